// Decode megakernel: one cooperative persistent launch runs every phase of a one-token
// decoder step.  One CTA per SM, ten warps:
//
//   warp 8       streams weight rows through a ring of 16 KB stages in shared memory, one
//                tensor-map copy per stage, a ring length ahead of the others and across phase
//                boundaries, because weights depend on nothing in the launch: HBM keeps streaming
//                while a phase waits for its activations.  The box of a copy is 32 reduction
//                elements x 8 or 16 rows x 16 or 32 such groups, which lands as the mma.sync fragments
//                of the lanes that read it: 16 bytes per lane, no bank conflicts, no padding, no
//                address arithmetic.  (Measured with nothing but the copies: 6.6 TB/s; 16-byte
//                copies by one producer warp reach 3.4 TB/s and by all warps 6.9, but then every
//                warp spends about as many instructions on copying as on everything else.)
//   warp 9       copies the phase records and resolves their addresses, up to four phases ahead.
//   warps 0..7   consumers: activation prologues (RMSNorm, embedding gather), the skinny GEMM on
//                mma.sync, epilogues, decode attention.
//
// Phases hand activations to one another through the plan's relay arena: every word of it that has
// not been written in this launch holds a pattern no result can have, so a consumer simply loads
// the activations it needs, in fragment layout, until they are there.  Data and "ready" are one L2
// round trip; there is no fence and no grid barrier.  (Records may also ask for plain
// tensors behind a counter, flagged cells, or a grid barrier.)  A warp multiplies a slice of the
// reduction for all rows of the CTA, with its slice of the activations in shared memory of its own,
// and the slices' products are added in shared memory in a fixed order.
//
// Replaces, for decode, the reference's generated persistent kernel
// (src/megabake/codegen.py:1634-1703), its sm100 swapAB GEMM bodies
// (src/megabake/bodies/cuda/sm100/cutlass_gemm.py:1072-1316), the split decode attention
// body (src/megabake/bodies/cuda/sm100/attention.py:909-1417), the generic row-reduction /
// map bodies used for RMSNorm, RoPE, residual and gated activations
// (src/megabake/bodies/cuda/generic.py:175-613) and the counting grid barrier
// (src/megabake/runtime.py:153-190).
#include <cuda.h>

#include <climits>
#include <cmath>
#include <cstring>
#include <mutex>

#include "mb_device.cuh"
#include "mb_kernels.h"

namespace mb {
namespace decode {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;        // consumers
constexpr int kAllThreads = kThreads + 64;   // and two more: weights, keys and values; phase records
constexpr int kRowTile = 8;          // ROW_TILE and K_CHUNK of a record describe the staging of
constexpr int kRowPad = 64;          // weight rows in units of these; the kernel's own stages are
constexpr int kStageBytes = 34816;   // 16 KB whatever they say
constexpr int kRingStage = 16384;    // 16 groups of 16 rows, 32 groups of 8, or 2 x 16 groups of 8
constexpr int kMaxStages = 8;
constexpr int kMapsPerPhase = 3;     // tensor maps: three weights, or keys and values
// Partial sums: two halves of 256 results (two blocks of 16 rows x 8 tokens; four blocks of 8) from
// eight slices each.
constexpr int kScratchBytes = 2 * 4 * kWarps * 512;
constexpr int kBarAll = 1;           // named barrier of the consumer warps
constexpr int kRopeRows = 8;         // batch rows the cos / sin table holds
constexpr int kEntryVectors = sizeof(PhaseEntry) / 16;
constexpr int kTraceEvents = 8;  // stamps per phase and CTA in the optional trace buffer

// How the key blocks of an attention phase are dealt over the CTAs, one piece of it: see
// find_segment.
struct Segment {
    int b, h, pair;
    int length;          // cached keys of the row
    int blk0, blk1;      // this CTA's blocks of the (row, kv head) pair
    int index, parts;    // which part of the pair this is, of how many
};

struct SharedCtl {
    unsigned long long full[kMaxStages];   // a stage's copies have landed
    unsigned long long empty[kMaxStages];  // all consumer warps have read it
    unsigned long long entry_ready[4];     // a phase record is there, its addresses resolved
    unsigned long long entry_done[4];      // all consumer warps are through with it
    volatile unsigned int issued;          // stages the producer armed
    unsigned long long limit_ns;           // bound of every wait of this launch
    unsigned long long relay_now, relay_next;  // this launch's half of the arena, the other half
    volatile int abort_flag;
    volatile int verdict;            // thread 0's decision at a grid barrier / at the end
    unsigned int tag_base;           // cells of phase q carry tag_base + q + 1 in this launch
    unsigned int calls;              // launches completed before this one
    Control* ctl;
    unsigned long long* trace;
    const PhaseEntry* entries;
    const CUtensorMap* maps;         // kMapsPerPhase per phase
    unsigned long long dyn[MB_MAX_DYNAMIC];
    int n_phases, stages, slots;
    unsigned long long rope_pos, rope_freq;  // what the cos / sin table was made from
    int rope_shape;
    float rope_scale;
    Segment segment[kWarps + 1];     // the segment a warp works on, the one the producer streams
    __align__(16) float norm_part[8][kWarps];      // sums of squares per activation row and slice
    float stat[kWarps][8][2];        // attention: (maximum, sum) per warp and head
    float exchange[2][kWarps][8];    // attention, exact mode: maxima and sums of the warps
    __align__(16) unsigned short new_row[2][256];  // rotated new key and new value of an item
    __align__(16) PhaseEntry entry[4];  // phase records ph .. ph + 3
};
constexpr int kCtlBytes = 5120;
constexpr int kFixedBytes = kCtlBytes + kScratchBytes;
static_assert(sizeof(SharedCtl) <= kCtlBytes, "control block too large");

// After the fixed part: the ring, the warps' slices (shared activations of GEMV phases; attention dumps
// its states there), the stream table, the cos / sin table.  Stages start on 1024-byte boundaries.
constexpr unsigned int kRingOffset = kFixedBytes;
static_assert(kRingOffset % 1024 == 0, "stages are 1024-byte aligned");
__host__ __device__ constexpr unsigned int slice_offset(int stages) {
    return kRingOffset + static_cast<unsigned int>(stages) * kRingStage;
}
__host__ __device__ constexpr unsigned int table_offset(int stages, int slots) {
    return slice_offset(stages) + static_cast<unsigned int>(kWarps * slots) * 512u;
}
__host__ __device__ constexpr unsigned int rope_offset(int stages, int slots, unsigned int n_phases) {
    return table_offset(stages, slots) +
           (n_phases * static_cast<unsigned int>(sizeof(StreamDesc)) + 127u) / 128u * 128u;
}

extern __shared__ __align__(1024) char g_smem[];
__device__ __forceinline__ SharedCtl* ctl_of() { return reinterpret_cast<SharedCtl*>(g_smem); }
__device__ __forceinline__ float* scratch_of() { return reinterpret_cast<float*>(g_smem + kCtlBytes); }
__device__ __forceinline__ StreamDesc* table_of() {
    return reinterpret_cast<StreamDesc*>(g_smem + table_offset(ctl_of()->stages, ctl_of()->slots));
}
__device__ __forceinline__ unsigned int* rope_of() {
    return reinterpret_cast<unsigned int*>(g_smem + rope_offset(ctl_of()->stages, ctl_of()->slots, ctl_of()->n_phases));
}

__device__ __forceinline__ void trace_stamp(int ph, int event) {
    SharedCtl* sc = ctl_of();
    if (threadIdx.x == 0 && sc->trace != nullptr)
        sc->trace[(static_cast<size_t>(blockIdx.x) * sc->n_phases + ph) * kTraceEvents + event] =
            global_timer_ns();
}

__device__ __forceinline__ unsigned long long resolve_address(unsigned long long v) {
    const SharedCtl* sc = ctl_of();
    if (v & kDynamicTag) return sc->dyn[v & (MB_MAX_DYNAMIC - 1)];  // the address comes with the launch
    if (v & kRelayTag) return sc->relay_now + (v & ~kRelayTag);
    return v;
}

// ---------------------------------------------------------------------------------------
// Bounded waits.  A wait gives up when the launch's limit has run out (status
// MB_ST_HANDOFF_TIMEOUT) or when this CTA or any other has recorded a fault; the caller goes on
// with whatever it has, without waiting any more, and the CTA leaves before the next phase or the one
// after that (consume_launch).
// ---------------------------------------------------------------------------------------
__device__ __noinline__ bool wait_gave_up(int ph, unsigned long long start) {
    SharedCtl* sc = ctl_of();
    if (sc->abort_flag) return true;
    if (peek_status(sc->ctl) != 0) {
        sc->abort_flag = 1;
        return true;
    }
    if (global_timer_ns() - start > sc->limit_ns) {
        record_status(sc->ctl, MB_ST_HANDOFF_TIMEOUT, ph, static_cast<int>(blockIdx.x));
        sc->abort_flag = 1;
        return true;
    }
    return false;
}

__device__ __noinline__ unsigned long long cell_wait(const void* src, unsigned int tag, int ph) {
    const unsigned long long start = global_timer_ns();
    for (unsigned int tries = 1;; ++tries) {
        const unsigned long long v = ld_cell(src);
        if (cell_tag(v) == tag) return v;
        if ((tries & 63u) == 0u && wait_gave_up(ph, start)) return v;
    }
}

__device__ __forceinline__ unsigned int relay_wait(const void* src, int ph) {
    const unsigned long long start = global_timer_ns();
    for (unsigned int tries = 1;; ++tries) {
        const unsigned int v = ld_relaxed_u32(src);
        if (v != kUnwritten) return v;
        if ((tries & 63u) == 0u && wait_gave_up(ph, start)) return 0u;
    }
}

// Finished-phase counters, for plans with hand-offs outside the relay arena: the count every CTA
// has to have reached once phase q of this launch is finished everywhere.
__device__ __forceinline__ unsigned int finished_target(const SharedCtl* sc, int q) {
    const unsigned int slot = static_cast<unsigned int>(q) & 3u;
    // phases of one launch that count on this slot, and how many of them up to phase q
    const unsigned int per_launch = (static_cast<unsigned int>(sc->n_phases) + 3u - slot) >> 2;
    return gridDim.x * (sc->calls * per_launch + (static_cast<unsigned int>(q) >> 2) + 1u);
}

// One thread: wait until every CTA has reported phase `q` finished.  The load is an acquire, so
// what those CTAs stored before a fenced report is visible to this thread afterwards (and,
// through a warp or CTA barrier, to the others).
__device__ __noinline__ void finished_wait(int ph, int q) {
    SharedCtl* sc = ctl_of();
    const unsigned int target = finished_target(sc, q);
    const unsigned int* counter = &sc->ctl->finished[q & 3].count;
    const unsigned long long start = global_timer_ns();
    for (unsigned int tries = 1;; ++tries) {
        unsigned int seen;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
        if (static_cast<int>(seen - target) >= 0) return;
        if ((tries & 63u) == 0u && wait_gave_up(ph, start)) return;
        __nanosleep(40);
    }
}

// ---------------------------------------------------------------------------------------
// Activations written earlier in the launch, eight bf16 values (16 bytes) at a time.
// ---------------------------------------------------------------------------------------
enum SourceKind { kPlain = 0, kRelay = 1, kCells = 2 };

__device__ __forceinline__ int source_kind(const PhaseEntry* E, bool cells) {
    return (E->modes & kModeInRelay) ? kRelay : (cells ? kCells : kPlain);
}

__device__ __forceinline__ bool unwritten(uint4 v) {
    return v.x == kUnwritten || v.y == kUnwritten || v.z == kUnwritten || v.w == kUnwritten;
}

// A pair of values as the arena may hold it: two NaNs that look like the blank pattern become two others.
__device__ __forceinline__ unsigned int as_written(unsigned int v) { return v == kUnwritten ? 0x7fff7fffu : v; }

// Eight values from four cells.
__device__ __noinline__ uint4 cells_load(const char* src, unsigned int tag, int ph) {
    unsigned int v[4];
    for (int i = 0; i < 4; ++i) {
        unsigned long long c = ld_cell(src + 8 * i);
        if (cell_tag(c) != tag) c = cell_wait(src + 8 * i, tag, ph);
        v[i] = cell_data(c);
    }
    return make_uint4(v[0], v[1], v[2], v[3]);
}

// Loads the first `count` of N vectors, vector i from `at(i)`, all of them in flight together, again
// and again until none has a word that is not written yet.  Whole warps only.  (No predicate per
// lane or vector: callers clamp addresses instead, because on the chain of a phase branches
// around single loads cost more than the loads.)
template <int N, typename At>
__device__ __forceinline__ void gather_source(uint4 (&x)[N], int count, bool relay, At at, int ph) {
    unsigned long long start = 0;
#pragma unroll 1
    for (unsigned int tries = 1;; ++tries) {
        bool missing = false;
#pragma unroll
        for (int i = 0; i < N; i += 2) {
            if (i >= count) break;
            x[i] = ld_relaxed_u4(at(i));
            if (i + 1 < N) x[i + 1] = ld_relaxed_u4(at(i + 1));
        }
        if (!relay) return;
#pragma unroll
        for (int i = 0; i < N; i += 2) {
            if (i >= count) break;
            missing |= unwritten(x[i]);
            if (i + 1 < N) missing |= unwritten(x[i + 1]);
        }
        if (!__any_sync(0xffffffffu, missing)) return;
        if ((tries & 63u) == 0u) {
            if (start == 0) start = global_timer_ns();
            if (__any_sync(0xffffffffu, wait_gave_up(ph, start))) return;  // garbage: the launch has failed
        }
    }
}

// Two neighbouring bf16 results on their way out: 4 bytes, or one cell.
__device__ __forceinline__ void store_result(char* base, size_t element, unsigned int packed,
                                             bool cells, unsigned int tag) {
    if (cells)
        st_cell(base + element * 4, packed, tag);
    else
        st_relaxed_u32(base + element * 2, packed);
}

// ---------------------------------------------------------------------------------------
// How the key blocks of an attention phase are dealt over the CTAs: every (row, kv head) pair is cut
// into `chunks` equal parts, and CTA c takes parts c, c + ctas, ... of all of them; the parts of a pair
// meet through the partial buffer.  The cut also decides, through the maxima a warp has seen, how the
// probabilities round.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ int row_length(const KvStream& d, int b) {
    if (d.len_count <= 1) return d.lens[0];
    if (d.batch <= 8) return d.lens[b];
    return __ldg(reinterpret_cast<const int*>(d.lengths) + b);
}

// Writes segment `which` of this CTA to `out`; false if there are fewer.
__device__ __noinline__ bool locate_segment(int ph, int which, Segment* out, bool writer) {
    const KvStream& d = table_of()[ph].kv;
    const int nc = d.chunks;
    int b, h, chunk, nblocks, parts;
    for (int item = blockIdx.x;; item += gridDim.x) {
        const int pair = item / nc;
        if (pair >= d.batch * d.kv_heads) return false;
        chunk = item - pair * nc;
        b = pair / d.kv_heads;
        h = pair - b * d.kv_heads;
        nblocks = (row_length(d, b) + 16) >> 4;
        parts = min(nc, nblocks);
        if (chunk < parts && which-- == 0) break;
    }
    if (writer) {
        out->b = b;
        out->h = h;
        out->pair = b * d.kv_heads + h;
        out->length = row_length(d, b);
        out->blk0 = static_cast<int>(static_cast<unsigned int>(chunk) * nblocks / parts);
        out->blk1 = static_cast<int>(static_cast<unsigned int>(chunk + 1) * nblocks / parts);
        out->index = chunk;
        out->parts = parts;
    }
    return true;
}
// The same for a consumer warp, into its own record.
__device__ __forceinline__ bool find_segment(int ph, int which) {
    __syncwarp();
    const bool found = locate_segment(ph, which, &ctl_of()->segment[threadIdx.x >> 5], (threadIdx.x & 31) == 0);
    __syncwarp();
    return found;
}

// log2 of the 16-key blocks per stage: 8 KB of keys.
__host__ __device__ constexpr int kv_shift(int head_dim) { return head_dim == 64 ? 2 : (head_dim == 128 ? 1 : 0); }

// Parts per pair (32 lanes): waves of parts over the CTAs times rounds of 16-key blocks over the eight
// warps, three rounds' worth of prologue and merge, and the fold, which grows with the parts.
__device__ __forceinline__ int choose_chunks(int pairs, int nblocks, int max_chunks) {
    int best_cost = INT_MAX, best = 1;
    for (int nc = (threadIdx.x & 31) + 1; nc <= min(max_chunks, nblocks); nc += 32) {
        const int waves = (pairs * nc + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
        const int rounds = ((nblocks + nc - 1) / nc + kWarps - 1) / kWarps;
        const int cost = 4 * waves * (rounds + 3) + nc;
        if (cost < best_cost) {
            best_cost = cost;
            best = nc;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const int cost = __shfl_xor_sync(0xffffffffu, best_cost, o), nc = __shfl_xor_sync(0xffffffffu, best, o);
        if (cost < best_cost || (cost == best_cost && nc < best)) {
            best_cost = cost;
            best = nc;
        }
    }
    return best;
}

// ---------------------------------------------------------------------------------------
// The weight ring.
// ---------------------------------------------------------------------------------------
// What a phase function hands on: the stage to consume next, its parity, and which half of the
// partial-sum scratch the next batch of rows uses.
struct Place {
    unsigned int stage, parity, flip;
};

// First virtual row of block `b` of this CTA, and the end of the segment it lies in: blocks never
// straddle two weight matrices.
__device__ __forceinline__ int block_row(const GemvStream& d, int b, int block_rows, int* end) {
    int lo = d.r0, hi = min(d.r1, d.n0);
    int blocks = hi > lo ? (hi - lo + block_rows - 1) / block_rows : 0;
    if (b >= blocks && hi < d.r1) {
        b -= blocks;
        lo = max(d.r0, d.n0);
        hi = min(d.r1, d.n01);
        blocks = hi > lo ? (hi - lo + block_rows - 1) / block_rows : 0;
        if (b >= blocks && hi < d.r1) {
            b -= blocks;
            lo = max(d.r0, d.n01);
            hi = d.r1;
        }
    }
    *end = hi;
    return lo + b * block_rows;
}
__device__ __forceinline__ int count_blocks(const GemvStream& d, int block_rows) {
    int total = 0;
    const int bounds[4] = {d.r0, min(max(d.n0, d.r0), d.r1), min(max(d.n01, d.r0), d.r1), d.r1};
    for (int s = 0; s < 3; ++s)
        total += (max(bounds[s + 1] - bounds[s], 0) + block_rows - 1) / block_rows;
    return total;
}

__device__ __forceinline__ void cp_async16(unsigned int dst_smem, unsigned long long src_gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_smem), "l"(src_gmem)
                 : "memory");
}
// All threads: orders what was stored to the tensor maps in global memory before this CTA's copies
// through them, which come after a barrier.
__device__ __noinline__ void acquire_maps(const CUtensorMap* maps, int count) {
    for (int m = threadIdx.x; m < count; m += kAllThreads)
        asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(maps + m) : "memory");
}
__device__ __forceinline__ void tma_load_3d(unsigned int dst, const CUtensorMap* map, int row, int group,
                                            unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
        "l"(map), "r"(0), "r"(row), "r"(group), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tma_load_5d(unsigned int dst, const CUtensorMap* map, int key, int head, int row,
                                            unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
        "l"(map), "r"(0), "r"(key), "r"(0), "r"(head), "r"(row), "r"(smem_u32(bar))
        : "memory");
}

// Producer: a warp walks the phases and fills stage after stage in the order they are consumed; its lanes stay
// together and one elected lane issues (elect_one says why).
__device__ __noinline__ void producer_loop() {
    SharedCtl* sc = ctl_of();
    const StreamDesc* table = table_of();
    const unsigned int ring = smem_u32(g_smem) + kRingOffset;
    const int lane = threadIdx.x & 31;
    int stage = 0;
    unsigned int parity = 1, issued = 0;
    // the next stage, once every warp has read what it held
    auto open_stage = [&](int ph) {
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(&sc->empty[stage], parity, &sc->abort_flag, 2 * sc->limit_ns))) {
            if (lane == 0) {
                if (!sc->abort_flag) record_status(sc->ctl, MB_ST_PIPE_TIMEOUT, ph, blockIdx.x);
                sc->abort_flag = 1;
            }
            return false;
        }
        ++issued;
        if (lane == 0) sc->issued = issued;
        return true;
    };
    auto next_stage = [&] {
        if (++stage == sc->stages) {
            stage = 0;
            parity ^= 1u;
        }
    };
    for (int ph = 0; ph < sc->n_phases; ++ph) {
        const CUtensorMap* maps = sc->maps + kMapsPerPhase * ph;
        if (table[ph].kind == kStreamKv) {
            const int head_dim = table[ph].kv.head_dim;
            Segment& seg = sc->segment[kWarps];
            for (int which = 0; locate_segment(ph, which, &seg, lane == 0); ++which) {
                __syncwarp();
                const int shift = kv_shift(head_dim);
                const unsigned int bytes = 8192;  // of the keys
                const int blk0 = seg.blk0, blk1 = seg.blk1, h = seg.h, b = seg.b;
                for (int blk = blk0; blk < blk1; blk += 1 << shift) {
                    if (!open_stage(ph)) return;
                    const unsigned int dst = ring + static_cast<unsigned int>(stage) * kRingStage;
                    if (elect_one()) {
                        mbar_arrive_expect_tx(&sc->full[stage], 2 * bytes);
                        tma_load_5d(dst, maps, blk * 16, h, b, &sc->full[stage]);
                        tma_load_5d(dst + bytes, maps + 1, blk * 16, h, b, &sc->full[stage]);
                    }
                    __syncwarp();
                    next_stage();
                }
                __syncwarp();
            }
            continue;
        }
        if (table[ph].kind != kStreamGemv) continue;
        const GemvStream& d = table[ph].gemv;
        const bool is_short = (d.shape & kShapeShort) != 0, paired = (d.shape & kShapePaired) != 0;
        const int block_rows = is_short || paired ? 8 : 16;
        const int step = is_short ? 32 : 16;  // groups per stage
        const char* nw = reinterpret_cast<const char*>(d.w_norm);
        if (nw != nullptr)  // every CTA reads the norm weights right after its wait: have them in L2
            for (int at = (static_cast<int>(blockIdx.x) + 8 * lane) * 128; at < d.row_bytes; at += 8 * 32 * 128)
                prefetch_l2(nw + at);
        for (int b = 0; b < d.nblocks; ++b) {
            int end;
            int row = block_row(d, b, block_rows, &end);
            const CUtensorMap* map = maps;
            if (row >= d.n01) {
                map = maps + 2;
                row -= d.n01;
            } else if (row >= d.n0) {
                map = maps + 1;
                row -= d.n0;
            }
            for (int g = 0; g < d.groups; g += step) {
                if (!open_stage(ph)) return;
                const unsigned int dst = ring + static_cast<unsigned int>(stage) * kRingStage;
                if (elect_one()) {
                    mbar_arrive_expect_tx(&sc->full[stage], kRingStage);
                    tma_load_3d(dst, map, row, g, &sc->full[stage]);
                    if (paired) tma_load_3d(dst + kRingStage / 2, maps + 1, row, g, &sc->full[stage]);
                }
                __syncwarp();
                next_stage();
            }
        }
    }
}
// After a fault: never leave while one of this CTA's copies is still in flight.  One thread.
__device__ __noinline__ void drain_ring() {
    SharedCtl* sc = ctl_of();
    const unsigned int stages = sc->stages, issued = sc->issued;
    for (unsigned int i = issued > stages ? issued - stages : 0u; i < issued; ++i)
        for (unsigned int tries = 0; tries < kDrainTryLimit; ++tries)
            if (mbar_try_wait(&sc->full[i % stages], (i / stages) & 1u)) break;
}

__device__ __forceinline__ uint4 lds128(unsigned int addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(addr)
                 : "memory");
    return v;
}
// Waits for a stage.  If the wait runs out the fault is recorded and the values are garbage; the
// CTA runs through the launch without waiting any more.  (No call: one in the loop of a phase costs
// more in spilled registers than the wait itself.)
__device__ __forceinline__ void ring_wait(unsigned int stage, unsigned int parity) {
    SharedCtl* sc = ctl_of();
    if (mbar_try_wait(&sc->full[stage], parity)) return;
    const unsigned long long start = global_timer_ns();
    for (unsigned int tries = 1; !mbar_try_wait(&sc->full[stage], parity); ++tries) {
        if ((tries & 127u) != 0u) continue;
        if (sc->abort_flag) return;
        if (global_timer_ns() - start > 2 * sc->limit_ns) {
            record_status(sc->ctl, MB_ST_PIPE_TIMEOUT, 0, blockIdx.x);
            sc->abort_flag = 1;
            return;
        }
    }
}
// The record of phase ph; it is there but for the first phases of a launch.  One thread, whose verdict all warps take
// (consume_launch).  False: a fault is on record in this CTA, or the record has not come in time.
__device__ __noinline__ bool await_record(int ph) {
    SharedCtl* sc = ctl_of();
    if (sc->abort_flag != 0) return false;
    if (mbar_wait_bounded(&sc->entry_ready[ph & 3], (ph >> 2) & 1, &sc->abort_flag, 2 * sc->limit_ns)) return true;
    if (sc->abort_flag == 0) record_status(sc->ctl, MB_ST_PIPE_TIMEOUT, ph, blockIdx.x);
    sc->abort_flag = 1;
    return false;
}
__device__ __forceinline__ bool record_ready(int ph) {
    SharedCtl* sc = ctl_of();
    return (sc->abort_flag == 0 && mbar_try_wait(&sc->entry_ready[ph & 3], (ph >> 2) & 1)) || await_record(ph);
}
// Hands the stage back once the warp has its values, and moves on.
__device__ __forceinline__ void ring_next(Place& s) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(&ctl_of()->empty[s.stage]);
    if (++s.stage == static_cast<unsigned int>(ctl_of()->stages)) {
        s.stage = 0;
        s.parity ^= 1u;
    }
}

// ---------------------------------------------------------------------------------------
// Skinny GEMM: out[row, n] = epilogue(prologue(x)[row, :] . W[n, :] + bias[n]), up to 8 rows.
// mma.sync m16n8k16 with the weight rows as A (16 of them, or 8 gate and 8 up rows) and the
// activation rows as B (n = row): one instruction takes 512 bytes of weights.  The reduction
// index is permuted identically in both, so that a lane's operand is 16 contiguous bytes per
// 32 elements.  The eight warps share a block of rows along K: of every stage a warp takes two
// groups of 32 elements (four where blocks have 8 rows).
//
// A phase is a chain -- activations arrive, norm, products, slices added, results leave -- on
// which every instruction counts, so whatever does not depend on the activations is done before
// they arrive.
// ---------------------------------------------------------------------------------------
// Element (virtual row) -> segment, and row inside it.
__device__ __forceinline__ int output_segment(const GemvStream& d, int& local) {
    if (local >= d.n01) {
        local -= d.n01;
        return 2;
    }
    if (local >= d.n0) {
        local -= d.n0;
        return 1;
    }
    return 0;
}
// Address of the packed pair that holds an element's residual.
__device__ __forceinline__ const char* residual_address(const PhaseEntry* E, int local, int tok) {
    const size_t index = static_cast<size_t>(tok) * E->rec.i[MB_GV_I_N0] + (local & ~1);
    const bool cells = (E->rec.i[MB_GV_I_CELLS] & MB_CELLS_RESIDUAL) && !(E->modes & kModeResidualRelay);
    return reinterpret_cast<const char*>(E->addr[MB_GV_S_RESIDUAL]) + index * (cells ? 4 : 2);
}

__device__ __forceinline__ float dot_self(uint4 v) {  // sum of squares of eight bf16 values
    const unsigned int w[4] = {v.x, v.y, v.z, v.w};
    float s = 0.f, t = 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        s = __fmaf_rn(lo_bf16(w[q]), lo_bf16(w[q]), s);
        t = __fmaf_rn(hi_bf16(w[q]), hi_bf16(w[q]), t);
    }
    return s + t;
}
// RMSNorm of eight values: the same roundings as normalise_vector, with the product of two bf16
// values -- exact in fp32 -- rounded by the packed multiplication.
__device__ __forceinline__ uint4 normalise_fast(uint4 x, uint4 w, float inv) {
    unsigned int xv[4] = {x.x, x.y, x.z, x.w};
    const unsigned int wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        asm("{\n\t.reg .b32 t;\n\tcvt.rn.bf16x2.f32 t, %1, %2;\n\tmul.rn.bf16x2 %0, t, %3;\n\t}"
            : "=r"(xv[q])
            : "f"(hi_bf16(xv[q]) * inv), "f"(lo_bf16(xv[q]) * inv), "r"(wv[q]));
    }
    return make_uint4(xv[0], xv[1], xv[2], xv[3]);
}

// What the code on a phase's chain needs of its record, read before the activations arrive.  (Every asm statement
// that touches memory makes the compiler read a record again.)
struct Recipe {
    int rows, prologue, epilogue, cells;
    unsigned int modes;
    bool gather;
};
__device__ __forceinline__ Recipe recipe_of(const PhaseEntry* E) {
    Recipe r;
    r.rows = E->rec.i[MB_GV_I_ROWS];
    r.prologue = E->rec.i[MB_GV_I_PROLOGUE];
    r.epilogue = E->rec.i[MB_GV_I_EPILOGUE];
    r.cells = E->rec.i[MB_GV_I_CELLS];
    r.modes = static_cast<unsigned int>(E->modes);
    r.gather = E->rec.i[MB_GV_I_GATHER] != 0;
    return r;
}

// A warp's share of the activations: of every stage the groups it multiplies ("vectors": 32
// elements of each row), R rows (the batch rounded up to a power of two) of four lanes x 16 bytes
// each, one after the other in the warp's own 8 KB (or 10 KB) of shared memory.  A lane brings and normalises the
// 16 bytes at slot * 512 + lane * 16 -- at small batches a slot holds several vectors, so that
// no lane works on a row that does not exist -- and reads them as B fragments of m16n8k16.  Reductions
// longer than the slice go chunk by chunk.
// A slice has 16 slots, or 20 in plans where that saves the chunks of some phase: five to eight rows
// of a reduction of 4,097 - 5,120 elements (0.5B shape, 8 rows, 4,096 keys: 1,060 -> 953 us).  The four
// take one stage from the ring, 1 % of a step where nobody needs them; more would take more.
constexpr int kSliceSlots = 16, kWideSlots = 20;
constexpr int kSliceBytes = kSliceSlots * 512;  // at least
struct Slice {
    int lp, rs;          // log2 of vectors per stage and of R
    int stages;          // of the whole reduction
    int chunk;           // stages per chunk
    int first, vectors, slots;   // of the current chunk
};
__device__ __forceinline__ Slice slice_of(int rows, const GemvStream& d, int c) {
    Slice v;
    v.lp = (d.shape & kShapeShort) ? 2 : 1;
    v.rs = rows > 2 ? (rows > 4 ? 3 : 2) : rows - 1;
    v.stages = (d.groups + (8 << v.lp) - 1) >> (3 + v.lp);
    v.chunk = (ctl_of()->slots * 8) >> (v.lp + v.rs);
    v.first = c * v.chunk << v.lp;
    v.vectors = min(v.chunk, v.stages - c * v.chunk) << v.lp;
    v.slots = ((v.vectors << v.rs) + 7) >> 3;
    return v;
}
// Group of 32 elements of vector `v` of warp `warp`, possibly past the end of the reduction.
__device__ __forceinline__ int vector_group(int lp, int warp, int v) {
    return ((v >> lp) << (3 + lp)) + (warp << lp) + (v & ((1 << lp) - 1));
}
__device__ __forceinline__ unsigned int slice_base(int warp) {
    return smem_u32(g_smem) + slice_offset(ctl_of()->stages) + warp * ctl_of()->slots * 512;
}
// Norm weights of the warp's vectors wait behind the slots where there is room (the usual case).
__device__ __forceinline__ bool weights_staged(const Slice& v) {
    return v.stages <= v.chunk && v.slots * 512 + v.vectors * 64 <= ctl_of()->slots * 512;
}
__device__ __forceinline__ void sts128(unsigned int addr, uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                 : "memory");
}

// N slots from `i` on (the last one repeated), all loads in flight together, again and again
// until no word is left unwritten.
template <int N>
__device__ __forceinline__ void fill_slots(const char* x, int lp, int warp, int vec, int step, int groups, int i,
                                           int slots, unsigned int out, bool relay, int ph) {
    uint4 v[N];
    unsigned int at[N];
#pragma unroll
    for (int q = 0; q < N; ++q)
        at[q] = static_cast<unsigned int>(min(vector_group(lp, warp, vec + min(i + q, slots - 1) * step), groups - 1)) * 64u;
    unsigned long long start = 0;
#pragma unroll 1
    for (unsigned int tries = 1;; ++tries) {
        bool missing = false;
#pragma unroll
        for (int q = 0; q < N; ++q) v[q] = ld_relaxed_u4(x + at[q]);
        if (!relay) break;
#pragma unroll
        for (int q = 0; q < N; ++q) missing |= unwritten(v[q]);
        if (!__any_sync(0xffffffffu, missing)) break;
        if ((tries & 63u) == 0u) {
            if (start == 0) start = global_timer_ns();
            if (__any_sync(0xffffffffu, wait_gave_up(ph, start))) break;  // garbage: the launch has failed
        }
    }
#pragma unroll
    for (int q = 0; q < N; ++q) sts128(out + static_cast<unsigned int>(min(i + q, slots - 1)) * 512u, v[q]);
}

// Activations kept as flagged cells.
__device__ __noinline__ void stage_cells(const int ph, const int c) {
    const SharedCtl* sc = ctl_of();
    const PhaseEntry* E = &sc->entry[ph & 3];
    const GemvStream& d = table_of()[ph].gemv;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const Slice sl = slice_of(E->rec.i[MB_GV_I_ROWS], d, c);
    const int row = min((lane >> 2) & ((1 << sl.rs) - 1), E->rec.i[MB_GV_I_ROWS] - 1);
    const char* x = reinterpret_cast<const char*>(E->addr[MB_GV_S_X]) + (lane & 3) * 32 +
                    static_cast<size_t>(row) * d.row_bytes * 2;
    const unsigned int tag = sc->tag_base + static_cast<unsigned int>(E->rec.i[MB_GV_I_X_SOURCE]) + 1u;
#pragma unroll 1
    for (int i = 0; i < sl.slots; ++i) {
        const int v = sl.first + (lane >> 2 >> sl.rs) + i * (8 >> sl.rs);
        sts128(slice_base(warp) + lane * 16 + i * 512,
               cells_load(x + static_cast<size_t>(min(vector_group(sl.lp, warp, v), d.groups - 1)) * 128, tag, ph));
    }
}

// Gathered rows, in the slice as they are in the table: the embedding scale, and the copy that the residual stream
// needs.  (Out of line: one phase of a launch.)
__device__ __noinline__ void finish_gather(const int ph, const int c, const bool store) {
    const SharedCtl* sc = ctl_of();
    const PhaseEntry* E = &sc->entry[ph & 3];
    const GemvStream& d = table_of()[ph].gemv;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gid = lane >> 2, tq = lane & 3;
    const Recipe rc = recipe_of(E);
    const Slice sl = slice_of(rc.rows, d, c);
    const int row = min(gid & ((1 << sl.rs) - 1), rc.rows - 1);
    const int vec = sl.first + (gid >> sl.rs), step = 8 >> sl.rs;
    const int groups = d.groups, row_bytes = d.row_bytes, flags = rc.cells;
    const unsigned int out = slice_base(warp) + lane * 16;
    // embedding scale; the residual stream needs the un-normalised rows
    const float scale = E->rec.f[MB_GV_F_EMBED_SCALE];
    char* keep = reinterpret_cast<char*>(E->addr[MB_GV_S_XSTORE]);
    const bool as_cells = (flags & MB_CELLS_XSTORE) && !(rc.modes & kModeStoreRelay);
    const unsigned int tag = sc->tag_base + static_cast<unsigned int>(ph) + 1u;
    const bool mine = store && E->rec.i[MB_GV_I_STORE_X] && blockIdx.x == 0 && row == (gid & ((1 << sl.rs) - 1));
#pragma unroll 1
    for (int i = 0; i < sl.slots; ++i) {
        const int g = vector_group(sl.lp, warp, vec + i * step);
        uint4 v = lds128(out + i * 512);
        if (scale != 0.f) {
            v = scale_vector(v, scale);
            sts128(out + i * 512, v);
        }
        if (rc.modes & kModeStoreRelay)  // rows of the table as they are: the one thing not converted
            v = make_uint4(as_written(v.x), as_written(v.y), as_written(v.z), as_written(v.w));
        if (mine && g < groups) {
            const size_t e = static_cast<size_t>(row) * (row_bytes / 2) + g * 32 + 8 * tq;
            store_result(keep, e, v.x, as_cells, tag);
            store_result(keep, e + 2, v.y, as_cells, tag);
            store_result(keep, e + 4, v.z, as_cells, tag);
            store_result(keep, e + 6, v.w, as_cells, tag);
        }
    }
}

// Brings chunk `c` of the warp's slice to shared memory, un-normalised, once its producers have
// written it; `store`: also hand on the gathered rows.  Returns this lane's part of its row's sum of
// squares when the phase normalises.
__device__ __forceinline__ float stage_slice(const int ph, const int c, const bool store, const Recipe& rc,
                                             const Slice& sl, const unsigned int base, const int groups,
                                             const int row_bytes) {
    SharedCtl* sc = ctl_of();
    const PhaseEntry* E = &sc->entry[ph & 3];
    const GemvStream& d = table_of()[ph].gemv;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gid = lane >> 2, tq = lane & 3;
    const int row = min(gid & ((1 << sl.rs) - 1), rc.rows - 1);
    const int vec = sl.first + (gid >> sl.rs), step = 8 >> sl.rs;
    const bool gather = rc.gather;
    const int flags = rc.cells;
    const bool relay = !gather && (rc.modes & kModeInRelay);
    const bool cells = !gather && !relay && (flags & MB_CELLS_X);
    const bool norm = rc.prologue != MB_PRO_NONE;
    const unsigned int out = base + lane * 16;
    __syncwarp();
    if (norm && weights_staged(sl)) {
        const unsigned long long w_norm = d.w_norm;
        const unsigned int end = base + sc->slots * 512;
        for (int v = gid; v < sl.vectors; v += 8)
            cp_async16(end - (sl.vectors - v) * 64 + tq * 16,
                       w_norm + min(vector_group(sl.lp, warp, v), groups - 1) * 64 + tq * 16);
    }
    const char* x = reinterpret_cast<const char*>(E->addr[MB_GV_S_X]) + 16 * tq;
    if (gather) {
        long long id = reinterpret_cast<const long long*>(E->addr[MB_GV_S_IDS])[row];
        if (id < 0 || id >= E->rec.i[MB_GV_I_VOCAB]) {
            record_status(sc->ctl, MB_ST_TOKEN_RANGE, ph, blockIdx.x);
            id = 0;
        }
        x += static_cast<size_t>(id) * row_bytes;
    } else {
        x += static_cast<size_t>(row) * row_bytes;
    }
    if (rc.modes & kModeWait) {
        if (lane == 0) finished_wait(ph, E->rec.i[MB_GV_I_X_SOURCE]);
        __syncwarp();
    }
    if (cells) {
        stage_cells(ph, c);
        __syncwarp();
    } else {
        int i = 0;
#pragma unroll 1
        for (; sl.slots - i > 4; i += 8)
            fill_slots<8>(x, sl.lp, warp, vec, step, groups, i, sl.slots, out, relay, ph);
        if (sl.slots - i == 1)
            fill_slots<1>(x, sl.lp, warp, vec, step, groups, i, sl.slots, out, relay, ph);
        else if (sl.slots > i)
            fill_slots<4>(x, sl.lp, warp, vec, step, groups, i, sl.slots, out, relay, ph);
    }
    if (gather) {
        finish_gather(ph, c, store);
    }
    float ss = 0.f;
    if (norm) {
#pragma unroll 4
        for (int i = 0; i < sl.slots; ++i) {
            const float part = dot_self(lds128(out + i * 512));
            ss += vector_group(sl.lp, warp, vec + i * step) < groups ? part : 0.f;
        }
    }
    __syncwarp();
    return ss;
}

// Normalises the staged chunk in place.  `ss`: the warp-summed squares are in norm_part.
__device__ __forceinline__ void normalise_slice(const int ph, const int kind, const Slice& sl, const unsigned int base,
                                                const int groups, const int row_bytes, const float eps) {
    SharedCtl* sc = ctl_of();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gid = lane >> 2, tq = lane & 3;
    const int row = gid & ((1 << sl.rs) - 1), step = 8 >> sl.rs;
    const float4 lo = *reinterpret_cast<const float4*>(&sc->norm_part[row][0]);
    const float4 hi = *reinterpret_cast<const float4*>(&sc->norm_part[row][4]);
    const float total = ((lo.x + lo.y) + (lo.z + lo.w)) + ((hi.x + hi.y) + (hi.z + hi.w));
    const float inv = 1.0f / sqrtf(total / static_cast<float>(row_bytes / 2) + eps);
    const unsigned int out = base + lane * 16;
    const bool staged = weights_staged(sl);
    const char* w = staged ? g_smem + slice_offset(sc->stages) + (warp + 1) * sc->slots * 512 - sl.vectors * 64
                           : reinterpret_cast<const char*>(table_of()[ph].gemv.w_norm);
    w += tq * 16;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    const int vec = gid >> sl.rs;
#pragma unroll 1
    for (int i = 0; i < sl.slots; ++i) {
        const int v = vec + i * step;
        const int at = staged ? min(v, sl.vectors - 1)
                              : min(vector_group(sl.lp, warp, sl.first + v), groups - 1);
        const uint4 nw = *reinterpret_cast<const uint4*>(w + at * 64);
        const uint4 x = lds128(out + i * 512);
        sts128(out + i * 512,
               kind == MB_PRO_RMS_LLAMA ? normalise_fast(x, nw, inv) : normalise_vector(x, nw, inv, kind));
    }
    __syncwarp();
}

// The same out of line, for slices of several chunks.
__device__ __noinline__ float stage_chunk(int ph, int c, bool store) {
    const GemvStream& d = table_of()[ph].gemv;
    const Recipe rc = recipe_of(&ctl_of()->entry[ph & 3]);
    return stage_slice(ph, c, store, rc, slice_of(rc.rows, d, c), slice_base(threadIdx.x >> 5), d.groups, d.row_bytes);
}
__device__ __noinline__ void normalise_chunk(int ph, int c) {
    const GemvStream& d = table_of()[ph].gemv;
    const PhaseEntry* E = &ctl_of()->entry[ph & 3];
    normalise_slice(ph, E->rec.i[MB_GV_I_PROLOGUE], slice_of(E->rec.i[MB_GV_I_ROWS], d, c),
                    slice_base(threadIdx.x >> 5), d.groups, d.row_bytes, E->rec.f[MB_GV_F_EPS]);
}

// The element of a batch of blocks that a thread finishes.
struct Result {
    int vrow, tok;               // virtual row (INT_MAX: none), activation row
    unsigned int residual;       // the packed pair that holds its residual
    float bias;
    char* out;                   // where an even row's pair goes
};
// `lr`: log2 of the rows of a block, 3 or 4; a block has 8 << lr results.
__device__ __forceinline__ Result request_result(const PhaseEntry* E, const GemvStream& d, const Recipe& rc, int lr,
                                                 int block) {
    const int t = threadIdx.x;
    Result r;
    r.vrow = INT_MAX;
    r.tok = t & 7;
    r.residual = kUnwritten;
    r.bias = 0.f;
    r.out = nullptr;
    const int b = block + (t >> (3 + lr));
    if (b < d.nblocks && r.tok < rc.rows) {
        int end;
        const int vrow = block_row(d, b, 1 << lr, &end) + (t >> 3 & ((1 << lr) - 1));
        if (vrow < end) {
            r.vrow = vrow;
            int local = vrow;
            const int seg = output_segment(d, local);
            const unsigned short* bias = reinterpret_cast<const unsigned short*>(E->addr[MB_GV_S_BIAS0 + seg]);
            if (bias != nullptr) r.bias = bf16_bits_to_float(__ldg(bias + local));
            // (a plain one of a phase that waits may not have been written yet: finish_result loads it)
            if (rc.epilogue == MB_EPI_RESIDUAL &&
                ((rc.modes & kModeResidualRelay) || !((rc.cells & MB_CELLS_RESIDUAL) || (rc.modes & kModeWait))))
                r.residual = ld_relaxed_u32(residual_address(E, vrow, r.tok));
            const bool out_cells = (rc.cells & MB_CELLS_OUT) != 0 && !(rc.modes & kModeOutRelay);
            r.out = reinterpret_cast<char*>(E->addr[MB_GV_S_OUT0 + seg]) +
                    (static_cast<size_t>(r.tok) * E->rec.i[MB_GV_I_N0 + seg] + local) * (out_cells ? 4 : 2);
        }
    }
    return r;
}

// The same out of line, for the blocks after the first.
__device__ __noinline__ Result next_result(int ph, int lr, int block) {
    const PhaseEntry* E = &ctl_of()->entry[ph & 3];
    return request_result(E, table_of()[ph].gemv, recipe_of(E), lr, block);
}

// The residual where it was not there when it was asked for.  (Out of line: it is there by then.)
__device__ __noinline__ unsigned int late_residual(int ph, int vrow, int tok) {
    const SharedCtl* sc = ctl_of();
    const PhaseEntry* E = &sc->entry[ph & 3];
    const char* at = residual_address(E, vrow, tok);
    if (E->modes & kModeResidualRelay) return relay_wait(at, ph);
    if (E->rec.i[MB_GV_I_CELLS] & MB_CELLS_RESIDUAL)
        return cell_data(cell_wait(at, sc->tag_base + static_cast<unsigned int>(E->rec.i[MB_GV_I_RES_SOURCE]) + 1u, ph));
    return ld_relaxed_u32(at);  // plain, of a phase that waits: stage_slice has waited for it
}

// Adds the slices of a thread's element, in slice order, runs the epilogue and stores the result
// together with its neighbour's (the odd row of a pair sits eight lanes further on).
__device__ __forceinline__ void finish_result(const Recipe& rc, const int ph, const int lr, const bool paired,
                                              const float* batch, Result r) {
    const int t = threadIdx.x;
    const float* part = batch + (t >> (3 + lr)) * (kWarps * 128) + (t & ((8 << lr) - 1));
    float v[kWarps];
#pragma unroll
    for (int w = 0; w < kWarps; ++w) v[w] = part[w * 128];
    const float sum = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
    const bool live = r.vrow != INT_MAX;
    float y = bf16_round(sum + r.bias);
    if (paired) {
#pragma unroll
        for (int w = 0; w < kWarps; ++w) v[w] = part[w * 128 + 64];
        const float up = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
        const float act = sigmoid_product(y, rc.epilogue == MB_EPI_SILU_MUL ? y : gelu_exponent(y));
        y = bf16_round(act) * bf16_round(up);
    } else if (rc.epilogue == MB_EPI_RESIDUAL) {
        const bool asked = (rc.modes & kModeResidualRelay) || !((rc.cells & MB_CELLS_RESIDUAL) || (rc.modes & kModeWait));
        // in the relay arena the blank pattern says that it was not there yet; elsewhere it may be a value
        if (live && (!asked || (r.residual == kUnwritten && (rc.modes & kModeResidualRelay))))
            r.residual = late_residual(ph, r.vrow, r.tok);
        y = (r.vrow & 1 ? hi_bf16(r.residual) : lo_bf16(r.residual)) + y;
    }
    const float other = __shfl_xor_sync(0xffffffffu, y, 8);
    if (live && (r.vrow & 1) == 0) {
        const unsigned int both = pack_bf16(y, other);
        if ((rc.cells & MB_CELLS_OUT) != 0 && !(rc.modes & kModeOutRelay))
            st_cell(r.out, both, ctl_of()->tag_base + static_cast<unsigned int>(ph) + 1u);
        else
            st_relaxed_u32(r.out, both);
    }
}

// SHORT: blocks of 8 rows, 32 groups per stage (a CTA's rows fit one block, or few); else 16 rows,
// or 8 gate and 8 up rows, 16 groups per stage.  (One body for all three shapes, told apart at run time, is 37 KB
// less code and slower: 1B 673 -> 695 us, 1.7B with 8 rows 3,520 -> 3,700.)
// WHOLE: the slices fit their place (host rule, kShapeWhole).
template <bool SHORT, bool WHOLE>
__device__ __noinline__ Place gemv_phase(const int ph, Place s) {
    SharedCtl* sc = ctl_of();
    const PhaseEntry* E = &sc->entry[ph & 3];
    const GemvStream& d = table_of()[ph].gemv;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nblocks = d.nblocks;
    const bool paired = !SHORT && (d.shape & kShapePaired);
    const Recipe rc = recipe_of(E);
    const bool norm = rc.prologue != MB_PRO_NONE;
    const int lr = SHORT || paired ? 3 : 4;
    const int groups = d.groups, row_bytes = d.row_bytes;
    const float eps = E->rec.f[MB_GV_F_EPS];
    const unsigned int base = slice_base(warp);
    Result result = request_result(E, d, rc, lr, 0);

    const Slice sl = slice_of(rc.rows, d, 0);
    float ss = 0.f;
    if (WHOLE) {
        ss = stage_slice(ph, 0, true, rc, sl, base, groups, row_bytes);
    } else if (norm) {
#pragma unroll 1
        for (int c = 0; c * sl.chunk < sl.stages; ++c) ss += stage_chunk(ph, c, true);
    }
    if (norm) {
        ss += __shfl_xor_sync(0xffffffffu, ss, 1);
        ss += __shfl_xor_sync(0xffffffffu, ss, 2);
        if (sl.rs < 3) ss += __shfl_xor_sync(0xffffffffu, ss, 16);
        if (sl.rs < 2) ss += __shfl_xor_sync(0xffffffffu, ss, 8);
        if (sl.rs < 1) ss += __shfl_xor_sync(0xffffffffu, ss, 4);
        if ((lane & 3) == 0) sc->norm_part[lane >> 2][warp] = ss;
        named_barrier(kBarAll, kThreads);
        if (WHOLE) normalise_slice(ph, rc.prologue, sl, base, groups, row_bytes, eps);
    }
    trace_stamp(ph, 1);

    // ---- blocks of rows
    constexpr int per = SHORT ? 4 : 2;
    float* batch = scratch_of() + s.flip * (kScratchBytes / 8);
    const unsigned int piece_step = SHORT || paired ? 512u : 1024u;
    const unsigned int piece_half = paired ? kRingStage / 2 : 512u;
    const unsigned int lane_ring = smem_u32(g_smem) + kRingOffset + lane * 16 + warp * per * piece_step;
    const unsigned int lane_x = base + (lane & ((4 << sl.rs) - 1)) * 16;
    const unsigned int x_step = 64u << sl.rs;
    int in_batch = 0;
#pragma unroll 1
    for (int b = 0; b < nblocks; ++b) {
        float acc[2][4];
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[0][q] = acc[1][q] = 0.f;
#pragma unroll 1
        for (int c = 0; WHOLE ? c == 0 : c * sl.chunk < sl.stages; ++c) {
            if (!WHOLE) {
                stage_chunk(ph, c, !norm && b == 0);
                if (norm) normalise_chunk(ph, c);
            }
            unsigned int at = lane_x;
#pragma unroll 1
            for (int left = WHOLE ? sl.stages : min(sl.chunk, sl.stages - c * sl.chunk); left > 0; --left) {
                const unsigned int piece = lane_ring + s.stage * kRingStage;
                uint4 x[per];
#pragma unroll
                for (int i = 0; i < per; ++i) x[i] = lds128(at + i * x_step);
                at += per * x_step;
                ring_wait(s.stage, s.parity);
                uint4 a[per], h[SHORT ? 1 : per];
#pragma unroll
                for (int i = 0; i < per; ++i) {
                    a[i] = lds128(piece + i * piece_step);
                    if (!SHORT) h[SHORT ? 0 : i] = lds128(piece + i * piece_step + piece_half);
                }
#pragma unroll
                for (int i = 0; i < per; ++i) {
                    if (SHORT) {
                        mma_bf16_16816(acc[0], a[i].x, 0u, a[i].y, 0u, x[i].x, x[i].y);
                        mma_bf16_16816(acc[1], a[i].z, 0u, a[i].w, 0u, x[i].z, x[i].w);
                    } else {
                        const uint4 g = h[SHORT ? 0 : i];
                        mma_bf16_16816(acc[0], a[i].x, g.x, a[i].y, g.y, x[i].x, x[i].y);
                        mma_bf16_16816(acc[1], a[i].z, g.z, a[i].w, g.w, x[i].z, x[i].w);
                    }
                }
                ring_next(s);
            }
        }
        float* cell = batch + (in_batch * kWarps + warp) * 128 + lane * 2;
        *reinterpret_cast<float2*>(cell) = make_float2(acc[0][0] + acc[1][0], acc[0][1] + acc[1][1]);
        if (!SHORT)
            *reinterpret_cast<float2*>(cell + 64) = make_float2(acc[0][2] + acc[1][2], acc[0][3] + acc[1][3]);
        if ((++in_batch << lr) == kThreads / 8 || b + 1 == nblocks) {
            named_barrier(kBarAll, kThreads);
            finish_result(rc, ph, lr, paired, batch, result);
            if (b + 1 < nblocks) result = next_result(ph, lr, b + 1);
            s.flip ^= 1u;
            batch = scratch_of() + s.flip * (kScratchBytes / 8);
            in_batch = 0;
        }
    }
    return s;
}

// ---------------------------------------------------------------------------------------
// Decode attention.  A CTA works on segments (the key blocks of one (row, kv head) it was dealt),
// which the producer streams through the weight ring ahead of the phase, 8 KB of keys and 8 KB of
// values per stage: the cached rows depend on nothing in the launch.  16-key block j of a segment belongs
// to warp j mod 8.  Queries (rows = heads of the group) are A and keys are B
// of the score product, transposed values (ldmatrix) A and the probabilities -- the score fragment as
// it stands -- B of the value product.  Every warp rotates the queries for itself: element pairs
// (i, i + D/2) sit in the same lane of two fragments.  The warp that owns the block with the new key
// rotates that key, appends both rows to the caches and puts them into the stage.
//
// Two softmax modes.  The reference normalises the probabilities in fp32 and rounds them to
// bf16 *before* the value product (ops/attention.py:82-84).
//   exact  (contexts of at most `exact_keys` <= 128 keys: one CTA per (row, kv head), at most one
//          16-key block per warp, scores stay in registers): row max and row sum are
//          exchanged through shared memory, then bf16(exp / sum) feeds the value product --
//          the reference's rounding.
//   online (longer contexts): online softmax per warp with unnormalised bf16 probabilities,
//          states merged across warps and, through tagged partials in global memory, across CTAs:
//          each part of a pair folds its share of the outputs from everybody's partials.  With
//          hundreds of keys the rounding of single probabilities averages out far below one
//          bf16 ulp of the result.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void ldmatrix_x4_trans(unsigned int (&r)[4], unsigned int addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}

// cos / sin of position `pos` for i = first, first + step ... < D/2, rounded to bf16 like the
// eager tables.
__device__ __noinline__ void fill_rope_row(unsigned int* table, const PhaseEntry* E, long long pos,
                                              int half_dim, int first, int step) {
    const void* invf = reinterpret_cast<const void*>(E->addr[MB_AT_S_INVFREQ]);
    const float rope_scale = E->rec.f[MB_AT_F_ROPE_SCALE];
    for (int i = first; i < half_dim; i += step) {
        const float f = E->rec.i[MB_AT_I_INVFREQ_BF16] != 0
                            ? bf16_bits_to_float(reinterpret_cast<const unsigned short*>(invf)[i])
                            : reinterpret_cast<const float*>(invf)[i];
        float sn, cn;
        sincosf(static_cast<float>(pos) * f, &sn, &cn);
        table[i] = pack_bf16(cn * rope_scale, sn * rope_scale);
    }
}

// The table of a launch's positions: the same for every layer of a model, made once.  All consumer threads.
__device__ __noinline__ void make_rope_table(int ph, int D, int shape) {
    SharedCtl* sc = ctl_of();
    const PhaseEntry* E = &sc->entry[ph & 3];
    const int batch = table_of()[ph].kv.batch;
    named_barrier(kBarAll, kThreads);
    const long long* pos = reinterpret_cast<const long long*>(E->addr[MB_AT_S_POS]);
    for (int b = threadIdx.x >> 5; b < batch; b += kWarps)
        fill_rope_row(rope_of() + b * (D / 2), E, pos[b], D / 2, threadIdx.x & 31, 32);
    if (threadIdx.x == 0) {
        sc->rope_pos = E->addr[MB_AT_S_POS];
        sc->rope_freq = E->addr[MB_AT_S_INVFREQ];
        sc->rope_shape = shape;
        sc->rope_scale = E->rec.f[MB_AT_F_ROPE_SCALE];
    }
    named_barrier(kBarAll, kThreads);
}

// Eight elements of the first half of a head and the eight they rotate with, in place.
__device__ __forceinline__ void rotate_vectors(uint4& lo, uint4& hi, const unsigned int* table,
                                               float q_scale) {
    unsigned int a[4] = {lo.x, lo.y, lo.z, lo.w}, b[4] = {hi.x, hi.y, hi.z, hi.w};
    const uint4 t0 = *reinterpret_cast<const uint4*>(table), t1 = *reinterpret_cast<const uint4*>(table + 4);
    const unsigned int t[8] = {t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w};
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const unsigned int c = __byte_perm(t[2 * w], t[2 * w + 1], 0x5410), x1 = a[w];
        const unsigned int sn = __byte_perm(t[2 * w], t[2 * w + 1], 0x7632), x2 = b[w];
        a[w] = sub_bf16_pair(mul_bf16_pair(x1, c), mul_bf16_pair(x2, sn));
        b[w] = add_bf16_pair(mul_bf16_pair(x2, c), mul_bf16_pair(x1, sn));
    }
    if (q_scale != 0.f && q_scale != 1.f) {
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            a[w] = pack_bf16(lo_bf16(a[w]) * q_scale, hi_bf16(a[w]) * q_scale);
            b[w] = pack_bf16(lo_bf16(b[w]) * q_scale, hi_bf16(b[w]) * q_scale);
        }
    }
    lo = make_uint4(a[0], a[1], a[2], a[3]);
    hi = make_uint4(b[0], b[1], b[2], b[3]);
}

// Queries (and the new key and value) kept as cells: one vector at a time, into the warp's slice.
__device__ __noinline__ void gather_cells(int ph, const char* qrow, const char* krow, const char* vrow, int groups,
                                          bool holder) {
    const SharedCtl* sc = ctl_of();
    const unsigned int tag =
        sc->tag_base + static_cast<unsigned int>(sc->entry[ph & 3].rec.i[MB_AT_I_QKV_SOURCE]) + 1u;
    const unsigned int keep = slice_base(threadIdx.x >> 5) + (threadIdx.x & 31) * 16;
#pragma unroll 1
    for (int i = 0; i < (holder ? 2 * groups + 1 : groups); ++i)
        sts128(keep + min(i, kSliceSlots - 1) * 512,
               cells_load(i < groups ? qrow + 128 * i : (i < 2 * groups ? krow + 128 * (i - groups) : vrow), tag, ph));
    __syncwarp();
}

template <int D, bool EXACT>
__device__ __noinline__ Place attention_phase(const int ph, Place s) {
    constexpr int DC = D / 32;                       // 32-element groups of the head dimension
    constexpr int DT = D / 16;                       // 16-row tiles of the value product
    constexpr int PS = 1 << kv_shift(D);             // 16-key blocks per stage
    constexpr unsigned int pitch = 1024u * PS;       // bytes of 32 dimensions of a stage's keys
    constexpr int DR = D < 128 ? D : 128;            // dimensions merged at a time
    constexpr int PR = DR + 4;                       // floats per dumped head: no bank conflicts
    static_assert(kSliceBytes >= 8 * PR * 4, "a dumped state fits the warp's slice");
    SharedCtl* sc = ctl_of();
    const PhaseEntry* E = &sc->entry[ph & 3];
    const KvStream& d = table_of()[ph].kv;
    unsigned int* rope = rope_of();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int gid = lane >> 2, tq = lane & 3;
    const int Hq = E->rec.i[MB_AT_I_HEADS], Hkv = E->rec.i[MB_AT_I_KV_HEADS];
    const int group = Hq / Hkv;  // query heads per kv head, <= 8
    const float scale = E->rec.f[MB_AT_F_SCALE];
    const int kind = source_kind(E, (E->rec.i[MB_AT_I_CELLS] & MB_CELLS_X) != 0);
    const unsigned int own_tag = sc->tag_base + static_cast<unsigned int>(ph) + 1u;
    const bool out_cells = (E->rec.i[MB_AT_I_CELLS] & MB_CELLS_OUT) != 0 && !(E->modes & kModeOutRelay);
    char* out = reinterpret_cast<char*>(E->addr[MB_AT_S_OUT]);
    const bool tabled = d.batch <= kRopeRows;

    // the slices still belong to the phase before until every warp is here
    named_barrier(kBarAll, kThreads);
    if (tabled) {
        const int shape = d.batch * 4096 + D * 2 + (E->rec.i[MB_AT_I_INVFREQ_BF16] ? 1 : 0);
        const bool fresh = sc->rope_pos == E->addr[MB_AT_S_POS] &&
                           sc->rope_freq == E->addr[MB_AT_S_INVFREQ] && sc->rope_shape == shape &&
                           sc->rope_scale == E->rec.f[MB_AT_F_ROPE_SCALE];
        if (__builtin_expect(!fresh, 0)) make_rope_table(ph, D, shape);
    }
    if (kind == kPlain && (E->rec.i[MB_AT_I_CELLS] & MB_CELLS_X_WAIT)) {
        if (lane == 0) finished_wait(ph, E->rec.i[MB_AT_I_QKV_SOURCE]);
        __syncwarp();
    }

    const unsigned int stages = static_cast<unsigned int>(sc->stages);
    const unsigned int ring = smem_u32(g_smem) + kRingOffset;
    float* dumps = reinterpret_cast<float*>(g_smem + slice_offset(sc->stages));
    const int dump_pitch = sc->slots * 128;  // floats
    const Segment& seg = sc->segment[warp];
    bool parted = false;  // some segment is one of several parts of its pair
    // One item a CTA at most, the usual case: its record still holds it when its parts are folded (a search takes
    // 1,000 cycles).
    const bool single = d.batch * d.kv_heads * d.chunks <= static_cast<int>(gridDim.x);
    for (int which = 0; find_segment(ph, which); ++which) {
        const int L = seg.length;
        const int b = seg.b, h = seg.h;
        const int blocks = seg.blk1 - seg.blk0;
        const bool has = warp < blocks;
        if (!tabled) {
            named_barrier(kBarAll, kThreads);
            fill_rope_row(rope, E, reinterpret_cast<const long long*>(E->addr[MB_AT_S_POS])[b], D / 2,
                          tid, kThreads);
            named_barrier(kBarAll, kThreads);
        }
        const unsigned int* row_rope = rope + (tabled ? b * (D / 2) : 0);

        // Queries, and in the warp whose stage includes the new key that key and its value: one
        // round trip for all of them (256-wide heads: one after the other, in as many registers).
        uint4 qf[DC];
        if (has) {
            const bool holder = seg.blk1 - 1 == (L >> 4) && ((blocks - 1) & (kWarps - 1)) == warp;
            const int elem = kind == kCells ? 4 : 2;
            const char* qrow = reinterpret_cast<const char*>(E->addr[MB_AT_S_Q]) +
                               (static_cast<size_t>(b) * Hq + h * group + min(gid, group - 1)) * D * elem +
                               8 * tq * elem;
            const size_t kv_row = (static_cast<size_t>(b) * Hkv + h) * D * elem;
            const char* krow = reinterpret_cast<const char*>(E->addr[MB_AT_S_K]) + kv_row + 8 * tq * elem;
            const char* vrow = reinterpret_cast<const char*>(E->addr[MB_AT_S_V]) + kv_row +
                               8 * (lane & (D / 8 - 1)) * elem;
            if (__builtin_expect(kind == kCells, 0)) gather_cells(ph, qrow, krow, vrow, DC, holder);
            const size_t at = ((static_cast<size_t>(b) * d.capacity + L) * Hkv + h) * D;
            auto place_new_row = [&](uint4 (&kn)[DC], uint4 vn) {
                if (gid == 0) {
#pragma unroll
                    for (int i = 0; i < DC / 2; ++i)
                        rotate_vectors(kn[i], kn[i + DC / 2], row_rope + 32 * i + 8 * tq, 0.f);
                    unsigned short* cache = reinterpret_cast<unsigned short*>(d.k) + at;
#pragma unroll
                    for (int i = 0; i < DC; ++i) {
                        *reinterpret_cast<uint4*>(cache + 32 * i + 8 * tq) = kn[i];
                        *reinterpret_cast<uint4*>(&sc->new_row[0][32 * i + 8 * tq]) = kn[i];
                    }
                }
                if (lane < D / 8) {
                    *reinterpret_cast<uint4*>(reinterpret_cast<unsigned short*>(d.v) + at + 8 * lane) = vn;
                    *reinterpret_cast<uint4*>(&sc->new_row[1][8 * lane]) = vn;
                }
            };
            if (D < 256 && kind != kCells) {
                uint4 in[2 * DC + 1], kn[DC];
                gather_source<2 * DC + 1>(
                    in, holder ? 2 * DC + 1 : DC, kind == kRelay,
                    [&](int i) { return i < DC ? qrow + 64 * i : (i < 2 * DC ? krow + 64 * (i - DC) : vrow); }, ph);
#pragma unroll
                for (int i = 0; i < DC; ++i) {
                    qf[i] = in[i];
                    kn[i] = in[DC + i];
                }
                if (holder) place_new_row(kn, in[2 * DC]);
            } else {
                if (holder) {
                    uint4 in[DC + 1], kn[DC];
                    const unsigned int kept = slice_base(warp) + lane * 16;
                    if (kind == kCells) {
#pragma unroll
                        for (int i = 0; i <= DC; ++i) in[i] = lds128(kept + min(DC + i, kSliceSlots - 1) * 512);
                        if (2 * DC >= kSliceSlots) {  // the slice holds one vector less: keys 0 .. DC - 2
                            in[DC] = in[DC - 1];
                            in[DC - 1] = cells_load(
                                krow + 128 * (DC - 1),
                                sc->tag_base + static_cast<unsigned int>(E->rec.i[MB_AT_I_QKV_SOURCE]) + 1u, ph);
                        }
                    } else {
                        gather_source<DC + 1>(
                            in, DC + 1, kind == kRelay, [&](int i) { return i < DC ? krow + 64 * i : vrow; }, ph);
                    }
#pragma unroll
                    for (int i = 0; i < DC; ++i) kn[i] = in[i];
                    place_new_row(kn, in[DC]);
                }
                if (kind == kCells) {
#pragma unroll
                    for (int i = 0; i < DC; ++i) qf[i] = lds128(slice_base(warp) + lane * 16 + i * 512);
                } else {
                    gather_source<DC>(qf, DC, kind == kRelay, [&](int i) { return qrow + 64 * i; }, ph);
                }
            }
#pragma unroll
            for (int i = 0; i < DC / 2; ++i)
                rotate_vectors(qf[i], qf[i + DC / 2], row_rope + 32 * i + 8 * tq, E->rec.f[MB_AT_F_Q_SCALE]);
            __syncwarp();
        }

        float m_run = -INFINITY, l_run = 0.f;
        // acc[t]: dims 16t + gid (+8), heads 2*tq (+1)
        float acc[DT][4];
#pragma unroll
        for (int t = 0; t < DT; ++t)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[t][q] = 0.f;
        unsigned int slot = s.stage, parity = s.parity;
        // The new row in its place and zeros after its value (0 * stale bits may be NaN), if block `q` of
        // the stage is the one.
        auto patch = [&](unsigned int base, int q, int first_key) {
            const int r0 = L - first_key;
            if (r0 >= 16) return;
            constexpr int C = D / 8;  // 16-byte pieces of a row
            const unsigned int keys = base + q * 1024u, values = keys + DC * pitch;
            for (int p = lane; p < 2 * C + (15 - r0) * C; p += 32) {
                const int r = p < 2 * C ? r0 : r0 + 1 + (p - 2 * C) / C, c = p & (C - 1);
                uint4 v = make_uint4(0u, 0u, 0u, 0u);
                if (p < 2 * C) v = *reinterpret_cast<const uint4*>(&sc->new_row[p < C ? 0 : 1][8 * c]);
                const unsigned int at = (c >> 2) * pitch + static_cast<unsigned int>(r) * 64u;
                sts128(p < C ? keys + at + (c & 3) * 16 : values + at + (((c & 3) ^ ((r >> 1) & 3)) << 4), v);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
        };
        // scores of block `q` of a stage: sv[2j + e] <-> head gid, key 8j + 2tq + e; bf16-rounded
        // product, scale applied in fp32, keys past the valid length masked
        auto block_scores = [&](unsigned int base, int q, int first_key, float (&sv)[4], bool masked) {
            float frag[2][4], frag2[2][4];  // two independent chains per tile, added at the end
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) frag[j][e] = frag2[j][e] = 0.f;
            unsigned int at = base + static_cast<unsigned int>(q) * 1024u + lane * 16;
#pragma unroll
            for (int i = 0; i < DC; ++i, at += pitch) {
                const uint4 k0 = lds128(at), k1 = lds128(at + 512);
                mma_bf16_16816(frag[0], qf[i].x, 0u, qf[i].y, 0u, k0.x, k0.y);
                mma_bf16_16816(frag[1], qf[i].x, 0u, qf[i].y, 0u, k1.x, k1.y);
                mma_bf16_16816(frag2[0], qf[i].z, 0u, qf[i].w, 0u, k0.z, k0.w);
                mma_bf16_16816(frag2[1], qf[i].z, 0u, qf[i].w, 0u, k1.z, k1.w);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float v = bf16_round(frag[j][e] + frag2[j][e]) * scale;
                    sv[2 * j + e] = !masked || first_key + 8 * j + 2 * tq + e <= L ? v : -INFINITY;
                }
        };
        // Lane's address for the value fragments of block 0: matrices (keys 0-7, dims 0-7), (keys
        // 0-7, dims 8-15), then keys 8-15; rows are 64 bytes, their four pieces permuted by the
        // tensor map so that eight rows touch all banks.
        const int vr = (lane & 7) + ((lane >> 4) << 3), vc = (lane >> 3) & 1;
        const unsigned int v_row = DC * pitch + static_cast<unsigned int>(vr) * 64u;
        const unsigned int v_even = v_row + ((vc ^ ((vr >> 1) & 3)) << 4);  // dims 0-15 of a group
        const unsigned int v_odd = v_row + (((vc + 2) ^ ((vr >> 1) & 3)) << 4);
        // acc += V^T P^T for one block; pb0 / pb1 = probabilities of keys (2tq, 2tq + 1) and
        // (8 + 2tq, 9 + 2tq) of head gid, packed bf16
        auto block_values = [&](unsigned int base, int q, unsigned int pb0, unsigned int pb1) {
            unsigned int at = base + static_cast<unsigned int>(q) * 1024u;
#pragma unroll
            for (int i = 0; i < DC; ++i, at += pitch) {
                unsigned int a[4], c[4];
                ldmatrix_x4_trans(a, at + v_even);
                ldmatrix_x4_trans(c, at + v_odd);
                mma_bf16_16816(acc[2 * i], a[0], a[1], a[2], a[3], pb0, pb1);
                mma_bf16_16816(acc[2 * i + 1], c[0], c[1], c[2], c[3], pb0, pb1);
            }
        };

        float sv[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        unsigned int vf[EXACT ? DT : 1][4];
        // Block j of the segment is warp j mod 8's, and every warp goes through every stage: the one
        // parity bit of a wait only tells the last two uses of a slot apart.
        // `last`: the new key, and keys past the valid length, can only be in a segment's last stage.  The loop over the
        // others is the shorter for it, which is what long contexts run in: 1.7B, 8 rows of 8,192 keys 3,425 -> 3,287 us.
        // (256-wide heads are the slower for the second copy of the body: 1,257 -> 1,280.)
        auto stage_of = [&](int j, bool last) {
            ring_wait(slot, parity);
            const int q = (warp - j) & (kWarps - 1);
            if (q < PS && j + q < blocks) {
                const unsigned int base = ring + slot * kRingStage;
                const int first_key = (seg.blk0 + j + q) * 16;
                if (last) patch(base, q, first_key);
                block_scores(base, q, first_key, sv, last);
                if (EXACT) {
                    // One block per warp at most.  The value fragments leave the ring before the
                    // warps meet, so that a ring shorter than the segment cannot stall the producer.
#pragma unroll
                    for (int i = 0; i < DC; ++i) {
                        ldmatrix_x4_trans(vf[EXACT ? 2 * i : 0], base + q * 1024u + i * pitch + v_even);
                        ldmatrix_x4_trans(vf[EXACT ? 2 * i + 1 : 0], base + q * 1024u + i * pitch + v_odd);
                    }
                } else {
                    float bmax = fmaxf(fmaxf(sv[0], sv[1]), fmaxf(sv[2], sv[3]));
                    bmax = fmaxf(bmax, __shfl_xor_sync(0xffffffffu, bmax, 1));
                    bmax = fmaxf(bmax, __shfl_xor_sync(0xffffffffu, bmax, 2));
                    if (__any_sync(0xffffffffu, bmax > m_run)) {  // a new maximum: rare after the first blocks
                        const float m_new = fmaxf(m_run, bmax);
                        const float alpha = expf(m_run - m_new);
                        l_run *= alpha;
                        m_run = m_new;
                        // rescale factors of the two heads this lane accumulates (columns 2tq, 2tq+1)
                        const float alpha0 = __shfl_sync(0xffffffffu, alpha, (2 * tq) * 4);
                        const float alpha1 = __shfl_sync(0xffffffffu, alpha, (2 * tq + 1) * 4);
#pragma unroll
                        for (int t = 0; t < DT; ++t) {
                            acc[t][0] *= alpha0;
                            acc[t][1] *= alpha1;
                            acc[t][2] *= alpha0;
                            acc[t][3] *= alpha1;
                        }
                    }
                    float pv[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) pv[e] = expf(sv[e] - m_run);
                    l_run += (pv[0] + pv[1]) + (pv[2] + pv[3]);
                    block_values(base, q, pack_bf16(pv[0], pv[1]), pack_bf16(pv[2], pv[3]));
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sc->empty[slot]);
            if (++slot == stages) {
                slot = 0;
                parity ^= 1u;
            }
        };
        int j = 0;
        if (!EXACT && D < 256) {
#pragma unroll 1
            for (; j + PS < blocks; j += PS) stage_of(j, false);
        }
#pragma unroll 1
        for (; j < blocks; j += PS) stage_of(j, true);
        s.stage = slot;
        s.parity = parity;
        if (EXACT) {
            float rmax = fmaxf(fmaxf(sv[0], sv[1]), fmaxf(sv[2], sv[3]));
            rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, 1));
            rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, 2));
            if (tq == 0) sc->exchange[0][warp][gid] = rmax;
            named_barrier(kBarAll, kThreads);
            float row_max = -INFINITY;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) row_max = fmaxf(row_max, sc->exchange[0][w][gid]);
            float ev[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) ev[q] = expf(sv[q] - row_max);  // 0 for masked keys
            float rsum = (ev[0] + ev[1]) + (ev[2] + ev[3]);
            rsum += __shfl_xor_sync(0xffffffffu, rsum, 1);
            rsum += __shfl_xor_sync(0xffffffffu, rsum, 2);
            if (tq == 0) sc->exchange[1][warp][gid] = rsum;
            named_barrier(kBarAll, kThreads);
            float row_sum = 0.f;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) row_sum += sc->exchange[1][w][gid];
            if (has) {  // normalised probabilities rounded to bf16, as the eager operator does
                const unsigned int pb0 = pack_bf16(ev[0] / row_sum, ev[1] / row_sum);
                const unsigned int pb1 = pack_bf16(ev[2] / row_sum, ev[3] / row_sum);
#pragma unroll
                for (int t = 0; t < DT; ++t) mma_bf16_16816(acc[t], vf[t][0], vf[t][1], vf[t][2], vf[t][3], pb0, pb1);
            }
            // already normalised: merge as plain sums (max 0, total weight 1)
            m_run = 0.f;
            l_run = (warp == 0 && tq == 0) ? 1.f : 0.f;
        }
        l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
        l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
        trace_stamp(ph, 5);

        // ---- merge the warp states: dumped DR dimensions at a time, added up in warp order
        if (tq == 0) {
            sc->stat[warp][gid][0] = m_run;
            sc->stat[warp][gid][1] = l_run;
        }
        if (seg.parts > 1) parted = true;
#pragma unroll
        for (int r = 0; r < D / DR; ++r) {
            if (r > 0) named_barrier(kBarAll, kThreads);
            __syncwarp();
            float* dump = dumps + warp * dump_pitch + gid;
#pragma unroll
            for (int t = 0; t < DR / 16; ++t) {
                const float(&v)[4] = acc[r * (DR / 16) + t];
                if (2 * tq < group) {
                    dump[(2 * tq) * PR + 16 * t] = v[0];
                    dump[(2 * tq) * PR + 16 * t + 8] = v[2];
                }
                if (2 * tq + 1 < group) {
                    dump[(2 * tq + 1) * PR + 16 * t] = v[1];
                    dump[(2 * tq + 1) * PR + 16 * t + 8] = v[3];
                }
            }
            named_barrier(kBarAll, kThreads);
            // Several outputs a thread (256-wide heads): the warps' weights are worked out once.
            constexpr bool kShared = D > DR;
            if (kShared && !EXACT && r == 0) {
                const int w = tid >> 3, head = tid & 7;
                if (tid < 8 * kWarps) {
                    float m_all = -INFINITY;
#pragma unroll
                    for (int q = 0; q < kWarps; ++q) m_all = fmaxf(m_all, sc->stat[q][head][0]);
                    sc->exchange[0][w][head] = __expf(sc->stat[w][head][0] - m_all);
                    if (w == 0) sc->exchange[1][0][head] = m_all;
                }
                named_barrier(kBarAll, kThreads);
            }
#pragma unroll 1
            for (int o = tid; o < group * (DR / 2); o += kThreads) {
                const int head = o / (DR / 2), dim = 2 * (o & (DR / 2 - 1));
                float m_all = -INFINITY, l_all = 0.f, y0 = 0.f, y1 = 0.f;
                if (EXACT) {  // normalised already: every weight is 1, and so is their sum
                    m_all = 0.f;
                } else if (kShared) {
                    m_all = sc->exchange[1][0][head];
                } else {
#pragma unroll
                    for (int w = 0; w < kWarps; ++w) m_all = fmaxf(m_all, sc->stat[w][head][0]);
                }
#pragma unroll
                for (int w = 0; w < kWarps; ++w) {
                    // weights between partial softmax states: no rounding point of the operator
                    // sits here, the fast exponential is accurate to 2^-21
                    const float wgt = EXACT ? 1.f : kShared ? sc->exchange[0][w][head]
                                              : __expf(sc->stat[w][head][0] - m_all);  // 0: a warp without a block
                    const float2 v =
                        *reinterpret_cast<const float2*>(dumps + w * dump_pitch + head * PR + dim);
                    if (!EXACT) l_all += sc->stat[w][head][1] * wgt;
                    y0 += v.x * wgt;
                    y1 += v.y * wgt;
                }
                const int column = r * DR + dim;
                if (seg.parts == 1) {
                    store_result(out, (static_cast<size_t>(b) * Hq + h * group + head) * D + column,
                                 EXACT ? pack_bf16(y0, y1) : pack_bf16(y0 / l_all, y1 / l_all), out_cells, own_tag);
                } else {
                    // cells of (fp32, tag): maximum, sum, D values per head
                    char* part = reinterpret_cast<char*>(E->addr[MB_AT_S_PARTIAL]) +
                                 ((static_cast<size_t>(seg.pair) * d.chunk_cap + seg.index) * group + head) *
                                     ((D + 2) * 8);
                    st_cell(part + (2 + column) * 8, __float_as_uint(y0), own_tag);
                    st_cell(part + (3 + column) * 8, __float_as_uint(y1), own_tag);
                    if (column == 0) {
                        st_cell(part, __float_as_uint(m_all), own_tag);
                        st_cell(part + 8, __float_as_uint(l_all), own_tag);
                    }
                }
            }
        }
        named_barrier(kBarAll, kThreads);  // slices and statistics are reused by the next segment
    }
    trace_stamp(ph, 7);

    // ---- fold the parts of the pairs this CTA has a part of: its share of their outputs.  Only
    // after ALL its partials are out, so no chain of CTAs waits for one another's folds.
    for (int which = 0; parted; ++which) {
        if (single ? which > 0 : !find_segment(ph, which)) break;
        if (seg.parts == 1) continue;
        const int total = group * (D / 2);  // pairs of neighbouring outputs
        const int lo = seg.index * total / seg.parts, hi = (seg.index + 1) * total / seg.parts;
        const char* base = reinterpret_cast<const char*>(E->addr[MB_AT_S_PARTIAL]) +
                           static_cast<size_t>(seg.pair) * d.chunk_cap * group * ((D + 2) * 8);
        // A thread takes up to eight parts of an output pair, four threads up to 32: the cells of all of
        // them are in flight together, again and again until none carries an older tag.  (One part a
        // thread, its four cells waited for one after the other, took 4.6 us on the 0.5B shape
        // and 9.7 on the 2B, after the last part was out; now 1.9 and 2.7.)
        // Only what is needed is asked for: a poll of all threads for eight parts each is 64 KB per CTA.
        const int lanes = seg.parts > 8 ? 4 : 1, j = tid & (lanes - 1);
        const int slots = seg.parts > 16 ? 8 : (seg.parts > 8 ? 4 : seg.parts);
        for (int o0 = lo; o0 + (tid & ~31) / lanes < hi; o0 += kThreads / lanes) {
            const int o = o0 + tid / lanes;
            const int head = min(o, hi - 1) / (D / 2), dim = 2 * (min(o, hi - 1) - head * (D / 2));
            const char* first = base + static_cast<size_t>(head) * ((D + 2) * 8);
            unsigned long long cm[8], cl[8], c0[8], c1[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) cm[i] = cl[i] = c0[i] = c1[i] = 0ull;
            unsigned long long start = 0;
#pragma unroll 1
            for (unsigned int tries = 1;; ++tries) {
                bool missing = false;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (i >= slots) break;
                    // a part that does not exist: the last one again, left out below
                    const int c = min(lanes == 1 ? i : j + 4 * (i & 3) + 16 * (i >> 2), seg.parts - 1);
                    const char* part = first + static_cast<size_t>(c) * group * ((D + 2) * 8);
                    ld_cell_pair(part, cm[i], cl[i]);
                    ld_cell_pair(part + (2 + dim) * 8, c0[i], c1[i]);
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (i >= slots) break;
                    missing |= cell_tag(cm[i]) != own_tag || cell_tag(cl[i]) != own_tag ||
                               cell_tag(c0[i]) != own_tag || cell_tag(c1[i]) != own_tag;
                }
                if (!__any_sync(0xffffffffu, missing)) break;
                if ((tries & 63u) == 0u) {
                    if (start == 0) start = global_timer_ns();
                    if (__any_sync(0xffffffffu, wait_gave_up(ph, start))) break;  // garbage: the launch has failed
                }
            }
            float m[8], mx = -INFINITY;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int c = lanes == 1 ? i : j + 4 * (i & 3) + 16 * (i >> 2);
                m[i] = c < seg.parts ? __uint_as_float(cell_data(cm[i])) : -INFINITY;
                mx = fmaxf(mx, m[i]);
            }
            for (int w = lanes >> 1; w > 0; w >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
            float den[8], s0[8], s1[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                // (not by a weight of zero: an infinity times zero is a NaN)
                const bool there = (lanes == 1 ? i : j + 4 * (i & 3) + 16 * (i >> 2)) < seg.parts;
                const float weight = m[i] == -INFINITY ? 0.f : expf(m[i] - mx);
                den[i] = there ? __uint_as_float(cell_data(cl[i])) * weight : 0.f;
                s0[i] = there ? __uint_as_float(cell_data(c0[i])) * weight : 0.f;
                s1[i] = there ? __uint_as_float(cell_data(c1[i])) * weight : 0.f;
            }
            // part c meets part c + 16, then c + 8, + 4, + 2, + 1, whoever holds them
#pragma unroll
            for (int w = 4; w > 0; w >>= 1)
#pragma unroll
                for (int i = 0; i < w; ++i) {
                    den[i] += den[i + w];
                    s0[i] += s0[i + w];
                    s1[i] += s1[i + w];
                }
            for (int w = lanes >> 1; w > 0; w >>= 1) {
                den[0] += __shfl_xor_sync(0xffffffffu, den[0], w);
                s0[0] += __shfl_xor_sync(0xffffffffu, s0[0], w);
                s1[0] += __shfl_xor_sync(0xffffffffu, s1[0], w);
            }
            if (j == 0 && o < hi)
                store_result(out, (static_cast<size_t>(seg.b) * Hq + seg.h * group + head) * D + dim,
                             pack_bf16(s0[0] / den[0], s1[0] / den[0]), out_cells, own_tag);
        }
    }
    return s;
}

// ---------------------------------------------------------------------------------------
// The kernel.
// ---------------------------------------------------------------------------------------
// Completes one stream record in shared memory for this CTA and this launch: its output rows, or
// the valid lengths and how the keys are dealt.  False: a length (`bad`) does not fit the cache.
__device__ __forceinline__ bool complete_stream(StreamDesc* desc, int* bad) {
    if (desc->kind == kStreamGemv) {
        GemvStream& d = desc->gemv;
        d.w_norm = resolve_address(d.w_norm);
        const int cta = blockIdx.x, q = d.r0, rem = d.r1;  // pairs of rows per CTA, and the rest
        d.r0 = 2 * (cta * q + min(cta, rem));
        d.r1 = d.r0 + 2 * (q + (cta < rem ? 1 : 0));
        d.nblocks = count_blocks(d, (d.shape & (kShapeShort | kShapePaired)) ? 8 : 16);
        return true;
    }
    if (desc->kind != kStreamKv) return true;
    KvStream& d = desc->kv;
    d.k = resolve_address(d.k);
    d.v = resolve_address(d.v);
    d.lengths = resolve_address(d.lengths);
    const int* lengths = reinterpret_cast<const int*>(d.lengths);
    const int count = d.len_count > 1 ? d.batch : 1;
    int longest = 0;
    bool fits = true;
    for (int r = 0; r < count; ++r) {
        const int L = *reinterpret_cast<const volatile int*>(lengths + r);
        if (L < 0 || L >= d.capacity) {
            fits = false;
            *bad = L;
        }
        if (r < 8) d.lens[r] = L;
        longest = max(longest, L);
    }
    if (!fits) return false;
    d.exact_keys = longest + 1 <= d.exact_keys ? 1 : 0;
    d.longest = longest;
    d.chunks = 1;
    return true;
}

// DIM: the head size of all attention phases of the plan (0: a mix of sizes, every body compiled
// in).  One kernel per head size keeps the code of a launch within the instruction caches and its
// loop operands in registers.
template <int D>
__device__ __forceinline__ Place attention_call(int ph, Place s) {
    return table_of()[ph].kv.exact_keys ? attention_phase<D, true>(ph, s) : attention_phase<D, false>(ph, s);
}
template <int DIM>
__device__ __forceinline__ Place run_attention(int ph, Place s) {
    if constexpr (DIM != 0) {
        return attention_call<DIM>(ph, s);
    } else {
        const int dim = table_of()[ph].kv.head_dim;
        if (dim == 64) return attention_call<64>(ph, s);
        if (dim == 128) return attention_call<128>(ph, s);
        return attention_call<256>(ph, s);
    }
}

// Start of a launch, all threads: control block, stream table, ring.  False: a fault is on record
// (now or from an earlier launch) and nothing may run.
__device__ __forceinline__ bool begin_launch(const KernelParams& p, const StreamDesc* streams, const void* maps,
                                             unsigned int tag_base, unsigned int parity,
                                             unsigned int calls) {
    SharedCtl* sc = ctl_of();
    StreamDesc* table = reinterpret_cast<StreamDesc*>(g_smem + table_offset(p.stages, p.slots));
    const int tid = threadIdx.x;
    for (int v = tid; v < p.n_phases * 6; v += kAllThreads)
        reinterpret_cast<uint4*>(table)[v] = reinterpret_cast<const uint4*>(streams)[v];
    if (tid == 0) {
        for (int i = 0; i < p.stages; ++i) {
            mbar_init(&sc->full[i], 1);
            mbar_init(&sc->empty[i], kWarps);
        }
        for (int i = 0; i < 4; ++i) {
            mbar_init(&sc->entry_ready[i], 1);
            mbar_init(&sc->entry_done[i], kWarps);
        }
        sc->issued = 0;
        mbar_init_fence();
        sc->abort_flag = peek_status(p.ctl) != 0 ? 1 : 0;  // a faulted plan runs nothing
        sc->limit_ns = static_cast<unsigned long long>(p.wait_limit_us) * 1000ull;
        sc->tag_base = tag_base;
        sc->calls = calls;
        sc->ctl = p.ctl;
        sc->trace = p.trace;
        sc->n_phases = p.n_phases;
        sc->stages = p.stages;
        sc->slots = p.slots;
        sc->maps = reinterpret_cast<const CUtensorMap*>(maps);
        sc->entries = p.entries;
        for (int i = 0; i < MB_MAX_DYNAMIC; ++i) sc->dyn[i] = p.dyn[i];
        sc->relay_now = p.relay + (parity & 1u) * p.relay_bytes;
        sc->relay_next = p.relay + ((parity & 1u) ^ 1u) * p.relay_bytes;
        sc->rope_pos = sc->rope_freq = 0;
        sc->rope_shape = -1;
    }
    __syncthreads();
    if (sc->abort_flag) return false;
    for (int ph = tid; ph < p.n_phases; ph += kAllThreads) {
        int bad = 0;
        if (!complete_stream(table + ph, &bad)) {
            record_status(p.ctl, MB_ST_KV_OVERFLOW, ph, bad);
            sc->abort_flag = 1;
        }
    }
    __syncthreads();
    for (int ph = tid >> 5; ph < p.n_phases; ph += kAllThreads / 32) {
        if (table[ph].kind != kStreamKv || table[ph].kv.exact_keys) continue;
        KvStream& d = table[ph].kv;
        const int chunks = choose_chunks(d.batch * d.kv_heads, (d.longest + 16) >> 4, d.chunk_cap);
        if ((tid & 31) == 0) d.chunks = chunks;
    }
    __syncthreads();
    return sc->abort_flag == 0;
}

// One 16-byte vector of a phase entry, addresses resolved.  addr[] starts in the upper half of
// vector kFirst; the last vector's upper half is `modes`.
__device__ __forceinline__ uint4 resolve_vector(uint4 v, int index) {
    constexpr int kFirst = offsetof(PhaseEntry, addr) / 16;
    static_assert(offsetof(PhaseEntry, addr) % 16 == 8 && offsetof(PhaseEntry, modes) % 16 == 8,
                  "addr[] starts mid-vector and modes ends one");
    if (index > kFirst) {
        const unsigned long long a =
            resolve_address(v.x | (static_cast<unsigned long long>(v.y) << 32));
        v.x = static_cast<unsigned int>(a);
        v.y = static_cast<unsigned int>(a >> 32);
    }
    if (index >= kFirst && index < kEntryVectors - 1) {
        const unsigned long long a =
            resolve_address(v.z | (static_cast<unsigned long long>(v.w) << 32));
        v.z = static_cast<unsigned int>(a);
        v.w = static_cast<unsigned int>(a >> 32);
    }
    return v;
}

// Phase entries: a warp of its own copies the records and resolves their addresses, up to four phases ahead of
// the consumers.  (Warp 0 did it at the start of each phase: 2,500 cycles on the chain of every phase of
// the 135M shape with a bulk copy, whose proxy fence waited for the results the warp had just stored, 1,700
// without, most of them instructions that are not in the cache after a phase.)
__device__ __noinline__ void entry_loop() {
    SharedCtl* sc = ctl_of();
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int ph = 0; ph < sc->n_phases; ++ph) {
        if (ph >= 4 && !__all_sync(0xffffffffu, mbar_wait_bounded(&sc->entry_done[ph & 3], ((ph >> 2) - 1) & 1,
                                                                 &sc->abort_flag, 8 * sc->limit_ns)))
            return;  // a fault is on record, or soon will be: the consumers have limits of their own
        if (lane < kEntryVectors) {
            uint4* v = reinterpret_cast<uint4*>(&sc->entry[ph & 3]) + lane;
            *v = resolve_vector(ld_cg_u4(reinterpret_cast<const uint4*>(sc->entries + ph) + lane), lane);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sc->entry_ready[ph & 3]);
    }
}

// The end of a phase in plans with hand-offs outside the relay arena: counters and the grid barrier.  False: the
// barrier failed.
__device__ __noinline__ bool close_phase(Control* ctl, int ph, int flags, bool meet, bool counters,
                                         unsigned int generation) {
    SharedCtl* sc = ctl_of();
    const int tid = threadIdx.x;
    if (meet || counters) named_barrier(kBarAll, kThreads);
    if (counters && tid == 0) {
        // This CTA has finished phase `ph`: counted for the CTAs that wait for its plain results
        // or are about to overwrite what it has read.
        if (ph >= 2 && !sc->abort_flag) finished_wait(ph, ph - 2);
        if (!sc->abort_flag) {
            if (flags & MB_FLAG_FENCE) asm volatile("fence.acq_rel.gpu;" ::: "memory");
            asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(&ctl->finished[ph & 3].count) : "memory");
        }
    }
    if (flags & MB_FLAG_BARRIER) {
        if (!grid_barrier(ctl, generation, kBarAll, kThreads, tid, &sc->abort_flag, &sc->verdict, ph, sc->limit_ns))
            return false;
        trace_stamp(ph, 3);
    }
    return true;
}

// The consumer warps' walk through the phase table.
template <int DIM>
__device__ __forceinline__ void consume_launch(const KernelParams& p, unsigned int calls) {
    SharedCtl* sc = ctl_of();
    const StreamDesc* table = table_of();
    const int tid = threadIdx.x;
    Place place{0u, 0u, 0u};
    // the other half of the arena becomes blank for the next launch
    for (unsigned long long at = (static_cast<unsigned long long>(blockIdx.x) * kThreads + tid) * 16;
         at < p.relay_bytes; at += static_cast<unsigned long long>(gridDim.x) * kThreads * 16)
        *reinterpret_cast<uint4*>(sc->relay_next + at) =
            make_uint4(kUnwritten, kUnwritten, kUnwritten, kUnwritten);
    if (tid == 0 && !record_ready(0)) table_of()[0].kind = kStreamStop;
    named_barrier(kBarAll, kThreads);

    const unsigned int barriers = calls * static_cast<unsigned int>(p.barriers_per_launch);
    int barrier_index = 0;
    // Optional per-phase trace: thread 0 of every CTA stamps the global timer at phase start (0),
    // when the first activations are ready (1), after the body (2) and after the closing grid
    // barrier, if the phase has one (3).
    for (int ph = 0; ph < p.n_phases; ++ph) {
        const int kind = table[ph].kind;
        if (kind == kStreamStop) break;
        // Whether there will be a phase ph + 1 -- its record has come, no fault is on record in this CTA -- is one
        // thread's verdict, through the kind of that phase, which the barrier inside this one publishes: all warps
        // leave there or none does, and that barrier also orders the record before their reads of it.  (Each
        // warp waiting for itself could leave some of them alone at the next barrier, which has no limit.)
        if (tid == 0 && ph + 1 < p.n_phases && !record_ready(ph + 1)) table_of()[ph + 1].kind = kStreamStop;
        const PhaseEntry* E = &sc->entry[ph & 3];
        trace_stamp(ph, 0);
        bool meet = true;  // the phase has not had a barrier of all threads
        if (kind == kStreamGemv) {
            const GemvStream& d = table[ph].gemv;
            if (d.shape & kShapeWhole)
                place = d.shape & kShapeShort ? gemv_phase<true, true>(ph, place) : gemv_phase<false, true>(ph, place);
            else
                place = d.shape & kShapeShort ? gemv_phase<true, false>(ph, place) : gemv_phase<false, false>(ph, place);
            meet = d.nblocks == 0;
        } else if (kind == kStreamKv) {
            place = run_attention<DIM>(ph, place);
            meet = false;
        }
        trace_stamp(ph, 2);
        const int flags = E->rec.flags;
        if (__builtin_expect(p.counters || (flags & MB_FLAG_BARRIER) != 0, 0)) {
            if (flags & MB_FLAG_BARRIER) ++barrier_index;
            if (!close_phase(p.ctl, ph, flags, meet, p.counters != 0, barriers + barrier_index)) break;  // all threads
        } else if (meet) {
            named_barrier(kBarAll, kThreads);
        }
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(&sc->entry_done[ph & 3]);
    }
}

template <int DIM>
__global__ void __launch_bounds__(kAllThreads, 1)
decode_kernel(const __grid_constant__ KernelParams p) {
    SharedCtl* sc = ctl_of();
    const int tid = threadIdx.x;
    // These words only change when the last CTA of a launch closes it (or by a host reset or bind).
    const unsigned int calls = *reinterpret_cast<volatile unsigned int*>(&p.ctl->calls);
    const unsigned int epoch = *reinterpret_cast<volatile unsigned int*>(&p.ctl->epoch);
    const unsigned int written = *reinterpret_cast<volatile unsigned int*>(&p.ctl->maps_written);
    // newer maps than this SM may have cached from their addresses (10 us for those of a model, so not always)
    if (*reinterpret_cast<volatile unsigned int*>(&p.ctl->maps_acquired) != written)
        acquire_maps(static_cast<const CUtensorMap*>(p.maps), p.n_phases * kMapsPerPhase);
    if (!begin_launch(p, p.streams, p.maps, epoch * static_cast<unsigned int>(p.n_phases), epoch, calls)) return;
    const StreamDesc* table = table_of();

    if (threadIdx.x >= kThreads) {
        if (threadIdx.x < kThreads + 32)
            producer_loop();
        else
            entry_loop();
    } else {
        consume_launch<DIM>(p, calls);
    }

    // End of the launch: the CTA that arrives last knows that every CTA has read the valid lengths,
    // `calls` and `epoch`, and advances them -- unless a fault was recorded anywhere (a token
    // outside the table ...): then the host has to reset the plan anyway.
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (sc->abort_flag && tid == 0) drain_ring();
    if (tid == 0) {
        __threadfence();
        const unsigned int before = atomicAdd(&p.ctl->arrived, 1u);
        __threadfence();
        const bool last = before == gridDim.x - 1;
        if (last) p.ctl->arrived = 0;
        sc->verdict = last && sc->abort_flag == 0 && peek_status(p.ctl) == 0 ? 1 : 0;
    }
    __syncthreads();
    if (sc->verdict) {
        for (int q = tid; q < p.n_phases; q += kAllThreads) {
            if (table[q].kind != kStreamKv || !(p.entries[q].rec.flags & MB_FLAG_BUMP_LENGTH)) continue;
            const KvStream& d = table[q].kv;
            int* lengths = reinterpret_cast<int*>(d.lengths);
            const int count = d.len_count > 1 ? d.batch : 1;
            for (int r = 0; r < count; ++r) lengths[r] += 1;
        }
        if (tid == 0) {
            p.ctl->calls = calls + 1;
            p.ctl->epoch = epoch + 1;
            // one CTA of this size fits an SM: a grid of one per SM has been on all of them
            if (static_cast<int>(gridDim.x) >= p.sm_count) p.ctl->maps_acquired = written;
        }
    }
}

// Slots of a slice that hold a warp's share of a phase's activations: the arithmetic of slice_of.
int slots_needed(const mb_phase& P, const GemvStream& d) {
    const int batch = P.i[MB_GV_I_ROWS], lp = (d.shape & kShapeShort) ? 2 : 1;
    const int rs = batch > 2 ? (batch > 4 ? 3 : 2) : batch - 1;
    const int stages = (d.groups + (8 << lp) - 1) >> (3 + lp);
    return ((stages << (lp + rs)) + 7) >> 3;
}

// Shape of a skinny GEMM: a CTA with at most 8 output rows (o and down projections, q|k|v of small
// models) takes blocks of 8 rows and twice the reduction per stage, so that no half of a stage and
// of the MMA runs empty; gate and up rows come eight and eight; everything else sixteen at a time.
void shape_gemv(const mb_phase& P, int ctas, int slots, GemvStream* d) {
    int total = 0;
    for (int s = 0; s < P.i[MB_GV_I_NSEG]; ++s) total += P.i[MB_GV_I_N0 + s];
    d->row_bytes = P.i[MB_GV_I_K] * 2;
    d->n0 = P.i[MB_GV_I_NSEG] > 1 ? P.i[MB_GV_I_N0] : INT_MAX;
    d->n01 = P.i[MB_GV_I_NSEG] > 2 ? d->n0 + P.i[MB_GV_I_N0 + 1] : INT_MAX;
    d->r0 = (total / 2) / ctas;
    d->r1 = (total / 2) % ctas;
    d->groups = P.i[MB_GV_I_K] / 32;
    const int rows = 2 * (d->r0 + (d->r1 > 0 ? 1 : 0));  // of the busiest CTA
    d->shape = P.i[MB_GV_I_NMAT] == 2 ? kShapePaired : (rows <= 8 ? kShapeShort : 0);
    if (slots_needed(P, *d) <= slots) d->shape |= kShapeWhole;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

bool encode_map(CUtensorMap* map, unsigned long long base, int rank, const cuuint64_t* dims, const cuuint64_t* strides,
                const cuuint32_t* box, bool swizzled, bool wide) {
    static EncodeTiledFn fn = [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult result;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &result) != cudaSuccess ||
            result != cudaDriverEntryPointSuccess)
            sym = nullptr;
        return reinterpret_cast<EncodeTiledFn>(sym);
    }();
    const cuuint32_t elem[5] = {1, 1, 1, 1, 1};
    return fn != nullptr &&
           fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, static_cast<cuuint32_t>(rank), reinterpret_cast<void*>(base),
              dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              swizzled ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_NONE,
              wide ? CU_TENSOR_MAP_L2_PROMOTION_L2_256B : CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// [rows, K] bf16 row-major as (32 elements, rows, groups of 32 elements); zeros outside.
bool encode_weight_map(CUtensorMap* map, unsigned long long base, int rows, int K, int box_rows,
                       int box_groups) {
    const cuuint64_t dims[3] = {32, static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(K / 32)};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(K) * 2, 64};
    const cuuint32_t box[3] = {32, static_cast<cuuint32_t>(box_rows), static_cast<cuuint32_t>(box_groups)};
    return encode_map(map, base, 3, dims, strides, box, false, true);
}
// A cache [batch, capacity, heads, D] as (32 elements, keys, groups of 32 elements, heads, batch); boxes
// of `keys` rows of one head.
bool encode_cache_map(CUtensorMap* map, unsigned long long base, const mb_phase& P, int keys, bool swizzled) {
    const cuuint64_t D = P.i[MB_AT_I_HEAD_DIM], heads = P.i[MB_AT_I_KV_HEADS], capacity = P.i[MB_AT_I_CAPACITY];
    const cuuint64_t dims[5] = {32, capacity, D / 32, heads, static_cast<cuuint64_t>(P.i[MB_AT_I_BATCH])};
    const cuuint64_t strides[4] = {heads * D * 2, 64, D * 2, capacity * heads * D * 2};
    const cuuint32_t box[5] = {32, static_cast<cuuint32_t>(keys), static_cast<cuuint32_t>(D / 32), 1, 1};
    return encode_map(map, base, 5, dims, strides, box, swizzled, D > 64);
}

}  // namespace decode

int decode_threads() { return decode::kAllThreads; }
int decode_fixed_smem() { return decode::kCtlBytes; }
int decode_stage_bytes() { return decode::kStageBytes; }
int decode_row_pad() { return decode::kRowPad; }
int decode_row_tile() { return decode::kRowTile; }

int decode_rope_bytes(const mb_phase* phases, unsigned int n) {
    int bytes = 0;
    for (unsigned int i = 0; i < n; ++i) {
        if (phases[i].body != MB_BODY_ATTN_DECODE) continue;
        const int batch = phases[i].i[MB_AT_I_BATCH];
        const int rows = batch <= decode::kRopeRows ? batch : 1;
        const int need = rows * (phases[i].i[MB_AT_I_HEAD_DIM] / 2) * 4;
        if (need > bytes) bytes = need;
    }
    return (bytes + 127) / 128 * 128;
}

// Shared memory of a plan: fixed part, slices, ring, stream table, cos / sin table.
static long long smem_bytes(int rope_bytes, unsigned int n_phases, int stages, int slots) {
    if (n_phases > 1u << 20) return LLONG_MAX;
    return static_cast<long long>(decode::rope_offset(stages, slots, n_phases)) + rope_bytes;
}
// Stages of the weight ring that fit; fewer than two means the plan does not.
int decode_ring_stages(int rope_bytes, unsigned int n_phases, int slots, int limit) {
    int stages = decode::kMaxStages;
    while (stages > 0 && smem_bytes(rope_bytes, n_phases, stages, slots) > limit) --stages;
    return stages;
}
int decode_smem_bytes(int rope_bytes, unsigned int n_phases, int slots, int stages) {
    return static_cast<int>(smem_bytes(rope_bytes, n_phases, stages, slots));
}
int decode_slice_slots(const mb_phase* phases, unsigned int n, int ctas) {
    int slots = decode::kSliceSlots;
    for (unsigned int i = 0; i < n; ++i) {
        if (phases[i].body != MB_BODY_GEMV) continue;
        GemvStream d;
        decode::shape_gemv(phases[i], ctas, 0, &d);
        const int need = decode::slots_needed(phases[i], d);
        if (need > decode::kSliceSlots && need <= decode::kWideSlots) slots = decode::kWideSlots;
    }
    return slots;
}

// The static part of a phase's stream record; `addr`: its resolved slots.
void decode_stream(const mb_phase& P, const unsigned long long* addr, int ctas, int slots, StreamDesc* out) {
    std::memset(out, 0, sizeof(*out));
    if (P.body == MB_BODY_GEMV) {
        GemvStream& d = out->gemv;
        d.kind = kStreamGemv;
        decode::shape_gemv(P, ctas, slots, &d);
        if (P.i[MB_GV_I_PROLOGUE] != MB_PRO_NONE) d.w_norm = addr[MB_GV_S_NORM_W];
    } else if (P.body == MB_BODY_ATTN_DECODE) {
        KvStream& d = out->kv;
        d.kind = kStreamKv;
        d.capacity = P.i[MB_AT_I_CAPACITY];
        d.k = addr[MB_AT_S_KCACHE];
        d.v = addr[MB_AT_S_VCACHE];
        d.lengths = addr[MB_AT_S_LEN];
        d.batch = P.i[MB_AT_I_BATCH];
        d.kv_heads = P.i[MB_AT_I_KV_HEADS];
        d.head_dim = P.i[MB_AT_I_HEAD_DIM];
        d.len_count = P.i[MB_AT_I_LEN_COUNT];
        // a partial is kept as (value, tag) pairs, twice the floats the record's buffer counts
        d.chunk_cap = P.i[MB_AT_I_MAX_CHUNKS] / 2 > 1 ? P.i[MB_AT_I_MAX_CHUNKS] / 2 : 1;
        d.exact_keys = P.i[MB_AT_I_EXACT_KEYS];
    }
}

// The tensor maps of a phase.  GEMV: the weight segments (the second one of a paired phase is the paired
// matrix); attention: keys and values.
bool decode_encode_maps(const mb_phase& P, const unsigned long long* addr, int ctas, void* out) {
    CUtensorMap* maps = static_cast<CUtensorMap*>(out);
    std::memset(maps, 0, decode::kMapsPerPhase * sizeof(CUtensorMap));
    if (P.body == MB_BODY_ATTN_DECODE) {
        const int keys = 16 << decode::kv_shift(P.i[MB_AT_I_HEAD_DIM]);
        if (!decode::encode_cache_map(maps, addr[MB_AT_S_KCACHE], P, keys, false) ||
            !decode::encode_cache_map(maps + 1, addr[MB_AT_S_VCACHE], P, keys, true))
            return false;
        return true;
    }
    if (P.body != MB_BODY_GEMV) return true;
    GemvStream d;
    decode::shape_gemv(P, ctas, 0, &d);
    const bool is_short = (d.shape & kShapeShort) != 0, paired = (d.shape & kShapePaired) != 0;
    const int box_rows = is_short || paired ? 8 : 16, box_groups = is_short ? 32 : 16;
    for (int s = 0; s < P.i[MB_GV_I_NSEG]; ++s)
        if (!decode::encode_weight_map(maps + s, addr[MB_GV_S_W0 + s], P.i[MB_GV_I_N0 + s], P.i[MB_GV_I_K],
                                       box_rows, box_groups))
            return false;
    return !paired || decode::encode_weight_map(maps + 1, addr[MB_GV_S_W_PAIR], P.i[MB_GV_I_N0],
                                                P.i[MB_GV_I_K], box_rows, box_groups);
}
namespace decode {
struct alignas(64) PhaseMaps {
    CUtensorMap map[kMapsPerPhase];
};
// One warp: the maps of one phase of the launch that follows, which finds them newer than those acquired.
__global__ void store_maps_kernel(const __grid_constant__ PhaseMaps maps, uint4* out, Control* ctl) {
    for (unsigned int v = threadIdx.x; v < sizeof(PhaseMaps) / 16; v += 32)
        out[v] = reinterpret_cast<const uint4*>(&maps)[v];
    asm volatile("fence.proxy.tensormap::generic.release.gpu;" ::: "memory");
    if (threadIdx.x == 0) ctl->maps_written += 1;
}
}  // namespace decode

cudaError_t decode_store_maps(const mb_phase& P, const unsigned long long* addr, int ctas, void* out, Control* ctl,
                              cudaStream_t stream) {
    decode::PhaseMaps maps;
    if (!decode_encode_maps(P, addr, ctas, &maps)) return cudaErrorInvalidValue;
    decode::store_maps_kernel<<<1, 32, 0, stream>>>(maps, static_cast<uint4*>(out), ctl);
    return cudaGetLastError();
}
size_t decode_map_bytes() { return decode::kMapsPerPhase * sizeof(CUtensorMap); }

namespace {
const void* kernel_of(int head_dim) {
    switch (head_dim) {
        case 64: return reinterpret_cast<const void*>(&decode::decode_kernel<64>);
        case 128: return reinterpret_cast<const void*>(&decode::decode_kernel<128>);
        case 256: return reinterpret_cast<const void*>(&decode::decode_kernel<256>);
        default: return reinterpret_cast<const void*>(&decode::decode_kernel<0>);
    }
}
}  // namespace

// The one head size of a plan's attention phases (64 if it has none), or 0.
int decode_head_dim(const mb_phase* phases, unsigned int n) {
    int dim = -1;
    for (unsigned int i = 0; i < n; ++i) {
        if (phases[i].body != MB_BODY_ATTN_DECODE) continue;
        const int d = phases[i].i[MB_AT_I_HEAD_DIM];
        if (dim >= 0 && d != dim) return 0;
        dim = d;
    }
    return dim < 0 ? 64 : dim;
}

cudaError_t decode_configure(int head_dim, int smem_bytes) {
    return cudaFuncSetAttribute(kernel_of(head_dim), cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
}

cudaError_t decode_occupancy(int head_dim, int smem_bytes, int* blocks_per_sm) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kernel_of(head_dim), decode::kAllThreads,
                                                         smem_bytes);
}

cudaError_t decode_launch(const KernelParams& params, int head_dim, int ctas, int smem_bytes,
                          cudaStream_t stream) {
    KernelParams copy = params;
    void* args[] = {&copy};
    return cudaLaunchCooperativeKernel(kernel_of(head_dim), dim3(ctas), dim3(decode::kAllThreads), args,
                                       static_cast<size_t>(smem_bytes), stream);
}

}  // namespace mb

// =======================================================================================
// Decode attention without any allocation.
//
// Some hosts may not allocate device memory at the point where they need one attention
// step: a plugin called from inside someone else's stream-ordered pipeline, a process that
// runs inside a fixed amount of memory handed out at start-up, a caller inside a region where
// cudaMalloc would synchronise the device.  For them this entry point runs the same
// attention body as the plan path, but everything the plan path keeps in allocated memory
// (phase table, control block, split-key partials) lives either in the
// kernel parameters or in one fixed-size array inside this library's device image.
//
// The array is a file-scope `static __device__` object of kStaticScratchBytes (4 MiB); every
// GPU that loads the library holds it until the process exits.  In host code its name is only
// a host-side stand-in, not a device address: the address the kernel gets is asked for once
// per device with cudaGetSymbolAddress, with that device current.
//
// All calls share the array.  The control words are cleared on the stream before every launch.  The
// partials need no clearing: they are cells tagged with the call's number, which is kept outside the
// cleared part and never repeats.  Two calls that overlap on the GPU (different streams, no
// dependency) race on the array -- callers serialise them.
// =======================================================================================
namespace mb {
namespace decode {

constexpr size_t kStaticScratchBytes = 4u << 20;
constexpr size_t kStaticControlBytes = 256;        // the head of a Control: status and arrivals
// The attention body and the end of the launch only touch the words before the finished-phase
// counters through the pointer they are given.
static_assert(offsetof(Control, finished) <= kStaticControlBytes, "the static control area is too small");
constexpr size_t kStaticCounterBytes = 4096;       // a word for each of up to 1024 (row, kv head): unused,
                                                   // but part of the size limits callers know
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];
// Tags the partials of a call; outside the area that is cleared before every call, so that no
// partial of an earlier call can be mistaken for one of this call.
static __device__ unsigned int g_static_epoch;

__global__ void __launch_bounds__(kAllThreads, 1)
attention_static_kernel(const __grid_constant__ KernelParams p, const __grid_constant__ PhaseEntry entry,
                        const __grid_constant__ StreamDesc stream, const __grid_constant__ PhaseMaps maps,
                        int* status_out) {
    SharedCtl* sc = ctl_of();
    const int tid = threadIdx.x;
    const unsigned int epoch = *reinterpret_cast<volatile unsigned int*>(&g_static_epoch);
    if (tid < kEntryVectors)
        reinterpret_cast<uint4*>(&sc->entry[0])[tid] = reinterpret_cast<const uint4*>(&entry)[tid];
    if (begin_launch(p, &stream, &maps, epoch, 0u, 0u)) {
        if (tid < kThreads)
            run_attention<0>(0, Place{0u, 0u, 0u});
        else if (tid < kThreads + 32)
            producer_loop();
        __syncthreads();
        if (sc->abort_flag && tid == 0) drain_ring();
    }
    __syncthreads();
    if (tid == 0) {
        // The valid length may only move once every CTA has read it: the last CTA to finish
        // advances it, reports the status and re-arms the counter for the next call.
        __threadfence();
        const unsigned int before = atomicAdd(&p.ctl->arrived, 1u);
        if (before == gridDim.x - 1) {
            __threadfence();
            const int code = peek_status(p.ctl);
            if (code == 0) {
                int* lenp = reinterpret_cast<int*>(entry.addr[MB_AT_S_LEN]);
                *lenp = *lenp + 1;
            }
            if (status_out != nullptr) *status_out = code;
            p.ctl->arrived = 0;
            g_static_epoch = epoch + 1;
        }
    }
}

struct StaticDevice {
    unsigned char* scratch = nullptr;  // device address of g_static_scratch on this device
    int sm_count = 0;
    int smem_limit = 0;
    bool ready = false;
};

}  // namespace decode
}  // namespace mb

namespace {
mb::decode::StaticDevice g_static_devices[64];
std::mutex g_static_mutex;
}  // namespace

// Declared in include/megabake_b200.h.  The first call on a device performs the one-time
// set-up (symbol address, kernel attribute); make that call before any stream capture.
extern "C" int mb_attention_decode_static(const mb_attention_args* a, void* stream) {
    using namespace mb::decode;
    if (a == nullptr) return MB_ERR_INVALID;
    if (a->batch < 1 || a->heads < 1 || a->kv_heads < 1 || a->capacity < 1) return MB_ERR_INVALID;
    if (a->heads % a->kv_heads != 0 || a->heads / a->kv_heads > 8) return MB_ERR_UNSUPPORTED;
    if (a->head_dim != 64 && a->head_dim != 128 && a->head_dim != 256) return MB_ERR_UNSUPPORTED;
    const unsigned long long pointers[] = {a->query, a->key, a->value, a->key_cache,
                                           a->value_cache, a->valid_length, a->position_ids,
                                           a->inv_freq, a->out};
    for (unsigned long long ptr : pointers)
        if (ptr == 0) return MB_ERR_INVALID;
    if ((a->query | a->key | a->value | a->key_cache | a->value_cache | a->out) & 15ull)
        return MB_ERR_INVALID;
    if ((a->position_ids & 7ull) || (a->valid_length & 3ull) || (a->inv_freq & 3ull) ||
        (a->status & 3ull))
        return MB_ERR_INVALID;

    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return MB_ERR_CUDA;
    StaticDevice& dev = g_static_devices[device];
    {
        std::lock_guard<std::mutex> lock(g_static_mutex);
        if (!dev.ready) {
            void* address = nullptr;
            cudaError_t err = cudaGetSymbolAddress(&address, g_static_scratch);
            if (err != cudaSuccess || address == nullptr) return MB_ERR_CUDA;
            cudaDeviceProp prop;
            if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return MB_ERR_CUDA;
            if (prop.major != 10) return MB_ERR_UNSUPPORTED;
            if (!prop.cooperativeLaunch) return MB_ERR_UNSUPPORTED;
            if (cudaFuncSetAttribute(attention_static_kernel,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(prop.sharedMemPerBlockOptin)) != cudaSuccess)
                return MB_ERR_CUDA;
            dev.scratch = static_cast<unsigned char*>(address);
            dev.sm_count = prop.multiProcessorCount;
            dev.smem_limit = static_cast<int>(prop.sharedMemPerBlockOptin);
            dev.ready = true;
        }
    }

    const int group = a->heads / a->kv_heads;
    const int pairs = a->batch * a->kv_heads;
    // What fits the fixed array: a word for every (row, kv head) and at least one
    // part of partials each; more parts if there is room, up to 32.
    if (static_cast<size_t>(pairs) * 4 > kStaticCounterBytes) return MB_ERR_RESOURCE;
    const size_t per_chunk = static_cast<size_t>(pairs) * group * (a->head_dim + 2) * 4;
    const size_t room = kStaticScratchBytes - kStaticControlBytes - kStaticCounterBytes;
    if (per_chunk > room) return MB_ERR_RESOURCE;  // shapes beyond the 4 MiB scratch
    int max_chunks = static_cast<int>(room / per_chunk);  // two for every part: cells take twice the room
    if (max_chunks > 64) max_chunks = 64;
    const int by_capacity = 2 * ((a->capacity + 15) / 16);
    if (max_chunks > by_capacity) max_chunks = by_capacity;

    mb::PhaseEntry entry;
    std::memset(&entry, 0, sizeof(entry));
    entry.rec.body = MB_BODY_ATTN_DECODE;
    entry.rec.i[MB_AT_I_BATCH] = a->batch;
    entry.rec.i[MB_AT_I_HEADS] = a->heads;
    entry.rec.i[MB_AT_I_KV_HEADS] = a->kv_heads;
    entry.rec.i[MB_AT_I_HEAD_DIM] = a->head_dim;
    entry.rec.i[MB_AT_I_CAPACITY] = a->capacity;
    entry.rec.i[MB_AT_I_INVFREQ_BF16] = a->inv_freq_is_bf16 ? 1 : 0;
    entry.rec.i[MB_AT_I_MAX_CHUNKS] = max_chunks;
    entry.rec.i[MB_AT_I_MERGE_SLOTS] = 1;
    entry.rec.i[MB_AT_I_EXACT_KEYS] = a->capacity < 128 ? a->capacity : 128;
    entry.rec.i[MB_AT_I_LEN_COUNT] = 1;
    entry.rec.f[MB_AT_F_SCALE] = 1.0f / sqrtf(static_cast<float>(a->head_dim));
    entry.rec.f[MB_AT_F_ROPE_SCALE] = a->rope_scale;
    entry.rec.f[MB_AT_F_Q_SCALE] = a->query_scale;
    unsigned char* control = dev.scratch;
    unsigned char* counters = dev.scratch + kStaticControlBytes;
    unsigned char* partials = counters + kStaticCounterBytes;
    entry.addr[MB_AT_S_Q] = a->query;
    entry.addr[MB_AT_S_K] = a->key;
    entry.addr[MB_AT_S_V] = a->value;
    entry.addr[MB_AT_S_KCACHE] = a->key_cache;
    entry.addr[MB_AT_S_VCACHE] = a->value_cache;
    entry.addr[MB_AT_S_LEN] = a->valid_length;
    entry.addr[MB_AT_S_POS] = a->position_ids;
    entry.addr[MB_AT_S_INVFREQ] = a->inv_freq;
    entry.addr[MB_AT_S_OUT] = a->out;
    entry.addr[MB_AT_S_PARTIAL] = reinterpret_cast<unsigned long long>(partials);
    entry.addr[MB_AT_S_COUNTER] = reinterpret_cast<unsigned long long>(counters);

    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // control words start every call at zero (a faulted earlier call may have left them set)
    if (cudaMemsetAsync(control, 0, kStaticControlBytes + kStaticCounterBytes, s) != cudaSuccess)
        return MB_ERR_CUDA;
    mb::StreamDesc desc;
    mb::decode_stream(entry.rec, entry.addr, dev.sm_count, kSliceSlots, &desc);
    mb::KernelParams params;
    std::memset(&params, 0, sizeof(params));
    params.ctl = reinterpret_cast<mb::Control*>(control);
    params.n_phases = 1;
    params.wait_limit_us = 2000000u;
    int* status_out = reinterpret_cast<int*>(a->status);
    // the parts of a split context wait for one another's partials: all CTAs have to be resident
    const int rope_bytes = mb::decode_rope_bytes(&entry.rec, 1);
    params.slots = kSliceSlots;
    params.stages = mb::decode_ring_stages(rope_bytes, 1, params.slots, dev.smem_limit);
    PhaseMaps maps;
    if (params.stages < 2 || !mb::decode_encode_maps(entry.rec, entry.addr, dev.sm_count, &maps)) return MB_ERR_CUDA;
    void* args[] = {&params, &entry, &desc, &maps, &status_out};
    const int smem = mb::decode_smem_bytes(rope_bytes, 1, params.slots, params.stages);
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(&attention_static_kernel),
                                       dim3(dev.sm_count), dim3(kAllThreads), args,
                                       static_cast<size_t>(smem), s) == cudaSuccess
               ? MB_OK
               : MB_ERR_CUDA;
}

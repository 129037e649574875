// Short prompts: a whole prefill as one cooperative launch.
//
// A short prompt is a chain of small dependent steps, and as one kernel per step (mb_prefill.cu) it is bound by
// the launch boundaries: 243 launches of 5.1 us for 19 tokens of a 30-layer model whose weights
// stream in 42 us.  Here one CTA per SM stays for the whole prompt and walks the steps
//
//     rows       embedding gather, rotary table, first norm
//     per layer  q|k|v  ->  attention  ->  o (slices)  ->  rows  ->  gate|up  ->  down (slices)  ->  rows
//     logits
//
// A step starts when every work unit of the step before it has been counted (one counter per step in global
// memory).  So a buffer is never written before its last readers are through: they belong to a step
// that was counted before the writer's step began.
//
//   warp 0      weight producer: one lane copies weight tiles (TMA) into a ring of stages.  Weights depend on
//               nothing, so it runs ahead, across steps, as far as the ring goes: what a step waits
//               for is its activations alone.
//   warp 1      issues tcgen05.mma.  The weights are the 64 or 128 rows of the product and the tokens its
//               columns: 16 tokens are padded to nothing, and a CTA's share of the features can be any
//               multiple of 8, so that every SM streams weights however few tokens there are.
//   warp 2      activation producer: one lane waits for the step before and copies the activations of each
//               k-block (TMA) into the same stages.
//   warps 4-11  workers: accumulators out of tensor memory (thread = feature), attention, rows.
//
// Sums over slices of a reduction meet in the row step, which needs whole rows anyway: it adds the slices in
// order, adds the residual, and normalises.  The rounding points are those of the kernels in mb_prefill.cu.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>

#include "mb_device.cuh"
#include "mb_kernels.h"
#include "mb_tensor.cuh"

namespace mb {
namespace prompt {

using namespace prefill;

constexpr int kWorkers = 256;
constexpr int kThreads = 128 + kWorkers;
constexpr int kMaxLayers = 30;     // what fits the parameters of one launch
// Tokens over all rows of the batch up to which one launch is the faster form, by the weights of a layer.  What it
// saves is launches; what it costs grows with the tokens and the weights (tiles of 128 tokens take more operand
// bytes than mb_prefill.cu's, attention does without tcgen05).  Between the points the limit is interpolated over the
// logarithm of the weights.  Time of the launches of their own over that of the one, each called directly /
// replayed from a graph, one prompt (four and sixteen prompts of as many tokens together do better):
//   0.6 M weights a layer  1.14 / 1.06 at 512 tokens, 1.02 / 0.97 at 640
//   3.5 M (135M shape)     1.18 / 1.12 at 512, 1.07 / 1.02 at 576, 0.98 / 0.96 at 608
//   5.9 M and 7.5 M        1.12 / 1.05 at 512, 1.04 / 1.00 at 576, 1.00 / 0.97 at 608
//   9.4 M                  1.09 / 1.02 at 512, 0.96 / 0.92 at 544
//   12.1 M                 1.05 / 0.99 at 448, 1.03 / 0.96 at 480
//   14.9 M (0.5B shape)    1.17 / 1.11 at 256, 1.03 / 0.98 at 384
//   19.9 M                 1.11 / 1.05 at 256, 1.01 / 0.96 at 288
//   23.3 M                 1.05 / 1.00 at 192, 0.97 / 0.92 at 256
//   29 M, 39 M, 47 M       1.17 / 1.10 at 160, 1.04 to 1.10 / 0.99 to 1.04 at 208
//   60.8 M (1B shape)      1.12 / 1.07 at 128, 1.06 / 1.00 at 160, 1.01 / 0.96 at 176
//   70 M to 212 M          1.13 to 1.22 / 1.09 to 1.15 at 128, 0.94 to 1.01 / 0.90 to 0.96 at 144
struct Limit {
    double weights;
    int rows;
};
constexpr Limit kLimits[] = {{1.0e6, 640}, {4.2e6, 592}, {8.0e6, 576}, {12.0e6, 432}, {16.0e6, 384},
                             {20.0e6, 272}, {24.0e6, 160}, {64.0e6, 160}, {66.0e6, 128}};
inline int most_rows(long long layer_weights) {
    const double w = static_cast<double>(layer_weights);
    const Limit* below = kLimits;
    for (const Limit& at : kLimits) {
        if (w <= at.weights)
            return &at == kLimits ? at.rows
                                  : below->rows + static_cast<int>((at.rows - below->rows) * std::log(w / below->weights) /
                                                                   std::log(at.weights / below->weights));
        below = &at;
    }
    return below->rows;
}
// Blocks of keys that the attention units of one CTA may go over where a prompt has more than one (tcgen05 takes less
// for them): 16 heads of 64 on a hidden size of 256, two waves of units and five blocks 1.01 / 0.96, three
// waves 0.89 / 0.85.  Prompts of one block do better the more there are (128 of one token, 32 heads, 28 waves: 2.26 / 2.23).
constexpr int kAttnSweeps = 10;
constexpr int kAttnRows = 32;      // query rows of an attention unit
constexpr int kSmemBytes = 232448 - 1024;  // 1 KB for what the kernel declares itself
// A 128-row MMA reads 16 KB of weights from wherever a tile starts, also where the tile has fewer rows
// (their products are never read): the ring ends that far before the end of shared memory.
constexpr int kStages = 4, kStageBytes = 52 * 1024;
constexpr int kRingBytes = kStages * kStageBytes;
static_assert(kRingBytes + 16384 + 1024 + 1024 <= kSmemBytes, "ring, over-read, barriers and alignment");

// One projection: how its output is cut into units, unit u being CTA (first + u) mod grid's.
struct Gemm {
    int rows;     // features per unit (per matrix of a gated pair), a multiple of 8
    int tokens;   // columns per unit, a multiple of 16
    int tiles_t;
    int start[3]; // first feature tile of each segment
    int n[3];
    int tiles;    // feature tiles over all segments
    int slices, kblocks, units, first;
    int accs;     // accumulators: 2 for a gated pair and for more than 128 features
    int pair, wide;
    int half;     // q|k|v: half the head dimension; a unit's features are pairs (i, i + half) of heads
    unsigned int idesc;
    int deep;     // k-blocks per stage of the ring
    int a_bytes, b_bytes;  // per stage
};

struct LayerArgs {
    CUtensorMap w[7];  // q, k, v, o, gate, up, down
    const unsigned short* norm[2];  // before attention, before the gated projections
    const unsigned short* bias[5];  // q, k, v, o, down
    unsigned short* kv[2];          // keys and values: one pair of tensors for all layers, or caches of the layer's own
    int* length;
};

struct Params {
    CUtensorMap b[5];  // activations of q|k|v, o, gate|up, down, logits
    CUtensorMap head;
    Gemm gemm[5];
    LayerArgs layer[kMaxLayers];
    const unsigned short* final_norm;
    const unsigned short* head_bias;
    const unsigned short* table;
    const long long* ids;
    const long long* pos;
    const void* inv_freq;
    unsigned short* hidden;
    unsigned short* normed;
    unsigned short* q;
    unsigned short* attn;
    unsigned short* glu;
    unsigned short* logits;
    float* parts;            // [slice][row][hidden]
    unsigned int* rotary;    // [row][head_dim / 2]: cos | sin << 16, bf16
    unsigned int* counters;  // one per step; then CTAs that are through, and the fault mark
    Control* ctl;
    unsigned long long* trace;
    int layers, rows, tokens, batch, hidden_size, vocab_in, heads, kv_heads, head_dim, intermediate;
    int norm_kind, activation, invfreq_bf16, kv_rows, length_value, length_count;  // kv_rows: per batch row
    float eps, embed_scale, rope_scale, q_scale, softmax_scale;
    int attn_units, attn_blocks;  // units of the attention step; query blocks of a (row, head)
    int steps, small;
    unsigned int limit_us;  // of a hand-over between steps; twice as much for the pipeline within a CTA
};

enum Step { kQkv = 0, kAttention, kOut, kRowsMid, kGated, kDown, kRowsEnd, kStepsPerLayer };
enum Projection { kProjQkv = 0, kProjOut, kProjGated, kProjDown, kProjHead };

struct Shared {
    unsigned char* ring;
    unsigned long long *full, *empty, *acc_full, *acc_empty, *attn_done;
    unsigned int* tmem_slot;
    volatile int* abort_flag;  // the word after it: the limit of a hand-over between steps, microseconds
};

// ---------------------------------------------------------------------------------------
// Code size is time here.  A step's code runs once a layer, and what does not stay in the instruction cache until
// the next layer comes from L2 again, behind the weights: with every wait and every step inlined wherever
// it is used (300 KB) an attention unit of the 1B shape took 15,700 cycles, and 4,500 when it was run
// twice in a row.  So a body has one place in the code, waits that do not succeed at once continue
// out of line, and loops stay rolled.
// ---------------------------------------------------------------------------------------
// (The limit comes from shared memory when it is looked at: as an argument it cost 0.8 % of the shortest prompt.)
__device__ __forceinline__ unsigned long long limit_ns(const volatile int* abort_flag) {
    return 1000ull * static_cast<unsigned int>(abort_flag[1]);
}
__device__ __noinline__ bool wait_long(unsigned int bar, unsigned int parity, volatile int* abort_flag) {
    const unsigned long long start = global_timer_ns();
    for (unsigned int tries = 1;; ++tries) {
        unsigned int done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if ((tries & 127u) == 0u && (*abort_flag || global_timer_ns() - start > 2 * limit_ns(abort_flag))) return false;
    }
}
// All lanes of a warp; the compiler knows the result to be the same in all of them.
__device__ __forceinline__ bool wait_warp(const Shared& sh, unsigned long long* bar, unsigned int parity) {
    bool done = mbar_try_wait(bar, parity);
    if (!__all_sync(0xffffffffu, done)) done = wait_long(smem_u32(bar), parity, sh.abort_flag);
    return __all_sync(0xffffffffu, done) != 0;
}

// ---------------------------------------------------------------------------------------
// Steps follow one another through counters.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned int* fault_mark(const Params& p) { return p.counters + p.steps + 1; }

__device__ __noinline__ void record_fault(Control* ctl, unsigned int* mark, volatile int* abort_flag, int code,
                                          int step, int where) {
    record_status(ctl, code, step, where);
    atomicExch(mark, 1u);  // the others need not wait for this CTA
    *abort_flag = 1;
}
__device__ __forceinline__ void give_up(const Params& p, const Shared& sh, int code, int step, int where) {
    record_fault(p.ctl, fault_mark(p), sh.abort_flag, code, step, where);
}

// Waits until `units` units of `step` are complete; one thread.
__device__ __noinline__ bool await_count(const unsigned int* counter, unsigned int units, const unsigned int* mark,
                                         volatile int* abort_flag, Control* ctl, int step) {
    unsigned long long start = 0;
    for (unsigned int tries = 1;; ++tries) {
        unsigned int seen;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
        if (seen >= units) return true;
        if ((tries & 63u) == 0u) {
            if (start == 0) start = global_timer_ns();
            if (*abort_flag != 0) return false;
            if (*reinterpret_cast<const volatile unsigned int*>(mark) != 0) {
                *abort_flag = 1;
                return false;
            }
            if (global_timer_ns() - start > limit_ns(abort_flag)) {
                record_fault(ctl, const_cast<unsigned int*>(mark), abort_flag, MB_ST_HANDOFF_TIMEOUT, step,
                             static_cast<int>(blockIdx.x));
                return false;
            }
        }
    }
}
__device__ __forceinline__ bool await_step(const Params& p, const Shared& sh, int step, unsigned int units) {
    return await_count(p.counters + step, units, fault_mark(p), sh.abort_flag, p.ctl, step);
}

// The workers of this CTA have finished `units` units of `step`.  False: some wait ran out.
__device__ __forceinline__ bool workers_done(const Params& p, const Shared& sh, int tid, int step, int units,
                                             bool ok) {
    if (named_barrier_or(1, kWorkers, !ok)) return false;
    if (tid == 0 && units > 0) {
        __threadfence();
        atomicAdd(p.counters + step, static_cast<unsigned int>(units));
    }
    return true;
}
__device__ __forceinline__ bool workers_await(const Params& p, const Shared& sh, int tid, int step,
                                              unsigned int units) {
    bool ok = true;
    if (tid == 0) ok = await_step(p, sh, step, units);
    return !named_barrier_or(1, kWorkers, !ok);
}

__device__ __forceinline__ int first_unit(int first) {
    const int c = static_cast<int>(blockIdx.x) - first;
    return c < 0 ? c + static_cast<int>(gridDim.x) : c;
}
__device__ __forceinline__ int units_here(int units, int first) {
    const int u = first_unit(first);
    return u < units ? (units - u + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x) : 0;
}

// Slices of a tile are neighbours, then the token tiles of the same features.
struct Unit {
    int slice, tile_t, seg, f0, kb0, kb1;
};
__device__ __noinline__ Unit unit_at(int u, int slices, int tiles_t, int start1, int start2, int rows, int kblocks) {
    Unit x;
    const int t = u / slices;
    x.slice = u - t * slices;
    const int tile = t / tiles_t;
    x.tile_t = t - tile * tiles_t;
    x.seg = (tile >= start1 ? 1 : 0) + (tile >= start2 ? 1 : 0);
    x.f0 = (tile - (x.seg == 0 ? 0 : x.seg == 1 ? start1 : start2)) * rows;
    x.kb0 = x.slice * kblocks / slices;
    x.kb1 = (x.slice + 1) * kblocks / slices;
    return x;
}
__device__ __forceinline__ Unit unit_of(const Gemm& g, int u) {
    return unit_at(u, g.slices, g.tiles_t, g.start[1], g.start[2], g.rows, g.kblocks);
}

__device__ __forceinline__ void stamp_at(const Params& p, int step, int slot) {
    if (p.trace != nullptr && blockIdx.x == 0) p.trace[static_cast<size_t>(step) * 8 + slot] = global_timer_ns();
}

struct RingPlace {
    int s = 0, round = 0;
    __device__ __forceinline__ void next() {
        if (++s == kStages) {
            s = 0;
            ++round;
        }
    }
};

// ---------------------------------------------------------------------------------------
// Producers and the MMA warp: one thread each, all walking the same units.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ bool produce_weights(const Params& p, const Shared& sh, const Gemm& g,
                                                const CUtensorMap* maps, RingPlace& at, int step) {
    for (int u = first_unit(g.first); u < g.units; u += gridDim.x) {
        const Unit x = unit_of(g, u);
        for (int kb = x.kb0; kb < x.kb1; kb += g.deep) {
            if (at.round > 0 && !wait_warp(sh, &sh.empty[at.s], (at.round - 1) & 1)) {
                give_up(p, sh, MB_ST_PIPE_TIMEOUT, step, 1);
                return false;
            }
            unsigned char* stage = sh.ring + at.s * kStageBytes;
            if (elect_one()) {
                mbar_arrive_expect_tx(&sh.full[at.s], g.a_bytes);
                if (g.half > 0) {
                    const int head = x.f0 / g.half, row = x.f0 - head * g.half;
                    tma_load_heads(stage, maps + x.seg, row, 0, head, kb, &sh.full[at.s]);
                    tma_load_heads(stage + g.a_bytes / 2, maps + x.seg, row, 1, head, kb, &sh.full[at.s]);
                } else {
                    tma_load_blocks(stage, maps + x.seg, x.f0, kb, &sh.full[at.s]);
                    if (g.pair) tma_load_blocks(stage + g.a_bytes / 2, maps + 1, x.f0, kb, &sh.full[at.s]);
                }
            }
            __syncwarp();
            at.next();
        }
    }
    return true;
}

__device__ __forceinline__ bool produce_activations(const Params& p, const Shared& sh, const Gemm& g,
                                                    const CUtensorMap* map, RingPlace& at, int step,
                                                    unsigned int before) {
    bool waited = false;
    for (int u = first_unit(g.first); u < g.units; u += gridDim.x) {
        const Unit x = unit_of(g, u);
        if (!waited) {
            // The lane that waits is the one that issues the copies: elect.sync chooses the same lane of the same mask
            // every time.  (A vote orders no memory between lanes; a warp barrier would, at 1.9 % of the shortest prompt.)
            bool ready = true;
            if (elect_one()) {
                ready = await_step(p, sh, step - 1, before);
                stamp_at(p, step, 3);
            }
            if (!__all_sync(0xffffffffu, ready)) return false;
            // the step before wrote through the generic proxy, TMA reads through the async proxy
            asm volatile("fence.proxy.async;" ::: "memory");
            waited = true;
        }
        for (int kb = x.kb0; kb < x.kb1; kb += g.deep) {
            if (at.round > 0 && !wait_warp(sh, &sh.empty[at.s], (at.round - 1) & 1)) {
                give_up(p, sh, MB_ST_PIPE_TIMEOUT, step, 2);
                return false;
            }
            if (elect_one()) {
                mbar_arrive_expect_tx(&sh.full[at.s], g.b_bytes);
                tma_load_blocks(sh.ring + at.s * kStageBytes + g.a_bytes, map, x.tile_t * g.tokens, kb,
                                &sh.full[at.s]);
            }
            __syncwarp();
            at.next();
        }
    }
    return true;
}

__device__ __forceinline__ bool issue_products(const Params& p, const Shared& sh, const Gemm& g, RingPlace& at,
                                               unsigned int tmem, int& turn, int step) {
    // where the second accumulator's weights start: the other matrix, or feature 128
    const unsigned long long second = (g.pair ? g.a_bytes / 2 : 128 * 128) / 16;
    for (int u = first_unit(g.first); u < g.units; u += gridDim.x, ++turn) {
        const Unit x = unit_of(g, u);
        const int buf = turn & 1;
        if (turn >= 2 && !wait_warp(sh, &sh.acc_empty[buf], ((turn >> 1) - 1) & 1)) {
            give_up(p, sh, MB_ST_PIPE_TIMEOUT, step, 3);
            return false;
        }
        tc_fence_after();
        const unsigned int acc = tmem + buf * 256;
        for (int kb = x.kb0; kb < x.kb1; kb += g.deep) {
            if (!wait_warp(sh, &sh.full[at.s], at.round & 1)) {
                give_up(p, sh, MB_ST_PIPE_TIMEOUT, step, 4);
                return false;
            }
            if (u == first_unit(g.first) && kb == x.kb0 && (threadIdx.x & 31) == 0) stamp_at(p, step, 4);
            tc_fence_after();
            const unsigned int base = smem_u32(sh.ring + at.s * kStageBytes);
            const int blocks = min(g.deep, x.kb1 - kb);
            if (elect_one()) {
                unsigned long long da = umma_desc(base), db = umma_desc(base + g.a_bytes);
                unsigned int accumulate = kb != x.kb0 ? 1u : 0u;
                for (int j = 0; j < blocks; ++j) {
#pragma unroll
                    for (int k = 0; k < kTileK / 16; ++k) {
                        umma_bf16(acc, da + 2 * k, db + 2 * k, g.idesc, accumulate);
                        if (g.accs == 2) umma_bf16(acc + g.tokens, da + second + 2 * k, db + 2 * k, g.idesc, accumulate);
                        accumulate = 1u;
                    }
                    da += g.rows * 8;  // descriptors count 16 bytes
                    db += g.tokens * 8;
                }
                umma_commit(&sh.empty[at.s]);
                if (kb + g.deep >= x.kb1) umma_commit(&sh.acc_full[buf]);
            }
            __syncwarp();
            at.next();
        }
        if ((threadIdx.x & 31) == 0) stamp_at(p, step, 5);
    }
    return true;
}

__device__ __forceinline__ void tmem_load8_pair(unsigned int addr_v, unsigned int addr_u, float (&v)[8],
                                                float (&u)[8]) {
    unsigned int r[8], q[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(addr_v)
                 : "memory");
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]), "=r"(q[4]), "=r"(q[5]), "=r"(q[6]), "=r"(q[7])
                 : "r"(addr_u)
                 : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        v[i] = __uint_as_float(r[i]);
        u[i] = __uint_as_float(q[i]);
    }
}

// ---------------------------------------------------------------------------------------
// Accumulators -> memory.  A thread has one feature (of both matrices of a pair) and 8 tokens at a time: the
// lanes of a warp write neighbouring features of a token.  With 64-row products the sixteen rows 16 i ..
// lie in lanes 32 i .. 32 i + 15.  The two sets of four warps take the groups of tokens in turn.
// ---------------------------------------------------------------------------------------
// act(gate) * up of eight tokens, bf16 pairs.  One branch for eight elements: their chains have to overlap.
__device__ __forceinline__ void gate_pairs(unsigned int (&out)[4], const float (&v)[8], const float (&up)[8],
                                           int epilogue) {
    float x[8], t[8];
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        const unsigned int both = pack_bf16_pair(v[i], v[i + 1]);
        t[i] = x[i] = lo_bf16(both);
        t[i + 1] = x[i + 1] = hi_bf16(both);
    }
    if (epilogue == MB_EPI_GELU_TANH_MUL) {
#pragma unroll
        for (int i = 0; i < 8; ++i) t[i] = gelu_exponent(x[i]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = sigmoid_product(x[i], t[i]);
#pragma unroll
    for (int i = 0; i < 4; ++i)
        out[i] = mul_bf16_pair(pack_bf16_pair(x[2 * i], x[2 * i + 1]), pack_bf16_pair(up[2 * i], up[2 * i + 1]));
}

// Eight tokens of this lane's feature, and of its neighbour's: an even lane writes both features of the even
// tokens, an odd lane those of the odd ones (4 bytes a store instead of 2).  Tokens from `left` on, and
// every `period` further, are `jump` elements further away.
__device__ __forceinline__ void store_pairs(unsigned short* dst, int pitch, const unsigned int (&v)[4], int lane,
                                            bool mine, int count, int left = 0x7fffffff, int period = 1,
                                            size_t jump = 0) {
    const int odd = lane & 1;
    unsigned short* at = dst - odd;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const unsigned int other = __shfl_xor_sync(0xffffffffu, v[i], 1);
        const unsigned int word = odd ? __byte_perm(other, v[i], 0x7632) : __byte_perm(v[i], other, 0x5410);
        const int t = 2 * i + odd;
        if (mine && t < count) {
            size_t offset = static_cast<size_t>(t) * pitch;
            if (t >= left) offset += static_cast<size_t>((t - left) / period + 1) * jump;
            *reinterpret_cast<unsigned int*>(at + offset) = word;
        }
    }
}

__device__ __forceinline__ bool drain_units(const Params& p, const Shared& sh, const Gemm& g, int proj,
                                            const LayerArgs& layer, int wid, int lane, unsigned int tmem,
                                            int& turn, int step) {
    const int quarter = wid & 3, set = wid >> 2;
    const unsigned int lane_addr = tmem + (static_cast<unsigned int>(quarter * 32) << 16);
    const int local = g.wide ? quarter * 32 + lane : quarter * 16 + lane;
    const bool live = g.wide || lane < 16;
    for (int u = first_unit(g.first); u < g.units; u += gridDim.x, ++turn) {
        const Unit x = unit_of(g, u);
        const int buf = turn & 1;
        if (!wait_warp(sh, &sh.acc_full[buf], (turn >> 1) & 1)) {
            if (lane == 0) give_up(p, sh, MB_ST_PIPE_TIMEOUT, step, 5);
            return false;
        }
        tc_fence_after();
        if (wid == 0 && lane == 0) stamp_at(p, step, 6);
        const int t0 = x.tile_t * g.tokens, limit = min(g.tokens, p.rows - t0);
        const int n = g.n[x.seg];
#pragma unroll 1
        for (int half = 0; half < (g.pair ? 1 : g.accs); ++half) {
            const int row = half * 128 + local, feature = x.f0 + row;
            const bool mine = live && row < g.rows && feature < n;
            const unsigned int addr = lane_addr + buf * 256 + half * g.tokens;
            const unsigned int second = g.pair ? addr + g.tokens : addr;
            // where the feature's column is, and how far the next token's is from it
            unsigned short* out = nullptr;
            float* sum = nullptr;
            int pitch, head = 0, i0 = 0;
            const unsigned short* bias = nullptr;
            const unsigned int* rotary = nullptr;
            if (proj == kProjGated) {
                pitch = p.intermediate;
                out = p.glu + feature;
            } else if (proj == kProjHead) {
                pitch = n;
                out = p.logits + feature;
                bias = p.head_bias;
            } else if (proj == kProjQkv) {
                // pairs of elements i and i + D / 2 of a head; q's and k's are turned by the row's angle
                head = feature / g.half;
                i0 = feature - head * g.half;
                pitch = 2 * n;
                out = (x.seg == 0 ? p.q : layer.kv[x.seg - 1]) + 2 * head * g.half + i0;
                bias = layer.bias[x.seg];
                if (x.seg < 2) rotary = p.rotary + static_cast<size_t>(t0) * g.half + i0;
            } else {
                pitch = p.hidden_size;
                sum = p.parts + (static_cast<size_t>(x.slice) * p.rows + t0) * pitch + feature;
            }
            // caches of keys and values have kv_rows rows for each prompt of the batch
            const bool gaps = proj == kProjQkv && x.seg > 0 && p.kv_rows != p.tokens;
            float b1 = 0.f, b2 = 0.f;
            if (mine && bias != nullptr) {
                b1 = bf16_bits_to_float(__ldg(bias + (proj == kProjQkv ? 2 * head * g.half + i0 : feature)));
                b2 = bf16_bits_to_float(__ldg(bias + (proj == kProjQkv ? (2 * head + 1) * g.half + i0 : feature)));
            }
            unsigned int cs[8];
            auto ask_angles = [&](int col) {  // a group ahead: they come from L2
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    cs[i] = mine && col + i < limit ? __ldcg(rotary + static_cast<size_t>(col + i) * g.half) : 0u;
            };
            if (rotary != nullptr) ask_angles(8 * set);
#pragma unroll 1
            for (int col = 8 * set; col < limit; col += 16) {
                float v[8], w[8];
                tmem_load8_pair(addr + col, second + col, v, w);
                const int count = limit - col;
                if (sum != nullptr) {
                    if (mine) {
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            if (i < count) __stcg(sum + static_cast<size_t>(col + i) * pitch, v[i]);
                    }
                    continue;
                }
                unsigned int v2[4], w2[4];
                if (proj == kProjGated) {
                    gate_pairs(v2, v, w, p.activation);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        v2[i] = pack_bf16_pair(v[2 * i] + b1, v[2 * i + 1] + b1);
                        w2[i] = pack_bf16_pair(w[2 * i] + b2, w[2 * i + 1] + b2);
                    }
                }
                if (rotary != nullptr) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const unsigned int c = __byte_perm(cs[2 * i], cs[2 * i + 1], 0x5410);
                        const unsigned int s = __byte_perm(cs[2 * i], cs[2 * i + 1], 0x7632);
                        const unsigned int x1 = v2[i], x2 = w2[i];
                        v2[i] = sub_bf16_pair(mul_bf16_pair(x1, c), mul_bf16_pair(x2, s));
                        w2[i] = add_bf16_pair(mul_bf16_pair(x2, c), mul_bf16_pair(x1, s));
                    }
                    if (x.seg == 0 && p.q_scale != 0.f && p.q_scale != 1.f) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            v2[i] = pack_bf16_pair(lo_bf16(v2[i]) * p.q_scale, hi_bf16(v2[i]) * p.q_scale);
                            w2[i] = pack_bf16_pair(lo_bf16(w2[i]) * p.q_scale, hi_bf16(w2[i]) * p.q_scale);
                        }
                    }
                    ask_angles(col + 16);
                }
                if (!gaps) {
                    unsigned short* dst = out + static_cast<size_t>(t0 + col) * pitch;
                    store_pairs(dst, pitch, v2, lane, mine, count);
                    if (proj == kProjQkv) store_pairs(dst + g.half, pitch, w2, lane, mine, count);
                } else {
                    const int r = t0 + col, b = r / p.tokens, left = (b + 1) * p.tokens - r;
                    const size_t gap = static_cast<size_t>(p.kv_rows - p.tokens) * pitch;
                    unsigned short* dst = out + static_cast<size_t>(r) * pitch + b * gap;
                    store_pairs(dst, pitch, v2, lane, mine, count, left, p.tokens, gap);
                    store_pairs(dst + g.half, pitch, w2, lane, mine, count, left, p.tokens, gap);
                }
            }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.acc_empty[buf]);
    }
    return true;
}

// ---------------------------------------------------------------------------------------
// Rows: the sum of a reduction's slices, the residual, the norm (and the embedding gather before layer 0).
// Row r is always CTA r mod grid's: it reads back the residual it wrote itself.
// ---------------------------------------------------------------------------------------
template <int AT_ONCE>
__device__ __forceinline__ bool row_step(const Params& p, const Shared& sh, int tid, int lane, float* sums,
                                         const unsigned short* norm, const unsigned short* bias, int slices,
                                         int step, unsigned int before) {
    constexpr int kShare = kWorkers / AT_ONCE;  // threads of a row; a thread has AT_ONCE vectors of it
    const int H = p.hidden_size, vectors = H / 8, sub = tid / kShare, t = tid - sub * kShare;
    const uint4* wv = reinterpret_cast<const uint4*>(norm);
    const size_t stride = static_cast<size_t>(p.rows) * H / 4;
    int done = 0, turn = 0;
    uint4 g[AT_ONCE];
#pragma unroll
    for (int j = 0; j < AT_ONCE; ++j)
        if (t + j * kShare < vectors) g[j] = __ldg(wv + t + j * kShare);
#pragma unroll 1
    for (int r0 = blockIdx.x * AT_ONCE; r0 < p.rows; r0 += gridDim.x * AT_ONCE, ++turn) {
        const int r = r0 + sub;
        const bool row_live = r < p.rows;
        done += min(AT_ONCE, p.rows - r0);
        uint4 v[AT_ONCE];
        uint4* hidden = reinterpret_cast<uint4*>(p.hidden + static_cast<size_t>(r) * H) + t;
#pragma unroll
        for (int j = 0; j < AT_ONCE; ++j) {
            v[j] = make_uint4(0u, 0u, 0u, 0u);
            if (slices > 0 && row_live && t + j * kShare < vectors) v[j] = hidden[j * kShare];
        }
        if (slices > 0) {
            if (turn == 0 && !workers_await(p, sh, tid, step - 1, before)) return false;
            if (tid == 0) stamp_at(p, step, 3);
#pragma unroll
            for (int j = 0; j < AT_ONCE; ++j) {
                const int idx = t + j * kShare;
                if (!row_live || idx >= vectors) continue;
                const float4* src = reinterpret_cast<const float4*>(p.parts + static_cast<size_t>(r) * H) + 2 * idx;
                float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
#pragma unroll 1
                for (int s = 0; s < slices; s += 4) {  // four at a time; past the last one it is read again, unused
                    float4 a[4], b[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float4* at = src + min(s + i, slices - 1) * stride;
                        a[i] = __ldcg(at);
                        b[i] = __ldcg(at + 1);
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (s + i >= slices) break;
                        lo.x += a[i].x;
                        lo.y += a[i].y;
                        lo.z += a[i].z;
                        lo.w += a[i].w;
                        hi.x += b[i].x;
                        hi.y += b[i].y;
                        hi.z += b[i].z;
                        hi.w += b[i].w;
                    }
                }
                float y[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
                if (bias != nullptr) {
                    const uint4 c = __ldg(reinterpret_cast<const uint4*>(bias) + idx);
                    const unsigned int w[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
                    for (int i = 0; i < 8; ++i) y[i] += i & 1 ? hi_bf16(w[i / 2]) : lo_bf16(w[i / 2]);
                }
                const unsigned int h[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
                unsigned int sum[4];
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    sum[e] = pack_bf16_pair(lo_bf16(h[e]) + bf16_round(y[2 * e]),
                                            hi_bf16(h[e]) + bf16_round(y[2 * e + 1]));
                v[j] = make_uint4(sum[0], sum[1], sum[2], sum[3]);
            }
        } else if (row_live) {
            long long id = p.ids[r];
            if (id < 0 || id >= p.vocab_in) {
                if (t == 0) record_status(p.ctl, MB_ST_TOKEN_RANGE, 0, r);
                id = 0;
            }
            const uint4* src = reinterpret_cast<const uint4*>(p.table + static_cast<size_t>(id) * H) + t;
#pragma unroll
            for (int j = 0; j < AT_ONCE; ++j) {
                if (t + j * kShare >= vectors) continue;
                v[j] = __ldg(src + j * kShare);
                if (p.embed_scale != 0.f) v[j] = scale_vector(v[j], p.embed_scale);
            }
            const int half = p.head_dim / 2;
            for (int i = t; i < half; i += kShare) {
                const float f = p.invfreq_bf16
                                    ? bf16_bits_to_float(reinterpret_cast<const unsigned short*>(p.inv_freq)[i])
                                    : reinterpret_cast<const float*>(p.inv_freq)[i];
                const float angle = static_cast<float>(p.pos[r]) * f;
                float sn, cn;
                sincosf(angle, &sn, &cn);
                p.rotary[static_cast<size_t>(r) * half + i] = pack_bf16(cn * p.rope_scale, sn * p.rope_scale);
            }
        }
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < AT_ONCE; ++j) {
            ss += sum_squares(v[j]);
            if (row_live && t + j * kShare < vectors) hidden[j * kShare] = v[j];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (lane == 0) sums[(tid >> 5) + 8 * (turn & 1)] = ss;
        if (tid == 0) stamp_at(p, step, 4);
        named_barrier(1, kWorkers);
        float total = 0.f;
#pragma unroll
        for (int i = 0; i < 8 / AT_ONCE; ++i) total += sums[sub * (8 / AT_ONCE) + i + 8 * (turn & 1)];
        const float inv = 1.0f / sqrtf(total / static_cast<float>(H) + p.eps);
        uint4* dst = reinterpret_cast<uint4*>(p.normed + static_cast<size_t>(r) * H) + t;
#pragma unroll
        for (int j = 0; j < AT_ONCE; ++j)
            if (row_live && t + j * kShare < vectors) dst[j * kShare] = normalise_vector(v[j], g[j], inv, p.norm_kind);
    }
    return workers_done(p, sh, tid, step, done, true);
}

// ---------------------------------------------------------------------------------------
// Attention: a unit is 32 query rows of one head.  Two groups of 16 rows x four groups of keys (later, of value
// columns) are the eight warps' shares.  A prompt of one block of keys keeps its scores in registers between the
// row sums and the probabilities; a longer one goes over its keys twice, so that probabilities are
// rounded after normalisation.  mma.sync: a unit of a short prompt is 2 to 17 MFLOP, and its time is
// the chain of loads and row sums around the products.  Its operands take the ring's place: the
// weight producer of a CTA that has units here waits for attn_done.
// ---------------------------------------------------------------------------------------
constexpr int kOneBlock = 128;  // keys a prompt may have for the form that needs one block of them
__host__ __device__ constexpr int attention_block(int D, bool one) { return !one && D == 256 ? 64 : kOneBlock; }
constexpr int attention_bytes(int D, bool one) {
    return (kAttnRows * (D + 8) + (one ? 2 : 4) * attention_block(D, one) * (D + 8) +
            kAttnRows * (attention_block(D, one) + 8)) * 2 + kAttnRows * 4 * 2 * 4;
}
static_assert(attention_bytes(128, false) <= kRingBytes && attention_bytes(256, false) <= kRingBytes &&
                  attention_bytes(256, true) <= kRingBytes, "attention's operands lie in the ring");

// `count` rows of D elements to pitch D + 8; rows from `live` on are zero (0 x NaN would not be 0).
template <int D>
__device__ __forceinline__ void copy_rows(unsigned short* dst, const unsigned short* src, size_t pitch, int count,
                                          int live, int tid) {
#pragma unroll 4
    for (int e = tid; e < count * (D / 8); e += kWorkers) {
        const int r = e / (D / 8), c = (e - r * (D / 8)) * 8;
        if (r < live)
            cp_async_16(dst + r * (D + 8) + c, src + r * pitch + c);
        else
            *reinterpret_cast<uint4*>(dst + r * (D + 8) + c) = make_uint4(0u, 0u, 0u, 0u);
    }
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void copies_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
}

template <int D, bool ONE>
__device__ __forceinline__ void attention_unit(const Params& p, const LayerArgs& layer, unsigned char* smem, int u,
                                               int tid, int warp, int lane) {
    constexpr int P = D + 8, KB = attention_block(D, ONE), KW = KB / 4, NT = KW / 8, PP = KB + 8;
    constexpr int kBuffers = ONE ? 1 : 2;
    const int T = p.tokens, group = p.heads / p.kv_heads;
    // the last rows see the most keys: they come first
    const int head = u % p.heads, rest = u / p.heads;
    const int b = rest % p.batch, block = p.attn_blocks - 1 - rest / p.batch;
    const int kvh = head / group, q0 = block * kAttnRows;
    const int queries = min(kAttnRows, T - q0), seen = min(T, q0 + kAttnRows);
    const int nblocks = ONE ? 1 : (seen + KB - 1) / KB;
    unsigned short* Qs = reinterpret_cast<unsigned short*>(smem);
    unsigned short* Ks = Qs + kAttnRows * P;      // [kBuffers][KB][P]
    unsigned short* Vs = Ks + kBuffers * KB * P;  // [kBuffers][KB][P]
    unsigned short* Ps = Vs + kBuffers * KB * P;  // [32][PP]
    float* stats = reinterpret_cast<float*>(Ps + kAttnRows * PP);  // [2][4 groups][32 rows]
    const int q_dim = p.heads * D, kv_dim = p.kv_heads * D;
    const size_t kv_at = static_cast<size_t>(b) * p.kv_rows * kv_dim + kvh * D;
    const unsigned short *queries_at = p.q + static_cast<size_t>(b * T + q0) * q_dim + head * D;
    const unsigned short *keys = layer.kv[0] + kv_at, *values = layer.kv[1] + kv_at;
    const int rg = warp & 1, kg = warp >> 1, gid = lane >> 2, tq = lane & 3;
    constexpr float kLog2e = 1.4426950408889634f;

    auto copy_keys = [&](int j) {
        copy_rows<D>(Ks + (j & 1) * KB * P, keys + static_cast<size_t>(j) * KB * kv_dim, kv_dim,
                     min(KB, (seen - j * KB + 31) / 32 * 32), seen - j * KB, tid);
    };
    auto copy_values = [&](int j) {
        copy_rows<D>(Vs + (j & 1) * KB * P, values + static_cast<size_t>(j) * KB * kv_dim, kv_dim,
                     min(KB, (seen - j * KB + 31) / 32 * 32), seen - j * KB, tid);
    };
    // scores of this warp's 16 rows and KW keys of block j, with the operator's rounding points
    float s[4 * NT];
    auto scores = [&](int j) {
        float acc[NT][4];
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[t][i] = 0.f;
        const int key0 = j * KB + kg * KW;
        const unsigned short* block_keys = Ks + (j & 1) * KB * P + kg * KW * P;
        if (key0 < seen) {
#pragma unroll 2
            for (int kk = 0; kk < D / 16; ++kk) {
                unsigned int a[4], bf[4];
                ldmatrix_x4(a, Qs + (rg * 16 + (lane & 15)) * P + kk * 16 + (lane >> 4) * 8);
#pragma unroll
                for (int np = 0; np < NT / 2; ++np) {
                    ldmatrix_x4(bf, block_keys + (np * 16 + ((lane >> 4) & 1) * 8 + (lane & 7)) * P + kk * 16 +
                                        ((lane >> 3) & 1) * 8);
                    mma_bf16_16816(acc[2 * np], a[0], a[1], a[2], a[3], bf[0], bf[1]);
                    mma_bf16_16816(acc[2 * np + 1], a[0], a[1], a[2], a[3], bf[2], bf[3]);
                }
            }
        }
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int key = key0 + t * 8 + 2 * tq + (i & 1), row = q0 + rg * 16 + gid + (i >> 1) * 8;
                const float x = bf16_round(bf16_round(acc[t][i]) * p.softmax_scale);
                s[4 * t + i] = key <= row && key < T ? x : -INFINITY;
            }
    };

    copy_rows<D>(Qs, queries_at, q_dim, kAttnRows, queries, tid);
    copy_keys(0);
    copies_commit();
    if (nblocks == 1) copy_values(0);
    copies_commit();

    // ---- first sweep: each warp's row maxima and denominators over its own keys ----
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll 1
    for (int j = 0; j < nblocks; ++j) {
        if (j + 1 < nblocks) copy_keys(j + 1);
        copies_commit();
        // in flight at most: the next block's keys, and a single block's values
        if (nblocks == 1)
            copies_wait<2>();
        else
            copies_wait<1>();
        named_barrier(1, kWorkers);
        scores(j);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float top = m[h];
#pragma unroll
            for (int t = 0; t < NT; ++t) top = fmaxf(top, fmaxf(s[4 * t + 2 * h], s[4 * t + 2 * h + 1]));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
            const float ref = top == -INFINITY ? 0.f : top;
            l[h] *= exp2_approx((m[h] - ref) * kLog2e);
#pragma unroll
            for (int t = 0; t < NT; ++t)
                l[h] += exp2_approx(__fmaf_rn(s[4 * t + 2 * h], kLog2e, -ref * kLog2e)) +
                        exp2_approx(__fmaf_rn(s[4 * t + 2 * h + 1], kLog2e, -ref * kLog2e));
            m[h] = top;
        }
        if (nblocks > 1) named_barrier(1, kWorkers);  // the block after next takes this one's place
    }
    if (nblocks > 1) {
        copy_keys(0);
        copy_values(0);
        copies_commit();
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 1);
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 2);
        const int at = kg * 32 + rg * 16 + gid + 8 * h;
        if (tq == 0) {
            stats[at] = m[h];
            stats[128 + at] = l[h];
        }
    }
    named_barrier(1, kWorkers);
    float inv[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int row = rg * 16 + gid + 8 * h;
        m[h] = fmaxf(fmaxf(stats[row], stats[32 + row]), fmaxf(stats[64 + row], stats[96 + row]));
        if (m[h] == -INFINITY) m[h] = 0.f;
        float total = 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            total += stats[128 + 32 * q + row] * exp2_approx((stats[32 * q + row] - m[h]) * kLog2e);
        inv[h] = total > 0.f ? __frcp_rn(total) : 0.f;
    }

    // ---- second sweep: probabilities, and their products with the values (16 rows x D / 4 columns a warp) ----
    float o[D / 32][4];
#pragma unroll
    for (int t = 0; t < D / 32; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) o[t][i] = 0.f;
    const int d0 = kg * (D / 4);
#pragma unroll 1
    for (int j = 0; j < nblocks; ++j) {
        if (nblocks > 1) {
            if (j + 1 < nblocks) {
                copy_keys(j + 1);
                copy_values(j + 1);
            }
            copies_commit();
            copies_wait<1>();
            named_barrier(1, kWorkers);
            scores(j);
        }
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float lo = exp2_approx(__fmaf_rn(s[4 * t + 2 * h], kLog2e, -m[h] * kLog2e)) * inv[h];
                const float hi = exp2_approx(__fmaf_rn(s[4 * t + 2 * h + 1], kLog2e, -m[h] * kLog2e)) * inv[h];
                *reinterpret_cast<unsigned int*>(Ps + (rg * 16 + gid + 8 * h) * PP + kg * KW + t * 8 + 2 * tq) =
                    pack_bf16_pair(lo, hi);
            }
        if (nblocks == 1) copies_wait<0>();
        named_barrier(1, kWorkers);
        const unsigned short* block_values = Vs + (j & 1) * KB * P;
        const int steps = (min(KB, seen - j * KB) + 15) / 16;
#pragma unroll 2
        for (int kk = 0; kk < steps; ++kk) {
            unsigned int a[4], bf[4];
            ldmatrix_x4(a, Ps + (rg * 16 + (lane & 15)) * PP + kk * 16 + (lane >> 4) * 8);
#pragma unroll
            for (int dp = 0; dp < D / 64; ++dp) {
                ldmatrix_x4_trans(bf, block_values + (kk * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * P + d0 +
                                          dp * 16 + (lane >> 4) * 8);
                mma_bf16_16816(o[2 * dp], a[0], a[1], a[2], a[3], bf[0], bf[1]);
                mma_bf16_16816(o[2 * dp + 1], a[0], a[1], a[2], a[3], bf[2], bf[3]);
            }
        }
        named_barrier(1, kWorkers);  // probabilities, this block and, after the last one, every place are free
    }
    unsigned short* out = p.attn + static_cast<size_t>(b * T + q0) * q_dim + head * D + d0;
#pragma unroll
    for (int t = 0; t < D / 32; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = rg * 16 + gid + 8 * h;
            if (row < queries)
                *reinterpret_cast<unsigned int*>(out + static_cast<size_t>(row) * q_dim + t * 8 + 2 * tq) =
                    pack_bf16_pair(o[t][2 * h], o[t][2 * h + 1]);
        }
}

// ---------------------------------------------------------------------------------------
// Projection i of the launch: four a layer, then the logits.
struct Place {
    int proj, step, first_map;
};
__device__ __forceinline__ Place place_of(const Params& p, int i) {
    Place x;
    const int l = i >> 2, j = i & 3, base = 1 + l * kStepsPerLayer;
    x.proj = l == p.layers ? kProjHead : j;
    x.step = l == p.layers ? base : base + (j == 0 ? kQkv : j == 1 ? kOut : j == 2 ? kGated : kDown);
    x.first_map = j == 0 ? 0 : j == 1 ? 3 : j == 2 ? 4 : 6;
    return x;
}

// SMALL: at most one block of keys and one row of tokens a CTA.  Any number of CTAs works that run at once.
template <int D, bool SMALL>
__global__ void __launch_bounds__(kThreads, 1) prompt_kernel(const __grid_constant__ Params p) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ float sums[16];  // [2 turns][8 warps]
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    Shared sh;
    sh.ring = smem;
    sh.full = reinterpret_cast<unsigned long long*>(smem + kRingBytes);
    sh.empty = sh.full + kStages;
    sh.acc_full = sh.empty + kStages;
    sh.acc_empty = sh.acc_full + 2;
    sh.attn_done = sh.acc_empty + 2;
    sh.tmem_slot = reinterpret_cast<unsigned int*>(sh.attn_done + 1);
    sh.abort_flag = reinterpret_cast<volatile int*>(sh.tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&sh.full[s], 2);  // the two producers
            mbar_init(&sh.empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&sh.acc_full[b], 1);
            mbar_init(&sh.acc_empty[b], kWorkers / 32);
        }
        mbar_init(sh.attn_done, 1);
        sh.abort_flag[0] = 0;
        sh.abort_flag[1] = static_cast<int>(p.limit_us);
        mbar_init_fence();
    }
    if (warp == 1) tmem_alloc(sh.tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned int tmem = *sh.tmem_slot;
    const int attn_here = units_here(p.attn_units, 0);
    const int projections = 4 * p.layers + 1;

    if (warp == 0) {
        RingPlace at;
        bool ok = true;
        for (int i = 0; ok && i < projections; ++i) {
            const Place x = place_of(p, i);
            if (x.proj == kProjOut && attn_here > 0 && !wait_warp(sh, sh.attn_done, (i >> 2) & 1)) {
                give_up(p, sh, MB_ST_PIPE_TIMEOUT, x.step, 6);
                break;
            }
            ok = produce_weights(p, sh, p.gemm[x.proj], x.proj == kProjHead ? &p.head : p.layer[i >> 2].w + x.first_map,
                                 at, x.step);
        }
    } else if (warp == 1) {
        RingPlace at;
        int turn = 0;
        bool ok = true;
        for (int i = 0; ok && i < projections; ++i) {
            const Place x = place_of(p, i);
            ok = issue_products(p, sh, p.gemm[x.proj], at, tmem, turn, x.step);
        }
    } else if (warp == 2) {
        RingPlace at;
        bool ok = true;
        for (int i = 0; ok && i < projections; ++i) {
            const Place x = place_of(p, i);
            // the step before: rows, attention, rows, the gated projection, rows
            const int before = x.proj == kProjOut    ? p.attn_units
                               : x.proj == kProjDown ? p.gemm[kProjGated].units
                                                     : p.rows;
            ok = produce_activations(p, sh, p.gemm[x.proj], &p.b[x.proj], at, x.step, static_cast<unsigned int>(before));
        }
    } else if (warp >= 4) {
        const int tid = static_cast<int>(threadIdx.x) - 128, wid = warp - 4;
        for (int l = blockIdx.x; l < p.layers; l += gridDim.x)
            if (p.layer[l].length != nullptr && tid < p.length_count) p.layer[l].length[tid] = p.length_value;
        int turn = 0, kind = kRowsEnd, l = -1;  // the first rows are those before layer 0
        bool ok = true;
        for (int step = 0; ok && step < p.steps; ++step) {
            const bool last = step == p.steps - 1;
            const LayerArgs& layer = p.layer[min(max(l, 0), p.layers - 1)];
            if (kind == kRowsMid || kind == kRowsEnd) {
                const bool mid = kind == kRowsMid;
                const unsigned short* norm = mid               ? layer.norm[1]
                                             : l + 1 < p.layers ? p.layer[l + 1].norm[0]
                                                                : p.final_norm;
                const Gemm& g = p.gemm[mid ? kProjOut : kProjDown];
                const unsigned short* bias = mid ? layer.bias[3] : layer.bias[4];
                const int slices = step == 0 ? 0 : g.slices;
                ok = row_step<SMALL ? 1 : 4>(p, sh, tid, lane, sums, norm, bias, slices, step, g.units);
            } else if (kind == kAttention) {
                if (attn_here > 0) {
                    ok = workers_await(p, sh, tid, step - 1, p.gemm[kProjQkv].units);
                    if (tid == 0) stamp_at(p, step, 3);
                    if (ok) {
                        for (int u = blockIdx.x; u < p.attn_units; u += gridDim.x)
                            attention_unit<D, SMALL>(p, layer, sh.ring, u, tid, wid, lane);
                        // weights are copied to where the operands were
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        ok = workers_done(p, sh, tid, step, attn_here, true);
                        if (tid == 0) mbar_arrive(sh.attn_done);
                    }
                }
            } else {
                const int proj = last ? kProjHead : kind == kQkv ? kProjQkv : kind == kOut ? kProjOut
                                        : kind == kGated ? kProjGated : kProjDown;
                const Gemm& g = p.gemm[proj];
                ok = drain_units(p, sh, g, proj, layer, wid, lane, tmem, turn, step);
                ok = workers_done(p, sh, tid, step, units_here(g.units, g.first), ok);
            }
            if (tid == 0) stamp_at(p, step, 2);
            if (++kind == kStepsPerLayer) {
                kind = 0;
                ++l;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (*sh.abort_flag) {
        // copies this CTA issued may still be landing in its shared memory: give them time
        const unsigned long long start = global_timer_ns();
        while (global_timer_ns() - start < 200000ull) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == 1) tmem_dealloc(tmem, 512);
    // the CTA that is through last leaves the counters as the next launch wants them
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(p.counters + p.steps, 1u) == gridDim.x - 1) {
            for (int s = 0; s < p.steps + 2; ++s) p.counters[s] = 0u;
        }
    }
}

// SMs that a launch on `stream` may use: fewer than the device has in a green context, which is the current context's
// or the stream's.
int usable_sms(cudaStream_t stream, int device_sms) {
    typedef CUresult (*CurrentFn)(CUcontext*);
    typedef CUresult (*ContextResourceFn)(CUcontext, CUdevResource*, CUdevResourceType);
    typedef CUresult (*StreamGreenFn)(CUstream, CUgreenCtx*);
    typedef CUresult (*GreenResourceFn)(CUgreenCtx, CUdevResource*, CUdevResourceType);
    static const auto entry = [](const char* name) -> void* {
        void* symbol = nullptr;
        cudaDriverEntryPointQueryResult result;
        return cudaGetDriverEntryPoint(name, &symbol, cudaEnableDefault, &result) == cudaSuccess &&
                       result == cudaDriverEntryPointSuccess
                   ? symbol
                   : nullptr;
    };
    static const auto current = reinterpret_cast<CurrentFn>(entry("cuCtxGetCurrent"));
    static const auto of_context = reinterpret_cast<ContextResourceFn>(entry("cuCtxGetDevResource"));
    static const auto green_of = reinterpret_cast<StreamGreenFn>(entry("cuStreamGetGreenCtx"));
    static const auto of_green = reinterpret_cast<GreenResourceFn>(entry("cuGreenCtxGetDevResource"));
    int sms = device_sms;
    auto at_most = [&](const CUdevResource& room) {
        if (room.sm.smCount > 0 && static_cast<int>(room.sm.smCount) < sms) sms = static_cast<int>(room.sm.smCount);
    };
    CUdevResource room;
    CUcontext context = nullptr;
    CUgreenCtx green = nullptr;
    if (current != nullptr && of_context != nullptr && current(&context) == CUDA_SUCCESS && context != nullptr &&
        of_context(context, &room, CU_DEV_RESOURCE_TYPE_SM) == CUDA_SUCCESS)
        at_most(room);
    if (green_of != nullptr && of_green != nullptr && stream != nullptr && green_of(stream, &green) == CUDA_SUCCESS &&
        green != nullptr && of_green(green, &room, CU_DEV_RESOURCE_TYPE_SM) == CUDA_SUCCESS)
        at_most(room);
    return sms;
}

template <bool SMALL>
const void* kernel_for(int head_dim) {
    return head_dim == 64    ? reinterpret_cast<const void*>(&prompt_kernel<64, SMALL>)
           : head_dim == 128 ? reinterpret_cast<const void*>(&prompt_kernel<128, SMALL>)
                             : reinterpret_cast<const void*>(&prompt_kernel<256, SMALL>);
}
// One kernel per head size and form: neither carries the other's code.
const void* kernel_of(const Params& p) { return p.small ? kernel_for<true>(p.head_dim) : kernel_for<false>(p.head_dim); }

// ---------------------------------------------------------------------------------------
// Host: does a list of phases describe such a prefill, and how is each projection cut?
// ---------------------------------------------------------------------------------------
// Cost of a cut in microseconds.  An SM takes 72 bytes a nanosecond from L2 while all of them stream; weights up to a ring come before
// the step begins; a product of 16 elements takes 27 cycles to issue and works through two columns a cycle; a
// stage costs 250 cycles of barriers around its products; the last unit's accumulators are drained
// with nothing beside them; a further unit of the same CTA costs half a microsecond of refilling (1B, logits of 19
// tokens: 106 us in units of 56 features, 80 in units of 128).
struct Cut {
    Gemm gemm;
    double cost;
};
Cut best_cut(const int* n, int segments, bool pair, bool sliced, int half, int K, int M, int hidden, int grid) {
    Cut best;
    best.cost = 1e30;
    const int padded = (M + 15) / 16 * 16;
    const int kblocks = K / kTileK, mats = pair ? 2 : 1;
    long long features = 0;
    for (int s = 0; s < segments; ++s) features += n[s];
    const double hbm = 2.0 * features * mats * K / 6.2e6;
    for (int tiles_t = 1; tiles_t <= 32; tiles_t = tiles_t < 4 ? 2 * tiles_t : tiles_t + 1) {
        const int tokens = ((padded + tiles_t - 1) / tiles_t + 15) / 16 * 16;
        if (tiles_t > 1 && tokens * (tiles_t - 1) >= padded) continue;
        for (int rows = 8; rows * mats <= 256; rows += 8) {
            const int accs = pair || rows > 128 ? 2 : 1;
            const bool wide = rows > 64;
            // pairs of a head: whole halves of heads, or an equal part of one
            if (half > 0 && (rows < half ? half % rows != 0 : rows % half != 0)) continue;
            if (accs * tokens > 256) continue;
            const int block = 128 * (rows * mats + tokens);
            if (block > kStageBytes) continue;
            int tiles = 0;
            for (int s = 0; s < segments; ++s) tiles += (n[s] + rows - 1) / rows;
            for (int slices = 1; slices <= (sliced ? 16 : 1); ++slices) {
                if (slices > 1 && kblocks / slices < 2) break;
                const int units = tiles * tiles_t * slices, waves = (units + grid - 1) / grid;
                const int kb = (kblocks + slices - 1) / slices;
                int deep = kStageBytes / block;
                if (deep > kb) deep = kb;
                const int stages = (kb + deep - 1) / deep;
                deep = (kb + stages - 1) / stages;
                const double a = 128.0 * rows * mats * kb;
                const double ahead = a < kStages * 128.0 * rows * mats * deep ? a : kStages * 128.0 * rows * mats * deep;
                const double load = (waves * (a + 128.0 * tokens * kb) - ahead) / 7.2e4;
                const double issue = tokens / 2.0 > 27.0 ? tokens / 2.0 : 27.0;
                const double product = waves * (kb * 4.0 * accs * issue + 250.0 * stages) / 1.85e3;
                const double drain = tokens * (pair ? 0.047 : accs * 0.012) * (wide ? 1.0 : 0.6);
                double cost = load > product ? load : product;
                if (cost < hbm) cost = hbm;
                if (cost < waves * drain) cost = waves * drain;
                cost += drain + 0.5 * (waves - 1);
                if (sliced) cost += slices * 8.0 * M * hidden / 5.0e6 + 0.05 * slices;
                if (cost >= best.cost - 1e-9) continue;
                best.cost = cost;
                Gemm& g = best.gemm;
                std::memset(&g, 0, sizeof(g));
                g.rows = rows;
                g.tokens = tokens;
                g.tiles_t = tiles_t;
                int at = 0;
                for (int s = 0; s < 3; ++s) {
                    g.start[s] = s < segments ? at : 0x7fffffff;
                    g.n[s] = s < segments ? n[s] : 0;
                    if (s < segments) at += (n[s] + rows - 1) / rows;
                }
                g.tiles = tiles;
                g.slices = slices;
                g.kblocks = kblocks;
                g.units = units;
                g.accs = accs;
                g.pair = pair ? 1 : 0;
                g.wide = wide ? 1 : 0;
                g.half = half;
                g.idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<unsigned int>(tokens >> 3) << 17) |
                          (static_cast<unsigned int>((wide ? 128 : 64) >> 4) << 24);
                g.deep = deep;
                g.a_bytes = 128 * rows * mats * deep;
                g.b_bytes = 128 * tokens * deep;
            }
        }
    }
    return best;
}

constexpr int kPhasesPerLayer = 8;  // norm, q|k|v, rotary, attention, o, norm, gate|up, down

// The records of a decoder prefill in the planner's order, every layer of one shape.
bool describes_prompt(const std::vector<mb_phase>& f, unsigned int n_dynamic, int sm_count) {
    const int count = static_cast<int>(f.size());
    if (count < 1 + kPhasesPerLayer + 2 || (count - 3) % kPhasesPerLayer != 0) return false;
    const int layers = (count - 3) / kPhasesPerLayer;
    if (layers > kMaxLayers) return false;
    const mb_phase& e = f[0];
    if (e.body != MB_BODY_EMBED_ROWS) return false;
    const int M = e.i[MB_EM_I_ROWS], H = e.i[MB_EM_I_K];
    const int hidden = e.slot[MB_EM_S_OUT];
    if (H > 8 * kWorkers || H % kTileK != 0) return false;
    auto is_norm = [&](const mb_phase& P, const mb_phase& like) {
        return P.body == MB_BODY_RMSNORM_ROWS && P.i[MB_RN_I_ROWS] == M && P.i[MB_RN_I_K] == H &&
               P.i[MB_RN_I_KIND] == like.i[MB_RN_I_KIND] && P.f[MB_RN_F_EPS] == like.f[MB_RN_F_EPS] &&
               P.slot[MB_RN_S_X] == hidden && P.slot[MB_RN_S_OUT] == like.slot[MB_RN_S_OUT];
    };
    auto is_gemm = [&](const mb_phase& P, int nseg, int nmat, int x) {
        return P.body == MB_BODY_GEMM_TC && P.i[MB_GV_I_ROWS] == M && P.i[MB_GV_I_NSEG] == nseg &&
               P.i[MB_GV_I_NMAT] == nmat && P.slot[MB_GV_S_X] == x;
    };
    const mb_phase* one = &f[1];
    const int normed = one[0].slot[MB_RN_S_OUT];
    const long long weights = static_cast<long long>(H) * (one[1].i[MB_GV_I_N0] + one[1].i[MB_GV_I_N0 + 1] +
                                                           one[1].i[MB_GV_I_N0 + 2] + one[4].i[MB_GV_I_K] +
                                                           3ll * one[6].i[MB_GV_I_N0]);
    if (M > most_rows(weights)) return false;
    for (int l = 0; l < layers; ++l) {
        const mb_phase* P = &f[1 + l * kPhasesPerLayer];
        if (!is_norm(P[0], one[0]) || !is_norm(P[5], one[0])) return false;
        const mb_phase &qkv = P[1], &rope = P[2], &attn = P[3], &out = P[4], &gated = P[6], &down = P[7];
        if (!is_gemm(qkv, 3, 1, normed) || !is_gemm(out, 1, 1, attn.slot[MB_AP_S_OUT]) ||
            !is_gemm(gated, 1, 2, normed) || !is_gemm(down, 1, 1, gated.slot[MB_GV_S_OUT0]))
            return false;
        if (rope.body != MB_BODY_ROPE_ROWS || attn.body != MB_BODY_ATTN_PREFILL) return false;
        // the same shapes, options and buffers in every layer
        for (int j = 0; j < kPhasesPerLayer; ++j)
            if (std::memcmp(P[j].i, one[j].i, sizeof(P[j].i)) != 0 || std::memcmp(P[j].f, one[j].f, sizeof(P[j].f)) != 0)
                return false;
        const int D = attn.i[MB_AP_I_HEAD_DIM], heads = attn.i[MB_AP_I_HEADS], kv = attn.i[MB_AP_I_KV_HEADS];
        const int T = attn.i[MB_AP_I_TOKENS];
        const long long units = static_cast<long long>(attn.i[MB_AP_I_BATCH]) * heads * ((T + kAttnRows - 1) / kAttnRows);
        if (T > kOneBlock && (units + sm_count - 1) / sm_count * ((T + kOneBlock - 1) / kOneBlock) > kAttnSweeps) return false;
        if (attn.i[MB_AP_I_BATCH] * T != M || attn.i[MB_AP_I_CAUSAL] != 1 || attn.slot[MB_AP_S_MASK] >= 0) return false;
        // without scratch for transposed values the phase has another arithmetic (expf, exact division), which it keeps
        if (attn.slot[MB_AP_S_VT] < 0) return false;
        if (qkv.i[MB_GV_I_K] != H || qkv.i[MB_GV_I_EPILOGUE] != MB_EPI_NONE || qkv.i[MB_GV_I_N0] != heads * D ||
            qkv.i[MB_GV_I_N0 + 1] != kv * D || qkv.i[MB_GV_I_N0 + 2] != kv * D)
            return false;
        if (rope.i[MB_RP_I_ROWS] != M || rope.i[MB_RP_I_HEADS] != heads || rope.i[MB_RP_I_KV_HEADS] != kv ||
            rope.i[MB_RP_I_HEAD_DIM] != D || rope.slot[MB_RP_S_POS] != one[2].slot[MB_RP_S_POS] ||
            rope.slot[MB_RP_S_INVFREQ] != one[2].slot[MB_RP_S_INVFREQ])
            return false;
        for (int s = 0; s < 3; ++s)
            if (attn.slot[MB_AP_S_Q + s] != qkv.slot[MB_GV_S_OUT0 + s]) return false;
        if (rope.slot[MB_RP_S_Q] != qkv.slot[MB_GV_S_OUT0] || rope.slot[MB_RP_S_K] != qkv.slot[MB_GV_S_OUT0 + 1])
            return false;
        if (attn.slot[MB_AP_S_OUT] != one[3].slot[MB_AP_S_OUT] || attn.slot[MB_AP_S_Q] != one[3].slot[MB_AP_S_Q])
            return false;
        // keys and values of their own per layer (caches the caller reads): all three records say so
        const int capacity = attn.i[MB_AP_I_KV_CAPACITY];
        if (capacity > 0) {
            if (qkv.i[MB_GV_I_OUT_TOKENS] != T || qkv.i[MB_GV_I_OUT_CAPACITY] != capacity ||
                rope.i[MB_RP_I_K_TOKENS] != T || rope.i[MB_RP_I_K_CAPACITY] != capacity || capacity < T)
                return false;
        } else if (qkv.i[MB_GV_I_OUT_TOKENS] != 0 || rope.i[MB_RP_I_K_TOKENS] != 0 || rope.slot[MB_RP_S_LEN] >= 0 ||
                   qkv.slot[MB_GV_S_OUT0 + 1] != one[1].slot[MB_GV_S_OUT0 + 1] ||
                   qkv.slot[MB_GV_S_OUT0 + 2] != one[1].slot[MB_GV_S_OUT0 + 2]) {
            return false;
        }
        if (rope.i[MB_RP_I_LEN_COUNT] > kWorkers) return false;
        for (const mb_phase* G : {&out, &down})
            if (G->i[MB_GV_I_EPILOGUE] != MB_EPI_RESIDUAL || G->i[MB_GV_I_N0] != H ||
                G->slot[MB_GV_S_RESIDUAL] != hidden || G->slot[MB_GV_S_OUT0] != hidden || G->i[MB_GV_I_OUT_TOKENS] != 0)
                return false;
        if (down.i[MB_GV_I_K] % kTileK != 0 || out.i[MB_GV_I_K] != heads * D || gated.i[MB_GV_I_K] != H || down.i[MB_GV_I_K] != gated.i[MB_GV_I_N0] ||
            gated.slot[MB_GV_S_BIAS0] >= 0 || gated.i[MB_GV_I_OUT_TOKENS] != 0 ||
            gated.slot[MB_GV_S_OUT0] != one[6].slot[MB_GV_S_OUT0])
            return false;
    }
    const mb_phase &last_norm = f[count - 2], &head = f[count - 1];
    if (!is_norm(last_norm, one[0]) || !is_gemm(head, 1, 1, normed) || head.i[MB_GV_I_K] != H ||
        head.i[MB_GV_I_EPILOGUE] != MB_EPI_NONE || head.i[MB_GV_I_OUT_TOKENS] != 0 || head.i[MB_GV_I_N0] % 2 != 0)
        return false;
    // buffers between the steps: all distinct, none given per launch
    const int own[] = {hidden, normed, one[3].slot[MB_AP_S_OUT], one[6].slot[MB_GV_S_OUT0]};
    for (int a = 0; a < 4; ++a) {
        if (own[a] < static_cast<int>(n_dynamic)) return false;
        for (int b = 0; b < a; ++b)
            if (own[a] == own[b]) return false;
    }
    return true;
}

// Sizes and options of such a list, and how its projections are cut.
void plan_steps(const std::vector<mb_phase>& f, int grid, unsigned int wait_limit_us, Params* params) {
    Params& p = *params;
    std::memset(&p, 0, sizeof(p));
    const mb_phase* one = &f[1];
    const mb_phase &attn = one[3], &rope = one[2], &head = f.back();
    p.limit_us = wait_limit_us;
    p.layers = (static_cast<int>(f.size()) - 3) / kPhasesPerLayer;
    p.steps = 2 + p.layers * kStepsPerLayer;
    p.rows = f[0].i[MB_EM_I_ROWS];
    p.hidden_size = f[0].i[MB_EM_I_K];
    p.vocab_in = f[0].i[MB_EM_I_VOCAB];
    p.embed_scale = f[0].f[MB_EM_F_SCALE];
    p.batch = attn.i[MB_AP_I_BATCH];
    p.tokens = attn.i[MB_AP_I_TOKENS];
    p.heads = attn.i[MB_AP_I_HEADS];
    p.kv_heads = attn.i[MB_AP_I_KV_HEADS];
    p.head_dim = attn.i[MB_AP_I_HEAD_DIM];
    p.kv_rows = attn.i[MB_AP_I_KV_CAPACITY] > 0 ? attn.i[MB_AP_I_KV_CAPACITY] : p.tokens;
    p.softmax_scale = attn.f[MB_AP_F_SCALE];
    p.intermediate = one[6].i[MB_GV_I_N0];
    p.activation = one[6].i[MB_GV_I_EPILOGUE];
    p.norm_kind = one[0].i[MB_RN_I_KIND];
    p.eps = one[0].f[MB_RN_F_EPS];
    p.invfreq_bf16 = rope.i[MB_RP_I_INVFREQ_BF16];
    p.rope_scale = rope.f[MB_RP_F_ROPE_SCALE];
    p.q_scale = rope.f[MB_RP_F_Q_SCALE];
    p.length_value = rope.i[MB_RP_I_LEN_VALUE];
    p.length_count = rope.i[MB_RP_I_LEN_COUNT] > 1 ? rope.i[MB_RP_I_LEN_COUNT] : 1;
    p.attn_blocks = (p.tokens + kAttnRows - 1) / kAttnRows;
    p.attn_units = p.batch * p.heads * p.attn_blocks;
    p.small = p.rows <= grid && p.tokens <= kOneBlock ? 1 : 0;

    const int M = p.rows, H = p.hidden_size;
    const int half = p.head_dim / 2, pairs[3] = {p.heads * half, p.kv_heads * half, p.kv_heads * half};
    p.gemm[kProjQkv] = best_cut(pairs, 3, true, false, half, H, M, H, grid).gemm;
    p.gemm[kProjOut] = best_cut(&one[4].i[MB_GV_I_N0], 1, false, true, 0, one[4].i[MB_GV_I_K], M, H, grid).gemm;
    p.gemm[kProjGated] = best_cut(&one[6].i[MB_GV_I_N0], 1, true, false, 0, H, M, H, grid).gemm;
    p.gemm[kProjDown] = best_cut(&one[7].i[MB_GV_I_N0], 1, false, true, 0, one[7].i[MB_GV_I_K], M, H, grid).gemm;
    p.gemm[kProjHead] = best_cut(&head.i[MB_GV_I_N0], 1, false, false, 0, H, M, H, grid).gemm;
    // CTAs with attention units cannot have their weights of the next projection ahead: others come first
    p.gemm[kProjOut].first = p.attn_units % grid;
}

}  // namespace prompt

struct PromptState {
    prompt::Params params;
    std::vector<mb_phase> phases;
    int grid = 0;
    unsigned char* scratch = nullptr;
    unsigned int n_dynamic = 0;
};

void prompt_destroy(PromptState* st) {
    if (st == nullptr) return;
    if (st->scratch != nullptr) cudaFree(st->scratch);
    delete st;
}

cudaError_t prompt_reset(PromptState* st) {
    if (st == nullptr) return cudaSuccess;
    return cudaMemset(st->params.counters, 0, sizeof(unsigned int) * (st->params.steps + 2));
}

// *out stays null where the phases are not a short prompt: they run as launches of their own.
cudaError_t prompt_create(const std::vector<mb_phase>& f, unsigned int n_dynamic, int sm_count,
                          unsigned int wait_limit_us, PromptState** out) {
    using namespace prompt;
    *out = nullptr;
    const char* env = std::getenv("MEGABAKE_B200_PREFILL_ONE_LAUNCH");
    if (env != nullptr && std::atoi(env) == 0) return cudaSuccess;
    // whoever sets how the launches of their own are cut or chained wants them
    for (const char* name : {"MEGABAKE_B200_ATTN_PARTS", "MEGABAKE_B200_ATTN_CHUNK", "MEGABAKE_B200_GEMM_PERSISTENT",
                             "MEGABAKE_B200_GEMM_BN", "MEGABAKE_B200_GEMM_STAGES", "MEGABAKE_B200_GEMM_SPLIT",
                             "MEGABAKE_B200_PREFILL_CHAIN"})
        if (std::getenv(name) != nullptr) return cudaSuccess;
    if (!describes_prompt(f, n_dynamic, sm_count)) return cudaSuccess;
    int device = 0, cooperative = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err == cudaSuccess) err = cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, device);
    if (err != cudaSuccess || cooperative == 0) return err;
    PromptState* st = new (std::nothrow) PromptState();
    if (st == nullptr) return cudaErrorMemoryAllocation;
    st->phases = f;
    st->grid = sm_count;
    st->n_dynamic = n_dynamic;
    Params& p = st->params;
    plan_steps(f, sm_count, wait_limit_us, &p);
    const int M = p.rows, H = p.hidden_size;
    const int slices = p.gemm[kProjOut].slices > p.gemm[kProjDown].slices ? p.gemm[kProjOut].slices
                                                                          : p.gemm[kProjDown].slices;
    auto room = [](size_t bytes) { return (bytes + 255) / 256 * 256; };
    const size_t parts = room(static_cast<size_t>(slices) * M * H * 4),
                 rotary = room(static_cast<size_t>(M) * (p.head_dim / 2) * 4), counters = room((p.steps + 2) * 4);
    err = cudaMalloc(&st->scratch, parts + rotary + counters);
    if (err == cudaSuccess) {
        p.parts = reinterpret_cast<float*>(st->scratch);
        p.rotary = reinterpret_cast<unsigned int*>(st->scratch + parts);
        p.counters = reinterpret_cast<unsigned int*>(st->scratch + parts + rotary);
        err = cudaMemset(p.counters, 0, counters);
    }
    // the form a launch takes, and the one it takes where it has fewer SMs
    const void* kernels[2] = {kernel_of(p), kernel_for<false>(p.head_dim)};
    int per_sm = 1;
    for (const void* kernel : kernels) {
        int room = 0;
        if (err == cudaSuccess) err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
        if (err == cudaSuccess) err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&room, kernel, kThreads, kSmemBytes);
        per_sm = room < per_sm ? room : per_sm;
    }
    if (err == cudaSuccess) err = cudaStreamSynchronize(cudaStreamLegacy);
    if (err != cudaSuccess || per_sm < 1) {
        prompt_destroy(st);
        return err;
    }
    *out = st;
    return cudaSuccess;
}

int prompt_cuts(const std::vector<mb_phase>& f, unsigned int n_dynamic, int sm_count, int* form, mb_prefill_cut* out) {
    using namespace prompt;
    *form = 0;
    if (!describes_prompt(f, n_dynamic, sm_count)) return MB_OK;
    Params* p = new (std::nothrow) Params;
    if (p == nullptr) return MB_ERR_RESOURCE;
    plan_steps(f, sm_count, 0, p);
    for (int j = 0; j < 5; ++j) {
        const Gemm& g = p->gemm[j];
        out[j] = {g.rows, g.tokens, g.slices, g.units, g.accs, g.first};
    }
    *form = p->small ? 1 : 2;
    delete p;
    return MB_OK;
}

int prompt_bind(PromptState* st, const std::vector<unsigned long long>& slots, Control* ctl) {
    using namespace prompt;
    Params& p = st->params;
    const std::vector<mb_phase>& f = st->phases;
    auto addr = [&](int s) -> unsigned long long { return s < 0 ? 0ull : slots[s]; };
    auto rows_at = [&](int s) { return reinterpret_cast<unsigned short*>(addr(s)); };
    const mb_phase* one = &f[1];
    p.ctl = ctl;
    p.table = rows_at(f[0].slot[MB_EM_S_TABLE]);
    p.hidden = rows_at(f[0].slot[MB_EM_S_OUT]);
    p.normed = rows_at(one[0].slot[MB_RN_S_OUT]);
    p.q = rows_at(one[1].slot[MB_GV_S_OUT0]);
    p.attn = rows_at(one[3].slot[MB_AP_S_OUT]);
    p.glu = rows_at(one[6].slot[MB_GV_S_OUT0]);
    p.inv_freq = reinterpret_cast<const void*>(addr(one[2].slot[MB_RP_S_INVFREQ]));
    const int H = p.hidden_size, I = p.intermediate, q_dim = p.heads * p.head_dim;
    const unsigned long long inputs[5] = {addr(one[0].slot[MB_RN_S_OUT]), addr(one[3].slot[MB_AP_S_OUT]),
                                          addr(one[0].slot[MB_RN_S_OUT]), addr(one[6].slot[MB_GV_S_OUT0]),
                                          addr(one[0].slot[MB_RN_S_OUT])};
    const int lengths[5] = {H, q_dim, H, I, H};
    for (int j = 0; j < 5; ++j)
        if (!make_block_map(&p.b[j], inputs[j], p.rows, lengths[j], p.gemm[j].tokens, p.gemm[j].deep))
            return MB_ERR_CUDA;
    for (int l = 0; l < p.layers; ++l) {
        const mb_phase* P = &f[1 + l * kPhasesPerLayer];
        LayerArgs& layer = p.layer[l];
        layer.norm[0] = rows_at(P[0].slot[MB_RN_S_W]);
        layer.norm[1] = rows_at(P[5].slot[MB_RN_S_W]);
        for (int s = 0; s < 3; ++s) layer.bias[s] = rows_at(P[1].slot[MB_GV_S_BIAS0 + s]);
        layer.bias[3] = rows_at(P[4].slot[MB_GV_S_BIAS0]);
        layer.bias[4] = rows_at(P[7].slot[MB_GV_S_BIAS0]);
        for (int s = 0; s < 2; ++s) layer.kv[s] = rows_at(P[1].slot[MB_GV_S_OUT0 + 1 + s]);
        layer.length = reinterpret_cast<int*>(addr(P[2].slot[MB_RP_S_LEN]));
        for (int w = 0; w < 3; ++w)
            if (!make_head_map(&layer.w[w], addr(P[1].slot[MB_GV_S_W0 + w]), w == 0 ? p.heads : p.kv_heads, p.head_dim,
                               H, p.gemm[kProjQkv].rows, p.gemm[kProjQkv].deep))
                return MB_ERR_CUDA;
        const struct {
            const mb_phase* record;
            int slot, n, proj;
        } weights[4] = {{&P[4], MB_GV_S_W0, H, kProjOut},
                        {&P[6], MB_GV_S_W0, I, kProjGated},
                        {&P[6], MB_GV_S_W_PAIR, I, kProjGated},
                        {&P[7], MB_GV_S_W0, H, kProjDown}};
        for (int w = 0; w < 4; ++w)
            if (!make_block_map(&layer.w[3 + w], addr(weights[w].record->slot[weights[w].slot]), weights[w].n,
                                lengths[weights[w].proj], p.gemm[weights[w].proj].rows,
                                p.gemm[weights[w].proj].deep))
                return MB_ERR_CUDA;
    }
    const mb_phase& head = f.back();
    p.final_norm = rows_at(f[f.size() - 2].slot[MB_RN_S_W]);
    p.head_bias = rows_at(head.slot[MB_GV_S_BIAS0]);
    if (!make_block_map(&p.head, addr(head.slot[MB_GV_S_W0]), head.i[MB_GV_I_N0], H, p.gemm[kProjHead].rows,
                        p.gemm[kProjHead].deep))
        return MB_ERR_CUDA;
    return MB_OK;
}

cudaError_t prompt_launch(const PromptState* st, const std::vector<unsigned long long>& slots,
                          const unsigned long long* dyn, unsigned long long* trace, cudaStream_t stream) {
    using namespace prompt;
    auto addr = [&](int s) -> unsigned long long {
        if (s < 0) return 0ull;
        return static_cast<unsigned int>(s) < st->n_dynamic ? dyn[s] : slots[s];
    };
    Params p = st->params;
    p.ids = reinterpret_cast<const long long*>(addr(st->phases[0].slot[MB_EM_S_IDS]));
    p.pos = reinterpret_cast<const long long*>(addr(st->phases[3].slot[MB_RP_S_POS]));
    p.logits = reinterpret_cast<unsigned short*>(addr(st->phases.back().slot[MB_GV_S_OUT0]));
    p.trace = trace;
    // All CTAs have to run at once.  What the projections are cut into does not depend on how many there are.
    const int grid = usable_sms(stream, st->grid);
    if (grid < st->grid) {
        p.gemm[kProjOut].first = p.attn_units % grid;
        if (p.rows > grid) p.small = 0;
    }
    void* args[] = {&p};
    return cudaLaunchCooperativeKernel(kernel_of(p), dim3(grid), dim3(kThreads), args, kSmemBytes, stream);
}

}  // namespace mb

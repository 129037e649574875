// The C ABI declared in include/megabake_b200.h: plan objects, validation, admission,
// binding and launch.  No torch types cross this boundary; device memory for tensors is the
// caller's, the plan only owns its own small tables (phase records, address table, control
// block).
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "mb_device.cuh"
#include "mb_kernels.h"

namespace {

thread_local std::string g_last_cuda_error;

int cuda_fail(cudaError_t err, const char* what) {
    g_last_cuda_error = std::string(what) + ": " + cudaGetErrorName(err) + " (" +
                        cudaGetErrorString(err) + ")";
    return MB_ERR_CUDA;
}

#define MB_CUDA(call)                                       \
    do {                                                    \
        cudaError_t err__ = (call);                         \
        if (err__ != cudaSuccess) return cuda_fail(err__, #call); \
    } while (0)

// Makes `device` current for the lifetime of the object and restores the previous one.
struct DeviceGuard {
    int previous = -1;
    bool switched = false;
    cudaError_t error = cudaSuccess;
    explicit DeviceGuard(int device) {
        error = cudaGetDevice(&previous);
        if (error == cudaSuccess && previous != device) {
            error = cudaSetDevice(device);
            switched = error == cudaSuccess;
        }
    }
    ~DeviceGuard() {
        if (switched) cudaSetDevice(previous);
    }
};


// Which operands of a decode phase live in the plan's relay arena, and where.
struct Relay {
    unsigned long long modes = 0;
    unsigned long long offset[MB_PHASE_SLOTS] = {};
    bool used[MB_PHASE_SLOTS] = {};
};

}  // namespace

struct mb_plan {
    int device = 0;
    int mode = MB_MODE_DECODE;
    std::vector<mb_phase> phases;
    std::vector<unsigned long long> slots;
    unsigned int n_dynamic = 0;
    unsigned int activation_bytes = 0;
    bool bound = false;
    int sm_count = 0;
    int ctas = 0;
    int threads = 0;
    int smem_bytes = 0;
    int stages = 0;
    int slots_per_slice = 0;  // decode: of a warp's slice of the activations
    int head_dim = 64;  // decode: of all attention phases, 0 if they differ
    int barriers = 0;
    bool counters = false;
    unsigned int wait_limit_us = 2000000u;
    std::vector<Relay> relays;            // per phase (decode)
    unsigned long long relay_bytes = 0;   // one half of the arena
    void* d_relay = nullptr;              // both halves
    mb::PhaseEntry* d_entries = nullptr;
    mb::StreamDesc* d_streams = nullptr;
    void* d_maps = nullptr;               // tensor maps of weights and caches, decode_map_bytes() per phase
    unsigned int maps_written = 0;        // Control::maps_written
    std::vector<size_t> late_maps;        // phases with such an operand that comes with the launch
    std::vector<mb::PhaseEntry> entries;  // as bound
    std::vector<unsigned long long> partials;  // per phase: split-key buffer that was cleared for it, or 0
    unsigned int wide_dynamic = 0;        // per-launch slots that must be 16-byte aligned, one bit each
    mb::Control* d_ctl = nullptr;
    unsigned long long trace = 0;
    mb::PrefillState* prefill = nullptr;  // MB_MODE_PREFILL plans only, one of the two:
    mb::PromptState* prompt = nullptr;    // a short prompt in one launch
};

namespace {

// What activation_bytes is checked against for an attention phase.  (The kernel's own scratch does not
// depend on it; the check stays as callers know it.)
long long attention_scratch_bytes(int head_dim, int group, int merge_slots) {
    const long long qs = 8LL * (head_dim + 32) * 2;
    const long long new_rows = 2LL * head_dim * 2;
    const long long cs = 4LL * head_dim;
    const long long stats = 4LL * (2 * 8 * 8 + 8 * 64 + 16);
    const long long states = 4LL * (head_dim + 2) * group * (merge_slots + 2);
    // per-warp K/V tile slots of the split-key loop (64-wide heads): 8 warps x 2 slots x 16 keys
    const long long staging = head_dim == 64 ? 8LL * 2 * 16 * ((head_dim * 2 + 64) + (head_dim * 2 + 16)) : 0;
    return qs + new_rows + cs + stats + states + staging;
}

int check_slot(const mb_plan_desc* d, int s, bool required) {
    if (s < 0) return required ? MB_ERR_INVALID : MB_OK;
    return static_cast<unsigned int>(s) < d->n_slots ? MB_OK : MB_ERR_INVALID;
}

int plan_stage_bytes(const mb_plan_desc* d) {
    return d->stage_bytes == 0 ? mb::decode_stage_bytes() : static_cast<int>(d->stage_bytes);
}

int validate_gemv(const mb_plan_desc* d, const mb_phase& P) {
    const int rows = P.i[MB_GV_I_ROWS], K = P.i[MB_GV_I_K], nseg = P.i[MB_GV_I_NSEG];
    const int nmat = P.i[MB_GV_I_NMAT], rt = P.i[MB_GV_I_ROW_TILE], kc = P.i[MB_GV_I_K_CHUNK];
    const int epi = P.i[MB_GV_I_EPILOGUE], pro = P.i[MB_GV_I_PROLOGUE];
    if (rows < 1 || rows > 8) return MB_ERR_UNSUPPORTED;
    if (K < 32 || K % 32 != 0) return MB_ERR_UNSUPPORTED;
    if (nseg < 1 || nseg > 3) return MB_ERR_INVALID;
    if (nmat != 1 && nmat != 2) return MB_ERR_INVALID;
    if (nmat == 2 && nseg != 1) return MB_ERR_INVALID;
    // a stage holds one 8-row tile, or two: the gate and up tiles of a paired phase, or 16
    // consecutive rows of a plain one
    if (rt != mb::decode_row_tile() && !(nmat == 1 && rt == 2 * mb::decode_row_tile()))
        return MB_ERR_INVALID;
    if (kc < 32 || kc % 32 != 0 || kc > K) return MB_ERR_INVALID;
    if (static_cast<long long>(rt) * nmat * (kc * 2 + mb::decode_row_pad()) > plan_stage_bytes(d))
        return MB_ERR_RESOURCE;
    const int cells = P.i[MB_GV_I_CELLS];
    if (cells & ~(MB_CELLS_X | MB_CELLS_OUT | MB_CELLS_RESIDUAL | MB_CELLS_XSTORE | MB_CELLS_X_WAIT))
        return MB_ERR_INVALID;
    if ((cells & MB_CELLS_X_WAIT) &&
        (P.i[MB_GV_I_X_SOURCE] < 0 || static_cast<unsigned int>(P.i[MB_GV_I_X_SOURCE]) >= d->n_phases))
        return MB_ERR_INVALID;
    if ((cells & MB_CELLS_X) && (P.i[MB_GV_I_GATHER] || K % 4 != 0)) return MB_ERR_INVALID;
    if ((cells & MB_CELLS_X) &&
        (P.i[MB_GV_I_X_SOURCE] < 0 || static_cast<unsigned int>(P.i[MB_GV_I_X_SOURCE]) >= d->n_phases))
        return MB_ERR_INVALID;
    if ((cells & MB_CELLS_RESIDUAL) &&
        (P.i[MB_GV_I_RES_SOURCE] < 0 ||
         static_cast<unsigned int>(P.i[MB_GV_I_RES_SOURCE]) >= d->n_phases))
        return MB_ERR_INVALID;
    // activation rows, plus one staged row of norm weights when the phase normalises
    const long long staged_rows = rows + (P.i[MB_GV_I_PROLOGUE] != MB_PRO_NONE ? 1 : 0);
    if (staged_rows * (K + 32) * 2 > d->activation_bytes) return MB_ERR_RESOURCE;
    if (pro < MB_PRO_NONE || pro > MB_PRO_RMS_GEMMA) return MB_ERR_INVALID;
    if (epi < MB_EPI_NONE || epi > MB_EPI_GELU_TANH_MUL) return MB_ERR_INVALID;
    const bool paired_epi = epi == MB_EPI_SILU_MUL || epi == MB_EPI_GELU_TANH_MUL;
    if (paired_epi != (nmat == 2)) return MB_ERR_INVALID;
    for (int s = 0; s < nseg; ++s) {
        if (P.i[MB_GV_I_N0 + s] < 2) return MB_ERR_INVALID;
        // results are stored as pairs of neighbouring rows (one 4-byte store or one cell)
        if (P.i[MB_GV_I_N0 + s] % 2 != 0) return MB_ERR_UNSUPPORTED;
        if (check_slot(d, P.slot[MB_GV_S_W0 + s], true)) return MB_ERR_INVALID;
        if (check_slot(d, P.slot[MB_GV_S_OUT0 + s], true)) return MB_ERR_INVALID;
        if (check_slot(d, P.slot[MB_GV_S_BIAS0 + s], false)) return MB_ERR_INVALID;
    }
    if (check_slot(d, P.slot[MB_GV_S_X], true)) return MB_ERR_INVALID;
    if (pro != MB_PRO_NONE && check_slot(d, P.slot[MB_GV_S_NORM_W], true)) return MB_ERR_INVALID;
    if (nmat == 2 && check_slot(d, P.slot[MB_GV_S_W_PAIR], true)) return MB_ERR_INVALID;
    if (epi == MB_EPI_RESIDUAL && check_slot(d, P.slot[MB_GV_S_RESIDUAL], true))
        return MB_ERR_INVALID;
    if (P.i[MB_GV_I_GATHER]) {
        if (check_slot(d, P.slot[MB_GV_S_IDS], true)) return MB_ERR_INVALID;
        if (P.i[MB_GV_I_VOCAB] < 1) return MB_ERR_INVALID;
        if (P.i[MB_GV_I_STORE_X] && check_slot(d, P.slot[MB_GV_S_XSTORE], true))
            return MB_ERR_INVALID;
    }
    return MB_OK;
}

int validate_attention(const mb_plan_desc* d, const mb_phase& P) {
    const int B = P.i[MB_AT_I_BATCH], Hq = P.i[MB_AT_I_HEADS], Hkv = P.i[MB_AT_I_KV_HEADS];
    const int D = P.i[MB_AT_I_HEAD_DIM], cap = P.i[MB_AT_I_CAPACITY];
    const int chunks = P.i[MB_AT_I_MAX_CHUNKS], slots = P.i[MB_AT_I_MERGE_SLOTS];
    if (B < 1 || Hq < 1 || Hkv < 1 || cap < 1) return MB_ERR_INVALID;
    if (Hq % Hkv != 0 || Hq / Hkv > 8) return MB_ERR_UNSUPPORTED;
    if (D != 64 && D != 128 && D != 256) return MB_ERR_UNSUPPORTED;
    if (chunks < 1 || chunks > 64) return MB_ERR_INVALID;
    if (slots < 1 || slots > 8) return MB_ERR_INVALID;
    const int exact = P.i[MB_AT_I_EXACT_KEYS];
    if (exact < 0 || exact > 128) return MB_ERR_INVALID;
    if (attention_scratch_bytes(D, Hq / Hkv, slots) > d->activation_bytes)
        return MB_ERR_RESOURCE;
    for (int s = MB_AT_S_Q; s <= MB_AT_S_COUNTER; ++s)
        if (check_slot(d, P.slot[s], true)) return MB_ERR_INVALID;
    const int cells = P.i[MB_AT_I_CELLS];
    if (cells & ~(MB_CELLS_X | MB_CELLS_OUT | MB_CELLS_X_WAIT)) return MB_ERR_INVALID;
    if ((cells & (MB_CELLS_X | MB_CELLS_X_WAIT)) &&
        (P.i[MB_AT_I_QKV_SOURCE] < 0 ||
         static_cast<unsigned int>(P.i[MB_AT_I_QKV_SOURCE]) >= d->n_phases))
        return MB_ERR_INVALID;
    const int lengths = P.i[MB_AT_I_LEN_COUNT];
    if (lengths != 0 && lengths != 1 && lengths != B) return MB_ERR_INVALID;
    return MB_OK;
}

// Gives every tensor that a phase with MB_FLAG_RELAY produces a place of its own in the relay arena
// and points the phases that read it there.  No place is used twice in a launch, so nothing ever
// has to wait before it overwrites.  Sets `counters` if some hand-off still needs the
// finished-phase counters: plain results behind MB_CELLS_X_WAIT, or cells, whose buffers are
// written again.
int lower_relays(mb_plan* plan) {
    plan->relays.assign(plan->phases.size(), Relay());
    plan->relay_bytes = 0;
    std::vector<long long> place(plan->slots.size(), -1);  // slot -> arena offset of its live contents
    auto produce = [&](Relay& r, const mb_phase& P, int s, unsigned long long bytes) {
        const int slot = P.slot[s];
        if (slot < 0) return MB_OK;
        if (!(P.flags & MB_FLAG_RELAY)) {
            place[slot] = -1;
            return MB_OK;
        }
        if (static_cast<unsigned int>(slot) < plan->n_dynamic) return MB_ERR_INVALID;
        place[slot] = static_cast<long long>(plan->relay_bytes);
        r.offset[s] = plan->relay_bytes;
        r.used[s] = true;
        plan->relay_bytes += (bytes + 255) / 256 * 256;
        return MB_OK;
    };
    auto consume = [&](Relay& r, const mb_phase& P, int s) {
        const int slot = P.slot[s];
        if (slot < 0 || place[slot] < 0) return false;
        r.offset[s] = static_cast<unsigned long long>(place[slot]);
        r.used[s] = true;
        return true;
    };
    for (size_t i = 0; i < plan->phases.size(); ++i) {
        const mb_phase& P = plan->phases[i];
        Relay& r = plan->relays[i];
        if (P.body == MB_BODY_GEMV) {
            const int cells = P.i[MB_GV_I_CELLS];
            if (!P.i[MB_GV_I_GATHER]) {
                if (consume(r, P, MB_GV_S_X))
                    r.modes |= mb::kModeInRelay;
                else if (cells & (MB_CELLS_X | MB_CELLS_X_WAIT))
                    plan->counters = true;
                if ((cells & MB_CELLS_X_WAIT) && !(cells & MB_CELLS_X) && !(r.modes & mb::kModeInRelay))
                    r.modes |= mb::kModeWait;
            }
            if (P.i[MB_GV_I_EPILOGUE] == MB_EPI_RESIDUAL) {
                if (consume(r, P, MB_GV_S_RESIDUAL))
                    r.modes |= mb::kModeResidualRelay;
                else if (cells & (MB_CELLS_RESIDUAL | MB_CELLS_X_WAIT))
                    plan->counters = true;
                if ((cells & MB_CELLS_X_WAIT) && !(cells & MB_CELLS_RESIDUAL) &&
                    !(r.modes & mb::kModeResidualRelay))
                    r.modes |= mb::kModeWait;  // whatever the activations are
            }
            if (P.i[MB_GV_I_GATHER] && P.i[MB_GV_I_STORE_X]) {
                if (P.flags & MB_FLAG_RELAY) r.modes |= mb::kModeStoreRelay;
                const int rc = produce(r, P, MB_GV_S_XSTORE, 2ull * P.i[MB_GV_I_ROWS] * P.i[MB_GV_I_K]);
                if (rc != MB_OK) return rc;
            }
            if (P.flags & MB_FLAG_RELAY) r.modes |= mb::kModeOutRelay;
            for (int s = 0; s < P.i[MB_GV_I_NSEG]; ++s) {
                const int rc = produce(r, P, MB_GV_S_OUT0 + s, 2ull * P.i[MB_GV_I_ROWS] * P.i[MB_GV_I_N0 + s]);
                if (rc != MB_OK) return rc;
            }
        } else if (P.body == MB_BODY_ATTN_DECODE) {
            const bool q = consume(r, P, MB_AT_S_Q), k = consume(r, P, MB_AT_S_K), v = consume(r, P, MB_AT_S_V);
            if (q != k || q != v) return MB_ERR_INVALID;
            if (q)
                r.modes |= mb::kModeInRelay;
            else if (P.i[MB_AT_I_CELLS] & (MB_CELLS_X | MB_CELLS_X_WAIT))
                plan->counters = true;
            if (P.flags & MB_FLAG_RELAY) r.modes |= mb::kModeOutRelay;
            const int rc = produce(r, P, MB_AT_S_OUT,
                                   2ull * P.i[MB_AT_I_BATCH] * P.i[MB_AT_I_HEADS] * P.i[MB_AT_I_HEAD_DIM]);
            if (rc != MB_OK) return rc;
        }
    }
    return MB_OK;
}

// Phases that read weights or caches from addresses known at launch only.
bool has_late_map(const mb::PhaseEntry& entry) {
    const bool gemv = entry.rec.body == MB_BODY_GEMV;
    static const int weights[] = {MB_GV_S_W0, MB_GV_S_W0 + 1, MB_GV_S_W0 + 2, MB_GV_S_W_PAIR};
    static const int caches[] = {MB_AT_S_KCACHE, MB_AT_S_VCACHE};
    if (!gemv && entry.rec.body != MB_BODY_ATTN_DECODE) return false;
    for (int k = 0; k < (gemv ? 4 : 2); ++k)
        if (entry.addr[gemv ? weights[k] : caches[k]] & mb::kDynamicTag) return true;
    return false;
}

// Blank arena: every word says "not written in this launch".
cudaError_t blank_relays(const mb_plan* plan) {
    if (plan->d_relay == nullptr) return cudaSuccess;
    return cudaMemset(plan->d_relay, 0xff, 2 * plan->relay_bytes);
}

// Bytes of split-key partials an attention phase may poll; 0 if its context is never cut.
size_t partial_bytes(const mb_phase& P) {
    if (P.body != MB_BODY_ATTN_DECODE || P.i[MB_AT_I_MAX_CHUNKS] < 4) return 0;
    if (P.i[MB_AT_I_CAPACITY] <= P.i[MB_AT_I_EXACT_KEYS]) return 0;
    return static_cast<size_t>(P.i[MB_AT_I_BATCH]) * P.i[MB_AT_I_HEADS] * (P.i[MB_AT_I_MAX_CHUNKS] / 2) *
           (P.i[MB_AT_I_HEAD_DIM] + 2) * 8;
}

// The partials are (value, tag) cells, and the tags of every plan start over: what an earlier owner of the
// memory left there may carry the very tags this plan is going to wait for.  So each buffer is
// cleared when its address is new to the phase, before any launch can poll it.
cudaError_t clear_partials(mb_plan* plan, const std::vector<mb::PhaseEntry>& entries) {
    plan->partials.resize(entries.size(), 0ull);
    bool cleared = false;
    for (size_t ph = 0; ph < entries.size(); ++ph) {
        const size_t bytes = partial_bytes(plan->phases[ph]);
        const unsigned long long address = entries[ph].addr[MB_AT_S_PARTIAL];
        if (bytes == 0 || (address & mb::kDynamicTag) || address == plan->partials[ph]) continue;
        const cudaError_t err = cudaMemset(reinterpret_cast<void*>(address), 0, bytes);
        if (err != cudaSuccess) return err;
        for (size_t other = ph; other < entries.size(); ++other)  // the layers of a model share one buffer
            if (entries[other].addr[MB_AT_S_PARTIAL] == address && partial_bytes(plan->phases[other]) <= bytes)
                plan->partials[other] = address;
        cleared = true;
    }
    return cleared ? cudaStreamSynchronize(cudaStreamLegacy) : cudaSuccess;  // launches may use any stream
}

unsigned int wait_limit_us(const mb_plan_desc* desc) {
    if (desc->wait_limit_ms == 0) return 2000000u;
    return desc->wait_limit_ms > 4000000u ? 4000000000u : desc->wait_limit_ms * 1000u;
}

// A prefill plan is a list of kernel launches; it shares the descriptor, the slot table, the
// status word and the entry points with decode plans.
int create_prefill_plan(const mb_plan_desc* desc, mb_plan** out) {
    for (unsigned int i = 0; i < desc->n_phases; ++i) {
        const int rc = mb::prefill_validate(desc->phases[i], desc->n_slots, desc->n_dynamic);
        if (rc != MB_OK) return rc;
    }
    DeviceGuard guard(desc->device);
    if (guard.error != cudaSuccess) return cuda_fail(guard.error, "cudaSetDevice");
    cudaDeviceProp prop;
    MB_CUDA(cudaGetDeviceProperties(&prop, desc->device));
    if (prop.major != 10) {
        g_last_cuda_error = "device is not sm_100 (compute capability " +
                            std::to_string(prop.major) + "." + std::to_string(prop.minor) + ")";
        return MB_ERR_UNSUPPORTED;
    }
    mb_plan* plan = new (std::nothrow) mb_plan();
    if (plan == nullptr) return MB_ERR_RESOURCE;
    plan->device = desc->device;
    plan->mode = desc->mode;
    plan->phases.assign(desc->phases, desc->phases + desc->n_phases);
    plan->slots.assign(desc->n_slots, 0ull);
    plan->n_dynamic = desc->n_dynamic;
    plan->sm_count = prop.multiProcessorCount;
    plan->ctas = prop.multiProcessorCount;
    cudaError_t err = cudaMalloc(&plan->d_ctl, sizeof(mb::Control));
    if (err == cudaSuccess) err = cudaMemset(plan->d_ctl, 0, sizeof(mb::Control));
    if (err == cudaSuccess)
        err = mb::prompt_create(plan->phases, plan->n_dynamic, plan->sm_count, wait_limit_us(desc), &plan->prompt);
    if (err == cudaSuccess && plan->prompt == nullptr)
        err = mb::prefill_create(plan->phases, plan->sm_count, &plan->prefill);
    if (err != cudaSuccess) {
        cuda_fail(err, "prefill plan allocation");
        mb_plan_destroy(plan);
        return MB_ERR_CUDA;
    }
    *out = plan;
    return MB_OK;
}

}  // namespace

extern "C" {

int mb_abi_version(void) { return MB_ABI_VERSION; }

const char* mb_last_cuda_error(void) { return g_last_cuda_error.c_str(); }

const char* mb_strerror(int code) {
    switch (code) {
        case MB_OK: return "ok";
        case MB_ERR_INVALID: return "invalid argument or malformed plan descriptor";
        case MB_ERR_CUDA: return "a CUDA runtime call failed";
        case MB_ERR_UNSUPPORTED: return "body or shape not implemented by the kernels";
        case MB_ERR_RESOURCE: return "shared memory or co-residency admission failed";
        case MB_ERR_UNBOUND: return "plan launched before its static slots were bound";
        case MB_ERR_VERSION: return "plan descriptor ABI version mismatch";
        default: return "unknown error code";
    }
}

const char* mb_status_string(int status_code) {
    switch (status_code) {
        case MB_ST_OK: return "ok";
        case MB_ST_BARRIER_TIMEOUT: return "grid barrier wait timed out";
        case MB_ST_PIPE_TIMEOUT: return "shared-memory pipeline wait timed out";
        case MB_ST_KV_OVERFLOW: return "KV cache is full";
        case MB_ST_TOKEN_RANGE: return "token id outside the embedding table";
        case MB_ST_BAD_PHASE: return "unknown body in the phase table";
        case MB_ST_TMEM: return "tensor memory allocation failed";
        case MB_ST_HANDOFF_TIMEOUT: return "an activation hand-off wait timed out";
        default: return "unknown status";
    }
}

int mb_max_smem_bytes(void) { return 232448; }  // 227 KiB opt-in limit of sm_100

int mb_fixed_smem_bytes(int mode) {
    if (mode == MB_MODE_DECODE) return mb::decode_fixed_smem();
    return -1;
}

int mb_stage_bytes(int mode) {
    if (mode == MB_MODE_DECODE) return mb::decode_stage_bytes();
    return -1;
}

int mb_plan_create(const mb_plan_desc* desc, mb_plan** out) {
    if (desc == nullptr || out == nullptr) return MB_ERR_INVALID;
    *out = nullptr;
    if (desc->abi_version != MB_ABI_VERSION) return MB_ERR_VERSION;
    if (desc->n_phases == 0 || desc->phases == nullptr) return MB_ERR_INVALID;
    if (desc->n_dynamic > MB_MAX_DYNAMIC || desc->n_dynamic > desc->n_slots) return MB_ERR_INVALID;
    if (desc->mode == MB_MODE_PREFILL) return create_prefill_plan(desc, out);
    if (desc->mode != MB_MODE_DECODE) return MB_ERR_UNSUPPORTED;
    if (desc->activation_bytes % 128 != 0) return MB_ERR_INVALID;
    if (desc->stage_bytes % 1024 != 0 ||
        desc->stage_bytes > static_cast<unsigned int>(mb::decode_stage_bytes()))
        return MB_ERR_INVALID;

    int barriers = 1;  // one more than the records ask for: the end of the launch
    for (unsigned int i = 0; i < desc->n_phases; ++i) {
        const mb_phase& P = desc->phases[i];
        int rc = MB_OK;
        switch (P.body) {
            case MB_BODY_NOP: break;
            case MB_BODY_GEMV: rc = validate_gemv(desc, P); break;
            case MB_BODY_ATTN_DECODE: rc = validate_attention(desc, P); break;
            default: rc = MB_ERR_UNSUPPORTED; break;
        }
        if (rc != MB_OK) return rc;
        if (P.flags & MB_FLAG_BARRIER) ++barriers;
    }

    DeviceGuard guard(desc->device);
    if (guard.error != cudaSuccess) return cuda_fail(guard.error, "cudaSetDevice");
    cudaDeviceProp prop;
    MB_CUDA(cudaGetDeviceProperties(&prop, desc->device));
    if (prop.major != 10) {
        g_last_cuda_error = "device is not sm_100 (compute capability " +
                            std::to_string(prop.major) + "." + std::to_string(prop.minor) + ")";
        return MB_ERR_UNSUPPORTED;
    }
    if (!prop.cooperativeLaunch) return MB_ERR_UNSUPPORTED;

    const int limit = static_cast<int>(prop.sharedMemPerBlockOptin);
    const int head_dim = mb::decode_head_dim(desc->phases, desc->n_phases);
    const int rope_bytes = mb::decode_rope_bytes(desc->phases, desc->n_phases);
    const int slots = mb::decode_slice_slots(desc->phases, desc->n_phases,
                                             desc->ctas == 0 ? prop.multiProcessorCount : static_cast<int>(desc->ctas));
    const int stages = mb::decode_ring_stages(rope_bytes, desc->n_phases, slots, limit);
    if (stages < 2) return MB_ERR_RESOURCE;
    const int smem = mb::decode_smem_bytes(rope_bytes, desc->n_phases, slots, stages);

    // The attribute belongs to the kernel, not to a plan: set it to the device's opt-in limit so
    // that plans of different sizes (two batch sizes, two models) can be launched in any order.
    MB_CUDA(mb::decode_configure(head_dim, limit));
    int per_sm = 0;
    MB_CUDA(mb::decode_occupancy(head_dim, smem, &per_sm));
    if (per_sm < 1) return MB_ERR_RESOURCE;
    int ctas = desc->ctas == 0 ? prop.multiProcessorCount : static_cast<int>(desc->ctas);
    if (ctas < 1 || ctas > prop.multiProcessorCount * per_sm) return MB_ERR_RESOURCE;

    mb_plan* plan = new (std::nothrow) mb_plan();
    if (plan == nullptr) return MB_ERR_RESOURCE;
    plan->device = desc->device;
    plan->mode = desc->mode;
    plan->phases.assign(desc->phases, desc->phases + desc->n_phases);
    for (mb_phase& P : plan->phases) {
        if (P.body != MB_BODY_GEMV) continue;
        // balanced split of the output rows over the CTAs, so the kernel needs no division
        // (in pairs of rows: a lane's two neighbouring results are stored together)
        int total = 0;
        for (int s = 0; s < P.i[MB_GV_I_NSEG]; ++s) total += P.i[MB_GV_I_N0 + s];
        P.i[MB_GV_I_SPLIT_Q] = (total / 2) / ctas;
        P.i[MB_GV_I_SPLIT_R] = (total / 2) % ctas;
    }
    plan->slots.assign(desc->n_slots, 0ull);
    plan->n_dynamic = desc->n_dynamic;
    for (const mb_phase& P : plan->phases)
        if (P.body == MB_BODY_ATTN_DECODE && static_cast<unsigned int>(P.slot[MB_AT_S_PARTIAL]) < desc->n_dynamic)
            plan->wide_dynamic |= 1u << P.slot[MB_AT_S_PARTIAL];
    plan->activation_bytes = desc->activation_bytes;
    plan->sm_count = prop.multiProcessorCount;
    plan->ctas = ctas;
    plan->threads = mb::decode_threads();
    plan->smem_bytes = smem;
    plan->stages = stages;
    plan->slots_per_slice = slots;
    plan->head_dim = head_dim;
    plan->barriers = barriers;
    plan->wait_limit_us = wait_limit_us(desc);

    const int lowered = lower_relays(plan);
    if (lowered != MB_OK) {
        mb_plan_destroy(plan);
        return lowered;
    }

    cudaError_t err = cudaMalloc(&plan->d_entries, sizeof(mb::PhaseEntry) * desc->n_phases);
    if (err == cudaSuccess) err = cudaMalloc(&plan->d_streams, sizeof(mb::StreamDesc) * desc->n_phases);
    if (err == cudaSuccess) err = cudaMalloc(&plan->d_maps, mb::decode_map_bytes() * desc->n_phases);
    if (err == cudaSuccess && plan->relay_bytes > 0) err = cudaMalloc(&plan->d_relay, 2 * plan->relay_bytes);
    if (err == cudaSuccess) err = blank_relays(plan);
    if (err == cudaSuccess) err = cudaMalloc(&plan->d_ctl, sizeof(mb::Control));
    if (err == cudaSuccess) err = cudaMemset(plan->d_ctl, 0, sizeof(mb::Control));
    if (err == cudaSuccess) err = cudaStreamSynchronize(cudaStreamLegacy);  // launches may use any stream
    if (err != cudaSuccess) {
        cuda_fail(err, "plan table allocation");
        mb_plan_destroy(plan);
        return MB_ERR_CUDA;
    }
    *out = plan;
    return MB_OK;
}

int mb_plan_query(const mb_plan* plan, mb_plan_info* out) {
    if (plan == nullptr || out == nullptr) return MB_ERR_INVALID;
    std::memset(out, 0, sizeof(*out));
    out->ctas = plan->ctas;
    out->threads = plan->threads;
    out->smem_bytes = plan->smem_bytes;
    out->stages = plan->stages;
    out->barriers = plan->mode == MB_MODE_PREFILL ? 0 : plan->barriers - 1;
    out->sm_count = plan->sm_count;
    out->launches = plan->prompt != nullptr           ? 1
                    : plan->mode == MB_MODE_PREFILL ? mb::prefill_launch_count(plan->prefill)
                                                    : 1 + static_cast<int>(plan->late_maps.size());
    return MB_OK;
}

int mb_plan_bind(mb_plan* plan, const uint64_t* slot_addresses, size_t n) {
    if (plan == nullptr || slot_addresses == nullptr) return MB_ERR_INVALID;
    if (n != plan->slots.size()) return MB_ERR_INVALID;
    for (size_t i = plan->n_dynamic; i < n; ++i) {
        if (slot_addresses[i] == 0 || (slot_addresses[i] & 15ull) != 0) return MB_ERR_INVALID;
        plan->slots[i] = slot_addresses[i];
    }
    if (plan->mode == MB_MODE_PREFILL) {
        DeviceGuard guard(plan->device);
        if (guard.error != cudaSuccess) return cuda_fail(guard.error, "cudaSetDevice");
        const int rc = plan->prompt != nullptr
                           ? mb::prompt_bind(plan->prompt, plan->slots, plan->d_ctl)
                           : mb::prefill_bind(plan->prefill, plan->phases, plan->slots, plan->d_ctl);
        if (rc != MB_OK) {
            g_last_cuda_error = "tensor map encoding failed";
            return rc;
        }
        plan->bound = true;
        return MB_OK;
    }
    // Resolve every slot a phase names into its entry, so the kernel reads one record per
    // phase and never a second table.
    std::vector<mb::PhaseEntry> entries(plan->phases.size());
    std::vector<mb::StreamDesc> streams(plan->phases.size());
    std::vector<unsigned char> maps(plan->phases.size() * mb::decode_map_bytes(), 0);
    plan->late_maps.clear();
    for (size_t ph = 0; ph < plan->phases.size(); ++ph) {
        entries[ph].rec = plan->phases[ph];
        entries[ph].modes = plan->relays[ph].modes;
        for (int j = 0; j < MB_PHASE_SLOTS; ++j) {
            const int slot = plan->phases[ph].slot[j];
            if (slot < 0)
                entries[ph].addr[j] = 0ull;
            else if (plan->relays[ph].used[j])
                entries[ph].addr[j] = mb::kRelayTag | plan->relays[ph].offset[j];
            else if (static_cast<unsigned int>(slot) < plan->n_dynamic)
                entries[ph].addr[j] = mb::kDynamicTag | static_cast<unsigned long long>(slot);
            else
                entries[ph].addr[j] = plan->slots[slot];
        }
        mb::decode_stream(plan->phases[ph], entries[ph].addr, plan->ctas, plan->slots_per_slice, &streams[ph]);
        if (has_late_map(entries[ph])) {
            plan->late_maps.push_back(ph);
        } else if (!mb::decode_encode_maps(plan->phases[ph], entries[ph].addr, plan->ctas,
                                           maps.data() + ph * mb::decode_map_bytes())) {
            g_last_cuda_error = "tensor map encoding failed";
            return MB_ERR_CUDA;
        }
    }
    DeviceGuard guard(plan->device);
    if (guard.error != cudaSuccess) return cuda_fail(guard.error, "cudaSetDevice");
    MB_CUDA(clear_partials(plan, entries));
    MB_CUDA(cudaMemcpy(plan->d_entries, entries.data(), sizeof(mb::PhaseEntry) * entries.size(),
                       cudaMemcpyHostToDevice));
    MB_CUDA(cudaMemcpy(plan->d_maps, maps.data(), maps.size(), cudaMemcpyHostToDevice));
    ++plan->maps_written;
    MB_CUDA(cudaMemcpy(&plan->d_ctl->maps_written, &plan->maps_written, sizeof(plan->maps_written),
                       cudaMemcpyHostToDevice));
    MB_CUDA(cudaMemcpy(plan->d_streams, streams.data(), sizeof(mb::StreamDesc) * streams.size(),
                       cudaMemcpyHostToDevice));
    plan->entries = std::move(entries);
    plan->bound = true;
    return MB_OK;
}

int mb_plan_launch(mb_plan* plan, const uint64_t* dynamic_addresses, size_t n, void* stream) {
    if (plan == nullptr) return MB_ERR_INVALID;
    if (!plan->bound) return MB_ERR_UNBOUND;
    if (n != plan->n_dynamic || (n > 0 && dynamic_addresses == nullptr)) return MB_ERR_INVALID;
    if (plan->mode == MB_MODE_PREFILL) {
        for (size_t i = 0; i < n; ++i)
            if (dynamic_addresses[i] == 0 || (dynamic_addresses[i] & 7ull) != 0) return MB_ERR_INVALID;
        DeviceGuard guard(plan->device);
        if (guard.error != cudaSuccess) return cuda_fail(guard.error, "cudaSetDevice");
        if (plan->prompt != nullptr) {
            MB_CUDA(mb::prompt_launch(plan->prompt, plan->slots,
                                      reinterpret_cast<const unsigned long long*>(dynamic_addresses),
                                      reinterpret_cast<unsigned long long*>(plan->trace),
                                      static_cast<cudaStream_t>(stream)));
            return MB_OK;
        }
        MB_CUDA(mb::prefill_launch(plan->prefill, plan->phases, plan->slots, plan->n_dynamic,
                                   reinterpret_cast<const unsigned long long*>(dynamic_addresses),
                                   plan->d_ctl, reinterpret_cast<unsigned long long*>(plan->trace),
                                   static_cast<cudaStream_t>(stream)));
        return MB_OK;
    }
    mb::KernelParams params;
    std::memset(&params, 0, sizeof(params));
    params.entries = plan->d_entries;
    params.streams = plan->d_streams;
    params.maps = plan->d_maps;
    params.stages = plan->stages;
    params.slots = plan->slots_per_slice;
    params.relay = reinterpret_cast<unsigned long long>(plan->d_relay);
    params.relay_bytes = plan->relay_bytes;
    params.ctl = plan->d_ctl;
    params.trace = reinterpret_cast<unsigned long long*>(plan->trace);
    for (size_t i = 0; i < n; ++i) {
        const unsigned long long unaligned = (plan->wide_dynamic >> i & 1u) ? 15ull : 7ull;
        if (dynamic_addresses[i] == 0 || (dynamic_addresses[i] & unaligned) != 0) return MB_ERR_INVALID;
        params.dyn[i] = dynamic_addresses[i];
    }
    params.n_phases = static_cast<int>(plan->phases.size());
    params.n_dynamic = static_cast<int>(plan->n_dynamic);
    params.barriers_per_launch = plan->barriers - 1;
    params.sm_count = plan->sm_count;
    params.counters = plan->counters ? 1 : 0;
    params.wait_limit_us = plan->wait_limit_us;
    DeviceGuard guard(plan->device);
    if (guard.error != cudaSuccess) return cuda_fail(guard.error, "cudaSetDevice");
    // Weights and caches that come with the launch: their maps travel as parameters of a kernel before it, so
    // that a captured launch keeps its own and the host may go on to the next one at once.
    for (size_t ph : plan->late_maps) {
        mb::PhaseEntry entry = plan->entries[ph];
        for (unsigned long long& a : entry.addr)
            if (a & mb::kDynamicTag) a = dynamic_addresses[a & (MB_MAX_DYNAMIC - 1)];
        MB_CUDA(mb::decode_store_maps(plan->phases[ph], entry.addr, plan->ctas,
                                      static_cast<unsigned char*>(plan->d_maps) + ph * mb::decode_map_bytes(),
                                      plan->d_ctl, static_cast<cudaStream_t>(stream)));
    }
    MB_CUDA(mb::decode_launch(params, plan->head_dim, plan->ctas, plan->smem_bytes,
                              static_cast<cudaStream_t>(stream)));
    return MB_OK;
}

int mb_plan_status(mb_plan* plan, mb_status* out) {
    if (plan == nullptr || out == nullptr) return MB_ERR_INVALID;
    DeviceGuard guard(plan->device);
    if (guard.error != cudaSuccess) return cuda_fail(guard.error, "cudaSetDevice");
    mb::Control host;
    MB_CUDA(cudaMemcpy(&host, plan->d_ctl, sizeof(host), cudaMemcpyDeviceToHost));
    out->code = host.status[0];
    out->phase = host.status[1];
    out->detail = host.status[2];
    out->calls = static_cast<int32_t>(host.calls);
    return MB_OK;
}

int mb_plan_set_trace(mb_plan* plan, uint64_t device_address, size_t bytes) {
    if (plan == nullptr) return MB_ERR_INVALID;
    if (device_address != 0) {
        // decode: 8 stamps per CTA and phase; prefill: 8 stamps per phase (CTA 0 of each GEMM)
        const size_t per_phase = plan->mode == MB_MODE_PREFILL ? 1 : static_cast<size_t>(plan->ctas);
        const size_t need = per_phase * plan->phases.size() * 8 * sizeof(uint64_t);
        if (bytes < need || (device_address & 7ull) != 0) return MB_ERR_INVALID;
    }
    plan->trace = device_address;
    return MB_OK;
}

int mb_plan_reset(mb_plan* plan) {
    if (plan == nullptr) return MB_ERR_INVALID;
    DeviceGuard guard(plan->device);
    if (guard.error != cudaSuccess) return cuda_fail(guard.error, "cudaSetDevice");
    MB_CUDA(cudaDeviceSynchronize());
    // Everything starts over except the epoch, which moves on: hand-off cells written by the
    // abandoned launch must never look like cells of the next one.
    unsigned int epoch = 0;
    MB_CUDA(cudaMemcpy(&epoch, &plan->d_ctl->epoch, sizeof(epoch), cudaMemcpyDeviceToHost));
    epoch += 1;
    MB_CUDA(cudaMemset(plan->d_ctl, 0, sizeof(mb::Control)));
    MB_CUDA(cudaMemcpy(&plan->d_ctl->epoch, &epoch, sizeof(epoch), cudaMemcpyHostToDevice));
    ++plan->maps_written;  // not acquired, as far as the cleared block knows
    MB_CUDA(cudaMemcpy(&plan->d_ctl->maps_written, &plan->maps_written, sizeof(plan->maps_written),
                       cudaMemcpyHostToDevice));
    MB_CUDA(blank_relays(plan));
    MB_CUDA(mb::prompt_reset(plan->prompt));
    MB_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
    return MB_OK;
}

int mb_prefill_cuts(const mb_phase* phases, uint32_t n_phases, uint32_t n_dynamic, int32_t sm_count,
                    int32_t* form, mb_prefill_cut out[5]) {
    if (phases == nullptr || form == nullptr || out == nullptr || n_phases == 0 || sm_count < 1) return MB_ERR_INVALID;
    for (unsigned int i = 0; i < n_phases; ++i) {
        const int rc = mb::prefill_validate(phases[i], UINT_MAX, n_dynamic);
        if (rc != MB_OK) return rc;
    }
    return mb::prompt_cuts(std::vector<mb_phase>(phases, phases + n_phases), n_dynamic, sm_count, form, out);
}

void mb_plan_destroy(mb_plan* plan) {
    if (plan == nullptr) return;
    {
        DeviceGuard guard(plan->device);
        if (plan->d_entries) cudaFree(plan->d_entries);
        if (plan->d_streams) cudaFree(plan->d_streams);
        if (plan->d_maps) cudaFree(plan->d_maps);
        if (plan->d_relay) cudaFree(plan->d_relay);
        if (plan->d_ctl) cudaFree(plan->d_ctl);
        mb::prefill_destroy(plan->prefill);
        mb::prompt_destroy(plan->prompt);
    }
    delete plan;
}

}  // extern "C"

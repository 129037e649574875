// Host-visible handles of the megakernels (one translation unit per kernel).
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "../../include/megabake_b200.h"

namespace mb {
struct KernelParams;
struct Control;
union StreamDesc;

int decode_threads();
int decode_fixed_smem();
int decode_stage_bytes();
int decode_row_pad();
int decode_row_tile();
int decode_rope_bytes(const mb_phase* phases, unsigned int n);
int decode_slice_slots(const mb_phase* phases, unsigned int n, int ctas);
int decode_ring_stages(int rope_bytes, unsigned int n_phases, int slots, int limit);  // < 2: does not fit
int decode_smem_bytes(int rope_bytes, unsigned int n_phases, int slots, int stages);
size_t decode_map_bytes();  // of the tensor maps of one phase
bool decode_encode_maps(const mb_phase& phase, const unsigned long long* addresses, int ctas, void* out);
// The same for one launch: encoded now, written to `out` on the device in stream order.
cudaError_t decode_store_maps(const mb_phase& phase, const unsigned long long* addresses, int ctas, void* out,
                              Control* ctl, cudaStream_t stream);
void decode_stream(const mb_phase& phase, const unsigned long long* addresses, int ctas, int slots,
                   StreamDesc* out);
int decode_head_dim(const mb_phase* phases, unsigned int n);  // of all attention phases; 0: a mix
cudaError_t decode_configure(int head_dim, int smem_bytes);
cudaError_t decode_occupancy(int head_dim, int smem_bytes, int* blocks_per_sm);
cudaError_t decode_launch(const KernelParams& params, int head_dim, int ctas, int smem_bytes,
                          cudaStream_t stream);

// Prefill plans (mb_prefill.cu): one kernel launch per phase; mb_prompt.cu below takes short prompts.
struct PrefillState;
int prefill_validate(const mb_phase& phase, unsigned int n_slots, unsigned int n_dynamic);
cudaError_t prefill_create(std::vector<mb_phase>& phases, int sm_count, PrefillState** out);
int prefill_launch_count(const PrefillState* state);  // kernels one prefill_launch enqueues
void prefill_destroy(PrefillState* state);
int prefill_bind(PrefillState* state, const std::vector<mb_phase>& phases,
                 const std::vector<unsigned long long>& slots, Control* ctl);
cudaError_t prefill_launch(PrefillState* state, const std::vector<mb_phase>& phases,
                           const std::vector<unsigned long long>& slots, unsigned int n_dynamic,
                           const unsigned long long* dynamic_addresses, Control* ctl,
                           unsigned long long* trace, cudaStream_t stream);

// Short prompts (mb_prompt.cu): the whole of a prefill plan as one launch.  The state stays null where the phases are
// no such prompt.
struct PromptState;
cudaError_t prompt_create(const std::vector<mb_phase>& phases, unsigned int n_dynamic, int sm_count,
                          unsigned int wait_limit_us, PromptState** out);
void prompt_destroy(PromptState* state);
int prompt_cuts(const std::vector<mb_phase>& phases, unsigned int n_dynamic, int sm_count, int* form,
                mb_prefill_cut* out);
cudaError_t prompt_reset(PromptState* state);
int prompt_bind(PromptState* state, const std::vector<unsigned long long>& slots, Control* ctl);
cudaError_t prompt_launch(const PromptState* state, const std::vector<unsigned long long>& slots,
                          const unsigned long long* dynamic_addresses, unsigned long long* trace,
                          cudaStream_t stream);
}  // namespace mb

// Host launchers of the activation prepare kernels (prepare.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace sharq {

// Bytes of scratch the scaled / RMSNorm-fused prepare needs for M rows:
// [0,4) tensor absmax bits (not written for a tensor-scale input of up to 64 K elements, 192 K without room for a word per
// CTA), [4,8) grid barrier counter, [256, 256 + 4*M) per-row inv_rms.
size_t prepare_workspace_bytes(int m);

// With that many bytes nothing has to be zeroed between the launches.
size_t prepare_workspace_best_bytes(int m);

// Prepare of an already scaled bf16 activation [m,k].  With q_sparse_dense != nullptr
// the debug variant runs (dense sparse payload instead of a_comp/e).
cudaError_t run_prepare(const void *x, int m, int k, void *a_comp, void *e, void *q_sparse_dense,
                        void *sfa_sparse, void *q_res, void *sf_res, cudaStream_t stream);

// Row statistics + prepare with the tensor scale (and RMSNorm when gamma != nullptr)
// applied inline.  inv_rms_external (optional) receives the per-row inv_rms instead of
// the workspace slot.  With absmax_words > 0 (gamma == nullptr only) the workspace already
// holds the bits of max|x|, the largest of that many words, and the statistics pass is skipped.  With residual (RMSNorm path
// only) the input is bf16(x + residual), which the statistics kernel also writes to sum_out.
// amax_out (optional, with absmax_words) receives the bits of the largest word.
// workspace_bytes beyond the minimum hold the maxima of the statistics kernel's CTAs (prepare_workspace_best_bytes).
cudaError_t run_scaled_prepare(const void *x, const void *gamma, float eps, int m, int k, void *workspace,
                               float *inv_rms_external, void *a_comp, void *e, void *sfa_sparse, void *q_res,
                               void *sf_res, float *scale_out, cudaStream_t stream, int absmax_words = 0,
                               const void *residual = nullptr, void *sum_out = nullptr, size_t workspace_bytes = 0,
                               unsigned int *amax_out = nullptr);

// The form that run_scaled_prepare takes on a GPU of `sms` SMs: 0 = every CTA scans the input for its maximum, 1 = every cluster of CTAs,
// 2 = a statistics launch and 8 elements per lane, 3 = a statistics launch (none with absmax_ready) and a 32-element group per lane, 4 = one cooperative launch.
int scaled_prepare_form(int m, int k, bool rms, bool residual, bool absmax_ready, size_t workspace_bytes, int sms);

// Tensor-scale prepare of a grouped activation (mixture-of-experts layers): rows sorted by group in
// 256-row units (m a multiple of 256), unit_group[u] < 0 = unit without rows (its outputs are
// zero metadata / scales and untouched payload), amax_bits[g] = bits of max|x| over group g
// (already computed), scale_vec_out[g] = clamp(amax_g / 2688, 1e-9).  With src_row the output row r is
// prepared from input row src_row[r] of x (a gather; < 0: a padding row, all-zero scales).  Every group is divided by
// its own scale, exactly as a separate call per group would do.
cudaError_t run_grouped_prepare(const void *x, int m, int k, const unsigned int *amax_bits, const int *unit_group, int groups,
                                void *a_comp, void *e, void *sfa_sparse, void *q_res, void *sf_res, float *scale_vec_out,
                                cudaStream_t stream, const int *src_row = nullptr);

// Grid barriers of the one-launch prepare that ran out on the current device since the library
// was loaded (0 in a healthy process; -1 when the counter cannot be read).
int prepare_timeouts();

}  // namespace sharq

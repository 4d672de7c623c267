/*
 * sharq_b200 - C ABI of the B200 (sm_100a) SharQ quantized-linear kernels.
 *
 * Every entry point takes plain device pointers, sizes and a CUDA stream handle
 * (cudaStream_t passed as void*; NULL = the legacy default stream), enqueues its work
 * on that stream and returns without synchronising.  Return value: 0 on success,
 * non-zero on an argument or launch error; sharq_last_error() then returns a message
 * (thread-local).  Unless stated otherwise an entry point allocates nothing and keeps
 * no state: every buffer, including scratch, is provided by the caller.
 *
 * The entry points are what a binding of the reference's `sharq_ops` module would call:
 * each comment names the reference op it stands behind (file:line in the reference
 * project, kernels/src/bindings.cpp unless another file is named).
 *
 * Buffer formats (identical to the reference's):
 *   payload     e2m1, two elements per byte (element 2i in the low nibble), row-major [rows, K/2]
 *   A_comp      per 8 logical K the two kept pair-bytes, row-major [M, K/4]
 *   E           per 8 logical K one nibble idx0 | idx1 << 2; layout [ceil(K/256)][ceil128(M)][16 B]
 *   scales      UE4M3, blocked: 512-byte tiles of 128 rows x 4 scales
 *               offset = (r/128)*(G/4)*512 + (g/4)*512 + (r%32)*16 + ((r/32)%4)*4 + g%4,
 *               G = K/16 (dense) or K/32 (sparse main path); allocation (rows/128+1)*128*K/16
 *   outputs     bf16 row-major [M, N]
 */
#ifndef SHARQ_B200_H_
#define SHARQ_B200_H_

#include <stddef.h>
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

/* Library version (major*10000 + minor*100 + patch). */
int sharq_version(void);

/* Message of the last failing call on this thread ("" if none). */
const char *sharq_last_error(void);

/* get_sparse_nvfp4_buffer_sizes(M,N,K) -> (A_comp, E, SFA, SFB) bytes.  bindings.cpp:232-241 */
int sharq_get_sparse_nvfp4_buffer_sizes(int m, int n, int k, int64_t out_bytes[4]);

/* get_fused_sparse_residual_buffer_sizes(M,N,K) -> (A_comp, E, SFA_sparse, Q_res, SF_res) bytes.
 * bindings.cpp:243-253 */
int sharq_get_fused_sparse_residual_buffer_sizes(int m, int n, int k, int64_t out_bytes[5]);

/* fused_sparse_residual_quantize_x(X, N): X is a pre-scaled bf16 [M,K], K % 128 == 0.
 * Writes every byte of the five output buffers (sizes from the call above), padding
 * included, so they need not be zero-initialised.  bindings.cpp:255-289 */
int sharq_fused_sparse_residual_quantize_x(const void *x_bf16, int m, int n, int k, void *a_comp, void *e,
                                           void *sfa_sparse, void *q_res, void *sf_res, void *stream);

/* fused_sparse_residual_quantize_x_debug(X, N): dense sparse payload [M,K/2] instead of
 * A_comp/E.  bindings.cpp:357-390 */
int sharq_fused_sparse_residual_quantize_x_debug(const void *x_bf16, int m, int n, int k, void *q_sparse,
                                                 void *sfa_sparse, void *q_res, void *sf_res, void *stream);

/* Scratch bytes needed by the scaled prepare calls below for M rows.  Layout:
 * bytes [0,4) tensor absmax (float bits; not written by a call without RMSNorm on up to 64 K elements, or up to 192 K where there
 * is no room for a word per CTA, see below), bytes [4,8) arrival counter of the grid-wide barrier,
 * bytes [256, 256+4*M) per-row inv_rms (float).  The calls initialise what they use. */
size_t sharq_prepare_workspace_bytes(int m);
/* With this many bytes (room for a maximum per CTA of the statistics launch, up to 4096 of them) nothing is zeroed between the launches. */
size_t sharq_prepare_workspace_best_bytes(int m);

/* A scaled prepare call runs its statistics and its quantisation as two launches or, with the smaller workspace and with the
 * residual add on middle sizes, as one cooperative launch whose CTAs meet at a grid-wide barrier with a bounded wait (about one
 * second).  Returns how many such
 * waits ran out on the current device since the library was loaded: 0 in a healthy process (the
 * outputs of a call that timed out are undefined), -1 if the counter cannot be read.  Synchronises
 * nothing itself: call it after synchronising the stream.  No counterpart in the reference. */
int sharq_prepare_timeouts(void);

/* fused_rmsnorm_sparse_residual_quantize_x(X, rmsnorm_weight, eps, N): RMSNorm, tensor
 * scale = clamp(amax/2688, 1e-9) and prepare, in two launches or one (see sharq_prepare_timeouts).
 * The normalised values are divided by the float32 scale, as the reference's kernel does
 * (kernels/src/fused_rmsnorm_sparse_prepare.cu:195-204).
 * K % 128 == 0 and K/32 <= 1024.  scale_out: one device float.  bindings.cpp:291-355 */
int sharq_fused_rmsnorm_sparse_residual_quantize_x(const void *x_bf16, const void *rmsnorm_weight_bf16,
                                                   float rmsnorm_eps, int m, int n, int k, void *workspace,
                                                   size_t workspace_bytes, void *a_comp, void *e, void *sfa_sparse,
                                                   void *q_res, void *sf_res, float *scale_out, void *stream);

/* The same with the decoder's residual add folded in (no counterpart in the reference, whose
 * layer wrapper adds with ATen before the call, model/qLlamaLayer.py:216-221): the input is
 * S = bf16(X + residual), rounded like the ATen add; the statistics kernel forms S, writes it
 * to sum_out [M,K] (may alias neither input) and the prepare reads it.  Outputs equal
 * sharq_fused_rmsnorm_sparse_residual_quantize_x(S, ...). */
int sharq_fused_add_rmsnorm_sparse_residual_quantize_x(const void *x_bf16, const void *residual_bf16, void *sum_out_bf16,
                                                       const void *rmsnorm_weight_bf16, float rmsnorm_eps, int m, int n,
                                                       int k, void *workspace, size_t workspace_bytes, void *a_comp,
                                                       void *e, void *sfa_sparse, void *q_res, void *sf_res,
                                                       float *scale_out, void *stream);

/* The non-RMSNorm activation path with its host-side passes folded in: computes
 * scale = clamp(max|X|/2688, 1e-9), X' = (X / scale).to(bf16) and the prepare of X'.  Equals
 * global_nvfp4_scale + divide + fused_sparse_residual_quantize_x of the reference
 * (model/quantize.py:43-44,179-183) as torch evaluates them on a CUDA device: dividing a bf16
 * tensor by a 0-dim float32 tensor there casts the divisor to bf16 first, so X' =
 * bf16(float(X) / float(bf16(scale))), while scale_out receives the unrounded float32 scale
 * (which the reference multiplies into the GEMM output). */
int sharq_scaled_sparse_residual_quantize_x(const void *x_bf16, int m, int n, int k, void *workspace,
                                            size_t workspace_bytes, void *a_comp, void *e, void *sfa_sparse,
                                            void *q_res, void *sf_res, float *scale_out, void *stream);

/* Decoder-layer steps between the SharQ linears, which the reference leaves to
 * HuggingFace's PyTorch code; each intermediate is rounded to bf16 where the PyTorch
 * composition rounds, so the results are those of the ATen ops.
 *
 * sharq_rope_inplace: rotary embedding x*cos + rotate_half(x)*sin, in place, on the first
 * `heads` heads of every row of a bf16 matrix (the query and key heads of a merged qkv
 * activation); row_stride in elements; position of a row = row % seq_len; cos/sin are bf16
 * [seq_len, head_dim].  Stands behind apply_rotary_pos_emb at model/qLlamaLayer.py:137-141.
 *
 * sharq_swiglu: H[rows, ffn] = silu(gate) * up of a contiguous merged activation
 * gate_up[rows, 2*ffn] (gate columns first).  model/qLlamaLayer.py:183-185.
 *
 * sharq_swiglu_sparse_residual_quantize_x: the same H (written to h_bf16, [M, K]) and the
 * scaled prepare of H for down_proj in two launches instead of the reference's five passes
 * (silu, mul, amax, divide, prepare): the SwiGLU kernel leaves max|H| in the workspace, so
 * the statistics pass of sharq_scaled_sparse_residual_quantize_x is not needed.  Outputs
 * equal sharq_scaled_sparse_residual_quantize_x(H).  workspace: 256 bytes, whose first word gets the bits of max|H|; with 8 KB behind them
 * (a maximum per CTA) nothing is zeroed first. */
int sharq_rope_inplace(void *x_bf16, int rows, int row_stride, int seq_len, int heads, int head_dim,
                       const void *cos_bf16, const void *sin_bf16, void *stream);
/* sharq_scatter_add_scaled: out[rows[i], :] += y[i, :] * w[i] in bf16 with the roundings of
 * `final.index_add_(0, rows, y * w[:, None])` (the expert loop of model/qMixtralLayer.py:228-231);
 * out [out_rows, width] and y [n_rows, width] contiguous bf16, rows int64 and pairwise distinct, w bf16;
 * an index outside [0, out_rows) is skipped. */
int sharq_scatter_add_scaled(void *out_bf16, int out_rows, const void *y_bf16, const int64_t *rows, const void *w_bf16,
                             int n_rows, int width, void *stream);
int sharq_swiglu(const void *gate_up_bf16, int rows, int ffn, void *h_bf16, void *stream);
/* sharq_add_rmsnorm: out[rows, K] = bf16(s * rsqrt(mean(s^2) + eps) * gamma) with s = bf16(x + residual) written to
 * sum_out (both NULL: s = x); mean and products in float, one rounding per element.  The normalised bf16
 * activation that the router and the experts of a mixture-of-experts layer both read
 * (model/qMixtralLayer.py:205-213; the reference calls HuggingFace's RMSNorm module there).  K % 8 == 0, K <= 8192. */
int sharq_add_rmsnorm(const void *x_bf16, const void *residual_bf16, void *sum_out_bf16, const void *gamma_bf16, float eps,
                      int rows, int k, void *out_bf16, void *stream);
int sharq_swiglu_sparse_residual_quantize_x(const void *gate_up_bf16, int m, int n, int k, void *h_bf16,
                                            void *workspace, size_t workspace_bytes, void *a_comp, void *e,
                                            void *sfa_sparse, void *q_res, void *sf_res, float *scale_out,
                                            void *stream);

/* quantize_w32_shared(W): bf16 [N,K] (already divided by the weight tensor scale),
 * K % 32 == 0 -> QW [N,K/2], SFW_sparse (32-groups), SFW_dense (each scale duplicated
 * into two 16-group slots).  bindings.cpp:392-417 */
int sharq_quantize_w32_shared(const void *w_bf16, int n, int k, void *qw, void *sfw_sparse, void *sfw_dense,
                              void *stream);

/* duplicate_sfa32_to_sfa16(SFA_sparse, M, N, K).  bindings.cpp:419-437 */
int sharq_duplicate_sfa32_to_sfa16(const void *sfa_sparse, int m, int n, int k, void *sfa_dense, void *stream);

/* quantize_x_nvfp4(X) / quantize_w_nvfp4(W) (and reorder_quantize_x/w with the identity
 * index and KE == 0): dense NVFP4, one scale per 16.  K % 16 == 0.  Only the used bytes
 * of the scale buffer are written, as in the reference.  bindings.cpp:74-160 */
int sharq_quantize_nvfp4(const void *x_bf16, int rows, int k, void *q, void *sf, void *stream);

/* The two with their host-side passes folded in (model/quantize.py:43-44,141-169): scale = clamp(max|x|/2688, 1e-9)
 * and the quantisation of (x / scale).to(bf16) as torch evaluates it on a CUDA device (the 0-dim divisor is cast
 * to bf16 first), in two launches.  x 16-byte aligned; workspace: sharq_scaled_quantize_workspace_bytes() bytes with
 * any content; scale_out: one device float.  nvfp4: K % 64 == 0, padding bytes of sf untouched.  w32_shared:
 * K % 128 == 0 and K/32 <= 1024, every byte of both scale buffers is written. */
size_t sharq_scaled_quantize_workspace_bytes(void);
int sharq_scaled_quantize_nvfp4(const void *x_bf16, int rows, int k, void *workspace, size_t workspace_bytes, void *q, void *sf,
                                float *scale_out, void *stream);
int sharq_scaled_quantize_w32_shared(const void *w_bf16, int n, int k, void *workspace, size_t workspace_bytes, void *qw,
                                     void *sfw_sparse, void *sfw_dense, float *scale_out, void *stream);

/* compress_sparse_a(A_q_dense, N): dense payload with at most two non-zero bytes per
 * 4-byte chunk -> A_comp, E.  bindings.cpp:164-230 */
int sharq_compress_sparse_a(const void *a_q_dense, int m, int n, int k, void *a_comp, void *e, void *stream);

/* matmul / matmul_tensor_scale / matmul_accum / matmul_accum_tensor_scale:
 * D = bf16(alpha * (A . B^T) + beta * C_in).  With alpha_dev (one device float) non-NULL
 * the factor is alpha * (*alpha_dev) (the reference passes alpha = 1 then); c_in may be
 * NULL when beta == 0.  K % 64 == 0.
 * error_flag: one device int the kernel sets non-zero if an internal bounded wait ran
 * out (never expected; the output is then undefined).  bindings.cpp:441-569 */
int sharq_matmul(const void *a, const void *b, const void *sfa, const void *sfb, int m, int n, int k, float alpha,
                 const float *alpha_dev, const void *c_in, float beta, void *d, int *error_flag, void *stream);

/* sparse_matmul / sparse_matmul_tensor_scale: beta must be 0.  K % 128 == 0.
 * bindings.cpp:571-701 */
int sharq_sparse_matmul(const void *a_comp, const void *b, const void *e, const void *sfa, const void *sfb, int m,
                        int n, int k, float alpha, const float *alpha_dev, float beta, void *d, int *error_flag,
                        void *stream);

/* The SharQ linear GEMM in one launch: D = bf16(alpha * (A_sparse + A_res) . W^T) (+ bias
 * in bf16), the sparse main pass and the dense residual pass reading the same weight tile
 * and accumulating into one tensor-memory tile.  Stands behind the two-launch composition
 * of model/qLinearLayer.py:130-154 (+ bias add at :177-179) and is what the optional
 * `sharq_linear_forward` op probed by benchmarks/vllm/sharq.py:206-213 runs. */
int sharq_linear_gemm(const void *a_comp, const void *e, const void *sfa_sparse, const void *q_res,
                      const void *sf_res, const void *qw, const void *sfw_sparse, const void *sfw_dense, int m, int n,
                      int k, float alpha, const float *alpha_dev, const void *bias_bf16, void *d, int *error_flag,
                      void *stream);

/* The three GEMMs with leave to split K (no counterpart in the reference).  With a workspace of
 * sharq_gemm_workspace_bytes(M, N) bytes (nothing is written to it: any 16-byte aligned device pointer will do) a GEMM
 * whose tiles alone would leave SMs idle, bound by streaming the weights, splits K over the CTAs of a cluster, which sum their fp32
 * partial tiles on chip in a fixed order: results are the same from call to call, in another order of additions
 * than the unsplit launch.  With workspace == NULL these are the plain entry points. */
size_t sharq_gemm_workspace_bytes(int m, int n);
int sharq_matmul_ws(const void *a, const void *b, const void *sfa, const void *sfb, int m, int n, int k, float alpha,
                    const float *alpha_dev, const void *c_in, float beta, void *d, void *workspace,
                    size_t workspace_bytes, int *error_flag, void *stream);
/* sharq_matmul_ws with a bias [N] (bf16) added to the bf16 result, rounded as a separate bf16 add would. */
int sharq_matmul_bias_ws(const void *a, const void *b, const void *sfa, const void *sfb, int m, int n, int k, float alpha,
                         const float *alpha_dev, const void *c_in, float beta, const void *bias_bf16, void *d, void *workspace,
                         size_t workspace_bytes, int *error_flag, void *stream);
int sharq_sparse_matmul_ws(const void *a_comp, const void *b, const void *e, const void *sfa, const void *sfb, int m,
                           int n, int k, float alpha, const float *alpha_dev, float beta, void *d, void *workspace,
                           size_t workspace_bytes, int *error_flag, void *stream);
int sharq_linear_gemm_ws(const void *a_comp, const void *e, const void *sfa_sparse, const void *q_res,
                         const void *sf_res, const void *qw, const void *sfw_sparse, const void *sfw_dense, int m, int n,
                         int k, float alpha, const float *alpha_dev, const void *bias_bf16, void *d, void *workspace,
                         size_t workspace_bytes, int *error_flag, void *stream);

/* Fused SharQ GEMM of a merged gate_up weight [2*ffn, K] (gate rows first, ffn % 128 == 0, no bias) whose epilogue
 * applies SwiGLU: h[m, ffn] = bf16(bf16(silu(gate)) * up), gate and up rounded to bf16 first, and the bits of max|h| go to
 * amax_bits (sharq_gemm_swiglu_absmax_words(m, ffn) uint32 words, whose largest is the maximum; 16-byte aligned rows of h).  The same bits as sharq_linear_gemm followed by sharq_swiglu, without the [m, 2*ffn]
 * intermediate.  sharq_absmax_sparse_residual_quantize_x is sharq_scaled_sparse_residual_quantize_x for an X whose max|X|
 * is already in amax_bits, the largest of amax_words words (no statistics pass).  sharq_gemm_swiglu_pays: 1 where this form is the faster one. */
int sharq_gemm_swiglu_pays(int m, int ffn, int k);
int sharq_linear_gemm_swiglu(const void *a_comp, const void *e, const void *sfa_sparse, const void *q_res, const void *sf_res,
                             const void *qw, const void *sfw_sparse, const void *sfw_dense, int m, int ffn, int k, float alpha,
                             const float *alpha_dev, void *h, void *amax_bits, int *error_flag, void *stream);
int sharq_gemm_swiglu_absmax_words(int m, int ffn);
int sharq_absmax_sparse_residual_quantize_x(const void *x_bf16, int m, int n, int k, const void *amax_bits, int amax_words,
                                            void *a_comp, void *e, void *sfa_sparse, void *q_res, void *sf_res, float *scale_out,
                                            void *stream);

/* sharq_linear_gemm_ws with a residual [M, N] (bf16, 16-byte aligned) added to the bf16 result in the epilogue, rounded as a
 * separate bf16 add would: the residual add behind a decoder layer's last linear. */
int sharq_linear_gemm_residual(const void *a_comp, const void *e, const void *sfa_sparse, const void *q_res, const void *sf_res,
                               const void *qw, const void *sfw_sparse, const void *sfw_dense, int m, int n, int k, float alpha,
                               const float *alpha_dev, const void *bias_bf16, const void *residual_bf16, void *d, void *workspace,
                               size_t workspace_bytes, int *error_flag, void *stream);

/* No counterpart in the reference.  Same work and outputs as
 * sharq_fused_rmsnorm_sparse_residual_quantize_x, for callers that cannot allocate device
 * memory and have no spare buffer to pass as workspace (a server that has given all free
 * HBM to its own pool; a thread on which cudaMalloc's device-wide synchronisation is not
 * allowed): the scratch lives in a fixed array inside the library (256 KiB + 256 B per GPU
 * that loads it).  M <= sharq_noalloc_max_rows() (65536), larger M is an error.  The first
 * call on a device looks up the array's address and should come before any stream capture;
 * no call allocates.  All calls on a device share the array: calls that overlap on the GPU
 * race, so order them on one stream (or with events).  Errors: non-zero return,
 * message from sharq_noalloc_last_error(). */
int sharq_fused_rmsnorm_sparse_residual_quantize_x_noalloc(const void *x_bf16, const void *rmsnorm_weight_bf16,
                                                           float rmsnorm_eps, int m, int n, int k, void *a_comp,
                                                           void *e, void *sfa_sparse, void *q_res, void *sf_res,
                                                           float *scale_out, void *stream);
int sharq_noalloc_max_rows(void);
const char *sharq_noalloc_last_error(void);

/* No counterpart in the reference (it has no tensor parallelism).  In-place sum, over the
 * `world` GPUs of one NVSwitch domain, of a bf16 buffer that every rank holds at the same
 * offset of a symmetric-memory allocation bound to an NVLink multicast object: the partial
 * outputs of a row-parallel SharQ linear (o_proj, down_proj).  One kernel per rank: rank r
 * reduces bytes [r, r+1) * n_bytes / world inside the switch (multimem.ld_reduce, fp32
 * accumulation) and stores the rounded bf16 sums to every rank's copy (multimem.st).
 *   multicast_data   multicast address of the buffer
 *   rank_flag_ptrs   HOST array of `world` device pointers: rank p's flag area as mapped in
 *                    this process (peer mapping; entry `rank` is the local one).  Each area
 *                    holds sharq_allreduce_flag_bytes() bytes, zeroed once (on every rank,
 *                    followed by a barrier) before the first call; afterwards it holds the
 *                    kernels' barrier counters and must not be touched.
 *   n_bytes          multiple of 16 * world; max_ctas: 0 = default.
 * All ranks must make the same calls in the same order with the same sizes.  The kernels of
 * the ranks wait for one another with bounded spins (about two seconds); a wait that runs
 * out sets *error_flag non-zero.  world <= 16. */
int sharq_allreduce_bf16_multimem(void *multicast_data, void *const *rank_flag_ptrs, int rank, int world,
                                  size_t n_bytes, int max_ctas, int *error_flag, void *stream);
size_t sharq_allreduce_flag_bytes(void);
/* The same sum with plain peer loads and stores instead of the multicast object, for
 * world <= 4 (it moves fewer bytes per link than the in-switch form at world == 2):
 * rank_data_ptrs[p] = rank p's copy of the buffer as mapped in this process.  Rank r sums
 * slice r of all copies in rank order (fp32) and writes the bf16 result into every copy. */
int sharq_allreduce_bf16_peer(void *const *rank_data_ptrs, void *const *rank_flag_ptrs, int rank, int world,
                              size_t n_bytes, int max_ctas, int *error_flag, void *stream);

/* Mixture-of-experts FFN in grouped launches.  The reference runs its experts in a Python loop
 * (model/qMixtralLayer.py:223-231): per expert a gather of its tokens, prepare, two GEMMs, SwiGLU, a
 * routing-weight multiply and index_add_.  These entry points do each step once for ALL experts on a
 * GROUPED activation: the token slots are sorted by expert, every expert's segment is padded to a
 * multiple of 256 rows, M is the padded total, and unit_group[u] (device, M/256 ints) is the expert
 * of rows [256u, 256u+256) or < 0 for a unit without rows.  Arithmetic per row is that of the
 * per-expert calls: every expert's rows are divided by that expert's own tensor scale.
 *   sharq_grouped_sparse_residual_quantize_x: per-expert max|X| (into amax_workspace, `groups`
 *     uint32 words) + scaled prepare; scale_vec_out[g] = clamp(amax_g / 2688, 1e-9).  src_row (optional,
 *     device, M ints) gathers: grouped row r is row src_row[r] of the token-major X (< 0: padding row).
 *   sharq_grouped_swiglu_sparse_residual_quantize_x: H = silu(gate) * up of gate_up [M, 2K] (written
 *     to h_bf16 [M, K]), per-expert max|H| and the scaled prepare of H.
 *   sharq_linear_gemm_grouped: D[r] = alpha * alpha_vec[g] * (A_sparse[r] + A_res[r]) . W_g^T for every
 *     row r of a unit of expert g (one launch; qw / sfw_sparse / sfw_dense: host arrays of `groups`
 *     device pointers; alpha_vec: device, e.g. activation scale x weight scale per expert).
 *   sharq_linear_gemm_grouped_swiglu / sharq_grouped_absmax_sparse_residual_quantize_x: the grouped
 *     forms of sharq_linear_gemm_swiglu and sharq_absmax_sparse_residual_quantize_x (amax_workspace: `groups` words).
 *   sharq_moe_plan: the grouping itself from selected [tokens * top_k] (expert of every token slot, experts <= 16, unit 256
 *     for the entry points below): dest[slot] = its grouped row (ascending slots inside an expert), src_row[row] = its
 *     token or -1, unit_group as above; rows >= (ceil(slots / unit) + experts) * unit, a multiple of unit.
 *     A slot whose expert is outside [0, experts) has no row: dest is -1.  sharq_moe_plan_flagged also stores the code
 *     0x401 in *error_flag (device) then.
 *   sharq_moe_combine: out[t] = sum over the top_k slots of token t, in ascending expert order, of
 *     y[dest[t,j]] * w[t,j] with bf16 rounding after every product and addition, which is what the
 *     reference's sequence of index_add_ calls on a zero buffer computes.  dest < 0: the token's row is NaN. */
int sharq_grouped_sparse_residual_quantize_x(const void *x_bf16, const int *src_row, int m, int n, int k,
                                            const int *unit_group, int groups, void *amax_workspace, void *a_comp, void *e,
                                            void *sfa_sparse, void *q_res, void *sf_res, float *scale_vec_out, void *stream);
int sharq_grouped_swiglu_sparse_residual_quantize_x(const void *gate_up_bf16, int m, int n, int k, void *h_bf16,
                                                   const int *unit_group, int groups, void *amax_workspace, void *a_comp,
                                                   void *e, void *sfa_sparse, void *q_res, void *sf_res,
                                                   float *scale_vec_out, void *stream);
int sharq_linear_gemm_grouped(const void *a_comp, const void *e, const void *sfa_sparse, const void *q_res, const void *sf_res,
                              int groups, const void *const *qw, const void *const *sfw_sparse, const void *const *sfw_dense,
                              const int *unit_group, const float *alpha_vec, float alpha, int m, int n, int k, void *d,
                              int *error_flag, void *stream);
int sharq_linear_gemm_grouped_swiglu(const void *a_comp, const void *e, const void *sfa_sparse, const void *q_res,
                                     const void *sf_res, int groups, const void *const *qw, const void *const *sfw_sparse,
                                     const void *const *sfw_dense, const int *unit_group, const float *alpha_vec, float alpha,
                                     int m, int ffn, int k, void *h, void *amax_workspace, int *error_flag, void *stream);
int sharq_grouped_absmax_sparse_residual_quantize_x(const void *x_bf16, int m, int n, int k, const int *unit_group, int groups,
                                                    const void *amax_workspace, void *a_comp, void *e, void *sfa_sparse,
                                                    void *q_res, void *sf_res, float *scale_vec_out, void *stream);
int sharq_moe_plan(const int64_t *selected, int64_t slots, int top_k, int experts, int unit, int64_t rows, void *workspace,
                   size_t workspace_bytes, int *dest, int *src_row, int *unit_group, void *stream);
int sharq_moe_plan_flagged(const int64_t *selected, int64_t slots, int top_k, int experts, int unit, int64_t rows, void *workspace,
                           size_t workspace_bytes, int *dest, int *src_row, int *unit_group, int *error_flag, void *stream);
size_t sharq_moe_plan_workspace_bytes(int64_t slots);
int sharq_moe_combine(void *out_bf16, const void *y_bf16, const int *dest, const int64_t *selected, const void *w_bf16,
                      int tokens, int top_k, int width, void *stream);
/* ... + residual [tokens, width] (bf16, 16-byte aligned), added last and rounded as a separate bf16 add would. */
int sharq_moe_combine_residual(void *out_bf16, const void *y_bf16, const int *dest, const int64_t *selected, const void *w_bf16,
                               const void *residual_bf16, int tokens, int top_k, int width, void *stream);

/* No counterpart in the reference (it has no tensor parallelism).  Row-parallel SharQ linear and the
 * transition to the next column-parallel one over the GPUs of one NVLink domain, with the residual
 * stream sharded by rows (GPU r owns rows [r*M/world, (r+1)*M/world)), in two launches per GPU:
 *
 * sharq_linear_gemm_scatter: sharq_linear_gemm whose epilogue deals the output rows to their owners:
 *   row q of this GPU's partial product goes, through the peer mapping d_rank_ptrs[o] of owner
 *   o = q / (M/world), into block `rank` of GPU o's collection buffer [world][M/world, N] bf16 (plain
 *   peer stores, so the transfer runs while the GEMM computes).  M % (128*world) == 0, N % 8 == 0.
 *
 * sharq_tp_reduce_rmsnorm_prepare_allgather (one cooperative kernel): waits until every GPU has delivered,
 *   S   = sum over the `world` blocks of partial_blocks (this GPU's collection buffer) in fp32 in rank
 *         order, rounded to bf16 (partial_blocks == NULL: no sum),
 *   X'  = bf16(residual_in + S) for this GPU's rows, written to residual_out [M/world, K]
 *         (partial_blocks == NULL: X' = residual_in; residual_in == NULL: X' = S),
 *   then RMSNorm statistics of X', the tensor scale from the absmax over ALL GPUs' rows, the
 *   4:8 sparse + residual prepare of this GPU's rows, and the packed rows stored into EVERY
 *   GPU's copy of the prepared activation (plain peer stores; multimem.st with SHARQ_TP_ALLGATHER=multicast).
 * On return of the kernel every GPU's (a_comp, e, sfa_sparse, q_res, sf_res, *scale_out) hold
 * exactly what sharq_fused_rmsnorm_sparse_residual_quantize_x produces for the whole [M,K]
 * matrix X' on one GPU.  The five output buffers are this GPU's copy inside ONE symmetric
 * allocation whose multicast mapping is at local address + multicast_delta; rank_state_ptrs[r]
 * is GPU r's state block (sharq_tp_transition_state_bytes() bytes inside the SAME symmetric
 * allocation, zero-filled once, then owned by these calls) as mapped on this GPU: the kernel
 * reaches GPU r's copy of an output byte at its local address + (rank_state_ptrs[r] -
 * rank_state_ptrs[rank]).  workspace:
 * sharq_tp_transition_workspace_bytes(M/world) bytes of local scratch.
 * Requirements: M % (128*world) == 0, K % 128 == 0, K/32 <= 1024, 16-byte aligned buffers, the
 * same sequence of calls on every GPU.  Every cross-GPU wait is bounded (about ten seconds); one
 * that runs out stores a code 0x301..0x306 in *error_flag and the outputs are undefined.  Uses
 * plain peer stores and multimem.st only. */
int sharq_linear_gemm_scatter(const void *a_comp, const void *e, const void *sfa_sparse, const void *q_res, const void *sf_res,
                              const void *qw, const void *sfw_sparse, const void *sfw_dense, int m, int n, int k, float alpha,
                              const float *alpha_dev, void *const *d_rank_ptrs, int rank, int world, int *error_flag,
                              void *stream);
size_t sharq_tp_transition_state_bytes(void);
size_t sharq_tp_transition_workspace_bytes(int rows);
int sharq_tp_reduce_rmsnorm_prepare_allgather(const void *partial_blocks, const void *residual_in_bf16,
                                              void *residual_out_bf16, const void *rmsnorm_weight_bf16, float rmsnorm_eps,
                                              int m, int n, int k, void *workspace, size_t workspace_bytes, void *a_comp,
                                              void *e, void *sfa_sparse, void *q_res, void *sf_res,
                                              long long multicast_delta, float *scale_out, void *const *rank_state_ptrs,
                                              int rank, int world, int *error_flag, void *stream);

/* Test/tuning hook: how many SM clock cycles a cross-GPU wait of the all-reduce and transition
 * kernels may take before the kernel gives up, stores its error code and returns (0 restores the
 * defaults of two to ten seconds).  Applies to launches made after the call. */
int sharq_set_wait_limit_cycles(long long cycles);

/* Test/tuning hook: force the GEMM kernel variant (0 = automatic; 128 or 256 = single-CTA kernel
 * with that tile width; 512 = CTA-pair kernel, 256 x 256 tile per pair).  Process-wide. */
int sharq_set_gemm_tile_n(int tile_n);
/* Test/tuning hook: the variant that the automatic choice takes for a shape on a GPU of `sms` SMs (128, 256 or 512 as above);
 * split_k: whether the call gives leave to split K.  Runs nothing. */
int sharq_gemm_tile_n(int m, int n, int k, int split_k, int sms);
/* Test hook: how the fp32 parts of an output tile with `rows` rows (1..128) meet when K is split over `splits` CTAs (2..8) of a
 * single-CTA kernel (tile_n 128 or 256): 0 = sent to the CTAs that sum them, from registers; 1 = by block copies; 2 = read behind a
 * cluster barrier; -1 for other arguments.  Runs nothing. */
int sharq_gemm_exchange(int tile_n, int sparse, int dense, int rows, int k, int splits);

/* Test hook: the form that a scaled prepare call takes on a GPU of `sms` SMs with that workspace: 0 = every CTA scans the input for its
 * maximum, 1 = every cluster of CTAs does, 2 = a statistics launch and 8 elements per lane, 3 = a statistics launch (none with absmax_ready)
 * and a group per lane, 4 = one cooperative launch; -1 for other arguments.  Runs nothing. */
int sharq_scaled_prepare_form(int m, int k, int rms, int residual, int absmax_ready, size_t workspace_bytes, int sms);

#ifdef __cplusplus
}
#endif

#endif /* SHARQ_B200_H_ */

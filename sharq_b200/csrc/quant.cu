// Weight preparation and dense NVFP4 quantisation kernels for sm_100a.
//
// Replaces, behind the same buffer formats, the reference's
//   kernels/src/shared_weight_nvfp4.cu:20-189   (32-group shared weight payload, scale duplication)
//   kernels/src/reorder.cu:69-203,381-555 and kernels/src/down.cu:72-233 with identity
//   reorder and KE == 0                         (dense NVFP4 quantisation, 16-group scales)
//   kernels/src/bindings.cpp:164-230            (structured-sparse compressor, debug path)
//   model/quantize.py:43-44,141-169             (tensor scale and division in front of the two)
// The kernels that take an already scaled input are written for clarity: one thread per scale
// group, 16-byte loads and stores.
#include "common.cuh"
#include "prepare_device.cuh"
#include "quant.cuh"
#include "sm100_ptx.cuh"

namespace sharq {

namespace {

__device__ __forceinline__ void unpack8(const uint4 &v, float *f) {
  uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    f[2 * t] = bf16_bits_to_float(w[t] & 0xFFFFu);
    f[2 * t + 1] = bf16_bits_to_float(w[t] >> 16);
  }
}

// One thread per 32-element group of one weight row.
__global__ void __launch_bounds__(256) quantize_w32_shared_kernel(const __nv_bfloat16 *__restrict__ w, int n, int k,
                                                                   uint8_t *__restrict__ qw,
                                                                   uint8_t *__restrict__ sf_sparse,
                                                                   uint8_t *__restrict__ sf_dense) {
  const int groups = k >> 5;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)n * groups) return;
  const int row = (int)(idx / groups), g = (int)(idx % groups);
  const uint4 *src = reinterpret_cast<const uint4 *>(w + (size_t)row * k + (size_t)g * 32);
  float x[32];
#pragma unroll
  for (int j = 0; j < 4; ++j) unpack8(__ldg(src + j), x + 8 * j);
  float mx = 0.0f;
#pragma unroll
  for (int i = 0; i < 32; ++i) mx = fmaxf(mx, fabsf(x[i]));
  float s = fminf(fmaxf(__fdiv_rn(mx, kFp4Max), kScaleEps), kFp8Max);
  uint32_t code = float_to_ue4m3(s);
  float inv = __frcp_rn(ue4m3_to_float(code));
  uint32_t out[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    out[j] = pack_e2m1x8(__fmul_rn(x[8 * j + 0], inv), __fmul_rn(x[8 * j + 1], inv), __fmul_rn(x[8 * j + 2], inv),
                         __fmul_rn(x[8 * j + 3], inv), __fmul_rn(x[8 * j + 4], inv), __fmul_rn(x[8 * j + 5], inv),
                         __fmul_rn(x[8 * j + 6], inv), __fmul_rn(x[8 * j + 7], inv));
  *reinterpret_cast<uint4 *>(qw + (size_t)row * (k / 2) + (size_t)g * 16) = make_uint4(out[0], out[1], out[2], out[3]);
  sf_sparse[sf_offset(row, g, groups)] = (uint8_t)code;
  // the two 16-group slots of the dense layout are neighbours: one 16-bit store
  *reinterpret_cast<uint16_t *>(sf_dense + sf_offset(row, 2 * g, k / 16)) = (uint16_t)(code | (code << 8));
}

__global__ void __launch_bounds__(256) duplicate_sf32_to_sf16_kernel(const uint8_t *__restrict__ sf32, int rows, int k,
                                                                      uint8_t *__restrict__ sf16) {
  const int groups = k >> 5;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)rows * groups) return;
  const int row = (int)(idx / groups), g = (int)(idx % groups);
  uint32_t code = sf32[sf_offset(row, g, groups)];
  *reinterpret_cast<uint16_t *>(sf16 + sf_offset(row, 2 * g, k / 16)) = (uint16_t)(code | (code << 8));
}

// One thread per 16-element group.
__global__ void __launch_bounds__(256) quantize_dense_nvfp4_kernel(const __nv_bfloat16 *__restrict__ x, int rows, int k,
                                                                    uint8_t *__restrict__ q, uint8_t *__restrict__ sf) {
  const int groups = k >> 4;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)rows * groups) return;
  const int row = (int)(idx / groups), g = (int)(idx % groups);
  const uint4 *src = reinterpret_cast<const uint4 *>(x + (size_t)row * k + (size_t)g * 16);
  float v[16];
  unpack8(__ldg(src), v);
  unpack8(__ldg(src + 1), v + 8);
  float mx = 0.0f;
#pragma unroll
  for (int i = 0; i < 16; ++i) mx = fmaxf(mx, fabsf(v[i]));
  float s = clamp_val(__fdiv_rn(mx, kFp4Max), kScaleEps, kFp8Max);
  uint32_t code = float_to_ue4m3(s);
  // The reference writes this reciprocal as a double division rounded to float; for
  // every UE4M3 value that equals the correctly rounded float reciprocal.
  float inv = __frcp_rn(ue4m3_to_float(code));
  uint32_t lo = pack_e2m1x8(__fmul_rn(v[0], inv), __fmul_rn(v[1], inv), __fmul_rn(v[2], inv), __fmul_rn(v[3], inv),
                            __fmul_rn(v[4], inv), __fmul_rn(v[5], inv), __fmul_rn(v[6], inv), __fmul_rn(v[7], inv));
  uint32_t hi = pack_e2m1x8(__fmul_rn(v[8], inv), __fmul_rn(v[9], inv), __fmul_rn(v[10], inv), __fmul_rn(v[11], inv),
                            __fmul_rn(v[12], inv), __fmul_rn(v[13], inv), __fmul_rn(v[14], inv), __fmul_rn(v[15], inv));
  *reinterpret_cast<uint2 *>(q + (size_t)row * (k / 2) + (size_t)g * 8) = make_uint2(lo, hi);
  sf[sf_offset(row, g, groups)] = (uint8_t)code;
}

// One thread per 32-element group (four 8-element chunks): a dense payload that
// already holds at most two non-zero bytes per 4-byte chunk -> compressed bytes +
// metadata.  A byte counts as zero when both nibbles are +-0.
__global__ void __launch_bounds__(256) compress_sparse_a_kernel(const uint8_t *__restrict__ a_dense, int m, int k,
                                                                 uint8_t *__restrict__ a_comp, uint8_t *__restrict__ e) {
  const int groups = k >> 5;
  const int aligned_m = (m + 127) / 128 * 128;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)m * groups) return;
  const int row = (int)(idx / groups), g = (int)(idx % groups);
  uint4 v = *reinterpret_cast<const uint4 *>(a_dense + (size_t)row * (k / 2) + (size_t)g * 16);
  uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t comp[2] = {0, 0};
  uint32_t meta = 0;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t idx0 = 0, idx1 = 0, v0 = 0, v1 = 0;
    int cnt = 0;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      uint32_t b = (w[c] >> (8 * p)) & 0xFFu;
      bool nz = (b & 0x77u) != 0;
      if (nz && cnt == 0) {
        idx0 = p;
        v0 = b;
      } else if (nz && cnt == 1) {
        idx1 = p;
        v1 = b;
      }
      cnt += nz ? 1 : 0;
    }
    if (cnt == 1 && idx0 == 3) {
      v1 = v0;
      v0 = 0;
      idx0 = 0;
      idx1 = 3;
    } else if (cnt == 1) {
      v1 = 0;
      idx1 = 3;
    }
    uint32_t two = v0 | (v1 << 8);
    comp[c >> 1] |= (c & 1) ? (two << 16) : two;
    meta |= (idx0 | (idx1 << 2)) << (4 * c);
  }
  *reinterpret_cast<uint2 *>(a_comp + (size_t)row * (k / 4) + (size_t)g * 8) = make_uint2(comp[0], comp[1]);
  *reinterpret_cast<uint16_t *>(e + (size_t)(g / 8) * aligned_m * 16 + (size_t)row * 16 + (size_t)(g % 8) * 2) =
      (uint16_t)meta;
}

// ---------------------------------------------------------------------------
// Unscaled bf16 matrix -> tensor scale, division and quantisation in two launches.
//
// HBM-bound: x has to be read twice (the scale depends on all of it), 4 B + 0.6 B per element.
// Launch 1 leaves one maximum per CTA in `partials`, so nothing has to be zeroed first; launch 2
// reduces them again in every CTA and walks the matrix from its END, so that the last ~100 MB launch 1
// read come from L2.  As ATen passes (abs, max, float, divide, clamp, divide, cast) and a
// quantisation kernel this took 668 us at 28672 x 4096, of which 442 us were ATen's division by a
// 0-dim tensor; now about 90 us (absmax 37 us = 6.4 TB/s, quantisation 53 us; 102 us with 64-bit index divisions, IEEE divisions and
// unpacked products, and a gap between the launches), and 85 -> 13 us at 1000 x 14336 (dense).
//
// Arithmetic: dividing a bf16 CUDA tensor by a 0-dim float32 tensor casts the divisor to bf16 first, so
// y = bf16(x / float(bf16(scale))).  Quotients of two 8-bit significands are either representable
// or at least 2^-17 (relative) away from every bf16 rounding boundary, and x * (1 / div) is within
// 2^-22 of them: the product rounds to the same y.  A subnormal quotient may round differently,
// but its group's scale is clamped to >= 2^-9, under which it becomes a zero of the same sign either way.
// A NaN in x makes the scale and with it every y NaN, as the ATen passes do.
// ---------------------------------------------------------------------------
constexpr int kScaledThreads = 256;

__device__ __forceinline__ float block_max_nan(float mx, float *warp_max) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float other = __shfl_xor_sync(0xffffffffu, mx, o);
    mx = (mx != mx || other != other) ? __int_as_float(0x7fffffff) : fmaxf(mx, other);
  }
  if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = mx;
  __syncthreads();
  mx = warp_max[0];
#pragma unroll
  for (int w = 1; w < kScaledThreads / 32; ++w) {
    const float other = warp_max[w];
    mx = (mx != mx || other != other) ? __int_as_float(0x7fffffff) : fmaxf(mx, other);
  }
  return mx;
}

__global__ void __launch_bounds__(kScaledThreads) absmax_partials_kernel(const uint4 *x, size_t n16, float *partials) {
  __shared__ float warp_max[kScaledThreads / 32];
  ptx::grid_launch_dependents();
  ptx::grid_dependency_wait();
  __nv_bfloat162 m2 = __floats2bfloat162_rn(0.0f, 0.0f);
  const size_t stride = (size_t)gridDim.x * kScaledThreads;
  for (size_t i = (size_t)blockIdx.x * kScaledThreads + threadIdx.x; i < n16; i += 4 * stride) {
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = (i + u * stride < n16) ? x[i + u * stride] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
      for (int t = 0; t < 4; ++t) m2 = __hmax2_nan(m2, __habs2(*reinterpret_cast<const __nv_bfloat162 *>(&w[t])));
    }
  }
  const float lo = __bfloat162float(m2.x), hi = __bfloat162float(m2.y);
  const float mx = block_max_nan((lo != lo || hi != hi) ? __int_as_float(0x7fffffff) : fmaxf(lo, hi), warp_max);
  if (threadIdx.x == 0) partials[blockIdx.x] = mx;
}

// The bytes of both scale views of a shared weight that belong to no row: rows [n, ceil128(n)) of the
// last band and everything behind the bands (K % 128 == 0, so whole 32-bit words).
__device__ __forceinline__ void zero_scale_padding(int n, int k, uint8_t *sf_sparse, uint8_t *sf_dense) {
  const size_t alloc = sf_alloc_bytes(n, k) / 4;
  const int bands = (n + 127) / 128, t_sp = k / 128, t_d = k / 64;  // 512-byte scale tiles per band
  const size_t worker = (size_t)blockIdx.x * blockDim.x + threadIdx.x, workers = (size_t)gridDim.x * blockDim.x;
  uint32_t *w_sp = reinterpret_cast<uint32_t *>(sf_sparse), *w_d = reinterpret_cast<uint32_t *>(sf_dense);
  for (size_t i = (size_t)bands * t_sp * 128 + worker; i < alloc; i += workers) w_sp[i] = 0u;
  for (size_t i = (size_t)bands * t_d * 128 + worker; i < alloc; i += workers) w_d[i] = 0u;
  const size_t pad = (size_t)(bands * 128 - n);
  for (size_t i = worker; i < pad * t_sp; i += workers) w_sp[sf_offset(n + (int)(i / t_sp), 4 * (int)(i % t_sp), k / 32) / 4] = 0u;
  for (size_t i = worker; i < pad * t_d; i += workers) w_d[sf_offset(n + (int)(i / t_d), 4 * (int)(i % t_d), k / 16) / 4] = 0u;
}

// kShared: 32 elements per thread, scale of 32, both scale views.  Else 16 elements per thread.
// The groups of a row are a multiple of 4, so four neighbouring lanes' scale bytes form a 32-bit word of
// the blocked layout: gathered by shuffles and stored once.
template <bool kShared>
__global__ void __launch_bounds__(kScaledThreads, kShared ? 4 : 6) scaled_quantize_kernel(const uint4 *x, int rows, int k, const float *partials,
                                                                         int n_partials, uint8_t *q, uint8_t *sf, uint8_t *sf2,
                                                                         float *scale_out) {
  constexpr int kVecs = kShared ? 4 : 2;  // 16-byte vectors of a group
  __shared__ float warp_max[kScaledThreads / 32];
  ptx::grid_launch_dependents();
  ptx::grid_dependency_wait();
  if (kShared) zero_scale_padding(rows, k, sf, sf2);
  float mx = 0.0f;
  for (int i = threadIdx.x; i < n_partials; i += kScaledThreads) {
    const float p = partials[i];
    mx = (mx != mx || p != p) ? __int_as_float(0x7fffffff) : fmaxf(mx, p);
  }
  const float amax = block_max_nan(mx, warp_max);
  // ATen divides by a host scalar by multiplying with its float reciprocal; clamp keeps a NaN
  const float raw = __fmul_rn(amax, 1.0f / 2688.0f);
  const float scale = raw != raw ? raw : fmaxf(raw, 1.0e-9f);
  if (blockIdx.x == 0 && threadIdx.x == 0) *scale_out = scale;
  const float recip = __frcp_rn(__bfloat162float(__float2bfloat16_rn(scale)));

  const int groups = k / (8 * kVecs);
  const long long total = (long long)rows * groups;
  const long long chunks = (total + kScaledThreads - 1) / kScaledThreads;
  for (long long c = chunks - 1 - blockIdx.x; c >= 0; c -= gridDim.x) {
    const long long idx = c * kScaledThreads + threadIdx.x;
    const bool live = idx < total;
    // a 32-bit division where it will do: the 64-bit one costs a third of the group's instructions
    int row = 0;
    if (live) row = total <= 0xffffffffLL ? (int)((uint32_t)idx / (uint32_t)groups) : (int)(idx / groups);
    const int g = live ? (int)(idx - (long long)row * groups) : 0;
    uint32_t code = 0;
    if (live) {
      uint32_t w[4 * kVecs];
#pragma unroll
      for (int j = 0; j < kVecs; ++j) {
        const uint4 t = x[idx * kVecs + j];
        w[4 * j] = t.x, w[4 * j + 1] = t.y, w[4 * j + 2] = t.z, w[4 * j + 3] = t.w;
      }
      float gm = 0.0f;
      const uint64_t recip2 = prep::pair_f32(recip, recip);
#pragma unroll
      for (int i = 0; i < 4 * kVecs; ++i) {
        const float2 y = prep::unpair_f32(prep::mul_f32x2(prep::pair_f32(prep::lo_f(w[i]), prep::hi_f(w[i])), recip2));
        w[i] = prep::pack_bf16x2(y.x, y.y);
        gm = prep::max3(gm, fabsf(prep::lo_f(w[i])), fabsf(prep::hi_f(w[i])));
      }
      code = prep::scale_code_from_max(gm);
      const float inv = __frcp_rn(ue4m3_to_float(code));
      const uint64_t inv2 = prep::pair_f32(inv, inv);
      uint32_t o[kVecs];
#pragma unroll
      for (int j = 0; j < kVecs; ++j) {
        float2 t[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          t[i] = prep::unpair_f32(prep::mul_f32x2(prep::pair_f32(prep::lo_f(w[4 * j + i]), prep::hi_f(w[4 * j + i])), inv2));
        o[j] = pack_e2m1x8(t[0].x, t[0].y, t[1].x, t[1].y, t[2].x, t[2].y, t[3].x, t[3].y);
      }
      uint8_t *dst = q + (size_t)idx * (4 * kVecs);
      if (kShared)
        *reinterpret_cast<uint4 *>(dst) = make_uint4(o[0], o[1], o[2], o[kVecs - 1]);
      else
        *reinterpret_cast<uint2 *>(dst) = make_uint2(o[0], o[1]);
    }
    const uint32_t s1 = __shfl_down_sync(0xffffffffu, code, 1);
    const uint32_t s2 = __shfl_down_sync(0xffffffffu, code, 2);
    const uint32_t s3 = __shfl_down_sync(0xffffffffu, code, 3);
    if (live && (g & 3) == 0)
      *reinterpret_cast<uint32_t *>(sf + sf_offset(row, g, groups)) = code | (s1 << 8) | (s2 << 16) | (s3 << 24);
    if (kShared && live && (g & 1) == 0)  // the two 16-group slots of a 32-group are neighbours
      *reinterpret_cast<uint32_t *>(sf2 + sf_offset(row, 2 * g, k / 16)) = code * 0x101u | (s1 * 0x1010000u);
  }
}

inline unsigned blocks_for(long long items) { return (unsigned)((items + 255) / 256); }

}  // namespace

cudaError_t run_quantize_w32_shared(const void *w, int n, int k, void *qw, void *sf_sparse, void *sf_dense,
                                    cudaStream_t stream) {
  cudaError_t err = cudaMemsetAsync(sf_sparse, 0, sf_alloc_bytes(n, k), stream);
  if (err != cudaSuccess) return err;
  err = cudaMemsetAsync(sf_dense, 0, sf_alloc_bytes(n, k), stream);
  if (err != cudaSuccess) return err;
  quantize_w32_shared_kernel<<<blocks_for((long long)n * (k / 32)), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16 *>(w), n, k, static_cast<uint8_t *>(qw), static_cast<uint8_t *>(sf_sparse),
      static_cast<uint8_t *>(sf_dense));
  return cudaGetLastError();
}

cudaError_t run_duplicate_sf32_to_sf16(const void *sf32, int rows, int k, void *sf16, cudaStream_t stream) {
  cudaError_t err = cudaMemsetAsync(sf16, 0, sf_alloc_bytes(rows, k), stream);
  if (err != cudaSuccess) return err;
  duplicate_sf32_to_sf16_kernel<<<blocks_for((long long)rows * (k / 32)), 256, 0, stream>>>(
      static_cast<const uint8_t *>(sf32), rows, k, static_cast<uint8_t *>(sf16));
  return cudaGetLastError();
}

cudaError_t run_quantize_dense_nvfp4(const void *x, int rows, int k, void *q, void *sf, cudaStream_t stream) {
  quantize_dense_nvfp4_kernel<<<blocks_for((long long)rows * (k / 16)), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16 *>(x), rows, k, static_cast<uint8_t *>(q), static_cast<uint8_t *>(sf));
  return cudaGetLastError();
}

cudaError_t run_scaled_quantize(const void *x, int rows, int k, bool shared, float *partials, void *q, void *sf, void *sf2,
                                float *scale_out, cudaStream_t stream) {
  int dev = 0, sms = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  if ((err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return err;
  const size_t n16 = (size_t)rows * k / 8;
  // four 16-byte loads in flight per thread, six CTAs per SM
  size_t parts = (n16 + 4 * kScaledThreads - 1) / (4 * kScaledThreads);
  const size_t cap = (size_t)6 * sms < (size_t)kScaledQuantPartials ? (size_t)6 * sms : (size_t)kScaledQuantPartials;
  if (parts > cap) parts = cap;
  // both launches may start while the kernel before them drains
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3((unsigned)parts);
  cfg.blockDim = dim3(kScaledThreads);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const auto *xv = static_cast<const uint4 *>(x);
  if ((err = cudaLaunchKernelEx(&cfg, absmax_partials_kernel, xv, n16, partials)) != cudaSuccess) return err;
  const long long chunks = ((long long)rows * (k / (shared ? 32 : 16)) + kScaledThreads - 1) / kScaledThreads;
  const long long full = (shared ? 4LL : 6LL) * sms;  // the CTAs that are resident at once
  cfg.gridDim = dim3((unsigned)(chunks < full ? chunks : full));
  return cudaLaunchKernelEx(&cfg, shared ? scaled_quantize_kernel<true> : scaled_quantize_kernel<false>, xv, rows, k,
                            static_cast<const float *>(partials), (int)parts, static_cast<uint8_t *>(q),
                            static_cast<uint8_t *>(sf), static_cast<uint8_t *>(sf2), scale_out);
}

cudaError_t run_compress_sparse_a(const void *a_dense, int m, int k, void *a_comp, void *e, cudaStream_t stream) {
  cudaError_t err = cudaMemsetAsync(a_comp, 0, a_comp_bytes(m, k), stream);
  if (err != cudaSuccess) return err;
  err = cudaMemsetAsync(e, 0, e_bytes(m, k), stream);
  if (err != cudaSuccess) return err;
  compress_sparse_a_kernel<<<blocks_for((long long)m * (k / 32)), 256, 0, stream>>>(
      static_cast<const uint8_t *>(a_dense), m, k, static_cast<uint8_t *>(a_comp), static_cast<uint8_t *>(e));
  return cudaGetLastError();
}

}  // namespace sharq

// Activation prepare kernels for sm_100a: row statistics, and the fused
// [RMSNorm ->] tensor-scale -> pair-wise 4:8 sparse main path + dense NVFP4 residual.
//
// Replaces, behind the same buffer formats, the reference's
//   kernels/src/fused_sparse_prepare.cu:89-251          (prepare of a pre-scaled input)
//   kernels/src/fused_rmsnorm_sparse_prepare.cu:85-325  (row stats + RMSNorm-fused prepare)
//   kernels/src/bindings.cpp:270-274,320-326,337        (zero fills and the tensor-scale glue)
// and the host-side amax / divide passes of model/quantize.py:179-183.
//
// Work split of the prepare kernel: one thread owns one 32-element group (one sparse scale,
// two residual scales).  A warp covers 4 rows x 8 groups = 4 rows x 256 columns, which makes
// its metadata (4 rows x 16 B) and its packed outputs contiguous per row; a CTA of 8 warps
// covers 32 rows x 256 columns.  Every byte of every output buffer is written by the kernel
// (payload by its owner thread, padding rows/columns and the spare tail of each buffer with
// zeros), so callers may hand in uninitialised memory.
//
// The kernel is instruction-bound, so the arithmetic is arranged to need few instructions
// while producing exactly the reference's bits:
//   * pair selection on integer keys: the pair score max(|a|,|b|) of two bf16-exact values
//     has 16 zero low bits as a float, so `bits | (3 - pair)` is a key whose integer order is
//     "larger score first, earlier pair first" - the reference's strict-'>' scan order;
//   * scale value and reciprocal of the 126 possible UE4M3 codes come from a shared-memory
//     table filled with ue4m3 -> float and the IEEE reciprocal;
//   * e2m1 encode/decode use the hardware conversions; x - q*s is one FMA (q*s is exact);
//   * products and the FMA on packed pairs (mul / fma.rn.f32x2), max / 6 as a product, maxima of three, the tile walk
//     without divisions: 16384 x 18944 with known absmax 285 -> 227 us (2.9 B per element: 4.0 TB/s), 2048 x 14336
//     31.7 -> 25.7 us, an already scaled 16384 x 4096 49.1 -> 41.2 us;
//   * x / scale (tensor scale) is y * (1/scale) when that product is provably on the same side
//     of every bf16 rounding boundary as the IEEE quotient, and an IEEE division otherwise.
#include "common.cuh"
#include "prepare.cuh"
#include "prepare_device.cuh"
#include "sm100_ptx.cuh"

#include <cstdlib>

namespace sharq {

using namespace prep;

namespace {

constexpr int kRowsPerWarp = 4;
constexpr int kGroupsPerWarp = 8;
constexpr int kWarpsPerCta = 8;
constexpr int kRowsPerCta = kRowsPerWarp * kWarpsPerCta;  // 32
constexpr int kColsPerCta = kGroupsPerWarp * 32;          // 256
constexpr int kPrepareThreads = 32 * kWarpsPerCta;

// Raise the tensor absmax (non-negative float bits, integer order = float order).  The read
// first keeps the number of same-address atomics small once the maximum has settled.
__device__ __forceinline__ void raise_amax(unsigned int *amax_bits, float mx) {
  const unsigned int bits = __float_as_uint(mx);
  if (bits > *reinterpret_cast<volatile unsigned int *>(amax_bits)) atomicMax(amax_bits, bits);
}

// The maximum of a CTA: into the CTA's own word (nothing has to be zeroed before the launch) or raised into the first.
__device__ __forceinline__ void publish_amax(unsigned int *amax_bits, float mx, bool word_per_cta) {
  if (word_per_cta)
    amax_bits[blockIdx.x] = __float_as_uint(mx);
  else
    raise_amax(amax_bits, mx);
}

// ---------------------------------------------------------------------------
// Row statistics for the RMSNorm path, one CTA per row, one thread per 32-element group:
//   inv_rms[r] = rsqrtf(sum(x^2)/K + eps) with the reference's summation order (each group
//   left to right - an FMA chain whose products are exact - then the group sums left to
//   right by one thread), and the tensor-wide max of |bf16(x * inv_rms * gamma)|.
// Many rows are resident per SM, so the serial sums of different rows overlap.
// ---------------------------------------------------------------------------
// With kAdd the row is first formed as bf16(x + residual) (the decoder's residual add, rounded
// like the ATen add), stored to sum_out, and the statistics are those of the sum.
template <bool kAdd>
__global__ void __launch_bounds__(1024, 2) rms_stats_kernel(const __nv_bfloat16 *x, const __nv_bfloat16 *residual,
                                                          __nv_bfloat16 *sum_out, const __nv_bfloat16 *gamma, float eps, int k,
                                                          float *inv_rms, unsigned int *amax_bits, bool word_per_cta) {
  ptx::grid_launch_dependents();
  ptx::grid_dependency_wait();
  extern __shared__ float partial[];  // [k/32] group sums, then [0] is reused for inv_rms
  __shared__ float warp_max[32];
  const int groups = k >> 5;
  const int g = threadIdx.x;
  const int row = blockIdx.x;
  const bool live = g < groups;
  uint32_t w[16];
  if (live) {
    const uint4 *src = reinterpret_cast<const uint4 *>(x + (size_t)row * k + (size_t)g * 32);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint4 v = src[j];
      w[4 * j + 0] = v.x;
      w[4 * j + 1] = v.y;
      w[4 * j + 2] = v.z;
      w[4 * j + 3] = v.w;
    }
    if (kAdd) {
      const uint4 *rsrc = reinterpret_cast<const uint4 *>(residual + (size_t)row * k + (size_t)g * 32);
      uint4 *dst = reinterpret_cast<uint4 *>(sum_out + (size_t)row * k + (size_t)g * 32);
      uint4 r[4];  // all loads ahead of the first store, which they may not pass
#pragma unroll
      for (int j = 0; j < 4; ++j) r[j] = rsrc[j];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t rw[4] = {r[j].x, r[j].y, r[j].z, r[j].w};
#pragma unroll
        for (int t = 0; t < 4; ++t)
          w[4 * j + t] = pack_bf16x2(__fadd_rn(lo_f(w[4 * j + t]), lo_f(rw[t])), __fadd_rn(hi_f(w[4 * j + t]), hi_f(rw[t])));
        dst[j] = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
      }
    }
    float s = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float a = lo_f(w[i]), b = hi_f(w[i]);
      s = __fmaf_rn(a, a, s);  // a*a is exact in float, so this equals s + a*a
      s = __fmaf_rn(b, b, s);
    }
    partial[g] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float total = 0.0f;
#pragma unroll 8
    for (int i = 0; i < groups; i += 4) {  // groups is a multiple of 4 (K % 128 == 0); the loads run ahead of the chain
      float4 v = *reinterpret_cast<const float4 *>(partial + i);
      total = __fadd_rn(total, v.x);
      total = __fadd_rn(total, v.y);
      total = __fadd_rn(total, v.z);
      total = __fadd_rn(total, v.w);
    }
    float inv = rsqrtf(__fadd_rn(__fdiv_rn(total, (float)k), eps));
    inv_rms[row] = inv;
    warp_max[31] = inv;  // slot 31 is free: at most 32 warps, reduction uses [0, nwarps)
  }
  __syncthreads();
  const float inv = warp_max[31];
  __syncthreads();
  float mx = 0.0f;
  if (live) {
    const uint4 *gsrc = reinterpret_cast<const uint4 *>(gamma + (size_t)g * 32);
    __nv_bfloat162 m2 = __floats2bfloat162_rn(0.0f, 0.0f);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint4 gv = gsrc[j];
      uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w};
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        float a = __fmul_rn(__fmul_rn(lo_f(w[4 * j + t]), inv), lo_f(gw[t]));
        float b = __fmul_rn(__fmul_rn(hi_f(w[4 * j + t]), inv), hi_f(gw[t]));
        m2 = __hmax2(m2, __habs2(__floats2bfloat162_rn(a, b)));
      }
    }
    mx = fmaxf(__bfloat162float(m2.x), __bfloat162float(m2.y));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = (blockDim.x + 31) >> 5;
  if (lane == 0) warp_max[warp] = mx;
  __syncthreads();
  if (warp == 0) {
    mx = lane < nwarps ? warp_max[lane] : 0.0f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) publish_amax(amax_bits, mx, word_per_cta);
  }
}

// Tensor-wide max |x| of a bf16 tensor (non-RMSNorm path): flat grid-stride reduction.
__global__ void __launch_bounds__(256) abs_stats_kernel(const __nv_bfloat16 *x, size_t n16, unsigned int *amax_bits,
                                                         bool word_per_cta) {
  ptx::grid_launch_dependents();
  ptx::grid_dependency_wait();
  __shared__ float warp_max[8];
  __nv_bfloat162 m2 = __floats2bfloat162_rn(0.0f, 0.0f);
  const uint4 *src = reinterpret_cast<const uint4 *>(x);
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += 4 * stride) {
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = (i + u * stride < n16) ? src[i + u * stride] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      m2 = __hmax2(m2, __habs2(*reinterpret_cast<__nv_bfloat162 *>(&v[u].x)));
      m2 = __hmax2(m2, __habs2(*reinterpret_cast<__nv_bfloat162 *>(&v[u].y)));
      m2 = __hmax2(m2, __habs2(*reinterpret_cast<__nv_bfloat162 *>(&v[u].z)));
      m2 = __hmax2(m2, __habs2(*reinterpret_cast<__nv_bfloat162 *>(&v[u].w)));
    }
  }
  float mx = fmaxf(__bfloat162float(m2.x), __bfloat162float(m2.y));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) warp_max[warp] = mx;
  __syncthreads();
  if (warp == 0) {
    mx = lane < 8 ? warp_max[lane] : 0.0f;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) publish_amax(amax_bits, mx, word_per_cta);
  }
}

// Zeros in the padding rows [m, ceil128(m)) of the metadata and of both scale buffers.
__device__ __forceinline__ void zero_padding_rows(uint8_t *e, uint8_t *sfa_sparse, uint8_t *sf_res, int m, int k, int worker, int workers) {
  const int groups32 = k >> 5, aligned_m = (m + 127) / 128 * 128;
  const int pad_rows = aligned_m - m;
  const int k_tiles = (k + 255) / 256;
  const int w_sp = groups32 >> 2, w_res = k >> 6;  // 32-bit scale words per row
  const int per_row = k_tiles * 4 + w_sp + w_res;  // 32-bit words to clear per padding row
  for (int i = worker; i < pad_rows * per_row; i += workers) {
    const int row = m + i / per_row;
    int j = i % per_row;
    if (j < k_tiles * 4) {
      *reinterpret_cast<uint32_t *>(e + ((size_t)(j >> 2) * aligned_m + row) * 16 + (size_t)(j & 3) * 4) = 0u;
    } else if ((j -= k_tiles * 4) < w_sp) {
      *reinterpret_cast<uint32_t *>(sfa_sparse + sf_offset(row, 4 * j, groups32)) = 0u;
    } else {
      j -= w_sp;
      *reinterpret_cast<uint32_t *>(sf_res + sf_offset(row, 4 * j, k / 16)) = 0u;
    }
  }
}

// ---------------------------------------------------------------------------
// Prepare kernel.
//   kMode 0: input already scaled (drop-in for fused_sparse_residual_quantize_x)
//   kMode 1: RMSNorm + tensor scale inline (needs inv_rms and the tensor absmax)
//   kMode 2: tensor scale inline only (x / scale rounded to bf16), scale from absmax
// Persistent: a fixed number of CTAs per SM loops over 32-row x 256-column tiles (rows up to
// ceil128(M)); every CTA first helps zero the spare tail of each buffer.
// ---------------------------------------------------------------------------
struct PrepareParams {
  const __nv_bfloat16 *x;
  const __nv_bfloat16 *gamma;
  const float *inv_rms;
  const unsigned int *amax_bits;
  unsigned int *amax_out;  // optional: the bits of the maximum
  int amax_words;    // one tensor: the maximum is the largest of that many words
  float *scale_out;  // optional, written by one thread (modes 1, 2)
  uint8_t *a_comp;
  uint8_t *e;
  uint8_t *q_sparse_dense;  // debug only
  uint8_t *sfa_sparse;
  uint8_t *q_res;
  uint8_t *sf_res;
  int m, k;
  int row_tiles;  // ceil128(m) / 32
  // grouped activation of a mixture-of-experts layer (mode 2, absmax ready): rows sorted by group in
  // 256-row units; unit_group[u] < 0 = unit without rows; amax_bits and scale_vec_out have `groups` entries
  const int *unit_group;
  float *scale_vec_out;
  int groups;
  const int *src_row;  // optional gather: output row r is prepared from input row src_row[r] (< 0: a padding row of zeros)
};

constexpr int kPrepareCtasPerSm = 3;
constexpr int kScaledCtasPerSm = 2;  // tensor-scale mode without a gather
// A tensor-scale input of up to kClusterScanElements needs no statistics launch: every CTA scans it for its maximum, or (from kCtaScanElements)
// every cluster of kScanCtas CTAs.  A prepare is followed by its GEMM, and what counts is the pair: us of both in a graph (o_proj of 4096
// columns behind it), clusters / statistics launch: 12 x 4096 9.9 / 10.4, 32 x 4096 11.9 / 11.8, 40 x 4096 12.5 / 12.2, 64 x 4096 13.6 / 14.5, 16 x 8192 12.1 / 13.0,
// 16 x 14336 15.5 / 16.1.  The prepare by itself behind a memset is slower from about 16 x 4096 on (16 x 14336 5.9 / 5.3).  A launch less is also 2 us
// less on the host (16 x 14336 and its GEMM, eager: 21.4 -> 19.2).  CTA / cluster by themselves: 8 x 4096 3.1 / 3.9, 16 x 4096 4.5 / 3.1.
constexpr size_t kCtaScanElements = 40 * 1024;
constexpr size_t kClusterScanElements = 256 * 1024;
constexpr int kClusterScanTiles = 256;  // CTAs that leave room for every cluster at once (8 x 18944, 296 of them: with its GEMM 19.2, launch 17.5)
constexpr int kScanCtas = 8;
// The scanning forms leave the maximum in the workspace only above these sizes (with and without room for a word per statistics CTA); up to
// the second one an input is scanned in any case where there is no such room.
constexpr size_t kInlineAbsmaxElements = 64 * 1024;
constexpr size_t kInlineAbsmaxElementsNoWords = 192 * 1024;
// Behind a statistics launch of its own and with more than one 32-row tile a lane takes 8 elements (prepare_narrow_kernel): RMSNorm up to
// kNarrowElements, tensor scale while its CTAs are at most one per SM.  us of the calls and their GEMM (4096 columns) in a graph, wide / narrow: RMSNorm
// 33 x 4096 14.4 / 13.8, 64 x 4096 15.4 / 15.2, 128 x 4096 17.3 / 16.7, 200 x 4096 17.9 / 17.9, 256 x 4096 18.3 / 18.8; tensor scale 72 x 4096 (144 CTAs) 15.4 / 13.9,
// 80 x 4096 (160) 15.8 / 17.9, 36 x 8192 (144) 15.5 / 13.9, 40 x 8192 (160) 15.6 / 17.5, 512 x 1152 (320) 12.6 / 14.9.  With a maximum that another kernel left
// (SwiGLU) 48 x 4096 14.6 / 13.1, but 72 x 4096 16.5 / 18.7, 128 x 1152 11.2 / 15.1 and 48 x 14336 19.6 / 20.2, and for an input that needs none 64 x 4096 11.1 / 12.7:
// these two keep the wide form.  Up to 32 rows the narrow one is faster by itself (RMSNorm 32 x 4096 6.1 / 5.1) but not between GEMMs: linears of a
// Llama-3-8B layer with 8 / 32 tokens wide 72.4 / 78.4, narrow 77.2 / 80.9.
constexpr size_t kNarrowElements = 640 * 1024;
constexpr unsigned kMaxAbsmaxWords = 4096;            // words of CTA maxima that every prepare CTA reduces

// kCtas: resident CTAs per SM the register allocation aims at.  The tensor-scale mode runs
// fastest with two (no spills) except on a gathered activation (src_row), where the third CTA
// hides more of the gather's latency (measured: 2048 x 14336 43.3 -> 41.1 us with two,
// 34816 x 4096 grouped 253 -> 264 us).
// kCluster (mode 2): a small input without a statistics launch: the CTAs of a cluster of kScanCtas CTAs look for the maximum of the whole input
// together, each over its share, and exchange what they found through distributed shared memory.
template <int kMode, bool kDebug, int kCtas = kPrepareCtasPerSm, bool kCluster = false>
__global__ void __launch_bounds__(kPrepareThreads, kCtas) prepare_kernel(const PrepareParams p) {
  const int m = p.m, k = p.k;
  const int groups32 = k >> 5;
  const int aligned_m = (m + 127) / 128 * 128;

  ptx::grid_launch_dependents();
  __shared__ ScaleTables tbl;
  extern __shared__ uint4 gamma_smem[];  // mode 1: the whole RMSNorm weight, k bf16
  if (threadIdx.x < 128) {
    const float v = ue4m3_to_float(threadIdx.x);
    tbl.value[threadIdx.x] = v;
    tbl.recip[threadIdx.x] = __frcp_rn(v);  // code 0 is never looked up (scales are clamped to >= 2^-9)
  }
  __shared__ float scan_max[kScanCtas];  // kCluster
  if (kCluster) ptx::cluster_arrive();
  ptx::grid_dependency_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k_tiles = (k + kColsPerCta - 1) / kColsPerCta;
  const int total_tiles = k_tiles * p.row_tiles;
  const int row_in_tile = warp * kRowsPerWarp + (lane >> 3);
  const int group_in_tile = lane & 7;

  // persistent loop over 32-row x 256-column tiles; the next tile's 64 bytes are loaded
  // before the current tile is processed, so the loads overlap the arithmetic
  uint4 next[4];
  float next_inv = 0.0f;
  bool next_row_ok = true;
  auto issue_loads = [&](int row_tile, int k_tile) {
    const int row = row_tile * kRowsPerCta + row_in_tile;
    const int group = k_tile * kGroupsPerWarp + group_in_tile;
    if (row < m && group < groups32) {
      int in_row = row;
      if (kMode == 2 && p.src_row != nullptr) in_row = p.src_row[row];
      next_row_ok = in_row >= 0;
      if (in_row >= 0) {
        const uint4 *src = reinterpret_cast<const uint4 *>(p.x + (size_t)in_row * k + (size_t)group * 32);
#pragma unroll
        for (int j = 0; j < 4; ++j) next[j] = src[j];
      }
      if (kMode == 1) next_inv = p.inv_rms[row];
    }
  };
  // the tile walk and the scale offsets are advanced instead of divided out per tile (the divisions were a
  // tenth of the instructions)
  const int step_rows = (int)gridDim.x / k_tiles, step_k = (int)gridDim.x % k_tiles;
  int next_row_tile = (int)blockIdx.x / k_tiles, next_k_tile = (int)blockIdx.x % k_tiles;
  // scale offset of (row, group): 512-byte tiles of 128 rows x 4 groups, see sf_offset
  const uint32_t sf_lane = (uint32_t)row_in_tile * 16u;  // row % 32 is row_in_tile
  const size_t band_sp = (size_t)(groups32 >> 2) * 512, band_res = (size_t)(k >> 6) * 512;
  issue_loads(next_row_tile, next_k_tile);

  // What the CTA needs first is loaded together, with one barrier behind it: its first tile (above), its words of the maximum, its
  // RMSNorm weight.  One after the other they were three latencies of a launch that lasts about four on a decode step (RMSNorm 32 x 4096
  // with its statistics 6.6 -> 6.1 us, 1 x 4096 with its scan 3.0 -> 2.6).
  float amax = 0.0f;
  if (kMode == 2 && p.amax_bits == nullptr) {
    // Small input (a decode step): every CTA, or every cluster, finds max|x| of the whole tensor itself, which
    // replaces the statistics launch; the tensor is read from L2.
    const uint4 *all = reinterpret_cast<const uint4 *>(p.x);
    const int n16 = m * (k / 8);
    __nv_bfloat162 m2 = __floats2bfloat162_rn(0.0f, 0.0f);
    const int share = kCluster ? (int)ptx::cluster_ctarank() : 0, shares = kCluster ? kScanCtas : 1;
    for (int i = share * kPrepareThreads + (int)threadIdx.x; i < n16; i += shares * kPrepareThreads) {
      const uint4 v = all[i];
      m2 = __hmax2(m2, __habs2(*reinterpret_cast<const __nv_bfloat162 *>(&v.x)));
      m2 = __hmax2(m2, __habs2(*reinterpret_cast<const __nv_bfloat162 *>(&v.y)));
      m2 = __hmax2(m2, __habs2(*reinterpret_cast<const __nv_bfloat162 *>(&v.z)));
      m2 = __hmax2(m2, __habs2(*reinterpret_cast<const __nv_bfloat162 *>(&v.w)));
    }
    amax = fmaxf(__bfloat162float(m2.x), __bfloat162float(m2.y));
  } else if (kMode != 0) {
    amax = __uint_as_float(*p.amax_bits);
    for (int i = threadIdx.x; i < p.amax_words; i += kPrepareThreads) amax = fmaxf(amax, __uint_as_float(p.amax_bits[i]));
  }
  if (kMode == 1) {
    // the columns this CTA will meet: those of its one tile, or all
    const bool one_tile = total_tiles <= (int)gridDim.x;
    const int lo = one_tile ? next_k_tile * (kColsPerCta / 8) : 0, hi = one_tile ? min(k / 8, lo + kColsPerCta / 8) : k / 8;
    const uint4 *gsrc = reinterpret_cast<const uint4 *>(p.gamma);
    for (int i = lo + (int)threadIdx.x; i < hi; i += blockDim.x) gamma_smem[i] = gsrc[i];
  }

  // zero what no owner thread writes: the spare tail of the scale buffers and of A_comp
  {
    const int worker = blockIdx.x * blockDim.x + threadIdx.x;
    const int workers = gridDim.x * blockDim.x;
    const size_t bands = (size_t)aligned_m / 128;
    zero_range(p.sfa_sparse, bands * (size_t)(groups32 / 4) * 512, sf_alloc_bytes(m, k), worker, workers);
    zero_range(p.sf_res, bands * (size_t)(k / 16 / 4) * 512, sf_alloc_bytes(m, k), worker, workers);
    if (!kDebug) zero_range(p.a_comp, (size_t)m * (k / 4), a_comp_bytes(m, k), worker, workers);
  }

  __shared__ float part_max[kWarpsPerCta];
  if (kMode != 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (lane == 0) part_max[warp] = amax;
  }
  __syncthreads();
  float scale = 1.0f, recip = 1.0f;
  if (kMode != 0) {
#pragma unroll
    for (int w = 0; w < kWarpsPerCta; ++w) amax = fmaxf(amax, part_max[w]);
    if (kCluster) {
      ptx::cluster_wait();  // the CTAs of the cluster are running
      if (threadIdx.x < kScanCtas) ptx::st_cluster_f32(&scan_max[ptx::cluster_ctarank()], threadIdx.x, amax);
      __syncwarp();
      ptx::cluster_sync();  // behind it no CTA writes to another
#pragma unroll
      for (int c = 0; c < kScanCtas; ++c) amax = fmaxf(amax, scan_max[c]);
    }
    // ATen divides a CUDA tensor by a host scalar by multiplying with the float
    // reciprocal; clamp(min=1e-9) follows (kernels/src/bindings.cpp:337 of the reference).
    scale = fmaxf(__fmul_rn(amax, 1.0f / 2688.0f), 1.0e-9f);
    if (p.scale_out != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *p.scale_out = scale;
    if (p.amax_out != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *p.amax_out = __float_as_uint(amax);
    if (kMode == 2 && p.unit_group != nullptr && blockIdx.x == 0 && (int)threadIdx.x < p.groups)
      p.scale_vec_out[threadIdx.x] = fmaxf(__fmul_rn(__uint_as_float(p.amax_bits[threadIdx.x]), 1.0f / 2688.0f), 1.0e-9f);
    if (kMode == 2) scale = round_to_bf16(scale);  // the divisor of the non-RMSNorm path, see round_to_bf16
    recip = __frcp_rn(scale);
  }

  for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x) {
    const int row_tile = next_row_tile, k_tile = next_k_tile;
    next_row_tile += step_rows;
    next_k_tile += step_k;
    if (next_k_tile >= k_tiles) {
      next_k_tile -= k_tiles;
      ++next_row_tile;
    }
    const int row = row_tile * kRowsPerCta + row_in_tile;
    const int group = k_tile * kGroupsPerWarp + group_in_tile;
    const bool col_ok = group < groups32;
    bool live = row < m && col_ok;
    float t_scale = scale, t_recip = recip;
    if (kMode == 2 && p.unit_group != nullptr) {  // per-group tensor scale; a 32-row tile lies inside one 256-row unit
      const int grp = p.unit_group[(row_tile * kRowsPerCta) >> 8];
      live = live && grp >= 0;
      t_scale = round_to_bf16(fmaxf(__fmul_rn(__uint_as_float(p.amax_bits[grp < 0 ? 0 : grp]), 1.0f / 2688.0f), 1.0e-9f));
      t_recip = __frcp_rn(t_scale);
    }

    uint32_t xw[16];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      xw[4 * j + 0] = next[j].x;
      xw[4 * j + 1] = next[j].y;
      xw[4 * j + 2] = next[j].z;
      xw[4 * j + 3] = next[j].w;
    }
    const float inv = next_inv;
    live = live && next_row_ok;
    issue_loads(next_row_tile, next_k_tile);

    GroupOut o;
    o.a_comp[0] = o.a_comp[1] = 0;
    o.meta = 0;
    o.sf_sparse = 0;
    o.sf_res = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) o.q_res[i] = o.q_sparse[i] = 0;

    if (live) {
      if (kMode == 1) {
        const uint4 *gsrc = gamma_smem + (size_t)group * 4;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4 gv = gsrc[j];
          uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w};
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            xw[4 * j + t] = normalise_word(xw[4 * j + t], gw[t], pair_f32(inv, inv));
          }
        }
      }
      scale_quantize_group<kMode, kDebug>(xw, t_scale, t_recip, tbl, o, [&](uint32_t (&w)[16]) {
        // mode 2, rare: the group is read again for the division form
        const int in_row = p.src_row != nullptr ? p.src_row[row] : row;
        const uint4 *src = reinterpret_cast<const uint4 *>(p.x + (size_t)in_row * k + (size_t)group * 32);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 v = src[j];
          w[4 * j + 0] = v.x;
          w[4 * j + 1] = v.y;
          w[4 * j + 2] = v.z;
          w[4 * j + 3] = v.w;
        }
      });

      uint4 q = make_uint4(o.q_res[0], o.q_res[1], o.q_res[2], o.q_res[3]);
      *reinterpret_cast<uint4 *>(p.q_res + (size_t)row * (k / 2) + (size_t)group * 16) = q;
      if (kDebug) {
        uint4 qs = make_uint4(o.q_sparse[0], o.q_sparse[1], o.q_sparse[2], o.q_sparse[3]);
        *reinterpret_cast<uint4 *>(p.q_sparse_dense + (size_t)row * (k / 2) + (size_t)group * 16) = qs;
      } else {
        *reinterpret_cast<uint2 *>(p.a_comp + (size_t)row * (k / 4) + (size_t)group * 8) = make_uint2(o.a_comp[0], o.a_comp[1]);
      }
    }
    // Metadata: rows up to ceil128(M), columns up to ceil256(K); dead lanes write zeros.
    // One warp writes 4 rows x 16 B = 64 contiguous bytes.
    if (!kDebug) {
      // combine the 16-bit metadata of two neighbouring groups into one 32-bit store
      uint32_t mine = o.meta & 0xFFFFu;
      uint32_t other = __shfl_down_sync(0xffffffffu, mine, 1);
      if ((lane & 1) == 0) {
        uint8_t *dst = p.e + (size_t)k_tile * aligned_m * 16 + (size_t)row * 16 + (size_t)group_in_tile * 2;
        *reinterpret_cast<uint32_t *>(dst) = mine | (other << 16);
      }
    }
    // Scale factors: 4 neighbouring groups share one 32-bit word of the sparse layout,
    // 2 neighbouring groups (4 residual scales) one word of the dense layout.
    {
      uint32_t sv = o.sf_sparse;
      uint32_t s1 = __shfl_down_sync(0xffffffffu, sv, 1);
      uint32_t s2 = __shfl_down_sync(0xffffffffu, sv, 2);
      uint32_t s3 = __shfl_down_sync(0xffffffffu, sv, 3);
      uint32_t r2 = o.sf_res;
      uint32_t r2n = __shfl_down_sync(0xffffffffu, r2, 1);
      if (col_ok) {
        const uint32_t at = sf_lane + (uint32_t)(row_tile & 3) * 4u;
        if ((lane & 3) == 0)
          *reinterpret_cast<uint32_t *>(p.sfa_sparse + (size_t)(row_tile >> 2) * band_sp + (uint32_t)(group >> 2) * 512u + at) =
              sv | (s1 << 8) | (s2 << 16) | (s3 << 24);
        if ((lane & 1) == 0)
          *reinterpret_cast<uint32_t *>(p.sf_res + (size_t)(row_tile >> 2) * band_res + (uint32_t)(group >> 1) * 512u + at +
                                        (uint32_t)(group & 1) * 2u) = r2 | (r2n << 16);
      }
    }
  }
}


// ---------------------------------------------------------------------------
// Prepare of a small input: latency is all there is, and one group per lane makes a serial chain of some 700 instructions that eight
// warps of a few SMs walk while the others idle.  Here a lane owns 8 elements, a warp 256 columns of one row, and a CTA has one task per
// warp (RMSNorm 48 x 4096 with its statistics 6.1 -> 5.3 us).  Modes 1 and 2 of prepare_kernel, the maximum ready; same bytes.
// ---------------------------------------------------------------------------
// Warps of a CTA: the tensor-scale mode has up to 8 maxima per SM to reduce in every CTA, the RMSNorm mode one per row.  us with 4 / 8
// warps: 96 x 4096 5.3 / 4.4, 32 x 14336 6.0 / 4.7 (tensor scale).
__host__ __device__ constexpr int narrow_warps(int mode) { return mode == 2 ? 8 : 4; }

template <int kMode>
__global__ void __launch_bounds__(32 * narrow_warps(kMode)) prepare_narrow_kernel(const PrepareParams p) {
  constexpr int kNarrowWarps = narrow_warps(kMode);
  const int m = p.m, k = p.k, groups32 = k >> 5;
  const int aligned_m = (m + 127) / 128 * 128;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ptx::grid_launch_dependents();
  __shared__ ScaleTables tbl;
  __shared__ float part_max[kNarrowWarps];
  if (threadIdx.x < 128) {
    const float v = ue4m3_to_float(threadIdx.x);
    tbl.value[threadIdx.x] = v;
    tbl.recip[threadIdx.x] = __frcp_rn(v);  // code 0 is never looked up (scales are clamped to >= 2^-9)
  }
  ptx::grid_dependency_wait();

  const int k_tiles = (k + 255) / 256;
  const int task = (int)blockIdx.x * kNarrowWarps + warp;
  const int row = task / k_tiles, k_tile = task - row * k_tiles;
  const int col8 = k_tile * 32 + lane;  // in units of 8 columns
  const bool live = row < m && col8 < (k >> 3);
  uint4 v = make_uint4(0, 0, 0, 0), gv = make_uint4(0, 0, 0, 0);
  float inv = 0.0f;
  if (live) {
    v = reinterpret_cast<const uint4 *>(p.x)[(size_t)row * (k >> 3) + col8];
    if (kMode == 1) {
      gv = reinterpret_cast<const uint4 *>(p.gamma)[col8];
      inv = p.inv_rms[row];
    }
  }
  float amax = __uint_as_float(*p.amax_bits);
  for (int i = threadIdx.x; i < p.amax_words; i += 32 * kNarrowWarps) amax = fmaxf(amax, __uint_as_float(p.amax_bits[i]));
  {
    const int worker = (int)(blockIdx.x * blockDim.x + threadIdx.x), workers = (int)(gridDim.x * blockDim.x);
    const size_t bands = (size_t)aligned_m / 128;
    zero_range(p.sfa_sparse, bands * (size_t)(groups32 / 4) * 512, sf_alloc_bytes(m, k), worker, workers);
    zero_range(p.sf_res, bands * (size_t)(k / 16 / 4) * 512, sf_alloc_bytes(m, k), worker, workers);
    zero_range(p.a_comp, (size_t)m * (k / 4), a_comp_bytes(m, k), worker, workers);
    zero_padding_rows(p.e, p.sfa_sparse, p.sf_res, m, k, worker, workers);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if (lane == 0) part_max[warp] = amax;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kNarrowWarps; ++w) amax = fmaxf(amax, part_max[w]);
  float scale = fmaxf(__fmul_rn(amax, 1.0f / 2688.0f), 1.0e-9f);  // as in prepare_kernel
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (p.scale_out != nullptr) *p.scale_out = scale;
    if (p.amax_out != nullptr) *p.amax_out = __float_as_uint(amax);
  }
  if (kMode == 2) scale = round_to_bf16(scale);
  const float recip = __frcp_rn(scale);
  if (row >= m) return;

  uint32_t w[4] = {v.x, v.y, v.z, v.w};
  if (kMode == 1) {
    const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = normalise_word(w[i], gw[i], pair_f32(inv, inv));
    scale_words(w, scale, recip);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 q = mul_word(w[i], pair_f32(recip, recip));
      w[i] = pack_bf16x2(q.x, q.y);
    }
  }
  ChunkPick pick = pick_pairs(w);
  if (kMode == 2 && pick.second - 4u < kTinyKey) {  // rare, see scale_quantize_group: a subnormal quotient takes part in the selection
    const uint32_t x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = pack_bf16x2(__fdiv_rn(lo_f(x[i]), scale), __fdiv_rn(hi_f(x[i]), scale));
    pick = pick_pairs(w);
  }
  __syncwarp();
  ChunkOut o;
  quantize_chunk8(w, pick, tbl, o);
  if (!live) o = ChunkOut{};

  if (live) *reinterpret_cast<uint32_t *>(p.q_res + (size_t)row * (k / 2) + (size_t)col8 * 4) = o.q_res;
  const uint32_t comp = o.a_comp | (__shfl_down_sync(0xffffffffu, o.a_comp, 1) << 16);
  if (live && (lane & 1) == 0) *reinterpret_cast<uint32_t *>(p.a_comp + (size_t)row * (k / 4) + (size_t)col8 * 2) = comp;
  uint32_t meta = o.meta << (4 * (lane & 7));  // 8 lanes: the metadata of two groups
  meta |= __shfl_xor_sync(0xffffffffu, meta, 1);
  meta |= __shfl_xor_sync(0xffffffffu, meta, 2);
  meta |= __shfl_xor_sync(0xffffffffu, meta, 4);
  if ((lane & 7) == 0) *reinterpret_cast<uint32_t *>(p.e + ((size_t)k_tile * aligned_m + row) * 16 + (size_t)(lane >> 3) * 4) = meta;
  uint32_t res = o.sf_res << (8 * ((lane >> 1) & 3));  // 8 lanes: four 16-groups
  res |= __shfl_xor_sync(0xffffffffu, res, 2);
  res |= __shfl_xor_sync(0xffffffffu, res, 4);
  if (live && (lane & 7) == 0) *reinterpret_cast<uint32_t *>(p.sf_res + sf_offset(row, col8 >> 1, k / 16)) = res;
  uint32_t sp = o.sf_sparse << (8 * ((lane >> 2) & 3));  // 16 lanes: four 32-groups
  sp |= __shfl_xor_sync(0xffffffffu, sp, 4);
  sp |= __shfl_xor_sync(0xffffffffu, sp, 8);
  if (live && (lane & 15) == 0) *reinterpret_cast<uint32_t *>(p.sfa_sparse + sf_offset(row, col8 >> 2, groups32)) = sp;
}

// ---------------------------------------------------------------------------
// One-launch scaled prepare (modes 1 and 2 with their statistics pass folded in).
//
// A cooperative grid of one CTA per SM; CTA b owns a contiguous block of rows.  Phase 1: the
// CTA streams its rows through shared memory in chunks, computes the row statistics of the
// RMSNorm path in the reference's summation order (group sums as FMA chains, then left to
// right over the groups by one thread per row), replaces the cached rows by the normalised
// bf16 values and folds max|y| into the tensor absmax word.  All CTAs then meet at a
// grid-wide barrier (a counter in the caller's workspace, bounded spin), read the absmax and
// quantise: the last chunk straight from shared memory, earlier chunks (when the CTA's rows
// do not fit) from a second read of the input.  At 2048 x 4096 every row stays on chip, so
// the input is read from HBM exactly once and the statistics cost no launch of their own.
// ---------------------------------------------------------------------------
constexpr int kFusedSmemBudget = 200 * 1024;       // dynamic shared memory the row cache may use
constexpr long long kGridBarrierLimitCycles = 2000000000LL;  // about one second

__device__ int g_prepare_timeouts = 0;  // grid barriers that ran out (the result of such a call is wrong)

struct FusedParams {
  const __nv_bfloat16 *x;
  const __nv_bfloat16 *residual;  // kAdd: the input is bf16(x + residual) ...
  __nv_bfloat16 *sum_out;         // ... which is also written here
  const __nv_bfloat16 *gamma;
  float eps;
  float *inv_rms;            // [m], mode 1
  unsigned int *amax_bits;   // zero on entry
  unsigned int *arrive;      // zero on entry: grid barrier counter
  float *scale_out;
  uint8_t *a_comp, *e, *sfa_sparse, *q_res, *sf_res;
  int m, k;
  int rows_per_cta;
  int chunk_rows;  // rows of one shared-memory chunk
};

// stores of one quantised group: payloads by the owner lane, metadata and scale factors
// combined over neighbouring lanes (groups g, g+1[, g+2, g+3] of the same row)
__device__ __forceinline__ void store_group(const FusedParams &p, const GroupOut &o, int row, int group, bool live,
                                            bool in_padded, int aligned_m, int lane) {
  const int k = p.k, groups32 = k >> 5;
  if (live) {
    *reinterpret_cast<uint4 *>(p.q_res + (size_t)row * (k / 2) + (size_t)group * 16) =
        make_uint4(o.q_res[0], o.q_res[1], o.q_res[2], o.q_res[3]);
    *reinterpret_cast<uint2 *>(p.a_comp + (size_t)row * (k / 4) + (size_t)group * 8) = make_uint2(o.a_comp[0], o.a_comp[1]);
  }
  const uint32_t mine = o.meta & 0xFFFFu;
  const uint32_t other = __shfl_down_sync(0xffffffffu, mine, 1);
  if ((lane & 1) == 0 && in_padded)
    *reinterpret_cast<uint32_t *>(p.e + (size_t)(group >> 3) * aligned_m * 16 + (size_t)row * 16 + (size_t)(group & 7) * 2) =
        mine | (other << 16);
  const uint32_t sv = o.sf_sparse;
  const uint32_t s1 = __shfl_down_sync(0xffffffffu, sv, 1);
  const uint32_t s2 = __shfl_down_sync(0xffffffffu, sv, 2);
  const uint32_t s3 = __shfl_down_sync(0xffffffffu, sv, 3);
  const uint32_t r2 = o.sf_res;
  const uint32_t r2n = __shfl_down_sync(0xffffffffu, r2, 1);
  if (live) {
    if ((lane & 3) == 0)
      *reinterpret_cast<uint32_t *>(p.sfa_sparse + sf_offset(row, group, groups32)) = sv | (s1 << 8) | (s2 << 16) | (s3 << 24);
    if ((lane & 1) == 0) *reinterpret_cast<uint32_t *>(p.sf_res + sf_offset(row, 2 * group, k / 16)) = r2 | (r2n << 16);
  }
}

template <int kMode, bool kAdd, int kFusedThreads>
__global__ void __launch_bounds__(kFusedThreads, 1) prepare_fused_kernel(const FusedParams p) {
  static_assert(kMode == 1 || kMode == 2, "modes with a statistics pass");
  constexpr int kFusedWarps = kFusedThreads / 32;
  const int m = p.m, k = p.k;
  const int groups32 = k >> 5;
  const int groups_padded = ((k + 255) / 256) * 8;  // groups of the metadata tiles (256 columns each)
  const int aligned_m = (m + 127) / 128 * 128;
  const int row_vecs = k >> 3;                     // uint4 per row
  const int partial_stride = groups32 + 4;         // padded: 16-byte reads of neighbouring rows hit different banks
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  __shared__ ScaleTables tbl;
  __shared__ float warp_red[32];
  extern __shared__ uint4 fused_smem[];
  uint4 *gamma_s = fused_smem;                                      // mode 1: k bf16, pieces permuted like the cache
  uint4 *cache = fused_smem + (kMode == 1 ? row_vecs : 0);          // chunk_rows x k bf16
  float *partial = reinterpret_cast<float *>(cache + (size_t)p.chunk_rows * row_vecs);  // mode 1: chunk_rows x partial_stride
  float *inv_s = partial + (kMode == 1 ? p.chunk_rows * partial_stride : 0);            // mode 1: rows_per_cta

  ptx::grid_launch_dependents();
  if (threadIdx.x < 128) {
    const float v = ue4m3_to_float(threadIdx.x);
    tbl.value[threadIdx.x] = v;
    tbl.recip[threadIdx.x] = __frcp_rn(v);  // code 0 is never looked up (scales are clamped to >= 2^-9)
  }
  ptx::grid_dependency_wait();
  if (kMode == 1) {
    const uint4 *gsrc = reinterpret_cast<const uint4 *>(p.gamma);
    for (int i = threadIdx.x; i < row_vecs; i += kFusedThreads) gamma_s[cache_slot(i >> 2, i & 3)] = gsrc[i];
  }

  // ---- zero what no owner thread writes: padding rows of the metadata and scale-factor
  // bands, the spare band of the scale buffers, the tail of A_comp
  {
    const int worker = blockIdx.x * kFusedThreads + threadIdx.x;
    const int workers = gridDim.x * kFusedThreads;
    const size_t bands = (size_t)aligned_m / 128;
    zero_range(p.sfa_sparse, bands * (size_t)(groups32 / 4) * 512, sf_alloc_bytes(m, k), worker, workers);
    zero_range(p.sf_res, bands * (size_t)(k / 16 / 4) * 512, sf_alloc_bytes(m, k), worker, workers);
    zero_range(p.a_comp, (size_t)m * (k / 4), a_comp_bytes(m, k), worker, workers);
    zero_padding_rows(p.e, p.sfa_sparse, p.sf_res, m, k, worker, workers);
  }

  const int row_begin = min(m, (int)blockIdx.x * p.rows_per_cta);
  const int row_end = min(m, row_begin + p.rows_per_cta);
  const int rows = row_end - row_begin;
  const int chunks = rows > 0 ? (rows + p.chunk_rows - 1) / p.chunk_rows : 0;
  const int first_chunk_rows = rows - (chunks - 1) * p.chunk_rows;  // the short chunk goes first, the cached (last) one is full
  auto chunk_first_row = [&](int c) { return c == 0 ? 0 : first_chunk_rows + (c - 1) * p.chunk_rows; };
  auto chunk_size = [&](int c) { return c == 0 ? first_chunk_rows : p.chunk_rows; };
  const __nv_bfloat16 *src = kAdd ? p.sum_out : p.x;  // what a second read of the (summed) input reads
  // no barrier here: the tables and gamma are first read after the barriers of phase 1 / the grid barrier

  // ------------------------------------------------------------------ phase 1: statistics
  __nv_bfloat162 m2 = __floats2bfloat162_rn(0.0f, 0.0f);
  for (int c = 0; c < chunks; ++c) {
    const int c_rows = chunk_size(c), c_row0 = row_begin + chunk_first_row(c);
    if (c > 0) __syncthreads();  // the previous chunk's cache and partial sums are no longer read
    // two tasks (32-element groups) per iteration, all loads issued before the first use
    const int n_tasks = c_rows * groups32;
    for (int t0 = threadIdx.x; t0 < n_tasks; t0 += 2 * kFusedThreads) {
      uint32_t w[2][16];
      int rl[2], g[2];
      bool on[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int t = t0 + u * kFusedThreads;
        on[u] = t < n_tasks;
        rl[u] = on[u] ? t / groups32 : 0;
        g[u] = on[u] ? t - rl[u] * groups32 : 0;
      }
      uint4 xv[2][4], rv[2][4];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (on[u]) {
          const size_t off = (size_t)(c_row0 + rl[u]) * k + (size_t)g[u] * 32;
          const uint4 *xs = reinterpret_cast<const uint4 *>(p.x + off);
#pragma unroll
          for (int j = 0; j < 4; ++j) xv[u][j] = xs[j];
          if (kAdd) {
            const uint4 *rs = reinterpret_cast<const uint4 *>(p.residual + off);
#pragma unroll
            for (int j = 0; j < 4; ++j) rv[u][j] = rs[j];
          }
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (!on[u]) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          w[u][4 * j + 0] = xv[u][j].x;
          w[u][4 * j + 1] = xv[u][j].y;
          w[u][4 * j + 2] = xv[u][j].z;
          w[u][4 * j + 3] = xv[u][j].w;
        }
        if (kAdd) {
          uint4 *dst = reinterpret_cast<uint4 *>(p.sum_out + (size_t)(c_row0 + rl[u]) * k + (size_t)g[u] * 32);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t rw[4] = {rv[u][j].x, rv[u][j].y, rv[u][j].z, rv[u][j].w};
#pragma unroll
            for (int q = 0; q < 4; ++q)
              w[u][4 * j + q] = pack_bf16x2(__fadd_rn(lo_f(w[u][4 * j + q]), lo_f(rw[q])),
                                            __fadd_rn(hi_f(w[u][4 * j + q]), hi_f(rw[q])));
            dst[j] = make_uint4(w[u][4 * j], w[u][4 * j + 1], w[u][4 * j + 2], w[u][4 * j + 3]);
          }
        }
        uint4 *row_cache = cache + (size_t)rl[u] * row_vecs;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          row_cache[cache_slot(g[u], j)] = make_uint4(w[u][4 * j], w[u][4 * j + 1], w[u][4 * j + 2], w[u][4 * j + 3]);
        if (kMode == 1) {
          float sq = 0.0f;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float a = lo_f(w[u][i]), b = hi_f(w[u][i]);
            sq = __fmaf_rn(a, a, sq);  // a*a is exact in float, so this equals sq + a*a
            sq = __fmaf_rn(b, b, sq);
          }
          partial[rl[u] * partial_stride + g[u]] = sq;
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) m2 = __hmax2(m2, __habs2(*reinterpret_cast<const __nv_bfloat162 *>(&w[u][i])));
        }
      }
    }
    if (kMode == 1) {
      __syncthreads();
      if (threadIdx.x < c_rows) {
        const float4 *pr = reinterpret_cast<const float4 *>(partial + threadIdx.x * partial_stride);
        float total = 0.0f;
        for (int i = 0; i < groups32 / 4; ++i) {  // groups32 is a multiple of 4 (K % 128 == 0)
          const float4 v = pr[i];
          total = __fadd_rn(total, v.x);
          total = __fadd_rn(total, v.y);
          total = __fadd_rn(total, v.z);
          total = __fadd_rn(total, v.w);
        }
        const float inv = rsqrtf(__fadd_rn(__fdiv_rn(total, (float)k), p.eps));
        inv_s[chunk_first_row(c) + threadIdx.x] = inv;
        p.inv_rms[c_row0 + threadIdx.x] = inv;
      }
      __syncthreads();
      // normalise in place: the cache then holds y = bf16(x * inv_rms * gamma)
      for (int t = threadIdx.x; t < c_rows * groups32; t += kFusedThreads) {
        const int rl = t / groups32, g = t - rl * groups32;
        const float inv = inv_s[chunk_first_row(c) + rl];
        uint4 *row_cache = cache + (size_t)rl * row_vecs;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int slot = cache_slot(g, j);
          const uint4 xv = row_cache[slot];
          const uint4 gv = gamma_s[slot];
          const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w}, gw[4] = {gv.x, gv.y, gv.z, gv.w};
          uint32_t y[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            y[q] = normalise_word(xw[q], gw[q], pair_f32(inv, inv));
            m2 = __hmax2(m2, __habs2(*reinterpret_cast<const __nv_bfloat162 *>(&y[q])));
          }
          row_cache[slot] = make_uint4(y[0], y[1], y[2], y[3]);
        }
      }
    }
  }

  // ---- CTA absmax -> tensor absmax, grid barrier, tensor scale
  {
    float mx = fmaxf(__bfloat162float(m2.x), __bfloat162float(m2.y));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) warp_red[warp] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
      for (int w = 1; w < kFusedWarps; ++w) mx = fmaxf(mx, warp_red[w]);
      if (mx > 0.0f) atomicMax(p.amax_bits, __float_as_uint(mx));
      __threadfence();
      atomicAdd(p.arrive, 1u);
      const long long t0 = clock64();
      while (ld_acquire_gpu(p.arrive) < gridDim.x) {
        if (clock64() - t0 > kGridBarrierLimitCycles) {
          atomicAdd(&g_prepare_timeouts, 1);
          break;
        }
      }
    }
    __syncthreads();
  }
  const float amax = __uint_as_float(ld_acquire_gpu(p.amax_bits));
  // ATen divides a CUDA tensor by a host scalar by multiplying with the float
  // reciprocal; clamp(min=1e-9) follows (kernels/src/bindings.cpp:337 of the reference).
  const float scale = fmaxf(__fmul_rn(amax, 1.0f / 2688.0f), 1.0e-9f);
  if (p.scale_out != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *p.scale_out = scale;
  const float div = kMode == 2 ? round_to_bf16(scale) : scale;  // see round_to_bf16
  const float recip = __frcp_rn(div);

  // ------------------------------------------------------------------ phase 2: quantise
  const int tasks_per_row = (groups_padded + 31) >> 5;  // a warp takes 32 neighbouring groups of one row
  for (int c = chunks - 1; c >= 0; --c) {
    const bool cached = c == chunks - 1;
    const int c_rows = chunk_size(c), c_row0 = row_begin + chunk_first_row(c);
    int rl = warp / tasks_per_row, piece = warp % tasks_per_row;
    const int step_rl = kFusedWarps / tasks_per_row, step_piece = kFusedWarps % tasks_per_row;
    for (int wt = warp; wt < c_rows * tasks_per_row; wt += kFusedWarps, rl += step_rl, piece += step_piece) {
      if (piece >= tasks_per_row) {
        piece -= tasks_per_row;
        ++rl;
      }
      const int group = piece * 32 + lane;
      const int row = c_row0 + rl;
      const bool live = group < groups32;
      uint32_t xw[16];
      GroupOut o;
      o.a_comp[0] = o.a_comp[1] = 0;
      o.meta = 0;
      o.sf_sparse = 0;
      o.sf_res = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) o.q_res[i] = o.q_sparse[i] = 0;
      // the group's 32 values from the row cache or, for a chunk that is not cached, from global memory
      auto load_group = [&](uint32_t (&w)[16]) {
        if (cached) {
          const uint4 *row_cache = cache + (size_t)rl * row_vecs;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint4 v = row_cache[cache_slot(group, j)];
            w[4 * j + 0] = v.x;
            w[4 * j + 1] = v.y;
            w[4 * j + 2] = v.z;
            w[4 * j + 3] = v.w;
          }
        } else {
          // plain loads: with kAdd these bytes were written by this CTA in phase 1
          const uint4 *xs = reinterpret_cast<const uint4 *>(src + (size_t)row * k + (size_t)group * 32);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint4 v = xs[j];
            w[4 * j + 0] = v.x;
            w[4 * j + 1] = v.y;
            w[4 * j + 2] = v.z;
            w[4 * j + 3] = v.w;
          }
        }
      };
      if (live) {
        load_group(xw);
        if (!cached) {
          if (kMode == 1) {
            const float inv = inv_s[chunk_first_row(c) + rl];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint4 gv = gamma_s[cache_slot(group, j)];
              const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w};
#pragma unroll
              for (int q = 0; q < 4; ++q) xw[4 * j + q] = normalise_word(xw[4 * j + q], gw[q], pair_f32(inv, inv));
            }
          }
        }
        scale_quantize_group<kMode, false>(xw, div, recip, tbl, o, load_group);
      }
      store_group(p, o, row, group, live, group < groups_padded, aligned_m, lane);
    }
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------

size_t prepare_workspace_bytes(int m) { return 256 + (size_t)m * sizeof(float); }

size_t prepare_workspace_best_bytes(int m) { return prepare_workspace_bytes(m) + kMaxAbsmaxWords * sizeof(float); }

// SM count of the current device (queried once per device).
static cudaError_t current_sms(int *dev_out, int *sms_out) {
  static int sms[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (sms[dev] == 0 && (e = cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  *dev_out = dev;
  *sms_out = sms[dev];
  return cudaSuccess;
}

// How a scaled prepare finds its maximum and quantises (scaled_prepare_form names them by number).
enum class PrepareForm {
  kCtaScan = 0,      // prepare_kernel, every CTA scans the input
  kClusterScan = 1,  // prepare_kernel, every cluster scans it
  kNarrow = 2,       // statistics launch, prepare_narrow_kernel
  kWide = 3,         // statistics launch (none where the maximum is ready), prepare_kernel
  kOneLaunch = 4     // prepare_fused_kernel
};

// 32-row x 256-column tiles of the padded activation.
static int prepare_tiles(int m, int k) { return (k + kColsPerCta - 1) / kColsPerCta * ((m + 127) / 128 * 128 / kRowsPerCta); }

// As many CTAs as are resident at once: a grid of 444 for the two-CTA kernel ran its last third at one CTA per SM.
static int prepare_grid(const PrepareParams &p, int ctas_per_sm) {
  int dev = 0, sms = 0;
  const int tiles = prepare_tiles(p.m, p.k);
  if (current_sms(&dev, &sms) != cudaSuccess) return tiles < 1024 ? tiles : 1024;
  const int full = sms * ctas_per_sm;
  return tiles < full ? tiles : full;
}

// CTAs of prepare_narrow_kernel.
static int narrow_ctas(int mode, int m, int k) { return (m * ((k + 255) / 256) + narrow_warps(mode) - 1) / narrow_warps(mode); }

static cudaError_t launch_prepare(int mode, bool debug, const PrepareParams &p, cudaStream_t stream, PrepareForm form = PrepareForm::kWide) {
  const bool cluster = form == PrepareForm::kClusterScan;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // the table set-up overlaps the kernel before
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(prepare_grid(p, mode == 2 && p.src_row == nullptr ? kScaledCtasPerSm : kPrepareCtasPerSm));
  cfg.blockDim = dim3(kPrepareThreads);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (form == PrepareForm::kNarrow) {
    cfg.gridDim = dim3((unsigned)narrow_ctas(mode, p.m, p.k));
    cfg.blockDim = dim3((unsigned)(32 * narrow_warps(mode)));
    return cudaLaunchKernelEx(&cfg, mode == 1 ? prepare_narrow_kernel<1> : prepare_narrow_kernel<2>, p);
  }
  if (cluster) {
    cfg.gridDim.x = (cfg.gridDim.x + kScanCtas - 1) / kScanCtas * kScanCtas;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = kScanCtas;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  }
  if (debug) return cudaLaunchKernelEx(&cfg, prepare_kernel<0, true>, p);
  if (mode == 0) return cudaLaunchKernelEx(&cfg, prepare_kernel<0, false>, p);
  if (mode == 1) {
    const size_t gamma_bytes = (size_t)p.k * sizeof(__nv_bfloat16);
    static bool attr_set[64] = {};
    int dev = 0;
    if (gamma_bytes > 48 * 1024 && cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 && !attr_set[dev]) {
      cudaError_t e = cudaFuncSetAttribute(prepare_kernel<1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
      if (e != cudaSuccess) return e;
      attr_set[dev] = true;
    }
    cfg.dynamicSmemBytes = gamma_bytes;
    return cudaLaunchKernelEx(&cfg, prepare_kernel<1, false>, p);
  }
  if (p.src_row != nullptr) return cudaLaunchKernelEx(&cfg, prepare_kernel<2, false>, p);
  if (cluster) return cudaLaunchKernelEx(&cfg, prepare_kernel<2, false, kScaledCtasPerSm, true>, p);
  return cudaLaunchKernelEx(&cfg, prepare_kernel<2, false, kScaledCtasPerSm>, p);
}

cudaError_t run_prepare(const void *x, int m, int k, void *a_comp, void *e, void *q_sparse_dense,
                        void *sfa_sparse, void *q_res, void *sf_res, cudaStream_t stream) {
  PrepareParams p{};
  p.x = static_cast<const __nv_bfloat16 *>(x);
  p.a_comp = static_cast<uint8_t *>(a_comp);
  p.e = static_cast<uint8_t *>(e);
  p.q_sparse_dense = static_cast<uint8_t *>(q_sparse_dense);
  p.sfa_sparse = static_cast<uint8_t *>(sfa_sparse);
  p.q_res = static_cast<uint8_t *>(q_res);
  p.sf_res = static_cast<uint8_t *>(sf_res);
  p.m = m;
  p.k = k;
  p.row_tiles = (m + 127) / 128 * 128 / kRowsPerCta;
  return launch_prepare(0, q_sparse_dense != nullptr, p, stream);
}

// One cooperative launch for statistics + prepare (see prepare_fused_kernel).  Returns
// cudaErrorNotSupported when the shape does not fit or the device cannot launch it, in which
// case the caller falls back to the separate statistics and prepare kernels.
// 512 threads per CTA: measured against 448, 768 and 896 (more threads spill or idle in the
// partly filled last round of 56 warp tasks per CTA at 2048 x 4096)
template <int kMode, bool kAdd>
static cudaError_t launch_fused(const FusedParams &p_in, cudaStream_t stream) {
  constexpr int kThreads = 512;
  static bool attr_set[64] = {};
  static int coop[64] = {};  // 0 unknown, 1 yes, -1 no
  int dev = 0, sms = 0;
  cudaError_t e = current_sms(&dev, &sms);
  if (e != cudaSuccess) return e;
  if (coop[dev] == 0) {
    int v = 0;
    coop[dev] = (cudaDeviceGetAttribute(&v, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && v) ? 1 : -1;
  }
  if (coop[dev] < 0) return cudaErrorNotSupported;
  FusedParams p = p_in;
  const int groups32 = p.k / 32;
  p.rows_per_cta = (p.m + sms - 1) / sms;
  const size_t row_bytes = (size_t)p.k * 2 + (kMode == 1 ? (size_t)(groups32 + 4) * 4 : 0);
  const size_t fixed = (kMode == 1 ? (size_t)p.k * 2 + (size_t)p.rows_per_cta * 4 : 0);
  if (fixed + row_bytes > (size_t)kFusedSmemBudget) return cudaErrorNotSupported;
  const size_t capacity = ((size_t)kFusedSmemBudget - fixed) / row_bytes;
  p.chunk_rows = (int)(capacity < (size_t)p.rows_per_cta ? capacity : (size_t)p.rows_per_cta);
  auto kernel = prepare_fused_kernel<kMode, kAdd, kThreads>;
  if (!attr_set[dev]) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFusedSmemBudget + 16);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.gridDim = dim3(sms);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = fixed + (size_t)p.chunk_rows * row_bytes + 16;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, p);
}

static bool fused_prepare_enabled() {
  static const bool on = [] {
    const char *v = getenv("SHARQ_PREPARE_FUSED");  // tuning hook: 0 selects the separate statistics + prepare kernels
    return !(v != nullptr && v[0] == '0');
  }();
  return on;
}

int prepare_timeouts() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_prepare_timeouts, sizeof(v)) != cudaSuccess) return -1;
  return v;
}

struct ScaledPlan {
  PrepareForm form;
  bool narrow;         // the quantisation behind a statistics launch
  unsigned stat_ctas;  // statistics launch: one CTA per row (RMSNorm) or a flat grid
  bool word_per_cta;   // its CTAs' maxima go behind the row statistics, where the caller's workspace has room for a word each
  size_t words_at;
};

static ScaledPlan plan_scaled_prepare(int m, int k, bool rms, bool residual, bool absmax_ready, bool inv_rms_external, size_t workspace_bytes,
                                      int sms) {
  ScaledPlan q{};
  const size_t elements = (size_t)m * (size_t)k;
  const size_t flat = (elements / 8 + 255) / 256;
  q.stat_ctas = rms ? (unsigned)m : (unsigned)(flat < (size_t)sms * 8 ? flat : (size_t)sms * 8);
  q.words_at = 256 + (rms && !inv_rms_external ? (size_t)m * sizeof(float) : 0);
  q.word_per_cta = q.stat_ctas <= kMaxAbsmaxWords && workspace_bytes >= q.words_at + (size_t)q.stat_ctas * sizeof(float);
  q.narrow = !absmax_ready && m > kRowsPerCta && (rms ? elements <= kNarrowElements : narrow_ctas(2, m, k) <= sms);
  q.form = q.narrow ? PrepareForm::kNarrow : PrepareForm::kWide;
  if (absmax_ready) return q;
  // Without room for the words the other forms are a cooperative launch behind a memset, and the scan pays longer: by every CTA where the
  // clusters would not fit at once (us per call in a graph, CTA / cluster: 2 x 18944 3.5 / 5.6, 8 x 18944 5.8 / 6.5, 10 x 18944 6.6 / 6.6).
  const bool clusters_fit = prepare_tiles(m, k) <= kClusterScanTiles;
  if (!rms && (elements <= kCtaScanElements || (clusters_fit && elements <= kClusterScanElements) ||
               (!q.word_per_cta && elements <= kInlineAbsmaxElementsNoWords))) {
    q.form = elements > kCtaScanElements && clusters_fit ? PrepareForm::kClusterScan : PrepareForm::kCtaScan;
    return q;
  }
  // Two launches that overlap, with nothing to zero, beat one cooperative launch behind its memset (us, two launches / one: tensor scale
  // 64 x 4096 5.0 / 8.4, 2048 x 4096 12.0 / 16.9, 4096 x 4096 19.6 / 27.1; RMSNorm 33 x 4096 7.0 / 10.5, 512 x 4096 9.1 / 12.5, 4096 x 4096
  // 29.8 / 33.0), except with the residual add on middle sizes, where the row caches spare the second read of the sum: 512 x 4096
  // 10.8 / 12.7, 2048 x 4096 24.7 / 24.9, 2048 x 8192 49.4 / 45.6, 700 x 14336 37.2 / 30.7.  Without room for the words the memset precedes both forms, and
  // one launch pays while the row caches hold most of the tensor.
  if (fused_prepare_enabled() && (q.word_per_cta ? residual && elements >= ((size_t)1 << 22) && elements < ((size_t)1 << 25)
                                                 : elements < (rms ? ((size_t)1 << 25) : ((size_t)1 << 24))))
    q.form = PrepareForm::kOneLaunch;
  return q;
}

int scaled_prepare_form(int m, int k, bool rms, bool residual, bool absmax_ready, size_t workspace_bytes, int sms) {
  return (int)plan_scaled_prepare(m, k, rms, residual, absmax_ready, false, workspace_bytes, sms).form;
}

cudaError_t run_scaled_prepare(const void *x, const void *gamma, float eps, int m, int k, void *workspace,
                               float *inv_rms_external, void *a_comp, void *e, void *sfa_sparse, void *q_res,
                               void *sf_res, float *scale_out, cudaStream_t stream, int absmax_words,
                               const void *residual, void *sum_out, size_t workspace_bytes, unsigned int *amax_out) {
  const bool absmax_ready = absmax_words > 0;
  if (residual != nullptr && (gamma == nullptr || sum_out == nullptr)) return cudaErrorInvalidValue;
  // workspace: [0,4) tensor absmax bits; [256, 256+4m) inv_rms
  auto *amax_bits = static_cast<unsigned int *>(workspace);
  float *inv_rms = inv_rms_external ? inv_rms_external
                                    : reinterpret_cast<float *>(static_cast<uint8_t *>(workspace) + 256);
  cudaError_t err = cudaSuccess;
  const bool rms = gamma != nullptr;
  const size_t elements = (size_t)m * (size_t)k;
  int dev = 0, sms = 0;
  if (current_sms(&dev, &sms) != cudaSuccess) sms = 128;
  const ScaledPlan plan = plan_scaled_prepare(m, k, rms, residual != nullptr, absmax_ready, inv_rms_external != nullptr, workspace_bytes, sms);
  const bool scan = plan.form == PrepareForm::kCtaScan || plan.form == PrepareForm::kClusterScan;
  const bool leave_absmax = scan ? elements > (plan.word_per_cta ? kInlineAbsmaxElements : kInlineAbsmaxElementsNoWords) : plan.word_per_cta;
  PrepareForm form = plan.form;
  if (form == PrepareForm::kOneLaunch) {
    FusedParams f{};
    f.x = static_cast<const __nv_bfloat16 *>(x);
    f.residual = static_cast<const __nv_bfloat16 *>(residual);
    f.sum_out = static_cast<__nv_bfloat16 *>(sum_out);
    f.gamma = static_cast<const __nv_bfloat16 *>(gamma);
    f.eps = eps;
    f.inv_rms = inv_rms;
    f.amax_bits = amax_bits;
    f.arrive = amax_bits + 1;
    f.scale_out = scale_out;
    f.a_comp = static_cast<uint8_t *>(a_comp);
    f.e = static_cast<uint8_t *>(e);
    f.sfa_sparse = static_cast<uint8_t *>(sfa_sparse);
    f.q_res = static_cast<uint8_t *>(q_res);
    f.sf_res = static_cast<uint8_t *>(sf_res);
    f.m = m;
    f.k = k;
    if ((err = cudaMemsetAsync(amax_bits, 0, 2 * sizeof(unsigned int), stream)) != cudaSuccess) return err;
    err = !rms ? launch_fused<2, false>(f, stream)
               : (residual != nullptr ? launch_fused<1, true>(f, stream) : launch_fused<1, false>(f, stream));
    if (err == cudaSuccess) return cudaSuccess;
    (void)cudaGetLastError();  // not launchable here: the separate kernels below do the same work
    if (err != cudaErrorNotSupported && err != cudaErrorCooperativeLaunchTooLarge) return err;
    err = cudaSuccess;
    form = plan.narrow ? PrepareForm::kNarrow : PrepareForm::kWide;
  }
  int words = absmax_words;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.stream = stream;
  cfg.attrs = attr;
  // The flat absolute maximum starts early (16 x 14336 and its GEMM 22.9 against 23.4 us); the row statistics don't: their few large
  // CTAs crowd the SMs that the kernel ahead leaves free (behind another prepare, with the residual add: 64 x 32768 25.6 against 18.0 us,
  // 129 x 14336 19.1 against 12.8, 512 x 8192 20.8 against 15.8, 2048 x 32768 222 against 182; behind a GEMM both take the same time).
  cfg.numAttrs = rms ? 0 : 1;
  const auto *xb = static_cast<const __nv_bfloat16 *>(x);
  if (absmax_ready) {
    // the producer of x already left max|x| in the workspace: no statistics pass
    if (rms) return cudaErrorInvalidValue;
  } else if (scan) {
    amax_bits = nullptr;
  } else {
    const int groups = k / 32;
    cfg.gridDim = dim3(plan.stat_ctas);
    cfg.blockDim = dim3(rms ? (unsigned)((groups + 31) / 32 * 32) : 256u);
    cfg.dynamicSmemBytes = rms ? (size_t)groups * sizeof(float) : 0;
    if (plan.word_per_cta) {
      amax_bits = reinterpret_cast<unsigned int *>(static_cast<uint8_t *>(workspace) + plan.words_at);
      words = (int)plan.stat_ctas;
    } else if ((err = cudaMemsetAsync(amax_bits, 0, sizeof(unsigned int), stream)) != cudaSuccess) {
      return err;
    }
    const auto *g = static_cast<const __nv_bfloat16 *>(gamma);
    if (!rms) {
      err = cudaLaunchKernelEx(&cfg, abs_stats_kernel, xb, (size_t)m * k / 8, amax_bits, plan.word_per_cta);
    } else if (residual != nullptr) {
      err = cudaLaunchKernelEx(&cfg, rms_stats_kernel<true>, xb, static_cast<const __nv_bfloat16 *>(residual),
                               static_cast<__nv_bfloat16 *>(sum_out), g, eps, k, inv_rms, amax_bits, plan.word_per_cta);
      x = sum_out;  // the prepare reads the sum
    } else {
      err = cudaLaunchKernelEx(&cfg, rms_stats_kernel<false>, xb, static_cast<const __nv_bfloat16 *>(nullptr),
                               static_cast<__nv_bfloat16 *>(nullptr), g, eps, k, inv_rms, amax_bits, plan.word_per_cta);
    }
    if (err != cudaSuccess) return err;
  }

  PrepareParams p{};
  p.x = static_cast<const __nv_bfloat16 *>(x);
  p.gamma = static_cast<const __nv_bfloat16 *>(gamma);
  p.inv_rms = inv_rms;
  p.amax_bits = amax_bits;
  p.amax_words = words;
  p.amax_out = !absmax_ready && leave_absmax ? static_cast<unsigned int *>(workspace) : amax_out;
  p.scale_out = scale_out;
  p.a_comp = static_cast<uint8_t *>(a_comp);
  p.e = static_cast<uint8_t *>(e);
  p.sfa_sparse = static_cast<uint8_t *>(sfa_sparse);
  p.q_res = static_cast<uint8_t *>(q_res);
  p.sf_res = static_cast<uint8_t *>(sf_res);
  p.m = m;
  p.k = k;
  p.row_tiles = (m + 127) / 128 * 128 / kRowsPerCta;
  return launch_prepare(rms ? 1 : 2, false, p, stream, form);
}

cudaError_t run_grouped_prepare(const void *x, int m, int k, const unsigned int *amax_bits, const int *unit_group, int groups,
                                void *a_comp, void *e, void *sfa_sparse, void *q_res, void *sf_res, float *scale_vec_out,
                                cudaStream_t stream, const int *src_row) {
  if (m <= 0 || m % 256 != 0 || groups < 1) return cudaErrorInvalidValue;
  PrepareParams p{};
  p.x = static_cast<const __nv_bfloat16 *>(x);
  p.amax_bits = amax_bits;
  p.a_comp = static_cast<uint8_t *>(a_comp);
  p.e = static_cast<uint8_t *>(e);
  p.sfa_sparse = static_cast<uint8_t *>(sfa_sparse);
  p.q_res = static_cast<uint8_t *>(q_res);
  p.sf_res = static_cast<uint8_t *>(sf_res);
  p.m = m;
  p.k = k;
  p.row_tiles = m / kRowsPerCta;
  p.unit_group = unit_group;
  p.scale_vec_out = scale_vec_out;
  p.groups = groups;
  p.src_row = src_row;
  return launch_prepare(2, false, p, stream);
}

}  // namespace sharq

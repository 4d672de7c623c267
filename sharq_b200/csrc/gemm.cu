// Block-scaled FP4 GEMMs for sm_100a, hand-written on tcgen05 / TMEM / TMA:
//   dense NVFP4      D = bf16(alpha * (A . B^T) + beta * C)         (one UE4M3 scale per 16 along K)
//   sparse NVFP4     the same with a pair-wise 4:8 compressed A     (one scale per 32 logical K)
//   fused SharQ      sparse main + dense residual against the SAME weight tile, both
//                    accumulated into one TMEM tile, one epilogue (+ optional bias).
// They replace the reference's CUTLASS-generated kernels behind the same buffers:
//   kernels/src/nvfp4.cu:432-455, kernels/src/sparse_nvfp4.cu:436-460 and the two-launch
//   composition at model/qLinearLayer.py:130-154.
//
// One persistent kernel, one CTA per SM (or one CTA pair per SM pair), looping over output
// tiles with the M index fastest so that CTAs working at the same time share weight tiles
// in L2.  K is consumed in stages of 256.  Warp roles:
//   warp 0     TMA producer: per stage three tensor-map loads (weight tile, dense A tile,
//              compressed A tile; 128-byte / 64-byte swizzle) and plain bulk copies of the
//              metadata tile and the scale-factor tiles, all landing on one mbarrier.  It runs
//              ahead across tile boundaries, so the pipeline never drains between tiles.
//   warp 1     MMA issuer: copies metadata and scale factors shared -> tensor memory
//              (tcgen05.cp), then issues 2 sparse (K=128) and 4 dense (K=64) MMAs per stage
//              into the same accumulator; tcgen05.commit releases the stage.
//   warps 2-9  epilogue: pull the whole accumulator into registers with tcgen05.ld, hand the
//              tensor memory back to the MMA warp at once, then alpha/beta/bias, bf16 (packed
//              conversions), a transpose through a small shared-memory tile and coalesced
//              global stores overlap the next tile's MMAs.
// Few tiles (decode batches, short chunks): K is split over the CTAs of a cluster, one tile per cluster; the fp32 partial tiles meet in
// distributed shared memory, where every element is summed in rank order (no scratch, no second kernel, a fixed order of
// additions).  How they meet depends on the rows of the tile, see Exchange.
// CTA-pair mode (cta_group::2, cluster of 2): the pair computes a 256 x 256 tile; CTA r owns
// rows [128r,128r+128) (its A operands, scales, metadata, accumulator) and loads weight rows
// [128r,128r+128) of the tile; the tensor cores of both SMs read both halves.  Every CTA
// loads with its own plain TMA copies - there is no multicast load anywhere.  Hand-shake:
// the peer CTA reports each loaded stage on the leader's peer barrier, the leader issues
// the pair's MMAs and commits to the barriers of both CTAs.
// All mbarrier waits are bounded; a timed-out wait sets *error_flag and every role drains
// to the common exit, where tensor memory is released.
#include "common.cuh"
#include "gemm.cuh"
#include "silu.cuh"
#include "sm100_ptx.cuh"

#include <cstring>
#include <mutex>

namespace sharq {

namespace {

constexpr int kBM = 128;
constexpr int kBK = 256;  // logical K per stage
constexpr int kEpiWarps = 8;
// K stages of weights a CTA prefetches into L2 while the activation is still being prepared: about what the ring holds.
// (Linears of a 32-token decode step, us: none 89.7, 3 87.3, 8 87.4; 28672 x 4096 at M = 32 right behind another GEMM 20.6 / 20.0 / 21.5.)
constexpr int kPrefetchStages = 3;
constexpr int kMaxSplits = 8;  // CTAs of a split-K cluster (the portable cluster size)
constexpr int kGemmThreads = 64 + 32 * kEpiWarps;

// Split launches: the columns of a tile are dealt over the CTAs of the cluster in runs of 8; run u belongs to rank
// u * splits / runs.
__host__ __device__ constexpr int first_run(int rank, int splits, int runs) { return (rank * runs + splits - 1) / splits; }
constexpr int kRecvPad = 4;  // floats behind each received row: neighbouring rows start on distinct banks

// How the partial tiles of a split launch meet:
//   kSendRegisters: every CTA sends the columns of its part to the CTAs that own them, 16 bytes at a time from its registers
//     (asynchronous stores that count on the owner's barrier), and sums its own columns.
//   kSendBlocks: the same by one block copy per owner, out of stages beside the receiving ones.
//   kPull: every CTA leaves its part in its own shared memory, and behind a cluster barrier all threads of the cluster read the others'.
// Sending saves the latency of the reads and a barrier, but its 16-byte stores and its few receiving CTAs are slower per byte.  us of a prepare
// and its fused GEMM, registers / blocks / pull: 1024 x 8192 (8 CTAs per tile) at M = 16 9.7 / 9.9 / 11.2, 32 11.1 / 11.1 / 12.1, 48 12.7 / 12.1 / 12.9,
// 64 14.7 / 13.4 / 13.8, 96 17.5 / 15.9 / 15.7, 128 21.2 / 19.1 / 18.2; 3584 x 18944 (4) at 48 20.6 / 20.2 / 20.4, 64 22.0 / 21.2 / 21.4, 128 27.3 / 26.0 / 24.0,
// 384 (3, wide tiles) 44.7 / 44.6 / 40.0; 6144 x 4096 (3) at 64 13.8 / 14.2 / 13.3; 3584 x 18944 (2) at 211 33.5 / 33.8 / 31.1.
enum Exchange { kSendRegisters = 0, kSendBlocks = 1, kPull = 2 };
constexpr int kRegisterRows = 32;  // rows of a tile up to which parts are sent from registers
constexpr int kBlockSplits = 4;    // fewer CTAs per tile: blocks are no faster than reads
constexpr int block_rows(int splits) { return 48 + 4 * splits; }  // rows up to which they are
constexpr int max_recv_bytes(int bn) {
  int most = 0;
  for (int s = 2; s <= kMaxSplits; ++s)
    for (int r = 0; r < s; ++r) {
      const int cols = 8 * (first_run(r + 1, s, bn / 8) - first_run(r, s, bn / 8));
      const int bytes = s * block_rows(s) * (cols + kRecvPad) * 4;
      most = bytes > most ? bytes : most;
    }
  return most;
}

// A wait that ran out: the first code of a launch stays.  Whatever gives up makes others give up behind it (a CTA that sends nothing lets the
// waits of its cluster run out), and their codes would hide the role that failed first.
__device__ __forceinline__ void report(int *error_flag, int code) { atomicCAS(error_flag, 0, code); }

// Shared-memory stage and tensor-memory column layout.  In pair mode BN is the pair's tile
// width (256) and each CTA stores half of the weight tile.
template <int BN, bool SPARSE, bool DENSE, bool PAIR>
struct StageLayout {
  static constexpr int kBands = BN / 128;  // 128-row scale-factor bands of the weight tile
  static constexpr int kWRows = PAIR ? BN / 2 : BN;
  static constexpr int kWBytes = kWRows * 128;
  static constexpr int kADenseBytes = DENSE ? kBM * 128 : 0;
  static constexpr int kACompBytes = SPARSE ? kBM * 64 : 0;
  static constexpr int kEBytes = SPARSE ? 2048 : 0;
  static constexpr int kSfaSpBytes = SPARSE ? 1024 : 0;
  static constexpr int kSfbSpBytes = SPARSE ? kBands * 1024 : 0;
  static constexpr int kSfaDBytes = DENSE ? 2048 : 0;
  static constexpr int kSfbDBytes = DENSE ? kBands * 2048 : 0;
  static constexpr int kOffW = 0;
  static constexpr int kOffADense = kOffW + kWBytes;
  static constexpr int kOffAComp = kOffADense + kADenseBytes;
  static constexpr int kOffE = kOffAComp + kACompBytes;
  static constexpr int kOffSfaSp = kOffE + kEBytes;
  static constexpr int kOffSfbSp = kOffSfaSp + kSfaSpBytes;
  static constexpr int kOffSfaD = kOffSfbSp + kSfbSpBytes;
  static constexpr int kOffSfbD = kOffSfaD + kSfaDBytes;
  static constexpr int kStageBytes = (kOffSfbD + kSfbDBytes + 1023) / 1024 * 1024;
  static constexpr int kOutStageBytes = kEpiWarps * 32 * 64;  // per epilogue warp 32 rows x 32 bf16 for the tile store
  static constexpr int kMaxSmem = 227 * 1024 - 2048 - kOutStageBytes;
  static constexpr int kStagesFit = kMaxSmem / kStageBytes;
  static constexpr int kStages = kStagesFit > 8 ? 8 : kStagesFit;
  // tensor memory columns
  static constexpr int kColAcc = 0;
  static constexpr int kColE = BN;
  static constexpr int kColSfaSp = kColE + 4;
  static constexpr int kColSfbSp = kColSfaSp + 8;
  static constexpr int kColSfaD = kColSfbSp + 2 * (BN / 32);
  static constexpr int kColSfbD = kColSfaD + 16;
  static constexpr int kColEnd = kColSfbD + 4 * (BN / 32);
  static constexpr int kTmemCols = kColEnd <= 256 ? 256 : 512;
  static constexpr int kPartStride = BN + 4;  // floats per row of a partial tile that is pulled (row starts on distinct banks)
  static_assert(PAIR || (max_recv_bytes(BN) <= kStages * kStageBytes && kBM * kPartStride * 4 <= kStages * kStageBytes),
                "the parts take the place of the stages");
  static constexpr int kSmemBytes =
      kStages * kStageBytes + kOutStageBytes + 1024 /*alignment slack*/ + 512 /*barriers*/;
};

// Where a rank receives the parts of its columns: in the stages that it is done with first (its last use of a slot lies furthest back).
struct RecvSlots {
  int first, count;
};
template <class L>
__host__ __device__ constexpr RecvSlots recv_slots(int rank, int splits, int rows, int k_stages, int runs) {
  const int stride = 4 * (8 * (first_run(rank + 1, splits, runs) - first_run(rank, splits, runs)) + kRecvPad);
  const int oldest = (k_stages * (rank + 1) / splits - k_stages * rank / splits) % L::kStages;
  const int count = (splits * rows * stride + L::kStageBytes - 1) / L::kStageBytes;
  return {oldest + count <= L::kStages ? oldest : 0, count};
}
// The stage that the blocks of a rank are laid out from: the first ones, or those behind the receiving slots; -1: neither holds them.
template <class L>
__host__ __device__ constexpr int send_slot(int rank, int splits, int rows, int k_stages, int bn) {
  const RecvSlots r = recv_slots<L>(rank, splits, rows, k_stages, bn / 8);
  const int need = (rows * (bn + splits * kRecvPad) * 4 + L::kStageBytes - 1) / L::kStageBytes;
  return r.first >= need ? 0 : (L::kStages - r.first - r.count >= need ? r.first + r.count : -1);
}
template <class L>
constexpr Exchange exchange_form(int rows, int splits, int k_stages, int bn) {
  if (rows <= kRegisterRows) return kSendRegisters;
  if (rows > block_rows(splits) || splits < kBlockSplits) return kPull;
  for (int r = 0; r < splits; ++r)
    if (send_slot<L>(r, splits, rows, k_stages, bn) < 0) return kPull;  // all CTAs of a cluster do the same
  return kSendBlocks;
}

struct GemmParams {
  const uint8_t *e;
  const uint8_t *sfa_sparse;
  const uint8_t *sfa_dense;
  const uint8_t *sfb_sparse;
  const uint8_t *sfb_dense;
  const __nv_bfloat16 *c_in;
  const __nv_bfloat16 *bias;
  const __nv_bfloat16 *residual;  // added to the finished bf16 value, as a separate bf16 add would
  __nv_bfloat16 *d;
  const float *alpha_ptr;
  float alpha;
  float beta;
  int m, n, k;
  int *error_flag;
  // Split K: the k_splits CTAs of a cluster compute one output tile, each over its share of the K stages.
  int k_splits;
  Exchange exchange, exchange_last;  // of the full tiles and of the last row of tiles
  int a_rows;        // rows of an activation box: the rows that exist when all are in one tile, else the tile's 128
  int staged_store;  // output tiles are transposed through shared memory for coalesced stores (N % 8 == 0)
  // Scatter mode (row-parallel linear under tensor parallelism): the output rows are dealt to their owner GPUs.
  // Row r belongs to GPU o = r / scatter_rows and is stored, through the peer mapping, into d_peer[o] at row
  // scatter_rank * scatter_rows + (r - o * scatter_rows): every GPU collects one [scatter_rows, n] block per
  // source GPU.  scatter_rows is a multiple of 128, so a tile has one owner.  scatter_rows == 0: plain output.
  __nv_bfloat16 *d_peer[kGemmMaxPeers];
  int scatter_rows, scatter_rank;
  unsigned int *amax_bits;  // SWIGLU: bits of max|h|, a word per CTA; grouped: a word per group, raised
};

// Grouped launch (mixture-of-experts layers): the rows of the activation are sorted by group
// (expert) in segments padded to whole 256-row units; every unit multiplies with the weight of
// its own group.  unit_group[u] < 0 marks a unit without rows (skipped).
constexpr int kMaxGroups = 16;
struct GroupTable {
  CUtensorMap tm_w[kMaxGroups];
  const uint8_t *sfb_sparse[kMaxGroups];
  const uint8_t *sfb_dense[kMaxGroups];
  const int *unit_group;  // [units along M] on the device
  const float *alpha;     // [groups] on the device: per-group factor (activation scale x weight scale)
};

// Epilogue of 8 accumulator columns: o = bf16(alpha * acc + beta * c_in), then (+ bias) in bf16, packed.  Columns >= N
// read nothing; what they hold is masked by the caller's store.
__device__ __forceinline__ void epilogue_8(const GemmParams &p, const float (&acc)[8], int row, int col, float alpha, float beta,
                                           bool has_c, uint32_t (&o)[4]) {
  const bool full = (col + 8 <= p.n) && ((p.n & 7) == 0);
  float f[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) f[i] = alpha * acc[i];
  if (has_c) {
    const __nv_bfloat16 *c = p.c_in + (size_t)row * p.n + col;
    if (full && (reinterpret_cast<uintptr_t>(p.c_in) & 15) == 0) {
      uint4 cv = *reinterpret_cast<const uint4 *>(c);
      uint32_t cw[4] = {cv.x, cv.y, cv.z, cv.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        f[2 * i] = __fmaf_rn(beta, bf16_bits_to_float(cw[i] & 0xFFFFu), f[2 * i]);
        f[2 * i + 1] = __fmaf_rn(beta, bf16_bits_to_float(cw[i] >> 16), f[2 * i + 1]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (col + i < p.n) f[i] = __fmaf_rn(beta, __bfloat162float(c[i]), f[i]);
    }
  }
  // two values per conversion instruction (the scalar conversion unit is the slow pipe here)
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    __nv_bfloat162 pair = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    o[i] = *reinterpret_cast<uint32_t *>(&pair);
  }
  if (p.bias != nullptr) {
    // bias is added to the bf16 result, as a separate bf16 add would (a bf16 add rounds the
    // exact sum once, which is what the fp32 add + rounding of two bf16 values gives)
    if (full && (reinterpret_cast<uintptr_t>(p.bias) & 15) == 0) {
      const uint4 bv = *reinterpret_cast<const uint4 *>(p.bias + col);
      const uint32_t bw[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        __nv_bfloat162 sum = __hadd2(*reinterpret_cast<__nv_bfloat162 *>(&o[i]),
                                     *reinterpret_cast<const __nv_bfloat162 *>(&bw[i]));
        o[i] = *reinterpret_cast<uint32_t *>(&sum);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int cc = col + 2 * i;
        const float b0 = cc < p.n ? __bfloat162float(p.bias[cc]) : 0.0f;
        const float b1 = cc + 1 < p.n ? __bfloat162float(p.bias[cc + 1]) : 0.0f;
        const uint32_t lo = float_to_bf16_bits(bf16_bits_to_float(o[i] & 0xFFFFu) + b0);
        const uint32_t hi = float_to_bf16_bits(bf16_bits_to_float(o[i] >> 16) + b1);
        o[i] = lo | (hi << 16);
      }
    }
  }
}

// o + residual[off, off + 8), every sum rounded to bf16; off a multiple of 8.  In place of an add pass of 6 bytes per element behind a
// layer's last linear (8 us at 2048 x 4096, 48 us at 16384 x 3584).
__device__ __forceinline__ void add_residual_8(const GemmParams &p, uint32_t (&o)[4], size_t off) {
  const uint4 rv = __ldcg(reinterpret_cast<const uint4 *>(p.residual + off));  // read once; the plain load cost 8 bytes of spills
  const uint32_t rw[4] = {rv.x, rv.y, rv.z, rv.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    __nv_bfloat162 sum = __hadd2(*reinterpret_cast<__nv_bfloat162 *>(&o[i]), *reinterpret_cast<const __nv_bfloat162 *>(&rw[i]));
    o[i] = *reinterpret_cast<uint32_t *>(&sum);
  }
}

// 8 packed columns (+ residual) to row `row` of D; columns >= N are masked.
__device__ __forceinline__ void store_8(const GemmParams &p, uint32_t (&o)[4], int row, int col) {
  __nv_bfloat16 *d = p.d + (size_t)row * p.n + col;
  if (p.residual != nullptr) {
    if ((p.n & 7) == 0) {
      if (col + 8 <= p.n) add_residual_8(p, o, (size_t)row * p.n + col);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const __nv_bfloat16 *r = p.residual + (size_t)row * p.n + col + 2 * i;
        const float r0 = col + 2 * i < p.n ? __bfloat162float(r[0]) : 0.0f;
        const float r1 = col + 2 * i + 1 < p.n ? __bfloat162float(r[1]) : 0.0f;
        o[i] = float_to_bf16_bits(bf16_bits_to_float(o[i] & 0xFFFFu) + r0) |
               (float_to_bf16_bits(bf16_bits_to_float(o[i] >> 16) + r1) << 16);
      }
    }
  }
  if (col + 8 <= p.n && (p.n & 7) == 0 && (reinterpret_cast<uintptr_t>(p.d) & 15) == 0) {
    *reinterpret_cast<uint4 *>(d) = make_uint4(o[0], o[1], o[2], o[3]);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (col + i < p.n) d[i] = __ushort_as_bfloat16((unsigned short)((o[i >> 1] >> (16 * (i & 1))) & 0xFFFFu));
  }
}

// epilogue_8 on 32 columns.  Where all of them exist the loads of C_in (and then of the bias) are issued together: a load and its
// checks per 8 columns cost a latency each (28672 x 4096 at M = 127 with C_in 18.3 against 16.6 us).
__device__ __forceinline__ void epilogue_32(const GemmParams &p, const uint32_t *acc, int row, int col0, float alpha, float beta,
                                            bool has_c, uint32_t (&o)[4][4]) {
  const bool vec = col0 + 32 <= p.n && (p.n & 7) == 0 &&
                   ((reinterpret_cast<uintptr_t>(p.c_in) | reinterpret_cast<uintptr_t>(p.bias)) & 15) == 0;
  if (!vec) {
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      float f[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(acc[8 * v + i]);
      epilogue_8(p, f, row, col0 + 8 * v, alpha, beta, has_c, o[v]);
    }
    return;
  }
  auto pack = [](float a, float b) {
    __nv_bfloat162 pair = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&pair);
  };
  if (has_c) {
    const uint4 *c = reinterpret_cast<const uint4 *>(p.c_in + (size_t)row * p.n + col0);
    const uint4 cv[4] = {c[0], c[1], c[2], c[3]};
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const uint32_t cw[4] = {cv[v].x, cv[v].y, cv[v].z, cv[v].w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
        o[v][i] = pack(__fmaf_rn(beta, bf16_bits_to_float(cw[i] & 0xFFFFu), alpha * __uint_as_float(acc[8 * v + 2 * i])),
                       __fmaf_rn(beta, bf16_bits_to_float(cw[i] >> 16), alpha * __uint_as_float(acc[8 * v + 2 * i + 1])));
    }
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      o[i >> 2][i & 3] = pack(alpha * __uint_as_float(acc[2 * i]), alpha * __uint_as_float(acc[2 * i + 1]));
  }
  if (p.bias != nullptr) {
    const uint4 *b = reinterpret_cast<const uint4 *>(p.bias + col0);
    const uint4 bv[4] = {b[0], b[1], b[2], b[3]};
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const uint32_t bw[4] = {bv[v].x, bv[v].y, bv[v].z, bv[v].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 sum = __hadd2(*reinterpret_cast<__nv_bfloat162 *>(&o[v][i]), *reinterpret_cast<const __nv_bfloat162 *>(&bw[i]));
        o[v][i] = *reinterpret_cast<const uint32_t *>(&sum);
      }
    }
  }
}

// Epilogue of 32 accumulator columns held in registers; rows >= M and columns >= N are masked.  A thread owns one row
// and stores 64 contiguous bytes.
// With `stage` non-null the 64 bytes go to row `stage_row` of a 32-row x 64-byte shared-memory
// tile instead, 16-byte chunk v at position v ^ ((row >> 1) & 3) (no bank conflicts on the way in
// or out); the caller stores the tile and masks rows >= M and columns >= N; requires N % 8 == 0.
// kWide: the tile is 16 rows x 128 bytes (two calls fill a row: chunk_base 0 and 4), chunk c of a
// row at position c ^ (row & 7).
template <bool kWide = false>
__device__ __forceinline__ void epilogue_chunk(const GemmParams &p, const uint32_t *acc, int row, int col0, float alpha,
                                               float beta, bool has_c, uint8_t *stage = nullptr, int stage_row = 0,
                                               int chunk_base = 0) {
  if (stage == nullptr && (row >= p.m || col0 >= p.n)) return;
  if (row >= p.m || col0 >= p.n) has_c = false;  // masked by the caller's store; C_in must not be read out of range
  uint32_t all[4][4];
  epilogue_32(p, acc, row, col0, alpha, beta, has_c, all);
#pragma unroll
  for (int v = 0; v < 4; ++v) {  // 8 columns per 16-byte store
    uint32_t(&o)[4] = all[v];
    if (stage != nullptr) {
      uint8_t *slot = kWide ? stage + stage_row * 128 + (((chunk_base + v) ^ (stage_row & 7)) << 4)
                            : stage + stage_row * 64 + ((v ^ ((stage_row >> 1) & 3)) << 4);
      *reinterpret_cast<uint4 *>(slot) = make_uint4(o[0], o[1], o[2], o[3]);
    } else {
      store_8(p, o, row, col0 + 8 * v);
    }
  }
}

// SwiGLU of 32 columns held in registers: h = bf16(bf16(silu(g)) * u), g and u rounded to bf16 as the plain epilogue
// stores them, into the warp's staging tile (layout of epilogue_chunk); returns the packed max |h| of this row.
__device__ __forceinline__ __nv_bfloat162 swiglu_chunk(const uint32_t *gate, const uint32_t *up, float alpha, uint8_t *stage,
                                                       int stage_row) {
  __nv_bfloat162 mx = __floats2bfloat162_rn(0.0f, 0.0f);
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int j = 8 * v + 2 * i;
      const float2 g = __bfloat1622float2(
          __floats2bfloat162_rn(alpha * __uint_as_float(gate[j]), alpha * __uint_as_float(gate[j + 1])));
      const float2 w = __bfloat1622float2(__floats2bfloat162_rn(alpha * __uint_as_float(up[j]), alpha * __uint_as_float(up[j + 1])));
      const float2 s = __bfloat1622float2(__floats2bfloat162_rn(silu_f32(g.x), silu_f32(g.y)));
      const __nv_bfloat162 h = __floats2bfloat162_rn(__fmul_rn(s.x, w.x), __fmul_rn(s.y, w.y));
      mx = __hmax2(mx, __habs2(h));
      o[i] = *reinterpret_cast<const uint32_t *>(&h);
    }
    *reinterpret_cast<uint4 *>(stage + stage_row * 64 + ((v ^ ((stage_row >> 1) & 3)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
  }
  return mx;
}

__device__ __forceinline__ float warp_max(__nv_bfloat162 mx2) {
  float mx = fmaxf(__bfloat162float(mx2.x), __bfloat162float(mx2.y));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  return mx;
}

// Warp-wide maximum raised into *amax_bits (non-negative floats order like their bit patterns); the read first keeps
// most warps from an atomic once the maximum has settled.
__device__ __forceinline__ void raise_absmax(unsigned int *amax_bits, __nv_bfloat162 mx2, int lane) {
  const unsigned int bits = __float_as_uint(warp_max(mx2));
  if (lane == 0 && bits > *reinterpret_cast<volatile unsigned int *>(amax_bits)) atomicMax(amax_bits, bits);
}

// SWIGLU: the weight is a merged gate_up matrix [2F, k] and the launch writes h = silu(gate) * up [m, F] and max|h|
// instead of the product: a pair tile takes 128 gate rows (CTA 0's half of the weight tile) and the 128 up rows of the
// same columns (CTA 1's half), so that an epilogue thread holds both factors of its elements.  The separate SwiGLU pass reads
// and writes 6 bytes per element of h (41 us at 2048 x 14336, 300 us at 16384 x 18944, about its memory time); here the
// arithmetic hides behind the next tile's MMAs: whole layers 518 -> 487 us (2048 tokens) and 4.26 -> 3.85 ms (16384).
template <int BN, bool SPARSE, bool DENSE, bool PAIR, bool GROUPED, bool WIDE = false, bool SWIGLU = false>
__device__ __forceinline__ void gemm_body(const CUtensorMap &tm_w, const CUtensorMap &tm_a_dense, const CUtensorMap &tm_a_comp,
                                          const GemmParams &p, const GroupTable *gt) {
  using L = StageLayout<BN, SPARSE, DENSE, PAIR>;
  constexpr int S = L::kStages;
  constexpr int CG = PAIR ? 2 : 1;
  constexpr int kColsPerEpiWarp = BN / 2;  // two warps share each tensor-memory lane quadrant

  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t *full_bar = reinterpret_cast<uint64_t *>(smem + S * L::kStageBytes);
  uint64_t *empty_bar = full_bar + S;
  uint64_t *peer_bar = empty_bar + S;  // pair mode, leader CTA: "the peer has loaded stage s"
  uint64_t *acc_full_bar = peer_bar + S;
  uint64_t *acc_empty_bar = acc_full_bar + 1;
  uint64_t *recv_bar = acc_empty_bar + 1;  // split launch: the parts of this CTA's columns have arrived
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(recv_bar + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  volatile int *never_set = abort_flag + 1;  // for the wait that another role's abort does not end
  int4 *recv_tab = reinterpret_cast<int4 *>(smem + S * L::kStageBytes + 256);  // split launch, see recv_entry

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta_rank = PAIR ? ptx::cluster_ctarank() : 0u;
  const bool leader = cta_rank == 0;
  const int k_stages = (p.k + kBK - 1) / kBK;
  const int aligned_m = (p.m + 127) / 128 * 128;
  const int a_bands = aligned_m / 128;     // 128-row bands of the activation operands
  const int b_bands = (p.n + 127) / 128;   // 128-row bands of the weight scale factors
  const int tiles_sp = p.k / 128;  // 512-byte scale tiles per 128-row band, 32-group layout
  const int tiles_d = p.k / 64;    // same, 16-group layout
  // work units: a unit is one output tile of a CTA (128 x BN) or of a pair (256 x BN)
  const int m_units = PAIR ? (p.m + 255) / 256 : (p.m + kBM - 1) / kBM;
  const int n_tiles = (p.n + BN - 1) / BN;
  const int ffn = p.n >> 1;  // SWIGLU: columns of h (a multiple of 128)
  const int k_splits = p.k_splits;
  const int num_units = m_units * n_tiles;  // tiles M-fastest
  const int unit0 = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x / k_splits;
  const int unit_stride = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x / k_splits;
  // this CTA's share of the K stages
  const int k_rank = PAIR ? 0 : (int)blockIdx.x % k_splits;  // the rank in the cluster of a split launch
  const int it_begin = k_stages * k_rank / k_splits, it_end = k_stages * (k_rank + 1) / k_splits;
  const bool split = !PAIR && k_splits > 1;
  const int split_rows = split ? min(kBM, p.m - (unit0 % m_units) * kBM) : 0;  // the rows of the cluster's tile
  constexpr int kRuns = BN / 8;
  const Exchange exchange = !split ? kPull : (split_rows < kBM ? p.exchange_last : p.exchange);
  // What the senders need of a rank: byte offset of the tile's column 0 in row 0 of rank 0's part, bytes per row, its first run.
  auto recv_entry = [&](int rank) {
    const int run0 = first_run(rank, k_splits, kRuns);
    const int stride = 4 * (8 * (first_run(rank + 1, k_splits, kRuns) - run0) + kRecvPad);
    return make_int4(recv_slots<L>(rank, k_splits, split_rows, k_stages, kRuns).first * L::kStageBytes - 32 * run0, stride, run0, 0);
  };

  if (threadIdx.x == 32) {
    // fetch the tensor maps while the barriers and tensor memory are being set up
    if (!GROUPED) ptx::tma_prefetch_desc(&tm_w);
    if (DENSE) ptx::tma_prefetch_desc(&tm_a_dense);
    if (SPARSE) ptx::tma_prefetch_desc(&tm_a_comp);
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      ptx::mbar_init(full_bar + s, 1);
      ptx::mbar_init(empty_bar + s, 1);
      ptx::mbar_init(peer_bar + s, 1);
    }
    ptx::mbar_init(acc_full_bar, 1);
    ptx::mbar_init(acc_empty_bar, PAIR ? 2 * kEpiWarps : kEpiWarps);
    ptx::mbar_init(recv_bar, 1);
    *abort_flag = 0;
    *never_set = 0;
    ptx::fence_barrier_init();
    if (exchange != kPull) {
      // what arrives: the columns, and with a block copy their padding too
      const int cols = 8 * (first_run(k_rank + 1, k_splits, kRuns) - first_run(k_rank, k_splits, kRuns));
      ptx::mbar_arrive_expect_tx(recv_bar, (uint32_t)(k_splits * split_rows * 4 * (cols + (exchange == kSendBlocks ? kRecvPad : 0))));
    }
  }
  if (exchange != kPull && threadIdx.x >= 64 && (int)threadIdx.x - 64 < k_splits)
    recv_tab[threadIdx.x - 64] = recv_entry((int)threadIdx.x - 64);
  if (warp == 1) {
    ptx::tmem_alloc<CG>(tmem_slot, L::kTmemCols);
    ptx::tmem_relinquish<CG>();
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (PAIR) ptx::cluster_sync();  // both CTAs' barriers exist before any remote arrive
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  auto stage_bytes = [&](int it) {
    const int n_sp = SPARSE ? min(2, tiles_sp - 2 * it) : 0, n_d = DENSE ? min(4, tiles_d - 4 * it) : 0;
    return L::kWBytes + (uint32_t)p.a_rows * ((DENSE ? 128 : 0) + (SPARSE ? 64 : 0)) + L::kEBytes +
           (uint32_t)((n_sp + n_d) * 512 * (1 + L::kBands));
  };
  // The metadata and scale-factor copies are plain bulk copies without bounds checks.  A
  // tile may hang over the last 128-row band (the second CTA of a pair when ceil(M/128) is
  // odd, the second weight band of a 256-wide tile when ceil(N/128) is odd): such a band
  // is loaded from the last band that exists.  Its rows / columns are masked on output.
  auto load_weight = [&](int it, int s, int n_tile, const CUtensorMap *tw, const uint8_t *sfb_dense, const uint8_t *sfb_sparse) {
    uint8_t *st = smem + s * L::kStageBytes;
    ptx::tma_load_2d(st + L::kOffW, tw, it * 128,
                     SWIGLU ? n_tile * 128 + (int)cta_rank * ffn : n_tile * BN + (PAIR ? (int)cta_rank * (BN / 2) : 0), full_bar + s);
#pragma unroll
    for (int b = 0; b < L::kBands; ++b) {
      const size_t band = SWIGLU ? n_tile + b * (ffn / 128) : min(n_tile * L::kBands + b, b_bands - 1);
      if (DENSE)
        ptx::bulk_load_1d(st + L::kOffSfbD + b * 2048, sfb_dense + (band * tiles_d + 4 * (size_t)it) * 512,
                          (uint32_t)min(4, tiles_d - 4 * it) * 512, full_bar + s);
      if (SPARSE)
        ptx::bulk_load_1d(st + L::kOffSfbSp + b * 1024, sfb_sparse + (band * tiles_sp + 2 * (size_t)it) * 512,
                          (uint32_t)min(2, tiles_sp - 2 * it) * 512, full_bar + s);
    }
  };
  auto load_activation = [&](int it, int s, int m_tile) {
    uint8_t *st = smem + s * L::kStageBytes;
    const int a_band = min(m_tile, a_bands - 1);
    if (DENSE) {
      ptx::tma_load_2d(st + L::kOffADense, &tm_a_dense, it * 128, m_tile * kBM, full_bar + s);
      ptx::bulk_load_1d(st + L::kOffSfaD, p.sfa_dense + ((size_t)a_band * tiles_d + 4 * (size_t)it) * 512,
                        (uint32_t)min(4, tiles_d - 4 * it) * 512, full_bar + s);
    }
    if (SPARSE) {
      ptx::tma_load_2d(st + L::kOffAComp, &tm_a_comp, it * 64, m_tile * kBM, full_bar + s);
      ptx::bulk_load_1d(st + L::kOffE, p.e + ((size_t)it * aligned_m + (size_t)a_band * 128) * 16, 2048, full_bar + s);
      ptx::bulk_load_1d(st + L::kOffSfaSp, p.sfa_sparse + ((size_t)a_band * tiles_sp + 2 * (size_t)it) * 512,
                        (uint32_t)min(2, tiles_sp - 2 * it) * 512, full_bar + s);
    }
  };

  // The set-up above and the prefetch below overlap the end of the kernel that prepares the activation; from the wait on
  // every role reads or writes what earlier kernels may still use.  The prefetch goes to L2, where it cannot make stale data visible.
  // Loads of the weight into the ring ahead of the wait were no faster (linears of a layer with 8 to 128 tokens within 2 % either way): they get
  // in the prepare's way.
  if (!PAIR && warp == 0 && unit0 < num_units) {
    // weight tiles of this CTA's first stages: nothing of them depends on the activation
    if (ptx::elect_one()) {
      const int n_tile = unit0 / m_units;
      const int ahead = min(it_end, it_begin + kPrefetchStages);
      for (int it = it_begin; it < ahead; ++it) {
        ptx::tma_prefetch_l2_2d(&tm_w, it * 128, n_tile * BN);
#pragma unroll
        for (int b = 0; b < L::kBands; ++b) {
          const size_t band = (size_t)min(n_tile * L::kBands + b, b_bands - 1);
          if (DENSE)
            ptx::bulk_prefetch_l2(p.sfb_dense + (band * tiles_d + 4 * (size_t)it) * 512, (uint32_t)min(4, tiles_d - 4 * it) * 512);
          if (SPARSE)
            ptx::bulk_prefetch_l2(p.sfb_sparse + (band * tiles_sp + 2 * (size_t)it) * 512, (uint32_t)min(2, tiles_sp - 2 * it) * 512);
        }
      }
    }
    __syncwarp();
  }
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (ptx::elect_one()) {
      uint32_t g = 0;  // stages issued so far, across tiles
      bool ok = true;
      for (int u = unit0; u < num_units && ok; u += unit_stride) {
        const int tile = u;
        const int grp = GROUPED ? gt->unit_group[tile % m_units] : 0;
        if (GROUPED && grp < 0) continue;
        const CUtensorMap *tw = GROUPED ? &gt->tm_w[grp] : &tm_w;
        const uint8_t *sfb_dense = GROUPED ? gt->sfb_dense[grp] : p.sfb_dense;
        const uint8_t *sfb_sparse = GROUPED ? gt->sfb_sparse[grp] : p.sfb_sparse;
        const int m_tile = PAIR ? 2 * (tile % m_units) + (int)cta_rank : (tile % m_units);
        const int n_tile = tile / m_units;
        for (int it = it_begin; it < it_end; ++it, ++g) {
          const int s = (int)(g % S);
          if (!ptx::mbar_wait(empty_bar + s, ((g / S) & 1u) ^ 1u, abort_flag)) {
            *abort_flag = 1;
            report(p.error_flag, 1);
            ok = false;
            break;
          }
          ptx::mbar_arrive_expect_tx(full_bar + s, stage_bytes(it));
          load_weight(it, s, n_tile, tw, sfb_dense, sfb_sparse);
          load_activation(it, s, m_tile);
        }
      }
      if (exchange != kPull) {
        // the slots that take the received parts are free once their last stage has been consumed
        const RecvSlots slots = recv_slots<L>(k_rank, k_splits, split_rows, k_stages, kRuns);
        const int slot0 = slots.first, n = it_end - it_begin;
        for (int s = slot0; s < slot0 + slots.count && ok; ++s) {
          if (s >= n) continue;
          ok = ptx::mbar_wait(empty_bar + s, (uint32_t)((n - 1 - s) / S) & 1u, abort_flag);
          if (!ok) {
            *abort_flag = 1;
            report(p.error_flag, 6);
          }
        }
      }
    }
    if (split) {
      __syncwarp();
      ptx::cluster_arrive();
      ptx::cluster_wait();  // all CTAs can receive, or all parts are written
      ptx::cluster_arrive();
    }
  } else if (warp == 1) {
    if (split) ptx::cluster_arrive();
    if (ptx::elect_one()) {
      if (PAIR && !leader) {
        // ---------------------------------------------------------- peer CTA: report loaded stages
        uint32_t g = 0;
        bool ok = true;
        for (int u = unit0; u < num_units && ok; u += unit_stride) {
          if (GROUPED && gt->unit_group[u % m_units] < 0) continue;
          for (int it = it_begin; it < it_end; ++it, ++g) {
            const int s = (int)(g % S);
            if (!ptx::mbar_wait(full_bar + s, (g / S) & 1u, abort_flag)) {
              *abort_flag = 1;
              report(p.error_flag, 4);
              ok = false;
              break;
            }
            ptx::mbar_arrive_cluster(peer_bar + s, 0);
          }
        }
      } else {
        // ---------------------------------------------------------- MMA issuer
        constexpr uint32_t idesc_d = ptx::make_idesc_nvf4(PAIR ? 256 : kBM, BN, false);
        constexpr uint32_t idesc_s = ptx::make_idesc_nvf4(PAIR ? 256 : kBM, BN, true);
        uint32_t g = 0;
        uint32_t tile_iter = 0;
        bool ok = true;
        for (int u = unit0; u < num_units && ok; u += unit_stride) {
          if (GROUPED && gt->unit_group[u % m_units] < 0) continue;
          // the epilogue warps must have pulled the previous tile out of tensor memory
          const bool drained = PAIR ? ptx::mbar_wait_cluster(acc_empty_bar, (tile_iter & 1u) ^ 1u, abort_flag)
                                    : ptx::mbar_wait(acc_empty_bar, (tile_iter & 1u) ^ 1u, abort_flag);
          if (!drained) {
            *abort_flag = 1;
            report(p.error_flag, 5);
            break;
          }
          ptx::tc_fence_after();
          uint32_t accumulate = 0;
          for (int it = it_begin; it < it_end; ++it, ++g) {
            const int s = (int)(g % S);
            const uint32_t ph = (g / S) & 1u;
            bool got = ptx::mbar_wait(full_bar + s, ph, abort_flag);
            if (PAIR && got) got = ptx::mbar_wait_cluster(peer_bar + s, ph, abort_flag);
            if (!got) {
              *abort_flag = 1;
              report(p.error_flag, 2);
              ok = false;
              break;
            }
            ptx::tc_fence_after();
            const uint32_t st = ptx::smem_u32(smem + s * L::kStageBytes);
            const int n_sp = SPARSE ? min(2, tiles_sp - 2 * it) : 0;
            const int n_d = DENSE ? min(4, tiles_d - 4 * it) : 0;
            if (SPARSE) {
              ptx::tmem_cp_128x128b<CG>(tmem_base + L::kColE, ptx::make_smem_desc(st + L::kOffE, 128, 0, 0));
#pragma unroll
              for (int t = 0; t < 2; ++t) {
                if (t < n_sp) {
                  ptx::tmem_cp_32x128b_warpx4<CG>(tmem_base + L::kColSfaSp + 4 * t,
                                                  ptx::make_smem_desc(st + L::kOffSfaSp + t * 512, 128, 0, 0));
#pragma unroll
                  for (int b = 0; b < L::kBands; ++b)
                    ptx::tmem_cp_32x128b_warpx4<CG>(
                        tmem_base + L::kColSfbSp + t * (BN / 32) + 4 * b,
                        ptx::make_smem_desc(st + L::kOffSfbSp + b * 1024 + t * 512, 128, 0, 0));
                }
              }
            }
            if (DENSE) {
#pragma unroll
              for (int t = 0; t < 4; ++t) {
                if (t < n_d) {
                  ptx::tmem_cp_32x128b_warpx4<CG>(tmem_base + L::kColSfaD + 4 * t,
                                                  ptx::make_smem_desc(st + L::kOffSfaD + t * 512, 128, 0, 0));
#pragma unroll
                  for (int b = 0; b < L::kBands; ++b)
                    ptx::tmem_cp_32x128b_warpx4<CG>(
                        tmem_base + L::kColSfbD + t * (BN / 32) + 4 * b,
                        ptx::make_smem_desc(st + L::kOffSfbD + b * 2048 + t * 512, 128, 0, 0));
                }
              }
            }
            if (SPARSE) {
              // compressed A: 64-byte swizzled rows, 32 bytes (128 logical K) per MMA;
              // weight: 128-byte swizzled rows, 64 bytes (128 K) per MMA.
#pragma unroll
              for (int t = 0; t < 2; ++t) {
                if (t < n_sp) {
                  uint64_t da = ptx::make_smem_desc(st + L::kOffAComp + t * 32, 512, 16, 4);
                  uint64_t db = ptx::make_smem_desc(st + L::kOffW + t * 64, 1024, 16, 2);
                  ptx::mma_nvf4_sparse<CG>(tmem_base + L::kColAcc, da, db, idesc_s, tmem_base + L::kColSfaSp + 4 * t,
                                           tmem_base + L::kColSfbSp + t * (BN / 32), tmem_base + L::kColE + 2 * t,
                                           accumulate);
                  accumulate = 1;
                }
              }
            }
            if (DENSE) {
#pragma unroll
              for (int t = 0; t < 4; ++t) {
                if (t < n_d) {
                  uint64_t da = ptx::make_smem_desc(st + L::kOffADense + t * 32, 1024, 16, 2);
                  uint64_t db = ptx::make_smem_desc(st + L::kOffW + t * 32, 1024, 16, 2);
                  ptx::mma_nvf4_dense<CG>(tmem_base + L::kColAcc, da, db, idesc_d, tmem_base + L::kColSfaD + 4 * t,
                                          tmem_base + L::kColSfbD + t * (BN / 32), accumulate);
                  accumulate = 1;
                }
              }
            }
            if (PAIR)
              ptx::tc_commit_multicast2(empty_bar + s, 3);
            else
              ptx::tc_commit<1>(empty_bar + s);
          }
          if (ok) {
            if (PAIR)
              ptx::tc_commit_multicast2(acc_full_bar, 3);
            else
              ptx::tc_commit<1>(acc_full_bar);
          }
          ++tile_iter;
        }
      }
    }
    if (split) {
      __syncwarp();
      ptx::cluster_wait();
      ptx::cluster_arrive();
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..9)
    const int ew = warp - 2;
    const int quad = warp & 3;  // tensor-memory lane quadrant this warp may read
    const int half = ew >> 2;   // which half of the tile's columns
    const float alpha0 = p.alpha_ptr ? p.alpha * (*p.alpha_ptr) : p.alpha;
    const float beta = p.beta;
    const bool has_c = (p.c_in != nullptr) && (beta != 0.0f);
    // Output path: a lane holds one row of the accumulator, so a direct store instruction would
    // touch 32 different rows with 16 bytes each (32 memory lines per instruction).  Every
    // epilogue warp owns a 32-row x 64-byte shared-memory tile instead: 32 columns at a time are
    // converted into it (swizzled, conflict-free), read back with four lanes per row, and
    // stored as 8 rows x 64 contiguous bytes per instruction.
    uint8_t *stage = p.staged_store ? smem + S * L::kStageBytes + 512 + ew * 2048 : nullptr;
    uint32_t tile_iter = 0;
    __nv_bfloat162 h_max = __floats2bfloat162_rn(0.0f, 0.0f);  // SWIGLU: running max |h|
    auto wait_acc = [&]() {  // the next tile's accumulator is complete (uniform over the warp)
      bool ok = ptx::mbar_wait(acc_full_bar, tile_iter & 1u, abort_flag);
      ++tile_iter;
      if (!ok) {
        *abort_flag = 1;
        report(p.error_flag, 3);
      }
      ok = __all_sync(0xffffffffu, ok);
      ptx::tc_fence_after();
      return ok;
    };
    if constexpr (!PAIR && !SWIGLU && !WIDE) {
      if (exchange == kPull && split) {
        bool ok = wait_acc();
        const uint32_t part = ptx::smem_u32(smem);
        const int r0 = quad * 32 + lane;
        if (ok && quad * 32 < split_rows) {
          const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(L::kColAcc + half * kColsPerEpiWarp);
#pragma unroll 1
          for (int c = 0; c < kColsPerEpiWarp / 32; ++c) {
            uint32_t acc[32];
            ptx::tmem_ld_32x32b_x32(taddr + 32 * c, acc);
            ptx::tmem_ld_wait();
            if (r0 < split_rows) {
              uint4 *dst = reinterpret_cast<uint4 *>(smem + ((size_t)r0 * L::kPartStride + half * kColsPerEpiWarp + 32 * c) * 4);
#pragma unroll
              for (int v = 0; v < 8; ++v) dst[v] = make_uint4(acc[4 * v], acc[4 * v + 1], acc[4 * v + 2], acc[4 * v + 3]);
            }
          }
        }
        __syncwarp();
        ptx::cluster_arrive();
        ptx::cluster_wait();  // every CTA's part is written
        const int m_tile = unit0 % m_units, n_tile = unit0 / m_units;
        // 8 columns per thread, dealt over the threads of all CTAs: neighbouring lanes read neighbouring 32 bytes
        for (int i = (int)threadIdx.x - 64 + k_rank * 32 * kEpiWarps; i < split_rows * kRuns && ok; i += k_splits * 32 * kEpiWarps) {
          const int r = i / kRuns, c8 = i % kRuns;
          const int row = m_tile * kBM + r, col = n_tile * BN + 8 * c8;
          if (col >= p.n) continue;
          const uint32_t at = part + (uint32_t)(r * L::kPartStride + 8 * c8) * 4u;
          float4 lo[kMaxSplits], hi[kMaxSplits];
#pragma unroll
          for (int s = 0; s < kMaxSplits; ++s) {
            if (s < k_splits) {
              lo[s] = ptx::ld_cluster_f32x4(at, s);
              hi[s] = ptx::ld_cluster_f32x4(at + 16, s);
            }
          }
          float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int s = 0; s < kMaxSplits; ++s) {
            if (s < k_splits) {
              f[0] += lo[s].x, f[1] += lo[s].y, f[2] += lo[s].z, f[3] += lo[s].w;
              f[4] += hi[s].x, f[5] += hi[s].y, f[6] += hi[s].z, f[7] += hi[s].w;
            }
          }
          uint32_t o[4];
          epilogue_8(p, f, row, col, alpha0, beta, has_c, o);
          store_8(p, o, row, col);
        }
        __syncwarp();
        ptx::cluster_arrive();
      } else if (split) {
        // The first of two passes only runs the code of the sum on one item, unstored, while the stages are still being
        // consumed: fetched when the last stage is done, it took longer than the sum.  From the last stage's MMAs to the end of the
        // launch 4096 x 4096 at M = 32 takes 2.6 us (3.6 with a cluster barrier, a sum that reads the other CTAs' memory, and a second
        // barrier), at M = 1 1.5 (2.6).
        const int run0 = first_run(k_rank, k_splits, kRuns), n_runs = first_run(k_rank + 1, k_splits, kRuns) - run0;
        const int m_tile = unit0 % m_units, n_tile = unit0 / m_units;
        const uint32_t ring = ptx::smem_u32(smem);
        const int items = split_rows * n_runs;
        bool ok = true;
        ptx::cluster_arrive();
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
          if (pass == 1) {
            ok = wait_acc();
            ptx::cluster_wait();  // all CTAs can receive
            const int r = quad * 32 + lane;
            const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(L::kColAcc + half * kColsPerEpiWarp);
            if (exchange == kSendBlocks) {
              const int send = send_slot<L>(k_rank, k_splits, split_rows, k_stages, BN) * L::kStageBytes;
              if (ok && quad * 32 < split_rows) {
#pragma unroll 1
                for (int c = 0; c < kColsPerEpiWarp / 32; ++c) {
                  uint32_t acc[32];
                  ptx::tmem_ld_32x32b_x32(taddr + 32 * c, acc);
                  ptx::tmem_ld_wait();
                  if (r < split_rows) {
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                      const int run = (half * kColsPerEpiWarp + 32 * c) / 8 + v;
                      const int owner = run * k_splits / kRuns;
                      const int4 entry = recv_tab[owner];
                      // the blocks ahead hold run0 runs and `owner` paddings per row
                      uint4 *dst = reinterpret_cast<uint4 *>(smem + send + split_rows * (32 * entry.z + 4 * kRecvPad * owner) +
                                                             r * entry.y + 32 * (run - entry.z));
                      dst[0] = make_uint4(acc[8 * v], acc[8 * v + 1], acc[8 * v + 2], acc[8 * v + 3]);
                      dst[1] = make_uint4(acc[8 * v + 4], acc[8 * v + 5], acc[8 * v + 6], acc[8 * v + 7]);
                    }
                  }
                }
              }
              ptx::fence_proxy_async();
              ptx::named_sync(1, 32 * kEpiWarps);
              if (ok && ew == 0 && lane < k_splits) {
                const int4 entry = recv_tab[lane];
                ptx::bulk_copy_cluster(ring + (uint32_t)(entry.x + k_rank * split_rows * entry.y + 32 * entry.z),
                                       smem + send + split_rows * (32 * entry.z + 4 * kRecvPad * lane), (uint32_t)(split_rows * entry.y),
                                       recv_bar, lane);
              }
            } else if (ok && quad * 32 < split_rows) {
#pragma unroll 1
              for (int c = 0; c < kColsPerEpiWarp / 32; ++c) {
                uint32_t acc[32];
                ptx::tmem_ld_32x32b_x32(taddr + 32 * c, acc);
                ptx::tmem_ld_wait();
                if (r < split_rows) {
#pragma unroll
                  for (int v = 0; v < 4; ++v) {
                    const int run = (half * kColsPerEpiWarp + 32 * c) / 8 + v;
                    const int owner = run * k_splits / kRuns;
                    const int4 entry = recv_tab[owner];
                    const uint32_t at = ring + (uint32_t)(entry.x + (k_rank * split_rows + r) * entry.y + 32 * run);
                    ptx::st_async_cluster_x4(at, recv_bar, owner, acc[8 * v], acc[8 * v + 1], acc[8 * v + 2], acc[8 * v + 3]);
                    ptx::st_async_cluster_x4(at + 16, recv_bar, owner, acc[8 * v + 4], acc[8 * v + 5], acc[8 * v + 6], acc[8 * v + 7]);
                  }
                }
              }
            }
            __syncwarp();
            // A CTA may leave once its parts are on their way; where they may be read from its memory, once they have arrived.
            if (exchange == kSendRegisters) ptx::cluster_arrive();
            // parts that are under way are waited for also when another role has given up
            if (!ptx::mbar_wait_cluster_acquire(recv_bar, 0, never_set)) {
              *abort_flag = 1;
              report(p.error_flag, 7);
              ok = false;
            }
            ok = __all_sync(0xffffffffu, ok);
            if (exchange == kSendBlocks) ptx::cluster_arrive();
          }
#pragma unroll 1
          for (int i = (int)threadIdx.x - 64; i < items && ok; i += 32 * kEpiWarps) {
            const int r = i / n_runs, c8 = i % n_runs;
            const int row = m_tile * kBM + r, col = n_tile * BN + 8 * (run0 + c8);
            if (col >= p.n) continue;
            float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            const int4 entry = recv_tab[k_rank];
            const uint32_t at = ring + (uint32_t)(entry.x + r * entry.y + 32 * (run0 + c8)), step = (uint32_t)(split_rows * entry.y);
#pragma unroll
            for (int s = 0; s < kMaxSplits; ++s) {
              if (s < k_splits) {
                const float4 lo = ptx::ld_shared_f32x4(at + s * step), hi = ptx::ld_shared_f32x4(at + s * step + 16);
                f[0] += lo.x, f[1] += lo.y, f[2] += lo.z, f[3] += lo.w;
                f[4] += hi.x, f[5] += hi.y, f[6] += hi.z, f[7] += hi.w;
              }
            }
            uint32_t o[4];
            epilogue_8(p, f, row, col, alpha0, beta, has_c, o);
            asm volatile("" : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]));  // computed in both passes
            if (pass == 0) break;
            store_8(p, o, row, col);
          }
        }
      }
    }
    for (int u = unit0; u < num_units && !split; u += unit_stride) {
      const int tile = u;
      const int grp = GROUPED ? gt->unit_group[tile % m_units] : 0;
      if (GROUPED && grp < 0) continue;
      const float alpha = GROUPED ? alpha0 * gt->alpha[grp] : alpha0;
      const int m_tile = PAIR ? 2 * (tile % m_units) + (int)cta_rank : (tile % m_units);
      const int n_tile = tile / m_units;
      if constexpr (!SWIGLU && !WIDE) {
        if (stage != nullptr && u + unit_stride >= num_units) {
          // The CTA's last tile: nothing waits for the tensor memory, so it is drained 32 columns at a time by a loop whose code is
          // a quarter of the unrolled form's, and which runs once on no rows ahead of the wait (28672 x 4096 at M = 32: 3.0 us behind the last MMA against 4.6, of which 2.8 went into
          // fetching code).
          const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(L::kColAcc + half * kColsPerEpiWarp);
          const int row0 = m_tile * kBM + quad * 32;
          bool ok = true;
#pragma unroll 1
          for (int c = -1; c < kColsPerEpiWarp / 32; ++c) {
            uint32_t acc[32] = {};
            if (c == 0) ok = wait_acc();
            if (!ok) break;
            if (c >= 0) {
              ptx::tmem_ld_32x32b_x32(taddr + 32 * c, acc);
              ptx::tmem_ld_wait();
            }
            const int rows = c < 0 ? 0 : p.m, col0 = n_tile * BN + half * kColsPerEpiWarp + 32 * max(c, 0);
            epilogue_chunk(p, acc, c < 0 ? p.m : row0 + lane, col0, alpha, beta, has_c, stage, lane);
            __syncwarp();
            const int gcol = col0 + (lane & 3) * 8;
#pragma unroll
            for (int it = 0; it < 4; ++it) {
              const int r = it * 8 + (lane >> 2);
              const uint4 v = *reinterpret_cast<const uint4 *>(stage + r * 64 + (((lane & 3) ^ ((r >> 1) & 3)) << 4));
              if (row0 + r < rows && gcol < p.n) {
                const size_t off = (size_t)(row0 + r) * p.n + gcol;
                uint32_t o[4] = {v.x, v.y, v.z, v.w};
                if (p.residual != nullptr) add_residual_8(p, o, off);
                *reinterpret_cast<uint4 *>(p.d + off) = make_uint4(o[0], o[1], o[2], o[3]);
              }
            }
            __syncwarp();
          }
          break;
        }
      }
      if (!wait_acc()) break;
      uint32_t acc[kColsPerEpiWarp];
      // SWIGLU: 64 gate columns and the 64 up columns that belong to them, else neighbouring columns
      const uint32_t taddr =
          tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(L::kColAcc + half * (SWIGLU ? 64 : kColsPerEpiWarp));
#pragma unroll
      for (int c = 0; c < kColsPerEpiWarp / 32; ++c)
        ptx::tmem_ld_32x32b_x32(taddr + (SWIGLU ? 32 * (c & 1) + 128 * (c >> 1) : 32 * c),
                                *reinterpret_cast<uint32_t(*)[32]>(&acc[32 * c]));
      ptx::tmem_ld_wait();
      // the accumulator is in registers: give tensor memory back before the slow part
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR && !leader)
          ptx::mbar_arrive_cluster(acc_empty_bar, 0);
        else
          ptx::mbar_arrive(acc_empty_bar);
      }
      const int row = m_tile * kBM + quad * 32 + lane;
      const int col_base = n_tile * BN + half * kColsPerEpiWarp;
      if constexpr (SWIGLU) {
        const int row0 = m_tile * kBM + quad * 32;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const __nv_bfloat162 mx = swiglu_chunk(&acc[32 * c], &acc[64 + 32 * c], alpha, stage, lane);
          if (row < p.m) h_max = __hmax2(h_max, mx);
          __syncwarp();
          const int gcol = n_tile * 128 + half * 64 + 32 * c + (lane & 3) * 8;
#pragma unroll
          for (int it = 0; it < 4; ++it) {
            const int r = it * 8 + (lane >> 2);
            const uint4 v = *reinterpret_cast<const uint4 *>(stage + r * 64 + (((lane & 3) ^ ((r >> 1) & 3)) << 4));
            if (row0 + r < p.m) *reinterpret_cast<uint4 *>(p.d + (size_t)(row0 + r) * ffn + gcol) = v;
          }
          __syncwarp();
        }
        if (GROUPED) {  // the unit's rows belong to one group
          raise_absmax(p.amax_bits + grp, h_max, lane);
          h_max = __floats2bfloat162_rn(0.0f, 0.0f);
        }
        continue;
      }
      if (stage != nullptr) {
        const int row0 = m_tile * kBM + quad * 32;
        __nv_bfloat16 *d_base = p.d;
        if (p.scatter_rows > 0) {
          const int owner = (m_tile * kBM) / p.scatter_rows;
          d_base = p.d_peer[owner] + ((long long)p.scatter_rank - owner) * p.scatter_rows * (long long)p.n;
        }
        if (WIDE) {
          // Scatter mode (rows that go to another GPU): a peer store moves 18 % more bytes per second in 128-byte
          // row pieces than in 64-byte ones (measured 605 against 511 GB/s), so the tile is staged
          // 64 columns at a time in two halves of 16 rows (the lanes of the other half wait) and
          // stored as 4 rows x 128 contiguous bytes per instruction.
#pragma unroll
          for (int c = 0; c < kColsPerEpiWarp / 64; ++c) {
            const int col0 = col_base + 64 * c;
            const int gcol = col0 + (lane & 7) * 8;
#pragma unroll 1
            for (int hrow = 0; hrow < 2; ++hrow) {
              if ((lane >> 4) == hrow) {
                epilogue_chunk<true>(p, &acc[64 * c], row, col0, alpha, beta, false, stage, lane & 15, 0);
                epilogue_chunk<true>(p, &acc[64 * c + 32], row, col0 + 32, alpha, beta, false, stage, lane & 15, 4);
              }
              __syncwarp();
#pragma unroll
              for (int it = 0; it < 4; ++it) {
                const int r = it * 4 + (lane >> 3);
                const uint4 v = *reinterpret_cast<const uint4 *>(stage + r * 128 + (((lane & 7) ^ (r & 7)) << 4));
                const int grow = row0 + 16 * hrow + r;
                if (grow < p.m && gcol < p.n) *reinterpret_cast<uint4 *>(d_base + (size_t)grow * p.n + gcol) = v;
              }
              __syncwarp();
            }
          }
          continue;
        }
#pragma unroll
        for (int c = 0; c < kColsPerEpiWarp / 32; ++c) {
          const int col0 = col_base + 32 * c;
          epilogue_chunk(p, &acc[32 * c], row, col0, alpha, beta, has_c, stage, lane);
          __syncwarp();
          const int gcol = col0 + (lane & 3) * 8;
#pragma unroll
          for (int it = 0; it < 4; ++it) {
            const int r = it * 8 + (lane >> 2);
            const uint4 v = *reinterpret_cast<const uint4 *>(stage + r * 64 + (((lane & 3) ^ ((r >> 1) & 3)) << 4));
            if (row0 + r < p.m && gcol < p.n) {
              const size_t off = (size_t)(row0 + r) * p.n + gcol;
              uint32_t o[4] = {v.x, v.y, v.z, v.w};
              if (p.residual != nullptr) add_residual_8(p, o, off);
              *reinterpret_cast<uint4 *>(d_base + off) = make_uint4(o[0], o[1], o[2], o[3]);
            }
          }
          __syncwarp();
        }
      } else {
#pragma unroll
        for (int c = 0; c < kColsPerEpiWarp / 32; ++c)
          epilogue_chunk(p, &acc[32 * c], row, col_base + 32 * c, alpha, beta, has_c);
      }
    }
    if (SWIGLU && !GROUPED) {
      const float mx = warp_max(h_max);
      if (lane == 0) reinterpret_cast<float *>(smem + S * L::kStageBytes + 256)[ew] = mx;
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (SWIGLU && !GROUPED && threadIdx.x == 0) {
    const float *mx = reinterpret_cast<const float *>(smem + S * L::kStageBytes + 256);  // behind the barriers
    float cta = mx[0];
#pragma unroll
    for (int w = 1; w < kEpiWarps; ++w) cta = fmaxf(cta, mx[w]);
    p.amax_bits[blockIdx.x] = __float_as_uint(cta);
  }
  if (split) ptx::cluster_wait();  // no CTA is sent to or read from any more
  if (PAIR) ptx::cluster_sync();  // neither CTA leaves (or frees tensor memory) while its peer may still use it
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc<CG>(tmem_base, L::kTmemCols);
  }
}

// WIDE: the scatter-mode epilogue (128-byte row pieces for the peer stores), its own instantiation so
// that the other kernels keep their register allocation.
template <int BN, bool SPARSE, bool DENSE, bool PAIR, bool WIDE = false, bool SWIGLU = false>
__global__ void __launch_bounds__(kGemmThreads, 1)
    gemm_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_a_dense,
                const __grid_constant__ CUtensorMap tm_a_comp, const GemmParams p) {
  gemm_body<BN, SPARSE, DENSE, PAIR, false, WIDE, SWIGLU>(tm_w, tm_a_dense, tm_a_comp, p, nullptr);
}

// The fused SharQ GEMM of all groups (experts) of a mixture-of-experts layer in one launch, CTA pairs.
template <bool SWIGLU>
__global__ void __launch_bounds__(kGemmThreads, 1)
    gemm_grouped_kernel(const __grid_constant__ GroupTable groups, const __grid_constant__ CUtensorMap tm_a_dense,
                        const __grid_constant__ CUtensorMap tm_a_comp, const GemmParams p) {
  gemm_body<256, true, true, true, true, false, SWIGLU>(groups.tm_w[0], tm_a_dense, tm_a_comp, p, &groups);
}

// ------------------------------------------------------------------ host side

using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  });
  return fn;
}

// 2-D byte tensor [rows, row_bytes] with a [box_rows, box_bytes] box.
bool make_tmap_bytes(CUtensorMap *map, const void *base, uint64_t rows, uint64_t row_bytes, uint32_t box_rows,
                     uint32_t box_bytes, CUtensorMapSwizzle swizzle) {
  EncodeTiledFn fn = get_encode_fn();
  if (fn == nullptr) return false;
  cuuint64_t dims[2] = {row_bytes, rows};
  cuuint64_t strides[1] = {row_bytes};
  cuuint32_t box[2] = {box_bytes, box_rows};
  cuuint32_t elem_strides[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box, elem_strides,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

struct DeviceInfo {
  bool known = false;
  int sms = 0;
};

// Per-device state: SM count and which kernel instantiations already have their
// shared-memory attribute set.
cudaError_t device_info(int *dev_out, int *sms_out) {
  static DeviceInfo info[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!info[dev].known) {
    e = cudaDeviceGetAttribute(&info[dev].sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    info[dev].known = true;
  }
  *dev_out = dev;
  *sms_out = info[dev].sms;
  return cudaSuccess;
}

template <int BN, bool SPARSE, bool DENSE, bool PAIR, bool WIDE = false, bool SWIGLU = false>
cudaError_t launch(const GemmArgs &a, cudaStream_t stream) {
  using L = StageLayout<BN, SPARSE, DENSE, PAIR>;
  static bool attr_set[64] = {};
  auto kernel = gemm_kernel<BN, SPARSE, DENSE, PAIR, WIDE, SWIGLU>;
  int dev = 0, sms = 0;
  cudaError_t e = device_info(&dev, &sms);
  if (e != cudaSuccess) return e;
  if (!attr_set[dev]) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kSmemBytes);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  CUtensorMap tm_w, tm_ad, tm_ac;
  memset(&tm_ad, 0, sizeof(tm_ad));
  memset(&tm_ac, 0, sizeof(tm_ac));
  if (!make_tmap_bytes(&tm_w, a.b, (uint64_t)a.n, (uint64_t)a.k / 2, L::kWRows, 128, CU_TENSOR_MAP_SWIZZLE_128B))
    return cudaErrorInvalidValue;
  // With one tile of rows only those that exist are loaded (whole 8-row groups of the swizzle): a 128-row box of a decode batch
  // is mostly zero fill, 24 of the 67 KB that a stage writes to shared memory.  The MMA then reads stale bytes for
  // the other rows, and whatever scales their padding holds (the dense quantisation leaves it unwritten): the rows of an
  // accumulator are independent, and those are masked.
  const int a_rows = !PAIR && a.m < kBM ? (a.m + 7) / 8 * 8 : kBM;
  if (DENSE && !make_tmap_bytes(&tm_ad, a.a_dense, (uint64_t)a.m, (uint64_t)a.k / 2, a_rows, 128, CU_TENSOR_MAP_SWIZZLE_128B))
    return cudaErrorInvalidValue;
  if (SPARSE && !make_tmap_bytes(&tm_ac, a.a_comp, (uint64_t)a.m, (uint64_t)a.k / 4, a_rows, 64, CU_TENSOR_MAP_SWIZZLE_64B))
    return cudaErrorInvalidValue;
  GemmParams p{};
  p.a_rows = a_rows;
  p.staged_store = (a.n % 8 == 0) && ((reinterpret_cast<uintptr_t>(a.scatter_world > 1 ? a.d_peer[0] : a.d) & 15) == 0);
  p.e = static_cast<const uint8_t *>(a.e);
  p.sfa_sparse = static_cast<const uint8_t *>(a.sfa_sparse);
  p.sfa_dense = static_cast<const uint8_t *>(a.sfa_dense);
  p.sfb_sparse = static_cast<const uint8_t *>(a.sfb_sparse);
  p.sfb_dense = static_cast<const uint8_t *>(a.sfb_dense);
  p.c_in = static_cast<const __nv_bfloat16 *>(a.c_in);
  p.bias = static_cast<const __nv_bfloat16 *>(a.bias);
  if (a.residual != nullptr && ((reinterpret_cast<uintptr_t>(a.residual) & 15) != 0 || a.scatter_world > 1 || SWIGLU))
    return cudaErrorInvalidValue;
  p.residual = static_cast<const __nv_bfloat16 *>(a.residual);
  p.d = static_cast<__nv_bfloat16 *>(a.d);
  p.alpha_ptr = a.alpha_ptr;
  p.alpha = a.alpha;
  p.beta = a.beta;
  p.m = a.m;
  p.n = a.n;
  p.k = a.k;
  p.error_flag = a.error_flag;
  p.amax_bits = a.amax_bits;
  p.scatter_rows = 0;
  if (a.scatter_world > 1) {
    // dealing rows to their owners needs whole 128-row tiles per owner and the coalesced store path
    if (a.scatter_world > kGemmMaxPeers || a.m % (128 * a.scatter_world) != 0 || !p.staged_store || a.c_in != nullptr)
      return cudaErrorInvalidValue;
    for (int r = 0; r < a.scatter_world; ++r) {
      if (a.d_peer[r] == nullptr || (reinterpret_cast<uintptr_t>(a.d_peer[r]) & 15) != 0) return cudaErrorInvalidValue;
      p.d_peer[r] = static_cast<__nv_bfloat16 *>(a.d_peer[r]);
    }
    p.scatter_rows = a.m / a.scatter_world;
    p.scatter_rank = a.scatter_rank;
  }
  const int n_tiles = (a.n + BN - 1) / BN;
  const int m_units = PAIR ? (a.m + 255) / 256 : (a.m + kBM - 1) / kBM;
  const int units = m_units * n_tiles;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  // see grid_dependency_wait in gemm_body; the linears of a 32-token decode step 90.8 -> 83.6 us, of 2048 tokens 429.6 -> 423.6
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 1;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  cfg.blockDim = dim3(kGemmThreads);
  cfg.dynamicSmemBytes = L::kSmemBytes;
  cfg.stream = stream;
  p.k_splits = 1;
  if (PAIR) {
    const int clusters = units < sms / 2 ? units : sms / 2;
    cfg.gridDim = dim3(2 * clusters);
    attr[1].val.clusterDim.x = 2;
  } else {
    // Split K where the tiles alone leave SMs idle (few rows: the launch is bound by streaming the weights, which
    // takes as many SMs as possible): the most CTAs per tile for which all clusters run at the same time, each
    // with at least two K stages.  Sums through distributed shared memory took the place of a memset, fp32 atomics and a
    // second kernel (4.5 us of 20 per launch at M = 32), for which only M <= 64 or K >= 8192 had paid.
    // The sum costs more the more rows a tile has and is set against K stages of 0.40 us (fused), 0.30 (dense) or 0.23 (sparse): split / one
    // pass of 4096 x 1024 at M = 129 took 8.6 / 6.4 us, 768 x 4096 sparse at M = 256 10.9 / 8.0, 1024 x 2048 at M = 64 7.0 / 7.2 and at M = 1 5.0 / 7.0,
    // 512 x 8192 at M = 256 12.1 / 16.8.  The line below lies within 6 % of the better form over M = 1 to 512, N = 128 to 6144, K = 512 to
    // 14336, but for 11 % at 16 x 4096 x 2048 sparse.  Rows of D that allow no 16-byte stores (N % 8 != 0) are always better dealt over
    // the threads of a cluster (300 x 1152 at M = 128 9.0 / 23.1 us).
    const int k_stages = (a.k + kBK - 1) / kBK;
    const int rows = a.m < kBM ? a.m : kBM;
    const bool split_pays = p.staged_store == 0 || k_stages >= 4 + rows / (SPARSE && DENSE ? 9 : (DENSE ? 8 : 5));
    if (a.split_k && split_pays && a.scatter_world <= 1) {
      static int capacity[64][kMaxSplits + 1] = {};  // clusters of a size that the device holds at once; 0 = not asked yet
      int s = k_stages / 2 < kMaxSplits ? k_stages / 2 : kMaxSplits;
      if (s > sms / units) s = sms / units;
      for (; s >= 2; --s) {
        if (capacity[dev][s] == 0) {
          attr[1].val.clusterDim.x = (unsigned)s;
          cudaLaunchConfig_t ask = cfg;
          ask.gridDim = dim3((unsigned)s);
          ask.attrs = attr + 1;
          ask.numAttrs = 1;
          int n = 0;
          if (cudaOccupancyMaxActiveClusters(&n, kernel, &ask) != cudaSuccess) {
            (void)cudaGetLastError();
            n = 0;
          }
          capacity[dev][s] = n > 0 ? n : -1;
        }
        if (capacity[dev][s] >= units) break;
      }
      if (s >= 2) {
        p.k_splits = s;
        p.exchange = exchange_form<L>(kBM, s, k_stages, BN);
        p.exchange_last = exchange_form<L>(a.m - (m_units - 1) * kBM, s, k_stages, BN);
      }
    }
    attr[1].val.clusterDim.x = (unsigned)p.k_splits;
    cfg.gridDim = dim3(p.k_splits > 1 ? units * p.k_splits : (units < sms ? units : sms));
    if (p.k_splits == 1) cfg.numAttrs = 1;
  }
  return cudaLaunchKernelEx(&cfg, kernel, tm_w, tm_ad, tm_ac, p);
}

}  // namespace

template <bool SWIGLU>
static cudaError_t launch_grouped(const GroupedGemmArgs &a, cudaStream_t stream) {
  using L = StageLayout<256, true, true, true>;
  static bool attr_set[64] = {};
  auto kernel = gemm_grouped_kernel<SWIGLU>;
  if (a.groups < 1 || a.groups > kMaxGroups || a.m <= 0 || a.m % 256 != 0 || a.n <= 0 || a.k <= 0 || a.k % 128 != 0)
    return cudaErrorInvalidValue;
  int dev = 0, sms = 0;
  cudaError_t e = device_info(&dev, &sms);
  if (e != cudaSuccess) return e;
  if (!attr_set[dev]) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kSmemBytes);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  GroupTable gt;
  memset(&gt, 0, sizeof(gt));
  for (int g = 0; g < a.groups; ++g) {
    if (!make_tmap_bytes(&gt.tm_w[g], a.b[g], (uint64_t)a.n, (uint64_t)a.k / 2, L::kWRows, 128, CU_TENSOR_MAP_SWIZZLE_128B))
      return cudaErrorInvalidValue;
    gt.sfb_sparse[g] = static_cast<const uint8_t *>(a.sfb_sparse[g]);
    gt.sfb_dense[g] = static_cast<const uint8_t *>(a.sfb_dense[g]);
  }
  gt.unit_group = a.unit_group;
  gt.alpha = a.alpha_vec;
  CUtensorMap tm_ad, tm_ac;
  if (!make_tmap_bytes(&tm_ad, a.a_dense, (uint64_t)a.m, (uint64_t)a.k / 2, kBM, 128, CU_TENSOR_MAP_SWIZZLE_128B))
    return cudaErrorInvalidValue;
  if (!make_tmap_bytes(&tm_ac, a.a_comp, (uint64_t)a.m, (uint64_t)a.k / 4, kBM, 64, CU_TENSOR_MAP_SWIZZLE_64B))
    return cudaErrorInvalidValue;
  GemmParams p{};
  p.a_rows = kBM;
  p.staged_store = (a.n % 8 == 0) && ((reinterpret_cast<uintptr_t>(a.d) & 15) == 0);
  p.e = static_cast<const uint8_t *>(a.e);
  p.sfa_sparse = static_cast<const uint8_t *>(a.sfa_sparse);
  p.sfa_dense = static_cast<const uint8_t *>(a.sfa_dense);
  p.d = static_cast<__nv_bfloat16 *>(a.d);
  p.alpha = a.alpha;
  p.m = a.m;
  p.n = a.n;
  p.k = a.k;
  p.error_flag = a.error_flag;
  p.amax_bits = a.amax_bits;
  p.k_splits = 1;
  const int units = (a.m / 256) * ((a.n + 255) / 256);
  const int clusters = units < sms / 2 ? units : sms / 2;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(2 * clusters);
  cfg.blockDim = dim3(kGemmThreads);
  cfg.dynamicSmemBytes = L::kSmemBytes;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, gt, tm_ad, tm_ac, p);
}

// What the SWIGLU epilogue takes: whole 128-column bands of gate and up, 16-byte aligned rows of h.
static bool swiglu_ok(int n, const void *d, const unsigned int *amax_bits) {
  return n > 0 && n % 256 == 0 && (reinterpret_cast<uintptr_t>(d) & 15) == 0 && amax_bits != nullptr;
}

cudaError_t run_gemm_grouped(const GroupedGemmArgs &a, cudaStream_t stream) {
  if (a.amax_bits == nullptr) return launch_grouped<false>(a, stream);
  if (a.groups < 1 || a.groups > kMaxGroups || !swiglu_ok(a.n, a.d, a.amax_bits)) return cudaErrorInvalidValue;
  cudaError_t e = cudaMemsetAsync(a.amax_bits, 0, sizeof(unsigned int) * a.groups, stream);
  return e != cudaSuccess ? e : launch_grouped<true>(a, stream);
}

int gemm_tile_n(int m, int n, int k, bool split_k, int sms) {
  const int pair_units = ((m + 255) / 256) * ((n + 255) / 256);
  const int units_128 = ((m + 127) / 128) * ((n + 127) / 128);
  const int units_256 = ((m + 127) / 128) * ((n + 255) / 256);
  if (m <= 128 || n <= 128) {
    // one row of tiles: narrow ones while they fit the GPU at once (split K fills it: 4096 x 4096 at M = 32 / 128 8.1 / 11.1 us
    // against 9.7 / 16.3 with 256-wide tiles, 4096 x 14336 13.7 / 16.4 against 15.8 / 22.5; without split K 10.3 / 10.9 against
    // 14.7 / 16.2 and 26.2 / 27.0 against 38.1 / 40.3); beyond that both take the same time (28672 x 4096) and the wide ones read the
    // activation half as often
    return n > 128 && units_128 > sms ? 256 : 128;
  }
  if (pair_units * 4 <= sms || k <= 512 || units_128 <= sms) {
    // 256 x 256 pair tiles would keep at most half of the SMs busy, or the K loop is too
    // short to hide the drain of a 256-wide accumulator: 128 x 128 tiles (measured at the
    // 8-way tensor-parallel shapes: 14.6 vs 18.8 us for N = 768, 12.7 vs 16.7 us for K = 512); also while these fit the GPU
    // at once (6144 x 4096 at M = 384: 12.6 against 16.1 us).  Where these fill more than half of it, so that their K is not split, and
    // 256-wide ones leave room for two CTAs per tile, the wide ones move fewer bytes through L2 and pay once a long K has
    // earned back the cluster sum (128-wide / 256-wide with K split, us, 84 to 140 narrow tiles of N = 2560 to 5120: K = 8192
    // 18.2 / 20.6, 12288 25.3 / 25.9, 14336 28.6 / 28.4, 16384 32.1 / 31.4, 18944 36.3 / 34.8; dense 16384 26.8 / 26.0, sparse 16384 21.5 / 21.4,
    // 18944 24.2 / 23.3).  Unsplit they never do (18944: 51.9).
    return split_k && k > 16384 && 2 * units_128 > sms && units_128 <= sms && 2 * units_256 <= sms ? 256 : 128;
  }
  return 512;
}

int gemm_exchange(int tile_n, bool sparse, bool dense, int rows, int k, int splits) {
  const int k_stages = (k + kBK - 1) / kBK;
  if (tile_n == 256) {
    if (sparse && dense) return exchange_form<StageLayout<256, true, true, false>>(rows, splits, k_stages, 256);
    return sparse ? exchange_form<StageLayout<256, true, false, false>>(rows, splits, k_stages, 256)
                  : exchange_form<StageLayout<256, false, true, false>>(rows, splits, k_stages, 256);
  }
  if (sparse && dense) return exchange_form<StageLayout<128, true, true, false>>(rows, splits, k_stages, 128);
  return sparse ? exchange_form<StageLayout<128, true, false, false>>(rows, splits, k_stages, 128)
                : exchange_form<StageLayout<128, false, true, false>>(rows, splits, k_stages, 128);
}

static cudaError_t choose_tile_n(int m, int n, int k, bool split_k, int *tile_n) {
  int dev = 0, sms = 0;
  cudaError_t e = device_info(&dev, &sms);
  if (e == cudaSuccess) *tile_n = gemm_tile_n(m, n, k, split_k, sms);
  return e;
}

bool gemm_swiglu_pays(int m, int ffn, int k) {
  int tile_n = 0;
  return ffn % 128 == 0 && choose_tile_n(m, 2 * ffn, k, true, &tile_n) == cudaSuccess && tile_n == 512;
}

cudaError_t run_gemm_swiglu(const GemmArgs &a, cudaStream_t stream) {
  if (a.a_comp == nullptr || a.a_dense == nullptr || a.bias != nullptr || a.c_in != nullptr || a.scatter_world > 1 ||
      !swiglu_ok(a.n, a.d, a.amax_bits))
    return cudaErrorInvalidValue;
  return launch<256, true, true, true, false, true>(a, stream);
}

int gemm_swiglu_absmax_words(int m, int ffn) {
  int dev = 0, sms = 0;
  if (device_info(&dev, &sms) != cudaSuccess) return 0;
  const int units = ((m + 255) / 256) * (2 * ffn / 256);
  return 2 * (units < sms / 2 ? units : sms / 2);  // the CTAs of the launch
}

cudaError_t run_gemm(const GemmArgs &a, cudaStream_t stream) {
  const bool sparse = a.a_comp != nullptr;
  const bool dense = a.a_dense != nullptr;
  if (!sparse && !dense) return cudaErrorInvalidValue;
  // tile_n: 0 = automatic, 128 / 256 = single-CTA tiles of that width, 512 = CTA pairs (256 x 256)
  int tile_n = a.tile_n;
  if (tile_n == 0) {
    cudaError_t e = choose_tile_n(a.m, a.n, a.k, a.split_k && a.scatter_world <= 1, &tile_n);
    if (e != cudaSuccess) return e;
  }
  const bool pair = tile_n == 512;
  const bool scatter = a.scatter_world > 1;  // validated by launch(): fused GEMM, staged stores, whole tiles per owner
  if (pair) {
    if (sparse && dense) return scatter ? launch<256, true, true, true, true>(a, stream) : launch<256, true, true, true>(a, stream);
    if (sparse) return launch<256, true, false, true>(a, stream);
    return launch<256, false, true, true>(a, stream);
  }
  const int bn = tile_n == 128 ? 128 : 256;
  if (bn == 256) {
    if (sparse && dense) return scatter ? launch<256, true, true, false, true>(a, stream) : launch<256, true, true, false>(a, stream);
    if (sparse) return launch<256, true, false, false>(a, stream);
    return launch<256, false, true, false>(a, stream);
  }
  if (sparse && dense) return scatter ? launch<128, true, true, false, true>(a, stream) : launch<128, true, true, false>(a, stream);
  if (sparse) return launch<128, true, false, false>(a, stream);
  return launch<128, false, true, false>(a, stream);
}

}  // namespace sharq

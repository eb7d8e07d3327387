// Backward of the NVFP4 flash attention with high-precision gradient GEMMs, sm_100a.
//
//   S  = Q K^T           recomputed from the NVFP4 packs (kind::mxf4nvf4, as the forward)
//   P  = exp2(S * scaling * log2e - lse * log2e)      (lse saved by the forward)
//   dP = dO V^T                                        bf16 tcgen05, exact operands
//   dS = P o (dP - delta),  delta = rowsum(dO o O)
//   dV = P^T dO,  dK = scaling * dS^T Q,  dQ = scaling * dS K      bf16 tcgen05
//
// Two kernels, both deterministic (no atomics):
//   bwd_dkdv_kernel  one CTA per 128-key tile of a (batch, kv-head) unit; walks 64-query steps of
//                    every query head of the GQA group, so dK / dV are reduced over the group in
//                    TMEM and written once.
//   bwd_dq_kernel    walks the 64-key steps of 128-query tiles of a head; at D = 128 a CTA takes over tiles of the grid
//                    that have not been launched.
// Every bf16 operand is read from the row-major [rows, 128] tensors by TMA into 128-byte-swizzled
// tiles; the same tile serves as a K-major operand (contraction along D) and as an MN-major
// operand (contraction along the rows), so no transposed copies exist anywhere.
//
// Pipeline of a dK/dV CTA (640 threads; dQ's is described at its kernel): warp 0 TMA producer, warp 1 issuer of S and dP,
// warp 2 scale-atom / row-statistics loader, warp 3 issuer of the gradient GEMMs, warps 4-11 and 12-19 two softmax teams
// that alternate steps, two threads per row.  S has one TMEM slot, which a team reads first and hands back at once, dP
// two; P^T / dS^T are written back as bf16 pairs over the dP^T columns that were read and enter the gradient
// GEMMs as TMEM A operands, so the probabilities never touch shared memory and the tensor pipe
// works on step t+1 while a team is still busy with step t.  (One team of eight warps that took every step:
// S8192 H32 Hk8 1629 -> 1554 us for pre-pass, dK/dV and dQ; two teams and one issuer 1525, an issuer of its own for dQ's
// gradient GEMMs and several query tiles a CTA 1398, for dK/dV's as well 1380.)
// Where the key tiles are too few or too unequal to fill the chip, the steps of a tile are dealt to the
// CTAs of a cluster and their accumulators added over distributed shared memory: S1024 H16 Hk4 101 -> 36 us
// (cluster_split chooses the number).  dQ does not depend on dK / dV and starts while their last CTAs run.
// Causal masking is bottom-right
// aligned; packed varlen is block-diagonal, expressed as a per-row visible range.  Head dim 128,
// or 256 as two 128-wide output halves per tile (both halves recompute S and dP).  Every barrier
// wait is bounded.
#include "common/abi.cuh"
#include "common/fp4.cuh"
#include "common/launch.cuh"
#include "common/sm100.cuh"
#include "common/tma_host.cuh"
#include "common/bwd_util.cuh"

namespace nvfp4 {

constexpr int kBwdThreads = 640;
constexpr float kBwdLog2e = 1.4426950408889634f;
constexpr int kBwdPrefetch = 8;   // stage loads are prefetched into L2 this many steps ahead

// ------------------------------------------------------------------------------------------
// Pre-pass over rows of x [B1, B2, S, D] (strided, unit stride along D): optional contiguous
// bf16 copy xc [B1*B2, S, D] and optional delta [B1*B2, S] = rowsum(x o y).
// 16-bit rows of D = 128 or 256 that are 32-byte aligned go to prep_wide_kernel: a lane takes 32 bytes with one
// 256-bit load, 8 or 16 lanes a row; `flat` rows (row r at r x stride, as contiguous tensors have them) cost
// no division.  Bound by memory, once the instructions are out of the way: half a warp per row with 16-byte
// loads and two divisions a row ran at 3.3 TB/s from HBM and from L2 alike (delta of [16, 8192, 256] with
// max|dO| 49 -> 29 us, of [32, 3000, 128] 14.7 -> 6 us).
// Others: half a warp per row, 16 bytes per lane and load; with D = 128 and aligned rows eight rows in flight.
// ------------------------------------------------------------------------------------------
// eight consecutive elements from a 16-byte aligned address: the loads only (no alignment test, no
// conversion), so that a thread can issue several before it uses the first
template <typename T> struct PrepRaw { uint4 q[sizeof(T) / 2]; };
template <typename T>
__device__ __forceinline__ void prep_load(const T* src, PrepRaw<T>& r) {
#pragma unroll
  for (int i = 0; i < (int)sizeof(T) / 2; ++i) r.q[i] = __ldg(reinterpret_cast<const uint4*>(src) + i);
}
template <typename T>
__device__ __forceinline__ void prep_unpack(const PrepRaw<T>& r, float (&v)[8]) {
  const T* t = reinterpret_cast<const T*>(&r);
#pragma unroll
  for (int e = 0; e < 8; ++e) v[e] = to_f32<T>(t[e]);
}

constexpr int kPrepRows = 4;   // rows per half-warp and trip on the aligned path

template <typename T>
__global__ void __launch_bounds__(256) bwd_prep_kernel(const T* __restrict__ x, int64_t sxb1, int64_t sxb2,
                                                       int64_t sxs, int nb2, const T* __restrict__ y,
                                                       int64_t syb1, int64_t syb2, int64_t sys, int S, int D,
                                                       int64_t rows, __nv_bfloat16* __restrict__ xc,
                                                       float* __restrict__ delta, float* __restrict__ amax,
                                                       int aligned) {
  griddep_launch();
  griddep_wait();
  const int lane = threadIdx.x & 31, l16 = lane & 15;
  float vmax = 0.0f;   // largest |x| this thread has seen (non-negative floats order like their bit patterns)
  // 32-bit divisions (the host keeps rows below 2^31): a 64-bit divide costs more instructions than
  // everything else a thread does for its 16 bytes
  auto row_ptrs = [&](int64_t row, const T*& xr, const T*& yr) {
    const uint32_t b = (uint32_t)row / (uint32_t)S;
    const int s = (int)((uint32_t)row - b * (uint32_t)S);
    const uint32_t b1 = b / (uint32_t)nb2, b2 = b - b1 * (uint32_t)nb2;
    xr = x + (int64_t)b1 * sxb1 + (int64_t)b2 * sxb2 + (int64_t)s * sxs;
    yr = y ? (y + (int64_t)b1 * syb1 + (int64_t)b2 * syb2 + (int64_t)s * sys) : nullptr;
  };
  if (aligned && D == 128) {
    // every row is 16 lanes x 16 bytes, all addresses 16-byte aligned: a warp takes 2 * kPrepRows
    // rows per trip and issues all their loads (x and y) before it reduces the first
    const int64_t base0 = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * (2 * kPrepRows);
    const int64_t step = (int64_t)gridDim.x * 16 * kPrepRows;
    for (int64_t base = base0; base < rows; base += step) {
      int64_t row[kPrepRows];
      bool live[kPrepRows];
      PrepRaw<T> rx[kPrepRows], ry[kPrepRows];
#pragma unroll
      for (int j = 0; j < kPrepRows; ++j) {
        const int64_t row0 = base + 2 * j + (lane >> 4);
        live[j] = row0 < rows;
        row[j] = live[j] ? row0 : rows - 1;
        const T *xr, *yr;
        row_ptrs(row[j], xr, yr);
        prep_load<T>(xr + l16 * 8, rx[j]);
        if (y) prep_load<T>(yr + l16 * 8, ry[j]);
      }
#pragma unroll
      for (int j = 0; j < kPrepRows; ++j) {
        float v[8], w8[8];
        prep_unpack<T>(rx[j], v);
        if (amax != nullptr && live[j]) {
#pragma unroll
          for (int e = 0; e < 8; ++e) vmax = fmaxf(vmax, fabsf(v[e]));
        }
        if (xc && live[j]) {
          uint4 w;
          w.x = pack_bf16x2(v[0], v[1]);
          w.y = pack_bf16x2(v[2], v[3]);
          w.z = pack_bf16x2(v[4], v[5]);
          w.w = pack_bf16x2(v[6], v[7]);
          *reinterpret_cast<uint4*>(xc + row[j] * D + l16 * 8) = w;
        }
        if (delta) {
          float acc = 0.0f;
          prep_unpack<T>(ry[j], w8);
#pragma unroll
          for (int e = 0; e < 8; ++e) acc = fmaf(v[e], w8[e], acc);
#pragma unroll
          for (int o = 8; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
          if (l16 == 0 && live[j]) delta[row[j]] = acc;
        }
      }
    }
  } else {
    const int64_t base0 = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * 2;
    const int64_t nhw = (int64_t)gridDim.x * 16;
    for (int64_t base = base0; base < rows; base += nhw) {    // both half-warps take every trip (shuffles)
      const int64_t row0 = base + (lane >> 4);
      const bool live = row0 < rows;
      const int64_t row = live ? row0 : rows - 1;
      const T *xr, *yr;
      row_ptrs(row, xr, yr);
      float acc = 0.0f;
      for (int c = l16 * 8; c < D; c += 128) {
        float v[8], w8[8];
        load8<T>(xr + c, v);
        if (amax != nullptr && live) {
#pragma unroll
          for (int e = 0; e < 8; ++e) vmax = fmaxf(vmax, fabsf(v[e]));
        }
        if (yr) {
          load8<T>(yr + c, w8);
#pragma unroll
          for (int e = 0; e < 8; ++e) acc = fmaf(v[e], w8[e], acc);
        }
        if (xc && live) {
          uint4 w;
          w.x = pack_bf16x2(v[0], v[1]);
          w.y = pack_bf16x2(v[2], v[3]);
          w.z = pack_bf16x2(v[4], v[5]);
          w.w = pack_bf16x2(v[6], v[7]);
          *reinterpret_cast<uint4*>(xc + row * D + c) = w;
        }
      }
      if (delta) {
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (l16 == 0 && live) delta[row] = acc;
      }
    }
  }
  if (amax != nullptr) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    if (lane == 0 && vmax > 0.0f && vmax < INFINITY)
      atomicMax(reinterpret_cast<unsigned int*>(amax), __float_as_uint(vmax));
  }
}

__device__ __forceinline__ void prep_ldg32(const void* p, uint32_t (&r)[8]) {
  asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "l"(p));
}

constexpr int kPrepWide = 2;   // rows per lane and trip of the wide kernel

template <typename T, int D, bool kDelta, bool kCopy>
__global__ void __launch_bounds__(256, 4) prep_wide_kernel(const T* __restrict__ x, int64_t sxb1, int64_t sxb2, int64_t sxs,
                                                           int nb2, const T* __restrict__ y, int64_t syb1, int64_t syb2,
                                                           int64_t sys, int S, int64_t rows, __nv_bfloat16* __restrict__ xc,
                                                           float* __restrict__ delta, float* __restrict__ amax, int flat) {
  griddep_launch();
  griddep_wait();
  constexpr int kLanes = D / 16, kPer = 32 / kLanes;      // lanes of a row, rows of a load
  const int lane = threadIdx.x & 31, sub = lane / kLanes, col = (lane % kLanes) * 16;
  float vmax = 0.0f;
  const int64_t step = (int64_t)gridDim.x * 8 * kPer * kPrepWide;
  for (int64_t base = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * (kPer * kPrepWide); base < rows; base += step) {
    uint32_t rx[kPrepWide][8], ry[kPrepWide][8];
#pragma unroll
    for (int j = 0; j < kPrepWide; ++j) {
      const int64_t r = min(base + kPer * j + sub, rows - 1);      // the tail re-reads the last row
      int64_t ox = r * sxs, oy = r * sys;
      if (!flat) {
        const uint32_t b = (uint32_t)r / (uint32_t)S, t = (uint32_t)r - b * (uint32_t)S, b1 = b / (uint32_t)nb2, b2 = b - b1 * (uint32_t)nb2;
        ox = (int64_t)b1 * sxb1 + (int64_t)b2 * sxb2 + (int64_t)t * sxs;
        oy = (int64_t)b1 * syb1 + (int64_t)b2 * syb2 + (int64_t)t * sys;
      }
      prep_ldg32(x + ox + col, rx[j]);
      if constexpr (kDelta) prep_ldg32(y + oy + col, ry[j]);
    }
#pragma unroll
    for (int j = 0; j < kPrepWide; ++j) {
      const int64_t r = base + kPer * j + sub;
      float v[16];
      const T* ex = reinterpret_cast<const T*>(rx[j]);
#pragma unroll
      for (int e = 0; e < 16; ++e) v[e] = to_f32<T>(ex[e]);
      if (amax != nullptr) {
#pragma unroll
        for (int e = 0; e < 16; ++e) vmax = fmaxf(vmax, fabsf(v[e]));
      }
      if constexpr (kCopy) {
        if (r < rows) {
          uint4* o = reinterpret_cast<uint4*>(xc + r * D + col);
#pragma unroll
          for (int h = 0; h < 2; ++h)
            o[h] = make_uint4(pack_bf16x2(v[8 * h], v[8 * h + 1]), pack_bf16x2(v[8 * h + 2], v[8 * h + 3]),
                              pack_bf16x2(v[8 * h + 4], v[8 * h + 5]), pack_bf16x2(v[8 * h + 6], v[8 * h + 7]));
        }
      }
      if constexpr (kDelta) {
        const T* ey = reinterpret_cast<const T*>(ry[j]);
        float a0 = 0.0f, a1 = 0.0f;
#pragma unroll
        for (int e = 0; e < 16; e += 2) {
          a0 = fmaf(v[e], to_f32<T>(ey[e]), a0);
          a1 = fmaf(v[e + 1], to_f32<T>(ey[e + 1]), a1);
        }
        a0 += a1;
#pragma unroll
        for (int o = kLanes / 2; o > 0; o >>= 1) a0 += __shfl_xor_sync(0xffffffffu, a0, o);
        if (col == 0 && r < rows) delta[r] = a0;
      }
    }
  }
  if (amax != nullptr) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    if (lane == 0 && vmax > 0.0f && vmax < INFINITY)
      atomicMax(reinterpret_cast<unsigned int*>(amax), __float_as_uint(vmax));
  }
}

// bf16 copies of up to four 16-bit operands (Q, K, V of an fp16 training step) in one launch, blockIdx.y the
// operand: bound by memory and, for short sequences, by the launches that three kernels would be (fp16 training step
// S1024 H16 Hk4 97 -> 91 us, S3000 H32 Hk8 418 -> 412).
struct CopyArgs {
  const void* x[4];
  __nv_bfloat16* out[4];
  int64_t sb1[4], sb2[4], ss[4], rows[4];
  int nb2[4], s[4], flat[4];
};
template <typename T, int D>
__global__ void __launch_bounds__(256, 4) bf16_copies_kernel(const CopyArgs a) {
  griddep_launch();
  griddep_wait();
  constexpr int kLanes = D / 16, kPer = 32 / kLanes, kRows = 4;
  const int k = blockIdx.y, lane = threadIdx.x & 31, sub = lane / kLanes, col = (lane % kLanes) * 16;
  const T* x = static_cast<const T*>(a.x[k]);
  const int64_t rows = a.rows[k], step = (int64_t)gridDim.x * 8 * kPer * kRows;
  for (int64_t base = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * (kPer * kRows); base < rows; base += step) {
    uint32_t rx[kRows][8];
#pragma unroll
    for (int j = 0; j < kRows; ++j) {
      const int64_t r = min(base + kPer * j + sub, rows - 1);
      int64_t o = r * a.ss[k];
      if (!a.flat[k]) {
        const uint32_t b = (uint32_t)r / (uint32_t)a.s[k], b1 = b / (uint32_t)a.nb2[k];
        o = (int64_t)b1 * a.sb1[k] + (int64_t)(b - b1 * (uint32_t)a.nb2[k]) * a.sb2[k] + (r - (int64_t)b * a.s[k]) * a.ss[k];
      }
      prep_ldg32(x + o + col, rx[j]);
    }
#pragma unroll
    for (int j = 0; j < kRows; ++j) {
      const int64_t r = base + kPer * j + sub;
      if (r >= rows) continue;
      const T* e = reinterpret_cast<const T*>(rx[j]);
      uint32_t w[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) w[i] = pack_bf16x2(to_f32<T>(e[2 * i]), to_f32<T>(e[2 * i + 1]));
      uint4* o = reinterpret_cast<uint4*>(a.out[k] + r * D + col);
      o[0] = make_uint4(w[0], w[1], w[2], w[3]);
      o[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
  }
}

struct BwdParams {
  const uint8_t* qsc;   // [ZH, Sq, 8]
  const uint8_t* ksc;   // [ZHk, Skv, 8]
  const __nv_bfloat16* v;    // [ZHk, Skv, D]
  const __nv_bfloat16* dout; // [ZH, Sq, D]
  const float* lse;     // [ZH, Sq] natural log
  const float* delta;   // [ZH, Sq]
  const float* bias;    // [Z, Skv] additive key bias (after the scaling) or null
  const int32_t* seq_start;  // [S] or null (varlen)
  const int32_t* seq_end;    // [S] or null
  void* dq;             // [ZH, Sq, D]
  void* dk;             // [ZHk, Skv, D]
  void* dv;             // [ZHk, Skv, D]
  int h, hk, g;
  int s_q, s_kv;
  float scaling;
  int causal;
  int split;            // CTAs (of one cluster) that share a tile's steps
  int late_wait;        // dQ kernel: wait for the kernel before it at the end, not at the start (launch.cuh)
  int* status;
};

// The operand of dP that a CTA keeps for all its steps -- V rows in the dK/dV kernel, dO rows in the dQ
// kernel -- goes to tensor memory as far as there is room: an N = 64 MMA with both operands in shared
// memory reads 4 KB of A and 2 KB of B, 48 clocks of its 128 bytes per clock for 32 clocks of arithmetic,
// and shared memory bandwidth (operands, TMA writes) is what the kernels run out of first.
// One thread fills kCols columns (two elements each) of its lane; a null row is zeros.
template <int kCols>
__device__ __forceinline__ void fill_a_tmem(uint32_t taddr, const __nv_bfloat16* row) {
#pragma unroll
  for (int c = 0; c < kCols; c += 32) {
    uint32_t r[32];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const uint4 w = row != nullptr ? __ldg(reinterpret_cast<const uint4*>(row + 2 * c) + e) : make_uint4(0u, 0u, 0u, 0u);
      r[4 * e] = w.x; r[4 * e + 1] = w.y; r[4 * e + 2] = w.z; r[4 * e + 3] = w.w;
    }
    tmem_st32(taddr + c, r);
  }
  tmem_st_wait();
  tc_fence_before();
}

// P for 16 columns of one accumulator row: exp2(s * c2 + offsets).  Per-column statistics (the
// dK/dV kernel): `nl` points at the raw lse of the 16 columns in shared memory and `nl_row` is a
// per-thread offset (the key's bias * log2e, or 0).  Per-row (the dQ kernel): `nl_row` is
// -lse*log2e of the row and `nl`, when not null, points at the raw key bias of the 16 columns.
// Columns outside [lo, hi) relative to the chunk's first column are masked when `masked`.
template <bool kPerColumn, bool kColumnBias = false>
__device__ __forceinline__ void prob_chunk(const uint32_t* sr, float (&pf)[16], float c2, const float* nl,
                                           float nl_row, bool masked, int lo, int hi) {
  const float2 c22 = make_float2(c2, c2);
  const float2 row2 = make_float2(nl_row, nl_row);
  const float2 ml2 = make_float2(kPerColumn ? -kBwdLog2e : kBwdLog2e, kPerColumn ? -kBwdLog2e : kBwdLog2e);
#pragma unroll
  for (int e = 0; e < 16; e += 4) {
    float2 n01 = row2, n23 = row2;
    if constexpr (kPerColumn || kColumnBias) {
      const float4 l4 = *reinterpret_cast<const float4*>(nl + e);
      n01 = __ffma2_rn(make_float2(l4.x, l4.y), ml2, row2);
      n23 = __ffma2_rn(make_float2(l4.z, l4.w), ml2, row2);
    }
    const float2 t0 = __ffma2_rn(make_float2(__uint_as_float(sr[e]), __uint_as_float(sr[e + 1])), c22, n01);
    const float2 t1 = __ffma2_rn(make_float2(__uint_as_float(sr[e + 2]), __uint_as_float(sr[e + 3])), c22, n23);
    pf[e] = ex2_bwd(t0.x);
    pf[e + 1] = ex2_bwd(t0.y);
    pf[e + 2] = ex2_bwd(t1.x);
    pf[e + 3] = ex2_bwd(t1.y);
  }
  if (masked) {
#pragma unroll
    for (int e = 0; e < 16; ++e) pf[e] = (e >= lo && e < hi) ? pf[e] : 0.0f;
  }
}
// dS = P o (dP - delta) for 16 columns, packed to bf16 pairs.  Per-column: `nd` points at the raw
// delta values; per-row: `nd_row` is -delta.
template <bool kPerColumn>
__device__ __forceinline__ void ds_chunk(const float (&pf)[16], const uint32_t* dr, uint32_t (&dw)[8],
                                         const float* nd, float nd_row) {
#pragma unroll
  for (int e = 0; e < 16; e += 4) {
    float2 a0, a1;
    const float2 d01 = make_float2(__uint_as_float(dr[e]), __uint_as_float(dr[e + 1]));
    const float2 d23 = make_float2(__uint_as_float(dr[e + 2]), __uint_as_float(dr[e + 3]));
    if constexpr (kPerColumn) {
      const float4 n4 = *reinterpret_cast<const float4*>(nd + e);
      const float2 m1 = make_float2(-1.0f, -1.0f);
      a0 = __ffma2_rn(make_float2(n4.x, n4.y), m1, d01);
      a1 = __ffma2_rn(make_float2(n4.z, n4.w), m1, d23);
    } else {
      a0 = __fadd2_rn(d01, make_float2(nd_row, nd_row));
      a1 = __fadd2_rn(d23, make_float2(nd_row, nd_row));
    }
    const float2 d0 = __fmul2_rn(make_float2(pf[e], pf[e + 1]), a0);
    const float2 d1 = __fmul2_rn(make_float2(pf[e + 2], pf[e + 3]), a1);
    dw[e >> 1] = pack_bf16x2(d0.x, d0.y);
    dw[(e >> 1) + 1] = pack_bf16x2(d1.x, d1.y);
  }
}
// ------------------------------------------------------------------------------------------
// dK / dV
// TMEM: dV [0,128) | dK [128,256) | S^T [256,320) | two dP^T slots [320,384) [384,448) |
//       SFK [448, 448+D/16) | two SFQ slots of D/16 columns
// Head dim 256: the accumulators of a full tile would need all 512 columns, so blockIdx.z picks a
// 128-wide half of dV / dK; S^T and dP^T still contract over the whole head dim.
// A team reads S^T first and hands its slot back, forms P^T while dP^T is still on its way, and writes P^T and dS^T (bf16
// pairs, 16 columns per 32 queries each) over the dP^T columns it has read: the gradient GEMMs take them as TMEM A
// operands.  Two threads issue, one S^T and dP^T and one the gradient GEMMs: a single one paid its waits, twenty MMAs and
// their commits one after the other, about as long as the ~1000 clocks that the products of a step take: S3072 H32 Hk8
// 239 -> 228 us, H16 Hk4 D256 S2048 218 -> 192 us for the whole backward.
// ------------------------------------------------------------------------------------------
template <int D>
struct DkdvSmem {
  static constexpr int DS = D / 64;      // 64-element (128-byte) sub-tiles of a bf16 row
  static constexpr int KSUB = D / 128;   // 64-byte sub-tiles of a pack row
  static constexpr int KB = D / 64;      // K = 64 block-scaled MMAs per S^T, scale atoms per tile
  static constexpr int V = DS * 16384;   // V bf16 [128 keys x D]
  static constexpr int KP = KSUB * 8192; // K pack tile, 128 keys x D/2 B (64-byte swizzle)
  static constexpr int KSF = KB * 512;   // K scale atoms
  // per stage: dO bf16 [64 q x D], the 128-wide half of Q bf16 [64 q x 128] (8 KB sub-tiles),
  // Q pack [64 q x D/2 B], Q scale atoms, lse [64] and delta [64]
  static constexpr int DO = DS * 8192, Q = 16384, QP = KSUB * 4096, QSF = KB * 512, AUX = 1024;
  static constexpr int O_DO = 0, O_Q = DO, O_QP = DO + Q, O_QSF = O_QP + QP, O_AUX = O_QSF + QSF;
  static constexpr int STAGE = DO + Q + QP + QSF + AUX;
  static constexpr int NSTAGE = D == 128 ? 4 : 2;
  static constexpr int TOTAL = V + KP + NSTAGE * STAGE + KSF + 1024;
  static_assert(STAGE % 1024 == 0 && (V + KP) % 1024 == 0, "128-byte-swizzled tiles need 1 KB alignment");
};

template <int D, typename TG, bool kSplit>
__global__ void __launch_bounds__(kBwdThreads, 1)
bwd_dkdv_kernel(const __grid_constant__ CUtensorMap tm_kp, const __grid_constant__ CUtensorMap tm_qp,
                const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                const __grid_constant__ CUtensorMap tm_q, const BwdParams p) {
  using L = DkdvSmem<D>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* s_v = smem;
  uint8_t* s_kp = s_v + L::V;
  uint8_t* s_stage = s_kp + L::KP;
  uint8_t* s_ksf = s_stage + L::NSTAGE * L::STAGE;

  __shared__ uint64_t full[L::NSTAGE], empty[L::NSTAGE];      // empty: also, the gradient GEMMs of the step are complete
  __shared__ uint64_t kv_full, ksf_full, a_full, s_full[2], s_free, dp_full[2], pds_full[2], acc_done;
  __shared__ uint32_t tmem_base_s;
  __shared__ int err;

  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int jt = blockIdx.y;           // key tile (low tiles have the most visible queries: first)
  const int unit = blockIdx.x;         // z * hk + kh
  const int split = kSplit ? p.split : 1;   // CTAs (of one cluster) that share the tile's steps
  const int half = blockIdx.z / split;      // 128-wide slice of the head dim owned by this CTA
  const int rank = kSplit ? blockIdx.z % split : 0;
  const int zi = unit / p.hk, kh = unit % p.hk;
  const int n0 = jt * 128;
  const int shift = p.s_kv - p.s_q;
  const bool varlen = p.seq_start != nullptr;
  if (tid == 0) {
    err = 0;
    for (int i = 0; i < L::NSTAGE; ++i) {
      mbar_init(&full[i], 2);              // TMA producer (and its bytes), scale loader
      mbar_init(&empty[i], 1);
    }
    mbar_init(&kv_full, 1);
    mbar_init(&ksf_full, 1);
    mbar_init(&a_full, 4);
    mbar_init(&s_free, 8);
    mbar_init(&acc_done, 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(&s_full[b], 1);
      mbar_init(&dp_full[b], 1);
      mbar_init(&pds_full[b], 8);
    }
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(&tmem_base_s, 512);
  griddep_wait();                 // before griddep_launch(): the dQ kernel behind it waits late (launch.cuh)
  // 64-query steps that can see a key of this tile
  int q_lo = 0, q_hi = p.s_q;
  if (p.causal) q_lo = max(0, n0 - shift);
  if (varlen) {
    q_lo = max(q_lo, (int)p.seq_start[min(n0, p.s_kv - 1)]);
    q_hi = min(q_hi, (int)p.seq_end[min(n0 + 127, p.s_kv - 1)]);
  }
  const int i_lo = q_lo / 64, i_hi = (q_hi + 63) / 64;
  const int n_i = max(i_hi - i_lo, 0);
  const int st0 = n_i * p.g * rank / split;
  const int nstep = n_i * p.g * (rank + 1) / split - st0;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  griddep_launch();
  const uint32_t tmem = tmem_base_s;
  constexpr uint32_t T_DV = 0, T_DK = 128, T_ST = 256, T_DPT = 320, T_SFK = 448, T_SFQ = T_SFK + L::KB * 4;
  constexpr uint32_t SFQ_SLOT = L::KB * 4;
  constexpr int KT = D == 128 ? 4 : 0;              // K = 16 blocks of V held in tensor memory
  constexpr uint32_t T_V = T_SFQ + 2 * SFQ_SLOT;
  static_assert(T_V + KT * 8 <= 512 && KT % 4 == 0, "TMEM budget");

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one() && nstep > 0) {
      mbar_expect_tx(&kv_full, L::KP + L::V - KT / 4 * 16384);
#pragma unroll
      for (int c = 0; c < L::KSUB; ++c) tma_load_3d(s_kp + c * 8192, &tm_kp, &kv_full, c * 64, n0, unit);
#pragma unroll
      for (int c = KT / 4; c < L::DS; ++c) tma_load_3d(s_v + c * 16384, &tm_v, &kv_full, c * 64, n0, unit);
      // L2 prefetch kBwdPrefetch steps ahead: co-resident CTAs walk the same query tiles in step,
      // so without it every stage load is a first touch that waits on HBM
      auto prefetch = [&](const StepCursor& c0) {
        const int i = i_lo + c0.i, zh = zi * p.h + kh * p.g + c0.gq;
#pragma unroll
        for (int c = 0; c < L::KSUB; ++c) tma_prefetch_3d(&tm_qp, c * 64, i * 64, zh);
#pragma unroll
        for (int c = 0; c < L::DS; ++c) tma_prefetch_3d(&tm_do, c * 64, i * 64, zh);
        tma_prefetch_3d(&tm_q, half * 128, i * 64, zh);
        tma_prefetch_3d(&tm_q, half * 128 + 64, i * 64, zh);
      };
      StepCursor cur(st0, n_i), ahead(st0 + L::NSTAGE, n_i);
      for (int t = L::NSTAGE; t < min(nstep, kBwdPrefetch); ++t, ahead.next(n_i)) prefetch(ahead);
      for (int st = 0; st < nstep; ++st, cur.next(n_i)) {
        const int s = st % L::NSTAGE;
        const int i = i_lo + cur.i;
        const int zh = zi * p.h + kh * p.g + cur.gq;
        if (st + kBwdPrefetch < nstep) {
          prefetch(ahead);
          ahead.next(n_i);
        }
        if (st >= L::NSTAGE) mbar_wait(&empty[s], ((st / L::NSTAGE) & 1) ^ 1, &err, 1);
        uint8_t* sb = s_stage + s * L::STAGE;
        mbar_expect_tx(&full[s], L::QP + L::DO + L::Q);
#pragma unroll
        for (int c = 0; c < L::KSUB; ++c)
          tma_load_3d(sb + L::O_QP + c * 4096, &tm_qp, &full[s], c * 64, i * 64, zh);
#pragma unroll
        for (int c = 0; c < L::DS; ++c)
          tma_load_3d(sb + L::O_DO + c * 8192, &tm_do, &full[s], c * 64, i * 64, zh);
        tma_load_3d(sb + L::O_Q, &tm_q, &full[s], half * 128, i * 64, zh);
        tma_load_3d(sb + L::O_Q + 8192, &tm_q, &full[s], half * 128 + 64, i * 64, zh);
      }
    }
    __syncwarp();
  } else if (warp == 2) {
    // ------------------------------------------------------------------ scale atoms / row statistics
    if (nstep > 0) {
      const uint8_t* ksrc = p.ksc + (int64_t)unit * p.s_kv * (D / 16);
#pragma unroll
      for (int r4 = 0; r4 < 4; ++r4) {
        const int r = lane + 32 * r4;
        const bool ok = n0 + r < p.s_kv;
        const uint8_t* g = ksrc + (int64_t)(ok ? n0 + r : 0) * (D / 16);
#pragma unroll
        for (int c = 0; c < L::KB; ++c)
          cp_async_4(smem_u32(s_ksf) + c * 512 + sf_atom_offset(r, 0), g + 4 * c, ok ? 4u : 0u);
      }
      cp_async_commit();
      cp_async_wait<0>();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ksf_full);
      StepCursor cur(st0, n_i);
      for (int st = 0; st < nstep; ++st, cur.next(n_i)) {
        const int s = st % L::NSTAGE;
        const int i = i_lo + cur.i;
        const int zh = zi * p.h + kh * p.g + cur.gq;
        if (st >= L::NSTAGE) mbar_wait(&empty[s], ((st / L::NSTAGE) & 1) ^ 1, &err, 2);
        uint8_t* sb = s_stage + s * L::STAGE;
        const uint32_t qsf = smem_u32(sb + L::O_QSF);
        float* aux = reinterpret_cast<float*>(sb + L::O_AUX);
#pragma unroll
        for (int r2 = 0; r2 < 2; ++r2) {
          const int r = lane + 32 * r2;
          const int qi = i * 64 + r;
          const bool ok = qi < p.s_q;
          const uint8_t* g = p.qsc + ((int64_t)zh * p.s_q + (ok ? qi : 0)) * (D / 16);
#pragma unroll
          for (int c = 0; c < L::KB; ++c) cp_async_4(qsf + c * 512 + sf_atom_offset(r, 0), g + 4 * c, ok ? 4u : 0u);
          // lse and delta land as they are (rows past the end read 0 and are masked by range)
          const int64_t gi = (int64_t)zh * p.s_q + (ok ? qi : 0);
          cp_async_4(smem_u32(aux + r), p.lse + gi, ok ? 4u : 0u);
          cp_async_4(smem_u32(aux + 64 + r), p.delta + gi, ok ? 4u : 0u);
        }
        cp_async_commit();
        cp_async_wait<0>();
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[s]);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ S^T and dP^T issuer
    // The whole warp waits and counts and one thread issues, here and in the other issuers: a branch of one thread has no
    // uniform registers, which descriptors and tensor-memory addresses have to be in.  Training step of 16384 packed tokens
    // 1578 -> 1525 us, with the forward's; S8192 D256 (block-scaled) 1485 -> 1465.
    if (nstep > 0) {
      const bool leader = elect_one();
      const uint32_t id_s = make_idesc_nvfp4(128, 64);
      const uint32_t id_dp = make_idesc_bf16(128, 64, false);
      mbar_wait(&kv_full, 0, &err, 3);
      mbar_wait(&ksf_full, 0, &err, 4);
      if (KT > 0) mbar_wait(&a_full, 0, &err, 15);
      tc_fence_after();
      if (leader) {
#pragma unroll
        for (int c = 0; c < L::KB; ++c) tmem_cp_32x128b_warpx4(tmem + T_SFK + 4 * c, smem_u32(s_ksf + c * 512));
      }
      // descriptors: constant fields once, then only the 16-byte-unit address field moves
      const uint64_t b_v = desc_sw128(s_v, 0), b_kp = desc_sw64(s_kp, 0);
      const uint64_t b_do = desc_sw128(s_stage + L::O_DO, 0), b_qp = desc_sw64(s_stage + L::O_QP, 0);
#pragma unroll 1
      for (int st = 0; st < nstep; ++st) {
        const int s = st % L::NSTAGE, b = st & 1;
        mbar_wait(&full[s], (st / L::NSTAGE) & 1, &err, 5);
        tc_fence_after();
        const uint32_t qsf = smem_u32(s_stage + L::O_QSF) + s * L::STAGE;
        if (leader) {
#pragma unroll
          for (int c = 0; c < L::KB; ++c) tmem_cp_32x128b_warpx4(tmem + T_SFQ + b * SFQ_SLOT + 4 * c, qsf + c * 512);
        }
        const uint64_t so = (uint64_t)(s * (L::STAGE >> 4));
        const uint64_t x_qp = b_qp + so, x_do = b_do + so;
        if (st > 0) {
          mbar_wait(&s_free, (st - 1) & 1, &err, 7);
          tc_fence_after();
        }
        __syncwarp();
        if (leader) {
#pragma unroll
          for (int k = 0; k < L::KB; ++k)
            umma_nvfp4(tmem + T_ST, b_kp + (k >> 1) * 512 + (k & 1) * 2, x_qp + (k >> 1) * 256 + (k & 1) * 2,
                       id_s, tmem + T_SFK + k * 4, tmem + T_SFQ + b * SFQ_SLOT + k * 4, k > 0);
          umma_commit(&s_full[b]);
        }
        if (st >= 2) {      // P^T and dS^T of step st - 2, in this dP^T slot, have been consumed
          mbar_wait_warp(&empty[(st - 2) % L::NSTAGE], ((st - 2) / L::NSTAGE) & 1, &err, 16);
          tc_fence_after();
        }
        const uint32_t dpt = tmem + T_DPT + b * 64;
        if (leader) {
#pragma unroll
          for (int k = 0; k < KT; ++k)
            umma_bf16_ta(dpt, tmem + T_V + k * 8, x_do + (k >> 2) * 512 + (k & 3) * 2, id_dp, k > 0);
#pragma unroll
          for (int k = KT; k < D / 16; ++k)
            umma_bf16(dpt, b_v + (k >> 2) * 1024 + (k & 3) * 2, x_do + (k >> 2) * 512 + (k & 3) * 2, id_dp, k > 0);
          umma_commit(&dp_full[b]);
        }
        __syncwarp();
      }
    }
    __syncwarp();
  } else if (warp == 3) {
    // ------------------------------------------------------------------ issuer of the gradient GEMMs
    if (nstep > 0) {
      const bool leader = elect_one();
      const uint32_t id_acc = make_idesc_bf16(128, 128, true);
      const uint64_t b_do_mn = desc_sw128_mn(s_stage + L::O_DO + half * 16384, 0, 8192);   // this half's two sub-tiles
      const uint64_t b_q_mn = desc_sw128_mn(s_stage + L::O_Q, 0, 8192);
#pragma unroll 1
      for (int st = 0; st < nstep; ++st) {
        const int s = st % L::NSTAGE, b = st & 1;
        // dO and Q of the stage landed before S^T and dP^T of the step were issued, but this thread has to observe them
        // itself; it does so while P^T and dS^T are still being written
        mbar_wait(&full[s], (st / L::NSTAGE) & 1, &err, 6);
        mbar_wait_warp(&pds_full[b], (st >> 1) & 1, &err, 8);
        tc_fence_after();
        // dV += P^T dO and dK += dS^T Q; slot columns: [P^T q0-31 | dS^T q0-31 | P^T q32-63 | dS^T q32-63], 16 each
        const uint64_t so = (uint64_t)(s * (L::STAGE >> 4));
        const uint32_t a_pt = tmem + T_DPT + b * 64, a_dst = a_pt + 16;
        const uint64_t x_do = b_do_mn + so, x_q = b_q_mn + so;
        if (leader) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_bf16_ta(tmem + T_DV, a_pt + (k >> 1) * 32 + (k & 1) * 8, x_do + 128 * k, id_acc, (k > 0 || st > 0) ? 1u : 0u);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_bf16_ta(tmem + T_DK, a_dst + (k >> 1) * 32 + (k & 1) * 8, x_q + 128 * k, id_acc, (k > 0 || st > 0) ? 1u : 0u);
          umma_commit(&empty[s]);
        }
        __syncwarp();
      }
      if (leader) umma_commit(&acc_done);
    }
    __syncwarp();
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ softmax groups, epilogue
    const int team = (warp - 4) >> 3;   // steps of this parity
    const int grp = ((warp - 4) >> 2) & 1;
    const int part = team * 2 + grp;    // 32-column slice of the gradients this thread stores
    const int wq = warp & 3;
    const int row = wq * 32 + lane;     // key within the tile
    const int key = n0 + row;
    const uint32_t lane_addr = (uint32_t)(wq * 32) << 16;
    if (KT > 0 && part == 0) {
      fill_a_tmem<(KT > 0 ? KT : 4) * 8>(tmem + lane_addr + T_V,
                                         key < p.s_kv ? p.v + ((int64_t)unit * p.s_kv + key) * D : nullptr);
      __syncwarp();
      if (lane == 0) mbar_arrive(&a_full);
    }
    const float c2 = p.scaling * kBwdLog2e;
    // additive bias of this key, in the exponent's base-2 units (-inf masks the key)
    const float bk2 = (p.bias != nullptr && key < p.s_kv) ? p.bias[(int64_t)zi * p.s_kv + key] * kBwdLog2e : 0.0f;
    // visible queries of this key: [ql, qh)
    int ql = 0, qh = 0;
    if (key < p.s_kv) {
      ql = p.causal ? max(key - shift, 0) : 0;
      qh = p.s_q;
      if (varlen) {
        ql = max(ql, (int)p.seq_start[key]);
        qh = min(qh, (int)p.seq_end[key]);
      }
      qh = max(qh, ql);
    }
    // the teams alternate steps; thread g of a row owns queries [32g, 32g+32) of the 64-query tile
    StepCursor cur(st0 + team, n_i);
    for (int st = team; st < nstep; st += 2) {
      const int s = st % L::NSTAGE, k2 = st >> 1;
      const int q0 = (i_lo + cur.i) * 64 + grp * 32;
      cur.next(n_i);
      cur.next(n_i);
      const float* aux = reinterpret_cast<const float*>(s_stage + s * L::STAGE + L::O_AUX) + grp * 32;
      const uint32_t slot = tmem + lane_addr + T_DPT + team * 64 + grp * 32;
      const bool masked = !__all_sync(0xffffffffu, q0 >= ql && q0 + 32 <= qh);
      // the row statistics have landed with the operands of the stage
      mbar_wait_all(&full[s], (st / L::NSTAGE) & 1, &s_full[team], k2 & 1, &err, 10);
      tc_fence_after();
      uint32_t sr[32], dr[32];
      tmem_ld32(tmem + lane_addr + T_ST + grp * 32, sr);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_free);
      float pf[2][16];
#pragma unroll
      for (int c = 0; c < 2; ++c)
        prob_chunk<true>(sr + 16 * c, pf[c], c2, aux + 16 * c, bk2, masked, ql - q0 - 16 * c, qh - q0 - 16 * c);
      mbar_wait(&dp_full[team], k2 & 1, &err, 13);
      tc_fence_after();
      tmem_ld32(slot, dr);
      tmem_ld_wait();
      // P^T -> 16 columns, dS^T -> the next 16, over the dP^T columns just read
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t w[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = pack_bf16x2(pf[c][2 * e], pf[c][2 * e + 1]);
        tmem_st8(slot + 8 * c, w);
        ds_chunk<true>(pf[c], dr + 16 * c, w, aux + 64 + 16 * c, 0.0f);
        tmem_st8(slot + 16 + 8 * c, w);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&pds_full[team]);
    }
    // ---- epilogue: thread `part` of a row writes gradient columns [32 part, 32 part + 32)
    TG* dkrow = static_cast<TG*>(p.dk) + ((int64_t)unit * p.s_kv + key) * D + half * 128 + part * 32;
    TG* dvrow = static_cast<TG*>(p.dv) + ((int64_t)unit * p.s_kv + key) * D + half * 128 + part * 32;
    const uint32_t red = smem_u32(smem);      // the operand tiles are idle once the accumulators are complete
    if (nstep > 0) {
      mbar_wait(&acc_done, 0, &err, 14);
      tc_fence_after();
    }
    if (nstep > 0 || kSplit) {
      uint32_t r[32];
      // One after the other at D = 256 where a cluster shares the tile: unrolled, the kernel spills 8 bytes stored and 20 loaded.
      // Backward H8 Hk2 D256 S384 18.33 -> 17.94 us, S512 23.95 -> 23.41 (before the spills grew 18.42 and 23.80).
#pragma unroll(kSplit && D == 256 ? 1 : 2)
      for (int o = 0; o < 2; ++o) {         // dV, dK
        if (nstep > 0) {
          tmem_ld32(tmem + lane_addr + (o ? T_DK : T_DV) + part * 32, r);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) r[e] = 0u;
        }
        if (kSplit) red_store32(red, row, o * 128 + part * 32, r);
        else store_rows32<TG>(smem + (warp - 4) * 4096, (o ? dkrow : dvrow) - (int64_t)lane * D, D, p.s_kv - key + lane, r,
                              o ? p.scaling : 1.0f, lane);
      }
      tc_fence_before();
    } else if (key < p.s_kv) {
      zero_row(dkrow, 32);
      zero_row(dvrow, 32);
    }
  }
  if (kSplit) {
    cluster_sync_all();
    TG* base_k = static_cast<TG*>(p.dk) + ((int64_t)unit * p.s_kv + n0) * D + half * 128;
    TG* base_v = static_cast<TG*>(p.dv) + ((int64_t)unit * p.s_kv + n0) * D + half * 128;
    red_sum_store<TG>(smem_u32(smem), rank, split, tid, kBwdThreads, p.s_kv - n0, base_v, base_k, D, 1.0f, p.scaling);
    cluster_sync_all();
  }
  tc_fence_before();
  __syncthreads();
  report_error(&err, p.status);
  if (warp == 1) tmem_dealloc(tmem, 512);
}

// ------------------------------------------------------------------------------------------
// dQ
// TMEM: dQ [0,128) | S 64 | three dP slots of 64 (D = 256: two) | SFQ, D/16 columns an item | two SFK slots of D/16
//       columns | dO, D/2 columns.  Head dim 256: blockIdx.z picks a 128-wide half of dQ.
// dS (bf16 pairs, 32 columns) is written back into the dP slot it came from and feeds the dQ GEMM
// as a TMEM A operand.  What bounded a step was the thread that issued its products: a wait that finds its phase complete
// costs it 110 to 130 clocks, fourteen MMAs and their commits 400 more, 1160 of a step's 1280 clocks where the
// products take 650.  So two threads issue, one S and dP and one the dQ GEMMs; the operands of a stage complete on one
// barrier; and the one slot that both teams share is that of S, which a team reads first and hands back before anything else.
// Whole backward (pre-pass, dK/dV, dQ), against one CTA per tile and one issuer: S3072 H32 Hk8 283 -> 239 us, S8192
// 1525 -> 1398, eight samples in 16384 tokens 1038 -> 900, H16 Hk4 D256 S2048 246 -> 220.
// An item is a query tile of a head.  At D = 128 a CTA that is through with one takes over another that has not been
// launched (clusterlaunchcontrol): a CTA's start and end were 13000 clocks, of 640 a step.  Steps count through all
// items; rings, parities and the turns of the teams run on, and the team that has no part in an item's last step is at
// the next item while the other brings out dQ.  At D = 256 the second item's operands do not fit: a CTA has one.
// dO lands in shared memory by TMA and goes from there to tensor memory (rows read by their threads from global
// memory took 2300 clocks of an item's start); dQ leaves through a tile in shared memory as 64-byte row segments.
// ------------------------------------------------------------------------------------------
template <int D>
struct DqSmem {
  static constexpr bool kMany = D == 128;  // a CTA walks several items
  static constexpr int NI = kMany ? 2 : 1; // items whose Q operands are held
  static constexpr int NG = D == 128 ? 3 : 2;   // dP slots
  static constexpr int DS = D / 64, KSUB = D / 128, KB = D / 64;
  static constexpr int QP = KSUB * 8192;   // Q pack tile, 128 queries x D/2 B
  static constexpr int QSF = KB * 512;
  static constexpr int LAND = DS * 16384;  // dO bf16 [128 queries x D] on its way to tensor memory
  static constexpr int OUT = 8 * 2048;     // per warp of a team 32 rows x 64 bytes of dQ
  // per stage: V bf16 [64 keys x D] and the 128-wide half of K bf16 (8 KB sub-tiles), K pack
  // [64 keys x D/2 B], K scale atoms
  static constexpr int V = DS * 8192, K = 16384, KP = KSUB * 4096, KSF = KB * 512, AUX = 1024;
  static constexpr int O_V = 0, O_K = V, O_KP = V + K, O_KSF = O_KP + KP, O_AUX = O_KSF + KSF;   // AUX: key bias [64]
  static constexpr int STAGE = V + K + KP + KSF + AUX;
  static constexpr int NSTAGE = D == 128 ? 4 : 2;
  static constexpr int TOTAL = NI * (QP + QSF) + LAND + OUT + NSTAGE * STAGE + 1024;
  static_assert(STAGE % 1024 == 0 && QP % 1024 == 0, "128-byte-swizzled tiles need 1 KB alignment");
  static_assert(NI * QSF % 512 == 0, "the output tiles are swizzled");
};

struct __align__(16) DqItem {   // one query tile of one head; steps count from the CTA's first one on
  int r0, r1;                   // its 64-key steps [r0, r1); r1 = -1: no more items
  int j0;                       // key step of running step 0 (may be negative)
  int m0, zh, unit, zi, half;
};

template <int D, typename TG>
__global__ void __launch_bounds__(kBwdThreads, 1)
bwd_dq_kernel(const __grid_constant__ CUtensorMap tm_qp, const __grid_constant__ CUtensorMap tm_kp,
              const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_k,
              const __grid_constant__ CUtensorMap tm_do, const BwdParams p) {
  using L = DqSmem<D>;
  constexpr int NI = L::NI;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* s_qp = smem;                          // NI items
  uint8_t* s_land = s_qp + NI * L::QP;
  uint8_t* s_stage = s_land + L::LAND;
  uint8_t* s_qsf = s_stage + L::NSTAGE * L::STAGE;   // NI items
  uint8_t* s_out = s_qsf + NI * L::QSF;

  __shared__ uint64_t full[L::NSTAGE], empty[L::NSTAGE];      // empty: also, the dQ GEMM of the stage's step is complete
  __shared__ uint64_t q_full[2], qsf_full[2], a_full[2], do_full, do_free;
  __shared__ uint64_t s_full[2], s_free, ds_full[2], acc_done, dq_free;
  __shared__ uint64_t item_full[2], item_free[2], clc_full;
  __shared__ __align__(16) uint4 clc_resp;
  __shared__ DqItem s_item[2];
  __shared__ float4 s_rows[NI][128];             // -lse * log2e, -delta, visible keys [first, end) of a row
  __shared__ uint32_t tmem_base_s;
  __shared__ int err;

  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int shift = p.s_kv - p.s_q;
  const bool varlen = p.seq_start != nullptr;
  if (warp == 0) {
    if (lane < L::NSTAGE) {
      mbar_init(&full[lane], 2);             // TMA producer (and its bytes), scale loader
      mbar_init(&empty[lane], 1);
    }
    if (lane < 2) {
      mbar_init(&q_full[lane], 1);
      mbar_init(&qsf_full[lane], 1);
      mbar_init(&a_full[lane], 8);
      mbar_init(&s_full[lane], 1);
      mbar_init(&ds_full[lane], 8);
      mbar_init(&item_full[lane], 1);
      mbar_init(&item_free[lane], 19);
    }
    if (lane == 0) {
      err = 0;
      mbar_init(&do_full, 1);
      mbar_init(&do_free, 8);
      mbar_init(&s_free, 8);
      mbar_init(&acc_done, 1);
      mbar_init(&dq_free, 8);
      mbar_init(&clc_full, 1);
    }
    mbar_fence_init();
    if (lane == 0) tma_prefetch_map(&tm_qp);
    if (lane == 1) tma_prefetch_map(&tm_kp);
    if (lane == 2) tma_prefetch_map(&tm_v);
    if (lane == 3) tma_prefetch_map(&tm_k);
    if (lane == 4) tma_prefetch_map(&tm_do);
  }
  if (warp == 1) tmem_alloc(&tmem_base_s, 512);
  // (warp 0) the query tile of the CTA with block index (bx, by, bz), as item `sl` whose steps count from r0
  auto decode = [&](int bx, int by, int bz, int r0, int sl) {
    const int m0 = ((int)gridDim.y - 1 - by) * 128;      // late query tiles see the most keys: first
    const int zi = bx / p.h, hi = bx - zi * p.h;
    int k_lo = 0, k_hi = p.s_kv;
    if (p.causal) k_hi = max(0, min(p.s_kv, m0 + 128 + shift));
    if (varlen) {
      k_lo = p.seq_start[min(m0, p.s_q - 1)];
      k_hi = min(k_hi, (int)p.seq_end[min(m0 + 127, p.s_q - 1)]);
    }
    const int j_lo = k_lo / 64;
    if (lane == 0) s_item[sl] = DqItem{r0, r0 + max((k_hi + 63) / 64 - j_lo, 0), j_lo - r0, m0, bx, zi * p.hk + hi / p.g, zi, bz};
    __syncwarp();
  };
  griddep_start(p.late_wait != 0);
  if (warp == 0) decode(blockIdx.x, blockIdx.y, blockIdx.z, 0, 0);
  if (tid == 0) mbar_arrive(&item_full[0]);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  griddep_launch();
  const uint32_t tmem = tmem_base_s;
  constexpr uint32_t SF = L::KB * 4;
  constexpr uint32_t T_DQ = 0, T_S = 128, T_DP = 192, T_SFQ = T_DP + L::NG * 64, T_SFK = T_SFQ + NI * SF;
  constexpr uint32_t T_DO = T_SFK + 2 * SF;
  static_assert(T_DO + D / 2 <= 512, "TMEM budget");

  if (warp == 0) {
    // ------------------------------------------------------------------ items, TMA producer
    const bool leader = elect_one();
    uint32_t landed = 0;             // dO tiles loaded
    for (int it = 0;; ++it) {
      const int sl = it & 1, sb_i = sl % NI;
      const int r0 = s_item[sl].r0, r1 = s_item[sl].r1, m0 = s_item[sl].m0, zh = s_item[sl].zh, unit = s_item[sl].unit;
      const int half = s_item[sl].half, j0 = s_item[sl].j0;
      if (leader) {
        mbar_expect_tx(&q_full[sl], L::QP);
#pragma unroll
        for (int c = 0; c < L::KSUB; ++c) tma_load_3d(s_qp + sb_i * L::QP + c * 8192, &tm_qp, &q_full[sl], c * 64, m0, zh);
      }
      if (r1 > r0) {
        if (landed > 0) mbar_wait_warp(&do_free, (landed - 1) & 1, &err, 18);
        ++landed;
        if (leader) {
          mbar_expect_tx(&do_full, L::LAND);
#pragma unroll
          for (int c = 0; c < L::DS; ++c) tma_load_3d(s_land + c * 16384, &tm_do, &do_full, c * 64, m0, zh);
        }
      }
      auto prefetch = [&](int r) {
        const int key0 = (j0 + r) * 64;
#pragma unroll
        for (int c = 0; c < L::KSUB; ++c) tma_prefetch_3d(&tm_kp, c * 64, key0, unit);
#pragma unroll
        for (int c = 0; c < L::DS; ++c) tma_prefetch_3d(&tm_v, c * 64, key0, unit);
        tma_prefetch_3d(&tm_k, half * 128, key0, unit);
        tma_prefetch_3d(&tm_k, half * 128 + 64, key0, unit);
      };
#pragma unroll 1
      for (int r = r0; r < r1; ++r) {
        const int s = r % L::NSTAGE, key0 = (j0 + r) * 64;
        if (leader && r + kBwdPrefetch < r1) prefetch(r + kBwdPrefetch);
        if (r >= L::NSTAGE) mbar_wait_warp(&empty[s], ((r / L::NSTAGE) & 1) ^ 1, &err, 1);
        if (leader) {
          uint8_t* sb = s_stage + s * L::STAGE;
          mbar_expect_tx(&full[s], L::KP + L::V + L::K);
#pragma unroll
          for (int c = 0; c < L::KSUB; ++c)
            tma_load_3d(sb + L::O_KP + c * 4096, &tm_kp, &full[s], c * 64, key0, unit);
#pragma unroll
          for (int c = 0; c < L::DS; ++c) tma_load_3d(sb + L::O_V + c * 8192, &tm_v, &full[s], c * 64, key0, unit);
          tma_load_3d(sb + L::O_K, &tm_k, &full[s], half * 128, key0, unit);
          tma_load_3d(sb + L::O_K + 8192, &tm_k, &full[s], half * 128 + 64, key0, unit);
        }
      }
      bool more = false;
      int bx = 0, by = 0, bz = 0;
      if (L::kMany) {
        if (leader) clc_request(&clc_resp, &clc_full);      // late: the next item goes to who is through first
        __syncwarp();
        more = mbar_wait_item_warp(&clc_full, it & 1, &err, 21) && clc_answer(&clc_resp, bx, by, bz);
        fence_proxy_async_smem();       // read before the next answer may overwrite it
        __syncwarp();
      }
      const int next = sl ^ 1;
      if (it >= 1) more = mbar_wait_item_warp(&item_free[next], (((it + 1) >> 1) & 1) ^ 1, &err, 20) && more;
      if (more) decode(bx, by, bz, r1, next);
      else if (lane == 0) s_item[next].r1 = -1;
      __syncwarp();
      if (lane == 0) mbar_arrive(&item_full[next]);
      if (!more) break;
    }
    __syncwarp();
  } else if (warp == 2) {
    // ------------------------------------------------------------------ scale atoms (+ key bias), row statistics, visible ranges
    for (int it = 0;; ++it) {
      const int sl = it & 1;
      if (!mbar_wait_item(&item_full[sl], (it >> 1) & 1, &err, 22)) break;
      const int r0 = s_item[sl].r0, r1 = s_item[sl].r1;
      if (r1 < 0) break;
      const int m0 = s_item[sl].m0, zh = s_item[sl].zh, unit = s_item[sl].unit, zi = s_item[sl].zi, j0 = s_item[sl].j0;
      const uint8_t* qsrc = p.qsc + (int64_t)zh * p.s_q * (D / 16);
      const uint32_t qsf = smem_u32(s_qsf + (sl % NI) * L::QSF);
#pragma unroll
      for (int r4 = 0; r4 < 4; ++r4) {
        const int r = lane + 32 * r4;
        const bool ok = m0 + r < p.s_q;
        const uint8_t* g = qsrc + (int64_t)(ok ? m0 + r : 0) * (D / 16);
#pragma unroll
        for (int c = 0; c < L::KB; ++c) cp_async_4(qsf + c * 512 + sf_atom_offset(r, 0), g + 4 * c, ok ? 4u : 0u);
      }
      cp_async_commit();
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int row = m0 + lane + 32 * j;
        float4 v = make_float4(0.0f, 0.0f, __int_as_float(0), __int_as_float(0));
        if (row < p.s_q) {
          int kl = 0, kh = p.causal ? min(p.s_kv, row + shift + 1) : p.s_kv;
          if (varlen) {
            kl = p.seq_start[row];
            kh = min(kh, (int)p.seq_end[row]);
          }
          v = make_float4(-p.lse[(int64_t)zh * p.s_q + row] * kBwdLog2e, -p.delta[(int64_t)zh * p.s_q + row],
                          __int_as_float(kl), __int_as_float(max(kh, kl)));
        }
        s_rows[sl % NI][lane + 32 * j] = v;
      }
      cp_async_wait<0>();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&qsf_full[sl]);
      const uint8_t* ksrc = p.ksc + (int64_t)unit * p.s_kv * (D / 16);
#pragma unroll 1
      for (int r = r0; r < r1; ++r) {
        const int s = r % L::NSTAGE, key0 = (j0 + r) * 64;
        if (r >= L::NSTAGE) mbar_wait(&empty[s], ((r / L::NSTAGE) & 1) ^ 1, &err, 2);
        const uint32_t ksf = smem_u32(s_stage + s * L::STAGE + L::O_KSF);
#pragma unroll
        for (int r2 = 0; r2 < 2; ++r2) {
          const int rr = lane + 32 * r2;
          const int key = key0 + rr;
          const bool ok = key < p.s_kv;
          const uint8_t* g = ksrc + (int64_t)(ok ? key : 0) * (D / 16);
#pragma unroll
          for (int c = 0; c < L::KB; ++c) cp_async_4(ksf + c * 512 + sf_atom_offset(rr, 0), g + 4 * c, ok ? 4u : 0u);
          if (p.bias != nullptr)
            cp_async_4(smem_u32(s_stage + s * L::STAGE + L::O_AUX) + rr * 4,
                       p.bias + (int64_t)zi * p.s_kv + (ok ? key : 0), ok ? 4u : 0u);
        }
        cp_async_commit();
        cp_async_wait<0>();
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[s]);
      }
      if (lane == 0) mbar_arrive(&item_free[sl]);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ S and dP issuer
    const bool leader = elect_one();
    const uint32_t id_s = make_idesc_nvfp4(128, 64);
    const uint32_t id_dp = make_idesc_bf16(128, 64, false);
    const uint64_t b_v = desc_sw128(s_stage + L::O_V, 0), b_kp = desc_sw64(s_stage + L::O_KP, 0);
    int r = 0;
    for (int it = 0;; ++it) {
      const int sl = it & 1, si = sl % NI;
      if (!mbar_wait_item_warp(&item_full[sl], (it >> 1) & 1, &err, 22)) break;
      const int r1 = __shfl_sync(0xffffffffu, s_item[sl].r1, 0);
      if (r1 < 0) break;
      mbar_wait(&q_full[sl], (it >> 1) & 1, &err, 3);
      mbar_wait(&qsf_full[sl], (it >> 1) & 1, &err, 4);
      if (r1 > r) mbar_wait(&a_full[sl], (it >> 1) & 1, &err, 15);
      __syncwarp();
      tc_fence_after();
      const uint64_t b_qp = desc_sw64(s_qp + si * L::QP, 0);
      const uint32_t sfq = tmem + T_SFQ + si * SF;
      if (leader) {
#pragma unroll
        for (int c = 0; c < L::KB; ++c) tmem_cp_32x128b_warpx4(sfq + 4 * c, smem_u32(s_qsf + si * L::QSF + c * 512));
      }
#pragma unroll 1
      for (; r < r1; ++r) {
        const int s = r % L::NSTAGE, b = r & 1;
        // the operands of the step; what its dP slot held, dS of step r - NG, has been consumed
        if (r >= L::NG)
          mbar_wait_all(&full[s], (r / L::NSTAGE) & 1, &empty[(r - L::NG) % L::NSTAGE], ((r - L::NG) / L::NSTAGE) & 1, &err, 5);
        else
          mbar_wait(&full[s], (r / L::NSTAGE) & 1, &err, 5);
        tc_fence_after();
        const uint64_t so = (uint64_t)(s * (L::STAGE >> 4));
        const uint64_t x_kp = b_kp + so, x_v = b_v + so;
        const uint32_t ksf = smem_u32(s_stage + L::O_KSF) + s * L::STAGE;
        if (leader) {
#pragma unroll
          for (int k = 0; k < D / 16; ++k)
            umma_bf16_ta(tmem + T_DP + (r % L::NG) * 64, tmem + T_DO + k * 8, x_v + (k >> 2) * 512 + (k & 3) * 2, id_dp, k > 0);
#pragma unroll
          for (int c = 0; c < L::KB; ++c) tmem_cp_32x128b_warpx4(tmem + T_SFK + b * SF + 4 * c, ksf + c * 512);
        }
        if (r > 0) {
          mbar_wait(&s_free, (r - 1) & 1, &err, 7);
          tc_fence_after();
        }
        __syncwarp();
        if (leader) {
#pragma unroll
          for (int k = 0; k < L::KB; ++k)
            umma_nvfp4(tmem + T_S, b_qp + (k >> 1) * 512 + (k & 1) * 2, x_kp + (k >> 1) * 256 + (k & 1) * 2,
                       id_s, sfq + k * 4, tmem + T_SFK + b * SF + k * 4, k > 0);
          umma_commit(&s_full[b]);
        }
        __syncwarp();
      }
      if (leader) mbar_arrive(&item_free[sl]);
    }
    __syncwarp();
  } else if (warp == 3) {
    // ------------------------------------------------------------------ dQ issuer
    const bool leader = elect_one();
    const uint32_t id_acc = make_idesc_bf16(128, 128, true);
    const uint64_t b_k_mn = desc_sw128_mn(s_stage + L::O_K, 0, 8192);
    int r = 0;
    uint32_t n = 0;                     // items with steps so far
    for (int it = 0;; ++it) {
      const int sl = it & 1;
      if (!mbar_wait_item_warp(&item_full[sl], (it >> 1) & 1, &err, 22)) break;
      const int r1 = __shfl_sync(0xffffffffu, s_item[sl].r1, 0);
      if (r1 < 0) break;
      const int first = r;
#pragma unroll 1
      for (; r < r1; ++r) {
        // K of the stage landed before S and dP of the step were issued, but this thread has to observe it itself;
        // it does so while dS is still being written
        mbar_wait(&full[r % L::NSTAGE], (r / L::NSTAGE) & 1, &err, 6);
        if (r == first && n > 0) mbar_wait(&dq_free, (n - 1) & 1, &err, 16);
        mbar_wait_warp(&ds_full[r & 1], (r >> 1) & 1, &err, 8);
        tc_fence_after();
        const uint32_t a_ds = tmem + T_DP + (r % L::NG) * 64;
        const uint64_t x_k = b_k_mn + (uint64_t)((r % L::NSTAGE) * (L::STAGE >> 4));
        if (leader) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_bf16_ta(tmem + T_DQ, a_ds + (k >> 1) * 32 + (k & 1) * 8, x_k + 128 * k, id_acc, (k > 0 || r > first) ? 1u : 0u);
          umma_commit(&empty[r % L::NSTAGE]);
        }
        __syncwarp();
      }
      if (r1 > first) {
        if (leader) umma_commit(&acc_done);
        ++n;
      }
      if (leader) mbar_arrive(&item_free[sl]);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ softmax teams, end of an item
    const int team = (warp - 4) >> 3;   // steps of this parity
    const int grp = ((warp - 4) >> 2) & 1;
    const int wq = warp & 3;
    const int row_in = wq * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(wq * 32) << 16;
    const float c2 = p.scaling * kBwdLog2e;
    uint32_t n = 0;                     // items with steps so far
    for (int it = 0;; ++it) {
      const int sl = it & 1, si = sl % NI;
      if (!mbar_wait_item(&item_full[sl], (it >> 1) & 1, &err, 22)) break;
      const int r0 = s_item[sl].r0, r1 = s_item[sl].r1;
      if (r1 < 0) break;
      if (team == (r0 & 1)) {           // the team of the first step: dO of the item to tensor memory, 2 threads a row
        if (r1 > r0) {
          mbar_wait(&do_full, n & 1, &err, 19);
          if (r0 > 0) {                 // the last dP of the item before has read its dO
            mbar_wait(&s_full[(r0 - 1) & 1], ((r0 - 1) >> 1) & 1, &err, 13);
            tc_fence_after();
          }
#pragma unroll 1
          for (int c = 0; c < L::DS / 2; ++c) {
            const int sub = grp * (L::DS / 2) + c;
            uint32_t w[32];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const uint4 v = *reinterpret_cast<const uint4*>(s_land + sub * 16384 + sw128_offset(row_in, e * 16));
              w[4 * e] = v.x; w[4 * e + 1] = v.y; w[4 * e + 2] = v.z; w[4 * e + 3] = v.w;
            }
            tmem_st32(tmem + lane_addr + T_DO + sub * 32, w);
          }
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&do_free);
        }
        if (lane == 0) mbar_arrive(&a_full[sl]);
      }
      mbar_wait(&qsf_full[sl], (it >> 1) & 1, &err, 12);
      const float4 st = s_rows[si][row_in];
      const float nl = st.x, nd = st.y;
      const int kl = __float_as_int(st.z), kh = __float_as_int(st.w);      // visible keys of this row: [kl, kh)
      const int j0 = s_item[sl].j0;
      // the teams alternate steps; thread g of a row owns keys [32g, 32g+32) of the 64-key tile
#pragma unroll 1
      for (int r = r0 + ((r0 ^ team) & 1); r < r1; r += 2) {
        const int key0 = (j0 + r) * 64 + grp * 32;
        const uint32_t slot = tmem + lane_addr + T_DP + (r % L::NG) * 64 + grp * 32;
        const bool masked = !__all_sync(0xffffffffu, key0 >= kl && key0 + 32 <= kh);
        const float* kbias = nullptr;
        if (p.bias != nullptr) {      // the stage's key bias (landed with the scale atoms)
          const int sg = r % L::NSTAGE;
          mbar_wait(&full[sg], (r / L::NSTAGE) & 1, &err, 10);
          kbias = reinterpret_cast<const float*>(s_stage + sg * L::STAGE + L::O_AUX) + grp * 32;
        }
        mbar_wait(&s_full[team], (r >> 1) & 1, &err, 11);
        tc_fence_after();
        uint32_t dr[32], sr[32];
        tmem_ld32(tmem + lane_addr + T_S + grp * 32, sr);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s_free);
        tmem_ld32(slot, dr);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          float pf[16];
          uint32_t w[8];
          if (kbias != nullptr) prob_chunk<false, true>(sr + 16 * c, pf, c2, kbias + 16 * c, nl, masked, kl - key0 - 16 * c, kh - key0 - 16 * c);
          else prob_chunk<false, false>(sr + 16 * c, pf, c2, nullptr, nl, masked, kl - key0 - 16 * c, kh - key0 - 16 * c);
          if (c == 0) tmem_ld_wait();
          ds_chunk<false>(pf, dr + 16 * c, w, nullptr, nd);
          // dS of keys [32g, 32g+32) replaces the first 16 of the dP columns this thread just read
          tmem_st8(slot + 8 * c, w);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ds_full[team]);
      }
      // ---- end of the item: the team of its last step brings out dQ, 64 columns a thread
      if (team == (r1 > r0 ? (r1 - 1) & 1 : 0)) {
        constexpr int PC = 64 / sizeof(TG);          // columns of a 64-byte row segment
        const int m0 = s_item[sl].m0 + wq * 32;
        TG* out = static_cast<TG*>(p.dq) + ((int64_t)s_item[sl].zh * p.s_q + m0) * D + s_item[sl].half * 128 + grp * 64;
        if (r1 > r0) {
          mbar_wait(&acc_done, n & 1, &err, 14);
          tc_fence_after();
        }
        uint8_t* stg = s_out + (grp * 4 + wq) * 2048;
#pragma unroll 1
        for (int c = 0; c < 64; c += PC) {
          uint4 seg[4];
          if (r1 > r0) {
            uint32_t w[16];
            if constexpr (sizeof(TG) == 2) {
              uint32_t o[32];
              tmem_ld32(tmem + lane_addr + T_DQ + grp * 64 + c, o);
              tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 16; ++e) {
                const float2 v = __fmul2_rn(make_float2(__uint_as_float(o[2 * e]), __uint_as_float(o[2 * e + 1])),
                                            make_float2(p.scaling, p.scaling));
                w[e] = pack_16x2<TG>(v.x, v.y);
              }
            } else {
              tmem_ld16(tmem + lane_addr + T_DQ + grp * 64 + c, w);
              tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 16; ++e) w[e] = __float_as_uint(__uint_as_float(w[e]) * p.scaling);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e)
              *reinterpret_cast<uint4*>(stg + sw64_offset(lane, e * 16)) = make_uint4(w[4 * e], w[4 * e + 1], w[4 * e + 2], w[4 * e + 3]);
            __syncwarp();
#pragma unroll
            for (int e = 0; e < 4; ++e) seg[e] = *reinterpret_cast<const uint4*>(stg + sw64_offset(8 * e + (lane >> 2), (lane & 3) * 16));
            __syncwarp();
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) seg[e] = make_uint4(0u, 0u, 0u, 0u);
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int row = 8 * e + (lane >> 2);
            if (m0 + row < p.s_q) *reinterpret_cast<uint4*>(out + (int64_t)row * D + c + (lane & 3) * (16 / sizeof(TG))) = seg[e];
          }
        }
        if (r1 > r0) {                // dQ and the staging tile are free for the next item
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&dq_free);
        }
      }
      if (r1 > r0) ++n;
      __syncwarp();
      if (lane == 0) mbar_arrive(&item_free[sl]);
    }
  }
  tc_fence_before();
  __syncthreads();
  report_error(&err, p.status);
  if (warp == 1) tmem_dealloc(tmem, 512);
  if (p.late_wait) griddep_wait();
}

template <typename T>
int prep_launch(const void* x, int64_t sxb1, int64_t sxb2, int64_t sxs, int64_t nb1, int64_t nb2, const void* y,
                int64_t syb1, int64_t syb2, int64_t sys, int S, int D, __nv_bfloat16* xc, float* delta,
                float* amax, cudaStream_t st) {
  const int64_t rows = nb1 * nb2 * S;
  if (rows >= (1LL << 31)) return fail(-1, "nvfp4_bwd_prep: more than 2^31 rows");
  auto al = [](const void* p, int64_t a, int64_t b, int64_t c) {
    return p == nullptr || ((reinterpret_cast<uintptr_t>(p) & 15) == 0 && (a * (int64_t)sizeof(T)) % 16 == 0 &&
                            (b * (int64_t)sizeof(T)) % 16 == 0 && (c * (int64_t)sizeof(T)) % 16 == 0);
  };
  if constexpr (sizeof(T) == 2) {
    auto al32 = [](const void* p, int64_t a, int64_t b, int64_t c) {
      return p == nullptr || (((uintptr_t)p | (uint64_t)(a * 2) | (uint64_t)(b * 2) | (uint64_t)(c * 2)) & 31) == 0;
    };
    if ((D == 128 || D == 256) && al32(x, sxb1, sxb2, sxs) && al32(y, syb1, syb2, sys)) {
      auto linear = [&](int64_t b1, int64_t b2, int64_t r) {
        return (nb2 == 1 || b2 == S * r) && (nb1 == 1 || b1 == nb2 * S * r);
      };
      const int flat = linear(sxb1, sxb2, sxs) && (y == nullptr || linear(syb1, syb2, sys));
      auto run = [&](auto kern) {
        const int64_t per_block = 8 * (512 / D) * kPrepWide, blocks = (rows + per_block - 1) / per_block;
        return launch("nvfp4_bwd_prep", kern, dim3((unsigned)std::min<int64_t>(blocks, 148 * 16)), 256, 0, st,
                      static_cast<const T*>(x), sxb1, sxb2, sxs, (int)nb2, static_cast<const T*>(y), syb1, syb2, sys, S, rows, xc,
                      delta, amax, flat);
      };
#define NVFP4_PREP(DD)                                                                                       \
  return delta ? (xc ? run(prep_wide_kernel<T, DD, true, true>) : run(prep_wide_kernel<T, DD, true, false>)) \
               : (xc ? run(prep_wide_kernel<T, DD, false, true>) : run(prep_wide_kernel<T, DD, false, false>))
      if (D == 128) { NVFP4_PREP(128); }
      NVFP4_PREP(256);
#undef NVFP4_PREP
    }
  }
  const int aligned = al(x, sxb1, sxb2, sxs) && al(y, syb1, syb2, sys) && D == 128;
  const int64_t per_block = aligned ? 16 * kPrepRows : 16;
  const int64_t blocks = (rows + per_block - 1) / per_block;
  const unsigned grid = (unsigned)(blocks < 148 * 16 ? blocks : 148 * 16);
  return launch("nvfp4_bwd_prep", bwd_prep_kernel<T>, dim3(grid), 256, 0, st, static_cast<const T*>(x), sxb1, sxb2, sxs,
                (int)nb2, static_cast<const T*>(y), syb1, syb2, sys, S, D, rows, xc, delta, amax, aligned);
}

}  // namespace nvfp4

extern "C" int nvfp4_bf16_copies(int n, const void* const* x, void* const* out, int dtype, const int64_t* strides,
                                 const int64_t* extents, int d, nvfp4_stream_t stream) {
  using namespace nvfp4;
  NVFP4_REQUIRE(n >= 1 && n <= 4 && x && out && strides && extents, "nvfp4_bf16_copies: one to four operands");
  NVFP4_REQUIRE(dtype == NVFP4_DT_BF16 || dtype == NVFP4_DT_FP16, "nvfp4_bf16_copies: operands must be bf16 or fp16");
  NVFP4_REQUIRE(d == 128 || d == 256, "nvfp4_bf16_copies: D must be 128 or 256");
  CopyArgs a = {};
  int64_t most = 0;
  for (int k = 0; k < n; ++k) {
    const int64_t *st = strides + 3 * k, b1 = extents[3 * k], b2 = extents[3 * k + 1], s = extents[3 * k + 2];
    NVFP4_REQUIRE(x[k] && out[k] && b1 >= 1 && b2 >= 1 && s >= 1 && b1 * b2 * s < (1LL << 31), "nvfp4_bf16_copies: bad extents");
    NVFP4_REQUIRE((((uintptr_t)x[k] | (uint64_t)(st[0] * 2) | (uint64_t)(st[1] * 2) | (uint64_t)(st[2] * 2)) & 31) == 0 &&
                      ((uintptr_t)out[k] & 15) == 0,
                  "nvfp4_bf16_copies: rows must be 32-byte aligned");
    a.x[k] = x[k]; a.out[k] = static_cast<__nv_bfloat16*>(out[k]);
    a.sb1[k] = st[0]; a.sb2[k] = st[1]; a.ss[k] = st[2];
    a.nb2[k] = (int)b2; a.s[k] = (int)s; a.rows[k] = b1 * b2 * s;
    a.flat[k] = (b2 == 1 || st[1] == s * st[2]) && (b1 == 1 || st[0] == b2 * s * st[2]);
    most = std::max(most, a.rows[k]);
  }
  const int64_t per_block = 8 * (512 / d) * 4;
  const dim3 grid((unsigned)std::min<int64_t>((most + per_block - 1) / per_block, 148 * 8), (unsigned)n);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto run = [&](auto kern) { return launch("nvfp4_bf16_copies", kern, grid, 256, 0, st, a); };
  if (dtype == NVFP4_DT_BF16) return d == 128 ? run(bf16_copies_kernel<__nv_bfloat16, 128>) : run(bf16_copies_kernel<__nv_bfloat16, 256>);
  return d == 128 ? run(bf16_copies_kernel<__half, 128>) : run(bf16_copies_kernel<__half, 256>);
}

extern "C" int nvfp4_bwd_prep(const void* x, int dtype, int64_t sxb1, int64_t sxb2, int64_t sxs,
                              int64_t nb1, int64_t nb2, const void* y, int64_t syb1, int64_t syb2,
                              int64_t sys, int64_t s, int d, void* xc, float* delta, float* amax,
                              nvfp4_stream_t stream) {
  using namespace nvfp4;
  NVFP4_REQUIRE(x != nullptr && (xc || delta || amax), "nvfp4_bwd_prep: nothing to do");
  NVFP4_REQUIRE(d >= 8 && d % 8 == 0 && s >= 1 && nb1 >= 1 && nb2 >= 1, "nvfp4_bwd_prep: bad extents");
  NVFP4_REQUIRE(s < (1LL << 31), "nvfp4_bwd_prep: sequence too long");
  NVFP4_REQUIRE(delta == nullptr || y != nullptr, "nvfp4_bwd_prep: delta needs the second operand");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto* c = static_cast<__nv_bfloat16*>(xc);
  switch (dtype) {
    case NVFP4_DT_BF16:
      return prep_launch<__nv_bfloat16>(x, sxb1, sxb2, sxs, nb1, nb2, y, syb1, syb2, sys, (int)s, d, c, delta, amax, st);
    case NVFP4_DT_FP16:
      return prep_launch<__half>(x, sxb1, sxb2, sxs, nb1, nb2, y, syb1, syb2, sys, (int)s, d, c, delta, amax, st);
    case NVFP4_DT_FP32:
      return prep_launch<float>(x, sxb1, sxb2, sxs, nb1, nb2, y, syb1, syb2, sys, (int)s, d, c, delta, amax, st);
    default:
      return fail(-1, "nvfp4_bwd_prep: unknown dtype %d", dtype);
  }
}

extern "C" int nvfp4_bwd_hp(const uint8_t* qnv, const uint8_t* qsc, const uint8_t* knv,
                            const uint8_t* ksc, const void* q_bf16, const void* k_bf16,
                            const void* v_bf16, const void* do_bf16, const float* lse,
                            const float* delta, const float* key_bias, const int32_t* seq_start,
                            const int32_t* seq_end, void* dq, void* dk, void* dv, int grad_dtype, int64_t z, int64_t h,
                            int64_t hk, int64_t s_q, int64_t s_kv, int d, float scaling, int flags,
                            int* status, nvfp4_stream_t stream) {
  using namespace nvfp4;
  NVFP4_REQUIRE(d == 128 || d == 256, "nvfp4_bwd_hp: head dim must be 128 or 256");
  NVFP4_REQUIRE(z >= 1 && h >= 1 && hk >= 1 && h % hk == 0, "nvfp4_bwd_hp: bad head counts");
  NVFP4_REQUIRE(s_q >= 1 && s_kv >= 1 && s_q < (1LL << 30) && s_kv < (1LL << 30), "nvfp4_bwd_hp: bad sequence extents");
  NVFP4_REQUIRE(qnv && qsc && knv && ksc && q_bf16 && k_bf16 && v_bf16 && do_bf16 && lse && delta && dq && dk && dv,
                "nvfp4_bwd_hp: null pointer");
  const bool varlen = seq_start != nullptr;
  NVFP4_REQUIRE(varlen == (seq_end != nullptr), "nvfp4_bwd_hp: seq_start and seq_end go together");
  NVFP4_REQUIRE(!varlen || (z == 1 && s_q == s_kv), "nvfp4_bwd_hp: varlen needs Z == 1 and Sq == Skv");
  NVFP4_REQUIRE(!(flags & NVFP4_FWD_CAUSAL) || varlen || s_kv >= s_q, "nvfp4_bwd_hp: causal needs Skv >= Sq");
  NVFP4_REQUIRE((s_kv + 127) / 128 < 65536 && z * h < (1LL << 31) && (s_q + 127) / 128 < 65536,
                "nvfp4_bwd_hp: grid too large");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t zh = z * h, zhk = z * hk;
  CUtensorMap t_qp64, t_qp128, t_kp64, t_kp128, t_v64, t_v128, t_do64, t_do128, t_q64, t_k64;
  int rc;
  const uint64_t pb = (uint64_t)d / 2, hb = (uint64_t)d * 2;   // bytes per pack row / bf16 row
  if ((rc = make_tmap_u8_3d_sw64(&t_qp64, qnv, pb, s_q, zh, pb, (uint64_t)s_q * pb, 64, "nvfp4_bwd_hp(Qp64)"))) return rc;
  if ((rc = make_tmap_u8_3d_sw64(&t_qp128, qnv, pb, s_q, zh, pb, (uint64_t)s_q * pb, 128, "nvfp4_bwd_hp(Qp128)"))) return rc;
  if ((rc = make_tmap_u8_3d_sw64(&t_kp64, knv, pb, s_kv, zhk, pb, (uint64_t)s_kv * pb, 64, "nvfp4_bwd_hp(Kp64)"))) return rc;
  if ((rc = make_tmap_u8_3d_sw64(&t_kp128, knv, pb, s_kv, zhk, pb, (uint64_t)s_kv * pb, 128, "nvfp4_bwd_hp(Kp128)"))) return rc;
  if ((rc = make_tmap_bf16_3d_sw128(&t_v64, v_bf16, d, s_kv, zhk, hb, (uint64_t)s_kv * hb, 64, "nvfp4_bwd_hp(V64)"))) return rc;
  if ((rc = make_tmap_bf16_3d_sw128(&t_v128, v_bf16, d, s_kv, zhk, hb, (uint64_t)s_kv * hb, 128, "nvfp4_bwd_hp(V128)"))) return rc;
  if ((rc = make_tmap_bf16_3d_sw128(&t_do64, do_bf16, d, s_q, zh, hb, (uint64_t)s_q * hb, 64, "nvfp4_bwd_hp(dO64)"))) return rc;
  if ((rc = make_tmap_bf16_3d_sw128(&t_do128, do_bf16, d, s_q, zh, hb, (uint64_t)s_q * hb, 128, "nvfp4_bwd_hp(dO128)"))) return rc;
  if ((rc = make_tmap_bf16_3d_sw128(&t_q64, q_bf16, d, s_q, zh, hb, (uint64_t)s_q * hb, 64, "nvfp4_bwd_hp(Q64)"))) return rc;
  if ((rc = make_tmap_bf16_3d_sw128(&t_k64, k_bf16, d, s_kv, zhk, hb, (uint64_t)s_kv * hb, 64, "nvfp4_bwd_hp(K64)"))) return rc;
  BwdParams p;
  p.v = static_cast<const __nv_bfloat16*>(v_bf16); p.dout = static_cast<const __nv_bfloat16*>(do_bf16);
  p.qsc = qsc; p.ksc = ksc; p.lse = lse; p.delta = delta; p.bias = key_bias;
  p.seq_start = seq_start; p.seq_end = seq_end;
  p.dq = dq; p.dk = dk; p.dv = dv;
  p.h = (int)h; p.hk = (int)hk; p.g = (int)(h / hk); p.s_q = (int)s_q; p.s_kv = (int)s_kv;
  p.scaling = scaling; p.causal = (flags & NVFP4_FWD_CAUSAL) ? 1 : 0; p.status = status;
  p.split = 1; p.late_wait = 0;
  const unsigned halves = (unsigned)(d / 128);
  auto launch = [&](auto kwhole, auto ksplit, auto kdq, int smem_dkdv, int smem_dq) -> int {
    if (int r0 = allow_smem("nvfp4_bwd_hp", reinterpret_cast<const void*>(kdq), smem_dq)) return r0;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t tiles = (s_kv + 127) / 128, longest = (h / hk) * ((s_q + 63) / 64);
    if (int r0 = allow_smem("nvfp4_bwd_hp", reinterpret_cast<const void*>(ksplit), smem_dkdv)) return r0;
    int slots[4];
    cluster_slots(reinterpret_cast<const void*>(ksplit), kBwdThreads, smem_dkdv, sms, slots);
    p.split = cluster_split(zhk * tiles * halves, longest, p.causal ? (h / hk) * 2 : longest, varlen, slots);
    auto kdkdv = p.split > 1 ? ksplit : kwhole;
    if (int r0 = allow_smem("nvfp4_bwd_hp", reinterpret_cast<const void*>(kdkdv), smem_dkdv)) return r0;
    dim3 g1((unsigned)zhk, (unsigned)tiles, halves * p.split);
    if (int r1 = launch_cluster("nvfp4_bwd_hp(dkdv)", kdkdv, g1, p.split, kBwdThreads, smem_dkdv, st, t_kp128, t_qp64, t_v128,
                                t_do64, t_q64, p))
      return r1;
    p.late_wait = 1;
    dim3 g2((unsigned)zh, (unsigned)((s_q + 127) / 128), halves);
    return nvfp4::launch("nvfp4_bwd_hp(dq)", kdq, g2, kBwdThreads, smem_dq, st, t_qp128, t_kp64, t_v64, t_k64, t_do128, p);
  };
#define NVFP4_BWD_LAUNCH(DD, TT) \
  launch(bwd_dkdv_kernel<DD, TT, false>, bwd_dkdv_kernel<DD, TT, true>, bwd_dq_kernel<DD, TT>, DkdvSmem<DD>::TOTAL, DqSmem<DD>::TOTAL)
  if (d == 128) {
    switch (grad_dtype) {
      case NVFP4_DT_BF16: return NVFP4_BWD_LAUNCH(128, __nv_bfloat16);
      case NVFP4_DT_FP16: return NVFP4_BWD_LAUNCH(128, __half);
      case NVFP4_DT_FP32: return NVFP4_BWD_LAUNCH(128, float);
      default: return fail(-1, "nvfp4_bwd_hp: unknown grad dtype %d", grad_dtype);
    }
  }
  switch (grad_dtype) {
    case NVFP4_DT_BF16: return NVFP4_BWD_LAUNCH(256, __nv_bfloat16);
    case NVFP4_DT_FP16: return NVFP4_BWD_LAUNCH(256, __half);
    case NVFP4_DT_FP32: return NVFP4_BWD_LAUNCH(256, float);
    default: return fail(-1, "nvfp4_bwd_hp: unknown grad dtype %d", grad_dtype);
  }
#undef NVFP4_BWD_LAUNCH
}

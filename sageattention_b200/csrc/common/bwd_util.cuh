// Small device helpers shared by the backward kernels (high-precision and all-FP4 gradient GEMMs).
#pragma once
#include <algorithm>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <cstring>
#include "fp4.cuh"
#include "sm100.cuh"

namespace nvfp4 {

__device__ __forceinline__ float ex2_bwd(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// K-major bf16 tile, rows of 128 bytes (64 elements), 128-byte swizzle: the MMA that consumes the
// 16 elements starting at element k16*16 of every row.
__device__ __forceinline__ uint64_t desc_sw128(const void* tile, int k16) {
  return make_smem_desc(smem_u32(tile) + (k16 & 3) * 32, 16, 1024, 2);
}
// The same kind of tile read as an MN-major operand: the contraction runs over the rows (16 rows
// = 2 KB per MMA), the 128 output columns are two 64-element sub-tiles `sub_bytes` apart.
__device__ __forceinline__ uint64_t desc_sw128_mn(const void* tile, int k16, uint32_t sub_bytes) {
  return make_smem_desc(smem_u32(tile) + k16 * 2048, sub_bytes, 1024, 2);
}
__device__ __forceinline__ uint64_t desc_sw64(const void* tile, int k64) {
  return make_smem_desc(smem_u32(tile) + (k64 & 1) * 32, 16, 512, 4);
}
// Instruction descriptor of kind::f16 (fp32 accumulate): 16-bit operands, bf16 unless `f16`.
__host__ __device__ inline uint32_t make_idesc_bf16(uint32_t m, uint32_t n, bool b_mn_major, bool f16 = false) {
  uint32_t d = 0;
  d |= 1u << 4;   // accumulator: fp32
  if (!f16) d |= (1u << 7) | (1u << 10);  // A and B: bf16 (0 = f16)
  if (b_mn_major) d |= 1u << 16;
  d |= (n >> 3) << 17;
  d |= (m >> 4) << 24;
  return d;
}
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                          uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// same, A operand read from TMEM (128 lanes x 8 columns of packed bf16 pairs per K = 16)
__device__ __forceinline__ void umma_bf16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc,
                                             uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// eight consecutive elements, one 16-byte load (two for fp32) when the address allows it
template <typename T>
__device__ __forceinline__ void load8(const T* src, float (&v)[8]) {
  if constexpr (sizeof(T) == 2) {
    if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
      const uint4 raw = *reinterpret_cast<const uint4*>(src);
      const T* t = reinterpret_cast<const T*>(&raw);
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = to_f32<T>(t[e]);
      return;
    }
  } else {
    if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
      const float4 a = *reinterpret_cast<const float4*>(src), c = *reinterpret_cast<const float4*>(src + 4);
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = c.x; v[5] = c.y; v[6] = c.z; v[7] = c.w;
      return;
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) v[e] = to_f32<T>(src[e]);
}

// 32 rows (one a lane) x 32 accumulator columns of a warp -> gradient rows `stride` elements apart, of which the first
// `rows` exist.  Through 32 x 64 (fp32: 128) bytes of shared memory, so that a store instruction covers whole 64- or
// 128-byte row segments: 16 bytes of 32 different rows each time kept the store path of a D = 256 CTA busy for 7700 clocks.
template <typename TG>
__device__ __forceinline__ void store_rows32(uint8_t* stg, TG* out, int64_t stride, int rows, const uint32_t (&r)[32], float mul,
                                             int lane) {
  constexpr int W = 8 * sizeof(TG);         // words of a row
  constexpr int CH = W / 4;                 // 16-byte chunks of a row: lanes of a row when it is stored
  auto at = [&](uint32_t row, uint32_t byte) { return stg + (CH == 4 ? sw64_offset(row, byte) : sw128_offset(row, byte)); };
  uint32_t w[W];
  if constexpr (sizeof(TG) == 2) {
#pragma unroll
    for (int e = 0; e < 16; ++e) w[e] = pack_16x2<TG>(__uint_as_float(r[2 * e]) * mul, __uint_as_float(r[2 * e + 1]) * mul);
  } else {
#pragma unroll
    for (int e = 0; e < 32; ++e) w[e] = __float_as_uint(__uint_as_float(r[e]) * mul);
  }
#pragma unroll
  for (int e = 0; e < CH; ++e) *reinterpret_cast<uint4*>(at(lane, e * 16)) = make_uint4(w[4 * e], w[4 * e + 1], w[4 * e + 2], w[4 * e + 3]);
  __syncwarp();
#pragma unroll
  for (int e = 0; e < CH; ++e) {
    const int row = (32 / CH) * e + lane / CH, ch = lane % CH;
    const uint4 v = *reinterpret_cast<const uint4*>(at(row, ch * 16));
    if (row < rows) *reinterpret_cast<uint4*>(out + row * stride + ch * (16 / (int)sizeof(TG))) = v;
  }
  __syncwarp();
}
template <typename TG>
__device__ __forceinline__ void zero_row(TG* dst, int n) {
  for (int e = 0; e < n; ++e) dst[e] = from_f32<TG>(0.0f);
}


// Position in the step list of a key tile: query head of the group, step among its n_i.
struct StepCursor {
  int gq, i;
  __device__ __forceinline__ StepCursor(int st, int n_i) : gq(n_i > 0 ? st / n_i : 0), i(n_i > 0 ? st - gq * n_i : 0) {}
  __device__ __forceinline__ void next(int n_i) {
    if (++i == n_i) {
      i = 0;
      ++gq;
    }
  }
};

// ---- split of a CTA's column steps over a thread-block cluster
// Where a grid has too few CTAs, or one CTA far more steps than the average, the steps of a tile are
// dealt to `n` CTAs of a cluster; each leaves its fp32 accumulators in its own shared memory and every
// rank adds up 128 / n rows over the cluster, in rank order (results do not depend on timing).
constexpr int kRedStride = 260;        // floats per row: 256 columns, padded so that 16-byte row accesses spread over the banks

// 32 accumulator columns of one row into the reduction buffer
__device__ __forceinline__ void red_store32(uint32_t buf, int row, int col, const uint32_t (&r)[32]) {
  const uint32_t a = buf + (uint32_t)(row * kRedStride + col) * 4u;
#pragma unroll
  for (int e = 0; e < 8; ++e)
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a + 16u * e), "r"(r[4 * e]), "r"(r[4 * e + 1]),
                 "r"(r[4 * e + 2]), "r"(r[4 * e + 3]) : "memory");
}
// Sum rows [rank * 128 / n, (rank + 1) * 128 / n) of the cluster's buffers: columns below 128 of a row go
// to o1 * mul1, the others to o2 * mul2 (with o1 null all 256 go to o2, with o2 null to o1); rows from `rows` on are not written.
template <typename TG>
__device__ __forceinline__ void red_sum_store(uint32_t buf, int rank, int n, int tid, int nthreads, int rows, TG* o1, TG* o2,
                                              int64_t stride, float mul1, float mul2) {
  const int per = 128 / n;
  for (int idx = tid; idx < per * 64; idx += nthreads) {
    const int row = rank * per + (idx >> 6), col = (idx & 63) * 4;
    if (row >= rows) continue;
    const uint32_t a = buf + (uint32_t)(row * kRedStride + col) * 4u;
    float4 v = ld_cluster_f4(a, 0);
    for (int k = 1; k < n; ++k) {
      const float4 w = ld_cluster_f4(a, k);
      v = make_float4(v.x + w.x, v.y + w.y, v.z + w.z, v.w + w.w);
    }
    const bool first = o2 == nullptr || (o1 != nullptr && col < 128);
    const float m = first ? mul1 : mul2;
    TG* o = (first ? o1 : o2) + row * stride + ((o1 != nullptr && o2 != nullptr) ? (col & 127) : col);
    if constexpr (sizeof(TG) == 2) {
      const TG t[4] = {from_f32<TG>(v.x * m), from_f32<TG>(v.y * m), from_f32<TG>(v.z * m), from_f32<TG>(v.w * m)};
      *reinterpret_cast<uint2*>(o) = *reinterpret_cast<const uint2*>(t);
    } else {
      *reinterpret_cast<float4*>(o) = make_float4(v.x * m, v.y * m, v.z * m, v.w * m);
    }
  }
}

// Smallest power of two >= a for a positive normal a; 1 for zero, denormals and non-finite input.
// Dividing a tensor by it is exact, which is what makes it usable as a global pre-scale of packs.
__host__ __device__ __forceinline__ float pow2_ceil(float a) {
#ifdef __CUDA_ARCH__
  uint32_t u = __float_as_uint(a) & 0x7FFFFFFFu;
#else
  uint32_t u;
  memcpy(&u, &a, 4);
  u &= 0x7FFFFFFFu;
#endif
  if (u < 0x00800000u || u >= 0x7F800000u) return 1.0f;
  uint32_t e = u >> 23;
  if (u & 0x7FFFFFu) ++e;
  if (e > 254u) e = 254u;
  const uint32_t r = e << 23;
#ifdef __CUDA_ARCH__
  return __uint_as_float(r);
#else
  float f;
  memcpy(&f, &r, 4);
  return f;
#endif
}

// CTAs per tile (n = 1, 2, 4, 8) for a pass of `tiles` tiles whose step counts run from `longest` down to
// `shortest`: the n with the shortest estimated schedule of clusters of n on the slots[log2 n] that are resident at
// once (cluster_slots; a B200 holds 148, 74, 33 and 15 clusters of such CTAs, so 16 tiles split by eight are two
// waves).  On top of its share a CTA costs kFixed steps (launch, operand loads, epilogue) and, split, kReduce more
// (133 KB exchanged through distributed shared memory).  Estimate: the longest CTA; or all work over the slots, plus
// the part of a last wave that stays empty.  Of packed rows the host does not know the sample lengths: half the
// row is taken for the longest.
// Measured with every n on 300 backward passes (128 to 16384 tokens, 1 to 8 key heads in groups of 1 to 8, D 128 and 256,
// causal or not, dense or 2 to 32 samples a row; half with bf16 gradients, steps of 64 queries, half block-scaled,
// steps of 128): the choice is 1.8 % behind the best n on average, 40 % in the worst pass; never splitting is 25 %
// behind, the same estimate with all SMs for slots and no cost of the exchange 7 % and 90 %.
inline int cluster_split(int64_t tiles, int64_t longest, int64_t shortest, bool packed, const int (&slots)[4]) {
  constexpr double kFixed = 4.0, kReduce = 4.0;
  if (packed) longest = std::max<int64_t>(longest / 2, shortest);
  int best = 1;
  double best_cost = 1e300;
  for (int i = 0; i < 4; ++i) {
    const int n = 1 << i;
    const double f = kFixed + (i > 0 ? kReduce : 0.0), hi = (double)longest / n + f, lo = (double)shortest / n + f;
    const int64_t m = std::max(slots[i], 1), waves = (tiles + m - 1) / m;
    const double cost = std::max(hi, (double)tiles * (hi + lo) * 0.5 / m + lo * ((double)waves - (double)tiles / m));
    if (cost < best_cost) { best_cost = cost; best = n; }
  }
  return best;
}

}  // namespace nvfp4

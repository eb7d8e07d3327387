// Backward of the NVFP4 flash attention with ALL GEMMs in NVFP4 (tcgen05.mma kind::mxf4nvf4,
// e4m3 scale per 16), sm_100a.  The "fp4_rownorm" mode of the training entry.
//
//   S  = Q K^T                     from the forward's packs of Q and K (along D)
//   P  = exp2(S * scaling * log2e - lse * log2e)
//   dP = dO' V^T                   dO' = dO / 2^e packed along D, V packed along D
//   dS = P o (dP - delta') * scaling
//   dV = P^T dO',  dK = dS^T Q,  dQ = dS K     A operand packed IN THE KERNEL along the contraction
//                                              axis, B operand = the transposed pack (dO'^T, Q^T, K^T)
//
// One kernel template serves all passes.  A CTA owns 128 "rows" and streams "columns" in stages
// of 128 (two 64-column steps per stage):
//   dV / dK passes  rows = keys of a (batch, kv-head) unit, columns = queries of every head of the GQA
//               group in turn (dV / dK are reduced over the group in TMEM and written once); one pass
//               for both at D = 128, one each at D = 256;
//   dQ pass     rows = queries of a head, columns = keys.
// Per step one issuer warp queues S (or S^T) and dP as N=64 block-scaled MMAs, another the gradient GEMMs; a
// softmax thread owns one row and 16-column chunks of the step's 64 columns, so the per-16 packs of
// P and dS along the columns are thread-local: nibbles and scale bytes go to shared memory in the
// operand layout and feed one MMA (M128, N = head dim, K64) per gradient and step.  FP4 MMAs replace
// the bf16 MMAs of the high-precision kernels.  Two teams of softmax warps alternate steps, so
// the TMEM loads and barrier waits of one step hide behind the arithmetic of the other; two threads share
// a row (the per-element exp + pack work is bound by how many warps a sub-partition has to interleave).
//
// Keeping the packed operands inside the e4m3 scale range (2^-9 .. 448) -- the job of the
// reference's per-row rms normalisation, flash.py:184-228 -- is done with factors that never change
// while a CTA accumulates, so the sums stay in TMEM:
//   * dO is divided once by 2^e, the smallest power of two >= max|dO| (exact; found by the pre-pass);
//   * P is packed as P * 2^11 and dS as dS * 2^9: with per-16 scales reaching down to 2^-9 this keeps
//     full precision for P >= 6e-6 (uniform attention over 170 k keys) and flushes only below 2e-7;
//   * the constant factors are undone on the accumulators in the epilogue.
// Causal masking is bottom-right aligned; packed varlen is block-diagonal; an additive key bias
// enters the recompute of P.  No atomics: results are run-to-run identical.  Every barrier wait is
// bounded.
#include "common/abi.cuh"
#include "common/fp4.cuh"
#include "common/launch.cuh"
#include "common/sm100.cuh"
#include "common/tma_host.cuh"
#include "common/bwd_util.cuh"

namespace nvfp4 {

constexpr float kB4Log2e = 1.4426950408889634f;
constexpr float kB4PShift = 11.0f;   // P is packed as P * 2^11
constexpr int kB4Prefetch = 2;       // stages prefetched into L2 ahead of the ring


// What a CTA computes.  At D = 128 dV and dK share one pass (both accumulators fit beside S and dP in
// tensor memory).  At D = 256 one 256-wide accumulator fills half of tensor memory, so every gradient
// has a pass of its own over its whole head dim: dV needs S and the P pack only, dK and dQ need S, dP
// and the dS pack.  Cutting the head dim in halves instead, each recomputing everything, ran S, dP and
// both packs twice: the three passes of S8192 H16 Hk4 2740 -> 1483 us with the pre-pass.
enum B4Pass { kB4DkDv = 0, kB4Dq = 1, kB4Dv = 2, kB4Dk = 3 };

// kFp8: the gradient GEMMs' operands (P^T, dS^T, dS packed in the kernel; dO'^T, Q^T, K^T from the
// pre-pass) are MXFP8 -- e4m3 bytes, e8m0 scale per 32 -- instead of NVFP4: tiles of 128-byte rows.
template <int D, int kPass, bool kFp8 = false>
struct B4Cfg {
  static constexpr bool kKeys = kPass != kB4Dq;                       // rows are keys
  static constexpr bool kP = kPass == kB4DkDv || kPass == kB4Dv;      // the P pack feeds a gradient
  static constexpr bool kDs = kPass != kB4Dv;                         // dP, and the dS pack
  static_assert(kPass != kB4DkDv || D == 128, "two 256-wide accumulators do not fit");
  static constexpr int KSUB = D / 128;      // 64-byte-wide sub-tiles of a pack row
  static constexpr int KB = D / 64;         // K = 64 MMAs per product over D
  static constexpr int NW = D / 128;        // 128-row pieces of a transposed tile (N of a gradient GEMM = D)
  static constexpr int X = KSUB * 8192;     // one pack tile: 128 rows x D/2 bytes
  static constexpr int AT = kFp8 ? 16384 : 8192;   // an in-kernel operand tile / a 128-row transposed-pack tile
  static constexpr int TB = NW * AT;        // a transposed-pack tile
  // resident part: X1, X2 (dP), the packed P and dS tiles, scale atoms
  static constexpr int O_X1 = 0, O_X2 = X, O_A1 = O_X2 + (kDs ? X : 0), O_A2 = O_A1 + (kP ? AT : 0);
  static constexpr int O_XSF = O_A2 + (kDs ? AT : 0);     // X1 atoms [KB], X2 atoms [KB]
  static constexpr int O_ASF = O_XSF + 2 * KB * 512;      // P atoms [2 parities], dS atoms [2]
  static constexpr int O_ASF2 = O_ASF + (kP ? 1024 : 0);
  static constexpr int RES = ((O_ASF2 + (kDs ? 1024 : 0) + 1023) / 1024) * 1024;
  // one stage = 128 columns
  static constexpr int S_Y1 = 0, S_Y2 = X, S_T1 = S_Y2 + (kDs ? X : 0), S_T2 = S_T1 + (kP ? TB : 0);
  // atoms [2 steps][KB]: rows 0-63 the 64 columns of the step of Y1, rows 64-127 those of Y2
  static constexpr int S_YSF = S_T2 + (kDs ? TB : 0);
  static constexpr int S_TSF1 = S_YSF + 2 * KB * 512;     // T1 atoms [2 parities][NW] (MXFP8: [NW])
  static constexpr int S_TSF2 = S_TSF1 + (kP ? 2 * NW * 512 : 0);
  static constexpr int S_AUX = S_TSF2 + (kDs ? 2 * NW * 512 : 0);     // two float[128]
  static constexpr int STAGE = ((S_AUX + 1024 + 1023) / 1024) * 1024;
  static constexpr int NSTAGE = (RES + 3 * STAGE + 1024 <= 227 * 1024) ? 3 : 2;
  // softmax threads per row: each owns 32 of a step's 64 columns (sixteen softmax warps, four on every SM
  // sub-partition; one thread per row and eight warps: S8192 D256 1483 -> 1702 us for the three passes)
  static constexpr int NP = 2;
  static constexpr int THREADS = 128 + 256 * NP;
  static constexpr int TOTAL = RES + NSTAGE * STAGE + 1024;
  // TMEM columns
  static constexpr uint32_t T_ACC1 = 0, T_ACC2 = kP ? 128 : 0, T_S = 256, T_G = 384;
  static constexpr uint32_t T_SFX1 = 448, T_SFX2 = T_SFX1 + KB * 4, T_SFY = T_SFX2 + KB * 4;
  static constexpr uint32_t T_SFA1 = T_SFY + KB * 4, T_SFT1 = T_SFA1 + (kP ? 4 : 0);
  static constexpr uint32_t T_SFA2 = T_SFT1 + (kP ? NW * 4 : 0), T_SFT2 = T_SFA2 + (kDs ? 4 : 0);
  static_assert(T_SFT2 + (kDs ? NW * 4 : 0) <= 512, "TMEM budget");
  static_assert(TOTAL <= 227 * 1024, "shared memory budget");
};

// kind::mxf8f6f4, e4m3 x e4m3, ue8m0 scale per 32, fp32 accumulate, both operands K-major; a_sf / b_sf
// pick the byte of the scale word in tensor memory that holds this K = 32 block's scale.
__host__ __device__ __forceinline__ uint32_t make_idesc_mx8(uint32_t m, uint32_t n, uint32_t a_sf, uint32_t b_sf) {
  uint32_t d = 0;
  d |= (b_sf & 3u) << 4;
  d |= (n >> 3) << 17;
  d |= 1u << 23;         // scale format: ue8m0
  d |= (m >> 4) << 24;
  d |= (a_sf & 3u) << 29;
  return d;              // A and B format 0 = e4m3
}
__device__ __forceinline__ void umma_mx8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t sfa_tmem, uint32_t sfb_tmem, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale.block32 [%0], %1, %2, %3, [%5], [%6], "
      "p;\n\t}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(sfa_tmem), "r"(sfb_tmem)
      : "memory");
}

struct B4Params {
  const uint8_t* x1sc;   // row side, along D: [RB, R, D/16]   (dK/dV: K scales; dQ: Q scales)
  const uint8_t* x2sc;   //                                    (dK/dV: V scales; dQ: dO' scales)
  const uint8_t* y1sc;   // column side, along D: [CB, C, D/16] (dK/dV: Q; dQ: K)
  const uint8_t* y2sc;   //                                    (dK/dV: dO'; dQ: V)
  const uint8_t* t1sc;   // transposed packs: [CB, D, c_pad/16] (dK/dV: dO'^T; dQ: unused)
  const uint8_t* t2sc;   //                                    (dK/dV: Q^T; dQ: K^T)
  const float* lse;      // [ZH, Sq] natural log
  const float* delta;    // [ZH, Sq] rowsum(dO o O), in units of dO
  const float* amax;     // device float: max|dO| (the pre-scale of the dO packs is 2^-ceil(log2 amax))
  const float* bias;     // [Z, Skv] additive key bias or null
  const int32_t* seq_start;  // [S] or null (packed varlen)
  const int32_t* seq_end;
  void* out1;            // dK/dV: dV [ZHk, Skv, D]
  void* out2;            // dK/dV: dK [ZHk, Skv, D]; dQ: dQ [ZH, Sq, D]
  int h, hk, g;
  int s_q, s_kv, c_pad;  // c_pad: padded column extent of the transposed packs
  float scaling;
  int causal;
  int split;             // dV / dK passes: CTAs (of one cluster along z) that share a tile's stages
  int late_wait;         // a later pass: wait for the kernel before it at the end, not at the start (launch.cuh)
  int sr_p, sr_ds;       // stochastic rounding of the in-kernel P / dS packs (fp4_legacy mode)
  uint32_t seed;
  int* status;
  int vec;                // scale tensors are aligned for one load a row
};

__device__ __forceinline__ float b4_max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float b4_absmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(fabsf(b)), "f"(fabsf(c)));
  return d;
}

// 16 values -> 8 nibble bytes (two words) and the e4m3 scale byte, with the packer's scale rule; the
// divisions are reciprocal multiplies here (these operands exist only inside the kernel).
// With sr the e2m1 convert rounds stochastically from the bits of (seed, ca, cb .. cb + 3).
template <bool kSigned>
__device__ __forceinline__ uint32_t b4_pack16(const float* x, uint32_t& lo, uint32_t& hi, bool sr = false,
                                              uint32_t seed = 0, uint32_t ca = 0, uint32_t cb = 0) {
  float m;
  if constexpr (kSigned) {
    m = fabsf(x[0]);
#pragma unroll
    for (int e = 1; e < 15; e += 2) m = b4_absmax3(m, x[e], x[e + 1]);
    m = fmaxf(m, fabsf(x[15]));
  } else {
    m = x[0];
#pragma unroll
    for (int e = 1; e < 15; e += 2) m = b4_max3(m, x[e], x[e + 1]);
    m = fmaxf(m, x[15]);
  }
  uint32_t sb;
  float inv;
  {
    const float s32 = fminf(fmaxf(m * 0.16666667f, kScaleFloor), kScaleMax);
    uint16_t sb16;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(sb16) : "f"(0.0f), "f"(s32));
    uint32_t h2;
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"(sb16));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(__half2float(__ushort_as_half((unsigned short)(h2 & 0xFFFF)))));
    sb = sb16 & 0xFFu;
  }
  const float2 i2 = make_float2(inv, inv);
  float2 y[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) y[e] = __fmul2_rn(make_float2(x[2 * e], x[2 * e + 1]), i2);
  if (sr) {
    uint32_t q[4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
      q[e] = e2m1x4_sr(y[2 * e].x, y[2 * e].y, y[2 * e + 1].x, y[2 * e + 1].y, sr_bits(seed, ca, cb + e));
    lo = q[0] | (q[1] << 16);
    hi = q[2] | (q[3] << 16);
    return sb;
  }
  lo = e2m1x8(y[0].x, y[0].y, y[1].x, y[1].y, y[2].x, y[2].y, y[3].x, y[3].y);
  hi = e2m1x8(y[4].x, y[4].y, y[5].x, y[5].y, y[6].x, y[6].y, y[7].x, y[7].y);
  return sb;
}

__device__ __forceinline__ void sts_v4(uint32_t saddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(saddr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void sts_b8(uint32_t saddr, uint32_t a) {
  asm volatile("st.shared.b8 [%0], %1;" ::"r"(saddr), "h"((uint16_t)a) : "memory");
}
__device__ __forceinline__ void sts_b16(uint32_t saddr, uint32_t a) {
  asm volatile("st.shared.b16 [%0], %1;" ::"r"(saddr), "h"((uint16_t)a) : "memory");
}

// kMode: 0 = NVFP4 gradient operands rounded to nearest, 1 = NVFP4 with the stochastic-rounding
// flags honoured (a kernel of its own, so the common case carries none of it), 2 = MXFP8.
template <int D, int kPass, typename TG, int kMode>
__global__ void __launch_bounds__((B4Cfg<D, kPass, kMode == 2>::THREADS), 1)
bwd4_kernel(const __grid_constant__ CUtensorMap tm_x1, const __grid_constant__ CUtensorMap tm_x2,
            const __grid_constant__ CUtensorMap tm_y1, const __grid_constant__ CUtensorMap tm_y2,
            const __grid_constant__ CUtensorMap tm_t1, const __grid_constant__ CUtensorMap tm_t2,
            const B4Params p) {
  constexpr bool kFp8 = kMode == 2, kSr = kMode == 1;
  using C = B4Cfg<D, kPass, kFp8>;
  constexpr bool kKeys = C::kKeys, kP = C::kP, kDs = C::kDs;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* s_res = smem;
  uint8_t* s_stage = smem + C::RES;

  __shared__ uint64_t full[C::NSTAGE], empty[C::NSTAGE];
  __shared__ uint64_t x_full, xsf_full, s_full[2], s_free[2], g_free, a_full[2], a_free[2], acc_done;
  __shared__ uint32_t tmem_base_s;
  __shared__ int err;
  __shared__ float gs_s;      // the power-of-two pre-scale of dO

  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int shift = p.s_kv - p.s_q;
  const bool varlen = p.seq_start != nullptr;

  if (tid == 0) {
    err = 0;
    for (int i = 0; i < C::NSTAGE; ++i) {
      mbar_init(&full[i], 2);              // TMA producer (and its bytes), scale loader
      mbar_init(&empty[i], 1);
    }
    mbar_init(&x_full, 1);
    mbar_init(&xsf_full, 1);
    mbar_init(&g_free, 4 * C::NP);
    mbar_init(&acc_done, 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(&s_full[b], 1);
      mbar_init(&s_free[b], 4 * C::NP);
      mbar_init(&a_full[b], 4 * C::NP);
      mbar_init(&a_free[b], 1);
    }
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(&tmem_base_s, 512);
  griddep_start(p.late_wait != 0);     // before griddep_launch(): the passes behind the first wait late (launch.cuh)
  if (tid == 0) gs_s = pow2_ceil(p.amax != nullptr ? *p.amax : 1.0f);

  // ---- rows of this CTA, and the range of 128-column stages it has to visit
  int rb, row0, zi, kh = 0, cb0;     // row batch entry, first row, batch index, kv head, first column batch entry
  int R, Ccols;                      // row / column extents
  int c_lo = 0, c_hi = 0;
  if constexpr (kKeys) {
    rb = blockIdx.x;                 // z * hk + kh
    row0 = blockIdx.y * 128;
    zi = rb / p.hk; kh = rb % p.hk;
    cb0 = zi * p.h + kh * p.g;
    R = p.s_kv; Ccols = p.s_q;
    c_lo = p.causal ? max(0, row0 - shift) : 0;
    c_hi = p.s_q;
    if (varlen) {
      c_lo = max(c_lo, (int)p.seq_start[min(row0, p.s_kv - 1)]);
      c_hi = min(c_hi, (int)p.seq_end[min(row0 + 127, p.s_kv - 1)]);
    }
  } else {
    rb = blockIdx.x;                 // z * h + hi
    row0 = (gridDim.y - 1 - blockIdx.y) * 128;   // late query tiles see the most keys: first
    zi = rb / p.h;
    cb0 = zi * p.hk + (rb % p.h) / p.g;
    R = p.s_q; Ccols = p.s_kv;
    c_hi = p.causal ? max(0, min(p.s_kv, row0 + 128 + shift)) : p.s_kv;
    if (varlen) {
      c_lo = p.seq_start[min(row0, p.s_q - 1)];
      c_hi = min(c_hi, (int)p.seq_end[min(row0 + 127, p.s_q - 1)]);
    }
  }
  const int i_lo = c_lo / 128;
  const int n_i = max((c_hi + 127) / 128 - i_lo, 0);
  const int rank = kKeys ? blockIdx.z : 0;
  const int sg0 = kKeys ? p.g * n_i * rank / p.split : 0;
  const int nstage = kKeys ? p.g * n_i * (rank + 1) / p.split - sg0 : n_i;
  const int nstep = 2 * nstage;

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  griddep_launch();
  const uint32_t tmem = tmem_base_s;
  const float gs = gs_s;

  // a stage's column batch entry and first column, from its position in the list
  auto stage_cols = [&](const StepCursor& c, int& cb, int& col0) {
    cb = cb0 + c.gq;
    col0 = (i_lo + c.i) * 128;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one() && nstep > 0) {
      mbar_expect_tx(&x_full, (kDs ? 2 : 1) * C::X);
#pragma unroll
      for (int c = 0; c < C::KSUB; ++c) {
        tma_load_3d(s_res + C::O_X1 + c * 8192, &tm_x1, &x_full, c * 64, row0, rb);
        if constexpr (kDs) tma_load_3d(s_res + C::O_X2 + c * 8192, &tm_x2, &x_full, c * 64, row0, rb);
      }
      auto prefetch = [&](const StepCursor& c) {
        int cb, col0;
        stage_cols(c, cb, col0);
        const int tc = kFp8 ? col0 : col0 / 2;
#pragma unroll
        for (int k = 0; k < C::KSUB; ++k) {
          tma_prefetch_3d(&tm_y1, k * 64, col0, cb);
          if constexpr (kDs) tma_prefetch_3d(&tm_y2, k * 64, col0, cb);
          if constexpr (kP) tma_prefetch_3d(&tm_t1, tc, k * 128, cb);
          if constexpr (kDs) tma_prefetch_3d(&tm_t2, tc, k * 128, cb);
        }
      };
      StepCursor cur(sg0, n_i), ahead(sg0 + C::NSTAGE, n_i);
      for (int sg = C::NSTAGE; sg < min(nstage, C::NSTAGE + kB4Prefetch); ++sg, ahead.next(n_i)) prefetch(ahead);
      for (int sg = 0; sg < nstage; ++sg, cur.next(n_i)) {
        const int s = sg % C::NSTAGE;
        int cb, col0;
        stage_cols(cur, cb, col0);
        if (sg + C::NSTAGE + kB4Prefetch < nstage) {
          prefetch(ahead);
          ahead.next(n_i);
        }
        if (sg >= C::NSTAGE) mbar_wait(&empty[s], ((sg / C::NSTAGE) & 1) ^ 1, &err, 1);
        uint8_t* sb = s_stage + s * C::STAGE;
        const int tc = kFp8 ? col0 : col0 / 2;
        mbar_expect_tx(&full[s], (kDs ? 2 : 1) * C::X + ((kP ? 1 : 0) + (kDs ? 1 : 0)) * C::TB);
#pragma unroll
        for (int c = 0; c < C::KSUB; ++c) {
          tma_load_3d(sb + C::S_Y1 + c * 8192, &tm_y1, &full[s], c * 64, col0, cb);
          if constexpr (kDs) tma_load_3d(sb + C::S_Y2 + c * 8192, &tm_y2, &full[s], c * 64, col0, cb);
          if constexpr (kP) tma_load_3d(sb + C::S_T1 + c * C::AT, &tm_t1, &full[s], tc, c * 128, cb);
          if constexpr (kDs) tma_load_3d(sb + C::S_T2 + c * C::AT, &tm_t2, &full[s], tc, c * 128, cb);
        }
      }
    }
    __syncwarp();
  } else if (warp == 2) {
    // ------------------------------------------------------------------ scale atoms, per-column statistics
    if (nstep > 0) {
      const uint32_t xsf = smem_u32(s_res + C::O_XSF);
#pragma unroll
      for (int r4 = 0; r4 < 4; ++r4) {
        const int r = lane + 32 * r4;
        const bool ok = row0 + r < R;
        const int64_t gi = ((int64_t)rb * R + (ok ? row0 + r : 0)) * (D / 16);
#pragma unroll
        for (int c = 0; c < C::KB; ++c) {
          cp_async_4(xsf + c * 512 + sf_atom_offset(r, 0), p.x1sc + gi + 4 * c, ok ? 4u : 0u);
          if constexpr (kDs) cp_async_4(xsf + (C::KB + c) * 512 + sf_atom_offset(r, 0), p.x2sc + gi + 4 * c, ok ? 4u : 0u);
        }
      }
      cp_async_commit();
      cp_async_wait<0>();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&xsf_full);
      // The bytes of the next stage are fetched into registers while this one is in use: a stage that is handed back costs
      // the warp its shared-memory stores, not a trip to L2.  Beside the softmax warps of its scheduler an instruction takes
      // this warp 6 to 8 clocks, so the packs' rows are taken with one load each where they are aligned (as allocated tensors
      // are) and stored 8 and 16 bytes at a time.  S8192 backward, D = 256 / D = 128: copies started when a stage is handed
      // back 1500 / 1947 us (a stage up to 1850 clocks late), a load and a store a word 1305 / 1640, wide ones 1265 / 1547,
      // with one address an operand 1231 / 1536 (column rows by the TMA warp instead: 1286 / 1540).
      const float inv_gs = 1.0f / gs;
      constexpr int PQ = kFp8 ? 1 : 2;                 // words of a transposed row's scale bytes in a stage
      const int csc = p.c_pad / (kFp8 ? 32 : 16);      // scale bytes per row of a transposed pack
      uint32_t y1[4][C::KB], y2[4][kDs ? C::KB : 1], t1[C::NW][PQ][4], t2[C::NW][PQ][4];
      float a0[4], a1[4];
      const bool vec = p.vec != 0;
      auto row_vec = [](const uint8_t* g, uint32_t (&w)[C::KB]) {
        if constexpr (C::KB == 4) {
          const uint4 v = __ldg(reinterpret_cast<const uint4*>(g));
          w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
        } else {
          const uint2 v = __ldg(reinterpret_cast<const uint2*>(g));
          w[0] = v.x; w[1] = v.y;
        }
      };
      auto col_vec = [](const uint8_t* g, uint32_t (&w)[PQ][4], int r4) {
        if constexpr (PQ == 2) {
          const uint2 v = __ldg(reinterpret_cast<const uint2*>(g));
          w[0][r4] = v.x; w[1][r4] = v.y;
        } else {
          w[0][r4] = __ldg(reinterpret_cast<const uint32_t*>(g));
        }
      };
      auto word = [](const uint8_t* g) { return __ldg(reinterpret_cast<const uint32_t*>(g)); };
      auto fetch = [&](const StepCursor& c) {
        int cb, col0;
        stage_cols(c, cb, col0);
        const int64_t y0 = ((int64_t)cb * Ccols + col0 + lane) * (D / 16);
        const int64_t t0 = ((int64_t)cb * D + lane) * csc + col0 / (kFp8 ? 32 : 16);
        if (vec && col0 + 128 <= Ccols) {
          // a whole stage of aligned packs: one address an operand
          const uint8_t *py1 = p.y1sc + y0, *py2 = kDs ? p.y2sc + y0 : nullptr;
          const uint8_t *pt1 = kP ? p.t1sc + t0 : nullptr, *pt2 = kDs ? p.t2sc + t0 : nullptr;
          const uint32_t step = 32u * (uint32_t)csc;
#pragma unroll
          for (int r4 = 0; r4 < 4; ++r4) {
            row_vec(py1 + r4 * 2 * D, y1[r4]);
            if constexpr (kDs) row_vec(py2 + r4 * 2 * D, y2[r4]);
          }
#pragma unroll
          for (int nw = 0; nw < C::NW; ++nw)
#pragma unroll
            for (int r4 = 0; r4 < 4; ++r4) {
              const uint32_t off = (uint32_t)(nw * 4 + r4) * step;
              if constexpr (kP) col_vec(pt1 + off, t1[nw], r4);
              if constexpr (kDs) col_vec(pt2 + off, t2[nw], r4);
            }
          if constexpr (kKeys) {
            const float *pl = p.lse + (int64_t)cb * p.s_q + col0 + lane, *pd = p.delta + (int64_t)cb * p.s_q + col0 + lane;
#pragma unroll
            for (int r4 = 0; r4 < 4; ++r4) {
              a0[r4] = pl[32 * r4];
              if constexpr (kDs) a1[r4] = pd[32 * r4];
            }
          } else {
#pragma unroll
            for (int r4 = 0; r4 < 4; ++r4) a0[r4] = p.bias != nullptr ? p.bias[(int64_t)zi * p.s_kv + col0 + lane + 32 * r4] : 0.0f;
          }
          return;
        }
#pragma unroll
        for (int r4 = 0; r4 < 4; ++r4) {
          const int col = col0 + lane + 32 * r4;   // column of the stage
          const bool ok = col < Ccols;
#pragma unroll
          for (int k = 0; k < C::KB; ++k) {
            y1[r4][k] = 0u;
            if constexpr (kDs) y2[r4][k] = 0u;
          }
          if (ok) {
#pragma unroll
            for (int k = 0; k < C::KB; ++k) {
              y1[r4][k] = word(p.y1sc + y0 + r4 * 2 * D + 4 * k);
              if constexpr (kDs) y2[r4][k] = word(p.y2sc + y0 + r4 * 2 * D + 4 * k);
            }
          }
          // transposed packs: row = feature, 8 (MXFP8: 4) scale bytes = this stage's columns
#pragma unroll
          for (int nw = 0; nw < C::NW; ++nw) {
            const int64_t ti = t0 + (int64_t)(nw * 128 + 32 * r4) * csc;
#pragma unroll
            for (int pq = 0; pq < PQ; ++pq) {
              if constexpr (kP) t1[nw][pq][r4] = word(p.t1sc + ti + 4 * pq);
              if constexpr (kDs) t2[nw][pq][r4] = word(p.t2sc + ti + 4 * pq);
            }
          }
          if constexpr (kKeys) {
            // per query: -lse * log2e + 11 (exponent offset of P * 2^11) and -delta' * scaling / 4
            const int64_t qi = (int64_t)cb * p.s_q + (ok ? col : 0);
            a0[r4] = ok ? p.lse[qi] : 0.0f;
            if constexpr (kDs) a1[r4] = ok ? p.delta[qi] : 0.0f;
          } else {
            // per key: the additive bias in base-2 units
            a0[r4] = (p.bias != nullptr && ok) ? p.bias[(int64_t)zi * p.s_kv + col] : 0.0f;
          }
        }
      };
      StepCursor cur(sg0, n_i);
      if (nstage > 0) fetch(cur);
#pragma unroll 1
      for (int sg = 0; sg < nstage; ++sg) {
        const int s = sg % C::NSTAGE;
        if (sg >= C::NSTAGE) mbar_wait(&empty[s], ((sg / C::NSTAGE) & 1) ^ 1, &err, 2);
        uint8_t* sb = s_stage + s * C::STAGE;
        float* aux = reinterpret_cast<float*>(sb + C::S_AUX);
        const uint32_t at = smem_u32(sb) + lane * 16;      // rows lane, lane + 32, .. of an atom are neighbours
#pragma unroll
        for (int k = 0; k < C::KB; ++k)
#pragma unroll
          for (int pp = 0; pp < 2; ++pp) {
            const uint32_t a = at + C::S_YSF + (pp * C::KB + k) * 512;
            if constexpr (kDs) sts_v4(a, y1[2 * pp][k], y1[2 * pp + 1][k], y2[2 * pp][k], y2[2 * pp + 1][k]);
            else sts_v2(a, y1[2 * pp][k], y1[2 * pp + 1][k]);
          }
#pragma unroll
        for (int nw = 0; nw < C::NW; ++nw)
#pragma unroll
          for (int pq = 0; pq < PQ; ++pq) {
            if constexpr (kP) sts_v4(at + C::S_TSF1 + (pq * C::NW + nw) * 512, t1[nw][pq][0], t1[nw][pq][1], t1[nw][pq][2], t1[nw][pq][3]);
            if constexpr (kDs) sts_v4(at + C::S_TSF2 + (pq * C::NW + nw) * 512, t2[nw][pq][0], t2[nw][pq][1], t2[nw][pq][2], t2[nw][pq][3]);
          }
#pragma unroll
        for (int r4 = 0; r4 < 4; ++r4) {
          const int r = lane + 32 * r4;
          if constexpr (kKeys) {
            const bool ok = (i_lo + cur.i) * 128 + r < Ccols;
            aux[r] = ok ? fmaf(-a0[r4], kB4Log2e, kB4PShift) : 0.0f;
            if constexpr (kDs) aux[128 + r] = -a1[r4] * inv_gs * (p.scaling * 0.25f);
          } else {
            aux[r] = a0[r4] * kB4Log2e;
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[s]);
        cur.next(n_i);
        if (sg + 1 < nstage) fetch(cur);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ S and dP issuer
    if (nstep > 0) {
      const bool leader = elect_one();
      const uint32_t id_n64 = make_idesc_nvfp4(128, 64);
      mbar_wait(&x_full, 0, &err, 3);
      mbar_wait(&xsf_full, 0, &err, 4);
      tc_fence_after();
      if (leader) {
#pragma unroll
        for (int c = 0; c < C::KB; ++c) {
          tmem_cp_32x128b_warpx4(tmem + C::T_SFX1 + 4 * c, smem_u32(s_res + C::O_XSF + c * 512));
          if constexpr (kDs) tmem_cp_32x128b_warpx4(tmem + C::T_SFX2 + 4 * c, smem_u32(s_res + C::O_XSF + (C::KB + c) * 512));
        }
      }
      const uint64_t d_x1 = desc_sw64(s_res + C::O_X1, 0), d_x2 = desc_sw64(s_res + C::O_X2, 0);
      const uint64_t d_y1 = desc_sw64(s_stage + C::S_Y1, 0), d_y2 = desc_sw64(s_stage + C::S_Y2, 0);
#pragma unroll 1
      for (int st = 0; st < nstep; ++st) {
        const int pp = st & 1, sg = st >> 1, s = sg % C::NSTAGE;
        uint8_t* sb = s_stage + s * C::STAGE;
        if (pp == 0) mbar_wait(&full[s], (sg / C::NSTAGE) & 1, &err, 5);
        if (st >= 2) mbar_wait(&s_free[pp], ((st >> 1) - 1) & 1, &err, 7);      // S slot: read by the team of step st - 2
        tc_fence_after();
        const uint64_t so = (uint64_t)(s * (C::STAGE >> 4)) + (uint64_t)(pp * 256);   // 64 rows x 64 bytes further
        if (leader) {
          // S (or S^T): rows x this step's 64 columns
#pragma unroll
          for (int c = 0; c < C::KB; ++c)
            tmem_cp_32x128b_warpx4(tmem + C::T_SFY + 4 * c, smem_u32(sb + C::S_YSF + (pp * C::KB + c) * 512));
#pragma unroll
          for (int k = 0; k < C::KB; ++k)
            umma_nvfp4(tmem + C::T_S + pp * 64, d_x1 + (k >> 1) * 512 + (k & 1) * 2, d_y1 + so + (k >> 1) * 512 + (k & 1) * 2,
                       id_n64, tmem + C::T_SFX1 + k * 4, tmem + C::T_SFY + k * 4, k > 0);
        }
        if constexpr (kDs) {
          // The one dP slot is read by the team of step st - 1.  Only dP waits for it: S and both scales are under way
          // meanwhile.  With both behind this wait the slot's round trip was the step of the dQ pass at D = 256
          // (1270 clocks of which 850 the next team's wait).  Both scales come with one copy a block of D: S8192 D128
          // 1427 -> 1381 us in all, S4100 D256 385 -> 373, S8192 D256 1170 -> 1140.
          if (st > 0) {
            mbar_wait(&g_free, (st - 1) & 1, &err, 9);
            tc_fence_after();
          }
          __syncwarp();
          if (leader) {
            // dP (or dP^T)
#pragma unroll
            for (int k = 0; k < C::KB; ++k)
              umma_nvfp4(tmem + C::T_G, d_x2 + (k >> 1) * 512 + (k & 1) * 2, d_y2 + so + (k >> 1) * 512 + (k & 1) * 2,
                         id_n64, tmem + C::T_SFX2 + k * 4, tmem + C::T_SFY + k * 4 + 2, k > 0);
          }
        }
        if constexpr (!kDs) __syncwarp();
        if (leader) umma_commit(&s_full[pp]);
        __syncwarp();
      }
    }
    __syncwarp();
  } else if (warp == 3) {
    // ------------------------------------------------------------------ issuer of the gradient GEMMs
    // A warp of its own: one issuer for all products paid its waits and commits one after the other, about 1100
    // clocks a step, and S and dP of the next step stood behind the wait for this one's operands.
    if (nstep > 0) {
      const bool leader = elect_one();
      const uint32_t id_acc = make_idesc_nvfp4(128, D);
      const uint64_t d_a1 = kFp8 ? desc_sw128(s_res + C::O_A1, 0) : desc_sw64(s_res + C::O_A1, 0);
      const uint64_t d_a2 = kFp8 ? desc_sw128(s_res + C::O_A2, 0) : desc_sw64(s_res + C::O_A2, 0);
      const uint64_t d_t1 = kFp8 ? desc_sw128(s_stage + C::S_T1, 0) : desc_sw64(s_stage + C::S_T1, 0);
      const uint64_t d_t2 = kFp8 ? desc_sw128(s_stage + C::S_T2, 0) : desc_sw64(s_stage + C::S_T2, 0);
      // acc += A T^T of step pp of stage s (columns [64 pp, 64 pp + 64)), one gradient
      auto one_grad = [&](int pp, int s, uint8_t* sb, uint32_t acc, uint32_t t_acc, uint64_t d_a, uint64_t d_t, int o_asf,
                          int s_tsf, uint32_t t_sfa, uint32_t t_sft) {
        tmem_cp_32x128b_warpx4(tmem + t_sfa, smem_u32(s_res + o_asf + pp * 512));
#pragma unroll
        for (int nw = 0; nw < C::NW; ++nw)
          tmem_cp_32x128b_warpx4(tmem + t_sft + nw * 4, smem_u32(sb + s_tsf + ((kFp8 ? 0 : pp * C::NW) + nw) * 512));
        const uint64_t sg = (uint64_t)(s * (C::STAGE >> 4));
        if constexpr (kFp8) {
          // a step is two K = 32 blocks (32 bytes each) of the 128-byte operand rows; block j of step pp
          // reads byte j of the A atom (one atom per step parity) and byte 2 pp + j of the T atom
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const uint32_t kk = (uint32_t)(pp * 2 + j);
            umma_mx8(tmem + t_acc, d_a + kk * 2, d_t + sg + kk * 2, make_idesc_mx8(128, D, (uint32_t)j, kk), tmem + t_sfa,
                     tmem + t_sft, j > 0 ? 1u : acc);
          }
        } else {      // stage, then the 32-byte half of a row
          umma_nvfp4(tmem + t_acc, d_a + pp * 2, d_t + sg + (uint64_t)(pp * 2), id_acc, tmem + t_sfa, tmem + t_sft, acc);
        }
      };
      auto grad_gemms = [&](int t) {
        const int pp = t & 1, s = (t >> 1) % C::NSTAGE;
        uint8_t* sb = s_stage + s * C::STAGE;
        if (pp == 0) mbar_wait(&full[s], ((t >> 1) / C::NSTAGE) & 1, &err, 6);   // the transposed tiles, seen by this thread
        mbar_wait_warp(&a_full[pp], (t >> 1) & 1, &err, 8);
        tc_fence_after();
        const uint32_t acc = t > 0 ? 1u : 0u;
        if (leader) {
          if constexpr (kP) one_grad(pp, s, sb, acc, C::T_ACC1, d_a1, d_t1, C::O_ASF, C::S_TSF1, C::T_SFA1, C::T_SFT1);
          if constexpr (kDs) one_grad(pp, s, sb, acc, C::T_ACC2, d_a2, d_t2, C::O_ASF2, C::S_TSF2, C::T_SFA2, C::T_SFT2);
          umma_commit(&a_free[pp]);
          if (pp == 1) umma_commit(&empty[s]);
        }
        __syncwarp();
      };
#pragma unroll 1
      for (int t = 0; t < nstep; ++t) grad_gemms(t);
      if (leader) umma_commit(&acc_done);
    }
    __syncwarp();
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ softmax teams, epilogue
    // Two teams alternate steps (team t owns the steps of parity t, hence S slot t and half t of the
    // operand tiles' rows), so one team's TMEM loads and barrier waits overlap the other team's
    // arithmetic.  NP threads share a row: thread h of a row owns 64 / NP of the step's 64 columns,
    // as 16-column chunks whose packs are thread-local.
    constexpr int NP = C::NP, NCH = 4 / NP;               // chunks per thread and step
    const int team = (warp - 4) / (4 * NP);
    const int h = ((warp - 4) >> 2) % NP;
    const int part = team * NP + h;       // epilogue: which 64 / NP accumulator columns this thread stores
    const int wq = warp & 3;
    const int row_in = wq * 32 + lane;
    const int row = row0 + row_in;
    const uint32_t lane_addr = (uint32_t)(wq * 32) << 16;
    const float c2 = p.scaling * kB4Log2e;
    const float cds = p.scaling * 0.25f;           // dS * 2^9 = (P * 2^11) * (dP - delta') * scaling / 4
    const bool row_ok = row < R;
    const bool has_bias = p.bias != nullptr;
    // visible columns of this row: [lo, hi); per-row terms of the exponent and of dS
    int lo = 0, hi = 0;
    float row_e = 0.0f, row_nd = 0.0f;
    if constexpr (kKeys) {
      if (row_ok) {
        lo = p.causal ? max(row - shift, 0) : 0;
        hi = p.s_q;
        if (varlen) {
          lo = max(lo, (int)p.seq_start[row]);
          hi = min(hi, (int)p.seq_end[row]);
        }
        hi = max(hi, lo);
        if (has_bias) row_e = p.bias[(int64_t)zi * p.s_kv + row] * kB4Log2e;
      }
    } else {
      if (row_ok) {
        hi = p.causal ? min(p.s_kv, row + shift + 1) : p.s_kv;
        if (varlen) {
          lo = p.seq_start[row];
          hi = min(hi, (int)p.seq_end[row]);
        }
        hi = max(hi, lo);
        row_e = fmaf(-p.lse[(int64_t)rb * p.s_q + row], kB4Log2e, kB4PShift);
        row_nd = -p.delta[(int64_t)rb * p.s_q + row] * (1.0f / gs) * cds;
      }
    }
    const uint32_t a1_s = smem_u32(s_res + C::O_A1), a2_s = smem_u32(s_res + C::O_A2);
    const uint32_t asf1_s = smem_u32(s_res + C::O_ASF), asf2_s = smem_u32(s_res + C::O_ASF2);
    const float2 c22 = make_float2(c2, c2), cds2 = make_float2(cds, cds);
    // dQ pass: the per-row exponent offset and -delta' term; dK/dV pass: these come per column from aux
    const float2 re2 = kKeys ? make_float2(0.0f, 0.0f) : make_float2(row_e, row_e);
    const float2 rnd2 = make_float2(row_nd, row_nd);
    StepCursor cur(sg0, n_i);
    for (int st = team; st < nstep; st += 2, cur.next(n_i)) {
      const int pp = team, sg = st >> 1, s = sg % C::NSTAGE;
      int cb, col0;
      stage_cols(cur, cb, col0);
      const float* aux0 = reinterpret_cast<const float*>(s_stage + s * C::STAGE + C::S_AUX) + 64 * pp;
      const int cs0 = col0 + 64 * pp;                // first column of the step
      const bool masked = !__all_sync(0xffffffffu, cs0 >= lo && cs0 + 64 <= hi);
      // the column statistics have landed with the operands of the stage
      mbar_wait_all(&full[s], (sg / C::NSTAGE) & 1, &s_full[pp], (st >> 1) & 1, &err, 11);
      tc_fence_after();
      uint32_t wp[4], wd[4], scp = 0u, scd = 0u;
      float pkeep[kFp8 ? 16 : 1], dkeep[kFp8 ? 16 : 1];     // MXFP8: the even chunk of a 32-column group
      // one 16-column chunk: S and dP (or dP^T) values -> P, dS -> packs -> operand tiles
      auto chunk = [&](int ch, const uint32_t (&cur)[16], const uint32_t* gsrc) {
        const float* aux = aux0 + 16 * ch;
        float pf[16], ds[16];
#pragma unroll
        for (int e = 0; e < 16; e += 4) {
          float2 eo01 = re2, eo23 = re2, nd01 = rnd2, nd23 = rnd2;
          if constexpr (kKeys) {
            const float4 a4 = *reinterpret_cast<const float4*>(aux + e);
            eo01 = make_float2(a4.x, a4.y); eo23 = make_float2(a4.z, a4.w);
            if constexpr (kDs) {
              const float4 n4 = *reinterpret_cast<const float4*>(aux + 128 + e);
              nd01 = make_float2(n4.x, n4.y); nd23 = make_float2(n4.z, n4.w);
            }
          }
          const float2 t01 = __ffma2_rn(make_float2(__uint_as_float(cur[e]), __uint_as_float(cur[e + 1])), c22, eo01);
          const float2 t23 = __ffma2_rn(make_float2(__uint_as_float(cur[e + 2]), __uint_as_float(cur[e + 3])), c22, eo23);
          pf[e] = t01.x; pf[e + 1] = t01.y; pf[e + 2] = t23.x; pf[e + 3] = t23.y;
          if constexpr (kDs) {
            const float2 a01 = __ffma2_rn(make_float2(__uint_as_float(gsrc[e]), __uint_as_float(gsrc[e + 1])), cds2, nd01);
            const float2 a23 = __ffma2_rn(make_float2(__uint_as_float(gsrc[e + 2]), __uint_as_float(gsrc[e + 3])), cds2, nd23);
            ds[e] = a01.x; ds[e + 1] = a01.y; ds[e + 2] = a23.x; ds[e + 3] = a23.y;
          }
        }
        if (has_bias) {           // row bias (dK/dV pass) or column bias (dQ pass), base-2 units
#pragma unroll
          for (int e = 0; e < 16; ++e) pf[e] += kKeys ? row_e : aux[e];
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) pf[e] = ex2_bwd(pf[e]);
        if (masked) {
#pragma unroll
          for (int e = 0; e < 16; ++e) pf[e] = (cs0 + 16 * ch + e >= lo && cs0 + 16 * ch + e < hi) ? pf[e] : 0.0f;
        }
        if constexpr (kDs) {
#pragma unroll
        for (int e = 0; e < 16; e += 2) {
          const float2 d2 = __fmul2_rn(make_float2(pf[e], pf[e + 1]), make_float2(ds[e], ds[e + 1]));
          ds[e] = d2.x; ds[e + 1] = d2.y;
        }
        }
        if constexpr (kFp8) {
          if (!(ch & 1)) {
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              if constexpr (kP) pkeep[e] = pf[e];
              if constexpr (kDs) dkeep[e] = ds[e];
            }
          } else {
            if (ch == NCH * h + 1 && st >= 2) mbar_wait(&a_free[pp], ((st >> 1) - 1) & 1, &err, 13);
            const int gi = ch >> 1;                       // which 32 columns of the step
            const uint32_t byte0 = (uint32_t)(pp * 64 + gi * 32);
            uint32_t w[8];
            if constexpr (kP) {
              const uint32_t sb8 = pack_group32_mx8(pkeep, pf, w);
              sts_v4(a1_s + sw128_offset(row_in, byte0), w[0], w[1], w[2], w[3]);
              sts_v4(a1_s + sw128_offset(row_in, byte0 + 16), w[4], w[5], w[6], w[7]);
              sts_b8(asf1_s + pp * 512 + sf_atom_offset(row_in, gi), sb8);
            }
            if constexpr (kDs) {
              const uint32_t sd8 = pack_group32_mx8(dkeep, ds, w);
              sts_v4(a2_s + sw128_offset(row_in, byte0), w[0], w[1], w[2], w[3]);
              sts_v4(a2_s + sw128_offset(row_in, byte0 + 16), w[4], w[5], w[6], w[7]);
              sts_b8(asf2_s + pp * 512 + sf_atom_offset(row_in, gi), sd8);
            }
          }
        } else {
        // random-bit counters: (tensor, row of the CTA's unit) and the quad's column within the unit
        if constexpr (kSr) {
          const uint32_t sr_row = (uint32_t)((int64_t)rb * R + row) * 4u + (kKeys ? 0u : 2u);
          const uint32_t sr_col = (uint32_t)((2 * sg0 + st) * 16 + ch * 4);
          if constexpr (kP)
            scp |= b4_pack16<false>(pf, wp[2 * (ch & 1)], wp[2 * (ch & 1) + 1], p.sr_p != 0, p.seed, sr_row + 1u, sr_col)
                   << (8 * (ch & 1));
          if constexpr (kDs)
            scd |= b4_pack16<true>(ds, wd[2 * (ch & 1)], wd[2 * (ch & 1) + 1], p.sr_ds != 0, p.seed, sr_row, sr_col)
                   << (8 * (ch & 1));
        } else {
          if constexpr (kP) scp |= b4_pack16<false>(pf, wp[2 * (ch & 1)], wp[2 * (ch & 1) + 1]) << (8 * (ch & 1));
          if constexpr (kDs) scd |= b4_pack16<true>(ds, wd[2 * (ch & 1)], wd[2 * (ch & 1) + 1]) << (8 * (ch & 1));
        }
        if (ch & 1) {
          // the operand tiles of step st - 2 (same half of the rows' bytes) must have been consumed
          if (ch == NCH * h + 1 && st >= 2) mbar_wait(&a_free[pp], ((st >> 1) - 1) & 1, &err, 13);
          const int c2i = ch >> 1;      // which 32 columns of the step
          if constexpr (kP) {
            sts_v4(a1_s + sw64_offset(row_in, pp * 32 + c2i * 16), wp[0], wp[1], wp[2], wp[3]);
            sts_b16(asf1_s + pp * 512 + sf_atom_offset(row_in, c2i * 2), scp);
            scp = 0u;
          }
          if constexpr (kDs) {
            sts_v4(a2_s + sw64_offset(row_in, pp * 32 + c2i * 16), wd[0], wd[1], wd[2], wd[3]);
            sts_b16(asf2_s + pp * 512 + sf_atom_offset(row_in, c2i * 2), scd);
            scd = 0u;
          }
        }
        }
      };
      // this thread's 32 columns of dP (or dP^T) arrive with the first S chunk, so the single dP slot
      // goes back to the issuer after one round trip; the S slot follows with the second chunk
      uint32_t gq[kDs ? 32 : 1];
      if constexpr (kDs) tmem_ld32(tmem + lane_addr + C::T_G + 32 * h, gq);
#pragma unroll
      for (int cc = 0; cc < NCH; ++cc) {
        const int ch = NCH * h + cc;
        uint32_t cur[16];
        tmem_ld16(tmem + lane_addr + C::T_S + pp * 64 + 16 * ch, cur);
        tmem_ld_wait();
        if (cc == 0 || cc == NCH - 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            if (kDs && cc == 0) mbar_arrive(&g_free);
            if (cc == NCH - 1) mbar_arrive(&s_free[pp]);
          }
        }
        chunk(ch, cur, kDs ? gq + 16 * cc : gq);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&a_full[pp]);
    }
    // ---- epilogue: thread `part` of a row writes gradient columns [EC part, EC part + EC)
    const float m1 = gs * 4.8828125e-4f;       // 2^-11
    const float m2 = gs * 1.953125e-3f;        // 2^-9
    constexpr int EC = D / (2 * NP);
    TG* o1 = kP ? static_cast<TG*>(p.out1) + ((int64_t)rb * R + row) * D + part * EC : nullptr;
    TG* o2 = kDs ? static_cast<TG*>(p.out2) + ((int64_t)rb * R + row) * D + part * EC : nullptr;
    const bool split = kKeys && p.split > 1;
    if (nstep > 0) {
      mbar_wait(&acc_done, 0, &err, 14);
      tc_fence_after();
    }
    if (nstep > 0 || split) {
      auto column32 = [&](uint32_t t_acc, int c, TG* o, float mul, int red_col) {
        uint32_t r[32];
        if (nstep > 0) {
          tmem_ld32(tmem + lane_addr + t_acc + part * EC + c * 32, r);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) r[e] = 0u;
        }
        if (split) red_store32(smem_u32(smem), row_in, red_col + part * EC + c * 32, r);   // the operand tiles are idle by now
        else store_rows32<TG>(smem + (warp - 4) * 4096, o + c * 32 - (int64_t)lane * D, D, R - row + lane, r, mul, lane);
      };
#pragma unroll
      for (int c = 0; c < EC / 32; ++c) {
        if constexpr (kP) column32(C::T_ACC1, c, o1, m1, 0);
        if constexpr (kDs) column32(C::T_ACC2, c, o2, m2, kP ? 128 : 0);
      }
      tc_fence_before();
    } else if (row_ok) {
      if constexpr (kP) zero_row(o1, EC);
      if constexpr (kDs) zero_row(o2, EC);
    }
  }
  if constexpr (kKeys) {
    if (p.split > 1) {
      cluster_sync_all();
      const int64_t first = ((int64_t)rb * R + row0) * D;
      red_sum_store<TG>(smem_u32(smem), rank, p.split, tid, C::THREADS, R - row0, kP ? static_cast<TG*>(p.out1) + first : nullptr,
                        kDs ? static_cast<TG*>(p.out2) + first : nullptr, D, gs * 4.8828125e-4f, gs * 1.953125e-3f);
      cluster_sync_all();
    }
  }
  tc_fence_before();
  __syncthreads();
  report_error(&err, p.status);
  if (warp == 1) tmem_dealloc(tmem, 512);
  if (p.late_wait) griddep_wait();
}

}  // namespace nvfp4

extern "C" int nvfp4_bwd_fp4(const uint8_t* qnv, const uint8_t* qsc, const uint8_t* knv, const uint8_t* ksc,
                             const uint8_t* vdnv, const uint8_t* vdsc, const uint8_t* donv,
                             const uint8_t* dosc, const uint8_t* dotnv, const uint8_t* dotsc,
                             const uint8_t* qtnv, const uint8_t* qtsc, const uint8_t* ktnv,
                             const uint8_t* ktsc, const float* lse, const float* delta,
                             const float* do_amax, const float* key_bias, const int32_t* seq_start,
                             const int32_t* seq_end, void* dq, void* dk, void* dv, int grad_dtype,
                             int64_t z, int64_t h, int64_t hk, int64_t s_q, int64_t s_kv,
                             int64_t sq_pad, int64_t skv_pad, int d, float scaling, int flags,
                             uint32_t seed, int* status, nvfp4_stream_t stream) {
  using namespace nvfp4;
  NVFP4_REQUIRE(d == 128 || d == 256, "nvfp4_bwd_fp4: head dim must be 128 or 256");
  NVFP4_REQUIRE(z >= 1 && h >= 1 && hk >= 1 && h % hk == 0, "nvfp4_bwd_fp4: bad head counts");
  NVFP4_REQUIRE(s_q >= 1 && s_kv >= 1 && s_q < (1LL << 30) && s_kv < (1LL << 30), "nvfp4_bwd_fp4: bad sequence extents");
  NVFP4_REQUIRE(sq_pad % 128 == 0 && sq_pad >= s_q && skv_pad % 128 == 0 && skv_pad >= s_kv,
                "nvfp4_bwd_fp4: transposed packs must be padded to a multiple of 128 columns");
  NVFP4_REQUIRE(qnv && qsc && knv && ksc && vdnv && vdsc && donv && dosc && dotnv && dotsc && qtnv && qtsc && ktnv &&
                    ktsc && lse && delta && do_amax && dq && dk && dv,
                "nvfp4_bwd_fp4: null pointer");
  const bool varlen = seq_start != nullptr;
  NVFP4_REQUIRE(varlen == (seq_end != nullptr), "nvfp4_bwd_fp4: seq_start and seq_end go together");
  NVFP4_REQUIRE(!varlen || (z == 1 && s_q == s_kv), "nvfp4_bwd_fp4: varlen needs Z == 1 and Sq == Skv");
  NVFP4_REQUIRE(!(flags & NVFP4_FWD_CAUSAL) || varlen || s_kv >= s_q, "nvfp4_bwd_fp4: causal needs Skv >= Sq");
  NVFP4_REQUIRE((s_kv + 127) / 128 < 65536 && z * h < (1LL << 31) && (s_q + 127) / 128 < 65536,
                "nvfp4_bwd_fp4: grid too large");
  NVFP4_REQUIRE((((uintptr_t)qsc | (uintptr_t)ksc | (uintptr_t)vdsc | (uintptr_t)dosc | (uintptr_t)dotsc |
                  (uintptr_t)qtsc | (uintptr_t)ktsc) & 3) == 0,
                "nvfp4_bwd_fp4: scale tensors must be 4-byte aligned");
  const bool fp8 = (flags & NVFP4_BWD_MXFP8) != 0;
  NVFP4_REQUIRE(!fp8 || !(flags & (NVFP4_BWD_SR_DS_DK | NVFP4_BWD_SR_P_DV | NVFP4_BWD_SR_DS_DQ)),
                "nvfp4_bwd_fp4: the MXFP8 operands round to nearest only");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t zh = z * h, zhk = z * hk;
  const uint64_t pb = (uint64_t)d / 2;
  CUtensorMap t_q, t_k, t_vd, t_do, t_dot, t_qt, t_kt;
  int rc;
  if ((rc = make_tmap_u8_3d_sw64(&t_q, qnv, pb, s_q, zh, pb, (uint64_t)s_q * pb, 128, "nvfp4_bwd_fp4(Q)"))) return rc;
  if ((rc = make_tmap_u8_3d_sw64(&t_k, knv, pb, s_kv, zhk, pb, (uint64_t)s_kv * pb, 128, "nvfp4_bwd_fp4(K)"))) return rc;
  if ((rc = make_tmap_u8_3d_sw64(&t_vd, vdnv, pb, s_kv, zhk, pb, (uint64_t)s_kv * pb, 128, "nvfp4_bwd_fp4(V)"))) return rc;
  if ((rc = make_tmap_u8_3d_sw64(&t_do, donv, pb, s_q, zh, pb, (uint64_t)s_q * pb, 128, "nvfp4_bwd_fp4(dO)"))) return rc;
  if (fp8) {      // transposed operands: one byte per element, 128-byte boxes
    if ((rc = make_tmap_u8_3d_sw128(&t_dot, dotnv, (uint64_t)sq_pad, d, zh, (uint64_t)sq_pad, (uint64_t)d * sq_pad, 128,
                                    "nvfp4_bwd_fp4(dO^T)"))) return rc;
    if ((rc = make_tmap_u8_3d_sw128(&t_qt, qtnv, (uint64_t)sq_pad, d, zh, (uint64_t)sq_pad, (uint64_t)d * sq_pad, 128,
                                    "nvfp4_bwd_fp4(Q^T)"))) return rc;
    if ((rc = make_tmap_u8_3d_sw128(&t_kt, ktnv, (uint64_t)skv_pad, d, zhk, (uint64_t)skv_pad, (uint64_t)d * skv_pad, 128,
                                    "nvfp4_bwd_fp4(K^T)"))) return rc;
  } else {
    if ((rc = make_tmap_u8_3d_sw64(&t_dot, dotnv, (uint64_t)sq_pad / 2, d, zh, (uint64_t)sq_pad / 2,
                                   (uint64_t)d * (sq_pad / 2), 128, "nvfp4_bwd_fp4(dO^T)"))) return rc;
    if ((rc = make_tmap_u8_3d_sw64(&t_qt, qtnv, (uint64_t)sq_pad / 2, d, zh, (uint64_t)sq_pad / 2,
                                   (uint64_t)d * (sq_pad / 2), 128, "nvfp4_bwd_fp4(Q^T)"))) return rc;
    if ((rc = make_tmap_u8_3d_sw64(&t_kt, ktnv, (uint64_t)skv_pad / 2, d, zhk, (uint64_t)skv_pad / 2,
                                   (uint64_t)d * (skv_pad / 2), 128, "nvfp4_bwd_fp4(K^T)"))) return rc;
  }
  B4Params p;
  p.lse = lse; p.delta = delta; p.amax = do_amax; p.bias = key_bias;
  p.seq_start = seq_start; p.seq_end = seq_end;
  p.h = (int)h; p.hk = (int)hk; p.g = (int)(h / hk); p.s_q = (int)s_q; p.s_kv = (int)s_kv;
  p.scaling = scaling; p.causal = (flags & NVFP4_FWD_CAUSAL) ? 1 : 0; p.status = status;
  p.seed = seed; p.sr_p = 0; p.sr_ds = 0;
  p.late_wait = 0; p.split = 1;
  p.vec = (((uintptr_t)qsc | (uintptr_t)ksc | (uintptr_t)vdsc | (uintptr_t)dosc | (uintptr_t)dotsc | (uintptr_t)qtsc | (uintptr_t)ktsc) & 15) == 0;
  // The passes are independent of one another: the first waits for the work before it, the later ones
  // start filling the SMs that its last CTAs leave and wait for it only at their end.
  bool first = true;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  auto launch_pass = [&](const char* what, auto kern, int smem, int threads, bool keys) -> int {
    if (int r0 = allow_smem(what, reinterpret_cast<const void*>(kern), smem)) return r0;
    B4Params a = p;
    a.late_wait = first ? 0 : 1;
    first = false;
    if (keys) {   // dV / dK: rows = keys (K, V packs), columns = queries (Q, dO' packs; dO'^T, Q^T transposed packs)
      a.x1sc = ksc; a.x2sc = vdsc; a.y1sc = qsc; a.y2sc = dosc; a.t1sc = dotsc; a.t2sc = qtsc;
      a.out1 = dv; a.out2 = dk; a.c_pad = (int)sq_pad;
      a.sr_p = (flags & NVFP4_BWD_SR_P_DV) ? 1 : 0; a.sr_ds = (flags & NVFP4_BWD_SR_DS_DK) ? 1 : 0;
      const int64_t g = h / hk, tiles = (s_kv + 127) / 128;
      int slots[4];
      cluster_slots(reinterpret_cast<const void*>(kern), threads, smem, sms, slots);
      a.split = cluster_split(zhk * tiles, g * ((s_q + 127) / 128), p.causal ? g : g * ((s_q + 127) / 128), varlen, slots);
      return launch_cluster(what, kern, dim3((unsigned)zhk, (unsigned)tiles, (unsigned)a.split), a.split, threads, smem, st, t_k,
                            t_vd, t_q, t_do, t_dot, t_qt, a);
    }
    // dQ: rows = queries (Q, dO' packs), columns = keys (K, V packs; K^T transposed pack)
    a.x1sc = qsc; a.x2sc = dosc; a.y1sc = ksc; a.y2sc = vdsc; a.t1sc = nullptr; a.t2sc = ktsc;
    a.out1 = nullptr; a.out2 = dq; a.c_pad = (int)skv_pad;
    a.sr_ds = (flags & NVFP4_BWD_SR_DS_DQ) ? 1 : 0;
    return launch(what, kern, dim3((unsigned)zh, (unsigned)((s_q + 127) / 128)), threads, smem, st, t_q, t_do, t_k, t_vd,
                  t_kt, t_kt, a);
  };
  const bool any_sr = (flags & (NVFP4_BWD_SR_DS_DK | NVFP4_BWD_SR_P_DV | NVFP4_BWD_SR_DS_DQ)) != 0;
#define NVFP4_B4_PASS(DD, PASS, TT, MODE)                                                                     \
  launch_pass("nvfp4_bwd_fp4(" #PASS ")", bwd4_kernel<DD, PASS, TT, MODE>, B4Cfg<DD, PASS, MODE == 2>::TOTAL,  \
              B4Cfg<DD, PASS, MODE == 2>::THREADS, PASS != kB4Dq)
#define NVFP4_B4_MODE(DD, TT, MODE)                                        \
  {                                                                        \
    if constexpr (DD == 128) {                                             \
      if ((rc = NVFP4_B4_PASS(128, kB4DkDv, TT, MODE))) return rc;         \
    } else {                                                               \
      if ((rc = NVFP4_B4_PASS(256, kB4Dk, TT, MODE))) return rc;           \
      if ((rc = NVFP4_B4_PASS(256, kB4Dv, TT, MODE))) return rc;           \
    }                                                                      \
    return NVFP4_B4_PASS(DD, kB4Dq, TT, MODE);                             \
  }
#define NVFP4_B4_LAUNCH(DD, TT)          \
  {                                      \
    if (fp8) NVFP4_B4_MODE(DD, TT, 2)    \
    if (any_sr) NVFP4_B4_MODE(DD, TT, 1) \
    NVFP4_B4_MODE(DD, TT, 0)             \
  }
  if (d == 128) {
    switch (grad_dtype) {
      case NVFP4_DT_BF16: NVFP4_B4_LAUNCH(128, __nv_bfloat16)
      case NVFP4_DT_FP16: NVFP4_B4_LAUNCH(128, __half);
      case NVFP4_DT_FP32: NVFP4_B4_LAUNCH(128, float);
      default: return fail(-1, "nvfp4_bwd_fp4: unknown grad dtype %d", grad_dtype);
    }
  }
  switch (grad_dtype) {
    case NVFP4_DT_BF16: NVFP4_B4_LAUNCH(256, __nv_bfloat16);
    case NVFP4_DT_FP16: NVFP4_B4_LAUNCH(256, __half);
    case NVFP4_DT_FP32: NVFP4_B4_LAUNCH(256, float);
    default: return fail(-1, "nvfp4_bwd_fp4: unknown grad dtype %d", grad_dtype);
  }
#undef NVFP4_B4_LAUNCH
#undef NVFP4_B4_MODE
#undef NVFP4_B4_PASS
}

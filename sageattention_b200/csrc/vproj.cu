// V projection with the NVFP4 pack as its epilogue: V = X W^T (+ bias) is computed on the tensor
// cores and leaves the kernel as the V^T pack along the keys that the attention kernels read (and,
// optionally, as the 16-bit V itself), so the projected tensor is never re-read for quantisation.
// This is the "v_proj epilogue" producer the reference's notes ask callers to fuse.
//
// The product is formed TRANSPOSED, V^T[feature, token] = W[feature, :] . X[token, :], so that the
// accumulator puts one output feature (one row of the V^T pack) on one TMEM lane and 128 consecutive
// tokens on its columns: the 16-token groups of the pack are thread-local in the epilogue and a
// thread writes 64 contiguous nibble bytes + 8 scale bytes of its row.
//
// One CTA = 128 features x NT tokens (128, 64 or 32) of one batch entry; K loop over the hidden dim in 64-element
// stages (TMA, 128-byte swizzle, ring of 3 to 8), tcgen05.mma kind::f16 M128 N=NT K16, accumulator in
// NT TMEM columns.  Warps: 0 TMA producer, 1 MMA issuer, the others epilogue (32 tokens of 32 features at a time).
//
// What bounds it: a stage's 32 KB (NT = 128) take ~470 clocks to arrive (an SM's share of L2; the MMAs need 260; a
// ring of six stages is no faster), so a tile of hidden 4096 costs 16 us however few there are.  The hidden dim
// is not split: V is rounded, packed to FP4 and attended, and a sum in another order moves single outputs by
// as much as their size.  Where tiles are fewer than SMs they are cut along the tokens instead, with
// 24 or 20 KB a stage.
#include "common/abi.cuh"
#include "common/fp4.cuh"
#include "common/launch.cuh"
#include "common/sm100.cuh"
#include "common/tma_host.cuh"
#include "common/bwd_util.cuh"

namespace nvfp4 {

constexpr int kVpTile = 128 * 64 * 2;      // bytes of the W tile of a stage

template <int kNT, int kPerSm>             // tokens of a tile, CTAs per SM the kernel is built for
struct VpCfg {
  static constexpr int STAGES = kPerSm == 2 ? 3 : (kNT == 128 ? 4 : 8);     // a narrow tile is bound by latency
  static constexpr int STAGE_BYTES = kVpTile + kNT * 128;
  static constexpr int EPI = kPerSm == 1 ? kNT * 4 : 256;   // epilogue threads
  static constexpr int THREADS = 64 + EPI;
};

struct VprojParams {
  const void* bias;      // [features] in the operand dtype, or null
  uint8_t* vnv;          // [Z*Hk, D, s_pad/2]
  uint8_t* vsc;          // [Z*Hk, D, s_pad/16]
  void* v_out;           // [Z, S, features] (element strides svb, svs; unit feature stride) or null
  int64_t svb, svs;
  int features, d, hk, s, s_pad, hidden;
  int f16;
  int* status;
};

// 16 tokens from `tok` of feature f: bias, rounding to the operand dtype (what an unfused projection would have
// stored), the value and its pack; tokens behind S are +0.0, groups behind the padded extent do not exist.
// Tiles of 128 tokens are held to 96 registers and divide: the quotient by products spilled 24 to 36 bytes there, fp16
// [8192, 4096] x 1024 79.3 -> 77.7 us; narrower ones have the registers, [128, 1024] x 256 6.57 -> 6.34.
template <typename T, int kNT>
__device__ __forceinline__ void vproj_store(const VprojParams& p, int zi, int f, int tok, float (&v)[16]) {
  if (f >= p.features || tok >= p.s_pad) return;
  const float b = p.bias != nullptr ? to_f32<T>(static_cast<const T*>(p.bias)[f]) : 0.0f;
  T* vo = p.v_out ? static_cast<T*>(p.v_out) + (int64_t)zi * p.svb + f : nullptr;
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const T hv = from_f32<T>(v[e] + b);
    v[e] = (tok + e < p.s) ? to_f32<T>(hv) : 0.0f;
    if (vo != nullptr && tok + e < p.s) vo[(int64_t)(tok + e) * p.svs] = hv;
  }
  uint32_t lo, hi;
  const uint8_t sb = kNT == 128 ? pack_group16(v, lo, hi) : pack_group16_of<T>(v, lo, hi);
  const int64_t row = ((int64_t)zi * p.hk + f / p.d) * p.d + f % p.d;
  *reinterpret_cast<uint2*>(p.vnv + row * (p.s_pad / 2) + tok / 2) = make_uint2(lo, hi);
  p.vsc[row * (p.s_pad / 16) + tok / 16] = sb;
}

// Tokens of a tile and CTAs per SM: the narrowest tile of which one wave covers the problem; beyond a wave of
// the widest, two CTAs per SM, one's start and epilogue under the other's loads.  [S, hidden] x features: 509 x 4096 x 1024
// 22.6 us (128 tokens) -> 17.4 (32), 128 x 2048 x 512 14.9 -> 10.3, 2430 x 4096 x 1024 44.9 -> 33, 8192 x 4096 x 1024 109 -> 76, 7486 x 1024 x 2048 80 -> 58.
struct VpPlan { int nt, per_sm; };
inline VpPlan vproj_plan(int64_t row_tiles, int64_t s_pad, int sms) {
  for (int nt = 32; nt <= 128; nt *= 2)
    if (row_tiles * ((s_pad + nt - 1) / nt) <= sms) return {nt, 1};
  return {128, 2};
}

template <typename T, int kNT, int kPerSm>
__global__ void __launch_bounds__(VpCfg<kNT, kPerSm>::THREADS, kPerSm)
vproj_pack_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                  const VprojParams p) {
  using C = VpCfg<kNT, kPerSm>;
  constexpr int kVpStages = C::STAGES;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  __shared__ uint64_t full[kVpStages], empty[kVpStages], acc_done;
  __shared__ uint32_t tmem_base_s;
  __shared__ int err;
  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int f0 = blockIdx.x * 128, t0 = blockIdx.y * kNT, zi = blockIdx.z;
  const int nstage = (p.hidden + 63) / 64;
  if (tid == 0) {
    err = 0;
    for (int i = 0; i < kVpStages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(&acc_done, 1);
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(&tmem_base_s, 128);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  griddep_launch();
  griddep_wait();
  const uint32_t tmem = tmem_base_s;

  if (warp == 0) {
    if (elect_one()) {
      for (int st = 0; st < nstage; ++st) {
        const int s = st % kVpStages;
        if (st >= kVpStages) mbar_wait(&empty[s], ((st / kVpStages) & 1) ^ 1, &err, 1);
        uint8_t* sb = smem + s * C::STAGE_BYTES;
        mbar_expect_tx(&full[s], C::STAGE_BYTES);
        tma_load_3d(sb, &tm_w, &full[s], st * 64, f0, 0);
        tma_load_3d(sb + kVpTile, &tm_x, &full[s], st * 64, t0, zi);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc_bf16(128, kNT, false, p.f16 != 0);
      for (int st = 0; st < nstage; ++st) {
        const int s = st % kVpStages;
        mbar_wait(&full[s], (st / kVpStages) & 1, &err, 2);
        tc_fence_after();
        const uint8_t* sb = smem + s * C::STAGE_BYTES;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_bf16(tmem, desc_sw128(sb, k), desc_sw128(sb + kVpTile, k), idesc, (st > 0 || k > 0) ? 1u : 0u);
        umma_commit(&empty[s]);
      }
      umma_commit(&acc_done);
    }
    __syncwarp();
  } else {
    // epilogue: thread = feature row 32 (warp % 4) + lane, 32 of the tokens
    const int row = (warp & 3) * 32 + lane;
    mbar_wait(&acc_done, 0, &err, 3);
    tc_fence_after();
#pragma unroll 1
    for (int c = (tid - 64) >> 7; c < kNT / 32; c += C::EPI / 128) {
      uint32_t r[32];
      tmem_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + c * 32, r);
      tmem_ld_wait();
#pragma unroll
      for (int gi = 0; gi < 2; ++gi) {
        float v[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = __uint_as_float(r[gi * 16 + e]);
        vproj_store<T, kNT>(p, zi, f0 + row, t0 + c * 32 + gi * 16, v);
      }
    }
    tc_fence_before();
  }
  __syncthreads();
  report_error(&err, p.status);
  if (warp == 1) tmem_dealloc(tmem, 128);
}

}  // namespace nvfp4

extern "C" int nvfp4_vproj_pack(const void* x, const void* w, const void* bias, int dtype, int64_t z,
                                int64_t s, int64_t hidden, int64_t hk, int d, int64_t sxb, int64_t sxs,
                                int64_t s_pad, uint8_t* vnv, uint8_t* vsc, void* v_out, int64_t svb,
                                int64_t svs, int* status, nvfp4_stream_t stream) {
  using namespace nvfp4;
  NVFP4_REQUIRE(dtype == NVFP4_DT_BF16 || dtype == NVFP4_DT_FP16, "nvfp4_vproj_pack: operands must be bf16 or fp16");
  NVFP4_REQUIRE(x && w && vnv && vsc, "nvfp4_vproj_pack: null pointer");
  NVFP4_REQUIRE(z >= 1 && s >= 1 && hk >= 1 && d >= 16 && d % 16 == 0, "nvfp4_vproj_pack: bad extents");
  NVFP4_REQUIRE(hidden >= 8 && hidden % 8 == 0, "nvfp4_vproj_pack: hidden size must be a multiple of 8");
  NVFP4_REQUIRE(s_pad % 16 == 0 && s_pad >= s, "nvfp4_vproj_pack: s_pad must be a multiple of 16 >= s");
  NVFP4_REQUIRE(sxb % 8 == 0 && sxs % 8 == 0, "nvfp4_vproj_pack: activation strides must be multiples of 8 elements");
  NVFP4_REQUIRE(((uintptr_t)vnv & 7) == 0 && (s_pad / 2) % 8 == 0, "nvfp4_vproj_pack: nibble rows must be 8-byte aligned");
  const int64_t features = hk * d;
  NVFP4_REQUIRE(features < (1LL << 30) && s_pad < (1LL << 30) && z < 65536 && (s_pad + 127) / 128 < 65536,
                "nvfp4_vproj_pack: problem too large");
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t tf = (features + 127) / 128;
  const VpPlan plan = vproj_plan(tf * z, s_pad, sms);
  CUtensorMap t_w, t_x;
  int rc;
  if ((rc = make_tmap_bf16_3d_sw128(&t_w, w, (uint64_t)hidden, (uint64_t)features, 1, (uint64_t)hidden * 2,
                                    (uint64_t)features * hidden * 2, 128, "nvfp4_vproj_pack(W)")))
    return rc;
  if ((rc = make_tmap_bf16_3d_sw128(&t_x, x, (uint64_t)hidden, (uint64_t)s, (uint64_t)z, (uint64_t)sxs * 2,
                                    (uint64_t)(z > 1 ? sxb : s * sxs) * 2, (uint32_t)plan.nt, "nvfp4_vproj_pack(X)")))
    return rc;
  VprojParams p;
  p.bias = bias; p.vnv = vnv; p.vsc = vsc; p.v_out = v_out; p.svb = svb; p.svs = svs;
  p.features = (int)features; p.d = d; p.hk = (int)hk; p.s = (int)s; p.s_pad = (int)s_pad; p.hidden = (int)hidden;
  p.f16 = dtype == NVFP4_DT_FP16 ? 1 : 0; p.status = status;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const dim3 grid((unsigned)tf, (unsigned)((s_pad + plan.nt - 1) / plan.nt), (unsigned)z);
  auto run = [&](auto kern, int threads, int ring) -> int {
    if (int r0 = allow_smem("nvfp4_vproj_pack", reinterpret_cast<const void*>(kern), ring + 1024)) return r0;
    return launch("nvfp4_vproj_pack", kern, grid, threads, ring + 1024, st, t_w, t_x, p);
  };
#define NVFP4_VP(T, NT, PER) \
  run(vproj_pack_kernel<T, NT, PER>, VpCfg<NT, PER>::THREADS, VpCfg<NT, PER>::STAGES * VpCfg<NT, PER>::STAGE_BYTES)
#define NVFP4_VP_T(T)                                      \
  return plan.per_sm == 2 ? NVFP4_VP(T, 128, 2)            \
         : plan.nt == 128 ? NVFP4_VP(T, 128, 1)            \
         : plan.nt == 64  ? NVFP4_VP(T, 64, 1)             \
                          : NVFP4_VP(T, 32, 1)
  if (dtype == NVFP4_DT_BF16) { NVFP4_VP_T(__nv_bfloat16); }
  NVFP4_VP_T(__half);
#undef NVFP4_VP_T
#undef NVFP4_VP
}

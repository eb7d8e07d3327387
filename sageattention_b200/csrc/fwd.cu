// NVFP4 flash-attention forward for sm_100a.
//
// One CTA owns a 128-row query tile of one (batch, head) and walks 128-key tiles:
//     S[128 x 128]  = Q_tile . K_tile^T        tcgen05.mma kind::mxf4nvf4, e4m3 scale per 16
//     P             = exp(S*scale - m) packed to NVFP4 per 16 keys (same scale rule as the packer)
//     O[128 x D]   += P . V_tile               same MMA kind, V held as V^T (packed along keys)
// Q/K/V^T nibble tiles arrive by TMA straight from the packed tensors; scale bytes are re-laid
// into the 32x16-byte form tcgen05.cp expects by a loader warp; S and O live in TMEM.  The running
// maximum is exact (O is rescaled in TMEM whenever a row's maximum moves), which keeps the P
// quantisation decisions those of a plain 128-key tile walk.
//
// Warps (608 threads): 0 TMA producer + scale loader (+bias), 1 QK^T issuer, 2 PV
// issuer, 3-18 softmax / correction / epilogue in two groups of eight that alternate key tiles.
// Within a group two threads share a query row, 64 key columns each, so the per-16-key P pack needs
// no cross-thread traffic.  Every barrier wait is bounded.
//
// What bounds it: the floor is one ex2 per score (16 lanes per clock and SM, 1024 clocks per tile at
// D = 128); a softmax warp's tile is a chain -- wait, read, maxima, exchange, exponentials and pack,
// rescale of O -- that is about four times its share of that, and two groups hide half of it.  What the
// layout does about the chain: the running maximum is not handed from tile to tile; every thread
// publishes the maximum of its 64 columns and forms the exact running maximum itself from its group's
// last one, the two of the tile in between and the other half's (one 64-thread barrier with the warp
// that holds it); reciprocal scales come from a table in shared memory, not from the pipe that ex2
// needs; P leaves in 16-byte stores.  Measured on a B200, causal bf16: Z4 H32 Hk8 S8192 D128
// 2228 -> 2035 us (1.08 PFLOP/s), H16 Hk4 S8192 D256 441 -> 335 us, S1024 D256 26.0 -> 17.5 us.
// Masks: a score is tested only in tiles at an edge of what a row may see -- diagonal, ragged end, ends of a
// packed sample -- as a bit of a 32-column word formed from the row's range; no sample ids are read per score.
// A bias is added, already divided by the scaling, only in tiles where some value of it is not zero, which in a
// padded batch are the few at the end.  Z2 H32 Sq1029 Skv2309 padded 152 -> 111 us (98 without a bias),
// packed 8 samples in 16384 tokens H32 D128 584 -> 498 us, H16 D256 364 -> 320 us.
// Registers decide here (96 per thread at nineteen warps): variants that spilled even a few hundred
// bytes took up to three times as long.
#include "common/abi.cuh"
#include "common/fp4.cuh"
#include "common/launch.cuh"
#include "common/sm100.cuh"
#include "common/tma_host.cuh"

namespace nvfp4 {

constexpr int kFwdRoleWarps = 3;
constexpr int kFwdThreads = 32 * (kFwdRoleWarps + 16);
constexpr float kFwdLog2e = 1.4426950408889634f;
// Tiles whose row maxima are kept for exchange.  A slot may be rewritten six tiles later at the earliest:
// a thread that publishes tile i has waited for tile i - 3 of the other group, which by then has read i - 6.
constexpr int kFwdMaxSlots = 8;

template <int D>
struct FwdCfg {
  static constexpr int KSUB = D / 128;  // 64-byte-wide sub-tiles of a Q/K row
  static constexpr int KB = D / 64;     // K=64 MMAs per QK tile
  static constexpr int NT = D / 128;    // 128-row pieces of the V^T tile (N of the PV MMA = D)
  static constexpr int NSBUF = (D == 128) ? 2 : 1;  // S buffers
  // D = 256: the one S buffer is emptied into registers at once; D = 128 reads it twice in 32-column
  // chunks instead (maxima, then exponentials), which keeps the loop free of spills
  static constexpr bool kOneRead = NSBUF == 1;
  static constexpr int NSTAGE = (D == 128) ? 4 : 3;
  static constexpr int Q_BYTES = KSUB * 8192;
  static constexpr int K_BYTES = KSUB * 8192;
  static constexpr int V_BYTES = NT * 8192;
  static constexpr int KSF_BYTES = KB * 512;
  static constexpr int VSF_BYTES = 2 * NT * 512;  // [kb][nt]
  static constexpr int AUX_BYTES = 1024;          // 128 fp32 bias; stages stay 1 KB aligned
  static constexpr int STAGE_BYTES = K_BYTES + V_BYTES + KSF_BYTES + VSF_BYTES + AUX_BYTES;
  static constexpr int QSF_BYTES = KB * 512;
  static constexpr int P_BYTES = 8192;
  static constexpr int PSF_BYTES = 1024;
  static constexpr int SMEM_BYTES = NSTAGE * STAGE_BYTES + Q_BYTES + QSF_BYTES + 2 * (P_BYTES + PSF_BYTES) + 1024;
  // TMEM columns
  static constexpr int T_S = 0;                       // NSBUF x 128
  static constexpr int T_O = NSBUF * 128;             // D
  static constexpr int T_SFQ = T_O + D;               // KB * 4
  static constexpr int T_SFK = T_SFQ + KB * 4;        // 2 x KB * 4
  static constexpr int T_SFP = T_SFK + 2 * KB * 4;    // 2 x 8
  static constexpr int T_SFV = T_SFP + 16;            // 2 x (2 * NT * 4)
  static constexpr int T_END = T_SFV + 2 * 2 * NT * 4;
  static_assert(T_END <= 512, "TMEM budget exceeded");
};

struct FwdParams {
  const uint8_t* qsc;  // [ZH, Sq, D/16]
  const uint8_t* ksc;  // [ZHk, Skv, D/16]
  const uint8_t* vsc;  // [ZHk, D, s_pad/16]
  const float* bias;   // [Z, Skv] or null
  const int32_t* seq_id;     // [S] or null
  const int32_t* seq_start;  // [S] or null
  void* out;
  int64_t so_z, so_h, so_s;
  float* lse;  // [ZH, Sq] or null
  int h, hk, g;
  int s_q, s_kv, s_pad;
  float scaling;
  int causal;
  int* status;
};

__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void fwd_sts_v4(uint32_t saddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(saddr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// kVarlen: packed rows with per-token sample ids; kBias: additive key bias.  Instantiations of their own keep
// the plain kernel free of the tests (with the bias as a run-time branch it took 9 % longer).
template <int D, typename TO, bool kVarlen, bool kBias>
__global__ void __launch_bounds__(kFwdThreads, 1)
fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
           const __grid_constant__ CUtensorMap tm_v, const FwdParams p) {
  using C = FwdCfg<D>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* s_stage = smem;
  uint8_t* s_q = s_stage + C::NSTAGE * C::STAGE_BYTES;
  uint8_t* s_p = s_q + C::Q_BYTES;
  uint8_t* s_psf = s_p + 2 * C::P_BYTES;
  uint8_t* s_qsf = s_psf + 2 * C::PSF_BYTES;

  __shared__ uint64_t full_kv[C::NSTAGE], full_sf[C::NSTAGE], empty[C::NSTAGE];
  __shared__ uint64_t s_full[2], s_free[2], p_full[2], pv_done[2], q_full, qsf_full;
  __shared__ uint64_t mx_ready[kFwdMaxSlots][4];     // row maxima of a tile, one barrier per 32-row quadrant
  __shared__ uint32_t tmem_base_s;
  __shared__ int err;
  __shared__ int s_lo_tile;
  __shared__ int s_biased[C::NSTAGE];                // the tile's bias has a value other than zero
  __shared__ float xmax[kFwdMaxSlots][2][128];       // [tile % slots][key half][row]
  __shared__ float xl[4][128];
  __shared__ float xm[2][128];
  __shared__ float inv_tab[128];                     // reciprocal of every (non-negative) e4m3 byte

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // grid = (heads, query tiles): all heads of the heaviest (last) query tile are scheduled first,
  // so the kernel ends on the cheapest tiles instead of on a long straggler
  const int mblk = gridDim.y - 1 - blockIdx.y;
  const int zh = blockIdx.x;
  const int zi = zh / p.h, hi = zh % p.h;
  const int unit = zi * p.hk + hi / p.g;  // (batch, kv head)
  const int m0 = mblk * 128;
  const int shift = p.s_kv - p.s_q;  // bottom-right aligned causal offset

  // key-tile range of this query tile
  int hi_key = p.s_kv;
  if (p.causal) hi_key = min(p.s_kv, m0 + 128 + shift);
  if (hi_key < 0) hi_key = 0;
  const int t_hi = (hi_key + 127) / 128;

  if (tid == 0) {
    err = 0;
    for (int i = 0; i < C::NSTAGE; ++i) {
      mbar_init(&full_kv[i], 1);
      mbar_init(&full_sf[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&s_free[i], 8);
      mbar_init(&p_full[i], 8);
      mbar_init(&pv_done[i], 1);
    }
    for (int i = 0; i < kFwdMaxSlots; ++i)
      for (int q = 0; q < 4; ++q) mbar_init(&mx_ready[i][q], 2);
    mbar_init(&q_full, 1);
    mbar_init(&qsf_full, 4);
    mbar_fence_init();
  }
  if (tid >= 128 && tid < 256) {
    float inv;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(e4m3_to_f32((uint8_t)(tid - 128))));
    inv_tab[tid - 128] = inv;
  }
  if (warp == 1) tmem_alloc(&tmem_base_s, 512);
  griddep_wait();
  if (tid == 0) s_lo_tile = kVarlen ? p.seq_start[min(m0, p.s_q - 1)] / 128 : 0;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  griddep_launch();
  const uint32_t tmem = tmem_base_s;
  // varlen: rows of a tile are sorted by sample, so the first row has the earliest start
  const int t_lo = s_lo_tile;
  const int ntile = max(t_hi - t_lo, 0);

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer, scale loader
    // K scales (+ key bias) and V^T scales of a tile, re-laid into the 32 x 16-byte
    // atoms tcgen05.cp copies.  The next tile's bytes are fetched into registers one tile
    // ahead, so per tile the warp pays a shared-memory store, not a trip to L2.
    const bool leader = elect_one();
    auto load_tile = [&](int i) {
      const int s = i % C::NSTAGE, t = t_lo + i;
      uint8_t* st = s_stage + s * C::STAGE_BYTES;
      mbar_expect_tx(&full_kv[s], C::K_BYTES + C::V_BYTES);
#pragma unroll
      for (int ks = 0; ks < C::KSUB; ++ks) tma_load_3d(st + ks * 8192, &tm_k, &full_kv[s], ks * 64, t * 128, unit);
#pragma unroll
      for (int nt = 0; nt < C::NT; ++nt)
        tma_load_3d(st + C::K_BYTES + nt * 8192, &tm_v, &full_kv[s], t * 64, nt * 128, unit);
    };
    if (leader && ntile > 0) {
      mbar_expect_tx(&q_full, C::Q_BYTES);
#pragma unroll
      for (int ks = 0; ks < C::KSUB; ++ks) tma_load_3d(s_q + ks * 8192, &tm_q, &q_full, ks * 64, m0, zh);
      for (int i = 0; i < min(ntile, C::NSTAGE); ++i) load_tile(i);
    }
    __syncwarp();
    const uint8_t* ksrc = p.ksc + (int64_t)unit * p.s_kv * (D / 16);
    const uint8_t* vsrc = p.vsc + (int64_t)unit * D * (p.s_pad / 16);
    const float inv_scaling = kBias ? 1.0f / p.scaling : 0.0f;      // the bias is added to the unscaled scores
    uint32_t kx[4][C::KB];
    float nb[4];
    uint2 vx[D / 32];
    auto fetch = [&](int t) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = t * 128 + lane + 32 * j;
#pragma unroll
        for (int k = 0; k < C::KB; ++k) kx[j][k] = 0u;
        nb[j] = 0.0f;
        if (key < p.s_kv) {
          const uint32_t* gsrc = reinterpret_cast<const uint32_t*>(ksrc + (int64_t)key * (D / 16));
#pragma unroll
          for (int k = 0; k < C::KB; ++k) kx[j][k] = __ldg(gsrc + k);
          if (kBias) nb[j] = __ldg(p.bias + (int64_t)zi * p.s_kv + key) * inv_scaling;
        }
      }
#pragma unroll
      for (int j = 0; j < D / 32; ++j)
        vx[j] = __ldg(reinterpret_cast<const uint2*>(vsrc + (int64_t)(lane + 32 * j) * (p.s_pad / 16) + (int64_t)t * 8));
    };
    if (ntile > 0) fetch(t_lo);
    for (int i = 0; i < ntile; ++i) {
      const int s = i % C::NSTAGE;
      if (i >= C::NSTAGE) {
        mbar_wait(&empty[s], ((i / C::NSTAGE) & 1) ^ 1, &err, 1);
        if (leader) load_tile(i);
      }
      uint8_t* st = s_stage + s * C::STAGE_BYTES + C::K_BYTES + C::V_BYTES;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int r = lane + 32 * j;
#pragma unroll
        for (int k = 0; k < C::KB; ++k)
          *reinterpret_cast<uint32_t*>(st + k * 512 + sf_atom_offset(r, 0)) = kx[j][k];
        if (kBias) reinterpret_cast<float*>(st + C::KSF_BYTES + C::VSF_BYTES)[r] = nb[j];
      }
      if (kBias) {
        const int any = __any_sync(0xffffffffu, nb[0] != 0.0f || nb[1] != 0.0f || nb[2] != 0.0f || nb[3] != 0.0f);
        if (lane == 0) s_biased[s] = any;
      }
      uint8_t* dst = st + C::KSF_BYTES;
#pragma unroll
      for (int j = 0; j < D / 32; ++j) {
        const int dr = lane + 32 * j;
        const int nt = dr >> 7, r = dr & 127;
        *reinterpret_cast<uint32_t*>(dst + (0 * C::NT + nt) * 512 + sf_atom_offset(r, 0)) = vx[j].x;
        *reinterpret_cast<uint32_t*>(dst + (1 * C::NT + nt) * 512 + sf_atom_offset(r, 0)) = vx[j].y;
      }
      if (i + 1 < ntile) fetch(t_lo + i + 1);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full_sf[s]);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ QK^T issuer
    if (elect_one() && ntile > 0) {
      const uint32_t idesc_qk = make_idesc_nvfp4(128, 128);
      mbar_wait(&q_full, 0, &err, 3);
      mbar_wait(&qsf_full, 0, &err, 4);
      tc_fence_after();
#pragma unroll
      for (int k = 0; k < C::KB; ++k)
        tmem_cp_32x128b_warpx4(tmem + C::T_SFQ + k * 4, smem_u32(s_qsf + k * 512));
      for (int j = 0; j < ntile; ++j) {
        const int s = j % C::NSTAGE, b = j % C::NSBUF;
        const uint32_t ph = (j / C::NSTAGE) & 1;
        mbar_wait(&full_kv[s], ph, &err, 5);
        mbar_wait(&full_sf[s], ph, &err, 6);
        if (j >= C::NSBUF) {      // the S buffer's last tile has been read into registers
          const int u = j - C::NSBUF;
          mbar_spin_wait(&s_free[u & 1], (u >> 1) & 1, &err, 7);
        }
        tc_fence_after();
        uint8_t* st = s_stage + s * C::STAGE_BYTES;
        const uint32_t sfk = tmem + C::T_SFK + (j & 1) * C::KB * 4;
#pragma unroll
        for (int k = 0; k < C::KB; ++k)
          tmem_cp_32x128b_warpx4(sfk + k * 4, smem_u32(st + C::K_BYTES + C::V_BYTES + k * 512));
#pragma unroll
        for (int k = 0; k < C::KB; ++k) {
          const uint64_t ad = make_smem_desc(smem_u32(s_q + (k >> 1) * 8192) + (k & 1) * 32, 16, 512, 4);
          const uint64_t bd = make_smem_desc(smem_u32(st + (k >> 1) * 8192) + (k & 1) * 32, 16, 512, 4);
          umma_nvfp4(tmem + C::T_S + b * 128, ad, bd, idesc_qk, tmem + C::T_SFQ + k * 4, sfk + k * 4,
                     k > 0);
        }
        umma_commit(&s_full[j & 1]);     // by tile parity: each group waits for its own tiles
      }
    }
    __syncwarp();
  } else if (warp == 2) {
    // ------------------------------------------------------------------ PV issuer
    // A thread of its own, so a QK^T for tile i+2 is never queued behind the wait for P(i).
    if (elect_one() && ntile > 0) {
      const uint32_t idesc_pv = make_idesc_nvfp4(128, D);
      for (int i = 0; i < ntile; ++i) {
        const int s = i % C::NSTAGE, b = i & 1;
        // the V tile and V scales of stage s landed before this tile's QK^T was issued, but this
        // thread has to observe them itself; it does so while P is still being written
        mbar_wait(&full_kv[s], (i / C::NSTAGE) & 1, &err, 15);
        mbar_wait(&full_sf[s], (i / C::NSTAGE) & 1, &err, 16);
        mbar_spin_wait(&p_full[b], (i >> 1) & 1, &err, 8);
        tc_fence_after();
        uint8_t* st = s_stage + s * C::STAGE_BYTES;
        const uint32_t sfp = tmem + C::T_SFP + b * 8;
        const uint32_t sfv = tmem + C::T_SFV + b * (2 * C::NT * 4);
#pragma unroll
        for (int k = 0; k < 2; ++k)
          tmem_cp_32x128b_warpx4(sfp + k * 4, smem_u32(s_psf + b * C::PSF_BYTES + k * 512));
#pragma unroll
        for (int k = 0; k < 2 * C::NT; ++k)
          tmem_cp_32x128b_warpx4(sfv + k * 4,
                                 smem_u32(st + C::K_BYTES + C::V_BYTES + C::KSF_BYTES + k * 512));
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const uint64_t ad = make_smem_desc(smem_u32(s_p + b * C::P_BYTES) + k * 32, 16, 512, 4);
          const uint64_t bd = make_smem_desc(smem_u32(st + C::K_BYTES) + k * 32, 16, 512, 4);
          umma_nvfp4(tmem + C::T_O, ad, bd, idesc_pv, sfp + k * 4, sfv + k * C::NT * 4,
                     (i > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(&pv_done[b]);
        umma_commit(&empty[s]);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ softmax / correction / epilogue
    const int sw = warp - kFwdRoleWarps;
    const int grp = sw >> 3;             // which tiles (parity)
    const int wq = warp & 3;             // TMEM lane quadrant
    const int half = (sw >> 2) & 1;      // which 64 key columns
    const int part = grp * 2 + half;     // 0..3: slice of O this thread stores in the epilogue
    const int row_in = wq * 32 + lane;
    const int row = m0 + row_in;
    const uint32_t lane_addr = (uint32_t)(wq * 32) << 16;
    constexpr int OC = D / 4;            // O columns stored per thread in the epilogue
    constexpr int RC = D / 2;            // O columns rescaled per thread (two threads per row in a group)
    if (part == 0) {
      uint32_t wds[C::KB];
#pragma unroll
      for (int k = 0; k < C::KB; ++k) wds[k] = 0u;
      if (row < p.s_q) {
        const uint32_t* gsrc =
            reinterpret_cast<const uint32_t*>(p.qsc + ((int64_t)zh * p.s_q + row) * (D / 16));
#pragma unroll
        for (int k = 0; k < C::KB; ++k) wds[k] = __ldg(gsrc + k);
      }
#pragma unroll
      for (int k = 0; k < C::KB; ++k)
        *reinterpret_cast<uint32_t*>(s_qsf + k * 512 + sf_atom_offset(row_in, 0)) = wds[k];
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&qsf_full);
    }
    // Visible keys of this row: one range, also in packed rows, whose ids are sorted (the row's sample, cut at
    // the row itself when causal).  Relative to this thread's first column of the first tile.
    const int row_c = min(row, p.s_q - 1);
    auto sample_end = [&](int r) {          // first key behind the sample of row r
      const int32_t id = p.seq_id[r];
      int lo = r + 1, hi = p.s_kv;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (p.seq_id[mid] == id) lo = mid + 1;
        else hi = mid;
      }
      return lo;
    };
    const int last = p.causal ? row + shift : (kVarlen ? sample_end(row_c) - 1 : p.s_kv - 1);
    const int rel = t_lo * 128 + half * 64;
    const int lim0 = min(last, p.s_kv - 1) - rel;
    const int beg0 = kVarlen ? p.seq_start[row_c] - rel : 0;
    // Tiles below i_first and from i_mask on need a test per score: the edge of a sample, the causal
    // diagonal, the ragged end.  A tile whose bias is all zero (the valid part of a padded batch) does not.
    const int last_full = min(p.causal ? m0 + shift + 1 : (kVarlen ? sample_end(min(m0, p.s_q - 1)) : p.s_kv), p.s_kv);
    const int i_mask = max(last_full, 0) / 128 - t_lo;     // keys below last_full are visible to every row
    const int i_first = kVarlen ? (p.seq_start[min(m0 + 127, p.s_q - 1)] + 127) / 128 - t_lo : 0;
    const float c2 = p.scaling * kFwdLog2e;
    float m_own = -INFINITY, l_run = 0.0f;   // running max (log2 units) after this group's last tile
    const uint32_t xmax_s = smem_u32(&xmax[0][0][0]) + (uint32_t)row_in * 4u;
    const uint32_t inv_s = smem_u32(inv_tab);
    const uint32_t pt = smem_u32(s_p + grp * C::P_BYTES) + sw64_offset(row_in, half * 32);   // the next 16 bytes: ^ 16
    const uint32_t psf = smem_u32(s_psf + grp * C::PSF_BYTES) + half * 512 + sf_atom_offset(row_in, 0);
    const uint32_t s_base = tmem + lane_addr + C::T_S + half * 64;

    // scores of N columns from column c of this thread's 64, masked where the tile needs it
    auto load_scores = [&](int i, int c, bool edge, bool biased, auto& sv) {
      constexpr int N = sizeof(sv) / sizeof(float);
      uint32_t r[N / 32][32];
      const uint32_t addr = s_base + (C::NSBUF == 2 ? grp * 128 : 0) + c;
#pragma unroll
      for (int k = 0; k < N / 32; ++k) tmem_ld32(addr + 32 * k, r[k]);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < N; ++e) sv[e] = __uint_as_float(r[e >> 5][e & 31]);
      if (kBias && biased) {
        const float* bp = reinterpret_cast<const float*>(s_stage + (i % C::NSTAGE) * C::STAGE_BYTES + C::K_BYTES + C::V_BYTES +
                                                         C::KSF_BYTES + C::VSF_BYTES) + half * 64 + c;
#pragma unroll
        for (int e = 0; e < N; e += 4) {
          const float4 b4 = *reinterpret_cast<const float4*>(bp + e);
          sv[e] += b4.x; sv[e + 1] += b4.y; sv[e + 2] += b4.z; sv[e + 3] += b4.w;
        }
      }
      if (edge) {
#pragma unroll
        for (int k = 0; k < N / 32; ++k) {
          const int off = i * 128 + c + 32 * k, lim = lim0 - off;         // last visible of these 32 columns
          // With a bias a compare and a select per score are faster at D = 128 than the bits: Z2 H32 Sq1029 Skv2309 111.3
          // us (113.3), causal Z1 H32 S4096 173.7 (176.1), Z2 H8 S3000 99.5 (101.1); equal at D = 256.
          if constexpr (kBias && !kVarlen) {
#pragma unroll
            for (int e = 0; e < 32; ++e) sv[32 * k + e] = (e <= lim) ? sv[32 * k + e] : -INFINITY;
          } else {
            uint32_t vis = lim < 0 ? 0u : 0xFFFFFFFFu >> (31 - min(lim, 31));
            if (kVarlen) {
              const int beg = beg0 - off;
              vis = beg > 31 ? 0u : vis & (0xFFFFFFFFu << max(beg, 0));
            }
#pragma unroll
            for (int e = 0; e < 32; ++e) sv[32 * k + e] = (vis >> e) & 1u ? sv[32 * k + e] : -INFINITY;
          }
        }
      }
    };
    auto free_scores = [&]() {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_free[grp]);
    };

    for (int i = grp; i < ntile; i += 2) {
      const int slot = i % kFwdMaxSlots;
      mbar_wait(&s_full[grp], (i >> 1) & 1, &err, 9);
      tc_fence_after();
      const bool edge = i >= i_mask || (kVarlen && i < i_first);
      const bool biased = kBias && s_biased[i % C::NSTAGE] != 0;
      // ---- maxima of the four 16-key groups and of the 64 columns; the latter goes to the exchange
      float gm[4];
      float sv1[C::kOneRead ? 64 : 32];
      auto group_max = [&](int g, const float* v16) {
        float v = fmax3(v16[0], v16[1], v16[2]);
#pragma unroll
        for (int e = 3; e < 15; e += 2) v = fmax3(v, v16[e], v16[e + 1]);
        gm[g] = fmaxf(v, v16[15]);
      };
      if constexpr (C::kOneRead) {
        load_scores(i, 0, edge, biased, sv1);
        free_scores();
#pragma unroll
        for (int g = 0; g < 4; ++g) group_max(g, sv1 + 16 * g);
      } else {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          load_scores(i, 32 * c, edge, biased, sv1);
          group_max(2 * c, sv1);
          group_max(2 * c + 1, sv1 + 16);
        }
      }
      const float mx = fmaxf(fmax3(gm[0], gm[1], gm[2]), gm[3]) * c2;      // c2 > 0: the scaled maximum
      sts_f32(xmax_s + (uint32_t)(slot * 2 + half) * 512u, mx);
      __syncwarp();
      if (lane == 0) mbar_arrive(&mx_ready[slot][wq]);
      // ---- the exact running maximum: own group's last tile, the tile in between, this tile's other half
      float m_prev = m_own;
      if (i > 0) {
        const int ps = (i - 1) % kFwdMaxSlots;
        mbar_wait(&mx_ready[ps][wq], ((i - 1) / kFwdMaxSlots) & 1, &err, 13);
        m_prev = fmax3(m_prev, lds_f32(xmax_s + (uint32_t)(ps * 2) * 512u), lds_f32(xmax_s + (uint32_t)(ps * 2 + 1) * 512u));
      }
      named_bar_sync(1 + grp * 4 + wq, 64);
      const float m_new = fmax3(m_prev, mx, lds_f32(xmax_s + (uint32_t)(slot * 2 + (half ^ 1)) * 512u));
      const float m_sf = (m_new == -INFINITY) ? 0.0f : m_new;
      uint32_t scw = 0u;
      float inv_g[4];
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const float a = ex2_approx(fmaf(gm[g], c2, -m_sf));
        const float s32 = fminf(fmaxf(a * 0.16666667f, kScaleFloor), kScaleMax);
        uint16_t sb16;
        asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(sb16) : "f"(0.0f), "f"(s32));
        const uint32_t sb = sb16 & 0xFFu;
        inv_g[g] = lds_f32(inv_s + sb * 4u);
        scw |= sb << (8 * g);
      }
      // P buffer of this group must have been consumed by the PV of tile i - 2
      if (i >= 2) mbar_wait(&pv_done[grp], ((i >> 1) & 1) ^ 1, &err, 10);
      float2 ls0 = make_float2(0.0f, 0.0f), ls1 = ls0;
      const float2 c22 = make_float2(c2, c2), nm2 = make_float2(-m_sf, -m_sf);
#pragma unroll
      for (int g2 = 0; g2 < 2; ++g2) {
        if constexpr (!C::kOneRead) {
          load_scores(i, 32 * g2, edge, biased, sv1);
          if (g2 == 1) free_scores();
        }
        const float* sv = sv1 + (C::kOneRead ? 32 * g2 : 0);
        uint32_t w[4];
#pragma unroll
        for (int h2 = 0; h2 < 2; ++h2) {
          const int g = g2 * 2 + h2;
          const float2 inv2 = make_float2(inv_g[g], inv_g[g]);
          float2 y[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float2 t2 = __ffma2_rn(make_float2(sv[h2 * 16 + 2 * e], sv[h2 * 16 + 2 * e + 1]), c22, nm2);
            const float2 pe = make_float2(ex2_approx(t2.x), ex2_approx(t2.y));
            if (e & 1) ls1 = __fadd2_rn(ls1, pe);
            else ls0 = __fadd2_rn(ls0, pe);
            y[e] = __fmul2_rn(pe, inv2);
          }
          w[2 * h2] = e2m1x8(y[0].x, y[0].y, y[1].x, y[1].y, y[2].x, y[2].y, y[3].x, y[3].y);
          w[2 * h2 + 1] = e2m1x8(y[4].x, y[4].y, y[5].x, y[5].y, y[6].x, y[6].y, y[7].x, y[7].y);
        }
        fwd_sts_v4(pt ^ (16u * g2), w[0], w[1], w[2], w[3]);
      }
      ls0 = __fadd2_rn(ls0, ls1);
      sts_b32(psf, scw);
      const float alpha = ex2_approx(m_prev - m_sf);
      const bool changed = (m_new > m_prev) && (i > 0);
      l_run = fmaf(l_run, ex2_approx(m_own - m_sf), ls0.x + ls0.y);
      m_own = m_new;
      if (__any_sync(0xffffffffu, changed)) {
        // O is rescaled (this thread: half of its row) once the PV of tile i - 1 has landed
        mbar_wait(&pv_done[grp ^ 1], ((i - 1) >> 1) & 1, &err, 11);
        tc_fence_after();
        const float a = changed ? alpha : 1.0f;
        const float2 a2 = make_float2(a, a);
#pragma unroll
        for (int c = 0; c < RC / 32; ++c) {
          uint32_t r[32];
          tmem_ld32(tmem + lane_addr + C::T_O + half * RC + c * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            const float2 v = __fmul2_rn(make_float2(__uint_as_float(r[e]), __uint_as_float(r[e + 1])), a2);
            r[e] = __float_as_uint(v.x);
            r[e + 1] = __float_as_uint(v.y);
          }
          tmem_st32(tmem + lane_addr + C::T_O + half * RC + c * 32, r);
        }
        tmem_st_wait();
        tc_fence_before();
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[grp]);
    }

    // ---- epilogue: bring the four partial row sums to the final maximum, O / l -> out, LSE
    xl[part][row_in] = l_run;
    if (half == 0) xm[grp][row_in] = m_own;
    named_bar_sync(9, 512);
    const float ma = xm[0][row_in], mb = xm[1][row_in];
    const float m_fin = fmaxf(ma, mb);
    {
      const float m_sf = (m_fin == -INFINITY) ? 0.0f : m_fin;
      l_run = (xl[0][row_in] + xl[1][row_in]) * ex2_approx(ma - m_sf) + (xl[2][row_in] + xl[3][row_in]) * ex2_approx(mb - m_sf);
    }
    TO* orow = nullptr;
    if (row < p.s_q)
      orow = static_cast<TO*>(p.out) + (int64_t)zi * p.so_z + (int64_t)hi * p.so_h +
             (int64_t)row * p.so_s + part * OC;
    if (ntile > 0) {
      const int last = ntile - 1;
      mbar_wait(&pv_done[last & 1], (last >> 1) & 1, &err, 12);
      tc_fence_after();
      float inv_l;
      asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv_l) : "f"((l_run == 0.0f) ? 1.0f : l_run));
#pragma unroll
      for (int c = 0; c < OC / 32; ++c) {
        uint32_t r[32];
        tmem_ld32(tmem + lane_addr + C::T_O + part * OC + c * 32, r);
        tmem_ld_wait();
        if (orow != nullptr) {
          if constexpr (sizeof(TO) == 2) {
            uint32_t w[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              const TO a0 = from_f32<TO>(__uint_as_float(r[2 * e]) * inv_l);
              const TO a1 = from_f32<TO>(__uint_as_float(r[2 * e + 1]) * inv_l);
              w[e] = (uint32_t)(*reinterpret_cast<const uint16_t*>(&a0)) |
                     ((uint32_t)(*reinterpret_cast<const uint16_t*>(&a1)) << 16);
            }
            uint4* dst = reinterpret_cast<uint4*>(orow + c * 32);
#pragma unroll
            for (int e = 0; e < 4; ++e) dst[e] = make_uint4(w[4 * e], w[4 * e + 1], w[4 * e + 2], w[4 * e + 3]);
          } else {
            float4* dst = reinterpret_cast<float4*>(orow + c * 32);
#pragma unroll
            for (int e = 0; e < 8; ++e)
              dst[e] = make_float4(__uint_as_float(r[4 * e]) * inv_l, __uint_as_float(r[4 * e + 1]) * inv_l,
                                   __uint_as_float(r[4 * e + 2]) * inv_l, __uint_as_float(r[4 * e + 3]) * inv_l);
          }
        }
      }
      tc_fence_before();
    } else if (orow != nullptr) {
      for (int e = 0; e < OC; ++e) orow[e] = from_f32<TO>(0.0f);
    }
    if (p.lse != nullptr && row < p.s_q && part == 0) {
      const float l_safe = (l_run == 0.0f) ? 1.0f : l_run;
      const float m_f = (m_fin == -INFINITY) ? 0.0f : m_fin;
      p.lse[(int64_t)zh * p.s_q + row] = m_f * 0.6931471805599453f + logf(l_safe);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && err != 0 && p.status != nullptr) atomicExch(p.status, err);
  if (warp == 1) tmem_dealloc(tmem, 512);
}

template <int D, typename TO>
int fwd_launch(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
               const FwdParams& p, int64_t zh, cudaStream_t st) {
  using C = FwdCfg<D>;
  auto kern = p.seq_id != nullptr ? (p.bias != nullptr ? fwd_kernel<D, TO, true, true> : fwd_kernel<D, TO, true, false>)
                                  : (p.bias != nullptr ? fwd_kernel<D, TO, false, true> : fwd_kernel<D, TO, false, false>);
  if (int rc = allow_smem("nvfp4_fwd", reinterpret_cast<const void*>(kern), C::SMEM_BYTES)) return rc;
  dim3 grid((unsigned)zh, (unsigned)((p.s_q + 127) / 128));
  return launch("nvfp4_fwd", kern, grid, kFwdThreads, C::SMEM_BYTES, st, tq, tk, tv, p);
}

}  // namespace nvfp4

extern "C" int nvfp4_fwd(const uint8_t* qnv, const uint8_t* qsc, const uint8_t* knv,
                         const uint8_t* ksc, const uint8_t* vnv, const uint8_t* vsc,
                         const float* bias, const int32_t* seq_id, const int32_t* seq_start,
                         void* out, int out_dtype, int64_t so_z, int64_t so_h, int64_t so_s,
                         float* lse, int64_t z, int64_t h, int64_t hk, int64_t s_q, int64_t s_kv,
                         int64_t s_pad, int d, float scaling, int flags, int* status,
                         nvfp4_stream_t stream) {
  using namespace nvfp4;
  NVFP4_REQUIRE(d == 128 || d == 256, "nvfp4_fwd: D must be 128 or 256");
  NVFP4_REQUIRE(z >= 1 && h >= 1 && hk >= 1 && h % hk == 0, "nvfp4_fwd: bad head counts");
  NVFP4_REQUIRE(s_q >= 1 && s_kv >= 1, "nvfp4_fwd: empty sequence");
  NVFP4_REQUIRE(s_pad % 128 == 0 && s_pad >= s_kv, "nvfp4_fwd: s_pad must be a multiple of 128 >= s_kv");
  NVFP4_REQUIRE(qnv && qsc && knv && ksc && vnv && vsc && out, "nvfp4_fwd: null pointer");
  NVFP4_REQUIRE((seq_id == nullptr) == (seq_start == nullptr), "nvfp4_fwd: seq_id/seq_start go together");
  NVFP4_REQUIRE(seq_id == nullptr || (z == 1 && s_q == s_kv), "nvfp4_fwd: varlen needs Z == 1 and Sq == Skv");
  NVFP4_REQUIRE((s_q + 127) / 128 < 65536, "nvfp4_fwd: too many query tiles");
  NVFP4_REQUIRE(s_q < (1LL << 30) && s_kv < (1LL << 30), "nvfp4_fwd: sequence too long");
  const size_t esz = out_dtype == NVFP4_DT_FP32 ? 4 : 2;
  NVFP4_REQUIRE(((uintptr_t)out % 16) == 0 && (so_z * esz) % 16 == 0 && (so_h * esz) % 16 == 0 &&
                    (so_s * esz) % 16 == 0,
                "nvfp4_fwd: out must be 16-byte aligned with 16-byte-multiple strides");
  NVFP4_REQUIRE(((uintptr_t)qsc % 4) == 0 && ((uintptr_t)ksc % 4) == 0 && ((uintptr_t)vsc % 8) == 0,
                "nvfp4_fwd: scale tensors must be aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t zh = z * h, zhk = z * hk;
  CUtensorMap tq, tk, tv;
  int rc = make_tmap_u8_3d_sw64(&tq, qnv, d / 2, s_q, zh, d / 2, (uint64_t)s_q * (d / 2), 128, "nvfp4_fwd(Q)");
  if (rc) return rc;
  rc = make_tmap_u8_3d_sw64(&tk, knv, d / 2, s_kv, zhk, d / 2, (uint64_t)s_kv * (d / 2), 128, "nvfp4_fwd(K)");
  if (rc) return rc;
  rc = make_tmap_u8_3d_sw64(&tv, vnv, s_pad / 2, d, zhk, s_pad / 2, (uint64_t)d * (s_pad / 2), 128, "nvfp4_fwd(V)");
  if (rc) return rc;
  FwdParams p;
  p.qsc = qsc; p.ksc = ksc; p.vsc = vsc; p.bias = bias; p.seq_id = seq_id; p.seq_start = seq_start;
  p.out = out; p.so_z = so_z; p.so_h = so_h; p.so_s = so_s; p.lse = lse;
  p.h = (int)h; p.hk = (int)hk; p.g = (int)(h / hk);
  p.s_q = (int)s_q; p.s_kv = (int)s_kv; p.s_pad = (int)s_pad;
  p.scaling = scaling; p.causal = (flags & NVFP4_FWD_CAUSAL) ? 1 : 0; p.status = status;
#define NVFP4_FWD(DD, T) return fwd_launch<DD, T>(tq, tk, tv, p, zh, st)
  if (d == 128) {
    switch (out_dtype) {
      case NVFP4_DT_BF16: NVFP4_FWD(128, __nv_bfloat16);
      case NVFP4_DT_FP16: NVFP4_FWD(128, __half);
      case NVFP4_DT_FP32: NVFP4_FWD(128, float);
    }
  } else {
    switch (out_dtype) {
      case NVFP4_DT_BF16: NVFP4_FWD(256, __nv_bfloat16);
      case NVFP4_DT_FP16: NVFP4_FWD(256, __half);
      case NVFP4_DT_FP32: NVFP4_FWD(256, float);
    }
  }
#undef NVFP4_FWD
  return fail(-1, "nvfp4_fwd: unknown out dtype %d", out_dtype);
}

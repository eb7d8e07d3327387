// NVFP4 flash-attention forward for sm_100a.
//
// An item is a 128-row query tile of one (batch, head); a CTA walks its 128-key tiles:
//     S[128 x 128]  = Q_tile . K_tile^T        tcgen05.mma kind::mxf4nvf4, e4m3 scale per 16
//     P             = exp(S*scale - m) packed to NVFP4 per 16 keys (same scale rule as the packer)
//     O[128 x D]   += P . V_tile               same MMA kind, V held as V^T (packed along keys)
// Q/K/V^T nibble tiles arrive by TMA straight from the packed tensors; scale bytes are re-laid
// into the 32x16-byte form tcgen05.cp expects by a loader warp; S and O live in TMEM.  The running
// maximum is exact (O is rescaled in TMEM whenever a row's maximum moves), which keeps the P
// quantisation decisions those of a plain 128-key tile walk.
//
// Warps (640 threads): 0 items and TMA producer, 1 QK^T issuer, 2 PV issuer, 3 scale loader (+bias), 4-19 softmax /
// correction / epilogue in two groups of eight that alternate key tiles.
// Within a group two threads share a query row, 64 key columns each, so the per-16-key P pack needs
// no cross-thread traffic.  Every barrier wait is bounded.
//
// Items.  The grid has a CTA per item, but a CTA that is through takes over one that has not been launched
// (clusterlaunchcontrol), so its start -- launch, barriers, tensor memory, code fetched anew -- is paid once per SM.
// Tiles are counted through all items of a CTA: rings, parities and the turns of the groups run on.  The group that
// has no part in an item's last tile is at the next item's first while the other merges the row sums and brings out O
// through a staging tile and TMA (32 rows x 128 bytes a warp; stores of 16 bytes a row took 3500 clocks).  An item
// costs ~3000 clocks besides its tiles where a CTA cost ~11000 (of 1750 a tile).  The next item is asked for only
// when the loads of this one are out: asked for at its start, S2048 H16 D256 takes 36.5 instead of 28.5 us.
//
// What bounds it: the floor is one ex2 per score (16 lanes per clock and SM, 1024 clocks per tile at
// D = 128); a softmax warp's tile is a chain -- wait, read, maxima, exchange, exponentials and pack,
// rescale of O -- that is about three times its share of that, and two groups hide half of it.  What the
// layout does about the chain: the running maximum is not handed from tile to tile; every thread
// publishes the maximum of its 64 columns and forms the exact running maximum itself from its group's
// last one, the two of the tile in between (read while its scores are on their way) and the other half's (one 64-thread
// barrier with the warp that holds it); a wait that usually finds its phase complete still costs 150 clocks, so the
// one for the P buffer stands behind the first exponentials; at D = 128 the 32 columns read last for the
// maxima are the first to be exponentiated, without another read; reciprocal scales come from a table in
// shared memory, not from the pipe that ex2 needs; P leaves in 16-byte stores.
// Measured on a B200, kernel alone, causal bf16, against one CTA per query tile and, the last figure, with uniform registers
// for addresses, six stages and whole scale rows: Z4 H32 Hk8 S8192 D128 2033 -> 1693 -> 1579 us (1.39 PFLOP/s), Z1 S2048
// 51.6 -> 37.7 -> 34.5; H16 Hk4 D256 S8192 334 -> 296 -> 269, S2048 33.2 -> 28.4 -> 26.2.
// Masks: only tiles at an edge of what a row may see -- diagonal, ragged end, ends of a packed sample -- and
// tiles whose bias has a value other than zero (added already divided by the scaling) are edited, in tensor memory
// before the maxima are taken, by bits of a 32-column word formed from the row's range; the loop over the others holds
// no mask code; keys at the end that the bias hides have no tiles.  Z2 H32 Sq1029 Skv2309 padded 111 -> 78 us.
// A bias that is non-zero in every tile edits them all: Z1 H32 S4096 not causal 235 -> 310 us at D = 128, 322 -> 374 at 256
// (added on the two reads of S instead, one CTA per query tile: 356 and 422).
// Registers decide here (96 per thread at twenty warps): variants that spilled even a few hundred
// bytes took up to three times as long; O is rescaled 32 columns at a time (64: prefill Z4 S8192 1883 -> 2049 us).
#include "common/abi.cuh"
#include "common/fp4.cuh"
#include "common/launch.cuh"
#include "common/sm100.cuh"
#include "common/tma_host.cuh"

namespace nvfp4 {

constexpr int kFwdRoleWarps = 4;
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
  // six instead of four stages: Z4 H32 S8192 D128 1609 -> 1586 us, S2048 34.8 -> 34.3 (five: 1600, 34.5); D = 256 has no room
  static constexpr int NSTAGE = (D == 128) ? 6 : 3;
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
  static constexpr int SMEM_BYTES = NSTAGE * STAGE_BYTES + 2 * (Q_BYTES + QSF_BYTES + P_BYTES + PSF_BYTES) + 32768 + 1024;
  static_assert(2 * (PSF_BYTES + QSF_BYTES) % 1024 == 0, "staging tiles are swizzled");
  // TMEM columns
  static constexpr int T_S = 0;                       // NSBUF x 128
  static constexpr int T_O = NSBUF * 128;             // D
  static constexpr int T_SFQ = T_O + D;               // 2 x KB * 4
  static constexpr int T_SFK = T_SFQ + 2 * KB * 4;    // 2 x KB * 4
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
  int tma_out;         // tm_o describes out
  int vec_sc;          // scale rows of Q and K are aligned to their size
  int* status;
};

struct __align__(16) FwdItem {   // one query tile of one head; tiles count from the CTA's first one on
  int r0, r1;                    // its key tiles [r0, r1); r1 = -1: no more items
  int r_first, r_mask;           // tiles whose scores are all visible: [r_first, r_mask)
  int zi, hi, m0;
  int t0;                        // key tile of running tile 0 (may be negative)
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
           const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o, const FwdParams p) {
  using C = FwdCfg<D>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* s_stage = smem;
  uint8_t* s_q = s_stage + C::NSTAGE * C::STAGE_BYTES;      // two items
  uint8_t* s_p = s_q + 2 * C::Q_BYTES;
  uint8_t* s_psf = s_p + 2 * C::P_BYTES;
  uint8_t* s_qsf = s_psf + 2 * C::PSF_BYTES;                // two items
  uint8_t* s_out = s_qsf + 2 * C::QSF_BYTES;                // per warp of a group 32 rows x 128 bytes

  __shared__ uint64_t full[C::NSTAGE], empty[C::NSTAGE];
  __shared__ uint64_t s_full[2], s_free[2], p_full[2], pv_done[2], q_full[2], qsf_full[2], part_done[2], o_free;
  __shared__ uint64_t item_full[2], item_free[2], clc_full;
  __shared__ uint64_t mx_ready[kFwdMaxSlots][4];     // row maxima of a tile, one barrier per 32-row quadrant
  __shared__ __align__(16) uint4 clc_resp;
  __shared__ uint32_t tmem_base_s;
  __shared__ int err;
  __shared__ FwdItem s_item[2];
  __shared__ int2 s_rows[kVarlen ? 2 : 1][kVarlen ? 128 : 1];   // [item][row] first and last visible key
  __shared__ int s_biased[C::NSTAGE];                // the tile's bias has a value other than zero
  __shared__ float xmax[kFwdMaxSlots][2][128];       // [tile % slots][key half][row]
  __shared__ float xl[2][2][2][128];                 // row sums [item][late group][key half][row]
  __shared__ float xm[2][128];                       // running maximum of the other group
  __shared__ float inv_tab[128];                     // reciprocal of every (non-negative) e4m3 byte

  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int shift = p.s_kv - p.s_q;  // bottom-right aligned causal offset

  if (warp == 0) {
    mbar_init(&mx_ready[lane >> 2][lane & 3], 2);
    if (lane < C::NSTAGE) {
      mbar_init(&full[lane], 2);        // TMA producer (and its bytes), scale loader
      mbar_init(&empty[lane], 1);
    }
    if (lane < 2) {
      mbar_init(&s_full[lane], 1);
      mbar_init(&s_free[lane], 8);
      mbar_init(&p_full[lane], 8);
      mbar_init(&pv_done[lane], 1);
      mbar_init(&q_full[lane], 1);
      mbar_init(&qsf_full[lane], 1);
      mbar_init(&part_done[lane], 8);
      mbar_init(&item_full[lane], 1);
      mbar_init(&item_free[lane], 19);
    }
    if (lane == 0) {
      err = 0;
      mbar_init(&o_free, 8);
      mbar_init(&clc_full, 1);
    }
    mbar_fence_init();
    if (lane == 0) tma_prefetch_map(&tm_q);
    if (lane == 1) tma_prefetch_map(&tm_k);
    if (lane == 2) tma_prefetch_map(&tm_v);
  }
  if (tid >= 128 && tid < 256) {
    float inv;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(e4m3_to_f32((uint8_t)(tid - 128))));
    inv_tab[tid - 128] = inv;
  }
  if (warp == 1) tmem_alloc(&tmem_base_s, 512);
  // (warp 0) the query tile of the CTA with block index (bx, by, bz), as item `sl` whose tiles count from r0
  auto decode = [&](int bx, int by, int bz, int r0, int sl) {
    // grid = (heads, batch, query tiles): all heads of the heaviest (last) query tile are scheduled first,
    // so the kernel ends on the cheapest tiles instead of on a long straggler
    const int m0 = ((int)gridDim.z - 1 - bz) * 128;
    int hi = bx, zi = by;
    if (hi >= p.h) {              // a batch beyond the grid's limit lies along x
      zi = hi / p.h;
      hi -= zi * p.h;
    }
    // Key tiles of the item.  Varlen: the visible keys of a row are its sample, cut at the row itself when causal;
    // ids are sorted, so the first row has the earliest start.
    int hi_key = p.causal ? min(p.s_kv, m0 + 128 + shift) : p.s_kv;
    if (hi_key < 0) hi_key = 0;
    int t_lo = 0, i_first = 0;
    int last_full = min(p.causal ? m0 + shift + 1 : p.s_kv, p.s_kv);     // keys below are visible to every row
    if (kVarlen) {
      int beg[4], end[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) beg[j] = p.seq_start[min(m0 + lane + 32 * j, p.s_q - 1)];
      if (p.causal) {
#pragma unroll
        for (int j = 0; j < 4; ++j) end[j] = m0 + lane + 32 * j + shift + 1;
      } else {          // first key behind the sample of the row
        int id[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) id[j] = p.seq_id[min(m0 + lane + 32 * j, p.s_q - 1)];
        // Behind the tile the last row's sample goes on up to a key in [lo, hi]: the last of 32 equal parts each round, three
        // trips to memory at 16384 tokens where a bisection by every row took fifteen: H16 Hk4 one sample of 1024 tokens D256
        // 19.5 -> 17.9 us, eight in 16384 D128 260 -> 231.
        const int id_last = __shfl_sync(0xffffffffu, id[3], 31);
        int lo = min(m0 + 128, p.s_q), hi = p.s_kv;
        while (lo < hi) {
          const int step = (hi - lo + 31) / 32, probe = lo + step * (lane + 1) - 1;
          const bool same = probe < hi && p.seq_id[min(probe, p.s_kv - 1)] == id_last;
          lo += step * __popc(__ballot_sync(0xffffffffu, same));
          hi = min(hi, lo + step - 1);
        }
        // inside the tile it ends where the next id begins
        int next = lo;
#pragma unroll
        for (int j = 3; j >= 0; --j) {
          int before = __shfl_up_sync(0xffffffffu, id[j], 1);
          const int seam = __shfl_sync(0xffffffffu, id[j > 0 ? j - 1 : 0], 31);
          if (lane == 0) before = j > 0 ? seam : id[0];
          const uint32_t begins = __ballot_sync(0xffffffffu, id[j] != before);
          const uint32_t behind = begins & ~((2u << lane) - 1u);
          end[j] = behind != 0u ? m0 + 32 * j + __ffs(behind) - 1 : next;
          if (begins != 0u) next = m0 + 32 * j + __ffs(begins) - 1;
        }
        last_full = __shfl_sync(0xffffffffu, end[0], 0);
        hi_key = __shfl_sync(0xffffffffu, end[3], 31);      // the last row's sample ends last
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) s_rows[sl][lane + 32 * j] = make_int2(beg[j], end[j] - 1);
      t_lo = __shfl_sync(0xffffffffu, beg[0], 0) / 128;
      i_first = (__shfl_sync(0xffffffffu, beg[3], 31) + 127) / 128 - t_lo;
    }
    if (kBias) {
      // Keys at the end that the bias hides from every row, as it does in a padded batch, have no tiles: 256 at a time from
      // behind until one is visible.  Z2 H32 Sq1029 Skv2309, 11 and 22 % padded: 86.2 -> 78.0 us,
      // eight prompts of up to 300 H8 Hk2 15.3 -> 11.9.  It is a trip to L2 before the loads, which calls of two or three tiles
      // without padding do not get back: Z1 H8 Hk2 S300 9.2 -> 9.7.  Left out below 256 or 384 keys, it cost padded batches of
      // short prompts more (Z32 H16 S512 causal 47.7 -> 53.2).
      const float* b = p.bias + (int64_t)zi * p.s_kv;
      int seen = 0;                       // visible key with the highest number, plus one
      for (; hi_key > t_lo * 128; hi_key -= 256) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int key = hi_key - 1 - lane - 32 * j;
          v[j] = key >= 0 ? __ldg(b + key) : -INFINITY;
        }
#pragma unroll
        for (int j = 7; j >= 0; --j)
          if (v[j] != -INFINITY) seen = hi_key - lane - 32 * j;
        seen = __reduce_max_sync(0xffffffffu, seen);
        if (seen > 0) break;
      }
      hi_key = seen;
    }
    const int r1 = r0 + max((hi_key + 127) / 128 - t_lo, 0);
    if (lane == 0)
      s_item[sl] = FwdItem{r0, r1, r0 + i_first, r0 - t_lo + max(last_full, 0) / 128, zi, hi, m0,
                           t_lo - r0};
    __syncwarp();
  };
  constexpr bool kReads = kVarlen || kBias;         // an item's extent depends on memory: sample ids, bias
  if (!kReads && warp == 0) decode(blockIdx.x, blockIdx.y, blockIdx.z, 0, 0);
  griddep_wait();
  if (kReads && warp == 0) decode(blockIdx.x, blockIdx.y, blockIdx.z, 0, 0);
  if (tid == 0) mbar_arrive(&item_full[0]);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  griddep_launch();
  const uint32_t tmem = tmem_base_s;

  if (warp == 0) {
    // ------------------------------------------------------------------ items, TMA producer
    const bool leader = elect_one();
    for (int it = 0;; ++it) {
      const int sl = it & 1;
      const int r0 = s_item[sl].r0, r1 = s_item[sl].r1, zi = s_item[sl].zi, hi = s_item[sl].hi, m0 = s_item[sl].m0;
      const int t0 = s_item[sl].t0, unit = zi * p.hk + hi / p.g;      // unit: (batch, kv head)
      if (leader) {
        mbar_expect_tx(&q_full[sl], C::Q_BYTES);
#pragma unroll
        for (int ks = 0; ks < C::KSUB; ++ks)
          tma_load_3d(s_q + sl * C::Q_BYTES + ks * 8192, &tm_q, &q_full[sl], ks * 64, m0, zi * p.h + hi);
      }
#pragma unroll 1
      for (int r = r0; r < r1; ++r) {
        const int s = r % C::NSTAGE, t = t0 + r;
        if (r >= C::NSTAGE) mbar_wait_warp(&empty[s], ((r / C::NSTAGE) & 1) ^ 1, &err, 1);
        if (leader) {
          uint8_t* st = s_stage + s * C::STAGE_BYTES;
          mbar_expect_tx(&full[s], C::K_BYTES + C::V_BYTES);
#pragma unroll
          for (int ks = 0; ks < C::KSUB; ++ks) tma_load_3d(st + ks * 8192, &tm_k, &full[s], ks * 64, t * 128, unit);
#pragma unroll
          for (int nt = 0; nt < C::NT; ++nt)
            tma_load_3d(st + C::K_BYTES + nt * 8192, &tm_v, &full[s], t * 64, nt * 128, unit);
        }
      }
      // The next item is asked for when this one's loads are out, three or four tiles before its end: asked for at its
      // start, the items of a grid of a wave or two would be dealt before it is known who is through first.
      if (leader) clc_request(&clc_resp, &clc_full);
      __syncwarp();
      int bx, by, bz;
      bool more = mbar_wait_item_warp(&clc_full, it & 1, &err, 21) && clc_answer(&clc_resp, bx, by, bz);
      fence_proxy_async_smem();         // read before the next answer may overwrite it
      __syncwarp();
      const int next = sl ^ 1;
      if (it >= 1) more = mbar_wait_item_warp(&item_free[next], (((it + 1) >> 1) & 1) ^ 1, &err, 20) && more;
      if (more) decode(bx, by, bz, r1, next);
      else if (lane == 0) s_item[next].r1 = -1;
      __syncwarp();
      if (lane == 0) mbar_arrive(&item_full[next]);
      if (!more) break;
    }
    __syncwarp();
  } else if (warp == 3) {
    // ------------------------------------------------------------------ scale loader (+ bias)
    // Q scales of an item, K scales (+ key bias) and V^T scales of a tile, re-laid into the 32 x 16-byte
    // atoms tcgen05.cp copies.  The next tile's bytes are fetched into registers one tile
    // ahead, so per tile the warp pays a shared-memory store, not a trip to L2.
    const float inv_scaling = kBias ? 1.0f / p.scaling : 0.0f;      // the bias is added to the unscaled scores
    for (int it = 0;; ++it) {
      const int sl = it & 1;
      if (!mbar_wait_item(&item_full[sl], (it >> 1) & 1, &err, 22)) break;
      const int r0 = s_item[sl].r0, r1 = s_item[sl].r1;
      if (r1 < 0) break;
      const int zi = s_item[sl].zi, hi = s_item[sl].hi, m0 = s_item[sl].m0;
      const int key0 = (s_item[sl].t0 + r0) * 128;
      const int unit = zi * p.hk + hi / p.g;
      const uint8_t* qsrc = p.qsc + (int64_t)(zi * p.h + hi) * p.s_q * (D / 16);
      const uint8_t* ksrc = p.ksc + (int64_t)unit * p.s_kv * (D / 16);
      const uint8_t* vsrc = p.vsc + (int64_t)unit * D * (p.s_pad / 16);
      uint32_t qx[4][C::KB], kx[4][C::KB];
      float nb[4];
      uint2 vx[D / 32];
      // The D / 16 scale bytes of a row: one load where rows are aligned to them, else words.  This warp's instructions are
      // taken from the softmax warps of its scheduler, which the others wait for (a fifth longer in their exponentials): one
      // load a row and one store of four rows an atom, S8192 H16 D256 278 -> 270 us, Z4 S8192 D128 1582 -> 1576.
      auto row_scales = [&](const uint8_t* src, uint32_t (&x)[C::KB]) {
        if (!p.vec_sc) {
#pragma unroll
          for (int k = 0; k < C::KB; ++k) x[k] = __ldg(reinterpret_cast<const uint32_t*>(src) + k);
        } else if constexpr (C::KB == 2) {
          const uint2 v = __ldg(reinterpret_cast<const uint2*>(src));
          x[0] = v.x; x[1] = v.y;
        } else {
          const uint4 v = __ldg(reinterpret_cast<const uint4*>(src));
          x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
        }
      };
      // Keys behind the last one take its scales: their scores are masked.
      auto fetch = [&](int first) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int key = min(first + lane + 32 * j, p.s_kv - 1);
          row_scales(ksrc + (int64_t)key * (D / 16), kx[j]);
          if (kBias) nb[j] = first + lane + 32 * j < p.s_kv ? __ldg(p.bias + (int64_t)zi * p.s_kv + key) * inv_scaling : 0.0f;
        }
#pragma unroll
        for (int j = 0; j < D / 32; ++j)
          vx[j] = __ldg(reinterpret_cast<const uint2*>(vsrc + (int64_t)(lane + 32 * j) * (p.s_pad / 16) + (first >> 4)));
      };
#pragma unroll
      for (int j = 0; j < 4; ++j) row_scales(qsrc + (int64_t)min(m0 + lane + 32 * j, p.s_q - 1) * (D / 16), qx[j]);
      if (r1 > r0) fetch(key0);
      // rows lane, lane + 32, .. of an atom are neighbours
#pragma unroll
      for (int k = 0; k < C::KB; ++k)
        fwd_sts_v4(smem_u32(s_qsf + sl * C::QSF_BYTES + k * 512) + lane * 16, qx[0][k], qx[1][k], qx[2][k], qx[3][k]);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&qsf_full[sl]);
#pragma unroll 1
      for (int r = r0; r < r1; ++r) {
        const int s = r % C::NSTAGE;
        if (r >= C::NSTAGE) mbar_wait(&empty[s], ((r / C::NSTAGE) & 1) ^ 1, &err, 4);
        uint8_t* st = s_stage + s * C::STAGE_BYTES + C::K_BYTES + C::V_BYTES;
        const uint32_t at = smem_u32(st) + lane * 16;
#pragma unroll
        for (int k = 0; k < C::KB; ++k) fwd_sts_v4(at + k * 512, kx[0][k], kx[1][k], kx[2][k], kx[3][k]);
        if (kBias) {
#pragma unroll
          for (int j = 0; j < 4; ++j) reinterpret_cast<float*>(st + C::KSF_BYTES + C::VSF_BYTES)[lane + 32 * j] = nb[j];
        }
        if (kBias) {
          const int any = __any_sync(0xffffffffu, nb[0] != 0.0f || nb[1] != 0.0f || nb[2] != 0.0f || nb[3] != 0.0f);
          if (lane == 0) s_biased[s] = any;
        }
#pragma unroll
        for (int nt = 0; nt < C::NT; ++nt) {
          fwd_sts_v4(at + C::KSF_BYTES + nt * 512, vx[4 * nt].x, vx[4 * nt + 1].x, vx[4 * nt + 2].x, vx[4 * nt + 3].x);
          fwd_sts_v4(at + C::KSF_BYTES + (C::NT + nt) * 512, vx[4 * nt].y, vx[4 * nt + 1].y, vx[4 * nt + 2].y, vx[4 * nt + 3].y);
        }
        if (r + 1 < r1) fetch(key0 + (r + 1 - r0) * 128);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[s]);
      }
      if (lane == 0) mbar_arrive(&item_free[sl]);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ QK^T issuer
    // The whole warp waits and counts, one thread issues: in a branch of one thread the compiler can use no uniform
    // registers, and the descriptors and addresses of every product are moved there one by one: S8192 H16 D256 284 -> 278.5 us.
    const bool leader = elect_one();
    const uint32_t idesc_qk = make_idesc_nvfp4(128, 128);
    int r = 0;
    for (int it = 0;; ++it) {
      const int sl = it & 1;
      if (!mbar_wait_item_warp(&item_full[sl], (it >> 1) & 1, &err, 22)) break;
      const int r1 = __shfl_sync(0xffffffffu, s_item[sl].r1, 0);
      if (r1 < 0) break;
      mbar_wait(&q_full[sl], (it >> 1) & 1, &err, 3);
      mbar_wait_warp(&qsf_full[sl], (it >> 1) & 1, &err, 6);
      tc_fence_after();
      const uint32_t sfq = tmem + C::T_SFQ + sl * C::KB * 4;
      uint8_t* q = s_q + sl * C::Q_BYTES;
      if (leader) {
#pragma unroll
        for (int k = 0; k < C::KB; ++k)
          tmem_cp_32x128b_warpx4(sfq + k * 4, smem_u32(s_qsf + sl * C::QSF_BYTES + k * 512));
      }
#pragma unroll 1
      for (; r < r1; ++r) {
        const int s = r % C::NSTAGE, b = r % C::NSBUF;
        const uint32_t ph = (r / C::NSTAGE) & 1;
        mbar_wait(&full[s], ph, &err, 5);
        if (r >= C::NSBUF) {      // the S buffer's last tile has been read into registers
          const int u = r - C::NSBUF;
          mbar_wait(&s_free[u & 1], (u >> 1) & 1, &err, 7);
        }
        tc_fence_after();
        uint8_t* st = s_stage + s * C::STAGE_BYTES;
        const uint32_t sfk = tmem + C::T_SFK + (r & 1) * C::KB * 4;
        __syncwarp();
        if (leader) {
#pragma unroll
          for (int k = 0; k < C::KB; ++k)
            tmem_cp_32x128b_warpx4(sfk + k * 4, smem_u32(st + C::K_BYTES + C::V_BYTES + k * 512));
#pragma unroll
          for (int k = 0; k < C::KB; ++k) {
            const uint64_t ad = make_smem_desc(smem_u32(q + (k >> 1) * 8192) + (k & 1) * 32, 16, 512, 4);
            const uint64_t bd = make_smem_desc(smem_u32(st + (k >> 1) * 8192) + (k & 1) * 32, 16, 512, 4);
            umma_nvfp4(tmem + C::T_S + b * 128, ad, bd, idesc_qk, sfq + k * 4, sfk + k * 4, k > 0);
          }
          umma_commit(&s_full[r & 1]);     // by tile parity: each group waits for its own tiles
        }
        __syncwarp();
      }
      if (leader) mbar_arrive(&item_free[sl]);
    }
    __syncwarp();
  } else if (warp == 2) {
    // ------------------------------------------------------------------ PV issuer
    // A warp of its own, so a QK^T for tile i+2 is never queued behind the wait for P(i).
    const bool leader = elect_one();
    const uint32_t idesc_pv = make_idesc_nvfp4(128, D);
    int r = 0;
    uint32_t o_phase = 0u;
    for (int it = 0;; ++it) {
      const int sl = it & 1;
      if (!mbar_wait_item_warp(&item_full[sl], (it >> 1) & 1, &err, 22)) break;
      const int r1 = __shfl_sync(0xffffffffu, s_item[sl].r1, 0);
      if (r1 < 0) break;
      if (r1 > r && r > 0) {          // O of the last item that had tiles has been read
        mbar_wait(&o_free, o_phase, &err, 2);
        o_phase ^= 1u;
      }
      const int r0 = r;
#pragma unroll 1
      for (; r < r1; ++r) {
        const int s = r % C::NSTAGE, b = r & 1;
        // the V tile and V scales of stage s landed before this tile's QK^T was issued, but this
        // thread has to observe them itself; it does so while P is still being written
        mbar_wait(&full[s], (r / C::NSTAGE) & 1, &err, 15);
        tc_fence_after();
        uint8_t* st = s_stage + s * C::STAGE_BYTES;
        const uint32_t sfp = tmem + C::T_SFP + b * 8;
        const uint32_t sfv = tmem + C::T_SFV + b * (2 * C::NT * 4);
        if (leader) {
#pragma unroll
          for (int k = 0; k < 2 * C::NT; ++k)
            tmem_cp_32x128b_warpx4(sfv + k * 4,
                                   smem_u32(st + C::K_BYTES + C::V_BYTES + C::KSF_BYTES + k * 512));
        }
        mbar_wait_warp(&p_full[b], (r >> 1) & 1, &err, 8);
        tc_fence_after();
        if (leader) {
#pragma unroll
          for (int k = 0; k < 2; ++k)
            tmem_cp_32x128b_warpx4(sfp + k * 4, smem_u32(s_psf + b * C::PSF_BYTES + k * 512));
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const uint64_t ad = make_smem_desc(smem_u32(s_p + b * C::P_BYTES) + k * 32, 16, 512, 4);
            const uint64_t bd = make_smem_desc(smem_u32(st + C::K_BYTES) + k * 32, 16, 512, 4);
            umma_nvfp4(tmem + C::T_O, ad, bd, idesc_pv, sfp + k * 4, sfv + k * C::NT * 4,
                       (r > r0 || k > 0) ? 1u : 0u);
          }
          umma_commit(&pv_done[b]);
          umma_commit(&empty[s]);
        }
        __syncwarp();
      }
      if (leader) mbar_arrive(&item_free[sl]);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ softmax / correction / epilogue
    const int sw = warp - kFwdRoleWarps;
    const int grp = sw >> 3;             // which tiles (parity)
    const int wq = warp & 3;             // TMEM lane quadrant
    const int half = (sw >> 2) & 1;      // which 64 key columns
    const int row_in = wq * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(wq * 32) << 16;
    constexpr int RC = D / 2;            // O columns of a thread: rescale and end of the item
    const float c2 = p.scaling * kFwdLog2e;
    const uint32_t xmax_s = smem_u32(&xmax[0][0][0]) + (uint32_t)row_in * 4u;
    const uint32_t inv_s = smem_u32(inv_tab);
    const uint32_t pt = smem_u32(s_p + grp * C::P_BYTES) + sw64_offset(row_in, half * 32);   // the next 16 bytes: ^ 16
    const uint32_t psf = smem_u32(s_psf + grp * C::PSF_BYTES) + half * 512 + sf_atom_offset(row_in, 0);
    const uint32_t s_base = tmem + lane_addr + C::T_S + half * 64 + (C::NSBUF == 2 ? grp * 128 : 0);

    // Visible keys of this row: one range, also in packed rows, whose ids are sorted.  Positions count from this thread's
    // first column of running tile 0 (modulo 2^32).
    uint32_t lim0 = 0u, beg0 = 0u;
    auto load_scores = [&](int c, uint32_t (&x)[32]) { tmem_ld32(s_base + c, x); };
    // Bias and mask of an edge tile, in tensor memory: a read and a write of the thread's 64 columns in the few tiles
    // that need it, so that the loop over the others holds none of it.
    auto edit_scores = [&](int r, bool edge, bool biased) {
#pragma unroll 1
      for (int c = 0; c < 64; c += 32) {
        uint32_t x[32];
        tmem_ld32(s_base + c, x);
        tmem_ld_wait();
        if (kBias && biased) {
          const float* bp = reinterpret_cast<const float*>(s_stage + (r % C::NSTAGE) * C::STAGE_BYTES + C::K_BYTES + C::V_BYTES +
                                                           C::KSF_BYTES + C::VSF_BYTES) + half * 64 + c;
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            const float4 b4 = *reinterpret_cast<const float4*>(bp + e);
            x[e] = __float_as_uint(__uint_as_float(x[e]) + b4.x);
            x[e + 1] = __float_as_uint(__uint_as_float(x[e + 1]) + b4.y);
            x[e + 2] = __float_as_uint(__uint_as_float(x[e + 2]) + b4.z);
            x[e + 3] = __float_as_uint(__uint_as_float(x[e + 3]) + b4.w);
          }
        }
        if (edge) {
          const uint32_t off = (uint32_t)r * 128u + c;
          const int lim = (int)(lim0 - off);                 // last visible of these 32 columns
          uint32_t vis = lim < 0 ? 0u : 0xFFFFFFFFu >> (31 - min(lim, 31));
          if (kVarlen) {
            const int beg = (int)(beg0 - off);
            vis = beg > 31 ? 0u : vis & (0xFFFFFFFFu << max(beg, 0));
          }
#pragma unroll
          for (int e = 0; e < 32; ++e) x[e] = (vis >> e) & 1u ? x[e] : 0xFF800000u;      // -inf
        }
        tmem_st32(s_base + c, x);
      }
      tmem_st_wait();
    };
    auto free_scores = [&]() {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_free[grp]);
    };

    for (int it = 0;; ++it) {
      const int sl = it & 1;
      if (!mbar_wait_item(&item_full[sl], (it >> 1) & 1, &err, 22)) break;
      const int r0 = s_item[sl].r0, r1 = s_item[sl].r1;
      if (r1 < 0) break;
      // Tiles below r_first and from r_mask on need a test per score: the edge of a sample, the causal
      // diagonal, the ragged end.  A tile whose bias is all zero (the valid part of a padded batch) does not.
      {
        const uint32_t rel = (uint32_t)s_item[sl].t0 * 128u + (uint32_t)half * 64u;
        const int last = kVarlen ? s_rows[sl][row_in].y : (p.causal ? s_item[sl].m0 + row_in + shift : p.s_kv - 1);
        lim0 = (uint32_t)min(last, p.s_kv - 1) - rel;
        if (kVarlen) beg0 = (uint32_t)s_rows[sl][row_in].x - rel;
      }
      float m_own = -INFINITY, l_run = 0.0f;   // running max (log2 units) after this group's last tile
#pragma unroll 1
      for (int r = r0 + ((r0 ^ grp) & 1); r < r1; r += 2) {
        const int slot = r % kFwdMaxSlots;
        mbar_wait(&s_full[grp], (r >> 1) & 1, &err, 17);
        tc_fence_after();
        const bool edge = r >= s_item[sl].r_mask || (kVarlen && r < s_item[sl].r_first);
        const bool biased = kBias && s_biased[r % C::NSTAGE] != 0;
        if (edge || biased) edit_scores(r, edge, biased);
        // ---- maxima of the four 16-key groups and of the 64 columns; the latter goes to the exchange
        float gm[4];
        uint32_t sv[C::kOneRead ? 2 : 1][32];      // scores; D = 128: of the 32 columns at hand
        auto group_max = [&](int g, const uint32_t* x) {
          float v = fmax3(__uint_as_float(x[0]), __uint_as_float(x[1]), __uint_as_float(x[2]));
#pragma unroll
          for (int e = 3; e < 15; e += 2) v = fmax3(v, __uint_as_float(x[e]), __uint_as_float(x[e + 1]));
          gm[g] = fmaxf(v, __uint_as_float(x[15]));
        };
        load_scores(0, sv[0]);
        if constexpr (C::kOneRead) load_scores(32, sv[1]);
        // while they are on their way: maxima of the tile in between, which the other group left half a tile ago
        float m_prev = m_own;
        if (r > r0) {
          const int ps = (r - 1) % kFwdMaxSlots;
          mbar_wait(&mx_ready[ps][wq], ((r - 1) / kFwdMaxSlots) & 1, &err, 13);
          m_prev = fmax3(m_prev, lds_f32(xmax_s + (uint32_t)(ps * 2) * 512u), lds_f32(xmax_s + (uint32_t)(ps * 2 + 1) * 512u));
        }
        tmem_ld_wait();
        if constexpr (C::kOneRead) {
          free_scores();
#pragma unroll
          for (int g = 0; g < 4; ++g) group_max(g, sv[g >> 1] + 16 * (g & 1));
        } else {
          group_max(0, sv[0]);
          group_max(1, sv[0] + 16);
          load_scores(32, sv[0]);
          tmem_ld_wait();
          group_max(2, sv[0]);
          group_max(3, sv[0] + 16);
        }
        const float mx = fmaxf(fmax3(gm[0], gm[1], gm[2]), gm[3]) * c2;      // c2 > 0: the scaled maximum
        sts_f32(xmax_s + (uint32_t)(slot * 2 + half) * 512u, mx);
        __syncwarp();
        if (lane == 0) mbar_arrive(&mx_ready[slot][wq]);
        // ---- the exact running maximum: own group's last tile, the tile in between, this tile's other half
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
        float2 ls0 = make_float2(0.0f, 0.0f), ls1 = ls0;
        const float2 c22 = make_float2(c2, c2), nm2 = make_float2(-m_sf, -m_sf);
#pragma unroll
        for (int k2 = 0; k2 < 2; ++k2) {
          const int g2 = C::kOneRead ? k2 : k2 ^ 1;           // the columns that the maxima were read from last are still here
          if constexpr (!C::kOneRead) {
            if (k2 == 1) {
              load_scores(32 * g2, sv[0]);
              tmem_ld_wait();
              free_scores();
            }
          }
          const uint32_t* x = sv[C::kOneRead ? g2 : 0];
          uint32_t w[4];
#pragma unroll
          for (int h2 = 0; h2 < 2; ++h2) {
            const int g = g2 * 2 + h2;
            const float2 inv2 = make_float2(inv_g[g], inv_g[g]);
            float2 y[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const float2 t2 = __ffma2_rn(make_float2(__uint_as_float(x[h2 * 16 + 2 * e]), __uint_as_float(x[h2 * 16 + 2 * e + 1])), c22, nm2);
              const float2 pe = make_float2(ex2_approx(t2.x), ex2_approx(t2.y));
              if (e & 1) ls1 = __fadd2_rn(ls1, pe);
              else ls0 = __fadd2_rn(ls0, pe);
              y[e] = __fmul2_rn(pe, inv2);
            }
            w[2 * h2] = e2m1x8(y[0].x, y[0].y, y[1].x, y[1].y, y[2].x, y[2].y, y[3].x, y[3].y);
            w[2 * h2 + 1] = e2m1x8(y[4].x, y[4].y, y[5].x, y[5].y, y[6].x, y[6].y, y[7].x, y[7].y);
          }
          // the P buffer of this group has been consumed by the PV of tile r - 2
          if (k2 == 0 && r >= 2) mbar_wait(&pv_done[grp], ((r >> 1) & 1) ^ 1, &err, 10);
          fwd_sts_v4(pt ^ (16u * g2), w[0], w[1], w[2], w[3]);
        }
        ls0 = __fadd2_rn(ls0, ls1);
        sts_b32(psf, scw);
        const float alpha = ex2_approx(m_prev - m_sf);
        const bool changed = (m_new > m_prev) && (r > r0);
        l_run = fmaf(l_run, ex2_approx(m_own - m_sf), ls0.x + ls0.y);
        m_own = m_new;
        if (__any_sync(0xffffffffu, changed)) {
          // O is rescaled (this thread: half of its row) once the PV of tile r - 1 has landed
          mbar_wait(&pv_done[grp ^ 1], ((r - 1) >> 1) & 1, &err, 11);
          tc_fence_after();
          const float a = changed ? alpha : 1.0f;
          const float2 a2 = make_float2(a, a);
#pragma unroll
          for (int c = 0; c < RC / 32; ++c) {
            uint32_t o[32];
            tmem_ld32(tmem + lane_addr + C::T_O + half * RC + c * 32, o);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; e += 2) {
              const float2 v = __fmul2_rn(make_float2(__uint_as_float(o[e]), __uint_as_float(o[e + 1])), a2);
              o[e] = __float_as_uint(v.x);
              o[e + 1] = __float_as_uint(v.y);
            }
            tmem_st32(tmem + lane_addr + C::T_O + half * RC + c * 32, o);
          }
          tmem_st_wait();
          tc_fence_before();
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[grp]);
      }
      // ---- end of the item.  The group without the last tile leaves its row sums and goes on to the next item; the
      // other one merges them (its running maximum is the final one), O / l -> out, LSE.
      const bool late = grp == (r1 > r0 ? (r1 - 1) & 1 : 0);
      xl[sl][late][half][row_in] = l_run;
      if (!late) {
        if (half == 0) xm[sl][row_in] = m_own;
        if (lane == 0) bulk_wait_read<0>();      // this group's stores have left the staging tiles
        __syncwarp();
        if (lane == 0) mbar_arrive(&part_done[sl]);
      } else {
        named_bar_sync(1 + grp * 4 + wq, 64);
        mbar_wait(&part_done[sl], (it >> 1) & 1, &err, 14);
        const float m_fin = (m_own == -INFINITY) ? 0.0f : m_own;
        l_run = fmaf(xl[sl][0][0][row_in] + xl[sl][0][1][row_in], ex2_approx(xm[sl][row_in] - m_fin),
                     xl[sl][1][0][row_in] + xl[sl][1][1][row_in]);
        const int m0 = s_item[sl].m0, zi = s_item[sl].zi, hi = s_item[sl].hi;
        if (r1 > r0) {
          mbar_wait(&pv_done[grp], ((r1 - 1) >> 1) & 1, &err, 12);
          tc_fence_after();
        }
        float inv_l;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv_l) : "f"((l_run == 0.0f) ? 1.0f : l_run));
        // A warp's 32 rows leave 128 bytes a row at a time, staged and stored as one box.  Not unrolled: code that runs
        // once per item is fetched each time.
        constexpr int CC = 128 / sizeof(TO);
        uint8_t* stg = s_out + (half * 4 + wq) * 4096;
        uint32_t ln;                             // lane, opaque: addresses of the staging tile are not kept over the loop
        asm volatile("mov.u32 %0, %%laneid;" : "=r"(ln));
#pragma unroll 1
        for (int c = 0; c < RC; c += CC) {
          if (p.tma_out && lane == 0) bulk_wait_read<0>();
          __syncwarp();
#pragma unroll
          for (int k = 0; k < CC / 32; ++k) {
            constexpr int W = 8 * sizeof(TO);    // words of 32 columns
            uint32_t o[32];
            if (r1 > r0) {
              tmem_ld32(tmem + lane_addr + C::T_O + half * RC + c + 32 * k, o);
              tmem_ld_wait();
            } else {
#pragma unroll
              for (int e = 0; e < 32; ++e) o[e] = 0u;
            }
            if constexpr (sizeof(TO) == 2) {
#pragma unroll
              for (int e = 0; e < 16; ++e) {
                const float2 v = __fmul2_rn(make_float2(__uint_as_float(o[2 * e]), __uint_as_float(o[2 * e + 1])),
                                            make_float2(inv_l, inv_l));
                o[e] = pack_16x2<TO>(v.x, v.y);
              }
            } else {
#pragma unroll
              for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * inv_l);
            }
            if (p.tma_out) {
#pragma unroll
              for (int e = 0; e < W; e += 4)
                fwd_sts_v4(smem_u32(stg) + sw128_offset(ln, (W * k + e) * 4), o[e], o[e + 1], o[e + 2], o[e + 3]);
            } else if (m0 + row_in < p.s_q) {
              uint4* dst = reinterpret_cast<uint4*>(static_cast<TO*>(p.out) + (int64_t)zi * p.so_z + (int64_t)hi * p.so_h +
                                                    (int64_t)(m0 + row_in) * p.so_s + half * RC + c + 32 * k);
#pragma unroll
              for (int e = 0; e < W; e += 4) dst[e >> 2] = make_uint4(o[e], o[e + 1], o[e + 2], o[e + 3]);
            }
          }
          if (c + CC == RC && r1 > r0) {         // O has been read: the next item's products may overwrite it
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&o_free);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (p.tma_out && lane == 0 && m0 + wq * 32 < p.s_q)
            tma_store_4d(&tm_o, stg, (half * RC + c) * (int)sizeof(TO), m0 + wq * 32, hi, zi);
        }
        const int row = m0 + wq * 32 + (int)ln;
        if (p.lse != nullptr && half == 0 && row < p.s_q) {
          const float l_safe = (l_run == 0.0f) ? 1.0f : l_run;
          p.lse[((int64_t)zi * p.h + hi) * p.s_q + row] = m_fin * 0.6931471805599453f + logf(l_safe);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&item_free[sl]);
    }
    if (lane == 0) bulk_wait_read<0>();
  }
  tc_fence_before();
  __syncthreads();
  report_error_call(&err, p.status);
  if (warp == 1) tmem_dealloc(tmem, 512);
}

template <int D, typename TO>
int fwd_launch(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to,
               const FwdParams& p, int64_t zh, cudaStream_t st) {
  using C = FwdCfg<D>;
  auto kern = p.seq_id != nullptr ? (p.bias != nullptr ? fwd_kernel<D, TO, true, true> : fwd_kernel<D, TO, true, false>)
                                  : (p.bias != nullptr ? fwd_kernel<D, TO, false, true> : fwd_kernel<D, TO, false, false>);
  if (int rc = allow_smem("nvfp4_fwd", reinterpret_cast<const void*>(kern), C::SMEM_BYTES)) return rc;
  const int64_t z = zh / p.h;
  const dim3 grid((unsigned)(z < 65536 ? p.h : zh), (unsigned)(z < 65536 ? z : 1), (unsigned)((p.s_q + 127) / 128));
  return launch("nvfp4_fwd", kern, grid, kFwdThreads, C::SMEM_BYTES, st, tq, tk, tv, to, p);
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
  p.vec_sc = (((uintptr_t)qsc | (uintptr_t)ksc) % (d / 16)) == 0;
  p.scaling = scaling; p.causal = (flags & NVFP4_FWD_CAUSAL) ? 1 : 0; p.status = status;
  // Rows leave through a tensor map; strides that a map cannot express (zero, negative, beyond 2^40 bytes) are stored
  // row by row.  A stride that is never taken is replaced by one that a map accepts.
  const int64_t pitch = (int64_t)d * esz, os = s_q > 1 ? so_s * esz : pitch, oh = h > 1 ? so_h * esz : pitch,
                oz = z > 1 ? so_z * esz : pitch;
  auto expressible = [](int64_t v) { return v > 0 && v < (1LL << 40); };
  p.tma_out = expressible(os) && expressible(oh) && expressible(oz);
  CUtensorMap to = tq;
  if (p.tma_out && (rc = make_tmap_u8_4d_sw128(&to, out, pitch, s_q, h, z, os, oh, oz, 32, "nvfp4_fwd(out)"))) return rc;
#define NVFP4_FWD(DD, T) return fwd_launch<DD, T>(tq, tk, tv, to, p, zh, st)
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

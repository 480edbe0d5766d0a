// Legacy (old-format mask) attention backward on tcgen05 tensor cores (f16/bf16, head_dim 64/128).
//
// Mathematics (the scalar kernels in legacy_bwd.cu derive it; reference: psa_kernel_legacy.py:947-1320): a pooled token t
// of level l stands for l identical expanded keys, of which c_t(i) exist and are visible to query row i, so with
// p_it = exp(q_i.k_t scale - lse_i):
//   ds_it = round(p_it (dO_i.v_t - delta_i)) c_t(i),   pc_it = round(p_it) c_t(i)
//   dQ_i = scale sum_t ds_it k_t,   dK_j (j in t) += scale / l sum_i ds_it q_i,   dV_j (j in t) += 1 / l sum_i pc_it dO_i
// Two kernels share one skeleton: a STATIONARY pair of 128-row operand tiles in shared memory, a STREAM of 128-row operand
// tiles through two rings, S and dP of a stream tile as products of the two, one thread per accumulator row turning them
// into the 16-bit operand of the accumulating products IN PLACE in TMEM, and a single MMA-issuing thread.
// The element-wise warps work in two phases per tile: the probabilities as soon as S is there (kept in registers), dS once
// dP is.  So half of their work runs under products: in the dK/dV kernel dV and the next S under phase 2, dK and the next dP
// under phase 1; in the dQ kernel (S double-buffered) dQ and the next dP under phase 1 of the next tile.
// Bound by the issuing thread and its hand-overs with the element-wise warps: with empty element-wise bodies 10.1 of 12.1 ms
// remained, without ex2 or with half of the copies all of it.  2 x 16 heads x 32768 tokens x 128, causal, random levels: dK/dV
// 14.3 -> 11.4 ms, dQ 7.3 -> 6.0 ms against both products of a tile before its whole element-wise pass with two stages per
// ring; 28 heads x 5003 tokens: 492 -> 410 and 334 -> 273 us.
//
//   bwd_dq_tc_kernel    stationary: Q and dO of one query block (rows = queries).  Stream: the selected key blocks of
//                       all levels, PACKED back to back into 128-token K and V tiles (tile images, one linear bulk copy
//                       per block and operand).  S = Q K^T, dP = dO V^T, dS over dP, dQ += dS K (K read MN-major from
//                       the same tile).  Per-column metadata (copies, first original position) comes from the producer.
//   bwd_dkdv_tc_kernel  stationary: 128 consecutive pooled K and V rows of ONE level (= l consecutive key blocks),
//                       rows = pooled keys.  Stream: Q and dO tiles of every query block that selected that level for at
//                       least one of those key blocks (rows whose block was not selected get zeros).  S^T = K Q^T,
//                       dP^T = V dO^T, P^T over S^T, dS^T over dP^T, dV += P^T dO, dK += dS^T Q.  The fp32 sums of the
//                       pooled rows go to scratch; bwd_fold_kernel spreads them over the original positions
//                       (mean-pool backward), folds the replicate-padded tail into the last token and rounds once.
// Every wait is bounded; on expiry the CTA records PSA_ERR_TIMEOUT, lets copies in flight land, frees TMEM and returns.
#include <cstddef>

#include "psa_common.cuh"
#include "fwd.h"
#include "tc_common.cuh"

namespace psa {
namespace {

constexpr int kSlab = 128 * 128;          // 128 rows x 128 B (64 16-bit channels)
constexpr int kThreadsBwd = 576;          // warp 0 producer, warp 1 MMA issuer, warps 2-17 element-wise (four groups)
constexpr int kEwWarps = 16;
constexpr int kMaxBlocks = 1472;          // key / query blocks per head that the entry points take

__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
template <int FMT> __device__ __forceinline__ uint32_t pack16(float a, float b);
template <> __device__ __forceinline__ uint32_t pack16<1>(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t pack16<0>(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
template <int FMT> __device__ __forceinline__ float round16(float x);
template <> __device__ __forceinline__ float round16<1>(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
template <> __device__ __forceinline__ float round16<0>(float x) { return __half2float(__float2half_rn(x)); }

// Visible copies of the pooled token whose first original position is j0, for the query at qpos.
__device__ __forceinline__ int copies(int64_t j0, int level, int64_t l_k, int causal, int64_t qpos) {
  int64_t hi = l_k;
  if (causal && qpos + 1 < hi) hi = qpos + 1;
  const int64_t c = hi - j0;
  return c < 0 ? 0 : (c > level ? level : (int)c);
}

struct BwdParams {
  const int32_t* mask;       // [bh][mq][mask_cols] levels
  const unsigned char* kimg; // tile images (block 128) of K and V, all levels
  const unsigned char* vimg;
  ImgLevels img;
  const float* nlse;         // [bh][s_pad]: -lse in log2 units of every query row; rows >= seq: -inf
  const float* ndelta;       // [bh][s_pad]: -delta; rows >= seq: 0
  void* dq;                  // [bh][seq][D]
  float* dkp[4];             // pooled fp32 sums per level: [bh][s_pad / l][D]
  float* dvp[4];
  const int2* items;         // dK/dV work list: (level index, group), heavy first
  int n_entries;             // entries of `items` (per head)
  int* counter;              // zero at launch: work beyond the first item of every CTA is claimed from it
  int32_t* status;
  int64_t seq, s_pad, bh;
  int mq, mask_cols, causal;
  float scale, scale_log2;
};

struct TmapQD {
  CUtensorMap q, d;          // {64 channels, 128 rows} boxes of Q and dO, [bh][seq][D]
};

// Shared memory of both kernels: two stationary tiles, a ring X for the stream operand that the first and the last product
// of a tile read (Q in the dK/dV kernel, K in the dQ kernel) and a ring Y for the one that is done with earlier (dO, V).  A
// copy takes some 2500 cycles from its issue to its last byte, so with two stages each the dQ kernel waited for K on every
// tile; X has one stage more, and at head_dim 128 the seven tiles, the per-column words and the control block fill the 227 KB
// to the last byte (the base needs no slack: it is declared 1024-byte aligned, and the kernels check it).
template <int D> struct KCfg {
  static constexpr int SLABS = D / 64;
  static constexpr int TILE = SLABS * kSlab;
  static constexpr int NX = D == 64 ? 4 : 3, NY = D == 64 ? 3 : 2;
  static constexpr int OFF_A0 = 0, OFF_A1 = TILE;       // stationary: K, V (dK/dV) or Q, dO (dQ)
  static constexpr int OFF_X = 2 * TILE, OFF_Y = OFF_X + NX * TILE;
  static constexpr int OFF_YW = OFF_Y + NY * TILE;      // dK/dV: per Y stage 128 x -lse.  dQ: per X stage 8 x (first position, level)
  static constexpr int OFF_XW = OFF_YW + NY * 512;      // per X stage 128 words: -delta of the queries (dK/dV), log2(copies) of the keys (dQ)
  static constexpr int OFF_CTRL = OFF_XW + NX * 512;
  static constexpr int SMEM = OFF_CTRL + 512;
  static_assert(SMEM <= 232448, "more than 227 KB of shared memory");
  static_assert(NX * 64 <= NY * 512, "dQ block words");
};

struct KCtrl {
  uint64_t a_full, a_free;               // stationary tiles loaded / all products that read them complete
  uint64_t x_full[4], x_free[4], y_full[3], y_free[3];
  uint64_t s_full[2], p_full;            // S of a tile ready (dQ: of even / odd tiles; dK/dV: [0] only) / P^T written over it (dK/dV)
  uint64_t dp_full, ds_full;             // dP of a tile ready / dS written over it
  uint64_t acc_full, acc_free;
  uint64_t job_ready[3], job_done[3];
  int job_id[3], job_n[3], job_bh[3];    // id < 0: no more work; n == 0: nothing selected
  uint32_t ent[4];                       // per X stage, the tile's entry; bit 31: last tile of the job
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(KCtrl) <= 512, "control block");

// ------------------------------------------------------------------------------------------------------------------
// dK / dV
// ------------------------------------------------------------------------------------------------------------------
template <int D, int FMT>
__global__ void __launch_bounds__(kThreadsBwd, 1) bwd_dkdv_tc_kernel(const __grid_constant__ TmapQD maps, const BwdParams p) {
  using C = KCfg<D>;
  extern __shared__ __align__(1024) unsigned char smem[];
  KCtrl* ctl = reinterpret_cast<KCtrl*>(smem + C::OFF_CTRL);
  volatile int* abort_flag = &ctl->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (tc::smem_u32(smem) & 1023) {          // the swizzled tiles need it; nothing has been started yet
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, PSA_ERR_TIMEOUT);
    return;
  }

  if (threadIdx.x == 0) {
    tc::mbar_init(&ctl->a_full, 1); tc::mbar_init(&ctl->a_free, 1);
    for (int i = 0; i < C::NX; ++i) { tc::mbar_init(&ctl->x_full[i], 1); tc::mbar_init(&ctl->x_free[i], 1); }
    for (int i = 0; i < C::NY; ++i) { tc::mbar_init(&ctl->y_full[i], 1); tc::mbar_init(&ctl->y_free[i], 1); }
    tc::mbar_init(&ctl->s_full[0], 1); tc::mbar_init(&ctl->p_full, kEwWarps);
    tc::mbar_init(&ctl->dp_full, 1); tc::mbar_init(&ctl->ds_full, kEwWarps);
    tc::mbar_init(&ctl->acc_full, 1); tc::mbar_init(&ctl->acc_free, kEwWarps);
    for (int i = 0; i < 3; ++i) { tc::mbar_init(&ctl->job_ready[i], 1); tc::mbar_init(&ctl->job_done[i], kEwWarps + 1); }
    ctl->abort_flag = 0;
    tc::fence_mbar_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(&ctl->tmem_base, 512);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;
  const int nk = p.mq;                                      // key blocks = query blocks
  const int64_t total_jobs = (int64_t)p.n_entries * p.bh;
  // TMEM columns: dK [0,D), dV [128,128+D), S^T [256,384), dP^T [384,512)
  constexpr uint32_t kAccK = 0, kAccV = 128, kST = 256, kDP = 384;

  if (warp == 0) {
    // ================================================================ producer
    bool ok = true;
    int gp = 0, ic = 0;                                    // stream tiles issued so far / jobs with work so far
    int64_t job = blockIdx.x;
    for (int it = 0; ok; ++it) {
      const int slot = it % 3;
      if (it >= 3) {
        ok = tc::mbar_wait(&ctl->job_done[slot], ((it / 3) - 1) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
      }
      if (job >= total_jobs) {
        if (lane == 0) { ctl->job_id[slot] = -1; __threadfence_block(); tc::mbar_arrive(&ctl->job_ready[slot]); }
        break;
      }
      // head-major order: the CTAs running at the same time stream the Q and dO rows of the same head (they stay in L2)
      const int2 e = p.items[job % p.n_entries];
      const int64_t bh = job / p.n_entries;
      const int li = e.x, g = e.y, l = 1 << li;
      const int n0 = g * l;                                // first key block of the group
      const int nsub = min(l, nk - n0);
      // Query blocks that selected level l for at least one of the group's key blocks, with the sub-block bits: found
      // while the job streams, 32 query blocks (one per lane) at a time and one pair ahead of the copies, so that a job
      // needs no list and does not start with a scan of the whole mask column.
      const int32_t* mbase = p.mask + (bh * p.mq) * (int64_t)p.mask_cols + n0;
      int m_next = p.causal ? n0 : 0, m_win = 0;
      uint32_t my_bits = 0;
      unsigned hits = 0;
      auto next_pair = [&](uint32_t& pair) -> bool {
        while (hits == 0 && m_next < p.mq) {
          m_win = m_next;
          const int m = m_win + lane;
          my_bits = 0;
          if (m < p.mq) {
            const int32_t* row = mbase + (int64_t)m * p.mask_cols;
            for (int i = 0; i < nsub; ++i)
              if (row[i] == l && (!p.causal || n0 + i <= m)) my_bits |= 1u << i;
          }
          hits = __ballot_sync(0xffffffffu, my_bits != 0);
          m_next += 32;
        }
        if (hits == 0) return false;
        const int at = __ffs(hits) - 1;
        hits &= hits - 1;
        pair = (uint32_t)(m_win + at) | __shfl_sync(0xffffffffu, my_bits, at) << 16;
        return true;
      };
      uint32_t pair = 0;
      bool have = next_pair(pair);
      if (lane == 0) {
        ctl->job_id[slot] = (int)job; ctl->job_n[slot] = have; ctl->job_bh[slot] = (int)bh;
        __threadfence_block();
        tc::mbar_arrive(&ctl->job_ready[slot]);
      }
      // next job (claimed now, so that the atomic's latency is hidden)
      int next = 0;
      if (lane == 0) next = atomicAdd(p.counter, 1);
      next = __shfl_sync(0xffffffffu, next, 0);
      job = (int64_t)gridDim.x + next;
      if (!have) continue;
      // stationary K and V rows [g*128, g*128+128) of level li (fewer at the end of the level)
      ok = tc::mbar_wait(&ctl->a_free, (ic & 1) ^ 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      if (lane == 0) {
        const int64_t n_l = p.s_pad >> li;
        const int rows = (int)min((int64_t)128, n_l - (int64_t)g * 128);
        const int64_t off = p.img.off[li] + (((int64_t)bh * p.img.groups[li] + (int64_t)g * 16) * C::SLABS << 10);
        const uint32_t bytes = (uint32_t)rows * D * 2;
        tc::bulk_load_a(tc::smem_u32(smem + C::OFF_A0), p.kimg + off, bytes, tc::smem_u32(&ctl->a_full));
        tc::bulk_load_a(tc::smem_u32(smem + C::OFF_A1), p.vimg + off, bytes, tc::smem_u32(&ctl->a_full));
        tc::mbar_arrive_expect_tx(&ctl->a_full, 2 * bytes);
      }
      ++ic;
      while (have) {
        uint32_t cur = pair;
        have = next_pair(pair);
        if (!have) cur |= 1u << 31;
        const int m = (int)(cur & 0xffffu), qs = gp % C::NX, ds = gp % C::NY;
        // Q: free once dK of the stage's previous tile is complete; dO: once its dV is, half a tile earlier
        ok = tc::mbar_wait(&ctl->x_free[qs], ((gp / C::NX) & 1) ^ 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if (lane == 0) {
          ctl->ent[qs] = cur;
          for (int s = 0; s < C::SLABS; ++s)
            tc::tma_load_3d(smem + C::OFF_X + qs * C::TILE + s * kSlab, &maps.q, &ctl->x_full[qs], s * 64, m * 128, (int)bh);
          tc::bulk_load_a(tc::smem_u32(smem + C::OFF_XW + qs * 512), p.ndelta + bh * p.s_pad + (int64_t)m * 128, 512,
                          tc::smem_u32(&ctl->x_full[qs]));
          tc::mbar_arrive_expect_tx(&ctl->x_full[qs], C::TILE + 512);
        }
        ok = tc::mbar_wait(&ctl->y_free[ds], ((gp / C::NY) & 1) ^ 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if (lane == 0) {
          for (int s = 0; s < C::SLABS; ++s)
            tc::tma_load_3d(smem + C::OFF_Y + ds * C::TILE + s * kSlab, &maps.d, &ctl->y_full[ds], s * 64, m * 128, (int)bh);
          tc::bulk_load_a(tc::smem_u32(smem + C::OFF_YW + ds * 512), p.nlse + bh * p.s_pad + (int64_t)m * 128, 512,
                          tc::smem_u32(&ctl->y_full[ds]));
          tc::mbar_arrive_expect_tx(&ctl->y_full[ds], C::TILE + 512);
        }
        ++gp;
      }
    }
  } else if (warp == 1) {
    // ================================================================ MMA issuer
    if (lane == 0) {
      bool ok = true;
      const uint32_t idesc_s = tc::make_idesc(FMT, 128, 128, 0, 0);
      const uint32_t idesc_acc = tc::make_idesc(FMT, 128, D, 0, 1);
      const uint64_t kdesc = tc::make_smem_desc(tc::smem_u32(smem + C::OFF_A0), 16, C::SLABS * 1024);
      const uint64_t vdesc = tc::make_smem_desc(tc::smem_u32(smem + C::OFF_A1), 16, C::SLABS * 1024);
      const uint64_t qk0 = tc::make_smem_desc(tc::smem_u32(smem + C::OFF_X), 16, 1024);       // stream tiles as K-major B
      const uint64_t dk0 = tc::make_smem_desc(tc::smem_u32(smem + C::OFF_Y), 16, 1024);
      const uint64_t qm0 = tc::make_smem_desc(tc::smem_u32(smem + C::OFF_X), kSlab, 1024);    // ... and as MN-major B
      const uint64_t dm0 = tc::make_smem_desc(tc::smem_u32(smem + C::OFF_Y), kSlab, 1024);
      const uint32_t ctl_a = tc::smem_u32(ctl);
      const uint32_t s_full_a = ctl_a + (uint32_t)offsetof(KCtrl, s_full), p_full_a = ctl_a + (uint32_t)offsetof(KCtrl, p_full);
      const uint32_t dp_full_a = ctl_a + (uint32_t)offsetof(KCtrl, dp_full), ds_full_a = ctl_a + (uint32_t)offsetof(KCtrl, ds_full);
      const uint32_t q_full_a = ctl_a + (uint32_t)offsetof(KCtrl, x_full), d_full_a = ctl_a + (uint32_t)offsetof(KCtrl, y_full);
      const volatile uint32_t* ent = ctl->ent;
      int gp = 0, ic = 0;
      auto q_off = [&](int u) { return (uint64_t)((uint32_t)((u % C::NX) * C::TILE) >> 4); };
      auto d_off = [&](int u) { return (uint64_t)((uint32_t)((u % C::NY) * C::TILE) >> 4); };
      // a stationary tile (image layout) times a stream tile, N = 128 query rows.  A look at a barrier takes ~170 cycles whether
      // its phase is complete or not, so the one the next product needs is looked at behind the last but two MMAs of this one (dK/dV
      // 12.5 -> 11.4 ms, the look at the next stage before an accumulating product included).
      auto issue_ss = [&](uint32_t dst, uint64_t adesc, uint64_t bdesc, uint32_t done, uint32_t next_bar, uint32_t next_par) -> bool {
        bool there = false;
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          tc::umma_ss(dst, adesc + (uint64_t)(((ks >> 2) * 1024 + (ks & 3) * 32) >> 4),
                      bdesc + (uint64_t)(((ks >> 2) * kSlab + (ks & 3) * 32) >> 4), idesc_s, ks > 0 ? 1u : 0u);
          if (ks == D / 16 - 3) there = tc::mbar_test_wait_a(next_bar, next_par);
        }
        tc::umma_commit_a(done);
        return there;
      };
      // an accumulating product.  k-step ks = query rows [16 ks, 16 ks + 16); its 16-bit operand sits at column
      // 32 (ks / 2) + 8 (ks % 2) of the buffer the fp32 values came from
      auto issue_acc = [&](uint32_t acc, uint32_t src, uint64_t bdesc, bool first) {
        tc::umma_ts(acc, src, bdesc, idesc_acc, first ? 0u : 1u);
#pragma unroll
        for (int ks = 1; ks < 8; ++ks)
          tc::umma_ts(acc, src + (ks >> 1) * 32 + (ks & 1) * 8, bdesc + (uint64_t)(ks * (2048 >> 4)), idesc_acc, 1u);
      };
      for (int it = 0; ok; ++it) {
        const int slot = it % 3;
        ok = tc::mbar_wait(&ctl->job_ready[slot], (it / 3) & 1, abort_flag);
        if (!ok || ctl->job_id[slot] < 0) break;
        if (ctl->job_n[slot] == 0) { tc::mbar_arrive(&ctl->job_done[slot]); continue; }
        ok = tc::mbar_wait(&ctl->a_full, ic & 1, abort_flag);
        if (ok) ok = tc::mbar_wait_a(q_full_a + (gp % C::NX) * 8, (gp / C::NX) & 1, abort_flag);
        if (!ok) break;
        tc::tc_fence_after();
        if (!issue_ss(tmem + kST, kdesc, qk0 + q_off(gp), s_full_a, d_full_a + (gp % C::NY) * 8, (gp / C::NY) & 1))
          ok = tc::mbar_wait_a(d_full_a + (gp % C::NY) * 8, (gp / C::NY) & 1, abort_flag);
        if (!ok) break;
        tc::tc_fence_after();
        bool p_there = issue_ss(tmem + kDP, vdesc, dk0 + d_off(gp), dp_full_a, p_full_a, gp & 1);
        // dV and S^T of the next tile run while the element-wise warps turn dP^T into dS^T, dK and dP^T of the next tile
        // while they take the probabilities of the next tile
        for (bool first = true; ok; first = false, ++gp) {
          const bool last = (ent[gp % C::NX] >> 31) != 0;
          if (!p_there) ok = tc::mbar_wait_a(p_full_a, gp & 1, abort_flag);
          if (ok && first && ic > 0) ok = tc::mbar_wait(&ctl->acc_free, (ic - 1) & 1, abort_flag);
          if (!ok) break;
          tc::tc_fence_after();
          bool ds_there = false;
          const uint32_t q_bar = q_full_a + ((gp + 1) % C::NX) * 8, q_par = ((gp + 1) / C::NX) & 1;
          const bool q_there = tc::mbar_test_wait_a(q_bar, q_par);
          issue_acc(tmem + kAccV, tmem + kST, dm0 + d_off(gp), first);
          if (!last) {
            if (!q_there) ok = tc::mbar_wait_a(q_bar, q_par, abort_flag);
            if (!ok) break;
            tc::tc_fence_after();
            ds_there = issue_ss(tmem + kST, kdesc, qk0 + q_off(gp + 1), s_full_a, ds_full_a, gp & 1);   // "S ready" also says: dV of this tile is complete
          }
          if (!ds_there) ok = tc::mbar_wait_a(ds_full_a, gp & 1, abort_flag);
          if (!ok) break;
          tc::tc_fence_after();
          const uint32_t d_bar = d_full_a + ((gp + 1) % C::NY) * 8, d_par = ((gp + 1) / C::NY) & 1;
          const bool d_there = tc::mbar_test_wait_a(d_bar, d_par);
          issue_acc(tmem + kAccK, tmem + kDP, qm0 + q_off(gp), first);
          if (last) { ++gp; break; }
          if (!d_there) ok = tc::mbar_wait_a(d_bar, d_par, abort_flag);
          if (!ok) break;
          tc::tc_fence_after();
          p_there = issue_ss(tmem + kDP, vdesc, dk0 + d_off(gp + 1), dp_full_a, p_full_a, (gp + 1) & 1);   // "dP ready" also says: dK of this tile is complete
        }
        if (!ok) break;
        tc::umma_commit(&ctl->acc_full);
        tc::umma_commit(&ctl->a_free);
        tc::mbar_arrive(&ctl->job_done[slot]);
        ++ic;
      }
    }
  } else {
    // ================================================================ element-wise warps: one thread per pooled key row
    // four groups of four warps; group cg works on query columns [32 cg, 32 cg + 32) of the tile
    const int quarter = warp & 3, cg = (warp - 2) >> 2;
    const int r = quarter * 32 + lane;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const uint32_t tST = tmem + kST + cg * 32 + lane_base, tDP = tmem + kDP + cg * 32 + lane_base;
    const bool relay = warp == 2 && lane == 0;                 // tells the producer which stream stages are free again
    bool ok = true;
    int gp = 0, ic = 0;
    for (int it = 0; ok; ++it) {
      const int slot = it % 3;
      ok = tc::mbar_wait(&ctl->job_ready[slot], (it / 3) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      const int job = ctl->job_id[slot];
      if (job < 0) break;
      const int64_t bh = ctl->job_bh[slot];
      const int2 e = p.items[job % p.n_entries];
      const int li = e.x, g = e.y, l = 1 << li;
      const int n0 = g * l;
      const int64_t n_l = p.s_pad >> li;
      const int64_t t = (int64_t)g * 128 + r;                 // pooled row of this thread
      const bool exists = t < n_l;
      const int sub = (r << li) >> 7;                        // key block of the group this row belongs to
      const int64_t j0 = t * l, l_k = li == 0 ? p.seq : p.s_pad;
      const bool any_copy = copies(j0, l, l_k, 0, 0) > 0;    // l = 2^li copies wherever there are any (level 1: 1)
      // the sums of this row: groups 0, 1 store the two halves of the dK channels, groups 2, 3 those of dV
      constexpr int HD = D / 2;
      float* dst = (cg < 2 ? p.dkp[li] : p.dvp[li]) + (bh * n_l + t) * D + (cg & 1) * HD;
      if (ctl->job_n[slot] == 0) {
        if (exists)
          for (int c = 0; c < HD; c += 4) *reinterpret_cast<float4*>(dst + c) = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&ctl->job_done[slot]);
        continue;
      }
      for (bool first = true; ok; first = false, ++gp) {
        const int qs = gp % C::NX, ds = gp % C::NY;
        // ---- phase 1: P^T over S^T.  The probabilities stay in registers for phase 2.
        ok = tc::mbar_wait(&ctl->y_full[ds], (gp / C::NY) & 1, abort_flag);        // the tile's -lse
        if (ok) ok = tc::mbar_wait(&ctl->x_full[qs], (gp / C::NX) & 1, abort_flag);  // ... -delta and entry
        if (ok) ok = tc::mbar_wait(&ctl->s_full[0], gp & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        // S^T of this tile was issued behind dV of the previous one: its dO stage may be refilled
        if (relay && !first) tc::mbar_arrive(&ctl->y_free[(gp - 1) % C::NY]);
        tc::tc_fence_after();
        const uint32_t ent = ctl->ent[qs];
        const int m = (int)(ent & 0xffffu);
        const bool act = exists && ((ent >> (16 + sub)) & 1u);
        const bool slow = __any_sync(0xffffffffu, p.causal && act && (n0 + sub == m));
        const int64_t qbase = (int64_t)m * 128 + cg * 32;
        const float4* lse4 = reinterpret_cast<const float4*>(smem + C::OFF_YW + ds * 512) + cg * 8;
        const float4* del4 = reinterpret_cast<const float4*>(smem + C::OFF_XW + qs * 512) + cg * 8;
        // Every copy that exists is visible away from the causal diagonal: the count c is a power of two (or 0), so it goes
        // into the exponent - p c = 2^(s scale - lse + log2 c), exact scaling - and one rounding after the product equals
        // the reference's rounding before it.  c = 0 (row not selected by this query block, or no copy exists): log2 c =
        // -inf gives p = 0 and ds = 0 * finite.  On the diagonal the copies a query sees depend on its position, and p is
        // kept without the count.  Two columns at a time on the packed fp32 pipe; the packed 16-bit results go back IN
        // PLACE into columns this thread has read itself - chunk c of 16 columns into [8 c, 8 c + 8) of its group's columns -
        // because the other groups work on the same buffers at the same time; the MMA takes every 16-element k-step from
        // its own TMEM address, so the operand need not be contiguous.
        const float lc = slow ? 0.f : (act && any_copy) ? (float)li : -INFINITY;
        const float2 lc2 = make_float2(lc, lc), sl2 = make_float2(p.scale_log2, p.scale_log2);
        auto seen = [&](int col) { return act ? (float)copies(j0, l, l_k, 1, qbase + col) : 0.f; };
        float2 pr[16];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t sv[16], pp[8];
          tc::tmem_ld16(tST + 16 * c, sv);
          tc::tmem_wait_ld();
#pragma unroll
          for (int k = 0; k < 8; k += 2) {
            const float4 s4 = lse4[c * 4 + (k >> 1)];
            const float2 xa = __ffma2_rn(make_float2(__uint_as_float(sv[2 * k]), __uint_as_float(sv[2 * k + 1])), sl2,
                                         __fadd2_rn(lc2, make_float2(s4.x, s4.y)));
            const float2 xb = __ffma2_rn(make_float2(__uint_as_float(sv[2 * k + 2]), __uint_as_float(sv[2 * k + 3])), sl2,
                                         __fadd2_rn(lc2, make_float2(s4.z, s4.w)));
            pr[c * 8 + k] = make_float2(ex2f(xa.x), ex2f(xa.y));
            pr[c * 8 + k + 1] = make_float2(ex2f(xb.x), ex2f(xb.y));
          }
#pragma unroll
          for (int k = 0; k < 8; ++k) pp[k] = pack16<FMT>(pr[c * 8 + k].x, pr[c * 8 + k].y);
          if (slow) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const float c0 = seen(c * 16 + 2 * k), c1 = seen(c * 16 + 2 * k + 1);
              pp[k] = pack16<FMT>(c0 > 0.f ? round16<FMT>(pr[c * 8 + k].x) * c0 : 0.f, c1 > 0.f ? round16<FMT>(pr[c * 8 + k].y) * c1 : 0.f);
            }
          }
          tc::tmem_st8(tST + 8 * c, pp);
        }
        tc::tmem_wait_st();
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&ctl->p_full);
        // ---- phase 2: dS^T over dP^T
        ok = tc::mbar_wait(&ctl->dp_full, gp & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        // dP^T of this tile was issued behind dK of the previous one: its Q stage may be refilled
        if (relay && !first) tc::mbar_arrive(&ctl->x_free[(gp - 1) % C::NX]);
        tc::tc_fence_after();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t dv[16], pd[8];
          tc::tmem_ld16(tDP + 16 * c, dv);
          tc::tmem_wait_ld();
          float2 y[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const float4 d4 = del4[c * 4 + (k >> 1)];
            y[k] = __fmul2_rn(pr[c * 8 + k], __fadd2_rn(make_float2(__uint_as_float(dv[2 * k]), __uint_as_float(dv[2 * k + 1])),
                                                        (k & 1) ? make_float2(d4.z, d4.w) : make_float2(d4.x, d4.y)));
            pd[k] = pack16<FMT>(y[k].x, y[k].y);
          }
          if (slow) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const float c0 = seen(c * 16 + 2 * k), c1 = seen(c * 16 + 2 * k + 1);
              pd[k] = pack16<FMT>(c0 > 0.f ? round16<FMT>(y[k].x) * c0 : 0.f, c1 > 0.f ? round16<FMT>(y[k].y) * c1 : 0.f);
            }
          }
          tc::tmem_st8(tDP + 8 * c, pd);
        }
        tc::tmem_wait_st();
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&ctl->ds_full);
        if (ent >> 31) { ++gp; break; }
      }
      if (!ok) break;
      // ---- the pooled rows' sums
      ok = tc::mbar_wait(&ctl->acc_full, ic & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      if (relay) { tc::mbar_arrive(&ctl->y_free[(gp - 1) % C::NY]); tc::mbar_arrive(&ctl->x_free[(gp - 1) % C::NX]); }   // the last tile's stages
      tc::tc_fence_after();
      const uint32_t tAcc = tmem + (cg < 2 ? kAccK : kAccV) + (cg & 1) * HD + lane_base;
#pragma unroll 1
      for (int c0 = 0; c0 < HD; c0 += 32) {
        uint32_t a[32];
        tc::tmem_ld32(tAcc + c0, a);
        tc::tmem_wait_ld();
        if (exists) {
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            *reinterpret_cast<float4*>(dst + c0 + i) = make_float4(__uint_as_float(a[i]), __uint_as_float(a[i + 1]),
                                                                    __uint_as_float(a[i + 2]), __uint_as_float(a[i + 3]));
        }
      }
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) { tc::mbar_arrive(&ctl->acc_free); tc::mbar_arrive(&ctl->job_done[slot]); }
      ++ic;
    }
  }

  tc::tc_fence_before();
  __syncthreads();
  if (ctl->abort_flag) {
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, PSA_ERR_TIMEOUT);
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    __syncwarp();
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, 512);
  }
}

// ------------------------------------------------------------------------------------------------------------------
// dQ
// ------------------------------------------------------------------------------------------------------------------
template <int D, int FMT>
__global__ void __launch_bounds__(kThreadsBwd, 1) bwd_dq_tc_kernel(const __grid_constant__ TmapQD maps, const BwdParams p) {
  using C = KCfg<D>;
  extern __shared__ __align__(1024) unsigned char smem[];
  KCtrl* ctl = reinterpret_cast<KCtrl*>(smem + C::OFF_CTRL);
  volatile int* abort_flag = &ctl->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (tc::smem_u32(smem) & 1023) {          // the swizzled tiles need it; nothing has been started yet
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, PSA_ERR_TIMEOUT);
    return;
  }

  if (threadIdx.x == 0) {
    tc::mbar_init(&ctl->a_full, 1); tc::mbar_init(&ctl->a_free, 1);
    for (int i = 0; i < C::NX; ++i) { tc::mbar_init(&ctl->x_full[i], 1); tc::mbar_init(&ctl->x_free[i], 1); }
    for (int i = 0; i < C::NY; ++i) { tc::mbar_init(&ctl->y_full[i], 1); tc::mbar_init(&ctl->y_free[i], 1); }
    tc::mbar_init(&ctl->s_full[0], 1); tc::mbar_init(&ctl->s_full[1], 1);
    tc::mbar_init(&ctl->dp_full, 1); tc::mbar_init(&ctl->ds_full, kEwWarps);
    tc::mbar_init(&ctl->acc_full, 1); tc::mbar_init(&ctl->acc_free, kEwWarps);
    for (int i = 0; i < 3; ++i) { tc::mbar_init(&ctl->job_ready[i], 1); tc::mbar_init(&ctl->job_done[i], kEwWarps + 1); }
    ctl->abort_flag = 0;
    tc::fence_mbar_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(&ctl->tmem_base, 512);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;
  const int nk = p.mq;
  const int64_t total_rows = (int64_t)p.mq * p.bh;
  // TMEM columns: dQ [0,D), S of even tiles [128,256), S of odd tiles [256,384), dP [384,512)
  constexpr uint32_t kAcc = 0, kS = 128, kDP = 384;
  constexpr int kGroup = C::SLABS * 1024;          // 8 rows of a tile image

  if (warp == 0) {
    // ================================================================ producer
    bool ok = true;
    int gt = 0, rc = 0;                                    // stream tiles issued so far / rows with work so far
    int64_t R = blockIdx.x;
    for (int it = 0; ok; ++it) {
      const int slot = it % 3;
      if (it >= 3) {
        ok = tc::mbar_wait(&ctl->job_done[slot], ((it / 3) - 1) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
      }
      if (R >= total_rows) {
        if (lane == 0) { ctl->job_id[slot] = -1; __threadfence_block(); tc::mbar_arrive(&ctl->job_ready[slot]); }
        break;
      }
      // head-major order (the CTAs running at the same time stream the K/V images of the same head: they stay in L2);
      // within a head the causal rows are walked from the last query block down, the long ones first
      const int m = p.causal ? p.mq - 1 - (int)(R % p.mq) : (int)(R % p.mq);
      const int64_t bh = R / p.mq;
      // The row's blocks, level by level, found in the dense level row 32 entries at a time and one block ahead of the tile
      // that is put together: entry = block | level index << 12.
      const int32_t* mrow = p.mask + (bh * p.mq + m) * (int64_t)p.mask_cols;
      const int end = p.causal ? min(nk, m + 1) : nk;
      int li_next = 0, c_next = 0, c_win = 0;
      unsigned hits = 0;
      auto next_block = [&](uint32_t& blk) -> bool {
        while (hits == 0 && li_next < 4) {
          if (c_next >= end) { ++li_next; c_next = 0; continue; }
          c_win = c_next;
          const int c = c_win + lane;
          hits = __ballot_sync(0xffffffffu, c < end && mrow[c] == (1 << li_next));
          c_next += 32;
        }
        if (hits == 0) return false;
        blk = (uint32_t)(c_win + __ffs(hits) - 1) | (uint32_t)li_next << 12;
        hits &= hits - 1;
        return true;
      };
      uint32_t blk = 0;
      bool have = next_block(blk);
      if (lane == 0) {
        ctl->job_id[slot] = (int)R; ctl->job_n[slot] = have;
        __threadfence_block();
        tc::mbar_arrive(&ctl->job_ready[slot]);
      }
      int next = 0;
      if (lane == 0) next = atomicAdd(p.counter, 1);
      next = __shfl_sync(0xffffffffu, next, 0);
      R = (int64_t)gridDim.x + next;
      if (!have) continue;
      // stationary Q and dO tiles of the query block
      ok = tc::mbar_wait(&ctl->a_free, (rc & 1) ^ 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      if (lane == 0) {
        for (int s = 0; s < C::SLABS; ++s) {
          tc::tma_load_3d(smem + C::OFF_A0 + s * kSlab, &maps.q, &ctl->a_full, s * 64, m * 128, (int)bh);
          tc::tma_load_3d(smem + C::OFF_A1 + s * kSlab, &maps.d, &ctl->a_full, s * 64, m * 128, (int)bh);
        }
        tc::mbar_arrive_expect_tx(&ctl->a_full, 2 * C::TILE);
      }
      ++rc;
      while (have) {
        // the next tile: blocks packed back to back (they come in falling width, a power of two, so none straddles a tile);
        // lane i holds block i
        uint32_t mine = 0, flag_diag = 0;
        int in_tile = 0, cols = 0, my_col = 0;
        do {
          if (lane == in_tile) { mine = blk; my_col = cols; }
          if (p.causal && (int)(blk & 0xfffu) == m) flag_diag = 1;
          cols += 128 >> (blk >> 12);
          ++in_tile;
          have = next_block(blk);
        } while (have && cols < 128);
        const int xs = gt % C::NX, ys = gt % C::NY;
        const int li = (int)(mine >> 12), b = (int)(mine & 0xfffu), P = 128 >> li;
        const int64_t off = p.img.off[li] + (((int64_t)bh * p.img.groups[li] + (((int64_t)b * P) >> 3)) * C::SLABS << 10);
        const uint32_t dstoff = (uint32_t)(my_col >> 3) * kGroup, my_bytes = (uint32_t)(P * D * 2), bytes = (uint32_t)(cols * D * 2);
        // K and the words beside it: free once dQ of the stage's previous tile is complete
        ok = tc::mbar_wait(&ctl->x_free[xs], ((gt / C::NX) & 1) ^ 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if (lane < in_tile)
          tc::bulk_load_a(tc::smem_u32(smem + C::OFF_X + xs * C::TILE) + dstoff, p.kimg + off, my_bytes, tc::smem_u32(&ctl->x_full[xs]));
        // Per 16 columns the first original position and the level of their block (read on the causal diagonal only), per
        // column log2 of the copies that exist (-inf: none), written by the whole warp block after block.
        int2* units = reinterpret_cast<int2*>(smem + C::OFF_YW + xs * 64);
        float* lcol = reinterpret_cast<float*>(smem + C::OFF_XW + xs * 512);
        for (int i = 0; i < in_tile; ++i) {
          const int b_li = __shfl_sync(0xffffffffu, li, i), b_b = __shfl_sync(0xffffffffu, b, i), b_col = __shfl_sync(0xffffffffu, my_col, i);
          const int b_l = 1 << b_li, b_P = 128 >> b_li;
          const int64_t l_k = b_li == 0 ? p.seq : p.s_pad, first = (int64_t)b_b * 128;
          for (int c = lane; c < b_P; c += 32) lcol[b_col + c] = first + (int64_t)c * b_l < l_k ? (float)b_li : -INFINITY;
          if (lane < b_P / 16) units[b_col / 16 + lane] = make_int2((int)first + lane * 16 * b_l, b_li);
        }
        for (int c = cols + lane; c < 128; c += 32) lcol[c] = -INFINITY;
        if (lane == 0) ctl->ent[xs] = (uint32_t)cols | flag_diag << 16 | (have ? 0u : 1u << 31);
        __syncwarp();
        if (lane == 0) tc::mbar_arrive_expect_tx(&ctl->x_full[xs], bytes);
        // V: free once dP of the stage's previous tile is complete
        ok = tc::mbar_wait(&ctl->y_free[ys], ((gt / C::NY) & 1) ^ 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if (lane < in_tile)
          tc::bulk_load_a(tc::smem_u32(smem + C::OFF_Y + ys * C::TILE) + dstoff, p.vimg + off, my_bytes, tc::smem_u32(&ctl->y_full[ys]));
        __syncwarp();
        if (lane == 0) tc::mbar_arrive_expect_tx(&ctl->y_full[ys], bytes);
        ++gt;
      }
    }
  } else if (warp == 1) {
    // ================================================================ MMA issuer
    if (lane == 0) {
      bool ok = true;
      const uint32_t idesc_acc = tc::make_idesc(FMT, 128, D, 0, 1);
      const uint32_t idesc_full = tc::make_idesc(FMT, 128, 128, 0, 0);
      const uint64_t qdesc = tc::make_smem_desc(tc::smem_u32(smem + C::OFF_A0), 16, 1024);
      const uint64_t ddesc = tc::make_smem_desc(tc::smem_u32(smem + C::OFF_A1), 16, 1024);
      const uint64_t kk0 = tc::make_smem_desc(tc::smem_u32(smem + C::OFF_X), 16, kGroup);      // stream tiles as K-major B
      const uint64_t vk0 = tc::make_smem_desc(tc::smem_u32(smem + C::OFF_Y), 16, kGroup);
      const uint64_t km0 = tc::make_smem_desc(tc::smem_u32(smem + C::OFF_X), 1024, kGroup);    // K tile as MN-major B
      const uint32_t ctl_a = tc::smem_u32(ctl);
      const uint32_t s_full_a = ctl_a + (uint32_t)offsetof(KCtrl, s_full), ds_full_a = ctl_a + (uint32_t)offsetof(KCtrl, ds_full);
      const uint32_t dp_full_a = ctl_a + (uint32_t)offsetof(KCtrl, dp_full);
      const uint32_t x_full_a = ctl_a + (uint32_t)offsetof(KCtrl, x_full), y_full_a = ctl_a + (uint32_t)offsetof(KCtrl, y_full);
      const volatile uint32_t* ent = ctl->ent;
      auto x_off = [&](int u) { return (uint64_t)((uint32_t)((u % C::NX) * C::TILE) >> 4); };
      auto y_off = [&](int u) { return (uint64_t)((uint32_t)((u % C::NY) * C::TILE) >> 4); };
      // a stationary tile times a stream tile, N = the tile's columns
      auto issue_ss = [&](uint32_t dst, uint64_t adesc, uint64_t bdesc, int cols, uint32_t done) {
        const uint32_t idesc = cols == 128 ? idesc_full : tc::make_idesc(FMT, 128, cols, 0, 0);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
          tc::umma_ss(dst, adesc + (uint64_t)(((ks >> 2) * kSlab + (ks & 3) * 32) >> 4),
                      bdesc + (uint64_t)(((ks >> 2) * 1024 + (ks & 3) * 32) >> 4), idesc, ks > 0 ? 1u : 0u);
        tc::umma_commit_a(done);
      };
      // dQ += dS K; k-step ks = columns [16 ks, 16 ks + 16) of the tile, whose 16-bit operand sits at column
      // 32 (ks / 2) + 8 (ks % 2) of the dP buffer
      auto issue_acc = [&](uint64_t kd, int cols, bool first) {
        if (cols == 128) {
          tc::umma_ts(tmem + kAcc, tmem + kDP, kd, idesc_acc, first ? 0u : 1u);
#pragma unroll
          for (int ks = 1; ks < 8; ++ks)
            tc::umma_ts(tmem + kAcc, tmem + kDP + (ks >> 1) * 32 + (ks & 1) * 8, kd + (uint64_t)(ks * ((2 * kGroup) >> 4)), idesc_acc, 1u);
        } else {
          for (int ks = 0; ks < cols / 16; ++ks)
            tc::umma_ts(tmem + kAcc, tmem + kDP + (ks >> 1) * 32 + (ks & 1) * 8, kd + (uint64_t)(ks * ((2 * kGroup) >> 4)), idesc_acc,
                        (first && ks == 0) ? 0u : 1u);
        }
      };
      int g0 = 0, rc = 0;                                   // stream tiles of the rows before this one / rows with work
      for (int it = 0; ok; ++it) {
        const int slot = it % 3;
        ok = tc::mbar_wait(&ctl->job_ready[slot], (it / 3) & 1, abort_flag);
        if (!ok || ctl->job_id[slot] < 0) break;
        if (ctl->job_n[slot] == 0) { tc::mbar_arrive(&ctl->job_done[slot]); continue; }
        ok = tc::mbar_wait(&ctl->a_full, rc & 1, abort_flag);
        if (!ok) break;
        tc::tc_fence_after();
        // Running tile numbers: next S, next dP, next dQ.  S runs up to two tiles ahead of dQ (two score buffers; the scores
        // of tile u-2 have been read once its dS is there), dP goes into the one buffer that dQ of the tile before has read
        // (the tensor pipe runs in issue order).  The issuer polls for whichever comes first.
        int ns = g0, np = g0, na = g0;
        bool s_done = false, done = false;
        uint32_t idle = 0;
        while (ok && !done) {
          bool progressed = false;
          // the three looks overlap (~170 cycles each); a phase that completes in between is found in the next round
          const bool ds_there = tc::mbar_test_wait_a(ds_full_a, na & 1);
          const bool y_there = tc::mbar_test_wait_a(y_full_a + (np % C::NY) * 8, (np / C::NY) & 1);
          const bool x_there = tc::mbar_test_wait_a(x_full_a + (ns % C::NX) * 8, (ns / C::NX) & 1);
          if (na < np && ds_there) {
            if (na == g0 && rc > 0) {
              ok = tc::mbar_wait(&ctl->acc_free, (rc - 1) & 1, abort_flag);
              if (!ok) break;
            }
            tc::tc_fence_after();
            const uint32_t e = ent[na % C::NX];
            issue_acc(km0 + x_off(na), (int)(e & 0xffffu), na == g0);
            done = (e >> 31) != 0;
            ++na;
            progressed = true;
          }
          if (np < ns && np == na && y_there) {
            tc::tc_fence_after();
            issue_ss(tmem + kDP, ddesc, vk0 + y_off(np), (int)(ent[np % C::NX] & 0xffffu), dp_full_a);   // also says: dQ of the tile before is complete
            ++np;
            progressed = true;
          }
          if (!s_done && ns <= na + 1 && x_there) {
            tc::tc_fence_after();
            const uint32_t e = ent[ns % C::NX];
            issue_ss(tmem + kS + (ns & 1) * 128, qdesc, kk0 + x_off(ns), (int)(e & 0xffffu), s_full_a + (ns & 1) * 8);
            s_done = (e >> 31) != 0;
            ++ns;
            progressed = true;
          }
          if (progressed) {
            idle = 0;
          } else if (++idle > (1u << 24) || ((idle & 1023) == 1023 && *abort_flag)) {
            *abort_flag = 1;
            ok = false;
          }
        }
        if (!ok) break;
        tc::umma_commit(&ctl->acc_full);
        tc::umma_commit(&ctl->a_free);
        tc::mbar_arrive(&ctl->job_done[slot]);
        ++rc;
        g0 = na;
      }
    }
  } else {
    // ================================================================ element-wise warps: one thread per query row
    // four groups of four warps; group cg works on columns [32 cg, 32 cg + 32) of the tile
    const int quarter = warp & 3, cg = (warp - 2) >> 2;
    const int r = quarter * 32 + lane;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const uint32_t tDP = tmem + kDP + cg * 32 + lane_base;
    const bool relay = warp == 2 && lane == 0;                 // tells the producer which stream stages are free again
    bool ok = true;
    int gt = 0, rc = 0;
    for (int it = 0; ok; ++it) {
      const int slot = it % 3;
      ok = tc::mbar_wait(&ctl->job_ready[slot], (it / 3) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      const int64_t R = ctl->job_id[slot];
      if (R < 0) break;
      const int m = p.causal ? p.mq - 1 - (int)(R % p.mq) : (int)(R % p.mq);
      const int64_t bh = R / p.mq;
      const int64_t qpos = (int64_t)m * 128 + r;
      constexpr int QD = D / 4;                               // channels of the row each group stores
      uint16_t* orow = reinterpret_cast<uint16_t*>(p.dq) + ((int64_t)bh * p.seq + qpos) * D + cg * QD;
      if (ctl->job_n[slot] == 0) {
        if (qpos < p.seq)
          for (int c = 0; c < QD; c += 8) *reinterpret_cast<uint4*>(orow + c) = make_uint4(0u, 0u, 0u, 0u);
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&ctl->job_done[slot]);
        continue;
      }
      // (-lse * log2 e, -delta) of this row; -inf for rows past the end
      const float2 my = make_float2(p.nlse[bh * p.s_pad + qpos], p.ndelta[bh * p.s_pad + qpos]);
      const float2 sl2 = make_float2(p.scale_log2, p.scale_log2), nlse2 = make_float2(my.x, my.x), ndel2 = make_float2(my.y, my.y);
      for (bool first = true; ok; first = false, ++gt) {
        const int xs = gt % C::NX;
        // ---- phase 1: the probabilities.  They need S only, which is computed while the tile before this one is still worked
        // on, so their ex2 (the longer half of the element-wise work) run under dQ of the previous tile and dP of this one.
        // They stay in registers until dP is there.
        ok = tc::mbar_wait(&ctl->s_full[gt & 1], (gt >> 1) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const uint32_t ent = ctl->ent[xs];
        const bool mine = cg * 32 < (int)(ent & 0xffffu), slow = (ent >> 16) & 1u;
        float2 pr[16];
        if (mine) {
          tc::tc_fence_after();
          const float4* lc4 = reinterpret_cast<const float4*>(smem + C::OFF_XW + xs * 512) + cg * 8;
          uint32_t sv[32];
          tc::tmem_ld32(tmem + kS + (gt & 1) * 128 + cg * 32 + lane_base, sv);
          tc::tmem_wait_ld();
          // the copy count of a column is a power of two (or 0): it goes into the exponent, p c = 2^(s scale - lse +
          // log2 c), so one rounding after the product equals the reference's rounding before it; log2 c = -inf
          // (no copy exists) gives 0.  On the causal diagonal the count follows in phase 2 and p is kept without it.  Two
          // columns at a time on the packed fp32 pipe.
          if (!slow) {
#pragma unroll
            for (int k = 0; k < 16; ++k) {
              const float4 l4 = lc4[k >> 1];
              const float2 x = __ffma2_rn(make_float2(__uint_as_float(sv[2 * k]), __uint_as_float(sv[2 * k + 1])), sl2,
                                          __fadd2_rn((k & 1) ? make_float2(l4.z, l4.w) : make_float2(l4.x, l4.y), nlse2));
              pr[k] = make_float2(ex2f(x.x), ex2f(x.y));
            }
          } else {
#pragma unroll
            for (int k = 0; k < 16; ++k) {
              const float2 x = __ffma2_rn(make_float2(__uint_as_float(sv[2 * k]), __uint_as_float(sv[2 * k + 1])), sl2, nlse2);
              pr[k] = make_float2(ex2f(x.x), ex2f(x.y));
            }
          }
        }
        // ---- phase 2: dS over dP
        ok = tc::mbar_wait(&ctl->dp_full, gt & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        // dP of this tile is complete, and so is dQ of the previous tile: V of this tile and K of the previous one may be
        // replaced
        if (relay) {
          tc::mbar_arrive(&ctl->y_free[gt % C::NY]);
          if (!first) tc::mbar_arrive(&ctl->x_free[(gt - 1) % C::NX]);
        }
        if (mine) {
          tc::tc_fence_after();
          const int2* units = reinterpret_cast<const int2*>(smem + C::OFF_YW + xs * 64) + cg * 2;
          // this thread's 32 columns in two chunks of 16, one after the other; the packed results go back in place into
          // columns of the dP buffer the thread has read itself (chunk c into [8 c, 8 c + 8) of its group's columns),
          // because the other groups work on the same buffer at the same time.  Columns past the tile's end hold stale
          // bits and are never read by a product.
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t dv[16], pd[8];
            tc::tmem_ld16(tDP + 16 * c, dv);
            tc::tmem_wait_ld();
            float2 y[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              y[k] = __fmul2_rn(pr[c * 8 + k], __fadd2_rn(make_float2(__uint_as_float(dv[2 * k]), __uint_as_float(dv[2 * k + 1])), ndel2));
              pd[k] = pack16<FMT>(y[k].x, y[k].y);
            }
            if (slow) {
              const int2 u = units[c];
              const int l = 1 << u.y;
              const int64_t l_k = u.y == 0 ? p.seq : p.s_pad;
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                const float c0 = (float)copies((int64_t)u.x + 2 * k * l, l, l_k, 1, qpos), c1 = (float)copies((int64_t)u.x + (2 * k + 1) * l, l, l_k, 1, qpos);
                pd[k] = pack16<FMT>(c0 > 0.f ? round16<FMT>(y[k].x) * c0 : 0.f, c1 > 0.f ? round16<FMT>(y[k].y) * c1 : 0.f);
              }
            }
            tc::tmem_st8(tDP + 8 * c, pd);
          }
          tc::tmem_wait_st();
          tc::tc_fence_before();
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&ctl->ds_full);
        if (ent >> 31) { ++gt; break; }
      }
      if (!ok) break;
      // ---- dQ rows: each group stores a quarter of the channels
      ok = tc::mbar_wait(&ctl->acc_full, rc & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      if (relay) tc::mbar_arrive(&ctl->x_free[(gt - 1) % C::NX]);   // K of the row's last tile
      tc::tc_fence_after();
      const uint32_t tAcc = tmem + kAcc + cg * QD + lane_base;
#pragma unroll
      for (int c0 = 0; c0 < QD; c0 += 16) {
        uint32_t a[16];
        tc::tmem_ld16(tAcc + c0, a);
        tc::tmem_wait_ld();
        if (qpos < p.seq) {
#pragma unroll
          for (int i = 0; i < 16; i += 8)
            *reinterpret_cast<uint4*>(orow + c0 + i) =
                make_uint4(pack16<FMT>(__uint_as_float(a[i]) * p.scale, __uint_as_float(a[i + 1]) * p.scale),
                           pack16<FMT>(__uint_as_float(a[i + 2]) * p.scale, __uint_as_float(a[i + 3]) * p.scale),
                           pack16<FMT>(__uint_as_float(a[i + 4]) * p.scale, __uint_as_float(a[i + 5]) * p.scale),
                           pack16<FMT>(__uint_as_float(a[i + 6]) * p.scale, __uint_as_float(a[i + 7]) * p.scale));
        }
      }
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) { tc::mbar_arrive(&ctl->acc_free); tc::mbar_arrive(&ctl->job_done[slot]); }
      ++rc;
    }
  }

  tc::tc_fence_before();
  __syncthreads();
  if (ctl->abort_flag) {
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, PSA_ERR_TIMEOUT);
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    __syncwarp();
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, 512);
  }
}

// ------------------------------------------------------------------------------------------------------------------
// Small kernels around the two: row statistics, the dK/dV work list, the fold of the pooled sums.
// ------------------------------------------------------------------------------------------------------------------
// Row statistics; block 0 also zeroes the work counters and writes the work list of the dK/dV kernel: every (level, group
// of 128 pooled rows), ordered by the group's first key block, so that under a causal mask the groups with the most query
// blocks come first.  HBM-bound (o and dO are read once): D/8 lanes share a row, 16 bytes each, and a thread has the words
// of four rows in flight.  32 heads x 32768 x 128: 204 -> 128 us (4.2 TB/s).
template <typename T, int D>
__global__ void __launch_bounds__(256) bwd_stat_kernel(const T* __restrict__ o, const T* __restrict__ dout, const float* __restrict__ lse,
                                                       float* __restrict__ nlse, float* __restrict__ ndelta, int64_t bh, int64_t seq,
                                                       int64_t s_pad, int2* __restrict__ items, int nk, int* __restrict__ counters, int o_aligned) {
  constexpr int CPR = D / 8, kRows = 256 / CPR, kUnroll = 4;
  if (blockIdx.x == 0) {
    if (threadIdx.x < 64) counters[threadIdx.x] = 0;
    for (int blk = threadIdx.x; blk < nk; blk += 256) {
      int n = blk + (blk + 1) / 2 + (blk + 3) / 4 + (blk + 7) / 8;      // entries of the blocks before this one
      for (int li = 0; li < 4; ++li)
        if ((blk & ((1 << li) - 1)) == 0) items[n++] = make_int2(li, blk >> li);
    }
  }
  const int c = threadIdx.x % CPR;
  const int64_t row0 = (int64_t)blockIdx.x * (kRows * kUnroll) + threadIdx.x / CPR;      // over bh * s_pad
  uint4 a[kUnroll], d[kUnroll];
  int64_t src[kUnroll];
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const int64_t row = row0 + u * kRows, b = row / s_pad, t = row - b * s_pad;
    src[u] = row < bh * s_pad && t < seq ? b * seq + t : -1;
    if (src[u] >= 0) {
      if (o_aligned) {
        a[u] = __ldg(reinterpret_cast<const uint4*>(o) + src[u] * CPR + c);
      } else {      // dO feeds a tensor map and is always aligned, o need not be
        T* e = reinterpret_cast<T*>(&a[u]);
#pragma unroll
        for (int i = 0; i < 8; ++i) e[i] = o[(src[u] * CPR + c) * 8 + i];
      }
      d[u] = __ldg(reinterpret_cast<const uint4*>(dout) + src[u] * CPR + c);
    }
  }
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const int64_t row = row0 + u * kRows;
    float acc = 0.f;
    if (src[u] >= 0) {
      const T* x = reinterpret_cast<const T*>(&a[u]);
      const T* y = reinterpret_cast<const T*>(&d[u]);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc = fmaf(Elem<T>::to_f(x[i]), Elem<T>::to_f(y[i]), acc);
    }
#pragma unroll
    for (int off = CPR / 2; off; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (c == 0 && row < bh * s_pad) {
      const float l = src[u] >= 0 ? lse[src[u]] : -INFINITY;
      // a row that saw no key has lse = -inf; its probabilities are taken as 0 (the reference leaves them undefined)
      nlse[row] = l == -INFINITY ? -INFINITY : -l * 1.4426950408889634f;
      ndelta[row] = src[u] >= 0 ? -acc : 0.f;
    }
  }
}

// dK[j] = scale * sum_l dKp_l[j / l] / l, dV[j] = sum_l dVp_l[j / l] / l; the replicate-padded positions [seq, s_pad)
// hand their share to token seq - 1.  HBM-bound (3.75 N fp32 sums read, 2 N elements written).  blockIdx.y: dK or dV.
// Blocks below n_main: one thread per 8 tokens (one row of level 8) and 4 channels, so that every pooled row is read once
// and all 15 loads are in flight together.  The blocks behind them take the last token of one head each when the sequence
// is padded: up to 128 positions, dealt to all threads (one thread walking them took 140 us of a 5003-token step).
// 32 heads x 32768 x 128: 458 -> 359 us (7 TB/s); 28 x 5003: 185 -> 57 us.
template <typename T>
__device__ __forceinline__ void store4(T* dst, const float4& v, float scale) {
  T e[4] = {Elem<T>::from_f(v.x * scale), Elem<T>::from_f(v.y * scale), Elem<T>::from_f(v.z * scale), Elem<T>::from_f(v.w * scale)};
  *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(e);
}

__device__ __forceinline__ void fma4(float4& s, const float4& a, float w) {
  s.x = fmaf(a.x, w, s.x); s.y = fmaf(a.y, w, s.y); s.z = fmaf(a.z, w, s.z); s.w = fmaf(a.w, w, s.w);
}

template <typename T, int D>
__global__ void __launch_bounds__(256) bwd_fold_kernel(BwdParams p, T* __restrict__ dk, T* __restrict__ dv, int n_main) {
  constexpr int CH = D / 4;
  float* const* src = blockIdx.y ? p.dvp : p.dkp;
  T* out = blockIdx.y ? dv : dk;
  const float scale = blockIdx.y ? 1.0f : p.scale;
  const bool tail = p.s_pad > p.seq;
  const int c = (int)(threadIdx.x % CH) * 4;
  auto at = [&](int li, int64_t bh, int64_t row) {
    return __ldg(reinterpret_cast<const float4*>(src[li] + (bh * (p.s_pad >> li) + row) * D + c));
  };
  if ((int)blockIdx.x < n_main) {
    const int64_t n8 = p.s_pad / 8, g = (int64_t)blockIdx.x * (256 / CH) + threadIdx.x / CH;
    if (g >= p.bh * n8) return;
    const int64_t bh = g / n8, j = g - bh * n8;
    if (j * 8 >= p.seq) return;
    float4 a1[8], a2[4], a4[2];
#pragma unroll
    for (int i = 0; i < 8; ++i) a1[i] = at(0, bh, j * 8 + i);
#pragma unroll
    for (int i = 0; i < 4; ++i) a2[i] = at(1, bh, j * 4 + i);
    a4[0] = at(2, bh, j * 2); a4[1] = at(2, bh, j * 2 + 1);
    const float4 a8 = at(3, bh, j);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int64_t tok = j * 8 + i;
      float4 s = a1[i];
      fma4(s, a2[i >> 1], 0.5f);
      fma4(s, a4[i >> 2], 0.25f);
      fma4(s, a8, 0.125f);
      if (tok < p.seq && !(tail && tok == p.seq - 1)) store4(out + (bh * p.seq + tok) * D + c, s, scale);
    }
    return;
  }
  __shared__ float4 part[256];
  const int64_t bh = (int64_t)blockIdx.x - n_main;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int64_t j = p.seq - 1 + threadIdx.x / CH; j < p.s_pad; j += 256 / CH)
#pragma unroll
    for (int li = 0; li < 4; ++li) fma4(s, at(li, bh, j >> li), 1.0f / (float)(1 << li));
  part[threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x < CH) {
    for (int i = 1; i < 256 / CH; ++i) fma4(s, part[i * CH + threadIdx.x], 1.0f);
    store4(out + (bh * p.seq + p.seq - 1) * D + c, s, scale);
  }
}

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

struct Scratch {
  size_t nlse, ndelta, pooled[8], items, counters, total;
};

Scratch scratch_layout(int64_t bh, int64_t seq, int D) {
  Scratch s;
  const int64_t nk = cdiv64(seq, 128), s_pad = nk * 128;
  size_t off = 0;
  s.nlse = off; off += align256((size_t)bh * s_pad * sizeof(float));
  s.ndelta = off; off += align256((size_t)bh * s_pad * sizeof(float));
  for (int i = 0; i < 8; ++i) {
    s.pooled[i] = off;
    off += align256((size_t)bh * (s_pad >> (i & 3)) * D * sizeof(float));
  }
  s.items = off; off += align256((size_t)2 * nk * sizeof(int2));
  s.counters = off; off += 256;
  s.total = off;
  return s;
}

template <typename T, int D, int FMT>
int launch_bwd_tc(const void* q, const void* kimg, const void* vimg, const int32_t* mask, const void* out, const float* lse,
                  const void* dout, void* dq, void* dk, void* dv, unsigned char* scratch, int64_t bh, int64_t seq, int mask_cols,
                  float scale, int causal, int32_t* status, cudaStream_t st) {
  constexpr int kSmem = KCfg<D>::SMEM;
  const int nk = (int)cdiv64(seq, 128);
  const int64_t s_pad = (int64_t)nk * 128;
  const Scratch L = scratch_layout(bh, seq, D);
  BwdParams p;
  p.mask = mask; p.kimg = (const unsigned char*)kimg; p.vimg = (const unsigned char*)vimg;
  p.img = make_img_levels(bh, seq, D, 128);
  p.nlse = reinterpret_cast<const float*>(scratch + L.nlse);
  p.ndelta = reinterpret_cast<const float*>(scratch + L.ndelta);
  p.dq = dq;
  for (int i = 0; i < 4; ++i) {
    p.dkp[i] = reinterpret_cast<float*>(scratch + L.pooled[i]);
    p.dvp[i] = reinterpret_cast<float*>(scratch + L.pooled[4 + i]);
  }
  p.items = reinterpret_cast<const int2*>(scratch + L.items);
  int n_entries = 0;
  for (int li = 0; li < 4; ++li) n_entries += (nk + (1 << li) - 1) >> li;
  p.n_entries = n_entries;
  p.status = status; p.seq = seq; p.s_pad = s_pad; p.bh = bh; p.mq = nk; p.mask_cols = mask_cols; p.causal = causal ? 1 : 0;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  int* counters = reinterpret_cast<int*>(scratch + L.counters);
  bwd_stat_kernel<T, D><<<(unsigned)cdiv64(bh * s_pad, 256 / (D / 8) * 4), 256, 0, st>>>(
      (const T*)out, (const T*)dout, lse, reinterpret_cast<float*>(scratch + L.nlse), reinterpret_cast<float*>(scratch + L.ndelta), bh, seq,
      s_pad, reinterpret_cast<int2*>(scratch + L.items), nk, counters,
      ((uintptr_t)out & 15) == 0);
  PSA_CHECK_LAUNCH("psa_legacy_bwd_tcgen05(row statistics)");

  TmapQD maps;
  int rc = encode_tmap_3d(&maps.q, q, 2, FMT == 1, D, seq, bh, 128);
  if (rc != PSA_OK) return rc;
  rc = encode_tmap_3d(&maps.d, dout, 2, FMT == 1, D, seq, bh, 128);
  if (rc != PSA_OK) return rc;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  PSA_REQUIRE(sms > 0, PSA_ERR_CUDA, "psa_legacy_bwd_tcgen05: cannot read the SM count");
  {
    cudaError_t e = cudaFuncSetAttribute(bwd_dq_tc_kernel<D, FMT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    PSA_REQUIRE(e == cudaSuccess, PSA_ERR_CUDA, "psa_legacy_bwd_tcgen05: shared-memory opt-in (%d B) failed: %s", kSmem, cudaGetErrorString(e));
    const int64_t rows = (int64_t)nk * bh;
    p.counter = counters;
    bwd_dq_tc_kernel<D, FMT><<<(unsigned)(rows < sms ? rows : sms), kThreadsBwd, kSmem, st>>>(maps, p);
    PSA_CHECK_LAUNCH("psa_legacy_bwd_tcgen05(dq)");
  }
  {
    cudaError_t e = cudaFuncSetAttribute(bwd_dkdv_tc_kernel<D, FMT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    PSA_REQUIRE(e == cudaSuccess, PSA_ERR_CUDA, "psa_legacy_bwd_tcgen05: shared-memory opt-in (%d B) failed: %s", kSmem, cudaGetErrorString(e));
    const int64_t jobs = (int64_t)n_entries * bh;
    p.counter = counters + 16;
    bwd_dkdv_tc_kernel<D, FMT><<<(unsigned)(jobs < sms ? jobs : sms), kThreadsBwd, kSmem, st>>>(maps, p);
    PSA_CHECK_LAUNCH("psa_legacy_bwd_tcgen05(dk, dv)");
  }
  const int64_t n_main = cdiv64(bh * (s_pad / 8), 256 / (D / 4));
  bwd_fold_kernel<T, D><<<dim3((unsigned)(n_main + (s_pad > seq ? bh : 0)), 2), 256, 0, st>>>(p, (T*)dk, (T*)dv, (int)n_main);
  PSA_CHECK_LAUNCH("psa_legacy_bwd_tcgen05(fold)");
  return PSA_OK;
}

}  // namespace
}  // namespace psa

extern "C" size_t psa_legacy_bwd_scratch_bytes(int64_t bh, int64_t seq, int head_dim) {
  if (bh <= 0 || seq <= 0 || (head_dim != 64 && head_dim != 128)) return 0;
  return psa::scratch_layout(bh, seq, head_dim).total;
}

extern "C" int psa_legacy_bwd_tcgen05(const void* q, const void* kimg, const void* vimg, const int32_t* mask, const void* out,
                                      const float* lse, const void* dout, void* dq, void* dk, void* dv, void* scratch,
                                      size_t scratch_bytes, int64_t bh, int64_t seq, int head_dim, int mask_cols, float sm_scale,
                                      int causal, int dtype, int32_t* status, void* stream) {
  using namespace psa;
  PSA_REQUIRE(q && kimg && vimg && mask && out && lse && dout && dq && dk && dv && scratch, PSA_ERR_ARG,
              "psa_legacy_bwd_tcgen05: null pointer");
  PSA_REQUIRE(dtype == PSA_F16 || dtype == PSA_BF16, PSA_ERR_UNSUPPORTED, "psa_legacy_bwd_tcgen05: f16/bf16 only");
  PSA_REQUIRE(head_dim == 64 || head_dim == 128, PSA_ERR_ARG, "psa_legacy_bwd_tcgen05: head_dim=%d (must be 64 or 128)", head_dim);
  PSA_REQUIRE(bh > 0 && bh < 65536 && seq > 0, PSA_ERR_ARG, "psa_legacy_bwd_tcgen05: bad shape");
  const int64_t nk = cdiv64(seq, 128);
  PSA_REQUIRE(nk <= kMaxBlocks, PSA_ERR_UNSUPPORTED, "psa_legacy_bwd_tcgen05: %lld key blocks, at most %d", (long long)nk, kMaxBlocks);
  PSA_REQUIRE(mask_cols >= nk, PSA_ERR_ARG, "psa_legacy_bwd_tcgen05: mask has %d columns, needs %lld", mask_cols, (long long)nk);
  PSA_REQUIRE(sm_scale > 0.f, PSA_ERR_ARG, "psa_legacy_bwd_tcgen05: sm_scale must be positive");
  PSA_REQUIRE(2 * nk * bh < ((int64_t)1 << 31), PSA_ERR_UNSUPPORTED, "psa_legacy_bwd_tcgen05: too many (head, block) pairs");
  const void* all[] = {q, kimg, vimg, dout, dq, dk, dv};
  for (const void* ptr : all) PSA_REQUIRE(((uintptr_t)ptr & 15) == 0, PSA_ERR_ARG, "psa_legacy_bwd_tcgen05: tensors must be 16-byte aligned");
  PSA_REQUIRE(((uintptr_t)scratch & 255) == 0, PSA_ERR_ARG, "psa_legacy_bwd_tcgen05: scratch must be 256-byte aligned");
  PSA_REQUIRE(scratch_bytes >= psa_legacy_bwd_scratch_bytes(bh, seq, head_dim), PSA_ERR_ARG,
              "psa_legacy_bwd_tcgen05: scratch too small (%zu bytes)", scratch_bytes);
  cudaStream_t st = (cudaStream_t)stream;
  unsigned char* sc = (unsigned char*)scratch;
#define PSA_BWD(TT, FMT)                                                                                                              \
  (head_dim == 64 ? launch_bwd_tc<TT, 64, FMT>(q, kimg, vimg, mask, out, lse, dout, dq, dk, dv, sc, bh, seq, mask_cols, sm_scale, causal, \
                                               status, st)                                                                            \
                  : launch_bwd_tc<TT, 128, FMT>(q, kimg, vimg, mask, out, lse, dout, dq, dk, dv, sc, bh, seq, mask_cols, sm_scale,     \
                                                causal, status, st))
  return dtype == PSA_F16 ? PSA_BWD(__half, 0) : PSA_BWD(__nv_bfloat16, 1);
#undef PSA_BWD
}

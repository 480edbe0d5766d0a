// Multi-level block-sparse flash-attention forward on tcgen05 tensor cores (f16/bf16, block_m = 128).
//
// Persistent CTAs, one per SM (up to 227 KB of shared memory and all 512 TMEM columns each), 12 warps.  A CTA starts with
// query row R = blockIdx.x (R = batch*head * Mq + query block) and claims further rows from a global counter; its roles run the
// rows as ONE continuous stream of 128-token tiles: ring stages, score buffers and barrier phases follow the running tile
// count, so nothing is drained between rows.
//   warp 0      K producer: finds the level segments of the next row's index list (asked into L1 a row ahead) and publishes
//               the row to the other roles, then gathers the selected K blocks of every pyramid level into 128-token tiles,
//               PACKING blocks of different levels into the same tile.  A block is P = block_n/level contiguous pooled rows.
//               From tile images it is ONE linear bulk copy; from row-major tensors one TMA box {64 ch, P rows} per 64-channel
//               slab (128-byte swizzle).  Never multicast.  Lane i stands for columns [4i, 4i+4) of the tile: it computes which
//               block they belong to, reads the list's entry, fetches the block if it starts there, and writes the columns'
//               logit bias (log2 of the level, -inf for columns that do not exist).  It also fetches the row's query tile as
//               soon as the previous row's last Q K^T has read the old one.
//   warp 1      V producer: the same for V, from the published row.  Each ring belongs to ONE warp, which waits for every phase
//               of its stages in order.
//   warps 2, 3  issuers (one thread each): S = Q K^T (operands in shared memory) into one of the TMEM score buffers, and
//               O += P V with P read from TMEM and V read MN-major from its swizzled tile.  A look at a barrier takes the
//               issuing thread 170 to 450 cycles while products run, an MMA 65 to 100: ONE thread for both products was busy all
//               the time (2270 cycles per tile at head_dim 128), with two the tile takes ~1750.
//   warps 4-11  softmax: two groups of four warps, ONE thread per query row.  Group g owns the tiles whose running index
//               is g (mod 2), so no thread needs another thread's partial result and the two warps on a scheduler work on
//               different tiles.  A tile is read from TMEM 32 columns at a time with the next chunk's load in flight: exp2 /
//               sum / round to the element type, written back IN PLACE over the scores.  The exact variant takes the maximum
//               first; its running maximum is only raised when the new one exceeds it by more than 2^8 ("lazy" rescale of the
//               accumulator).  The group that owns a row's last tile finishes the row: it takes the other one's sums from
//               shared memory, reads the accumulators from TMEM and stores 32 bytes per thread and instruction, while the other
//               group works on the next row's first tile.
// What bounds it: ~1750 cycles per tile = a chain of softmax (2000-2500), P V (~720), Q K^T (~720) and their hand-overs over
// three score buffers, against 1024 cycles of the tensor pipe and as many of the ex2 unit; and the 1000 W power cap (at 75600
// tokens the SM clock falls from 1965 to 1500-1700 MHz).  A copy takes its warp ~90 cycles: a tile of 32 blocks of 4 columns (row-major,
// head_dim 128: 64 boxes per operand) takes 5600.
// CODE SIZE counts: an SM holds about 32 KB of instructions, and the twelve warps are in five different places of the code.
// What does not fit is fetched through a cache that up to six SMs share (with 143 KB of unrolled code the softmax of a tile took
// 2120 cycles on an SM with that cache for two, 2990 on one with six).  Hence loops that are not unrolled, waits that are not,
// ring positions that are counted and not divided, one place each where a row is planned and a tile is looked up.
// TMEM (512 columns), head_dim 128: S0/P0 [0,128), S1/P1 [128,256), O of even tiles [256,384), O of odd tiles [384,512);
// head_dim 64: three score buffers [0,384), O of even tiles [384,448), O of odd tiles [448,512).
//
// bf16 calls run the FIXED-REFERENCE variant of the same kernel first: the exponent that the probabilities of a query row
// are taken relative to is the maximum of the row's FIRST tile (the group that owns that tile leaves it in shared memory
// for the other one) and is never raised.  A bf16 probability has the exponent range of fp32, so later scores may exceed the
// reference by dozens of octaves without losing a bit.  (Not so fp16, which takes the exact kernel: a probability below 2^-14
// is subnormal, and with one reference for both groups more of them are - error against 64 bits up to 4 % larger.)  The sum
// stays in fp32.  That removes the maximum pass from every tile but
// the first, the rescaling of the accumulator, so both groups add into ONE accumulator ([384, 384 + head_dim)), a third
// score buffer fits at head_dim 128 as well, and the row's end needs only the two sums.  With the causal rule a row sees a
// key of its first tile or none at all: only the diagonal block hides keys; at level 1 it shows every row at least one, and
// at the other levels it fills half a tile at most, with any other block of the row packed beside it.
// A row whose sum of probabilities exceeds 2^90, is below 2^-60 or is NaN, or whose accumulated values are not all finite
// (probabilities above 1 times values beyond 2^37 can overflow fp32 where probabilities of at most 2^8 do not), sets a guard
// word; the exact kernel is launched right behind on the same stream and returns at once unless that word is set, in which case
// it redoes the call.
//
// Every wait is bounded (mbarriers only, never bar.sync, inside the role loops); on expiry the CTA records PSA_ERR_TIMEOUT in the status word, lets copies in
// flight land, frees its TMEM and returns.
#include <cstddef>
#include <mutex>

#include "psa_common.cuh"
#include "fwd.h"
#include "tc_common.cuh"

namespace psa {

namespace {

constexpr int kSlabBytes = 128 * 128;  // 128 rows x 128 B (64 16-bit channels)
constexpr int kSoftmaxThreads = 256;
constexpr int kThreads = 4 * 32 + kSoftmaxThreads;   // 384
constexpr int kSlotWords = 44;         // per tile: 32 bias words (one per 4 columns), flag, diagonal word, pad, 32 validity bytes

struct TmapPack {
  CUtensorMap q;
  CUtensorMap k[4];   // levels 1, 2, 4, 8
  CUtensorMap v[4];
};

struct TcParams {
  const int32_t* mask;
  void* out;
  int32_t* status;
  int64_t seq_q;
  int64_t n[4];
  int mq, nblocks, bn, tn, width, quirk;
  int total_rows;     // query blocks of all heads: mq * bh
  int* row_counter;   // device word, zero at launch: rows beyond the first one of every CTA are claimed from it
  float scale_log2;   // sm_scale * log2(e)
  // tile-image mode: K/V of all levels pre-laid-out as shared-memory images (one linear bulk copy per block)
  const unsigned char* kimg;
  const unsigned char* vimg;
  ImgLevels img;
  OutScatter scatter;   // n_peers > 0: rows go to the peer that owns the token (plain stores over NVLink)
  float* lse;           // optional log-sum-exp output
  int legacy;           // rows without a visible key give 0 / -inf instead of 0/0
  int causal;           // legacy causal rule on the diagonal block (index rows hold no block beyond the diagonal)
  int* guard;           // fixed-reference variant: set when a row's probabilities left the safe exponent range
  const int* only_if;   // run only if this word is non-zero (the exact kernel as the fixed-reference variant's fallback)
};

// FIXED: the reference exponent of a query row is the maximum of its FIRST tile and is never raised (see the head of the
// file).  No maximum pass after the first tile, no rescaling of the accumulator, hence ONE accumulator for both softmax
// groups and room for a third score buffer.
template <int D, bool FIXED = false, bool CAUSAL = false> struct Cfg {
  static constexpr int SLABS = D / 64;
  static constexpr int NK = D == 64 ? 4 : 3;                 // K-tile ring
  static constexpr int NV = D == 64 ? 4 : FIXED ? 3 : 2;     // V-tile ring
  // Score buffers in TMEM.  At D = 128 the two accumulators leave room for two; at D = 64 for three, and the third one
  // lets Q K^T run two tiles ahead of P V, so that a softmax group finds its next scores ready when it is done with a tile.
  static constexpr int NSB = (D == 64 || FIXED) ? 3 : 2;
  static constexpr int O_BASE = NSB * 128;          // first TMEM column of the accumulators
  static constexpr int O_STRIDE = FIXED ? 0 : (NSB == 3 ? 64 : 128);
  // Two score buffers: one thread issues both products, in the order QK0 QK1 PV0 QK2 PV1 ..., so that Q K^T follows the product
  // that frees its buffer at once.  Three: one thread for each, neither of which ever waits behind the other's barriers.
  static constexpr bool ONE_ISSUER = NSB == 2;
  // A whole tile's MMAs one after the other in the code, or as a loop.  Unrolled, the eight of P V take 718 cycles instead of 880 and those
  // of Q K^T 717 instead of 815 at head_dim 128 (12x32760x128 629 -> 620 us, fp16 12x16384x128 247 -> 239); where the loops of a tile
  // fill the instruction cache already they cost more than that (causal 14x32768x128 1779 -> 1930 us), and at head_dim 64 the softmax is the bound
  // (48x17776x64 694 -> 701 us).
  static constexpr bool UNROLL_MMA = D == 128 && !CAUSAL;
  // The second pass of a full tile, two chunks at a time in a loop or all four in the code.  The loop is the better one
  // (exact kernel, 16 x 9973 x 128 168 against 205 us, 6 x 32760 x 128 387 / 438, causal 8 x 16384 x 64 318 / 344) except in the exact kernel at
  // head_dim 64 without the causal rule, where three score buffers keep both groups in this pass (6 x 32760 365 / 311, 8 x 20011 704 / 610).
  static constexpr bool UNROLL_EXP = D == 64 && !FIXED && !CAUSAL;
  // Bias words of tile t are written when the scores of tile t-NK are complete; these were issued behind P V of tile
  // t-NK-NSB, whose softmax is therefore done with its words.
  static constexpr int SLOTS = NK + NSB;
  static constexpr int TILE_BYTES = SLABS * kSlabBytes;
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_K = OFF_Q + TILE_BYTES;
  static constexpr int OFF_V = OFF_K + NK * TILE_BYTES;
  static constexpr int OFF_BIAS = OFF_V + NV * TILE_BYTES;
  // exchange of the softmax groups: a row's sum of one of them and the reference exponents of two rows (FIXED), or (sum, maximum)
  static constexpr int OFF_XCH = OFF_BIAS + SLOTS * kSlotWords * 4;
  static constexpr int OFF_CTRL = OFF_XCH + (FIXED ? 3 : 2) * 128 * 4;
};

// A query row as the K producer publishes it: the row (>= total_rows: no more rows), the first four separators of its index list,
// its tiles.
struct RowSlot { int R, sep0, sep1, sep2, sep3, n_tiles, last_cols; };

template <class C> struct Ctrl {
  uint64_t k_full[C::NK], v_full[C::NV];
  // "Scores of tile t complete": its K stage may be refilled and its softmax group may start.  Two barriers per stage, used by
  // alternate fills: a group owns every other tile, and a parity wait must see every phase of its barrier in order.
  uint64_t k_empty[2 * C::NK];
  uint64_t v_empty[C::NV];      // "P V of tile t complete": its V stage may be refilled, its score buffer overwritten
  uint64_t pv_done[C::O_STRIDE ? 2 : 1], q_full, mref_full[2];
  // probabilities of a tile written: two barriers per group, used by the group's alternate tiles.  With three score
  // buffers a group can finish its NEXT tile before the issuer has seen this one (P V also waits for the V tile), and a
  // parity wait must never fall two phases behind its barrier.
  uint64_t p_full[4];
  uint64_t row_ready[4], row_done[4], o_free;   // hand-over of query rows between the roles of a persistent CTA
  uint64_t xch_full;                            // one group's sums of a row, for the group that finishes the row
  RowSlot row[4];
  uint32_t tmem_base;
  int abort_flag;
};

template <int D, bool FIXED, bool CAUSAL> constexpr int smem_bytes() {
  using C = Cfg<D, FIXED, CAUSAL>;
  return C::OFF_CTRL + (int)sizeof(Ctrl<C>);
}

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int FMT> __device__ __forceinline__ uint32_t pack2(float a, float b);
template <> __device__ __forceinline__ uint32_t pack2<1>(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t pack2<0>(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

// 32 bytes of an output row (32-byte aligned)
__device__ __forceinline__ void store32(void* dst, const uint32_t* v) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
               "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

// A query row's stream of gathered columns: level li's blocks start at column col[li] (its blocks one after the other, then the
// extra blocks of a narrow level), list entry seg[li] is the first one.  From that any lane finds the block of any column by
// itself, so a row needs no table of its blocks in shared memory.
struct RowPlan {
  const int32_t* list;
  int R, n_tiles, tokens, last_cols, last_li;
  int seg1, seg2, seg3, cnt0, cnt1, cnt2, cnt3, col1, col2, col3;
};
__device__ __forceinline__ int pick4(int i, int a, int b, int c, int d) { return i < 2 ? (i == 0 ? a : b) : (i == 2 ? c : d); }

// s0..s3: positions of the first four separators (the list's length where there is none).  A row that ended early leaves the
// later levels empty.
__device__ __forceinline__ void plan_from_separators(RowPlan& c, const TcParams& p, int s0, int s1, int s2, int s3) {
  c.list = p.mask + (int64_t)c.R * p.width;
  c.seg1 = s0 + 1; c.seg2 = s1 + 1; c.seg3 = s2 + 1;
  c.cnt0 = s0; c.cnt1 = max(s1 - c.seg1, 0); c.cnt2 = max(s2 - c.seg2, 0); c.cnt3 = max(s3 - c.seg3, 0);
  const int cnt[4] = {c.cnt0, c.cnt1, c.cnt2, c.cnt3};
  int tokens = 0, col[4];
  c.last_li = 0;
#pragma unroll
  for (int li = 0; li < 4; ++li) {
    const int P = p.bn >> li;
    const int items = cnt[li] + (p.quirk && P < p.tn && cnt[li] >= 2 ? p.tn / P - 2 : 0);
    if (items > 0) c.last_li = li;
    col[li] = tokens;
    tokens += items * P;
  }
  c.col1 = col[1]; c.col2 = col[2]; c.col3 = col[3];
  c.tokens = tokens;
  c.n_tiles = (tokens + 127) >> 7;
  c.last_cols = tokens - (c.n_tiles - 1) * 128;
}

// Columns [4 lane, 4 lane + 4) of tile t: the block they belong to, whether it starts there, and where in it they lie.  (Blocks are at
// least 4 wide, and each starts at a multiple of its own width.)
struct LaneColumns {
  int li, blk, inside, col;
  bool in, start, extra, pad;      // in: the tile has these columns; extra: block of a narrow level added for reference compatibility
};
// The row's last tile is filled up: K to a multiple of 32 columns, the chunk of the softmax, with copies of the row's last block (bias
// -inf: a score that is not finite enters no row that did not select it), V to a multiple of 16, the step of its product, with zeros
// (a probability of 0 times a copied value that is not finite would be NaN, where the block's own product may be infinite or 0).
__device__ __forceinline__ int tile_columns(const RowPlan& c, int t, int multiple) {
  return t == c.n_tiles - 1 ? (c.last_cols + multiple - 1) & -multiple : 128;
}
__device__ __forceinline__ LaneColumns lane_columns(const RowPlan& c, int t, int cols, int lane, int bn_shift) {
  LaneColumns b;
  b.col = lane * 4;
  const int x = t * 128 + b.col;
  b.in = b.col < cols;
  b.pad = x >= c.tokens;
  b.li = b.pad ? c.last_li : (x >= c.col1) + (x >= c.col2) + (x >= c.col3);
  const int off = x - (b.pad ? c.tokens : pick4(b.li, 0, c.col1, c.col2, c.col3));
  const int shift = bn_shift - b.li, cnt = pick4(b.li, c.cnt0, c.cnt1, c.cnt2, c.cnt3), e = b.pad ? cnt - 1 : off >> shift;
  b.inside = off & ((1 << shift) - 1);
  b.start = b.in && b.inside == 0;
  b.extra = e >= cnt;
  b.blk = 2 + e - cnt;
  if (b.in && !b.extra) b.blk = __ldg(c.list + pick4(b.li, 0, c.seg1, c.seg2, c.seg3) + e);
  return b;
}

// One block into its columns of a tile.  A block number that no list should hold is held inside the operand.
template <int D, bool IMG>
__device__ __forceinline__ void fetch_block(const TcParams& p, const LaneColumns& b, int bh, uint32_t tile_a, uint32_t bar_a,
                                            const unsigned char* img, uint64_t map0) {
  constexpr int SLABS = D / 64;
  const int P = p.bn >> b.li;
  const int blk = (unsigned)b.blk < (unsigned)p.nblocks ? b.blk : p.nblocks - 1;
  if (IMG) {
    const unsigned char* src = img + p.img.off[b.li] + (((int64_t)bh * p.img.groups[b.li] + ((blk * P) >> 3)) * SLABS << 10);
    tc::bulk_load_a(tile_a + (b.col >> 3) * (SLABS * 1024), src, (uint32_t)(P * D * 2), bar_a);
  } else {
#pragma unroll
    for (int sl = 0; sl < SLABS; ++sl)
      tc::tma_load_3d_a(tile_a + sl * kSlabBytes + b.col * 128, map0 + (uint64_t)b.li * sizeof(CUtensorMap), bar_a, sl * 64, blk * P, bh);
  }
}

// A ring of N stages: the stage of the running tile and how often it was filled before.
template <int N> struct Ring {
  int stage = 0, fill = 0;
  __device__ __forceinline__ void next(int by = 1) {
    stage += by;
    if (stage >= N) { stage -= N; ++fill; }
  }
};

// Bounded spins.  The roles that feed the tensor pipe look again at once: a parked try_wait was seen to resume several hundred
// cycles after its phase completed.  Two barriers are looked at together (a look takes ~170 cycles or more, complete or not).
__device__ __forceinline__ bool spin_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
#pragma unroll 1
  for (uint32_t it = 0; it < (1u << 24); ++it) {
    if (tc::mbar_test_wait_a(bar, parity)) return true;
    if ((it & 255) == 255 && *abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}
__device__ __forceinline__ bool spin_wait2(uint32_t bar0, uint32_t parity0, uint32_t bar1, uint32_t parity1, volatile int* abort_flag) {
  if (bar1 == 0) return spin_wait(bar0, parity0, abort_flag);
#pragma unroll 1
  for (uint32_t it = 0; it < (1u << 24); ++it) {
    const bool a = tc::mbar_test_wait_a(bar0, parity0), b = tc::mbar_test_wait_a(bar1, parity1);
    if (a && b) return true;
    if ((it & 255) == 255 && *abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}

// Logit bias of the four columns of group q, column by column: absent ones (validity bits, looked at only where the tile has
// any) and, on the causal diagonal, those in [hide_lo, hide_hi) are hidden.
template <bool CAUSAL>
__device__ __forceinline__ float4 column_bias(const float* bias, const unsigned char* valid, int q, int hide_lo, int hide_hi) {
  const float b = bias[q];
  const int bits = valid[q];
  float4 ba = make_float4(bits & 1 ? b : -INFINITY, bits & 2 ? b : -INFINITY, bits & 4 ? b : -INFINITY, bits & 8 ? b : -INFINITY);
  if (CAUSAL) {
    const int c = 4 * q;
    if (c >= hide_lo && c < hide_hi) ba.x = -INFINITY;
    if (c + 1 >= hide_lo && c + 1 < hide_hi) ba.y = -INFINITY;
    if (c + 2 >= hide_lo && c + 2 < hide_hi) ba.z = -INFINITY;
    if (c + 3 >= hide_lo && c + 3 < hide_hi) ba.w = -INFINITY;
  }
  return ba;
}

// IMG = true: K/V tiles use the image layout [8-row group][slab][8 rows][128 B] and are filled by linear bulk copies from
// the tile-image buffers; IMG = false: [slab][128 rows][128 B] filled by tensor-map TMA boxes from row-major tensors.
template <int D, int FMT, bool IMG, bool CAUSAL, bool FIXED>
__global__ void __launch_bounds__(kThreads, 1) psa_fwd_tc_kernel(const __grid_constant__ TmapPack maps, const TcParams p) {
  using C = Cfg<D, FIXED, CAUSAL>;
  using Ctl = Ctrl<C>;
  if (p.only_if && *p.only_if == 0) return;
  extern __shared__ __align__(1024) unsigned char smem[];
  if (tc::smem_u32(smem) & 1023) {          // the swizzled tiles need it; nothing has been started yet
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, PSA_ERR_CUDA);
    return;
  }
  unsigned char* sQ = smem + C::OFF_Q;
  unsigned char* sK = smem + C::OFF_K;
  unsigned char* sV = smem + C::OFF_V;
  // [slot][32 bias words, one per 4 columns | flag: look at single columns | diagonal block (causal) | pad | 32 validity bytes]
  float* sBias = reinterpret_cast<float*>(smem + C::OFF_BIAS);
  float* sXch = reinterpret_cast<float*>(smem + C::OFF_XCH);
  Ctl* ctl = reinterpret_cast<Ctl*>(smem + C::OFF_CTRL);
  volatile int* abort_flag = &ctl->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // ---------------------------------------------------------------- setup (once per CTA)
  if (threadIdx.x == 0) {
    for (int i = 0; i < C::NK; ++i) {
      tc::mbar_init(&ctl->k_full[i], 1);
      tc::mbar_init(&ctl->k_empty[2 * i], 1); tc::mbar_init(&ctl->k_empty[2 * i + 1], 1);
    }
    for (int i = 0; i < C::NV; ++i) {
      tc::mbar_init(&ctl->v_full[i], 1);
      tc::mbar_init(&ctl->v_empty[i], 1);
    }
    ctl->abort_flag = 0;
    tc::fence_mbar_init();
  } else if (threadIdx.x == 32) {
    for (int i = 0; i < 4; ++i) tc::mbar_init(&ctl->p_full[i], 4);   // one arrival per softmax warp of the group
    for (int i = 0; i < (C::O_STRIDE ? 2 : 1); ++i) tc::mbar_init(&ctl->pv_done[i], 1);
    tc::mbar_init(&ctl->q_full, 1);
    for (int i = 0; i < 2; ++i) tc::mbar_init(&ctl->mref_full[i], 4);     // the four warps of the group that owns a row's first tile
    tc::mbar_init(&ctl->o_free, 4);        // ... that finishes the row
    tc::mbar_init(&ctl->xch_full, 4);      // ... of the other one
    tc::fence_mbar_init();
  } else if (threadIdx.x == 64) {
    for (int i = 0; i < 4; ++i) {
      tc::mbar_init(&ctl->row_ready[i], 1);
      tc::mbar_init(&ctl->row_done[i], 11);   // eight softmax warps, both issuers, the V producer
    }
    tc::fence_mbar_init();
  }
  if (warp == 3) {
    tc::tmem_alloc(&ctl->tmem_base, 512);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;

  // A CTA is persistent: it starts with query row R = blockIdx.x (R = bh * mq + m) and claims further rows from a global
  // counter (SMs do not all run at the same speed, so a fixed split would leave the fast ones idle at the end); its
  // roles run the rows as one continuous stream of tiles.  Ring stages, score buffers and barrier phases follow
  // the running tile count, so the producers plan and prefetch the next row while the MMAs and the softmax of
  // the current row are still in flight, and the first scores of the next row are computed under the epilogue.
  if (warp == 0) {
    // ============================================================ K producer, query tiles, planning of the rows
    const uint32_t ctl_a = tc::smem_u32(ctl);
    const uint32_t k_full_a = ctl_a + (uint32_t)offsetof(Ctl, k_full), k_empty_a = ctl_a + (uint32_t)offsetof(Ctl, k_empty);
    const uint32_t sK_a = tc::smem_u32(sK);
    const uint64_t kmap0 = reinterpret_cast<uint64_t>(&maps.k[0]);
    const int n0 = (int)p.n[0], n1 = (int)p.n[1], n2 = (int)p.n[2], n3 = (int)p.n[3];
    const int bn_shift = 31 - __clz(p.bn);
    int claim = (int)blockIdx.x;                 // the next row; lane 0's counts
    bool ok = true;
    // A row's index list is asked into L1 (the 28 KB beside the shared memory, through which little else passes) long before it is
    // looked at.
    auto prefetch_list = [&](int R_n) {
      if (R_n >= p.total_rows) return;
      const int32_t* list = p.mask + (int64_t)R_n * p.width;
      for (int i = lane * 32; i < p.width + 31; i += 32 * 32) {      // one request per 128 bytes
        const int32_t* at = list + (i < p.width ? i : p.width - 1);
        asm volatile("prefetch.global.L1 [%0];" ::"l"(at));
      }
    };
    // Take the claimed row, find its level segments (the first four separators of its list), publish it, claim the row after it
    // and ask for that one's list.
    auto plan_row = [&](int rit_n, RowPlan& c) -> bool {
      c.R = __shfl_sync(0xffffffffu, claim, 0);
      const int rs = rit_n & 3;
      int s0 = p.width, s1 = p.width, s2 = p.width, s3 = p.width;
      if (c.R < p.total_rows) {
        if (lane == 0) claim = (int)gridDim.x + atomicAdd(p.row_counter, 1);
        const int32_t* list = p.mask + (int64_t)c.R * p.width;
        int found = 0;
#pragma unroll 1
        for (int i0 = 0; i0 < p.width && found < 4; i0 += 64) {      // (lists are in L1; the fourth separator ends the search)
          const int v0 = i0 + lane < p.width ? __ldg(list + i0 + lane) : 0;
          const int v1 = i0 + 32 + lane < p.width ? __ldg(list + i0 + 32 + lane) : 0;
          const unsigned b0 = __ballot_sync(0xffffffffu, v0 == -1), b1 = __ballot_sync(0xffffffffu, v1 == -1);
          unsigned long long bits = (unsigned long long)b1 << 32 | b0;
#pragma unroll 1
          while (bits && found < 4) {
            const int at = i0 + __ffsll(bits) - 1;
            if (found == 0) s0 = at; else if (found == 1) s1 = at; else if (found == 2) s2 = at; else s3 = at;
            ++found;
            bits &= bits - 1;
          }
        }
        plan_from_separators(c, p, s0, s1, s2, s3);
        prefetch_list(__shfl_sync(0xffffffffu, claim, 0));
      }
      // Publish the row (or "no more rows") to the other roles.  The slot was last used four rows ago: wait until that row is
      // finished.
      if (rit_n >= 4) {
        const bool good = tc::mbar_wait(&ctl->row_done[rs], ((rit_n >> 2) - 1) & 1, abort_flag);
        if (!__all_sync(0xffffffffu, good)) return false;
      }
      if (lane == 0) {
        volatile RowSlot& s = ctl->row[rs];
        s.R = c.R;
        s.sep0 = s0; s.sep1 = s1; s.sep2 = s2; s.sep3 = s3;
        s.n_tiles = c.n_tiles; s.last_cols = c.last_cols;
        __threadfence_block();
        tc::mbar_arrive(&ctl->row_ready[rs]);
      }
      __syncwarp();
      return true;
    };
    RowPlan cur = {}, nxt = {};      // before the first row: one without tiles, in which the first is planned
    Ring<C::NK> ring;                // stage of the next tile
    int slot = 0;                    // its bias words
    int last_empty = -1, last_phase = 0;      // "scores complete" barrier of the last tile so far
#pragma unroll 1
    for (int rit = -1; ok && cur.R < p.total_rows; ++rit) {
      const int m = cur.R % p.mq, bh = cur.R / p.mq;
      const int n_tiles = cur.n_tiles;
      const int plan_step = n_tiles < C::NK ? n_tiles : C::NK;   // where the next row is planned: the ring is full by then
      // The query tile replaces the previous row's one as soon as the scores of that row's last tile are complete.
      bool q_pending = n_tiles > 0, planned = false, have = false;
      const int q_empty = last_empty, q_phase = last_phase;
      int kt = 0;
      uint32_t spins = 0;
      LaneColumns b;                   // of the next tile, looked up before its stage is free
#pragma unroll 1
      while (ok && (kt < n_tiles || !planned || q_pending)) {
        bool progressed = false;
        if (!have && kt < n_tiles) {
          b = lane_columns(cur, kt, tile_columns(cur, kt, 32), lane, bn_shift);
          have = true;
        }
        if (q_pending) {
          const bool ready = q_empty < 0 || tc::mbar_test_wait_a(k_empty_a + q_empty * 8, q_phase);
          if (__all_sync(0xffffffffu, ready)) {
            if (lane == 0) {
              for (int s = 0; s < C::SLABS; ++s) tc::tma_load_3d(sQ + s * kSlabBytes, &maps.q, &ctl->q_full, s * 64, m * 128, bh);
              tc::mbar_arrive_expect_tx(&ctl->q_full, C::TILE_BYTES);
            }
            q_pending = false;
            progressed = true;
          }
        }
        if (kt < n_tiles) {
          // fill number f of the stage waits for the scores of fill f-1 (barrier and phase of that fill)
          const bool ready = ring.fill == 0 || tc::mbar_test_wait_a(k_empty_a + (ring.stage * 2 + ((ring.fill - 1) & 1)) * 8, ((ring.fill - 1) >> 1) & 1);
          if (__all_sync(0xffffffffu, ready)) {
            const uint32_t bar_a = k_full_a + ring.stage * 8;
            if (b.start) fetch_block<D, IMG>(p, b, bh, sK_a + ring.stage * C::TILE_BYTES, bar_a, p.kimg, kmap0);
            // logit bias of this lane's four columns
            float* words = sBias + slot * kSlotWords;
            const int nvalid = pick4(b.li, n0, n1, n2, n3) - b.blk * (p.bn >> b.li) - b.inside;
            float bias2 = (float)b.li;
            if (b.extra) bias2 += log2f((float)(pick4(b.li, cur.cnt0, cur.cnt1, cur.cnt2, cur.cnt3) >> 1));
            words[lane] = b.in && !b.pad && nvalid > 0 ? bias2 : -INFINITY;
            const bool diag = CAUSAL && b.in && b.blk == m && !b.pad && !b.extra;
            // a block that ends inside a group of 4 columns, the diagonal block of a causal row, or the end of the row's tokens
            // 16 columns or more before the tile's makes the tile take the per-column path of the softmax
            const unsigned odd_lanes = __ballot_sync(0xffffffffu, (b.in && !b.pad && ((nvalid > 0 && nvalid < 4) || diag)) ||
                                                                      (kt == n_tiles - 1 && cur.last_cols <= 112));
            if (odd_lanes) reinterpret_cast<unsigned char*>(words + 36)[lane] = (unsigned char)(nvalid > 0 && nvalid < 4 ? (1 << nvalid) - 1 : 15);
            if (lane == 0) reinterpret_cast<int*>(words)[32] = odd_lanes != 0;
            if (CAUSAL) {
              const unsigned diag_start = __ballot_sync(0xffffffffu, diag && b.start);
              if (diag_start ? diag && b.start : lane == 0) reinterpret_cast<int*>(words)[33] = diag_start ? (b.li << 8 | lane * 4) : -1;
            }
            // the bias of this tile must be complete before the tile is announced: the softmax warps read it once the
            // scores are ready, and "scores ready" follows "K tile full" through the MMA issuer
            __syncwarp();
            if (lane == 0) tc::mbar_arrive_expect_tx_a(bar_a, (uint32_t)(tile_columns(cur, kt, 32) * D * 2));
            last_empty = ring.stage * 2 + (ring.fill & 1);
            last_phase = (ring.fill >> 1) & 1;
            ring.next();
            slot = slot + 1 == C::SLOTS ? 0 : slot + 1;
            ++kt;
            have = false;
            progressed = true;
          }
        }
        if (!planned && kt >= plan_step) {
          ok = plan_row(rit + 1, nxt);
          planned = true;
          progressed = true;
        }
        if (!progressed) __nanosleep(40);      // (the ring holds three or four tiles; a spinning warp takes issue slots and power)
        if (progressed) {
          spins = 0;
        } else if (++spins > (1u << 24) || ((spins & 255) == 255 && *abort_flag)) {
          *abort_flag = 1;
          ok = false;
        }
      }
      cur = nxt;
    }
  } else if (warp == 1) {
    // ============================================================ V producer
    const uint32_t ctl_a = tc::smem_u32(ctl);
    const uint32_t v_full_a = ctl_a + (uint32_t)offsetof(Ctl, v_full), v_empty_a = ctl_a + (uint32_t)offsetof(Ctl, v_empty);
    const uint32_t sV_a = tc::smem_u32(sV);
    const uint64_t vmap0 = reinterpret_cast<uint64_t>(&maps.v[0]);
    const int bn_shift = 31 - __clz(p.bn);
    Ring<C::NV> ring;
    bool ok = true;
    for (int rit = 0; ok; ++rit) {
      const int rs = rit & 3;
      ok = tc::mbar_wait(&ctl->row_ready[rs], (rit >> 2) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      const volatile RowSlot& s = ctl->row[rs];
      RowPlan cur;
      cur.R = s.R;
      if (cur.R >= p.total_rows) break;
      plan_from_separators(cur, p, s.sep0, s.sep1, s.sep2, s.sep3);
      const int n_tiles = cur.n_tiles, bh = cur.R / p.mq;
#pragma unroll 1
      for (int vt = 0; vt < n_tiles; ++vt) {
        const int cols = tile_columns(cur, vt, 1), zero_rows = tile_columns(cur, vt, 16) - cols;
        const LaneColumns b = lane_columns(cur, vt, cols, lane, bn_shift);
        // fill number f of the stage waits for P V of fill f-1
        if (ring.fill > 0) ok = tc::mbar_wait_a(v_empty_a + ring.stage * 8, (ring.fill - 1) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const uint32_t bar_a = v_full_a + ring.stage * 8;
        if (b.start) fetch_block<D, IMG>(p, b, bh, sV_a + ring.stage * C::TILE_BYTES, bar_a, p.vimg, vmap0);
        if (zero_rows) {       // 4 to 12 rows of 128 bytes per slab (whole rows: the swizzle moves nothing out of them)
          unsigned char* tile = sV + ring.stage * C::TILE_BYTES;
#pragma unroll 1
          for (int i = lane; i < zero_rows * C::SLABS * 8; i += 32) {
            const int sl = (i >> 3) % C::SLABS, row = cols + (i >> 3) / C::SLABS;
            const int at = IMG ? (row >> 3) * (C::SLABS * 1024) + sl * 1024 + (row & 7) * 128 : sl * kSlabBytes + row * 128;
            *reinterpret_cast<uint4*>(tile + at + (i & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
          }
          tc::fence_proxy_async();      // the tensor pipe reads them
          __syncwarp();
        }
        if (lane == 0) tc::mbar_arrive_expect_tx_a(bar_a, (uint32_t)(cols * D * 2));
        __syncwarp();
        ring.next();
      }
      __syncwarp();       // every lane has read the row's slot, also of a row without tiles, before it is handed back
      if (ok && lane == 0) tc::mbar_arrive(&ctl->row_done[rs]);
    }
  } else if (warp < 4) {
    // ============================================================ issuers: warp 2 S = Q K^T, warp 3 O += P V
    if (lane == 0) {
      bool ok = true;
      // ready-made descriptors: per tile only the stage offset is added, per MMA only an immediate
      const uint32_t idesc_qk = tc::make_idesc(FMT, 128, 128, 0, 0), idesc_pv = tc::make_idesc(FMT, 128, D, 0, 1);
      // image layout: 8-row groups are SLABS KiB apart and the slabs of a group follow each other
      constexpr uint32_t kGroupStride = IMG ? C::SLABS * 1024 : 1024;
      constexpr uint32_t kSlabStride = IMG ? 1024 : kSlabBytes;
      const uint64_t qdesc = tc::make_smem_desc(tc::smem_u32(sQ), 16, 1024);
      const uint64_t kdesc0 = tc::make_smem_desc(tc::smem_u32(sK), 16, kGroupStride);
      const uint64_t vdesc0 = tc::make_smem_desc(tc::smem_u32(sV), kSlabStride, kGroupStride);
      const uint32_t ctl_a = tc::smem_u32(ctl);
      const uint32_t k_full_a = ctl_a + (uint32_t)offsetof(Ctl, k_full), k_empty_a = ctl_a + (uint32_t)offsetof(Ctl, k_empty);
      const uint32_t v_full_a = ctl_a + (uint32_t)offsetof(Ctl, v_full), v_empty_a = ctl_a + (uint32_t)offsetof(Ctl, v_empty);
      const uint32_t p_full_a = ctl_a + (uint32_t)offsetof(Ctl, p_full), pv_done_a = ctl_a + (uint32_t)offsetof(Ctl, pv_done);
      Ring<C::NK> kring;
      Ring<C::NV> vring;       // of the next P V; in the thread that issues Q K^T, of the tile NSB before the next one
      int qk_buf = 0, pv_buf = 0, lead = C::NSB, pv_tile = 0;
      auto issue_qk = [&](bool last, int last_cols) -> bool {
        // the K tile is there, and P V of the tile NSB before is done with the probabilities that lie in this score buffer (issued
        // by this thread: the tensor pipe runs in issue order)
        if (!spin_wait2(k_full_a + kring.stage * 8, kring.fill & 1, !C::ONE_ISSUER && lead == 0 ? v_empty_a + vring.stage * 8 : 0u,
                        vring.fill & 1, abort_flag))
          return false;
        tc::tc_fence_after();
        uint64_t kdesc = kdesc0 + (uint64_t)(kring.stage * (C::TILE_BYTES >> 4)), qd = qdesc;
        const uint32_t idesc = last ? tc::make_idesc(FMT, 128, (last_cols + 31) & ~31, 0, 0) : idesc_qk;
        const uint32_t tSb = tmem + qk_buf * 128;
#pragma unroll(C::UNROLL_MMA ? C::SLABS : 1)
        for (int sl = 0; sl < C::SLABS; ++sl) {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) tc::umma_ss(tSb, qd + ks * 2, kdesc + ks * 2, idesc, (uint32_t)(sl + ks));
          qd += kSlabBytes >> 4;
          kdesc += kSlabStride >> 4;
        }
        tc::umma_commit_a(k_empty_a + (kring.stage * 2 + (kring.fill & 1)) * 8);   // scores ready, K tile may be refilled
        kring.next();
        qk_buf = qk_buf + 1 == C::NSB ? 0 : qk_buf + 1;
        if (!C::ONE_ISSUER) {
          if (lead > 0) --lead; else vring.next();
        }
        return true;
      };
      auto issue_pv = [&](int t, int n_tiles, int last_cols) -> bool {
        const int b = pv_tile & 1;
        if (!spin_wait2(p_full_a + (b * 2 + ((pv_tile >> 1) & 1)) * 8, (pv_tile >> 2) & 1, v_full_a + vring.stage * 8, vring.fill & 1, abort_flag))
          return false;
        tc::tc_fence_after();
        uint64_t vdesc = vdesc0 + (uint64_t)(vring.stage * (C::TILE_BYTES >> 4));
        uint32_t tP = tmem + pv_buf * 128;                           // probabilities overwrite the scores they came from
        const uint32_t tO = tmem + C::O_BASE + b * C::O_STRIDE;      // two accumulators: even and odd tiles separately
        uint32_t accumulate = t > (FIXED ? 0 : 1) ? 1u : 0u;
        if (C::UNROLL_MMA && t < n_tiles - 1) {
          tc::umma_ts(tO, tP, vdesc, idesc_pv, accumulate);
#pragma unroll
          for (int ks = 1; ks < 8; ++ks) tc::umma_ts(tO, tP + ks * 8, vdesc + (uint64_t)(ks * ((2 * kGroupStride) >> 4)), idesc_pv, 1u);
        } else {
          const int steps = t == n_tiles - 1 ? (last_cols + 15) >> 4 : 8;      // of 16 keys
#pragma unroll 1
          for (int ks = 0; ks < steps; ++ks) {
            tc::umma_ts(tO, tP, vdesc, idesc_pv, accumulate);
            accumulate = 1u;
            tP += 8;
            vdesc += (2 * kGroupStride) >> 4;
          }
        }
        tc::umma_commit_a(v_empty_a + vring.stage * 8);   // V tile may be refilled, score buffer may be overwritten
        // "accumulator final", for the last product of the row; with two accumulators for the last one of each.  Three score
        // buffers and two accumulators: every product (the softmax waits for it before it rescales the accumulator).
        if (FIXED) {
          if (t == n_tiles - 1) tc::umma_commit_a(pv_done_a);
        } else if (C::NSB == 3 || t >= n_tiles - 2) tc::umma_commit_a(pv_done_a + b * 8);
        vring.next();
        ++pv_tile;
        pv_buf = pv_buf + 1 == C::NSB ? 0 : pv_buf + 1;
        return true;
      };
      const bool does_qk = C::ONE_ISSUER ? warp == 3 : warp == 2, does_pv = warp == 3;
      int q_rows = 0;
#pragma unroll 1
      for (int rit = 0; ok; ++rit) {
        const int rs = rit & 3;
        ok = tc::mbar_wait(&ctl->row_ready[rs], (rit >> 2) & 1, abort_flag);
        const volatile RowSlot& s = ctl->row[rs];
        if (!ok || s.R >= p.total_rows) break;
        const int n_tiles = s.n_tiles, last_cols = s.last_cols;
        if (n_tiles > 0) {
          if (does_qk) ok = tc::mbar_wait(&ctl->q_full, q_rows & 1, abort_flag);
          int qk = 0;
          if (does_qk)
            for (; ok && qk < n_tiles && qk < (C::ONE_ISSUER ? C::NSB : n_tiles); ++qk) ok = issue_qk(qk == n_tiles - 1, last_cols);
          // the accumulators are overwritten by this row's first products: the previous row's epilogue must have read them
          if (ok && does_pv && q_rows > 0) ok = tc::mbar_wait(&ctl->o_free, (q_rows - 1) & 1, abort_flag);
          if (does_pv)
#pragma unroll 1
            for (int t = 0; ok && t < n_tiles; ++t) {
              ok = issue_pv(t, n_tiles, last_cols);
              if (C::ONE_ISSUER && ok && qk < n_tiles) { ok = issue_qk(qk == n_tiles - 1, last_cols); ++qk; }
            }
          ++q_rows;
        }
        if (ok) tc::mbar_arrive(&ctl->row_done[rs]);
      }
    }
  } else {
    // ============================================================ softmax / epilogue
    // Two groups of four warps, one thread per query row.  Group g owns the tiles whose running index is g (mod 2), so the two
    // warps that share a scheduler are in different phases of different tiles and no thread ever needs its neighbour's partial
    // result.  The group that owns a row's LAST tile finishes the row (a warp may read any column of its own TMEM lanes); the
    // other one, which owns the next row's first tile, leaves its sums in shared memory and goes straight on to that.
    // Both first wait until the row before has been read out of the accumulators (o_free): what was exchanged for it has been
    // read by then, and every barrier below is at most one phase ahead of any of its waiters.
    const int quarter = warp & 3;                 // TMEM lanes this warp may touch
    const int g = (warp - 4) >> 2;                // softmax group = tile parity = score buffer = accumulator
    const int r = quarter * 32 + lane;            // row inside the query block
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const uint32_t tO = tmem + C::O_BASE + g * C::O_STRIDE + lane_base;   // my accumulator
    const uint32_t tO_other = tmem + C::O_BASE + (g ^ 1) * C::O_STRIDE + lane_base;
    const float2 scale2 = make_float2(p.scale_log2, p.scale_log2);
    bool ok = true;
    int g0 = 0, ne = 0, pv_rows = 0;               // ne: rows with tiles before this one
    // of this group's next tile: K stage, score buffer, bias words; its number among the group's tiles
    Ring<C::NK> ring;
    ring.next(g);
    int buf = g, slot = g, mine = 0;
    float* sMref = sXch + 128;                    // fixed reference: the exponents of two rows, behind the sums
    constexpr float kSumMax = 1.2379400e27f, kSumMin = 8.6736174e-19f;      // 2^90, 2^-60
#pragma unroll 1
    for (int rit = 0; ok; ++rit) {
      const int rslot = rit & 3;
      ok = tc::mbar_wait(&ctl->row_ready[rslot], (rit >> 2) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      const volatile RowSlot& row = ctl->row[rslot];
      const int R = row.R;
      if (R >= p.total_rows) break;
      const int m = R % p.mq, bh = R / p.mq;
      const int n_tiles = row.n_tiles, last_cols = row.last_cols;
      float m_run = -INFINITY, l_run = 0.f;
      const int first = ((g0 & 1) == g) ? 0 : 1;    // my first tile of this row
      bool have_ref = false;                        // fixed reference: m_run holds the row's reference exponent
#pragma unroll 1
        for (int j = first; j < n_tiles; j += 2) {
          // scores ready (and the tile's bias words visible)
          ok = tc::mbar_wait(&ctl->k_empty[ring.stage * 2 + (ring.fill & 1)], (ring.fill >> 1) & 1, abort_flag);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          // Two score buffers: the scores of this tile were issued once P V of the group's previous one was complete, so the
          // accumulator may be rescaled below.  Three: see the wait before the rescale.
          tc::tc_fence_after();
          const uint32_t tS = tmem + buf * 128 + lane_base;
          const int chunks = j == n_tiles - 1 ? (last_cols + 31) >> 5 : 4;     // of 32 columns
          const float* slot_words = sBias + slot * kSlotWords;
          const float4* bg4 = reinterpret_cast<const float4*>(slot_words);     // one bias word per 4 columns
          const unsigned char* valid4 = reinterpret_cast<const unsigned char*>(slot_words + 36);   // 4 bits per group of 4 columns
          // Fast path: the bias is uniform inside every aligned group of 4 columns (blocks are at least 4 wide), so the
          // maximum is taken on raw scores per group and the bias enters once per group.  A tile with a block that ends
          // inside a group, with the causal diagonal, or that ends 16 columns early or more takes the per-column path (which rounds
          // score times scale before it subtracts the reference, so that the column with the maximum has exactly 1, whatever its size).
          // So the fast path's tiles have four chunks, and its loops no tests of their number: with them the exact kernel at head_dim 128
          // spilled 12 bytes and took 8 to 14 % longer (fp16 8 x 20011 x 128 878 -> 776 us, bf16 645 -> 630).
          const bool odd = reinterpret_cast<const int*>(slot_words)[32] != 0;
          // causal: of the diagonal block's pooled tokens (level li, columns [c0, c0 + 128 / l)) number i ends at position
          // (i + 1) l - 1, so row r sees the first (r + 1) / l of them
          int hide_lo = 128, hide_hi = 128;
          if (CAUSAL) {
            const int dw = reinterpret_cast<const int*>(slot_words)[33];
            if (odd && dw >= 0) {
              const int li = dw >> 8, c0 = dw & 255;
              hide_lo = c0 + ((r + 1) >> li);
              hide_hi = c0 + (128 >> li);
            }
          }
          uint32_t va[32], vb[32];      // two chunks of 32 score columns in flight
          float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
          const bool ref_tile = !FIXED || j == 0;      // fixed reference: only a row's first tile takes the maximum pass
          if (ref_tile && !odd) {
            // pass 1: running maximum; the load of the next chunk is issued before the current one is used
#define PSA_MAX_CHUNK(v, c)                                                                                                  \
  do {                                                                                                                       \
    const float4 ga = bg4[2 * (c)], gb = bg4[2 * (c) + 1];                                                                   \
    const float* f = reinterpret_cast<const float*>(v);                                                                      \
    mx0 = fmaxf(mx0, fmaf(fmaxf(fmaxf(f[0], f[1]), fmaxf(f[2], f[3])), p.scale_log2, ga.x));                                 \
    mx1 = fmaxf(mx1, fmaf(fmaxf(fmaxf(f[4], f[5]), fmaxf(f[6], f[7])), p.scale_log2, ga.y));                                 \
    mx2 = fmaxf(mx2, fmaf(fmaxf(fmaxf(f[8], f[9]), fmaxf(f[10], f[11])), p.scale_log2, ga.z));                               \
    mx3 = fmaxf(mx3, fmaf(fmaxf(fmaxf(f[12], f[13]), fmaxf(f[14], f[15])), p.scale_log2, ga.w));                             \
    mx0 = fmaxf(mx0, fmaf(fmaxf(fmaxf(f[16], f[17]), fmaxf(f[18], f[19])), p.scale_log2, gb.x));                             \
    mx1 = fmaxf(mx1, fmaf(fmaxf(fmaxf(f[20], f[21]), fmaxf(f[22], f[23])), p.scale_log2, gb.y));                             \
    mx2 = fmaxf(mx2, fmaf(fmaxf(fmaxf(f[24], f[25]), fmaxf(f[26], f[27])), p.scale_log2, gb.z));                             \
    mx3 = fmaxf(mx3, fmaf(fmaxf(fmaxf(f[28], f[29]), fmaxf(f[30], f[31])), p.scale_log2, gb.w));                             \
  } while (0)
            tc::tmem_ld32(tS, va);
#pragma unroll 1
            for (int c = 0; c < 4; c += 2) {
              tc::tmem_wait_ld();
              tc::tmem_ld32(tS + 32 * c + 32, vb);
              PSA_MAX_CHUNK(va, c);
              tc::tmem_wait_ld();
              if (c == 0) tc::tmem_ld32(tS + 64, va);
              PSA_MAX_CHUNK(vb, c + 1);
            }
#undef PSA_MAX_CHUNK
          } else if (ref_tile) {
#pragma unroll 1
            for (int h = 0; h < chunks; ++h) {
              tc::tmem_ld32(tS + h * 32, va);
              tc::tmem_wait_ld();
#pragma unroll
              for (int q4 = 0; q4 < 8; ++q4) {
                const float4 ba = column_bias<CAUSAL>(slot_words, valid4, h * 8 + q4, hide_lo, hide_hi);
                mx0 = fmaxf(mx0, fmaf(__uint_as_float(va[4 * q4 + 0]), p.scale_log2, ba.x));
                mx1 = fmaxf(mx1, fmaf(__uint_as_float(va[4 * q4 + 1]), p.scale_log2, ba.y));
                mx2 = fmaxf(mx2, fmaf(__uint_as_float(va[4 * q4 + 2]), p.scale_log2, ba.z));
                mx3 = fmaxf(mx3, fmaf(__uint_as_float(va[4 * q4 + 3]), p.scale_log2, ba.w));
              }
            }
          }
          const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
          // raise the running maximum only when it is far off (or still unset)
          float alpha = 1.f;
          bool raise = false;
          if (FIXED) {
            if (j == 0) {
              // the group that owns the row's first tile sets the reference for both groups
              m_run = mx == -INFINITY ? 0.f : mx;
              sMref[(ne & 1) * 128 + r] = m_run;
              __syncwarp();
              if (lane == 0) tc::mbar_arrive(&ctl->mref_full[ne & 1]);
              have_ref = true;
            } else if (!have_ref) {
              ok = tc::mbar_wait(&ctl->mref_full[ne & 1], (ne >> 1) & 1, abort_flag);
              ok = __all_sync(0xffffffffu, ok);
              if (!ok) break;
              m_run = sMref[(ne & 1) * 128 + r];
              have_ref = true;
            }
          } else {
            raise = mx > m_run + 8.f;
            if (raise) {
              alpha = m_run == -INFINITY ? 0.f : ex2(m_run - mx);
              m_run = mx;
              l_run *= alpha;
            }
          }
          if (!FIXED && C::NSB == 3 && j >= 2) {
            // Every product of this group is signalled; each signal is waited for exactly once and in order (here for the
            // product of tile j-2, in the epilogue for the last one), so the waiter is never more than one phase behind.
            // By now - a whole maximum pass after the scores were found ready - it has normally long completed.
            ok = tc::mbar_wait(&ctl->pv_done[g], pv_rows & 1, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            ++pv_rows;
            tc::tc_fence_after();
          }
          if (!FIXED && j >= 2 && __any_sync(0xffffffffu, raise)) {
            // the accumulator may only be touched between two of its P V products: the one of tile j-2 is complete (see
            // above), the one of tile j waits for the probabilities written below
#pragma unroll 1
            for (int c0 = 0; c0 < D; c0 += 32) {
              tc::tmem_ld32(tO + c0, vb);
              tc::tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 32; ++i) vb[i] = __float_as_uint(__uint_as_float(vb[i]) * alpha);
              tc::tmem_st32(tO + c0, vb);
            }
            tc::tmem_wait_st();
          }
          // pass 2: probabilities (rounded to the element type) written over the scores, running sum.  Chunk c reads score
          // columns [32c, 32c+32) and writes packed columns [16c, 16c+16): always columns that were read before.
          const float m_use = m_run == -INFINITY ? 0.f : m_run;
          float2 ls_a = make_float2(0.f, 0.f), ls_b = make_float2(0.f, 0.f);
          if (!odd) {
#define PSA_EXP_GROUP(f, cg, k, acc)                                                                                          \
  do {                                                                                                                       \
    const float2 cc = make_float2(cg, cg);                                                                                   \
    const float2 x01 = __ffma2_rn(make_float2(f[4 * (k)], f[4 * (k) + 1]), scale2, cc);                                      \
    const float2 x23 = __ffma2_rn(make_float2(f[4 * (k) + 2], f[4 * (k) + 3]), scale2, cc);                                  \
    const float2 e01 = make_float2(ex2(x01.x), ex2(x01.y)), e23 = make_float2(ex2(x23.x), ex2(x23.y));                       \
    acc = __fadd2_rn(acc, __fadd2_rn(e01, e23));                                                                             \
    pk[2 * (k)] = pack2<FMT>(e01.x, e01.y);                                                                                  \
    pk[2 * (k) + 1] = pack2<FMT>(e23.x, e23.y);                                                                              \
  } while (0)
#define PSA_EXP_CHUNK(v, c)                                                                                                  \
  do {                                                                                                                       \
    const float4 ga = bg4[2 * (c)], gb = bg4[2 * (c) + 1];                                                                   \
    const float* f = reinterpret_cast<const float*>(v);                                                                      \
    uint32_t pk[16];                                                                                                         \
    PSA_EXP_GROUP(f, ga.x - m_use, 0, ls_a); PSA_EXP_GROUP(f, ga.y - m_use, 1, ls_b);                                        \
    PSA_EXP_GROUP(f, ga.z - m_use, 2, ls_a); PSA_EXP_GROUP(f, ga.w - m_use, 3, ls_b);                                        \
    PSA_EXP_GROUP(f, gb.x - m_use, 4, ls_a); PSA_EXP_GROUP(f, gb.y - m_use, 5, ls_b);                                        \
    PSA_EXP_GROUP(f, gb.z - m_use, 6, ls_a); PSA_EXP_GROUP(f, gb.w - m_use, 7, ls_b);                                        \
    tc::tmem_st16(tS + 16 * (c), pk);                                                                                        \
  } while (0)
            tc::tmem_ld32(tS, va);
#pragma unroll(C::UNROLL_EXP ? 2 : 1)
            for (int c = 0; c < 4; c += 2) {
              tc::tmem_wait_ld();
              tc::tmem_ld32(tS + 32 * c + 32, vb);
              PSA_EXP_CHUNK(va, c);
              tc::tmem_wait_ld();
              if (c == 0) tc::tmem_ld32(tS + 64, va);
              PSA_EXP_CHUNK(vb, c + 1);
            }
#undef PSA_EXP_CHUNK
#undef PSA_EXP_GROUP
          } else {
#pragma unroll 1
            for (int h = 0; h < chunks; ++h) {
              tc::tmem_ld32(tS + h * 32, va);
              tc::tmem_wait_ld();
              uint32_t pk[16];
#pragma unroll
              for (int q4 = 0; q4 < 8; ++q4) {
                const float4 ba = column_bias<CAUSAL>(slot_words, valid4, h * 8 + q4, hide_lo, hide_hi);
                const float a0 = ex2(fmaf(__uint_as_float(va[4 * q4 + 0]), p.scale_log2, ba.x) - m_use);
                const float a1 = ex2(fmaf(__uint_as_float(va[4 * q4 + 1]), p.scale_log2, ba.y) - m_use);
                const float a2 = ex2(fmaf(__uint_as_float(va[4 * q4 + 2]), p.scale_log2, ba.z) - m_use);
                const float a3 = ex2(fmaf(__uint_as_float(va[4 * q4 + 3]), p.scale_log2, ba.w) - m_use);
                ls_a.x += a0 + a1;
                ls_b.x += a2 + a3;
                pk[2 * q4] = pack2<FMT>(a0, a1);
                pk[2 * q4 + 1] = pack2<FMT>(a2, a3);
              }
              tc::tmem_st16(tS + h * 16, pk);
            }
          }
          l_run += (ls_a.x + ls_a.y) + (ls_b.x + ls_b.y);
          tc::tmem_wait_st();
          tc::tc_fence_before();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&ctl->p_full[g * 2 + (mine & 1)]);   // one arrival per warp
          ++mine;
          ring.next(2);
          buf = buf + 2 >= C::NSB ? buf + 2 - C::NSB : buf + 2;
          slot = slot + 2 >= C::SLOTS ? slot + 2 - C::SLOTS : slot + 2;
        }
      if (!ok) break;
      // ---- end of the row
      const int my_tiles = n_tiles > first ? (n_tiles - first + 1) >> 1 : 0;
      const bool finishes = n_tiles == 0 ? g == 0 : ((g0 + n_tiles - 1) & 1) == g;
      if (n_tiles > 0) {
        if (ne > 0) ok = tc::mbar_wait(&ctl->o_free, (ne - 1) & 1, abort_flag);
        if (!FIXED && ok && my_tiles > 0) {      // my accumulator is final (signalled once per row after the last of my tiles)
          ok = tc::mbar_wait(&ctl->pv_done[g], pv_rows & 1, abort_flag);
          ++pv_rows;
        }
        if (finishes) {
          if (FIXED && ok) ok = tc::mbar_wait(&ctl->pv_done[0], ne & 1, abort_flag);      // the one accumulator is final
          if (ok) ok = tc::mbar_wait(&ctl->xch_full, ne & 1, abort_flag);
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if (!finishes) {
          sXch[r] = l_run;
          if (!FIXED) sXch[128 + r] = m_run;
          tc::tc_fence_before();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&ctl->xch_full);
        }
      }
      if (finishes) {
        const int64_t qrow = (int64_t)m * 128 + r;
        const bool stored = qrow < p.seq_q;
        const float l_o = n_tiles > 0 ? sXch[r] : 0.f, m_o = FIXED || n_tiles == 0 ? m_run : sXch[128 + r];
        const float m_all = FIXED ? m_run : fmaxf(m_run, m_o);      // fixed reference: both groups used the same exponent
        const float w_me = FIXED ? 1.f : (m_run == -INFINITY ? 0.f : ex2(m_run - m_all));
        const float w_ot = FIXED ? 1.f : (m_o == -INFINITY ? 0.f : ex2(m_o - m_all));
        const float l_all = l_run * w_me + l_o * w_ot;
        // legacy kernel: no visible key -> 0, lse -inf (fixed reference: a row that sees any key sees one of its first tile,
        // so "no key" = sum 0); otherwise a row without keys is 0/0 like the reference, also one without any block
        const bool dead = p.legacy && (FIXED ? l_all == 0.f : m_all == -INFINITY);
        const float inv = dead ? 0.f : 1.0f / l_all;
        const float w = w_me * inv, wo = w_ot * inv;
        if (p.lse && stored)
          p.lse[(int64_t)bh * p.seq_q + qrow] = dead ? -INFINITY : n_tiles == 0 ? __int_as_float(0x7fc00000) : (m_all + log2f(l_all)) * 0.6931471805599453f;
        const bool other_has = !FIXED && n_tiles > my_tiles;
        uint16_t* orow;
        {
          const int64_t drow = p.scatter.row_perm && stored ? (int64_t)p.scatter.row_perm[qrow] : qrow;
          if (p.scatter.n_peers > 0) {
            const int64_t owner = stored ? drow / p.scatter.tokens_per_rank : 0, local = drow - owner * p.scatter.tokens_per_rank;
            orow = reinterpret_cast<uint16_t*>(p.scatter.peer_out[owner]) + (local * p.scatter.heads_total + p.scatter.head0 + bh) * D;
          } else {
            orow = reinterpret_cast<uint16_t*>(p.out) + ((int64_t)bh * p.seq_q + drow) * D;
          }
        }
        tc::tc_fence_after();
        float z = 0.f;               // NaN if any value is not finite
        const float none = dead ? 0.f : __int_as_float(0x7fc00000);
        // A thread stores its own row, 32 bytes (a whole sector) at a time; an output that is only 16-byte aligned in halves.
        const bool wide = (reinterpret_cast<uintptr_t>(orow) & 31) == 0;
#pragma unroll 1
        for (int c0 = 0; c0 < D; c0 += 32) {
          uint32_t va[32], vb[32], pk[16];
          if (n_tiles > 0) {
            tc::tmem_ld32(tO + c0, va);
            if (other_has) tc::tmem_ld32(tO_other + c0, vb);
            tc::tmem_wait_ld();
          }
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float f0 = n_tiles > 0 ? __uint_as_float(va[i]) * w : none, f1 = n_tiles > 0 ? __uint_as_float(va[i + 1]) * w : none;
            if (other_has) {
              f0 += __uint_as_float(vb[i]) * wo;
              f1 += __uint_as_float(vb[i + 1]) * wo;
            }
            if (FIXED) z = fmaf(f0, 0.f, fmaf(f1, 0.f, z));
            pk[i >> 1] = pack2<FMT>(f0, f1);
          }
          if (stored) {
            if (wide) {
              store32(orow + c0, pk);
              store32(orow + c0 + 16, pk + 8);
            } else {
#pragma unroll
              for (int i = 0; i < 16; i += 4) *reinterpret_cast<uint4*>(orow + c0 + 2 * i) = make_uint4(pk[i], pk[i + 1], pk[i + 2], pk[i + 3]);
            }
          }
        }
        if (n_tiles > 0) {
          // the accumulators may be overwritten by the next row from here on
          tc::tc_fence_before();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&ctl->o_free);
        }
        // The sum near the end of the exponent range (or NaN), or a product of such probabilities with large values past it.
        // A sum far below 1: every score of the first tile was -inf, which leaves the reference at 0 (a row of one tile
        // is then a row without a key in the exact kernel as well).
        if (FIXED && p.guard && n_tiles > 0 && stored && !(l_all < kSumMax && (l_all > kSumMin || n_tiles == 1) && z == 0.f)) *p.guard = 1;
      }
      ne += n_tiles > 0;
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&ctl->row_done[rslot]);
      g0 += n_tiles;
    }
  }

  // ---------------------------------------------------------------- teardown
  tc::tc_fence_before();
  __syncthreads();
  if (ctl->abort_flag) {
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, PSA_ERR_TIMEOUT);
    for (int i = 0; i < 64; ++i) __nanosleep(1000);   // let copies in flight land before the CTA retires
    __syncthreads();
  }
  if (warp == 3) {
    __syncwarp();
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, 512);
  }
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link-time dependency on libcuda).
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)ptr;
  }
  return fn;
}

}  // namespace

int encode_tmap_3d(CUtensorMap* map, const void* base, int elem_bytes, int is_bf16, int64_t channels, int64_t tokens,
                   int64_t bh, int box_rows) {
  EncodeTiledFn fn = get_encode_fn();
  PSA_REQUIRE(fn != nullptr, PSA_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t dims[3] = {(cuuint64_t)channels, (cuuint64_t)tokens, (cuuint64_t)bh};
  cuuint64_t strides[2] = {(cuuint64_t)channels * elem_bytes, (cuuint64_t)tokens * channels * elem_bytes};
  cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base),
                  dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  PSA_REQUIRE(r == CUDA_SUCCESS, PSA_ERR_CUDA, "cuTensorMapEncodeTiled failed with CUresult %d (tokens=%lld box_rows=%d)", (int)r,
              (long long)tokens, box_rows);
  return PSA_OK;
}

bool fwd_tc_supported(const FwdArgs& a) {
  if (a.dtype != PSA_F16 && a.dtype != PSA_BF16) return false;
  if (a.bm != 128 || a.tn != 32) return false;
  if (a.D != 64 && a.D != 128) return false;
  // (no table in the kernel bounds these: what its lists have been tested at, and what callers route by)
  if (a.width > (a.kimg || a.causal ? PSA_FWD_LIST_MAX : PSA_FWD_LIST_MAX_ROWS)) return false;
  if (cdiv64(a.seq_k, a.bn) > (a.width > PSA_FWD_LIST_MAX ? PSA_FWD_BLOCKS_MAX_ROWS : PSA_FWD_BLOCKS_MAX)) return false;
  if (a.bh > 65535) return false;
  if (!(a.scale > 0.f)) return false;
  const void* ptrs[] = {a.q, a.out, a.k[0], a.k[1], a.k[2], a.k[3], a.v[0], a.v[1], a.v[2], a.v[3]};
  for (const void* ptr : ptrs)
    if ((uintptr_t)ptr & 15) return false;
  return true;
}

// Row counters of the persistent forward: a ring of device words; every launch takes the next one and zeroes it on its
// own stream right before the kernel, so launches in flight on different streams do not share a counter (unless more than
// kCounterRing launches of one device overlap in time).
constexpr int kCounterRing = 256;
__device__ int g_row_counters[kCounterRing];

// n (1 to 3) neighbouring words, zeroed by one memset.
static int next_counters(int n, int** out, cudaStream_t st) {
  constexpr int kMaxDevices = 64;
  static int* base[kMaxDevices] = {nullptr};
  static unsigned next[kMaxDevices] = {0};
  static std::mutex mu;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  PSA_REQUIRE(e == cudaSuccess && dev >= 0 && dev < kMaxDevices, PSA_ERR_CUDA, "psa_fwd: cudaGetDevice failed: %s", cudaGetErrorString(e));
  std::lock_guard<std::mutex> lock(mu);
  if (!base[dev]) {
    void* ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_row_counters);
    PSA_REQUIRE(e == cudaSuccess && ptr, PSA_ERR_CUDA, "psa_fwd: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
    base[dev] = (int*)ptr;
  }
  unsigned pos = next[dev] % kCounterRing;
  if (pos + n > kCounterRing) pos = 0;      // the words of one call do not wrap around
  next[dev] = pos + n;
  int* c = base[dev] + pos;
  e = cudaMemsetAsync(c, 0, n * sizeof(int), st);
  PSA_REQUIRE(e == cudaSuccess, PSA_ERR_CUDA, "psa_fwd: cudaMemsetAsync failed: %s", cudaGetErrorString(e));
  *out = c;
  return PSA_OK;
}

template <int D, int FMT, bool IMG, bool CAUSAL, bool FIXED>
static int launch_tc(const FwdArgs& a, cudaStream_t st, int* row_counter, int* guard = nullptr, const int* only_if = nullptr) {
  constexpr int kSmem = smem_bytes<D, FIXED, CAUSAL>();
  static_assert(kSmem <= 232448, "more than 227 KB of shared memory");
  TmapPack maps;
  const int is_bf16 = FMT == 1;
  int rc = encode_tmap_3d(&maps.q, a.q, 2, is_bf16, D, a.seq_q, a.bh, 128);
  if (rc != PSA_OK) return rc;
  for (int li = 0; li < 4 && !IMG; ++li) {
    const int P = a.bn >> li;
    rc = encode_tmap_3d(&maps.k[li], a.k[li], 2, is_bf16, D, a.n[li], a.bh, P);
    if (rc != PSA_OK) return rc;
    rc = encode_tmap_3d(&maps.v[li], a.v[li], 2, is_bf16, D, a.n[li], a.bh, P);
    if (rc != PSA_OK) return rc;
  }
  TcParams p;
  p.mask = a.mask; p.out = a.out; p.status = a.status; p.seq_q = a.seq_q;
  for (int i = 0; i < 4; ++i) p.n[i] = a.n[i];
  p.mq = (int)cdiv64(a.seq_q, 128); p.nblocks = (int)cdiv64(a.seq_k, a.bn); p.bn = a.bn; p.tn = a.tn; p.width = a.width; p.quirk = a.quirk;
  p.scale_log2 = a.scale * 1.4426950408889634f;
  p.total_rows = (int)((int64_t)p.mq * a.bh);
  p.kimg = (const unsigned char*)a.kimg; p.vimg = (const unsigned char*)a.vimg;
  p.img = make_img_levels(a.bh, a.seq_k, D, IMG ? a.bn : 64);
  p.scatter = a.scatter;
  p.lse = a.lse; p.legacy = a.legacy; p.causal = a.causal;
  p.guard = guard; p.only_if = only_if;
  cudaError_t e = cudaFuncSetAttribute(psa_fwd_tc_kernel<D, FMT, IMG, CAUSAL, FIXED>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
  PSA_REQUIRE(e == cudaSuccess, PSA_ERR_CUDA, "psa_fwd: shared-memory opt-in (%d B) failed: %s", kSmem,
              cudaGetErrorString(e));
  // persistent: one CTA per SM (up to 227 KB of shared memory and all 512 TMEM columns each); rows are claimed from a counter in
  // ascending order, so the CTAs running at the same time work on neighbouring rows of the same head (K/V stay in L2)
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  PSA_REQUIRE(sms > 0, PSA_ERR_CUDA, "psa_fwd: cannot read the SM count");
  const unsigned grid = (unsigned)(p.total_rows < sms ? p.total_rows : sms);
  p.row_counter = row_counter;
  psa_fwd_tc_kernel<D, FMT, IMG, CAUSAL, FIXED><<<grid, kThreads, kSmem, st>>>(maps, p);
  PSA_CHECK_LAUNCH("psa_fwd(tcgen05)");
  return PSA_OK;
}

// The fixed-reference kernel, then the exact one, which returns at once unless the first one raised its guard word (a row
// whose probabilities came near the end of the exponent range) - no host round trip.
template <int D, int FMT, bool IMG, bool CAUSAL>
static int launch_fixed_then_exact(const FwdArgs& a, cudaStream_t st) {
  static_assert(FMT == 1, "bf16 only");
  int* words = nullptr;                       // row counters of both kernels and the guard word
  int rc = next_counters(3, &words, st);
  if (rc != PSA_OK) return rc;
  rc = launch_tc<D, FMT, IMG, CAUSAL, true>(a, st, words, words + 2, nullptr);
  if (rc != PSA_OK) return rc;
  return launch_tc<D, FMT, IMG, CAUSAL, false>(a, st, words + 1, nullptr, words + 2);
}

template <int D, int FMT, bool IMG, bool CAUSAL>
static int launch_exact(const FwdArgs& a, cudaStream_t st) {
  int* words = nullptr;
  const int rc = next_counters(1, &words, st);
  return rc != PSA_OK ? rc : launch_tc<D, FMT, IMG, CAUSAL, false>(a, st, words);
}

int fwd_tc_launch(const FwdArgs& a, cudaStream_t st) {
  const int fmt = a.dtype == PSA_BF16 ? 1 : 0;
  const bool img = a.kimg != nullptr && a.vimg != nullptr;
  if (img) {
    PSA_REQUIRE(a.bn >= 64, PSA_ERR_UNSUPPORTED, "tile images need block_n >= 64 (blocks of at least 8 pooled rows)");
    PSA_REQUIRE((((uintptr_t)a.kimg | (uintptr_t)a.vimg) & 15) == 0, PSA_ERR_ARG, "tile images must be 16-byte aligned");
    if (a.causal) {   // only the legacy forward asks for it; a variant of its own keeps the common kernel lean
      if (a.D == 64) return fmt ? launch_fixed_then_exact<64, 1, true, true>(a, st) : launch_exact<64, 0, true, true>(a, st);
      return fmt ? launch_fixed_then_exact<128, 1, true, true>(a, st) : launch_exact<128, 0, true, true>(a, st);
    }
    if (a.D == 64) return fmt ? launch_fixed_then_exact<64, 1, true, false>(a, st) : launch_exact<64, 0, true, false>(a, st);
    return fmt ? launch_fixed_then_exact<128, 1, true, false>(a, st) : launch_exact<128, 0, true, false>(a, st);
  }
  PSA_REQUIRE(!a.causal, PSA_ERR_UNSUPPORTED, "the causal rule needs the tile-image path");
  if (a.D == 64) return fmt ? launch_fixed_then_exact<64, 1, false, false>(a, st) : launch_exact<64, 0, false, false>(a, st);
  return fmt ? launch_fixed_then_exact<128, 1, false, false>(a, st) : launch_exact<128, 0, false, false>(a, st);
}

}  // namespace psa

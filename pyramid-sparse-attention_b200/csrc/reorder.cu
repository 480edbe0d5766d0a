// Token reordering (space-filling-curve order of the video tokens) folded into the attention kernels.
//
// The reference reorders q, k, v with three index_select copies before the attention and the output with a fourth one
// after it (src/psa_triton/utils/rearranger.py:69-132).  Here one int32 table `perm` [seq] (token t of the attention's
// sequence = row perm[t] of the stored tensor) is read by the kernels that touch the rows anyway: the tile-image builder
// and the sample gather of the block scores read k, v (and the sampled quarter of q) through it, and the forward's
// epilogue stores output row t at row perm[t].  Only q needs a copy of its own (the forward fetches query tiles with
// one bulk tensor copy per tile), which is the kernel in this file.
#include "psa_common.cuh"
#include "fwd.h"

namespace psa {
namespace {

// The four kernels up to gather_heads_rope_kernel take rows of any whole number cpr of 16-byte words: fp32 rows, and 16-bit
// rows of other widths than the 64 and 128 channels that gather_views_kernel below is made for.
// dst[bh][t][:] = src[bh][perm[t]][:].
__global__ void __launch_bounds__(256) gather_rows_kernel(const uint4* __restrict__ src, const int32_t* __restrict__ perm,
                                                          uint4* __restrict__ dst, int64_t seq, int cpr) {
  const int64_t bh = blockIdx.y;
  const uint4* s = src + bh * seq * cpr;
  uint4* d = dst + bh * seq * cpr;
  const int64_t total = seq * cpr;
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = w / cpr;
    const int c = (int)(w - t * cpr);
    d[w] = s[(int64_t)perm[t] * cpr + c];
  }
}

// dst[h][t][:] = src[perm ? perm[t] : t][h][:]: token-major rows regrouped by head (and reordered) in one pass.
__global__ void __launch_bounds__(256) gather_heads_kernel(const uint4* __restrict__ src, const int32_t* __restrict__ perm,
                                                           uint4* __restrict__ dst, int64_t seq, int heads, int cpr) {
  const int64_t h = blockIdx.y;
  uint4* d = dst + h * seq * cpr;
  const int64_t total = seq * cpr;
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = w / cpr;
    const int c = (int)(w - t * cpr);
    const int64_t row = perm ? (int64_t)perm[t] : t;
    d[w] = src[(row * heads + h) * cpr + c];
  }
}

// dst[bh][t][:] = rotated src[bh][perm ? perm[t] : t][:] (16-bit rows; see RopeTables in fwd.h for the arithmetic).
__global__ void __launch_bounds__(256) gather_rows_rope_kernel(const uint4* __restrict__ src, const int32_t* __restrict__ perm,
                                                               uint4* __restrict__ dst, int64_t seq, int cpr,
                                                               const float* __restrict__ rope_a, const float* __restrict__ rope_b,
                                                               int64_t rope_first, int bf16) {
  const int64_t bh = blockIdx.y;
  const uint4* s = src + bh * seq * cpr;
  uint4* d = dst + bh * seq * cpr;
  const int64_t total = seq * cpr;
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = w / cpr;
    const int c = (int)(w - t * cpr);
    const int64_t row = perm ? (int64_t)perm[t] : t;
    uint4 x = s[row * cpr + c];
    if (row >= rope_first) {
      const int64_t off = ((row - rope_first) * cpr + c) * 8;
      x = rotate_word(x, rope_a + off, rope_b + off, bf16 != 0);
    }
    d[w] = x;
  }
}

// The same with every row rotated on the way (16-bit rows; see RopeTables in fwd.h for the arithmetic).
__global__ void __launch_bounds__(256) gather_heads_rope_kernel(const uint4* __restrict__ src, const int32_t* __restrict__ perm,
                                                                uint4* __restrict__ dst, int64_t seq, int heads, int cpr,
                                                                const float* __restrict__ rope_a, const float* __restrict__ rope_b,
                                                                int64_t rope_first, int bf16) {
  const int64_t h = blockIdx.y;
  uint4* d = dst + h * seq * cpr;
  const int64_t total = seq * cpr;
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = w / cpr;
    const int c = (int)(w - t * cpr);
    const int64_t row = perm ? (int64_t)perm[t] : t;
    uint4 x = src[(row * heads + h) * cpr + c];
    if (row >= rope_first) {
      const int64_t off = ((row - rope_first) * cpr + c) * 8;
      x = rotate_word(x, rope_a + off, rope_b + off, bf16 != 0);
    }
    d[w] = x;
  }
}

// Up to three strided operands [batch][heads][seq][D] copied head-major and contiguous in one launch, each read through
// the row table and, where asked, rotated on the way (RopeTables in fwd.h).
struct ViewSet {
  const uint4* src[3];
  int64_t batch_stride[3], head_stride[3], token_stride[3];   // in 16-byte words
  uint4* dst[3];
  int rotate[3];
};

// HBM-bound: every row is read and written once.  A thread moves the same 16-byte word of kUnroll rows, with all loads
// issued before the first store: the address of a row hangs on its table entry, so one row at a time leaves a warp with a
// single load in flight behind another one.  Rows are 128 or 256 contiguous bytes, whatever the order of the tokens.
// 12 heads x 32760 tokens x 128, q, k, v from token-major views, ordered, q and k rotated: 134 us (4.5 TB/s of rows; the
// rotary tables come on top, from L2).  The framework's element-wise operations took 2.5 ms for the same copies.
template <int CPR, bool ROPE>
__global__ void __launch_bounds__(256) gather_views_kernel(const ViewSet v, const int32_t* __restrict__ perm, int64_t seq, int heads,
                                                           int bh_count, const RopeTables rope) {
  constexpr int kUnroll = 4, kRows = 256 / CPR;
  const int z = blockIdx.z, c = threadIdx.x % CPR;
  // blocks walk the heads fastest where the rows of a token lie together (token-major), so that one DRAM page and one row of
  // the rotary tables serve all heads; head by head otherwise
  const unsigned stretches = gridDim.x / (unsigned)bh_count;
  const bool heads_fastest = v.head_stride[z] < v.token_stride[z];
  const int bh = (int)(heads_fastest ? blockIdx.x % (unsigned)bh_count : blockIdx.x / stretches);
  const int64_t stretch = heads_fastest ? blockIdx.x / (unsigned)bh_count : blockIdx.x % stretches;
  const int64_t b = bh / heads, h = bh % heads;
  const uint4* src = v.src[z] + b * v.batch_stride[z] + h * v.head_stride[z] + c;
  uint4* dst = v.dst[z] + (int64_t)bh * seq * CPR + c;
  const int64_t t0 = stretch * (kRows * kUnroll) + threadIdx.x / CPR;
  int64_t row[kUnroll];
  uint4 x[kUnroll];
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const int64_t t = t0 + u * kRows;
    row[u] = t < seq ? (perm ? (int64_t)perm[t] : t) : -1;
  }
#pragma unroll
  for (int u = 0; u < kUnroll; ++u)
    if (row[u] >= 0) x[u] = __ldg(src + row[u] * v.token_stride[z]);
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    if (row[u] < 0) continue;
    if (ROPE && v.rotate[z] && row[u] >= rope.first) {
      const int64_t off = ((row[u] - rope.first) * CPR + c) * 8;
      x[u] = rotate_word(x[u], rope.a + off, rope.b + off, rope.bf16 != 0);
    }
    dst[(t0 + u * kRows) * CPR] = x[u];
  }
}

int launch_views(const ViewSet& v, int n, const int32_t* perm, const RopeTables& rope, int64_t batch, int heads, int64_t seq, int head_dim,
                 cudaStream_t st) {
  const int64_t blocks = cdiv64(seq, 256 / (head_dim / 8) * 4) * batch * heads;
  PSA_REQUIRE(blocks < ((int64_t)1 << 31), PSA_ERR_ARG, "row copy: too many rows");
  const dim3 grid((unsigned)blocks, 1, (unsigned)n);
  const int bh = (int)(batch * heads);
  if (head_dim == 64) {
    if (rope.a) gather_views_kernel<8, true><<<grid, 256, 0, st>>>(v, perm, seq, heads, bh, rope);
    else gather_views_kernel<8, false><<<grid, 256, 0, st>>>(v, perm, seq, heads, bh, rope);
  } else {
    if (rope.a) gather_views_kernel<16, true><<<grid, 256, 0, st>>>(v, perm, seq, heads, bh, rope);
    else gather_views_kernel<16, false><<<grid, 256, 0, st>>>(v, perm, seq, heads, bh, rope);
  }
  PSA_CHECK_LAUNCH("row copy");
  return PSA_OK;
}

// One operand of 16-bit rows of 64 or 128 channels, its strides in elements.
int launch_one_view(const void* src, void* dst, int64_t head_stride, int64_t token_stride, const int32_t* perm, const RopeTables& rope,
                    int heads, int64_t seq, int head_dim, cudaStream_t st) {
  ViewSet v = {};
  v.src[0] = (const uint4*)src;
  v.dst[0] = (uint4*)dst;
  v.head_stride[0] = head_stride / 8;
  v.token_stride[0] = token_stride / 8;
  v.rotate[0] = rope.a != nullptr;
  return launch_views(v, 1, perm, rope, 1, heads, seq, head_dim, st);
}

}  // namespace
}  // namespace psa

extern "C" int psa_gather_views(const void* const* src, const int64_t* strides, const int32_t* rotate, void* const* dst, int n,
                                const int32_t* perm, const float* rope_a, const float* rope_b, int64_t rope_first, int64_t batch,
                                int heads, int64_t seq, int head_dim, int dtype, void* stream) {
  using namespace psa;
  PSA_REQUIRE(src && strides && rotate && dst && n >= 1 && n <= 3, PSA_ERR_ARG, "psa_gather_views: 1 to 3 operands");
  PSA_REQUIRE(dtype == PSA_F16 || dtype == PSA_BF16, PSA_ERR_UNSUPPORTED, "psa_gather_views: f16/bf16 only");
  PSA_REQUIRE(head_dim == 64 || head_dim == 128, PSA_ERR_ARG, "psa_gather_views: head_dim=%d unsupported (64/128)", head_dim);
  PSA_REQUIRE(batch > 0 && heads > 0 && batch * heads < 65536 && seq > 0 && seq < ((int64_t)1 << 31), PSA_ERR_ARG,
              "psa_gather_views: bad shape");
  PSA_REQUIRE((rope_a != nullptr) == (rope_b != nullptr) && (!rope_a || (rope_first >= 0 && rope_first <= seq)), PSA_ERR_ARG,
              "psa_gather_views: bad rotary tables");
  PSA_REQUIRE((((uintptr_t)rope_a | (uintptr_t)rope_b) & 15) == 0, PSA_ERR_ARG, "psa_gather_views: tables must be 16-byte aligned");
  ViewSet v = {};
  for (int i = 0; i < n; ++i) {
    PSA_REQUIRE(src[i] && dst[i] && src[i] != dst[i], PSA_ERR_ARG, "psa_gather_views: operand %d", i);
    PSA_REQUIRE((((uintptr_t)src[i] | (uintptr_t)dst[i]) & 15) == 0, PSA_ERR_ARG, "psa_gather_views: operand %d is not 16-byte aligned", i);
    PSA_REQUIRE(!rotate[i] || rope_a, PSA_ERR_ARG, "psa_gather_views: operand %d is to be rotated without tables", i);
    for (int d = 0; d < 3; ++d)
      PSA_REQUIRE(strides[3 * i + d] >= 0 && strides[3 * i + d] % 8 == 0, PSA_ERR_ARG,
                  "psa_gather_views: strides of operand %d must be multiples of 8 elements", i);
    v.src[i] = (const uint4*)src[i];
    v.dst[i] = (uint4*)dst[i];
    v.batch_stride[i] = strides[3 * i] / 8;
    v.head_stride[i] = strides[3 * i + 1] / 8;
    v.token_stride[i] = strides[3 * i + 2] / 8;
    v.rotate[i] = rotate[i] != 0;
  }
  return launch_views(v, n, perm, {rope_a, rope_b, rope_first, dtype == PSA_BF16}, batch, heads, seq, head_dim, (cudaStream_t)stream);
}

extern "C" int psa_gather_rows(const void* src, const int32_t* perm, void* dst, int64_t bh, int64_t seq, int head_dim,
                               int elem_bytes, void* stream) {
  using namespace psa;
  PSA_REQUIRE(src && perm && dst, PSA_ERR_ARG, "psa_gather_rows: null pointer");
  PSA_REQUIRE(src != dst, PSA_ERR_ARG, "psa_gather_rows: cannot reorder in place");
  PSA_REQUIRE(bh > 0 && bh < 65536 && seq > 0 && seq < ((int64_t)1 << 31), PSA_ERR_ARG, "psa_gather_rows: bad shape");
  PSA_REQUIRE(elem_bytes == 2 || elem_bytes == 4, PSA_ERR_ARG, "psa_gather_rows: elem_bytes=%d (2 or 4)", elem_bytes);
  PSA_REQUIRE(head_dim > 0 && (head_dim * elem_bytes) % 16 == 0, PSA_ERR_ARG,
              "psa_gather_rows: rows of %d bytes are not a multiple of 16", head_dim * elem_bytes);
  PSA_REQUIRE((((uintptr_t)src | (uintptr_t)dst) & 15) == 0, PSA_ERR_ARG, "psa_gather_rows: src and dst must be 16-byte aligned");
  if (elem_bytes == 2 && (head_dim == 64 || head_dim == 128))
    return launch_one_view(src, dst, seq * head_dim, head_dim, perm, RopeTables{}, (int)bh, seq, head_dim, (cudaStream_t)stream);
  const int cpr = head_dim * elem_bytes / 16;
  int64_t blocks = cdiv64(seq * cpr, 256);
  // enough CTAs to cover the machine several times over once the heads (grid.y) are counted in
  const int64_t cap = cdiv64(148 * 16, bh);
  if (blocks > cap) blocks = cap;
  dim3 grid((unsigned)blocks, (unsigned)bh);
  gather_rows_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((const uint4*)src, perm, (uint4*)dst, seq, cpr);
  PSA_CHECK_LAUNCH("psa_gather_rows");
  return PSA_OK;
}

extern "C" int psa_gather_heads(const void* src, const int32_t* perm, void* dst, int heads, int64_t seq, int head_dim,
                                int elem_bytes, void* stream) {
  using namespace psa;
  PSA_REQUIRE(src && dst, PSA_ERR_ARG, "psa_gather_heads: null pointer");
  PSA_REQUIRE(src != dst, PSA_ERR_ARG, "psa_gather_heads: cannot regroup in place");
  PSA_REQUIRE(heads > 0 && heads < 65536 && seq > 0 && seq < ((int64_t)1 << 31), PSA_ERR_ARG, "psa_gather_heads: bad shape");
  PSA_REQUIRE(elem_bytes == 2 || elem_bytes == 4, PSA_ERR_ARG, "psa_gather_heads: elem_bytes=%d (2 or 4)", elem_bytes);
  PSA_REQUIRE(head_dim > 0 && (head_dim * elem_bytes) % 16 == 0, PSA_ERR_ARG,
              "psa_gather_heads: rows of %d bytes are not a multiple of 16", head_dim * elem_bytes);
  PSA_REQUIRE((((uintptr_t)src | (uintptr_t)dst) & 15) == 0, PSA_ERR_ARG, "psa_gather_heads: src and dst must be 16-byte aligned");
  if (elem_bytes == 2 && (head_dim == 64 || head_dim == 128))
    return launch_one_view(src, dst, head_dim, (int64_t)heads * head_dim, perm, RopeTables{}, heads, seq, head_dim, (cudaStream_t)stream);
  const int cpr = head_dim * elem_bytes / 16;
  int64_t blocks = cdiv64(seq * cpr, 256);
  const int64_t cap = cdiv64(148 * 16, heads);
  if (blocks > cap) blocks = cap;
  dim3 grid((unsigned)blocks, (unsigned)heads);
  gather_heads_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((const uint4*)src, perm, (uint4*)dst, seq, heads, cpr);
  PSA_CHECK_LAUNCH("psa_gather_heads");
  return PSA_OK;
}

extern "C" int psa_gather_heads_rope(const void* src, const int32_t* perm, const float* rope_a, const float* rope_b,
                                     int64_t rope_first, void* dst, int heads, int64_t seq, int head_dim, int dtype, void* stream) {
  using namespace psa;
  PSA_REQUIRE(src && dst && rope_a && rope_b, PSA_ERR_ARG, "psa_gather_heads_rope: null pointer");
  PSA_REQUIRE(src != dst, PSA_ERR_ARG, "psa_gather_heads_rope: cannot regroup in place");
  PSA_REQUIRE(dtype == PSA_F16 || dtype == PSA_BF16, PSA_ERR_UNSUPPORTED, "psa_gather_heads_rope: f16/bf16 only");
  PSA_REQUIRE(heads > 0 && heads < 65536 && seq > 0 && seq < ((int64_t)1 << 31) && rope_first >= 0 && rope_first <= seq, PSA_ERR_ARG,
              "psa_gather_heads_rope: bad shape");
  PSA_REQUIRE(head_dim > 0 && head_dim % 8 == 0, PSA_ERR_ARG, "psa_gather_heads_rope: head_dim=%d is not a multiple of 8", head_dim);
  PSA_REQUIRE((((uintptr_t)src | (uintptr_t)dst | (uintptr_t)rope_a | (uintptr_t)rope_b) & 15) == 0, PSA_ERR_ARG,
              "psa_gather_heads_rope: src, dst and the tables must be 16-byte aligned");
  if (head_dim == 64 || head_dim == 128)
    return launch_one_view(src, dst, head_dim, (int64_t)heads * head_dim, perm, {rope_a, rope_b, rope_first, dtype == PSA_BF16}, heads, seq,
                           head_dim, (cudaStream_t)stream);
  const int cpr = head_dim * 2 / 16;
  int64_t blocks = cdiv64(seq * cpr, 256);
  const int64_t cap = cdiv64(148 * 16, heads);
  if (blocks > cap) blocks = cap;
  dim3 grid((unsigned)blocks, (unsigned)heads);
  gather_heads_rope_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((const uint4*)src, perm, (uint4*)dst, seq, heads, cpr, rope_a, rope_b,
                                                                    rope_first, dtype == PSA_BF16);
  PSA_CHECK_LAUNCH("psa_gather_heads_rope");
  return PSA_OK;
}

extern "C" int psa_gather_rows_rope(const void* src, const int32_t* perm, const float* rope_a, const float* rope_b, int64_t rope_first,
                                    void* dst, int64_t bh, int64_t seq, int head_dim, int dtype, void* stream) {
  using namespace psa;
  PSA_REQUIRE(src && dst && rope_a && rope_b, PSA_ERR_ARG, "psa_gather_rows_rope: null pointer");
  PSA_REQUIRE(src != dst, PSA_ERR_ARG, "psa_gather_rows_rope: cannot reorder in place");
  PSA_REQUIRE(dtype == PSA_F16 || dtype == PSA_BF16, PSA_ERR_UNSUPPORTED, "psa_gather_rows_rope: f16/bf16 only");
  PSA_REQUIRE(bh > 0 && bh < 65536 && seq > 0 && seq < ((int64_t)1 << 31) && rope_first >= 0 && rope_first <= seq, PSA_ERR_ARG,
              "psa_gather_rows_rope: bad shape");
  PSA_REQUIRE(head_dim > 0 && head_dim % 8 == 0, PSA_ERR_ARG, "psa_gather_rows_rope: head_dim=%d is not a multiple of 8", head_dim);
  PSA_REQUIRE((((uintptr_t)src | (uintptr_t)dst | (uintptr_t)rope_a | (uintptr_t)rope_b) & 15) == 0, PSA_ERR_ARG,
              "psa_gather_rows_rope: src, dst and the tables must be 16-byte aligned");
  if (head_dim == 64 || head_dim == 128)
    return launch_one_view(src, dst, seq * head_dim, head_dim, perm, {rope_a, rope_b, rope_first, dtype == PSA_BF16}, (int)bh, seq, head_dim,
                           (cudaStream_t)stream);
  const int cpr = head_dim * 2 / 16;
  int64_t blocks = cdiv64(seq * cpr, 256);
  const int64_t cap = cdiv64(148 * 16, bh);
  if (blocks > cap) blocks = cap;
  dim3 grid((unsigned)blocks, (unsigned)bh);
  gather_rows_rope_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((const uint4*)src, perm, (uint4*)dst, seq, cpr, rope_a, rope_b, rope_first,
                                                                   dtype == PSA_BF16);
  PSA_CHECK_LAUNCH("psa_gather_rows_rope");
  return PSA_OK;
}

// K-similarity cap: per key block, the mean cosine similarity of token pairs (2i,2i+1), (4i,4i+3) and
// (8i,8i+7) decides the coarsest pyramid level the block may be pooled to.
//
// K is read once (N*e bytes), one int32 per block is written.  One warp per key block; the warp walks the block 8 tokens at
// a time, lanes split the channels.  Bound by its instructions, not by HBM: 28 x 32768 x 128 takes 89 us (101 with one butterfly per sum).
#include "psa_common.cuh"

namespace psa {

template <typename T>
__global__ void __launch_bounds__(128) ksim_kernel(const T* __restrict__ k, const int32_t* __restrict__ perm, int32_t* __restrict__ out,
                                                   int64_t seq, int D, int bn, int nblk, float t2, float t4, float t8) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int blk = blockIdx.x * 4 + warp;
  if (blk >= nblk) return;
  const int64_t bh = blockIdx.y;
  const T* kh = k + bh * seq * D;
  float c2 = 0.f, c4 = 0.f, c8 = 0.f;
  // which two norms divide the product this lane ends up with (see below)
  const int held = lane >> 1;
  const int norm_a = held < 8 ? 0 : held < 12 ? 2 * (held - 8) : held == 13 ? 4 : 0;
  const int norm_b = held < 8 ? 0 : held < 12 ? 2 * (held - 8) + 1 : held == 12 ? 3 : 7;
  for (int g0 = 0; g0 < bn; g0 += 8) {
    // sums of this lane's channels: 8 squared norms, 4 + 2 + 1 products
    float v[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) v[t] = 0.f;
    const T* rows[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      int64_t tok = (int64_t)blk * bn + g0 + t;
      tok = tok < seq ? tok : seq - 1;
      if (perm) tok = perm[tok];              // token `tok` of the reordered sequence is stored row perm[tok]
      rows[t] = kh + tok * D;
    }
#pragma unroll 4
    for (int c = lane; c < D; c += 32) {
      float x[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        x[t] = Elem<T>::to_f(rows[t][c]);
        v[t] = fmaf(x[t], x[t], v[t]);
      }
#pragma unroll
      for (int t = 0; t < 4; ++t) v[8 + t] = fmaf(x[2 * t], x[2 * t + 1], v[8 + t]);
      v[12] = fmaf(x[0], x[3], v[12]);
      v[13] = fmaf(x[4], x[7], v[13]);
      v[14] = fmaf(x[0], x[7], v[14]);
    }
    // All 15 sums over the 32 lanes at once: at every step of the butterfly a lane passes on half of the values it holds and
    // adds its partner's share to the other half, so lane 2i (and 2i+1) ends up with value i after 16 shuffles instead of 75.
    // The additions are those of 15 butterflies.
#pragma unroll
    for (int n = 8; n >= 1; n >>= 1) {
      const bool upper = (lane & (2 * n)) != 0;
#pragma unroll
      for (int i = 0; i < n; ++i) {
        const float send = upper ? v[i] : v[i + n], keep = upper ? v[i + n] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * n);
      }
    }
    const float sum = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
    const float norm = sqrtf(sum + 1e-12f);
    const float na = __shfl_sync(0xffffffffu, norm, 2 * norm_a), nb = __shfl_sync(0xffffffffu, norm, 2 * norm_b);
    const float cosine = sum / (na * nb + 1e-6f);          // lanes 16..29
#pragma unroll
    for (int t = 0; t < 4; ++t) c2 += __shfl_sync(0xffffffffu, cosine, 16 + 2 * t);
    c4 += __shfl_sync(0xffffffffu, cosine, 24) + __shfl_sync(0xffffffffu, cosine, 26);
    c8 += __shfl_sync(0xffffffffu, cosine, 28);
  }
  if (lane == 0) {
    const float s2 = c2 / (float)(bn / 2), s4 = c4 / (float)(bn / 4), s8 = c8 / (float)(bn / 8);
    int r = 1;
    if (s2 > t2) r = 2;
    if (s4 > t4) r = 4;
    if (s8 > t8) r = 8;
    out[bh * nblk + blk] = r;
  }
}

}  // namespace psa

static int ksim_launch(const void* k, const int32_t* perm, int32_t* out, int64_t bh, int64_t seq, int head_dim, int block_n, float t2,
                       float t4, float t8, int dtype, void* stream) {
  using namespace psa;
  PSA_REQUIRE(k && out, PSA_ERR_ARG, "psa_ksim: null pointer");
  PSA_REQUIRE(bh > 0 && bh < 65536 && seq > 0, PSA_ERR_ARG, "psa_ksim: bad shape");
  PSA_REQUIRE(block_n >= 8 && block_n % 8 == 0, PSA_ERR_ARG, "psa_ksim: blocksize must be divisible by 8");
  const int nblk = (int)cdiv64(seq, block_n);
  dim3 grid((nblk + 3) / 4, (unsigned)bh);
  cudaStream_t st = (cudaStream_t)stream;
  PSA_DISPATCH_DTYPE(dtype, T, (ksim_kernel<T><<<grid, 128, 0, st>>>((const T*)k, perm, out, seq, head_dim, block_n, nblk, t2, t4, t8)));
  PSA_CHECK_LAUNCH("psa_ksim");
  return PSA_OK;
}

extern "C" int psa_ksim(const void* k, int32_t* out, int64_t bh, int64_t seq, int head_dim, int block_n, float t2,
                        float t4, float t8, int dtype, void* stream) {
  return ksim_launch(k, nullptr, out, bh, seq, head_dim, block_n, t2, t4, t8, dtype, stream);
}

extern "C" int psa_ksim_perm(const void* k, const int32_t* perm, int32_t* out, int64_t bh, int64_t seq, int head_dim, int block_n,
                             float t2, float t4, float t8, int dtype, void* stream) {
  PSA_REQUIRE(perm, PSA_ERR_ARG, "psa_ksim_perm: null pointer");
  return ksim_launch(k, perm, out, bh, seq, head_dim, block_n, t2, t4, t8, dtype, stream);
}

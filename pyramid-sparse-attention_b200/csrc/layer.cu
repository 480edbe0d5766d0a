// The plug-and-play layer in one call: block scores -> level mask -> tile images -> forward, on caller scratch.
//
// A layer of a short clip is a chain of small kernels, and four entry points with their own operands, scratch and checks
// cost the host more than the kernels take (12 heads x 1560 tokens: 85 us of kernels).  This entry point runs the same
// kernels in the same order; the scores' scratch and the tile images share memory, because the images are only built once
// the scores are there.
#include <algorithm>

#include "psa_common.cuh"
#include "scores.h"

namespace {
size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
size_t po_bytes(int64_t bh, int64_t seq_q, int64_t seq_k, int block_m, int block_n) {
  return align256((size_t)bh * psa::cdiv64(seq_q, block_m) * psa::cdiv64(seq_k, block_n) * 2);
}
}  // namespace

extern "C" size_t psa_layer_scratch_bytes(int64_t bh, int64_t seq_q, int64_t seq_k, int head_dim, int block_m, int block_n, int dtype) {
  if (dtype != PSA_F16 && dtype != PSA_BF16) return 0;
  const size_t img = psa_kv_image_bytes(bh, seq_k, head_dim, block_n);
  const size_t scores = seq_q > 0 ? psa_block_scores_scratch_bytes(bh, seq_q, seq_k, block_m, block_n, dtype) : 0;
  if (img == 0 || scores == 0) return 0;
  return po_bytes(bh, seq_q, seq_k, block_m, block_n) + std::max(scores, 2 * align256(img));
}

extern "C" int psa_layer(const void* q, const void* k, const void* v, const int64_t* idx_q, const int64_t* idx_k, int32_t* mask, void* out,
                         void* scratch, size_t scratch_bytes, int64_t bh, int64_t seq_q, int64_t seq_k, int head_dim, int block_m,
                         int block_n, int tile_n, int threshold_mode, int n_levels, const int32_t* level_values, const int32_t* starts,
                         const int32_t* ends, const float* thresholds, const int32_t* aligns, int min_index, float sm_scale,
                         int compat_quirk, int dtype, int32_t* status, void* stream) {
  using namespace psa;
  PSA_REQUIRE(q && k && v && idx_q && idx_k && mask && out && scratch, PSA_ERR_ARG, "psa_layer: null pointer");
  PSA_REQUIRE(bh > 0 && bh < 65536 && seq_q > 0 && seq_k > 0, PSA_ERR_ARG, "psa_layer: bad shape");
  PSA_REQUIRE((((uintptr_t)q | (uintptr_t)k) & 15) == 0 && ((uintptr_t)scratch & 255) == 0, PSA_ERR_ARG,
              "psa_layer: scratch must be 256-byte aligned, q and k 16-byte aligned");
  const size_t need = psa_layer_scratch_bytes(bh, seq_q, seq_k, head_dim, block_m, block_n, dtype);
  PSA_REQUIRE(need > 0, PSA_ERR_UNSUPPORTED, "psa_layer: needs f16/bf16, head_dim 64/128, block_n 64/128");
  PSA_REQUIRE(scratch_bytes >= need, PSA_ERR_ARG, "psa_layer: scratch too small (%zu bytes)", scratch_bytes);
  const int mq = (int)cdiv64(seq_q, block_m), nk = (int)cdiv64(seq_k, block_n);
  unsigned char* po = (unsigned char*)scratch;
  unsigned char* rest = po + po_bytes(bh, seq_q, seq_k, block_m, block_n);
  int rc = block_scores_idx64(q, k, idx_q, idx_k, po, rest, bh, seq_q, seq_k, head_dim, block_m, block_n, dtype, (cudaStream_t)stream);
  if (rc != PSA_OK) return rc;
  rc = psa_assign_levels(po, mask, bh * mq, nk, dtype, threshold_mode, 1, n_levels, level_values, starts, ends, thresholds, aligns,
                         min_index, 0, stream);
  if (rc != PSA_OK) return rc;
  unsigned char* vimg = rest + align256(psa_kv_image_bytes(bh, seq_k, head_dim, block_n));
  rc = psa_pyramid_kv_images(k, v, rest, vimg, bh, seq_k, head_dim, block_n, dtype, stream);
  if (rc != PSA_OK) return rc;
  return psa_fwd_images(q, rest, vimg, mask, out, bh, seq_q, seq_k, head_dim, block_m, block_n, tile_n, nk + n_levels, sm_scale,
                        compat_quirk, dtype, status, stream);
}

// Mask prediction of one denoising step in one call: block means of q and k, pooled map, line fit, features, line
// selection, mask and work lists: the single stages one after the other on one stream, with their scratch carved out of one
// workspace, so that a caller that goes through an interpreter pays for one call and one scratch allocation instead of ten
// of each.  It matters where the stages themselves are a few microseconds each.  Three launches of the single stages are
// not made here: query and key are pooled together and their means leave split into the terms that the logits read, and
// the solve writes its unknowns where the features go (the prediction of four heads over 8,448 tokens 71 -> 58 us on the
// device, of two heads over 4,096 tokens 67 -> 54: launches and the gaps between them).
#include "common.cuh"

namespace moddit {
namespace {

size_t up256(size_t x) { return (x + 255) / 256 * 256; }

struct Scratch {
  size_t map_ws, mts_ws, mts, solve_ws, selected, total;
};

Scratch layout(int H, int D, int n, int top_k, bool small) {
  Scratch s = {};
  size_t at = 0;
  auto take = [&](size_t bytes) { const size_t p = at; at += up256(bytes); return p; };
  s.map_ws = take(moddit_pooled_map_workspace_bytes(H, n, D));
  s.mts_ws = take(moddit_mts_workspace_bytes(H, n));
  s.mts = take(sizeof(float) * static_cast<size_t>(H) * 3 * n);
  s.solve_ws = take(small ? 0 : moddit_solve_workspace_bytes(H, n));
  const int k = top_k < 3 * n - 1 ? top_k : 3 * n - 1;
  s.selected = take(sizeof(int64_t) * static_cast<size_t>(H) * (k > 0 ? k : 1));
  s.total = at;
  return s;
}

}  // namespace
}  // namespace moddit

using namespace moddit;

extern "C" size_t moddit_predict_workspace_bytes(int H, int nb, int D, int n, int top_k, int small_solve) {
  if (H <= 0 || nb <= 0 || D <= 0 || n <= 0 || top_k <= 0) return 0;
  return layout(H, D, n, top_k, small_solve != 0).total;
}

extern "C" int moddit_predict_lines(const void* q, const void* k, int dtype, int H, int N, int D, int block_size, int first,
                                    int n, int blocks_per_frame, int mask_layout, float scale, const void* factor,
                                    int small_solve, const float* last_c, const float* last_d, int top_k, float predict_T,
                                    float mode_threshold, void* map_f16, float* d, float* c, float* b_d, int32_t* modes,
                                    uint8_t* mask, int32_t* counts, int32_t* entries, int32_t* order, void* workspace,
                                    size_t workspace_bytes, void* stream) {
  // what the stages cannot see for themselves; everything else they check
  clear_error();
  MODDIT_CHECK_ARG(factor && d && c && b_d && modes && mask && counts && entries, "predict_lines: null pointer");
  MODDIT_CHECK_ARG(H > 0 && N > 0 && D > 0 && n > 0 && top_k > 0 && blocks_per_frame > 0, "predict_lines: sizes must be positive");
  if (block_size != 64 && block_size != 128)
    return fail(MODDIT_E_UNSUPPORTED, "predict_lines: block_size must be 64 or 128, got %d", block_size);
  const int nb = ceil_div(N, block_size);
  MODDIT_CHECK_ARG(first >= 0 && n <= nb && first <= nb - n, "predict_lines: video region [%d, %d + %d) exceeds %d blocks",
                   first, first, n, nb);
  // The mask stage places the video region by its layout alone, and the list stage reads nb x nb blocks of what it wrote.
  if (mask_layout == MODDIT_LAYOUT_WAN) {
    MODDIT_CHECK_ARG(first == 0 && n == nb, "predict_lines: wan layout needs first == 0 and n == %d (got %d, %d)", nb, first, n);
  } else if (mask_layout == MODDIT_LAYOUT_HUNYUAN) {
    MODDIT_CHECK_ARG(first == 0, "predict_lines: hunyuan layout needs first == 0 (got %d)", first);
  } else if (mask_layout == MODDIT_LAYOUT_COGVIDEOX) {
    MODDIT_CHECK_ARG(first + n == nb, "predict_lines: cogvideox layout needs first + n == %d (got %d, %d)", nb, first, n);
  } else {
    return fail(MODDIT_E_ARG, "predict_lines: unknown layout %d", mask_layout);
  }
  const Scratch s = layout(H, D, n, top_k, small_solve != 0);
  if (workspace == nullptr || workspace_bytes < s.total || !aligned16(workspace))
    return fail(MODDIT_E_WORKSPACE, "predict_lines: %zu bytes of 16-byte aligned workspace needed", s.total);
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  float* mts = reinterpret_cast<float*>(ws + s.mts);
  int64_t* selected = reinterpret_cast<int64_t*>(ws + s.selected);
  if (int rc = pooled_map_of_blocks(q, k, dtype, H, N, D, block_size, first, n, scale, map_f16, ws + s.map_ws, as_stream(stream)))
    return rc;
  if (int rc = moddit_mts(map_f16, nullptr, nullptr, 0, 0, 0, nullptr, H, n, blocks_per_frame, mts, ws + s.mts_ws,
                          moddit_mts_workspace_bytes(H, n), stream))
    return rc;
  if (int rc = solve_features(mts, factor, small_solve != 0, H, n, mode_threshold, d, c, b_d, modes, ws + s.solve_ws,
                              moddit_solve_workspace_bytes(H, n), stream))
    return rc;
  if (int rc = moddit_select_lines(c, d, last_c, last_d, H, n, top_k, predict_T, selected, stream)) return rc;
  const int chosen = top_k < 3 * n - 1 ? top_k : 3 * n - 1;
  const int text_blocks = mask_layout == MODDIT_LAYOUT_COGVIDEOX ? first : nb - n;
  if (int rc = moddit_mask_from_lines(selected, chosen, modes, H, n, blocks_per_frame, mask_layout, text_blocks,
                                      mask_layout == MODDIT_LAYOUT_WAN ? n : nb, mask, stream))
    return rc;
  return moddit_tile_lists(mask, H, nb, nb, block_size, N, nb, counts, entries, order, stream);
}

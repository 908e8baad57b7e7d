// Launch geometry as plain functions of the sizes: what fb_pass.cu and fb_spec.cu launch, how the decode kernel cuts its phases, and what a host-side test can
// ask. No CUDA here (the device code uses the constexpr ones).
// Times: engine calls back to back.
#pragma once

namespace fb {

// rows of a tile of the streaming layout
constexpr int tile_rt(int k) { return (k / 128) % 2 == 0 ? 8 : 16; }
// the first of the rows of a phase that CTA b of G owns (they end where those of b + 1 start); `unit` rows stay together
constexpr int cta_first_row(int rows, int unit, int b, int G) {
  const int r = (int)((long long)((rows + unit - 1) / unit) * b / G) * unit;
  return r < rows ? r : rows;
}
// Columns of the O projection a rank reads: its heads' columns widened to whole int4 groups (a rank of the 3B-class
// model split 8 ways owns 320 columns = 2.5 groups: it reads 384 and takes zeros for its neighbour's 64). off: where its own start.
struct OWindow { int ko, off; };
constexpr OWindow o_window(int width, int rank) {
  const int start = rank * width, lo = start / 128 * 128, hi = (start + width + 127) / 128 * 128;
  return OWindow{hi - lo, start - lo};
}
// ... as pairs of tagged words (four columns a pair; a head is a multiple of eight): the only ones that this rank's attention publishes
struct WordPairs { int first, end; };
constexpr WordPairs o_words(int width, int off) { return WordPairs{off / 4, (off + width) / 4}; }

constexpr int kTcRowBlock = 128;  // weight rows of a GEMM's work item

// One GEMM of an M-token pass. nt: tokens that a tile can hold. 16, 32, 64: one tile, v_gemm_tl<nt>. 128 with nsplit > 1: v_gemm_tl<128>. 128 or 192
// with nsplit 1: the persistent kernel, v_gemm_tc<nt>.
struct GemmGeometry {
  int nt, ntok, ntile, nsplit;    // ntok: tokens of a tile (a multiple of 16); ntile: tiles; nsplit: CTAs of a cluster that share K
};

inline int token_tile(int M) { return M <= 16 ? 16 : (M <= 32 ? 32 : (M <= 64 ? 64 : 128)); }

inline GemmGeometry cut_tokens(int M, int nt) {                 // tiles of up to nt tokens, cut evenly
  GemmGeometry g{nt, 0, (M + nt - 1) / nt, 1};
  g.ntok = ((M + g.ntile - 1) / g.ntile + 15) / 16 * 16;
  return g;
}

inline GemmGeometry gemm_geometry(int M, int rows, int k, bool zeros, int sms) {
  GemmGeometry g = cut_tokens(M, token_tile(M));
  const int nrb = (rows + kTcRowBlock - 1) / kTcRowBlock, items = nrb * g.ntile, groups = k / 128;
  if (g.nt <= 64) {
    // trees: two CTAs share an SM; matrices with few row blocks are cut while all CTAs are resident at once and each keeps two groups to multiply
    while (g.nsplit < 8 && items * g.nsplit * 2 <= 2 * sms && groups / (g.nsplit * 2) >= 2 && g.nt / (g.nsplit * 2) >= 2) g.nsplit *= 2;
    return g;
  }
  // The same for the tiles of a prompt, one CTA per SM, at least four groups each. Clusters of eight fit only in 120 of 148 SMs: at most four.
  // Not split: the persistent kernel, which overlaps an item's epilogue with the next item. All prompts in it / split: 70 / 100 / 128 / 180 / 250 / 300 / 384
  // tokens of the 3B shape 3214 / 3411 / 3579 / 3594 / 4153 / 4282 / 4603 -> 2592 / 2678 / 2773 / 3612 / 3936 / 4036 / 4303 us, 100 / 180 / 250 of the 8B shape
  // 4300 / 4605 / 5569 -> 3239 / 4075 / 5023. Two tiles gain least just above 128 tokens: -0.7 to +2 % at 129 to 190 tokens
  // of the 3B shapes.
  while (g.nsplit < 4 && items * g.nsplit * 2 <= sms && groups / (g.nsplit * 2) >= 4) g.nsplit *= 2;
  if (g.nsplit > 1 || zeros) return g;                           // no 192-token tiles for zero points: tensor memory is full
  // 192-token tiles where they need fewer than 3/4 of the rounds of items that 128-token tiles need (a round of them takes about 4/3 of the time).
  // 180 / 300 / 520 / 725 / 900 tokens of the 3B shape 3712 / 4167 / 5911 / 6800 / 9049 us with 128-token tiles alone, 3612 / 4036 / 5288 / 6312 / 8107 with the
  // rule; 520 / 725 of the 8B shape 10802 / 13396 -> 8689 / 11576. Nowhere slower from 65 to 1000 tokens.
  const GemmGeometry w = cut_tokens(M, 192);
  const int rounds128 = (items + sms - 1) / sms, rounds192 = (nrb * w.ntile + sms - 1) / sms;
  return rounds192 * 4 < rounds128 * 3 ? w : g;
}

// The attention of an M-token pass behind `pos` cached positions. Few row tiles (16 query rows: r query heads of a kv head per token): one or two a
// CTA, its warps share the span's positions instead; four where that many CTAs would not fit the GPU with four spans each. Spans (CTAs of a
// cluster): a power of two up to 8 while there is a stage of 64 positions for each and all CTAs are resident at once (with one CTA per SM the GPU
// holds 15 clusters of 8 -- the 16th waited for a second wave, 22 us instead of 12 -- but 36 of 4).
struct AttnGeometry {
  int rt, groups, nspan, span;    // row tiles of a CTA, row groups of a kv head, spans, positions of a span
};

inline AttnGeometry attn_geometry(int M, int pos, int n_kv, int r, int sms) {
  const int tiles = (M * r + 15) / 16, per4 = sms / (4 * n_kv), stages = (pos + M + 63) / 64;
  AttnGeometry a{tiles <= per4 ? 1 : (tiles <= 2 * per4 ? 2 : 4), 0, 1, 0};
  a.groups = (tiles + a.rt - 1) / a.rt;
  const int clusters = n_kv * a.groups;
  while (a.nspan < 8 && a.nspan * 2 <= stages && clusters * a.nspan * 2 <= (a.nspan == 4 ? sms * 2 / 3 : sms)) a.nspan *= 2;
  a.span = (stages + a.nspan - 1) / a.nspan * 64;
  return a;
}

// A linear of the draft head: `blocks` CTAs of its rows, K in `chunks` of 32 columns, nt tiles of 8 tokens. CTAs of a cluster that share K: while all
// CTAs are resident at once (three per SM for up to eight tokens, else two) and every warp keeps two chunks.
constexpr int kDraftSplits = 3;
constexpr int kDraftWarps = 8;
inline int draft_splits(int blocks, int chunks, int nt, int sms) {
  const int slots = sms * (nt == 1 ? 3 : 2);
  int ks = 1;
  while (ks < kDraftSplits && blocks * (ks + 1) <= slots && chunks >= 2 * kDraftWarps * (ks + 1)) ks++;
  return ks;
}

}  // namespace fb

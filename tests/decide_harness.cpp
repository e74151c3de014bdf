// Host build of the selector's decision rules (csrc/fftopk_decide.h) for the CPU tests: the same
// header the kernels include, compiled by g++ and exposed as plain C functions.
#include "fftopk_decide.h"

#include <vector>

using namespace fftopk;

extern "C" {

uint32_t dh_key_from_bits(uint32_t bits) { return fftopk_key_from_bits(bits); }
uint32_t dh_bits_from_key(uint32_t key) { return fftopk_bits_from_key(key); }
uint32_t dh_sample_lower_rank(uint32_t k, uint32_t n_s, float len) { return sample_lower_rank(k, n_s, len); }
uint32_t dh_sample_upper_rank(uint32_t k, uint32_t n_s, float len) { return sample_upper_rank(k, n_s, len); }
int dh_sample_bin_too_coarse(uint32_t cnt, uint32_t total, float len, uint32_t k, float factor) {
  return sample_bin_too_coarse(cnt, total, len, k, factor) ? 1 : 0;
}
uint32_t dh_sample_digit(uint32_t bits) { return sample_digit(bits); }
uint32_t dh_sample_digit_low(uint32_t bin) { return sample_digit_low(bin); }
uint32_t dh_sample_digit_high(uint32_t bin) { return sample_digit_high(bin); }
int dh_sample_admits_too_much(uint32_t admitted, uint32_t total, float len, uint32_t room) {
  return sample_admits_too_much(admitted, total, len, room) ? 1 : 0;
}
int dh_sample_piece(void) { return kSamplePiece; }
uint32_t dh_sample_piece_start(uint32_t gi, uint32_t piece, int log_pieces, uint32_t off) {
  return sample_piece_start(gi, piece, log_pieces, off);
}
int dh_sample_log_batches(int len, uint32_t k) { return sample_log_batches(len, k); }
int dh_gather_region(int cand_cap, int list_cap, int ctas) { return gather_region(cand_cap, list_cap, ctas); }
int dh_fine_histogram_usable(int built, uint32_t total, uint32_t group) {
  return fine_histogram_usable(built != 0, total, group) ? 1 : 0;
}
uint32_t dh_guess_edge_bits(uint32_t gkey) { return guess_edge_bits(gkey); }
uint32_t dh_guess_low_key(uint32_t gkey) { return guess_low_key(gkey); }
int dh_sampled_attempt_ok(uint32_t over, uint32_t admitted, uint32_t k, uint32_t room) {
  return sampled_attempt_ok(over, admitted, k, room) ? 1 : 0;
}
// One guess from a sample (n float bit patterns; n_s of them count, as in the kernel), made step by step
// the way the selection kernel makes it. out: guess, focus, flags, second looks. Returns 0, or -1 when
// the second looks do not come to an end.
int dh_sample_guess(const uint32_t* bits, uint32_t n, uint32_t n_s, float len, uint32_t k, uint32_t room, int whole, uint32_t* out) {
  std::vector<uint32_t> hist(kSampleBins, 0u);
  uint32_t guess = 0u, focus = 0u, flags = 0u, width = 0u, above0 = 0u, rest = 0u, cnt0 = 0u;
  // the bin of rank `need` from the top
  auto pick = [&](uint32_t need, uint32_t& above, uint32_t& cnt) {
    above = 0u;
    for (int b = kSampleBins - 1; b >= 0; --b) {
      cnt = hist[b];
      if (above < need && need <= above + cnt) return b;
      above += cnt;
    }
    return -1;
  };
  auto weigh = [&](uint32_t low, uint32_t w, uint32_t above, uint32_t cnt, uint32_t r, uint32_t parent) {
    const uint32_t f = weigh_guess(w, above, cnt, parent, n_s, len, k, 2.0f, room);
    if (f & kGuessCopies) focus = low + w - 1u;
    guess = low;
    flags = f & ~kGuessCopies;
    if (f & kGuessCoarse) width = w, cnt0 = cnt, above0 = above, rest = r;
  };
  const SampleRanks ranks = sample_ranks(whole != 0, k, n_s, len);
  for (uint32_t i = 0; i < n; ++i) ++hist[sample_digit(bits[i])];
  uint32_t above, cnt;
  int b = pick(ranks.need, above, cnt);
  if (b >= 0) weigh(sample_digit_low(b), sample_digit_width(b), above, cnt, ranks.need - above, 0xffffffffu);
  b = pick(ranks.need_hi, above, cnt);
  if (b >= 0) focus = sample_digit_high(b);
  uint32_t looks = 0u;
  for (; flags & kGuessCoarse; ++looks) {
    if (looks == 8u) return -1;
    const uint32_t low = guess, w = width, a0 = above0, r = rest, c0 = cnt0;
    const int shift = second_look_shift(w);
    hist.assign(kSampleBins, 0u);
    flags = kGuessGiveUp;
    for (uint32_t i = 0; i < n; ++i) {
      const uint32_t off = fftopk_key_from_bits(bits[i]) - low;
      if (off < w) ++hist[(off >> shift) & (uint32_t)(kSampleBins - 1)];
    }
    b = pick(r, above, cnt);
    if (b >= 0) weigh(low + ((uint32_t)b << shift), 1u << shift, a0 + above, cnt, r - above, c0);
  }
  out[0] = guess, out[1] = focus, out[2] = flags, out[3] = looks;
  return 0;
}
int dh_finish_bins(void) { return kFinishBins; }
// the digit rule on 64-bit composites (key << 32 | inverted index) ...
int dh_finish_shift(uint64_t lo, uint64_t focus) { return make_field_digit<uint64_t>(lo, focus).shift; }
int dh_finish_key_only(uint64_t lo, uint64_t focus) { return dh_finish_shift(lo, focus) >= 32 && (uint32_t)lo == 0u ? 1 : 0; }
uint32_t dh_finish_digit(uint64_t lo, uint64_t focus, uint64_t c) { return make_field_digit<uint64_t>(lo, focus).of(c); }
void dh_finish_bin_range(uint64_t lo, uint64_t focus, uint64_t cap, int t, uint64_t* t_lo, uint64_t* t_hi) {
  const FieldDigit<uint64_t> dg = make_field_digit<uint64_t>(lo, focus);
  *t_lo = dg.bin_low((uint32_t)t);
  *t_hi = dg.bin_high((uint32_t)t, cap);
}
// ... and on their keys
uint32_t dh_finish_digit_of_key(uint64_t lo, uint64_t focus, uint32_t key) {
  return make_key_digit((uint32_t)(lo >> 32), (uint32_t)(focus >> 32)).of(key);
}
void dh_key_bin_range(uint32_t lo, uint32_t focus, uint32_t cap, uint32_t t, uint32_t* t_lo, uint32_t* t_hi) {
  const KeyDigit dg = make_key_digit(lo, focus);
  *t_lo = dg.bin_low(t);
  *t_hi = dg.bin_high(t, cap);
}
uint32_t dh_key_digit(uint32_t lo, uint32_t focus, uint32_t v) { return make_key_digit(lo, focus).of(v); }
uint64_t dh_single_key_floor(uint64_t lo, int idx_bits) { return (lo & 0xffffffff00000000ull) | inverted_index_floor(idx_bits); }
int dh_lone_segment(int list_cap, int threads) { return lone_segment(list_cap, threads); }
int dh_lone_room(int list_cap, int threads) { return lone_room(list_cap, threads); }
int dh_lone_regs(int threads) { return lone_regs(threads); }
int dh_rows_inside(uint64_t score, int64_t row_stride, int32_t B, int64_t L, int element_bytes, uint64_t base, uint64_t size) {
  return rows_inside(score, row_stride, B, L, element_bytes, base, size) ? 1 : 0;
}
int dh_lone_edge_warp(int threads) { return lone_edge_warp(threads); }

// Walks every CTA's run of tiles the way the fused indexer's producer does (tile_run, tile_row_at,
// then tile_segment row after row) and adds, for every (row, row-local tile) the CTAs visit, one to
// visits[first_tile[row] + tile]. segs_out receives the number of segments each CTA went through.
// Returns 0, or a negative code when a walk leaves the table.
int dh_walk_tile_split(const uint32_t* first_tile, int rows, uint32_t ctas, uint32_t* visits, uint32_t* segs_out) {
  const uint32_t total = first_tile[rows];
  for (uint32_t c = 0; c < ctas; ++c) {
    const TileRun run = tile_run(total, ctas, c);
    if (run.g1 < run.g0 || run.g1 > total) return -1;
    uint32_t segs = 0;
    if (run.g0 < run.g1) {
      int row = tile_row_at(first_tile, rows, run.g0);
      for (uint32_t g = run.g0; g < run.g1; ++row) {
        if (row >= rows) return -2;
        int t_lo, n;
        if (!tile_segment(first_tile[row], first_tile[row + 1] - first_tile[row], g, run.g1, t_lo, n)) continue;
        if (n <= 0 || t_lo < 0 || (uint32_t)(t_lo + n) > first_tile[row + 1] - first_tile[row]) return -3;
        for (int i = 0; i < n; ++i) ++visits[first_tile[row] + (uint32_t)(t_lo + i)];
        g += (uint32_t)n;
        ++segs;
      }
    }
    segs_out[c] = segs;
  }
  return 0;
}
void dh_tile_run(uint32_t total, uint32_t ctas, uint32_t cta, uint32_t* g0, uint32_t* g1) {
  const TileRun r = tile_run(total, ctas, cta);
  *g0 = r.g0;
  *g1 = r.g1;
}

}  // extern "C"

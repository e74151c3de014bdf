// Decision rules of the selector that do not depend on where they run: the sample-rank bounds,
// the choice between the two sample histograms, the float edge of a key guess, the digit rule of
// the finish and the conditions under which the sampled attempt is abandoned. The kernels call
// these functions; a host compiler can compile them too (tests drive them with generated inputs
// where no GPU is present).
#pragma once
#include <math.h>
#include <stdint.h>

#include "fftopk_key.h"

#if defined(__CUDACC__)
#define FFTOPK_DECIDE_HD __host__ __device__ __forceinline__
#else
#define FFTOPK_DECIDE_HD inline
#endif

namespace fftopk {

constexpr int kFinishBits = 11;  // digit width of the single-CTA finish
constexpr int kFinishBins = 1 << kFinishBits;

FFTOPK_DECIDE_HD int clz64(uint64_t v) {
#if defined(__CUDA_ARCH__)
  return __clzll((long long)v);
#else
  return v ? __builtin_clzll(v) : 64;
#endif
}

// ---------------------------------------------------------------------------------------------
// Sample ranks. A row of `len` elements is sampled at n_s positions; m = k * n_s / len of the
// sample are expected among the row's k largest. The element of sample rank
//     lower_rank = m + 5 sqrt(m) + 14   (capped at n_s)
// is, except with probability of the order 1e-6, not larger than the row's k-th largest: filtering
// with it admits at least k elements. The mirror image,
//     upper_rank = m - 5 sqrt(m) - 14   (0 when there is no such rank),
// is a sample element the k-th largest does not exceed with the same confidence.
// ---------------------------------------------------------------------------------------------
FFTOPK_DECIDE_HD uint32_t sample_lower_rank(uint32_t k, uint32_t n_s, float len) {
  const float m = (float)k * (float)n_s / len;
  const uint32_t rk = (uint32_t)(m + 5.0f * sqrtf(m) + 14.0f);
  return rk < n_s ? rk : n_s;
}

FFTOPK_DECIDE_HD uint32_t sample_upper_rank(uint32_t k, uint32_t n_s, float len) {
  const float m = (float)k * (float)n_s / len;
  const float rk = m - 5.0f * sqrtf(m) - 14.0f;
  return rk >= 1.0f ? (uint32_t)rk : 0u;
}

// Where the sample lies. A row too long to be read completely is sampled in pieces of 32 consecutive
// elements (eight granules of four): the `gi` granules that lie completely inside the row are cut into
// 2^log_pieces equal stretches, and every stretch holds one piece near its start: four neighbouring
// pieces 0 to 3 lines behind it, so that a row with a period of up to 128 elements (a page of keys, say) is
// seen at every phase. (Places at random within the stretch see any period; they cost 64 rows of 128K 0.25 us of
// 15.1 per call.)
// `off` is the first granule's position within eight of the address space. Pieces start on such a boundary -
// a 128-byte line of fp32 -, so that the 32 lanes of a load touch four lines, as many as one slab of 512 bytes.
// The rank bounds above take every sample element for an independent one, and neighbouring logits are
// alike in practice: the shorter the pieces, the closer that is to the truth. Share of rows of 98,304
// elements for which fewer than k elements pass (150 rows of a kind), with slabs of 128 elements / pieces of
// 32 / of 8: one window of 2,048 consecutive winners 27 / 0 / 0 %; 90 % of the variance smooth over 64
// positions 13 / 5 / 0 %, over 256 positions 22 / 4 / 0 %. Pieces of 8 touch 16 lines per load, which costs every
// row: 2,048 rows of 32K elements 112 us instead of 104, one row of 1M 16.0 instead of 15.0.
constexpr int kSamplePiece = 8;  // granules
FFTOPK_DECIDE_HD uint32_t sample_piece_start(uint32_t gi, uint32_t piece, int log_pieces, uint32_t off) {
  const uint32_t play = (gi >> log_pieces) - (uint32_t)kSamplePiece;  // (a stretch is longer than a piece)
  const uint32_t shift = (piece & 3u) * (uint32_t)kSamplePiece;
  const uint32_t at = (uint32_t)(((uint64_t)gi * piece) >> log_pieces) + (shift < play ? shift : play);
  const uint32_t line = (at + off) & ~(uint32_t)(kSamplePiece - 1);
  return line > off ? line - off : 0u;
}

// How much of a row is sampled: 2^log batches of 8K elements. With m of them expected among the k largest,
// the rank bound admits about k (1 + 5 / sqrt(m) + 14 / m) elements, so the sample grows with the row:
// 16K elements beyond 256K, and twice as many each time a row beyond 4M (2M for k beyond 2048) doubles. For
// k = 2048 m stays above 8, and no more than 9.3K elements are expected to pass (a cluster's buffer holds 16K, a lone CTA's list
// 10K or 12K). (With 16K elements for rows of any length, a row beyond
// 10M passed more than a cluster's buffer holds and went through three full-histogram rounds: one row of
// 12M 273 us instead of 43, of 32M 760 instead of 193. With twice the sample, from 2M on, 12M took 48 us.)
FFTOPK_DECIDE_HD int sample_log_batches(int len, uint32_t k) {
  return len <= 262144 ? 0 : 1 + 64 - clz64((uint64_t)((uint32_t)(len - 1) >> (k > 2048u ? 21 : 22)));
}

// A second sample round sharpens the guess when the guessed bin alone would admit more than
// factor * k row elements (estimated from the bin's share of the sample).
FFTOPK_DECIDE_HD bool sample_bin_too_coarse(uint32_t bin_count, uint32_t sample_total, float len, uint32_t k,
                                            float factor) {
  // (no division: one thread of a CTA decides this while the others wait)
  return (float)bin_count * len > factor * (float)k * (float)(sample_total ? sample_total : 1u);
}

// ---------------------------------------------------------------------------------------------
// Sample digit: a monotone map of the float's bits onto 4096 bins that is fine where logits live, and
// costs six integer instructions. Magnitudes in [2^-16, 2^16) get 64 bins per octave (bits [30:17]),
// for either sign; smaller ones share the two bins around zero, larger ones (and NaN) the outermost
// two. A bin then holds about 1/64 octave of values: the guess made on it admits few elements beyond
// the sampling margin (a plain 12-bit digit has 8 bins per octave, which on crowded rows - sums over
// heads, all of one sign and magnitude - costs thousands of extra candidates or a second look).
// -0 falls into the bin just below zero, although its key is the first one above it: a second look at that
// bin takes it in (sample_digit_width). A NaN of negative sign counts as the smallest value here and is
// the largest key: the guess then lies lower than it need. The sample only makes a guess, which is checked
// afterwards.
// ---------------------------------------------------------------------------------------------
constexpr int kSampleBins = 4096;
constexpr int kSampleShift = 17;
constexpr int32_t kSampleBase = 111 << 23;              // 2^-16
constexpr int32_t kSampleSpan = (32 << 23) - 1;         // 32 octaves
// ... as the byte offset of the bin's counter from that of the bin above zero: what a histogram update wants
FFTOPK_DECIDE_HD int32_t sample_digit_offset(uint32_t bits) {
  const int32_t sign = (int32_t)bits >> 31;
  const int32_t mag = (int32_t)(bits & 0x7fffffffu);
#if defined(__CUDA_ARCH__)
  const int32_t d = __viaddmin_s32_relu(mag, -kSampleBase, kSampleSpan);
#else
  const int32_t a = mag - kSampleBase;
  const int32_t d = a < 0 ? 0 : (a < kSampleSpan ? a : kSampleSpan);
#endif
  return ((d >> (kSampleShift - 2)) ^ sign) & ~3;
}
FFTOPK_DECIDE_HD uint32_t sample_digit(uint32_t bits) { return (uint32_t)((sample_digit_offset(bits) >> 2) + kSampleBins / 2); }
// the smallest key of a bin (a bin ends where the next one starts; the last one holds every key above)
FFTOPK_DECIDE_HD uint32_t sample_digit_low(uint32_t bin) {
  if (bin >= (uint32_t)kSampleBins / 2) {
    const uint32_t e = bin - kSampleBins / 2;
    return 0x80000000u | (e == 0u ? 0u : (uint32_t)kSampleBase + (e << kSampleShift));
  }
  const uint32_t e = kSampleBins / 2 - 1 - bin;  // magnitudes [e, e + 1) of the negative side
  return e == (uint32_t)kSampleBins / 2 - 1 ? 0u : ~(0x80000000u | ((uint32_t)kSampleBase + ((e + 1u) << kSampleShift))) + 1u;
}
FFTOPK_DECIDE_HD uint32_t sample_digit_high(uint32_t bin) {
  return bin == (uint32_t)kSampleBins - 1 ? 0xffffffffu : sample_digit_low(bin + 1u) - 1u;
}

// the number of keys, from the smallest on, that the elements of a bin may have
FFTOPK_DECIDE_HD uint32_t sample_digit_width(uint32_t bin) {
  return sample_digit_high(bin) - sample_digit_low(bin) + (bin == (uint32_t)kSampleBins / 2 - 1 ? 2u : 1u);
}

// A guess whose share of the sample stands for a quarter more row elements than there is room for is
// given up before the row is read for it (rows with thousands of copies of one value).
FFTOPK_DECIDE_HD bool sample_admits_too_much(uint32_t admitted, uint32_t sample_total, float len, uint32_t room) {
  return (float)admitted * len > 1.25f * (float)room * (float)(sample_total ? sample_total : 1u);
}

// The ranks sought in a sample of n_s elements: the guess is the bin of rank `need` (0: there is none,
// and no element is filtered out), and the finish is focused below the bin of rank `need_hi`. Of a row
// that was read completely (but for the granules that straddle its ends) rank k itself.
struct SampleRanks {
  uint32_t need, need_hi;
};
FFTOPK_DECIDE_HD SampleRanks sample_ranks(bool whole, uint32_t k, uint32_t n_s, float len) {
  if (whole) return SampleRanks{k <= n_s ? k : 0u, k <= n_s ? k : 0u};
  const uint32_t hi = sample_upper_rank(k, n_s, len);
  return SampleRanks{sample_lower_rank(k, n_s, len), hi > 1u ? hi : 1u};
}

// What to do about a guess: a bin of `width` keys that holds `cnt` sample elements, `above` of them lie
// above it, and the bin it was cut out of holds `parent`.
//   look again   the bin stands for more than factor * k row elements - values crowded into a sliver of
//                the key space -, and cutting it thins it out: not if it still holds most of the bin it
//                was cut out of, which are then copies of one value. (Below factor * k, carrying the
//                extra candidates is cheaper than the second look.)
//   give up      it admits far more than there is room for: not worth the pass
//   copies       the threshold is the value the bin holds copies of: the finish need not search above it
constexpr uint32_t kGuessCoarse = 1u, kGuessGiveUp = 2u, kGuessCopies = 4u;
FFTOPK_DECIDE_HD uint32_t weigh_guess(uint32_t width, uint32_t above, uint32_t cnt, uint32_t parent, uint32_t n_s,
                                      float len, uint32_t k, float factor, uint32_t room) {
  const bool copies = cnt >= parent - parent / 4u;
  if (width > 1u && !copies && sample_bin_too_coarse(cnt, n_s, len, k, factor)) return kGuessCoarse;
  if (sample_admits_too_much(above + cnt, n_s, len, room)) return kGuessGiveUp;
  return copies ? kGuessCopies : 0u;
}
// ... and how a second look cuts a bin of `width` keys into at most kSampleBins (key offset >> shift)
FFTOPK_DECIDE_HD int second_look_shift(uint32_t width) {
  const int bits = 64 - clz64((uint64_t)(width - 1u));
  return bits > 12 ? bits - 12 : 0;
}

// The finer sample histogram (key bits [27:16]) may replace the coarse one (bits [31:20]) only if
// one group of four consecutive coarse super-bins - one value of the key's top four bits - holds
// the whole sample.
FFTOPK_DECIDE_HD bool fine_histogram_usable(bool built, uint32_t sample_total, uint32_t group_total) {
  return built && sample_total > 0u && group_total == sample_total;
}

// Lower edge of a key guess as float bits: key(x) >= gkey <=> !(x < edge), NaN included. Keys
// outside the range that real values map to (below -inf's key, above +inf's) give -inf: the filter
// then admits everything, which only lengthens the lists.
FFTOPK_DECIDE_HD bool guess_has_edge(uint32_t gkey) { return gkey > 0x007fffffu && gkey <= 0xff800000u; }
FFTOPK_DECIDE_HD uint32_t guess_edge_bits(uint32_t gkey) {
  return guess_has_edge(gkey) ? fftopk_bits_from_key(gkey) : 0xff800000u;
}
// ... and the smallest key the filter can then admit (what the finish may assume as its lower bound)
FFTOPK_DECIDE_HD uint32_t guess_low_key(uint32_t gkey) { return guess_has_edge(gkey) ? gkey : 0u; }

// After the filter: keep the sampled attempt only if no list overflowed, at least k elements were
// admitted and they fit where they were gathered; otherwise the full-histogram path takes over.
FFTOPK_DECIDE_HD bool sampled_attempt_ok(uint32_t overflowed, uint32_t admitted, uint32_t k, uint32_t room) {
  return overflowed == 0u && admitted >= k && admitted <= room;
}

// The gather buffer of a cluster: every CTA has a region of its own, which it fills without asking for
// slots, and what does not fit there goes behind the last region, for a remote atomic per CTA. The regions
// leave room behind them for 4/3 of a whole list of any one CTA - what a window of recent keys fills, or a sorted
// row -, and take no more than three quarters of the buffer. (With three quarters whatever the list, one CTA
// could hand on 4,864 candidates at 16 CTAs per row and 2,112 at 8 in the throughput plan, and such rows
// went through full histograms. The walk over the part behind is shared by all warps of the finish, so
// they are also faster with small regions: 2,048 consecutive winners in a row of 98,305 elements 11.1 us
// instead of 12.0. One row of 1M elements leaves some 300 candidates per CTA, for 546 slots.)
FFTOPK_DECIDE_HD int gather_region(int cand_cap, int list_cap, int ctas) {
  const int most = (cand_cap - cand_cap / 4) / ctas;
  const int room = (cand_cap - list_cap - list_cap / 3) / (ctas > 1 ? ctas - 1 : 1);
  return room < 0 ? 0 : (most < room ? most : room) & ~15;  // (whole 128-byte lines: 3 % of a call at k = 4096, 1M)
}
// ... and of the list of a cluster's CTA: the warps' segments, and an area behind them for what a warp's segment does not
// hold. Where all candidates of a row may lie in one CTA's shard, a few thousand consecutive elements fall
// on the warps unevenly: a quarter of a short list (the throughput plan's), else an eighth. (A quarter of
// a long one as well cost 64 rows with 6,500 copies of the threshold 26.3 us instead of 24.4.)
FFTOPK_DECIDE_HD int list_spill(int list_cap) { return list_cap / (list_cap >= 4096 ? 8 : 4); }

// A lone CTA's segments hold row indices (words, in the memory of list_cap composites), and the finish has their keys in
// registers: so many per thread, and no more candidates per warp than that. There is no spill area: one warp over its
// segment sends the row through full histograms, and its call waits for it. So a segment has to hold what a guess may
// admit of one warp's share - up to 9.5K expected per row, and that unevenly -, or many copies of the threshold. With 8
// and 16 keys a thread (8,192 a row) most calls had such a row; us per call then / now: 100 rows of 160K, k = 4096, 78 / 19;
// 80 of 512K, k = 4096, 189 / 39; 40 of 2M, overlapping, 150 / 42; 160 of 256K with 6,500 copies 253 / 57. Rows that need fewer
// registers do not pay for the others (2,048 rows of 32K, k = 2048, 80.7 / 80.2). A row that gets 256 threads fits as it is.
FFTOPK_DECIDE_HD constexpr int lone_regs(int threads) { return threads >= 1024 ? 12 : (threads >= 512 ? 20 : 16); }
FFTOPK_DECIDE_HD int lone_segment(int list_cap, int threads) {
  const int own = 2 * list_cap / (threads / 32);
  return own < 32 * lone_regs(threads) ? own : 32 * lone_regs(threads);
}
// The warp that reads the granules a row's ends cut through (up to three elements each): the one with the fewest others. All
// of a row of up to 4,096 elements may pass - rows of mostly zeros -, and 256 threads hold 512 a warp: with the ends in the
// first two warps most rows that were not 16-byte aligned overflowed (2,048 rows of 4,095, 70 % zeros: 163 us, now 96.5).
FFTOPK_DECIDE_HD constexpr int lone_edge_warp(int threads) { return threads / 32 - 1; }
// ... the whole list in candidates (words)
FFTOPK_DECIDE_HD int lone_room(int list_cap, int threads) { return threads / 32 * lone_segment(list_cap, threads); }
// ... and what a guess is weighed against (sample_admits_too_much tries a quarter more, since the sample's share is an
// estimate): less than the larger lists hold, because the warps' shares differ. Rows with copies of the threshold, us for 160
// rows of 128K / 256K with weights of 8,192, this and 10,240: 7,500 copies 36 / 111 (given up for nothing),
// 36 / 59, 36 / 59; 12,000 copies 195 / 356, 194 / 359, 206 / 385 (read for nothing).
FFTOPK_DECIDE_HD int lone_room_weighed(int list_cap, int threads) {
  const int room = lone_room(list_cap, threads);
  return room < 9216 ? room : 9216;
}

// ---------------------------------------------------------------------------------------------
// Rows that are asked for in L2 ahead of time are asked for up to a length that may be out of date, so up to L: more than the call
// reads, and more than a caller has to have. The request is made only where B rows of L elements lie inside the allocation
// that the first of them lies in ([base, base + size), addresses in bytes).
// ---------------------------------------------------------------------------------------------
FFTOPK_DECIDE_HD bool rows_inside(uint64_t score, int64_t row_stride, int32_t B, int64_t L, int element_bytes, uint64_t base, uint64_t size) {
  if (B < 1 || L < 0 || row_stride < 0 || score < base || score - base > size) return false;
  const int64_t room = (int64_t)((size - (score - base)) / (uint64_t)element_bytes);
  return L <= room && (B == 1 || row_stride <= (room - L) / (B - 1));
}

// ---------------------------------------------------------------------------------------------
// Digit rule of a finish round over a field's range [lo, cap]: digit(v) = min((v - lo) >>
// shift, kFinishBins - 1). The shift is chosen so that [lo, focus] spreads over the bins below the
// last one; everything above `focus` (cap >= focus >= lo) lands in the last bin. With focus == cap
// this is a plain radix digit of the range; a caller that knows where in the range the threshold
// will fall passes a tighter focus and gets finer bins there. The rounds work on 32-bit fields: the keys, and
// the inverted indices under one key.
// ---------------------------------------------------------------------------------------------
template <class V>
struct FieldDigit {
  V lo;
  int shift;
  FFTOPK_DECIDE_HD uint32_t of(V v) const {
    const V d = (V)(v - lo) >> shift;
    return d < (V)(kFinishBins - 1) ? (uint32_t)d : (uint32_t)(kFinishBins - 1);
  }
  // the values of bin t (one that holds a value of [lo, cap])
  FFTOPK_DECIDE_HD V bin_low(uint32_t t) const { return lo + ((V)t << shift); }
  FFTOPK_DECIDE_HD V bin_high(uint32_t t, V cap) const {
    const V low = bin_low(t), high = low + (((V)1 << shift) - 1u);
    return t == (uint32_t)kFinishBins - 1u || high > cap || high < low ? cap : high;
  }
};
template <class V>
FFTOPK_DECIDE_HD FieldDigit<V> make_field_digit(V lo, V focus) {
  const V width = focus - lo;
  const int bits = 64 - clz64((uint64_t)width);
  int shift = bits > kFinishBits ? bits - kFinishBits : 0;
  if ((width >> shift) >= (V)(kFinishBins - 1)) ++shift;  // keep the last bin for what lies above
  return FieldDigit<V>{lo, shift};
}
using KeyDigit = FieldDigit<uint32_t>;
FFTOPK_DECIDE_HD KeyDigit make_key_digit(uint32_t lo, uint32_t focus) { return make_field_digit<uint32_t>(lo, focus); }

// (indices are < 2^idx_bits and stored inverted: the smallest inverted index)
FFTOPK_DECIDE_HD uint32_t inverted_index_floor(int idx_bits) { return ~((idx_bits >= 32 ? 0u : (1u << idx_bits)) - 1u); }

// ---------------------------------------------------------------------------------------------
// Work split of the fused indexer's producer. The tiles of all rows, row after row, form one
// sequence of `total` tiles; first_tile[r] (r <= rows) is the number of tiles of the rows before r.
// CTA c of `ctas` takes the run [g0, g1): total = each * ctas + rest, and the first `rest` CTAs
// take one tile more. The part of a run inside one row is a segment.
// ---------------------------------------------------------------------------------------------
struct TileRun {
  uint32_t g0, g1;
};
FFTOPK_DECIDE_HD TileRun tile_run(uint32_t total, uint32_t ctas, uint32_t cta) {
  const uint32_t each = total / ctas, rest = total % ctas;
  const uint32_t g0 = cta * each + (cta < rest ? cta : rest);
  return TileRun{g0, g0 + each + (cta < rest ? 1u : 0u)};
}
// the last row that starts at or before tile g (rows >= 1)
FFTOPK_DECIDE_HD int tile_row_at(const uint32_t* first_tile, int rows, uint32_t g) {
  int lo = 0, hi = rows;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (first_tile[mid] <= g) lo = mid; else hi = mid;
  }
  return lo;
}
// Segment of the run [g, g1) inside a row that starts at tile row_g0 and has ntiles tiles: the
// first row-local tile and the tile count; false if the row has no tile at or behind g.
FFTOPK_DECIDE_HD bool tile_segment(uint32_t row_g0, uint32_t ntiles, uint32_t g, uint32_t g1, int& t_lo, int& n) {
  if (row_g0 + ntiles <= g) return false;
  const uint32_t end = g1 < row_g0 + ntiles ? g1 : row_g0 + ntiles;
  t_lo = (int)(g - row_g0);
  n = (int)(end - g);
  return true;
}

}  // namespace fftopk

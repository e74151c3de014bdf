// Per-row top-2048 radix selector for B200 (sm_100a): one thread-block cluster per row.
//
// What it replaces in the reference: topk_kernel and fast_topk_split_kv_cuda_tl
// (jit_kernel/csrc/topk_indexer/topk_indexer_radix.cu:456-869) and the host launcher
// fast_topk_interface (:1051-1158).
//
// Shape of the computation for one row of `len` > 2048 valid fp32 logits, C CTAs in the cluster,
// each owning a contiguous shard of the row:
//   1. SAMPLE. Every CTA reads the same 8K elements (more of rows beyond 256K), in pieces of 32
//      spread evenly over the row, and histograms them on a digit of 64 bins per octave. A CTA whose
//      whole shard fits in registers has those loads in flight at the same time.
//   2. PICK. One block-wide suffix scan finds the bin whose sample rank is the expected rank of the k-th
//      element plus five standard deviations - a lower bound of the true threshold with overwhelming
//      probability where the sample elements are independent (see sample_piece_start) - and the mirror-image
//      upper bound. All CTAs of a cluster find the same bin by
//      themselves: no histogram is exchanged and no cluster barrier is waited for here (exchanging
//      them took 0.8 us for the barrier and 1.8 us for two rounds of remote reads).
//   3. FILTER. ONE float compare per element against the bin's lower edge, on the shard in registers
//      (counted, scanned over the warp, stored: no second read) or in one streaming pass (128-bit
//      loads, four or eight in flight per thread); the few thousand elements that pass go to dense
//      per-warp segments of a list in shared memory.
//   4. GATHER + FINISH. They become (key << 32 | ~index) composites on their way into rank 0's shared
//      memory, where every CTA owns a region; every CTA also tells every other its count, so that
//      after the one cluster barrier each knows whether the guess held and all but rank 0 leave. Rank 0
//      finishes (cta_finish): radix rounds over the keys in the composites, a counting and a writing pass, and the
//      last <= 256 undecided candidates ranked by votes. A lone CTA gathers nothing: it keeps its candidates'
//      indices in shared memory and their keys in registers, and finishes on those (lone_finish). Equal values resolve
//      to the lower index: votes compare whole composites, and more copies than are ranked go through
//      rounds over the inverted indices.
//      Measured (us per call in a chain of calls on B200, when histograms were exchanged -> as it is now):
//      B=1, L=96K 12.9 -> 10.5, 1M 15.4 -> 14.2 from L2; B=64 ragged rows of up to 128K 20.0 -> 18.0, calls that may
//      overlap 5.4 -> 3.2; B=2048, one CTA per row, L=32K 132 -> 80.2, 8K 106 -> 54.0, 4K 62 -> 35.8. What bounds it is no
//      bandwidth but the chain of short phases and the instructions in it.
//   5. If the guess admitted fewer than k elements, a list overflowed or the threshold bin is
//      larger than rank 0's buffer (heavy ties, rows of equal values), the cluster falls back to
//      full histograms over the data: 12 + 12 + 8 key bits, re-reading the shard from L2 each
//      round, and exact ties left after 32 bits are taken in index order, shard by shard.
//
// Build-time knobs (all optional, for experiments; the defaults are what was measured best):
//   FFTOPK_REG_SLABS        granules per thread up to which the shard stays in registers (4; see reg_slabs)
//   FFTOPK_1B_FACTOR        second look at the sample when the guessed bin holds more than factor*k (2)
//   FFTOPK_U512             128-bit loads in flight per thread of the 512-thread filter (8; 16 allowed)
//   FFTOPK_CTAS_512         512-thread CTAs per SM the register budget allows (2)
//   FFTOPK_KSMALL           undecided candidates ranked by votes (256)
//   FFTOPK_TRACE            phase timestamps of block 0 (changes no result)
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>

#include "../../include/fftopk.h"
#include "fftopk_trace.cuh"
#include "fftopk_device.cuh"
#include "fftopk_host.h"
#include "fftopk_internal.h"
#include "fftopk_key.h"
#include "fftopk_merge.cuh"

namespace fftopk {


#ifndef FFTOPK_REG_SLABS
#define FFTOPK_REG_SLABS 4
#endif

struct SelectParams {
  const void* score;  // fp32, or fp16 / bf16 for the kernels instantiated on those types
  int64_t row_stride;
  int64_t L;
  const int32_t* lengths;
  const int32_t* row_starts;
  int32_t* out_idx;
  uint32_t* out_key;
  uint32_t* status;
  int32_t B;
  int32_t k;  // elements selected per row (the reference's op: 2048); output rows have k slots
  int32_t idx_offset;
  int32_t list_cap;  // per-CTA candidate list capacity (entries), multiple of 16
  int32_t cand_cap;  // rank 0's gathered-candidate capacity (entries), multiple of 16
  int32_t region;    // slots of each CTA in it (gather_region; two divisions that no thread has to wait for)
  int32_t force_slow;  // tests: skip the filter path and run the full-histogram path
  int32_t overlap;     // let the next launch on the stream start before this one has finished
  int32_t prefetch;    // ask for the rows to be brought into L2 while the launch in front of this one still runs
  // fused output transforms (all optional; reference: topk_transform_decode_kernel,
  // topk_transform_prefill_kernel, topk_transform_prefill_ragged_kernel, radix.cu:871-995)
  const int32_t* src_page_table;  // [prefill_bs, src_stride]: out = table_row[idx]
  int64_t src_stride;
  const int32_t* cu_seqlens_q;    // [prefill_bs + 1] or NULL (then table row = score row)
  int32_t prefill_bs;
  const int32_t* row_offsets;     // [B]: out = idx + row_offsets[row]
  // context-parallel publication with a device-side epoch: when cp_flag is set, the output planes
  // are shifted by ((*cp_flag + 1) & 1) * cp_half_words (the half of the comm buffer that the NEXT
  // epoch writes), so that a captured CUDA graph can be replayed
  const uint32_t* cp_flag;
  int64_t cp_half_words;
  // ... and its announcement: when cp_publish is set, the last CTA of the grid to finish (arrival
  // counter at cp_publish[kCommArriveWord]) fences and releases the epoch flag cp_publish[0] at
  // system scope, so that peers that acquire the flag see every output of this launch. cp_epoch is
  // the value to store, or 0 for "the flag's current value plus one".
  uint32_t* cp_publish;
  uint32_t cp_epoch;
  // warm start (select2048_kernel<NT, false, true> only): prev_threshold[row] is a key guess of the
  // row's k-th largest element from an earlier call (0: none), from which warm_margin is
  // subtracted; next_threshold[row] receives this call's k-th largest key (or a lower bound of it)
  const uint32_t* prev_threshold;
  uint32_t* next_threshold;
  uint32_t warm_margin;
  // (warm-start kernel only) fused indexer: a row whose guess cand_guess[row] held is finished on its candidates
  uint64_t* cand;
  const uint32_t* cand_guess;
};


constexpr int kPrefetchers = 16;  // threads of a CTA that ask for a part of its row each
constexpr uint32_t kOverflowed = 1u << 31;   // in a CTA's candidate count: one of its lists has overflowed
#ifndef FFTOPK_1B_FACTOR
#define FFTOPK_1B_FACTOR 2.0f
#endif
constexpr float kCoarseFactor = FFTOPK_1B_FACTOR;
#ifndef FFTOPK_U512
#define FFTOPK_U512 8
#endif


// digit schedule of the full-histogram rounds: 12 + 12 + 8 bits
__device__ __forceinline__ int round_width(int r) { return r < 2 ? 12 : 8; }
__device__ __forceinline__ int round_shift(int r) { return r == 0 ? 20 : (r == 1 ? 8 : 0); }

// Element types of the score matrix. The kernel works on granules of FOUR elements of the aligned
// view of the row - 16 bytes of fp32, 8 bytes of fp16 / bf16 - and widens 16-bit elements to fp32
// (exactly, order-preserving) as it loads them, so that keys, edges and composites are the fp32
// ones everywhere and a 16-bit row is read once, in its own width.
template <class T>
struct Elem;
template <>
struct Elem<float> {
  static __device__ __forceinline__ float4 ld4(const float* gbase, int g) {
    return __ldg(reinterpret_cast<const float4*>(gbase) + g);
  }
  static __device__ __forceinline__ float ld1(const float* p) { return __ldg(p); }
};
template <>
struct Elem<__half> {
  static __device__ __forceinline__ float4 ld4(const __half* gbase, int g) {
    const uint2 r = __ldg(reinterpret_cast<const uint2*>(gbase) + g);
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&r.x));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&r.y));
    return make_float4(a.x, a.y, b.x, b.y);
  }
  static __device__ __forceinline__ float ld1(const __half* p) { return __half2float(__ldg(p)); }
};
template <>
struct Elem<__nv_bfloat16> {
  static __device__ __forceinline__ float4 ld4(const __nv_bfloat16* gbase, int g) {
    const uint2 r = __ldg(reinterpret_cast<const uint2*>(gbase) + g);  // bf16 = the upper half of an fp32
    return make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xffff0000u), __uint_as_float(r.y << 16),
                       __uint_as_float(r.y & 0xffff0000u));
  }
  static __device__ __forceinline__ float ld1(const __nv_bfloat16* p) {
    return __uint_as_float((uint32_t)__bfloat16_as_ushort(__ldg(p)) << 16);
  }
};

// Shard of one CTA, in granules of four elements of the aligned view of the row: granule g covers
// row elements 4g-a .. 4g-a+3, where a in 0..3 is the row's misalignment in elements.
template <class T>
struct Shard {
  const T* gbase;      // granule-aligned address of granule 0
  int g0, g1;          // granule range of this CTA
  int i0, i1;          // the part of [g0, g1) whose granules lie completely inside the row
  int a;               // misalignment (elements)
  int len;             // valid elements in the row
};

// A granule that straddles the start or the end of the row (at most two per row): scalar loads of
// the elements that belong to the row, `fill` elsewhere. Kept out of line so that the streaming
// loops stay small enough to unroll with every load in flight.
template <class T>
__device__ __noinline__ float4 load_granule_partial(const T* gbase, int a, int len, int g, float fill) {
  const int i0 = 4 * g - a;
  float4 x = make_float4(fill, fill, fill, fill);
  const T* p = gbase + 4 * (int64_t)g;
  if ((unsigned)(i0 + 0) < (unsigned)len) x.x = Elem<T>::ld1(p + 0);
  if ((unsigned)(i0 + 1) < (unsigned)len) x.y = Elem<T>::ld1(p + 1);
  if ((unsigned)(i0 + 2) < (unsigned)len) x.z = Elem<T>::ld1(p + 2);
  if ((unsigned)(i0 + 3) < (unsigned)len) x.w = Elem<T>::ld1(p + 3);
  return x;
}

// One granule from global memory; reads only bytes that belong to the row.
template <class T>
__device__ __forceinline__ float4 load_granule(const Shard<T>& sh, int g, float fill) {
  if (g >= sh.i0 && g < sh.i1) return Elem<T>::ld4(sh.gbase, g);
  return load_granule_partial(sh.gbase, sh.a, sh.len, g, fill);
}

// A kept element on its way into the list: the raw float bits (high word) and the row index. It becomes
// a (key << 32 | ~idx) composite later, in a dense pass - the loop that finds the hits is the divergent
// part of the filter and every instruction in it is paid by a whole warp for one or two lanes.
__device__ __forceinline__ uint64_t raw_to_composite(uint64_t raw) {
  return ((uint64_t)fftopk_key_from_bits((uint32_t)(raw >> 32)) << 32) | (uint64_t)(~(uint32_t)raw);
}

// Overflow of a warp's segment: a shared spill area, slots from one counter
// (rare, so the serialising atomic does not matter). Converts on the spot. Out of line to keep
// the filter loop small.
__device__ __noinline__ void spill_push(Ctrl* ctrl, uint64_t* spill, uint32_t spill_cap, uint64_t raw) {
  const uint32_t slot = warp_alloc(&ctrl->lcount);
  if (slot < spill_cap) {
    spill[slot] = raw_to_composite(raw);
  } else {
    ctrl->pub_flag = 1u;
  }
}

// The one full read of the shard: every element x with !(x < edge) is kept as a
// (key << 32 | ~idx) composite. Per loop trip a thread has U 128-bit loads in flight and spends
// one compare and one predicated OR per element on a pass mask. Candidates go to a segment of the
// shared-memory list that belongs to the WARP and is filled densely: the warp walks its lanes'
// hits together, one hit per lane and loop trip, and a ballot gives each its slot - no atomic, and
// the segment's length lives in a register that is the same in all lanes. (Allocating from one
// shared counter serialised at ~20 cycles per candidate; slots private to a thread left more than
// half of the list empty, and every later pass paid for the empty slots.) A hit's value cannot be
// selected out of 4*U registers by a computed index, so it is fetched again. kStage = false does
// that inside the hit loop (the loads of the warps of a CTA overlap; best when hits are few and
// the latency of one call counts); kStage = true stores only the row index there and fetches all
// values in the dense pass that builds the composites afterwards, several loads in flight per
// lane (best when most trips have hits: a dependent load per trip of the hit loop would stall
// the warp each time). Candidates beyond the segment's capacity go to the shared spill area.
// Returns the number of candidates the warp found (those beyond seg_cap went to the spill area).
template <int NT, int U, bool kStage, class T>
__device__ __forceinline__ uint32_t filter_shard(const Shard<T>& sh, float edge, uint64_t* seg, uint32_t seg_cap, Ctrl* ctrl,
                                                 uint64_t* spill, uint32_t spill_cap) {
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const unsigned lt = (1u << lane) - 1u;
  const float ninf = __uint_as_float(0xff800000u);
  const T* gbase = sh.gbase;
  const int fa = sh.a, fi1 = sh.i1, len = sh.len;
  uint32_t wcnt = 0;  // candidates of this warp so far (warp-uniform)
  const uint32_t seg_s = smem_u32(seg);  // staging: candidate j's row index in word j
  auto keep = [&](bool has, int idx) {  // called by the whole warp
    const unsigned b = __ballot_sync(kFull, has);
    if (has) {
      const uint32_t pos = wcnt + (uint32_t)__popc(b & lt);
      if (kStage && pos < seg_cap) {
        sts32(seg_s + pos * 4u, (uint32_t)idx);
      } else {
        const uint32_t bits = __float_as_uint(Elem<T>::ld1(gbase + idx + fa));
        if (pos < seg_cap) {
          sts64(seg_s + pos * 8u, (uint32_t)idx, bits);
        } else {
          spill_push(ctrl, spill, spill_cap, ((uint64_t)bits << 32) | (uint64_t)(uint32_t)idx);
        }
      }
    }
    wcnt += (uint32_t)__popc(b);
  };
  // one trip over granules gb + u*NT + tid, u < U; a `full` trip lies inside the shard entirely
  auto trip = [&](int gb, auto full) {
    float4 x[U];
    using Mask = std::conditional_t<(U > 8), uint64_t, uint32_t>;
    Mask vmask = ~(Mask)0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int g = gb + u * NT + tid;
      if constexpr (decltype(full)::value) {
        x[u] = Elem<T>::ld4(gbase, g);
      } else {
        x[u] = make_float4(ninf, ninf, ninf, ninf);
        if (g < fi1) {
          x[u] = Elem<T>::ld4(gbase, g);
        } else {
          vmask &= ~((Mask)0xfu << (4 * u));  // (padding would pass an edge of -inf)
        }
      }
    }
    // pass mask of this thread's 4*U elements: bit 4u+e
    Mask mask = 0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      mask |= !(x[u].x < edge) ? (Mask)1u << (4 * u) : (Mask)0;
      mask |= !(x[u].y < edge) ? (Mask)2u << (4 * u) : (Mask)0;
      mask |= !(x[u].z < edge) ? (Mask)4u << (4 * u) : (Mask)0;
      mask |= !(x[u].w < edge) ? (Mask)8u << (4 * u) : (Mask)0;
    }
    if constexpr (!decltype(full)::value) mask &= vmask;
    const int el0 = 4 * (gb + tid);
    while (__any_sync(kFull, mask != 0)) {
      const bool has = mask != 0;
      const int bit = (sizeof(Mask) == 8 ? __ffsll((long long)mask) : __ffs((int)mask)) - 1;
      mask &= mask - 1;
      keep(has, el0 + (bit >> 2) * (4 * NT) + (bit & 3) - fa);
    }
  };
  int gb = sh.i0;
  for (; gb + NT * U <= fi1; gb += NT * U) trip(gb, std::true_type{});
  if (gb < fi1) trip(gb, std::false_type{});
  // edge granules [g0, i0) and [i1, g1): at most one each, visited by lane 0 of warps 0 and 1
  if (tid < 64) {  // (whole warps: keep() votes)
    const int ge = (tid == 0) ? sh.g0 : ((tid == 32) ? sh.i1 : -1);
    const int ge_end = (tid == 0) ? sh.i0 : sh.g1;
    const bool mine = ge >= 0 && ge < ge_end;
    if (__any_sync(kFull, mine)) {
      float4 x = make_float4(ninf, ninf, ninf, ninf);
      if (mine) x = load_granule_partial(sh.gbase, sh.a, len, ge, ninf);
      const int e0 = 4 * ge - fa;
      const float xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int e = 0; e < 4; ++e)
        keep(mine && (unsigned)(e0 + e) < (unsigned)len && !(xv[e] < edge), e0 + e);
    }
  }
  return wcnt;
}

// The dense pass over a warp's segment of `own` entries that follows the filter: sink(j, composite) for
// each of them. Staged segments hold row indices only: the values are fetched again (L1/L2 hits, four
// loads in flight per lane). From the top down, so that a sink may put composite j back into the
// segment as its j-th 64-bit word: the composites of entries [j0, j0 + 128) cover words
// [2*j0, 2*j0 + 256), which hold no index not yet read.
template <class T, class Sink>
__device__ __forceinline__ void drain_segment(bool staged, const Shard<T>& sh, const uint64_t* seg, uint32_t own, Ctrl* ctrl, Sink&& sink) {
  const int lane = lane_id();
  const uint32_t seg_s = smem_u32(seg);
  __syncwarp();
  if (staged) {
    for (int j0 = (int)((own + 127u) & ~127u) - 128; j0 >= 0; j0 -= 128) {
      uint32_t idx[4], bits[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t j = (uint32_t)j0 + 32u * u + lane;
        idx[u] = j < own ? lds32(seg_s + j * 4u) : 0u;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (!FFTOPK_CHECK(7, idx[u], sh.len, ctrl_status(ctrl))) idx[u] = 0u;
        bits[u] = __float_as_uint(Elem<T>::ld1(sh.gbase + idx[u] + sh.a));  // (index 0 is always readable)
      }
      __syncwarp();
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t j = (uint32_t)j0 + 32u * u + lane;
        if (j < own) sink(j, raw_to_composite(((uint64_t)bits[u] << 32) | idx[u]));
      }
      __syncwarp();
    }
  } else {
    for (uint32_t j = lane; j < own; j += 32) sink(j, raw_to_composite(lds64(seg_s + j * 8u)));
  }
}

// Visit every valid element of the shard: op(key, idx). Interior granules are read with
// unconditional 128-bit loads, four in flight per thread; the at most two granules that straddle
// the row's ends are visited by one thread each through scalar loads.
template <int NT, class T, class Op>
__device__ __forceinline__ void scan_shard(const Shard<T>& sh, Op&& op) {
  const int tid = threadIdx.x;
  const T* gbase = sh.gbase;
  const int a = sh.a, i1 = sh.i1;
  constexpr int U = 4;
  for (int gb = sh.i0; gb < i1; gb += NT * U) {
    float4 x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int g = gb + u * NT + tid;
      x[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (g < i1) x[u] = Elem<T>::ld4(gbase, g);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int g = gb + u * NT + tid;
      if (g < i1) {
        const int e0 = 4 * g - a;
        op(fftopk_key_from_bits(__float_as_uint(x[u].x)), e0 + 0);
        op(fftopk_key_from_bits(__float_as_uint(x[u].y)), e0 + 1);
        op(fftopk_key_from_bits(__float_as_uint(x[u].z)), e0 + 2);
        op(fftopk_key_from_bits(__float_as_uint(x[u].w)), e0 + 3);
      }
    }
  }
  // edge granules of this shard: [g0, i0) and [i1, g1), at most one granule each
  const int ge = (tid == 0) ? sh.g0 : ((tid == 32) ? sh.i1 : -1);
  const int ge_end = (tid == 0) ? sh.i0 : sh.g1;
  if (ge >= 0 && ge < ge_end) {
    const float4 x = load_granule_partial(sh.gbase, sh.a, sh.len, ge, 0.f);
    const int e0 = 4 * ge - a;
    const float xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if ((unsigned)(e0 + e) < (unsigned)sh.len) op(fftopk_key_from_bits(__float_as_uint(xv[e])), e0 + e);
    }
  }
}

// The filter of a shard that sits in registers (x[j]: granule j*NT + thread of the shard, -inf where an
// element is not the row's; `edge` > -inf). Every lane counts its hits, a scan over the warp gives it
// its slots, and a predicated store per element writes what passes: no second read of the value, no
// loop over hits. Same result as filter_shard.
template <int R>
__device__ __forceinline__ uint32_t filter_regs(const float4 (&x)[R], int slabs, int el0, int el_step, float edge, uint64_t* seg,
                                                uint32_t seg_cap, Ctrl* ctrl, uint64_t* spill, uint32_t spill_cap) {
  const int lane = lane_id();
  uint32_t n = 0u;
  auto count = [&](float v) {
    asm("{\n\t.reg .pred p;\n\tsetp.geu.f32 p, %1, %2;\n\t@p add.u32 %0, %0, 1;\n\t}" : "+r"(n) : "f"(v), "f"(edge));
  };
#pragma unroll
  for (int j = 0; j < R; ++j) {
    if (j < slabs) {  // (uniform)
      count(x[j].x);
      count(x[j].y);
      count(x[j].z);
      count(x[j].w);
    }
  }
  uint32_t incl = n;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t v = __shfl_up_sync(kFull, incl, off);
    if (lane >= off) incl += v;
  }
  const uint32_t total = __shfl_sync(kFull, incl, 31);
  uint32_t pos = incl - n;
  uint32_t at = smem_u32(seg) + pos * 8u;
  auto put = [&](float v, int idx) {
#ifdef FFTOPK_CHECKED
    if (!(v < edge) && !FFTOPK_CHECK(13, (at - smem_u32(seg)) / 8u, seg_cap, ctrl_status(ctrl))) return;
#endif
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.geu.f32 p, %1, %2;\n\t@p st.shared.v2.u32 [%0], {%3, %4};\n\t@p add.u32 %0, %0, 8;\n\t}"
        : "+r"(at)
        : "f"(v), "f"(edge), "r"(idx), "r"(__float_as_uint(v))
        : "memory");
  };
  auto put_checked = [&](float v, int idx) {
    if (!(v < edge)) {
      const uint64_t raw = ((uint64_t)__float_as_uint(v) << 32) | (uint32_t)idx;
      if (pos < seg_cap) {
        seg[pos] = raw;
      } else {
        spill_push(ctrl, spill, spill_cap, raw);
      }
      ++pos;
    }
  };
  if (total <= seg_cap) {  // (uniform over the warp)
#pragma unroll
    for (int j = 0; j < R; ++j) {
      if (j < slabs) {
        put(x[j].x, el0 + j * el_step);
        put(x[j].y, el0 + j * el_step + 1);
        put(x[j].z, el0 + j * el_step + 2);
        put(x[j].w, el0 + j * el_step + 3);
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < R; ++j) {
      put_checked(x[j].x, el0 + j * el_step);
      put_checked(x[j].y, el0 + j * el_step + 1);
      put_checked(x[j].z, el0 + j * el_step + 2);
      put_checked(x[j].w, el0 + j * el_step + 3);
    }
  }
  return total;
}

// The filters of a lone CTA. They leave the candidates' row indices in the warp's segment (word j: candidate j) and
// nothing else: the values are fetched again by the pass that follows, several loads in flight per lane.
// What bounds a batch of such rows is the instructions their warps issue, so: two per element for the pass mask, one
// from the FMA pipe (the sign of x - edge; a NaN has none) and one that shifts the sign in; slots by a scan over the
// warp, once per trip; and every lane walks its own hits, without the votes and the warp-wide counter of a
// loop that the warp walks together (10,500 warp instructions for a row of 32K elements then).
// A segment that does not hold its warp's candidates says so, and the row goes through full histograms.
struct LoneList {
  uint32_t seg_s;  // shared address of the warp's segment
  uint32_t seg_cap;
  Ctrl* ctrl;
};
__device__ __forceinline__ uint32_t warp_excl_scan(uint32_t n, uint32_t& total) {
  const int lane = lane_id();
  uint32_t incl = n;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t v = __shfl_up_sync(kFull, incl, off);
    if (lane >= off) incl += v;
  }
  total = __shfl_sync(kFull, incl, 31);
  return incl - n;
}
// hits: bit 31 - e for element e (of at most 32) of the lane; index_of(e) is its place in the row
template <class IndexOf>
__device__ __forceinline__ void keep_hits(const LoneList& l, uint32_t hits, uint32_t& wcnt, IndexOf&& index_of) {
  uint32_t total;
  const uint32_t pos = wcnt + warp_excl_scan((uint32_t)__popc(hits), total);
  if (wcnt + total <= l.seg_cap) {  // (uniform over the warp)
    wcnt += total;
    uint32_t at = l.seg_s + pos * 4u;
    while (hits != 0u) {
      const int e = __clz((int)hits);
      hits &= ~(0x80000000u >> e);
      sts32(at, (uint32_t)index_of(e));
      at += 4u;
    }
  } else {
    l.ctrl->pub_flag = 1u;  // (what is counted is what the segment holds)
  }
}
// (x >= edge or NaN: 0) shifted into the mask from the right. An edge of zero has to be the negative one: -0 - (-0) is +0,
// -0 - (+0) would be -0.
__device__ __forceinline__ uint32_t shift_in_below(uint32_t mask, float x, float edge) {
  return __funnelshift_l(__float_as_uint(x - edge), mask, 1);
}
__device__ __forceinline__ uint32_t shift_in_below4(uint32_t mask, const float4& x, float edge) {
  return shift_in_below(shift_in_below(shift_in_below(shift_in_below(mask, x.x, edge), x.y, edge), x.z, edge), x.w, edge);
}
template <int NT, class T>
__device__ __forceinline__ uint32_t filter_stream_lone(const Shard<T>& sh, float edge, const LoneList& l) {
  constexpr int U = 8;
  static_assert(4 * U <= 32, "the mask");
  const int tid = threadIdx.x;
  const float ninf = __uint_as_float(0xff800000u);
  const T* gbase = sh.gbase;
  uint32_t wcnt = 0u;
  auto trip = [&](int gb, auto full) {
    float4 x[U];
    uint32_t valid = 0xffffffffu;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int g = gb + u * NT + tid;
      if constexpr (decltype(full)::value) {
        x[u] = Elem<T>::ld4(gbase, g);
      } else {
        x[u] = make_float4(ninf, ninf, ninf, ninf);
        if (g < sh.i1) {
          x[u] = Elem<T>::ld4(gbase, g);
        } else {
          valid &= ~(0xf0000000u >> (4 * u));  // (padding would pass an edge of -inf)
        }
      }
    }
    uint32_t below = 0u;
#pragma unroll
    for (int u = 0; u < U; ++u) below = shift_in_below4(below, x[u], edge);
    const int el0 = 4 * (gb + tid) - sh.a;
    const uint32_t hits = ~below << (32 - 4 * U);  // (bit 31 - e: element e; none beyond the 4 * U that were read)
    keep_hits(l, decltype(full)::value ? hits : hits & valid, wcnt,
              [&](int e) { return el0 + e * NT - (e & 3) * (NT - 1); });  // element e & 3 of granule e >> 2
  };
  int gb = sh.i0;
  for (; gb + NT * U <= sh.i1; gb += NT * U) trip(gb, std::true_type{});
  if (gb < sh.i1) trip(gb, std::false_type{});
  // edge granules [g0, i0) and [i1, g1): at most one each, two lanes of the same warp
  if (tid >> 5 == lone_edge_warp(NT)) {
    const int lane = lane_id();
    const int ge = lane == 0 ? sh.g0 : (lane == 1 ? sh.i1 : -1);
    const int ge_end = lane == 0 ? sh.i0 : sh.g1;
    const bool mine = ge >= 0 && ge < ge_end;
    if (__any_sync(kFull, mine)) {
      uint32_t hits = 0u;
      const int e0 = 4 * ge - sh.a;
      if (mine) {
        const float4 x = load_granule_partial(sh.gbase, sh.a, sh.len, ge, ninf);
        const uint32_t below = shift_in_below4(0u, x, edge);
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if ((unsigned)(e0 + e) < (unsigned)sh.len && !((below >> (3 - e)) & 1u)) hits |= 0x80000000u >> e;
      }
      keep_hits(l, hits, wcnt, [&](int e) { return e0 + e; });
    }
  }
  return wcnt;
}
// ... of a shard that sits in registers (x[j]: granule j*NT + thread, -inf where an element is not the row's; edge > -inf):
// a quarter of a short row passes, so a predicated store per element is cheaper than a walk over the hits.
template <int R>
__device__ __forceinline__ uint32_t filter_regs_lone(const float4 (&x)[R], int slabs, int el0, int el_step, float edge,
                                                     const LoneList& l) {
  static_assert(R <= 8, "");
  uint32_t below = 0u;
#pragma unroll
  for (int j = 0; j < R; ++j) below = j < slabs ? shift_in_below4(below, x[j], edge) : (below << 4) | 0xfu;
  const uint32_t hits = ~below << (32 - 4 * R);
  uint32_t total;
  const uint32_t pos = warp_excl_scan((uint32_t)__popc(hits), total);
  if (total <= l.seg_cap) {  // (uniform over the warp)
    uint32_t at = l.seg_s + pos * 4u;
    auto put = [&](float v, int idx) {
      asm volatile(
          "{\n\t.reg .pred p;\n\tsetp.geu.f32 p, %1, %2;\n\t@p st.shared.u32 [%0], %3;\n\t@p add.u32 %0, %0, 4;\n\t}"
          : "+r"(at)
          : "f"(v), "f"(edge), "r"(idx)
          : "memory");
    };
#pragma unroll
    for (int j = 0; j < R; ++j) {
      if (j < slabs) {  // (uniform)
        put(x[j].x, el0 + j * el_step);
        put(x[j].y, el0 + j * el_step + 1);
        put(x[j].z, el0 + j * el_step + 2);
        put(x[j].w, el0 + j * el_step + 3);
      }
    }
    return total;
  }
  l.ctrl->pub_flag = 1u;
  return 0u;
}

// The sample of a row: `nb` batches of G loads of 32 granules per warp, spread over the whole row in pieces
// (see sample_piece_start). Every CTA of a cluster takes the SAME sample, so each finds the same guess by
// itself: no exchange of histograms and no cluster barrier in front of the search. A row that is no larger
// than the sample is read completely. Granules that straddle the row's ends are left out.
template <int NT, int G>
struct RowSample {
  int i0, gi;  // first granule completely inside the row, and how many there are
  int nb;      // batches, a power of two
  int gu;      // loads per thread and batch: G, or half of that
  uint32_t off;  // granule i0's position within a piece
  bool whole;
  // load u of batch b: which of the sample's loads of 32 granules it is
  __device__ __forceinline__ int load_no(int b, int u) const { return (b * gu + u) * (NT / 32) + (int)(threadIdx.x >> 5); }
  __device__ __forceinline__ int granules() const { return NT * gu * nb; }
  __device__ __forceinline__ uint32_t size() const { return 4u * (uint32_t)(whole ? gi : granules()); }
  // (one branch around all loads of a batch, so that they are in flight together; x may be longer than G)
  template <class T, int N>
  __device__ __forceinline__ void load(const T* gbase, int b, float4 (&x)[N]) const {
    static_assert(N >= G, "");
    if (whole) {
#pragma unroll
      for (int u = 0; u < G; ++u) {
        const int g = load_no(b, u) * 32 + lane_id();
        if (u < gu && g < gi) x[u] = Elem<T>::ld4(gbase, i0 + g);
      }
    } else {
      constexpr int kPer = 32 / kSamplePiece;  // pieces per load
      const int log_pieces = 31 - __clz(granules() / kSamplePiece);
#pragma unroll
      for (int u = 0; u < G; ++u) {
        const uint32_t piece = (uint32_t)(load_no(b, u) * kPer + lane_id() / kSamplePiece);
        const uint32_t first = sample_piece_start((uint32_t)gi, piece, log_pieces, off);
        if (u < gu) x[u] = Elem<T>::ld4(gbase, i0 + (int)first + (lane_id() & (kSamplePiece - 1)));
      }
    }
  }
  template <int N, class Op>
  __device__ __forceinline__ void use(int b, const float4 (&x)[N], Op&& op) const {
    auto four = [&](const float4& v) {
      op(__float_as_uint(v.x));
      op(__float_as_uint(v.y));
      op(__float_as_uint(v.z));
      op(__float_as_uint(v.w));
    };
    if (whole) {
#pragma unroll
      for (int u = 0; u < G; ++u)
        if (u < gu && load_no(b, u) * 32 + lane_id() < gi) four(x[u]);
    } else {
#pragma unroll
      for (int u = 0; u < G; ++u)
        if (u < gu) four(x[u]);
    }
  }
};

// Everything one CTA needs to know about its row and its shared memory.
template <int NT, class T>
struct RowCtx {
  int C, rank;
  Shard<T> sh;
  uint32_t* hist0;  // two histograms of kMaxBins words, back to back; a lone CTA has one that serves as both
  uint32_t* sup0;   // two super-bin arrays of kSup words, back to back
  // (computed addresses instead of pointer arrays: indexing an array member with the round number
  // would force the whole struct into local memory)
  __device__ __forceinline__ uint32_t* hist(int i) const { return C == 1 ? hist0 : hist0 + i * kMaxBins; }
  __device__ __forceinline__ uint32_t* sup(int i) const { return sup0 + i * kSup; }
  uint32_t* xch;
  Ctrl* ctrl;
  Ctrl* ctrl0;
  uint64_t* list;
  uint64_t* cand;
  uint64_t* cand0;
  int32_t* out_idx;
  uint32_t* out_key;
  int32_t idx_offset;
  const int32_t* page;  // fused page-table transform: out = page[idx] (NULL: out = idx + idx_offset)
  int32_t cand_cap;
  uint32_t* status;
  uint32_t k;  // elements to select per row (2048 for the reference's op)
};

template <class Cx>
__device__ __forceinline__ void emit_winner(const Cx& cx, uint32_t base_w, uint32_t key, int idx) {
  const uint32_t pos = base_w + warp_alloc(&cx.ctrl->wslot);
  if (FFTOPK_CHECK(1, pos, cx.k, cx.status) && pos < cx.k) {
    cx.out_idx[pos] = cx.page ? __ldg(cx.page + idx) : idx + cx.idx_offset;
    if (cx.out_key) cx.out_key[pos] = key;
  }
}

// -----------------------------------------------------------------------------------------
// Full-histogram path: every round re-reads the shard (from L2) and histograms the next key
// digit of the elements that still match the threshold prefix. Handles anything: lists that
// would overflow, threshold bins larger than rank 0's buffer, rows of identical values.
// Returns the final mode; `need`, `P` and `r` describe where it stopped.
// -----------------------------------------------------------------------------------------
template <int NT, class T>
__device__ __forceinline__ int refine_from_data(const RowCtx<NT, T>& cx, uint32_t& need_out, uint32_t& P_out, int& r_out) {
  cg::cluster_group cluster = cg::this_cluster();
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int C = cx.C, rank = cx.rank;
  const Shard<T>& sh = cx.sh;
  Ctrl* ctrl = cx.ctrl;
  uint32_t* xch = cx.xch;

  // peers may still be reading this CTA's histograms from the attempt that fell back
  cluster_sync(cluster, C);
  {
    uint4* h4 = reinterpret_cast<uint4*>(cx.hist(0));
    for (int i = tid; i < kMaxBins / 4; i += NT) h4[i] = make_uint4(0u, 0u, 0u, 0u);
    if (tid == 0) {
      ctrl->pub_flag = 0u;
      ctrl->win_count = 0u;   // rank 0's copies are the cluster-wide counters; nobody touches
      ctrl->cand_count = 0u;  // them again before the cluster barrier of the first histogram pass
    }
    if (tid < kSup) {
      ctrl->tot[0][tid] = ctrl->tot[1][tid] = 0u;
      ctrl->tot2[0][tid] = ctrl->tot2[1][tid] = 0u;
    }
  }
  int pick_no = 0;  // number of cluster-wide searches so far (selects their total buffers)
  __syncthreads();
  {
    uint32_t* h0 = cx.hist(0);
    scan_shard<NT, T>(sh, [&](uint32_t key, int) { hist_add(h0, key >> 20, true); });
  }
  __syncthreads();

  uint32_t need = cx.k, P = 0;
  int mode = kModeAbort;
  int r = 0;
  for (;; ++r) {
    const int w = round_width(r);
    const int shift = round_shift(r);
    const int nb = 1 << w;
    uint32_t* h = cx.hist(r & 1);
    uint32_t* s = cx.sup(r & 1);
    compute_sup<NT>(h, s, nb);
    cluster_sync(cluster, C);  // every CTA's histogram and super-bin sums of this round are complete
    const uint32_t need_now = need;
    cluster_pick<NT>(
        cluster, C, h, s, xch, ctrl, pick_no, nb, [&](uint32_t) { return need_now; },
        [&](Picked& pk) {
          const bool last = (shift == 0);
          decide_and_allocate(cx, pk, last ? kModeTies : kModeNext);
          if (pk.ok && last && pk.cnt > (uint32_t)cx.cand_cap && pk.cnt != pk.need2) {
            // exact duplicates of the threshold key: ties before this shard, in rank order
            const uint32_t tp = (lane < rank) ? xch[lane * kSup + pk.tf] : 0u;
            const uint32_t tie_prefix = warp_sum(tp);
            if (lane == 0) ctrl->tie_prefix = tie_prefix;
          }
        });
    // clear the next round's histogram (peers finished reading that buffer before they arrived
    // at this round's cluster barrier)
    {
      uint4* n4 = reinterpret_cast<uint4*>(cx.hist((r + 1) & 1));
      for (int i = tid; i < kMaxBins / 4; i += NT) n4[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    __syncthreads();
    mode = ctrl->mode;
    if (mode == kModeAbort) break;
    const uint32_t Pn = (P << w) | (uint32_t)ctrl->t;
    const uint32_t Pold = P;
    const uint32_t base_w = ctrl->base_w;
    const uint32_t base_c = ctrl->base_c;
    need = ctrl->above;
    P = Pn;

    if (mode == kModeNext) {
      const int shift2 = round_shift(r + 1);
      const uint32_t mask2 = (1u << round_width(r + 1)) - 1u;
      uint32_t* h2 = cx.hist((r + 1) & 1);
      scan_shard<NT, T>(sh, [&](uint32_t key, int idx) {
        const uint32_t hh = key >> shift;
        if ((hh >> w) == Pold) {
          if (hh > Pn) emit_winner(cx, base_w, key, idx);
          hist_add(h2, (key >> shift2) & mask2, hh == Pn);
        }
      });
      __syncthreads();
      continue;
    }
    if (mode == kModeGather) {
      scan_shard<NT, T>(sh, [&](uint32_t key, int idx) {
        const uint32_t hh = key >> shift;
        if ((hh >> w) == Pold) {
          if (hh > Pn) {
            emit_winner(cx, base_w, key, idx);
          } else if (hh == Pn) {
            const uint32_t slot = base_c + warp_alloc(&ctrl->cslot);
            if (FFTOPK_CHECK(2, slot, cx.cand_cap, cx.status) && slot < (uint32_t)cx.cand_cap)
              cx.cand0[slot] = ((uint64_t)key << 32) | (uint64_t)(~(uint32_t)idx);
          }
        }
      });
    } else if (mode == kModeTakeAll) {
      scan_shard<NT, T>(sh, [&](uint32_t key, int idx) {
        const uint32_t hh = key >> shift;
        if (((hh >> w) == Pold) && hh >= Pn) emit_winner(cx, base_w, key, idx);
      });
    } else {  // kModeTies: all 32 key bits are fixed; Pn is the threshold key itself
      // (only keys under this round's prefix: larger prefixes were written by the earlier rounds,
      // and the slots reserved here are for this round's winners alone)
      scan_shard<NT, T>(sh, [&](uint32_t key, int idx) {
        if ((key >> w) == Pold && key > Pn) emit_winner(cx, base_w, key, idx);
      });
      // Exact duplicates of the threshold key: the first `need` of them in index order win.
      // Shards are contiguous and ordered by rank, so this CTA takes its first `quota`.
      const uint32_t tie_prefix = ctrl->tie_prefix;
      const uint32_t local_c = ctrl->local_c;
      const uint32_t quota = need > tie_prefix ? min(need - tie_prefix, local_c) : 0u;
      const uint32_t obase = cx.k - need + tie_prefix;
      uint32_t run = 0;  // ties seen so far in this shard (uniform over the CTA)
      for (int gb = sh.g0; gb < sh.g1 && run < quota; gb += NT) {
        const int g = gb + tid;
        const bool in = g < sh.g1;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (in) x = load_granule(sh, g, 0.f);
        const int i0 = 4 * g - sh.a;
        const float xv[4] = {x.x, x.y, x.z, x.w};
        bool m[4];
        uint32_t c = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          m[j] = in && (unsigned)(i0 + j) < (unsigned)sh.len && fftopk_key_from_bits(__float_as_uint(xv[j])) == Pn;
          c += m[j] ? 1u : 0u;
        }
        uint32_t incl = c;  // block exclusive scan of c in thread order
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const uint32_t v = __shfl_up_sync(kFull, incl, off);
          if (lane >= off) incl += v;
        }
        if (lane == 31) ctrl->wtot[warp] = incl;
        __syncthreads();
        const uint32_t wv = (lane < NT / 32) ? ctrl->wtot[lane] : 0u;
        const uint32_t before = warp_sum(lane < warp ? wv : 0u);
        const uint32_t total = warp_sum(wv);
        uint32_t rnk = run + before + incl - c;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (m[j]) {
            if (rnk < quota && FFTOPK_CHECK(6, obase + rnk, cx.k, cx.status) && obase + rnk < cx.k) {
              cx.out_idx[obase + rnk] = cx.page ? __ldg(cx.page + i0 + j) : i0 + j + cx.idx_offset;
              if (cx.out_key) cx.out_key[obase + rnk] = Pn;
            }
            ++rnk;
          }
        }
        run += total;
        __syncthreads();
      }
    }
    break;
  }
  need_out = need;
  P_out = P;
  r_out = r;
  return mode;
}

// The full-histogram path from start to finish, out of line (the common path neither pays its registers
// nor its instructions). Returns the row's threshold as the next call's guess (rank 0; 0: none).
template <int NT, bool kTrack, class T>
__device__ __noinline__ uint32_t select_by_full_histograms(const RowCtx<NT, T> passed) {
  const RowCtx<NT, T> cx = passed;  // (out of the stack, into registers)
  cg::cluster_group cluster = cg::this_cluster();
  uint32_t need = 0u, P = 0u;
  int r = 0;
  const int mode = refine_from_data<NT, T>(cx, need, P, r);
  cluster_sync(cluster, cx.C);  // candidates that peers pushed into rank 0 are complete
  if (cx.rank != 0) return 0u;
  uint32_t thr = 0u;
  if (mode == kModeGather) {
    // every candidate shares the key prefix P above bit `shift` of the key
    const int shift = round_shift(r);
    const uint32_t lo = P << shift;
    const uint32_t cap = lo | ((1u << shift) - 1u);
    const DenseCands<NT> src{cx.cand, (int)min(cx.ctrl->cand_count, (uint32_t)cx.cand_cap)};
    cta_finish<NT, DenseCands<NT>, kTrack>(src, need, lo, cap, cap, 32 - __clz(cx.sh.len - 1), cx.hist(1), cx.ctrl,
                                           cx.out_idx, cx.out_key, cx.k - need, cx.k, cx.idx_offset, cx.status, cx.page,
                                           (uint32_t)src.n);
    if constexpr (kTrack) {
      __syncthreads();
      thr = cx.ctrl->thr_key != 0xffffffffu ? cx.ctrl->thr_key : 0u;
    }
  } else if (mode == kModeTakeAll || mode == kModeTies) {
    // no finish ran: the lower edge of the bin the threshold was found in (a lower bound: the next
    // call then admits a few more candidates and tightens it again)
    thr = P << round_shift(r);
  } else if (threadIdx.x == 0 && cx.status) {
    atomicOr(cx.status, (uint32_t)FFTOPK_ST_INTERNAL);
  }
  return thr;
}

#ifndef FFTOPK_CTAS_512
#define FFTOPK_CTAS_512 2
#endif
// Form of the kernel: a row has one CTA (a grid of clusters of one), or a cluster of 2 to 16 with one CTA
// per SM, or one of which two CTAs - of different calls - share an SM (512 threads; the others have the
// registers for one form only).
enum Form : int { kLoneForm = 0, kRoomyForm = 1, kTightForm = 2 };
template <int NT>
__host__ __device__ constexpr int min_ctas(int form) {
  return NT == 512 ? (form == kRoomyForm ? 1 : FFTOPK_CTAS_512) : 1024 / NT;
}
// Granules a thread keeps in registers when its CTA's whole shard fits: with 512 threads and one CTA
// per SM (128 registers a thread) rows of up to 256K elements over 16 CTAs.
template <int NT>
__host__ __device__ constexpr int reg_slabs(int form) {
  return (NT == 512 && form == kRoomyForm) ? 2 * FFTOPK_REG_SLABS : FFTOPK_REG_SLABS;
}
// Where a row's output goes, its page table (NULL: none) and the offset of its indices. Worked out where they are
// needed: kept from the start they would cost every thread the registers through sample and filter.
struct RowOutput {
  int32_t* idx;
  uint32_t* key;
};
__device__ __forceinline__ RowOutput row_output(const SelectParams& p, int row, uint32_t K) {
  const int64_t at = (p.cp_flag ? (int64_t)((__ldcg(p.cp_flag) + 1u) & 1u) * p.cp_half_words : 0) + (int64_t)row * K;
  return RowOutput{p.out_idx + at, p.out_key ? p.out_key + at : nullptr};
}
__device__ __forceinline__ const int32_t* row_page(const SelectParams& p, int row) {
  if (!p.src_page_table) return nullptr;
  // which table row serves this score row: the request i with cu_seqlens_q[i] <= row < cu_seqlens_q[i+1]
  // (radix.cu:925-939); without cu_seqlens_q, the row itself (decode, :880)
  int64_t req = row;
  if (p.cu_seqlens_q) {
    int lo = 0, hi = p.prefill_bs;  // invariant: cu[lo] <= row, answer in [lo, hi)
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (__ldg(p.cu_seqlens_q + mid) <= row) lo = mid; else hi = mid;
    }
    req = lo;
  }
  return p.src_page_table + req * p.src_stride;
}
__device__ __forceinline__ int32_t row_idx_offset(const SelectParams& p, int row) {
  return p.idx_offset + (p.row_offsets ? __ldg(p.row_offsets + row) : 0);
}
// A row of the fused indexer whose producer has filtered it with a guess: if the guess held - at least k candidates, no more
// than the list has room for - the cluster's first CTA finishes it on them, keys in registers like a lone
// CTA's. False: the row has to be selected on its logits. All CTAs of the cluster decide the same.
template <int NT, bool kLone, class T>
__device__ __forceinline__ bool finish_given_candidates(const SelectParams& p, const RowCtx<NT, T>& cx, int row, int len, uint32_t raw,
                                                        uint32_t count) {
  constexpr int R = kIdxCandCap / NT;
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  cg::cluster_group cluster = cg::this_cluster();
  if (raw == 0u) return false;  // (not filtered, nothing to set back)
  const uint32_t gkey = raw > p.warm_margin ? raw - p.warm_margin : 1u;
  const bool held = count >= cx.k && count <= (uint32_t)kIdxCandCap;
  // everybody has read the count before the first CTA sets it back
  if (!kLone) cluster.barrier_arrive();
  if (held && cx.rank != 0) return true;
  if (held) {
    const uint32_t hist_s = smem_u32(cx.hist0);
    const uint32_t lowkey = guess_low_key(gkey);
    const uint32_t reach = 2u * min(p.warm_margin, 0x3fffffffu) + (1u << 19);
    const uint32_t focus = lowkey > 0xffffffffu - reach ? 0xffffffffu : lowkey + reach;
    // candidates [own * warp, ...) are this warp's
    const int own = (int)(((count + NT - 1u) / NT) * 32u);
    const uint64_t* const src = idx_row_cand(p.cand, row) + warp * own;
    RegSegCands<NT, R> cands;
    cands.seg = smem_u32(cx.list) + (uint32_t)(warp * own) * 4u;
    cands.wn = max(0, min(own, (int)count - warp * own));
    uint32_t inv[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      cands.key[i] = inv[i] = 0u;
      if (i * 32 + lane < cands.wn) {
        const uint2 c = __ldcg(reinterpret_cast<const uint2*>(src) + i * 32 + lane);
        inv[i] = c.x;
        cands.key[i] = c.y;
      }
    }
    for (int i = tid; i < kFinishBins / 4; i += NT) sts_zero16(hist_s + i * 16);
    if (tid == 0) cx.ctrl->thr_key = 0xffffffffu;
    __syncthreads();
    const KeyDigit dg = make_key_digit(lowkey, focus);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if (i * 32 + lane < cands.wn) {
        sts32(cands.seg + (uint32_t)(i * 32 + lane) * 4u, ~inv[i]);
        red_shared_inc(hist_s + dg.of(cands.key[i]) * 4u);
      }
    }
    __syncthreads();
    const RowOutput ro = row_output(p, row, cx.k);
    const FinishOut o{{ro.idx, ro.key, p.status, nullptr, 0u, cx.k, p.idx_offset, cx.k}, cx.ctrl};
    lone_finish<NT, R, true>(cands, o, cx.k, lowkey, focus, 32 - __clz(len - 1), cx.hist0);
    __syncthreads();
  }
  if (!kLone) {
    cluster.barrier_wait();
  } else {
    __syncthreads();
  }
  if (tid == 0 && cx.rank == 0) {
    *idx_row_count(p.cand, row) = 0u;
    if (held) {
      p.next_threshold[row] = cx.ctrl->thr_key != 0xffffffffu ? cx.ctrl->thr_key : 0u;
    } else if (p.status) {
      atomicOr(p.status, (uint32_t)FFTOPK_ST_GUESS_MISSED);
    }
  }
  return held;
}

// kAnyK = false: k is the constant 2048 of the reference's op (the compiler folds it: one register
// less in a kernel that sits at its register limit); true: k comes from the parameters.
template <int NT, bool kAnyK, bool kWarm, class T, int kForm>
__device__ __forceinline__ void select_row(const SelectParams& p) {
  constexpr bool kLone = kForm == kLoneForm;
  constexpr int kRegSlabs = reg_slabs<NT>(kForm);
  RowCtx<NT, T> cx;
  cg::cluster_group cluster = cg::this_cluster();
  const int C = cx.C = kLone ? 1 : (int)cluster.num_blocks();
  const int rank = cx.rank = kLone ? 0 : (int)cluster.block_rank();
  const int row = (int)(blockIdx.x / (unsigned)C);
  // Back-to-back kernels on one stream (every launch of this kernel is a programmatic dependent
  // launch): once every CTA of this grid has passed this point - or exited - the next kernel on
  // the stream may become resident on whatever the grid leaves free. By default this kernel then
  // waits, before its first access to global memory, until the kernel in front of it has
  // completed and its writes are visible - stream order as ever, but the launch latency of a call
  // hides behind the call before it (2 to 3 us per call in a chain of dependent calls). Only when
  // the caller has declared consecutive calls independent (fftopk_set_overlap) does it not wait:
  // the next call then fills the SMs that short rows free early.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // What it can do before that is to have its row brought into L2 (prefetch_part_l2): in a chain of calls whose rows lie
  // in HBM the few SMs of a cluster would wait for them afterwards.
  if constexpr (!kWarm) {
    if (p.prefetch && threadIdx.x < kPrefetchers) {
      const int64_t n = min((int64_t)max(hint_s32(p.lengths + row), 0), p.L);
      prefetch_part_l2(static_cast<const T*>(p.score) + (int64_t)row * p.row_stride, n * (int64_t)sizeof(T),
                       rank * kPrefetchers + (int)threadIdx.x, C * kPrefetchers);
    }
  }
  if (!p.overlap) asm volatile("griddepcontrol.wait;" ::: "memory");
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  constexpr int NW = NT / 32;

  int64_t row_start = p.row_starts ? (int64_t)p.row_starts[row] : 0;
  row_start = row_start < 0 ? 0 : (row_start > p.L ? p.L : row_start);
  int64_t len64 = (int64_t)p.lengths[row];
  len64 = len64 < 0 ? 0 : len64;
  len64 = len64 > p.L - row_start ? p.L - row_start : len64;
  const int len = (int)len64;
  uint32_t given_guess = 0u, given_count = 0u;  // (fused indexer; on their way together with the length)
  if constexpr (kWarm) {
    if (p.cand != nullptr) {
      given_guess = __ldcg(p.cand_guess + row);
      given_count = __ldcg(idx_row_count(p.cand, row));
    }
  }
  const T* rowp = static_cast<const T*>(p.score) + (int64_t)row * p.row_stride + row_start;
  const uint32_t K = cx.k = kAnyK ? (uint32_t)p.k : (uint32_t)kK;
  cx.cand_cap = p.cand_cap;
  cx.status = p.status;

  // Short rows: 0..len-1 then -1 (reference: naive_topk_cuda, topk_indexer_radix.cu:152-163).
  if (len <= (int)K) {
    if (rank == 0) {
      const RowOutput ro = row_output(p, row, K);
      int32_t* out_idx = ro.idx;
      uint32_t* out_key = ro.key;
      cx.page = row_page(p, row);
      cx.idx_offset = row_idx_offset(p, row);
      for (int i = tid; i < (int)K; i += NT) {
        out_idx[i] = i < len ? (cx.page ? __ldg(cx.page + i) : i + cx.idx_offset) : -1;
        if (out_key) out_key[i] = i < len ? fftopk_key_from_bits(__float_as_uint(Elem<T>::ld1(rowp + i))) : 0u;
      }
      if constexpr (kWarm) {
        if (tid == 0 && p.next_threshold) p.next_threshold[row] = 0u;  // nothing to guess for such a row
        if (tid == 0 && p.cand) {
          *idx_row_count(p.cand, row) = 0u;
          if (given_guess != 0u && len > 0 && p.status) atomicOr(p.status, (uint32_t)FFTOPK_ST_GUESS_MISSED);
        }
      }
    }
    return;  // uniform over the cluster; no shared memory of this CTA is ever read by a peer
  }

  FFTOPK_MARK(0);
  // ---- shared memory carve ---------------------------------------------------------------
  extern __shared__ __align__(128) unsigned char smem_raw[];
  cx.hist0 = reinterpret_cast<uint32_t*>(smem_raw);
  cx.sup0 = cx.hist0 + (kLone ? 1 : 2) * kMaxBins;
  cx.xch = cx.sup0 + 2 * kSup;                                             // 64 words per CTA of the cluster
  Ctrl* ctrl = cx.ctrl = reinterpret_cast<Ctrl*>(cx.xch + (kLone ? 1 : kMaxCluster) * kSup);  // 16-byte aligned
  cx.list = reinterpret_cast<uint64_t*>(reinterpret_cast<unsigned char*>(ctrl) + ((sizeof(Ctrl) + 127) & ~127u));
  // a cluster of one CTA has nobody to gather from: its candidate buffer IS the list
  cx.cand = C == 1 ? cx.list : cx.list + p.list_cap;
  cx.ctrl0 = C == 1 ? ctrl : cluster.map_shared_rank(ctrl, 0);
  cx.cand0 = C == 1 ? cx.cand : cluster.map_shared_rank(cx.cand, 0);
  uint64_t* list = cx.list;

  // ---- shard geometry --------------------------------------------------------------------
  Shard<T>& sh = cx.sh;
  sh.a = (int)((reinterpret_cast<uintptr_t>(rowp) / sizeof(T)) & 3u);
  sh.len = len;
  sh.gbase = rowp - sh.a;
  const int gn = (sh.a + len + 3) >> 2;
  const int per = (((gn + C - 1) / C) + 31) & ~31;
  sh.g0 = min(rank * per, gn);
  sh.g1 = min(sh.g0 + per, gn);
  sh.i0 = max(sh.g0, sh.a > 0 ? 1 : 0);
  sh.i1 = max(sh.i0, min(sh.g1, ((sh.a + len) & 3) ? gn - 1 : gn));
  // Whole shard in registers (same answer in every CTA of the cluster: `per` is rank-independent).
  const bool in_regs = per <= NT * kRegSlabs;
  const int slabs = (per + NT - 1) / NT;  // granules of the shard per thread
  constexpr int G = NT >= 1024 ? 2 : 4;  // sample granules per thread and batch
  RowSample<NT, G> smp;
  smp.i0 = sh.a > 0 ? 1 : 0;
  smp.gi = ((sh.a + len) & 3 ? gn - 1 : gn) - smp.i0;
  // 8K elements, more for rows so long that 8K would need a margin of several thousand candidates
  smp.nb = (NT >= 512 ? 1 : 2) << sample_log_batches(len, K);
  // ... and 4K for rows of up to 32K elements over several CTAs that cannot be read completely: a CTA's
  // shard is no more than that, and the sample would be most of its work (one row, us per call with 8K / 4K: 16K
  // elements 9.7 / 9.4, 32K 10.1 / 9.8; one of 8K, where it would no longer be all of the row, 9.2 / 9.5)
  smp.gu = !kLone && len <= 32768 && smp.gi > NT * G * smp.nb ? G / 2 : G;
  smp.whole = smp.gi <= smp.granules();
  smp.off = (uint32_t)(reinterpret_cast<uintptr_t>(sh.gbase + 4 * smp.i0) / (4 * sizeof(T))) & (uint32_t)(kSamplePiece - 1);

  // ---- fused indexer: the row's candidates are there already ----------------------------------------
  if constexpr (kWarm && NT >= 512) {
    if (finish_given_candidates<NT, kLone>(p, cx, row, len, given_guess, given_count)) return;  // (uniform over the cluster)
  }

  // ---- warm start: a key guess of the row's k-th largest element from an earlier call ----------
  // With a guess the row skips the sample, its histogram and the search: it is filtered at once
  // against the guess (minus the caller's margin). The checks after the filter are the same as for
  // a sampled guess - at least k admitted, no list overflowed - and a guess that fails them sends
  // the row to the full-histogram path, so the result is exact whatever the guess was.
  uint32_t warm_key = 0u;
  if constexpr (kWarm) {
    if (p.prev_threshold != nullptr && !p.force_slow) {
      const uint32_t g = __ldg(p.prev_threshold + row);
      if (g != 0u) warm_key = g > p.warm_margin ? g - p.warm_margin : 1u;
    }
  }
  const bool warm = kWarm && warm_key != 0u;  // (uniform over the cluster)
  const bool sampled = !warm && !p.force_slow;

  // ---- loads: the shard, if it fits in registers, and the sample ----------------------------------
  float4 xr[kRegSlabs];
  const float ninf = __uint_as_float(0xff800000u);
  if (in_regs) {
#pragma unroll
    for (int j = 0; j < kRegSlabs; ++j) {
      const int g = sh.g0 + j * NT + tid;
      xr[j] = make_float4(ninf, ninf, ninf, ninf);
      if (j < slabs && g >= sh.i0 && g < sh.i1) xr[j] = Elem<T>::ld4(sh.gbase, g);
    }
  }
  float4 xs[G];
  // (a row that a lone CTA holds whole is its own sample)
  const bool own_sample = kLone && in_regs && smp.whole;
  if (sampled && !own_sample) smp.load(sh.gbase, 0, xs);
  // ---- clear the histograms and the control block --------------------------------------------------
  // (round 0 of the finish: a histogram of its own, or a lone CTA's only one, cleared for it after the search)
  uint32_t* const fin_hist = kLone ? cx.hist0 : cx.hist0 + kMaxBins;
  const uint32_t h0 = smem_u32(cx.hist0), fh = smem_u32(fin_hist);  // shared addresses
  {
    constexpr int kOwnFin = kLone ? 0 : kFinishBins / 4;
    if (!warm) {
      for (int i = tid; i < kMaxBins / 4 + kOwnFin; i += NT) sts_zero16(h0 + i * 16);
    } else {
      for (int i = tid; i < kFinishBins / 4; i += NT) sts_zero16(fh + i * 16);
    }
    if (tid == 0) {
      if constexpr (kWarm) ctrl->thr_key = 0xffffffffu;
      ctrl->extra_count = 0u;
      ctrl->pub_flag = 0u;
      ctrl->lcount = 0u;
      ctrl->guess_flags = 0u;
      ctrl->guess = 0u;
      ctrl->focus = 0u;
#ifdef FFTOPK_CHECKED
      ctrl->status_ptr = p.status;
#endif
    }
    if (tid == 32) {  // (a search in a table, while the loads travel)
      ctrl->row_page = row_page(p, row);
      ctrl->row_idx_offset = row_idx_offset(p, row);
    }
    if (sampled && warp == NW - 1) {
      // The ranks sought in the sample (see sample_lower_rank). One warp works them out while the loads
      // travel (a division and a square root in every warp would cost the CTA as much as the search itself).
      const SampleRanks ranks = sample_ranks(smp.whole, K, smp.size(), (float)len);
      if (lane == 0) {
        ctrl->need = ranks.need;
        ctrl->need_hi = ranks.need_hi;
      }
    }
  }
  if (in_regs) {  // granules straddling the row's ends (at most two per row)
#pragma unroll
    for (int j = 0; j < kRegSlabs; ++j) {
      const int g = sh.g0 + j * NT + tid;
      if (j < slabs && g < sh.g1 && (g < sh.i0 || g >= sh.i1)) xr[j] = load_granule_partial(sh.gbase, sh.a, sh.len, g, ninf);
    }
  }
  __syncthreads();  // histograms and counters are clear
  // Every CTA tells the cluster so, and checks just before its first remote access: the barrier's
  // latency hides behind the sample and the filter.
  if (C > 1) cluster.barrier_arrive();
  FFTOPK_MARK(1);

  uint32_t gkey = warm_key;  // what the shard is filtered with: a lower bound of the k-th largest key
  // A bound the threshold will not lie above (the finish's first digit spreads [guess, focus] over
  // its bins): from the sample; of a warm guess, twice the margin and 1/16 octave.
  uint32_t focus_key = 0u;
  bool guessed = warm;
  if constexpr (kWarm) {
    const uint32_t reach = 2u * min(p.warm_margin, 0x3fffffffu) + (1u << 19);
    focus_key = warm_key > 0xffffffffu - reach ? 0xffffffffu : warm_key + reach;
  }
  if (sampled) {
    const uint32_t wtot_s = smem_u32(ctrl->wtot);
    const uint32_t mid = h0 + kSampleBins / 2 * 4u;
    auto tally = [&](uint32_t bits) { red_shared_inc(mid + (uint32_t)sample_digit_offset(bits)); };
    if (own_sample) {
#pragma unroll
      for (int j = 0; j < kRegSlabs; ++j) {
        const int g = sh.g0 + j * NT + tid;
        if (j < slabs && g >= sh.i0 && g < sh.i1) {
          tally(__float_as_uint(xr[j].x));
          tally(__float_as_uint(xr[j].y));
          tally(__float_as_uint(xr[j].z));
          tally(__float_as_uint(xr[j].w));
        }
      }
    } else if constexpr (kForm != kRoomyForm) {
      // The next batch of a long row is on its way while this one is counted: its shards are far too long for
      // the registers, and the next batch takes their place. (Not where a thread has registers to spare: a
      // row of two batches over 16 CTAs took 15.1 us like this, and 14.85 with one batch after the other.)
      static_assert(NT * kRegSlabs * 4 * kMaxCluster <= 262144, "rows of one batch");
      for (int b = 0;; b += 2) {
        if (b + 1 < smp.nb) smp.load(sh.gbase, b + 1, xr);
        smp.use(b, xs, tally);
        if (b + 1 >= smp.nb) break;
        if (b + 2 < smp.nb) smp.load(sh.gbase, b + 2, xs);
        smp.use(b + 1, xr, tally);
        if (b + 2 >= smp.nb) break;
      }
    } else {
      for (int b = 0;;) {
        smp.use(b, xs, tally);
        if (++b >= smp.nb) break;
        smp.load(sh.gbase, b, xs);
      }
    }
    __syncthreads();
    FFTOPK_MARK(2);
    const uint32_t room = (uint32_t)(kLone ? lone_room_weighed(p.list_cap, NT) : p.cand_cap);
    // (one thread, when it has found the bin) what the guess is and what to do about it: see weigh_guess
    auto weigh = [&](uint32_t low, uint32_t width, uint32_t above, uint32_t cnt, uint32_t rest, uint32_t parent) {
      const uint32_t flags = weigh_guess(width, above, cnt, parent, smp.size(), (float)len, K, kCoarseFactor, room);
      if (flags & kGuessCopies) ctrl->focus = low + width - 1u;
      ctrl->guess = low;
      ctrl->guess_flags = flags & ~kGuessCopies;
      if (flags & kGuessCoarse) {
        ctrl->cnt = width;
        ctrl->local_c = cnt;
        ctrl->above = above;
        ctrl->need = rest;
      }
    };
    {
      const uint32_t need_s = ctrl->need, need_hi = ctrl->need_hi;
      block_pick_sample<NT>(h0, need_s, need_hi, wtot_s,
                            [&](uint32_t bin, uint32_t above, uint32_t cnt) {
                              weigh(sample_digit_low(bin), sample_digit_width(bin), above, cnt, need_s - above, 0xffffffffu);
                            },
                            [&](uint32_t bin) { ctrl->focus = sample_digit_high(bin); });
    }
    FFTOPK_MARK(3);
    uint32_t flags = ctrl->guess_flags;
    while (flags & kGuessCoarse) {  // (uniform; every round narrows the bin by 12 bits)
      const uint32_t low = ctrl->guess, width = ctrl->cnt, above0 = ctrl->above, rest = ctrl->need;
      const uint32_t cnt0 = ctrl->local_c;
      const int shift = second_look_shift(width);
      __syncthreads();  // everybody has read the result of the search before
      for (int i = tid; i < kMaxBins / 4; i += NT) sts_zero16(h0 + i * 16);
      if (tid == 0) ctrl->guess_flags = kGuessGiveUp;
      __syncthreads();
      for (int b = 0; b < smp.nb; ++b) {
        smp.load(sh.gbase, b, xs);
        smp.use(b, xs, [&](uint32_t bits) {
          const uint32_t off = fftopk_key_from_bits(bits) - low;
          if (off < width) red_shared_inc(h0 + ((off >> shift) & (uint32_t)(kMaxBins - 1)) * 4u);
        });
      }
      __syncthreads();
      block_pick_sample<NT>(h0, rest, 0u, wtot_s,
                            [&](uint32_t bin, uint32_t above, uint32_t cnt) {
                              weigh(low + (bin << shift), 1u << shift, above0 + above, cnt, rest - above, cnt0);
                            },
                            [&](uint32_t) {});
      flags = ctrl->guess_flags;
      FFTOPK_MARK(11);
    }
    gkey = ctrl->guess;
    focus_key = ctrl->focus;
    guessed = flags == 0u;
    if constexpr (kLone) {
      for (int i = tid; i < kFinishBins / 4; i += NT) sts_zero16(fh + i * 16);
      __syncthreads();
    }
  }
  FFTOPK_MARK(4);

  uint32_t thr = 0u;  // this call's threshold key
  int mode = kModeFallback;
  // list layout: one segment per warp, then the spill area
  // (a lone CTA's segments hold indices only, as many as its warps have registers for)
  constexpr int kLoneRegs = lone_regs(NT);
  const uint32_t spill_cap = kLone ? 0u : (uint32_t)list_spill(p.list_cap);
  const uint32_t seg_cap = kLone ? (uint32_t)lone_segment(p.list_cap, NT) : ((uint32_t)p.list_cap - spill_cap) / NW;
  uint64_t* const seg = kLone ? nullptr : list + (size_t)warp * seg_cap;
  uint64_t* const spill = kLone ? nullptr : list + (size_t)NW * seg_cap;
  const LoneList lone{smem_u32(list) + (uint32_t)warp * seg_cap * 4u, seg_cap, ctrl};

  // ---- filter the shard against the guess -------------------------------------------------------
  // Lower edge of the guess as a float: key(x) >= gkey  <=>  !(x < edge), NaN included. Keys outside
  // the range real values map to (below -inf's key / above +inf's) admit everything instead; that
  // only lengthens the lists.
  const float edge = __uint_as_float(guess_edge_bits(gkey));
  const uint32_t lowkey = guess_low_key(gkey);  // every candidate's key lies in [lowkey, 0xffffffff]
  if (focus_key < lowkey) focus_key = 0xffffffffu;
  constexpr int U = NT >= 1024 ? 4 : FFTOPK_U512;
  uint32_t wcnt = 0u;
  bool staged = false;
  if (!guessed) {
    // No guess to filter with: say so the way an overflowed list does. (Every step from here on
    // depends on what the cluster's CTAs tell each other, not on what each has read for itself.)
    if (tid == 0) ctrl->pub_flag = 1u;
  } else if (kLone) {
    const float cut = edge == 0.f ? -0.f : edge;
    if (in_regs && edge > ninf) {
      wcnt = filter_regs_lone<kRegSlabs>(xr, slabs, 4 * (sh.g0 + tid) - sh.a, 4 * NT, cut, lone);
    } else {
      wcnt = filter_stream_lone<NT>(sh, cut, lone);
    }
  } else if (in_regs && edge > ninf) {
    wcnt = filter_regs<kRegSlabs>(xr, slabs, 4 * (sh.g0 + tid) - sh.a, 4 * NT, edge, seg, seg_cap, ctrl, spill, spill_cap);
  } else if (len <= 196608) {  // about 1.5 k candidates per row: most trips of the hit loop have work
    staged = true;
    wcnt = filter_shard<NT, U, true>(sh, edge, seg, seg_cap, ctrl, spill, spill_cap);
  } else {
    wcnt = filter_shard<NT, U, false>(sh, edge, seg, seg_cap, ctrl, spill, spill_cap);
  }
  const uint32_t wown = min(wcnt, seg_cap);
  FFTOPK_MARK(8);
  const int region = kLone ? 0 : p.region;  // slots of each CTA in rank 0's buffer
  int extra = 0;           // candidates beyond their CTAs' regions
  uint32_t total = 0u;     // candidates of the row
  RegSegCands<NT, kLoneRegs> held;
  if constexpr (kLone) {
    // ---- a lone CTA keeps its candidates where they are ------------------------------------------
    // Their keys go into registers, and the histogram of the finish's first round is built on the way.
    const KeyDigit dg = make_key_digit(lowkey, focus_key);
    held.seg = lone.seg_s;
    held.wn = (int)wown;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kLoneRegs; i += 4) {
      if (i * 32 >= held.wn) break;  // (uniform over the warp; nobody looks at registers beyond)
      uint32_t bits[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = (i + u) * 32 + lane;
        uint32_t idx = lds32_below(j, held.wn, held.seg + (uint32_t)j * 4u);
        if (!FFTOPK_CHECK(7, idx, sh.len, p.status)) idx = 0u;
        bits[u] = __float_as_uint(Elem<T>::ld1(sh.gbase + idx + sh.a));  // (index 0 is always readable)
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        held.key[i + u] = 0u;
        if ((i + u) * 32 < held.wn) {  // (uniform)
          if ((i + u) * 32 + lane < held.wn) {
            held.key[i + u] = fftopk_key_from_bits(bits[u]);
            red_shared_inc(fh + dg.of(held.key[i + u]) * 4u);
          }
        }
      }
    }
    const uint32_t wn_s = smem_u32(ctrl->wmax);
    if (lane == 0) sts32(wn_s + warp * 4, wown);  // (not wtot: the finish's search may write that before every warp has read it)
    __syncthreads();
    total = __reduce_add_sync(kFull, lane < NW ? lds32(wn_s + lane * 4) : 0u);
    mode = sampled_attempt_ok(ctrl->pub_flag, total, K, 0xffffffffu) ? kModeGather : kModeFallback;
  } else {
    // ---- gather in rank 0 ----------------------------------------------------------------------
    // Every CTA owns a region of rank 0's buffer and fills it densely, so no slot has to be asked
    // for; only what does not fit there (a window of winners in one shard) takes a remote atomic and
    // goes behind the last region. Every CTA tells every other its count, so that each decides by
    // itself whether the guess held.
    const uint32_t wn_s = smem_u32(ctrl->wtot);
    if (lane == 0) sts32(wn_s + warp * 4, wown);
    cluster.barrier_wait();  // every CTA's control block is clear (see the prologue)
    __syncthreads();
    FFTOPK_MARK(44);
    const uint32_t w = lane < NW ? lds32(wn_s + lane * 4) : 0u;
    const uint32_t own = __reduce_add_sync(kFull, w);
    const uint32_t before = __reduce_add_sync(kFull, lane < warp ? w : 0u);
    const uint32_t sn = min(ctrl->lcount, spill_cap);
    if (warp == 0 && lane < C)
      st_peer32(peer_smem(smem_u32(&ctrl->cnt_of[rank]), lane), (own + sn) | (ctrl->pub_flag ? kOverflowed : 0u));
    uint32_t xbase = 0u;  // where the candidates beyond the region go: region * C + xbase + (their number - region)
    if (own + sn > (uint32_t)region) {  // (uniform over the CTA)
      if (tid == 0) ctrl->base_c = atomicAdd(&cx.ctrl0->extra_count, own + sn - (uint32_t)region);
      __syncthreads();
      xbase = ctrl->base_c;
    }
    const uint32_t cand0 = peer_smem(smem_u32(cx.cand), 0);
    bool dropped = false;
    auto push = [&](uint32_t q, uint64_t c) {  // candidate number q of this CTA
      uint32_t at = (uint32_t)(rank * region) + q;
      if (q >= (uint32_t)region) at = (uint32_t)(C * region) + xbase + (q - (uint32_t)region);
      dropped = dropped || at >= (uint32_t)p.cand_cap;
      if (at < (uint32_t)p.cand_cap) st_peer64(cand0 + at * 8u, c);
    };
    drain_segment(staged, sh, seg, wown, ctrl, [&](uint32_t j, uint64_t c) { push(before + j, c); });
    for (uint32_t j = tid; j < sn; j += NT) push(own + j, spill[j]);
    FFTOPK_MARK(46);
    cluster.sync();  // every candidate has landed in rank 0, every CTA knows the counts
    FFTOPK_MARK(9);
    const uint32_t n_r = lane < C ? lds32(smem_u32(ctrl->cnt_of) + lane * 4) : 0u;
    const uint32_t over = __any_sync(kFull, n_r >= kOverflowed) ? 1u : 0u;
    const uint32_t cnt_r = n_r & (kOverflowed - 1u);
    total = __reduce_add_sync(kFull, cnt_r);
    extra = (int)__reduce_add_sync(kFull, cnt_r > (uint32_t)region ? cnt_r - (uint32_t)region : 0u);
    // fewer than k admitted (the guess was too high), a list overflowed, or more than rank 0
    // can hold: start over with full histograms
    mode = sampled_attempt_ok(over | (extra > p.cand_cap - C * region ? 1u : 0u), total, K, 0xffffffffu) ? kModeGather
                                                                                                       : kModeFallback;
#ifdef FFTOPK_CHECKED
    // (a candidate may be dropped only where the counts tell every CTA that the buffer was too small)
    if (dropped && mode == kModeGather) check_fail(14, (uint32_t)extra, (uint32_t)p.cand_cap, p.status);
#endif
  }
  if constexpr (kWarm) {
    // (a miss is worth knowing about: the row is then selected by the full-histogram path)
    if (warm && mode == kModeFallback && rank == 0 && tid == 0 && p.status)
      atomicOr(p.status, (uint32_t)FFTOPK_ST_GUESS_MISSED);
  }
  // The candidates are rank 0's business now. Nobody reads a peer's memory any more, so the others may
  // leave, and rank 0 needs no barrier at the end.
  if (mode == kModeGather && rank != 0) return;
  FFTOPK_MARK(5);
  const RowOutput ro = row_output(p, row, K);
  int32_t* const out_idx = cx.out_idx = ro.idx;
  uint32_t* const out_key = cx.out_key = ro.key;
  cx.page = ctrl->row_page;
  cx.idx_offset = ctrl->row_idx_offset;

  const int idx_bits = 32 - __clz(len - 1);
  if (rank == 0) FFTOPK_ROUTE(mode == kModeGather ? kRouteHeld : kRouteHistograms);
  if (rank == 0 && mode == kModeGather && extra > 0) FFTOPK_ROUTE(kRouteBeyond);
  if (mode == kModeGather) {
    if constexpr (kLone) {
      const FinishOut o{{out_idx, out_key, p.status, cx.page, 0u, K, cx.idx_offset, K}, ctrl};
      lone_finish<NT, kLoneRegs, kWarm>(held, o, K, lowkey, focus_key, idx_bits, fin_hist);
    } else {
      const RegionCands<NT> src{smem_u32(cx.cand), smem_u32(ctrl->cnt_of), region, C, extra};
      constexpr int kCopies = NT == 512 && kForm == kRoomyForm ? kCopiesBack : kCopiesRest;  // (128 registers a thread, or 64)
      cta_finish<NT, RegionCands<NT>, kWarm, kCopies>(src, K, lowkey, 0xffffffffu, focus_key, idx_bits, fin_hist, ctrl, out_idx, out_key, 0u,
                                             K, cx.idx_offset, p.status, cx.page, total, true);
    }
    // This call's threshold for the next one: the smallest key the finish let win (the row's k-th
    // largest key).
    if constexpr (kWarm) {
      __syncthreads();
      thr = ctrl->thr_key != 0xffffffffu ? ctrl->thr_key : 0u;
    }
  } else {
    const RowCtx<NT, T> ctx = cx;  // (a copy: an object that is passed on this way lives on the stack)
    thr = select_by_full_histograms<NT, kWarm, T>(ctx);
    if (rank != 0) return;
  }
  if constexpr (kWarm) {
    if (tid == 0 && p.next_threshold != nullptr) p.next_threshold[row] = thr;
  }
  FFTOPK_MARK(7);
}

template <int NT, int kForm, bool kAnyK = false, bool kWarm = false, class T = float>
__global__ void __launch_bounds__(NT, min_ctas<NT>(kForm)) select2048_kernel(const SelectParams p) {
  select_row<NT, kAnyK, kWarm, T, kForm>(p);
  if (p.cp_publish) {
    // Context-parallel publication folded into the selection: the CTA's barrier orders every
    // thread's output writes before thread 0's arrival, a release at device scope (one operation
    // by the arriving thread, as in a grid-wide barrier, instead of a fence per thread); the last
    // CTA of the grid, which has acquired all the others' arrivals, releases the epoch flag
    // system-wide (peers acquire it in their merge kernel). The counter goes back to zero for the
    // next launch, which stream order keeps behind this one.
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t* arrive = p.cp_publish + kCommArriveWord;
      uint32_t old;
      asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(arrive) : "memory");
      if (old == gridDim.x - 1u) {
        *arrive = 0u;
        const uint32_t epoch = p.cp_epoch ? p.cp_epoch : __ldcg(p.cp_publish) + 1u;
        __threadfence_system();
        asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p.cp_publish), "r"(epoch) : "memory");
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Context-parallel top-2048 in ONE launch per GPU: local selection, exchange and merge. Every GPU
// holds a contiguous slice of each row. The row's cluster first selects the local top 2048 of its
// slice (keys and global indices) exactly as select2048_kernel does; its first CTA then PUSHES the
// 2048 candidates as self-validating packets {index, epoch, key, epoch} into the inbox of every
// GPU, its own included, with plain 16-byte stores over NVLink - no flag, no fence (a system-scope
// fence was measured at 4.5 us per publication), no round trip. After that CTA g of the cluster
// (g < G) polls, in its own GPU's memory and with a time limit, the packets shard g sent for the
// row, and the cluster merges the G lists (merge_row). No second launch, no collective call, no
// launch-wide synchronisation: a row is merged as soon as its own G slices have been selected.
// The inbox has two halves that alternate by epoch parity: a GPU can only start call e+2 after
// its own call e+1 has seen every peer's packets of e+1, which the peer sent after it had finished
// call e and with it every read of its inbox half e.
// ---------------------------------------------------------------------------------------------
struct CpFused {
  uint4* inbox[kMaxShards];   // inbox (half 0, source shard 0, row 0) of every GPU, own included
  uint32_t* row_epoch;        // this GPU's epoch counter of row 0; row r's is kCommRowFlagWords * r further
  int64_t inbox_half_packets; // packets between the two halves of an inbox
  unsigned long long wait_ns;
  int32_t* out_idx;           // [B, 2048] merged result
  uint32_t epoch;             // epoch of this call, or 0: each row counter's value plus one
  int32_t G, own, b_cap;
};

template <int NT>
__global__ void __launch_bounds__(NT, min_ctas<NT>(kRoomyForm)) select_merge2048_kernel(const SelectParams p, const CpFused f) {
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks();
  const int rank = (int)cluster.block_rank();
  const int row = (int)(blockIdx.x / (unsigned)C);
  const int tid = threadIdx.x;
  uint32_t* my_epoch = f.row_epoch + (int64_t)row * kCommRowFlagWords;
  // launched as a programmatic dependent, like the selection kernel (see select_row): the call in
  // front of this one has to have completed before the row's epoch counter is read
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // (the previous call's update of the counter is complete - stream order - and this call's comes
  // at the very end: every CTA of the cluster reads the same value)
  const uint32_t epoch = f.epoch ? f.epoch : __ldcg(my_epoch) + 1u;
  if (C == 1) {
    select_row<NT, false, false, float, kLoneForm>(p);
  } else {
    select_row<NT, false, false, float, kRoomyForm>(p);
  }
  // Every output of the row is written: by this CTA, or by its peers before a cluster barrier
  // this CTA has passed.
  FFTOPK_MARK(60);
  // packets of (half, source shard, row): ((half * 8 + shard) * b_cap + row) * 2048
  const int64_t half_off = (int64_t)(epoch & 1u) * f.inbox_half_packets;
  if (rank == 0) {
    __syncthreads();
    constexpr int PER = kK / NT;
    const int32_t* lidx = p.out_idx + (int64_t)row * kK;
    const uint32_t* lkey = p.out_key + (int64_t)row * kK;
    const int64_t dst_off = half_off + ((int64_t)f.own * f.b_cap + row) * kK;
    int32_t ci[PER];
    uint32_t ck[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      ci[u] = __ldcg(lidx + u * NT + tid);
      ck[u] = __ldcg(lkey + u * NT + tid);
    }
    for (int d = 0; d < f.G; ++d) {
      uint4* dst = f.inbox[d] + dst_off;
#pragma unroll
      for (int u = 0; u < PER; ++u) st_packet(dst + u * NT + tid, ci[u], ck[u], epoch);
    }
  }
  FFTOPK_MARK(61);
  // ---- merge: same carve of the dynamic shared memory as the selection --------------------------
  extern __shared__ __align__(128) unsigned char smem_raw[];
  MergeSmem sm;
  sm.hist = reinterpret_cast<uint32_t*>(smem_raw);
  sm.sup = sm.hist + 2 * kMaxBins;
  sm.xch = sm.sup + 2 * kSup;
  sm.ctrl = reinterpret_cast<Ctrl*>(sm.xch + kMaxCluster * kSup);
  sm.cand = reinterpret_cast<uint64_t*>(reinterpret_cast<unsigned char*>(sm.ctrl) + ((sizeof(Ctrl) + 127) & ~127u));
  sm.cand_cap = C == 1 ? p.list_cap : p.list_cap + p.cand_cap;
  const uint4* mine = rank < f.G ? f.inbox[f.own] + half_off + ((int64_t)rank * f.b_cap + row) * kK : nullptr;
  merge_row<NT>(cluster, C, f.G, rank, sm, nullptr, nullptr, nullptr, mine, epoch, f.wait_ns,
                f.out_idx + (int64_t)row * kK, nullptr, p.status);
  // the row's epoch counter moves on only now: every CTA of the cluster read it before the first
  // cluster barrier of the merge
  if (rank == 0 && tid == 0 && f.epoch == 0u) *my_epoch = epoch;
  FFTOPK_MARK(69);
}

}  // namespace fftopk

// =============================================================================================
// Host side: launch plan and C ABI
// =============================================================================================
namespace {

using namespace fftopk;

// Process-wide overrides (fftopk_set_tuning, fftopk_set_overlap). Writers and readers go through
// the mutex; every launch works on its own snapshot.
struct Tuning {
  int cluster = -1, threads = -1, list_cap = -1, cand_cap = -1, force_slow = 0, overlap = 0;
};
std::mutex g_tuning_mu;
Tuning g_tuning;

Tuning tuning_snapshot() {
  std::lock_guard<std::mutex> lock(g_tuning_mu);
  return g_tuning;
}

using AddressRangeFn = CUresult (*)(CUdeviceptr*, size_t*, CUdeviceptr);  // cuMemGetAddressRange

struct DeviceInfo {
  DeviceOnce once;
  AddressRangeFn address_range = nullptr;
  int sm_count = 0;
  int smem_optin = 0;
  int cc_major = 0;
  int max_cluster = 0;  // largest cluster size that can be scheduled with the latency-mode footprint
  int active16 = 0, active8 = 0;  // clusters of that size the device holds at once (same footprint)
};
DeviceInfo g_dev[kMaxDevices];

// (everything but the lists; a lone CTA has one histogram and nobody to exchange super-bins with)
constexpr size_t fixed_smem_bytes(bool lone) {
  return (size_t)((lone ? 1 : 2) * kMaxBins + 2 * kSup + (lone ? 1 : kMaxCluster) * kSup) * 4 + ((sizeof(Ctrl) + 127) & ~(size_t)127);
}

constexpr int64_t kPrefetchRow = 1 << 20, kPrefetchBytes = 48 << 20;
constexpr int kLatencyListCap = 6144, kLatencyCandCap = 16384;  // one CTA per SM: use the shared memory
// One CTA per row, whatever its length and k: 640 or 384 candidates a warp (lone_segment), some 70 KB per CTA with the buffer
// that the full-histogram path gathers in. With two CTAs per SM the rest stays L1, which the second read of a candidate's value
// hits: a larger buffer for rows beyond 192K and for k > 2048 (9,216 composites, 94 KB) cost 150 rows of 1M 137 us instead
// of 114, 64 of 256K in overlapping calls 14.1 instead of 13.5.
constexpr int kOverlapListCap1 = 6144;
constexpr int kOverlapListCap = 3072, kOverlapCandCap = 6144;   // two CTAs per SM
// Rows so short that the list of a CTA of 256 threads holds all of them, whatever they are and wherever they start
// (make_plan, lone_edge_warp)
constexpr int kLoneListCap256 = 2560, kLoneCandCap256 = 2560;
constexpr int64_t kLoneRow256 = 4096;


using SelectFn = void (*)(SelectParams);

// The instantiations of the selection kernel.
enum Variant : int { kVar2048 = 0, kVarAnyK, kVarF16, kVarBF16, kVarWarm, kVariants };
template <int NT, int kForm>
SelectFn select_fn(int variant) {
  if constexpr (NT >= 512) {  // (256 threads: fp32 without a warm start only)
    switch (variant) {
      case kVarF16: return select2048_kernel<NT, kForm, true, false, __half>;
      case kVarBF16: return select2048_kernel<NT, kForm, true, false, __nv_bfloat16>;
      case kVarWarm: return select2048_kernel<NT, kForm, false, true>;
      default: break;
    }
  }
  return variant == kVarAnyK ? select2048_kernel<NT, kForm, true> : select2048_kernel<NT, kForm>;
}
SelectFn select_fn(int threads, int form, int variant) {
  const bool lone = form == kLoneForm;
  if (threads == 1024) return lone ? select_fn<1024, kLoneForm>(variant) : select_fn<1024, kRoomyForm>(variant);
  if (threads == 256) return lone ? select_fn<256, kLoneForm>(variant) : select_fn<256, kRoomyForm>(variant);
  return lone ? select_fn<512, kLoneForm>(variant)
              : (form == kTightForm ? select_fn<512, kTightForm>(variant) : select_fn<512, kRoomyForm>(variant));
}

template <class Fn>
int setup_fn(Fn fn, int smem_optin) {
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return e == cudaSuccess ? 0 : cuda_fail(e);
}
int setup_kernels(int smem_optin) {
  for (int threads = 256; threads <= 1024; threads *= 2) {
    for (int v = 0; v < kVariants; ++v) {
      for (int form = kLoneForm; form <= kTightForm; ++form) {
        const int rc = setup_fn(select_fn(threads, form, v), smem_optin);
        if (rc) return rc;
      }
    }
  }
  const int rc = setup_fn(select_merge2048_kernel<512>, smem_optin);
  return rc ? rc : setup_fn(select_merge2048_kernel<1024>, smem_optin);
}

int init_device(DeviceInfo& d, int dev) {
  cudaDeviceProp prop;
  cudaError_t e = cudaGetDeviceProperties(&prop, dev);
  if (e != cudaSuccess) return cuda_fail(e);
  d.sm_count = prop.multiProcessorCount;
  d.smem_optin = (int)prop.sharedMemPerBlockOptin;
  d.cc_major = prop.major;
  if (prop.major < 10) return FFTOPK_EDEVICE;
  const int rc = setup_kernels(d.smem_optin);
  if (rc) return rc;
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult qres;
  if (cudaGetDriverEntryPoint("cuMemGetAddressRange", &fn, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess)
    d.address_range = reinterpret_cast<AddressRangeFn>(fn);
  (void)cudaGetLastError();  // (without it no row is asked for ahead of time)
  // can a 16-CTA cluster with the latency-mode shared-memory footprint be co-scheduled, and how
  // many clusters of 16 / of 8 CTAs does the device hold at once? (A cluster lives inside one
  // GPC, so fewer 16-CTA clusters fit than SM count / 16: a batch with more rows than that would
  // run in two waves.)
  d.max_cluster = 8;
  d.active16 = 0;
  d.active8 = d.sm_count / 8;
  for (int cs = 16; cs >= 8; cs /= 2) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cs * 32, 1, 1);
    cfg.blockDim = dim3(512, 1, 1);  // (the form that such a plan launches)
    cfg.dynamicSmemBytes = fixed_smem_bytes(false) + (size_t)(kLatencyListCap + kLatencyCandCap) * 8;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int nclusters = 0;
    e = cudaOccupancyMaxActiveClusters(&nclusters, select2048_kernel<512, kRoomyForm>, &cfg);
    if (e == cudaSuccess && nclusters >= 1) {
      if (cs == 16) {
        d.max_cluster = 16;
        d.active16 = nclusters;
      } else {
        d.active8 = nclusters;
      }
    }
    (void)cudaGetLastError();
  }
  return 0;
}

// Properties of the current device; the first call on a device (any thread) sets the kernels'
// function attributes.
int device_info(DeviceInfo** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e);
  if (dev < 0 || dev >= kMaxDevices) return FFTOPK_EDEVICE;
  DeviceInfo& d = g_dev[dev];
  const int rc = d.once.run([&] { return init_device(d, dev); });
  if (rc) return rc;
  *out = &d;
  return 0;
}

// Whether all rows of a call lie inside one allocation, as far as L. A query of the driver on the host (an eager call
// takes 9.14 us of host time with it, 9.10 without), which fails for memory that it knows nothing about.
bool rows_allocated(const DeviceInfo& d, const SelectCall& c, int element_bytes) {
  if (d.address_range == nullptr) return false;
  CUdeviceptr base = 0;
  size_t size = 0;
  const uint64_t score = reinterpret_cast<uint64_t>(c.score);
  if (d.address_range(&base, &size, (CUdeviceptr)score) != CUDA_SUCCESS) return false;
  return rows_inside(score, c.row_stride, c.B, c.L, element_bytes, (uint64_t)base, (uint64_t)size);
}

struct Plan {
  int cluster, threads, smem_bytes, list_cap, cand_cap;
};

int floor_pow2(int64_t v) {
  int r = 1;
  while ((int64_t)r * 2 <= v) r *= 2;
  return r;
}

// The lists of a lone CTA: one for the filter, and in the same memory the one the full-histogram path gathers in.
// What they leave of the SM's 256 KB is L1, through which every load of the stream passes.
void lone_lists(Plan& pl, int list_cap) {
  pl.list_cap = list_cap;
  pl.cand_cap = pl.threads == 256 ? std::min(list_cap, kLoneCandCap256) : list_cap;
  pl.smem_bytes = (int)(fixed_smem_bytes(true) + std::max((size_t)lone_room(list_cap, pl.threads) * 4, (size_t)pl.cand_cap * 8));
}

// Replaces the reference's split heuristic (topk_indexer_radix.cu:1081-1111: at most 8 CTAs per
// row, a hard-coded SM count of 132). `overlap`: the launch may overlap its neighbours on the
// stream (throughput plan). `narrow`: the call's kernel exists for 256 threads.
Plan make_plan(const DeviceInfo& d, const Tuning& tn, bool overlap, int B, int64_t L, bool narrow) {
  Plan pl;
  const int rows = B > 0 ? B : 1;
  // CTAs per row: as many as keep the whole grid resident at once with one CTA per SM, but never
  // so many that a shard drops below ~2K elements.
  int c = floor_pow2(d.sm_count / rows > 0 ? d.sm_count / rows : 1);
  if (c > d.max_cluster) c = d.max_cluster;
  if (c == 16 && rows > d.active16) c = 8;  // all rows in one wave
  if (c == 8 && rows > d.active8) c = 4;
  const int by_len = floor_pow2(L / 2048 > 0 ? L / 2048 : 1);
  if (c > by_len) c = by_len;
  pl.cluster = c < 1 ? 1 : c;
  // A cluster's CTAs are bound by the instructions their warps issue, and much of that is per warp
  // (scans, searches, address arithmetic): 512 threads do it with half the warps and, one CTA per SM,
  // twice the registers. Measured, us per call in a chain, 512 / 1024 threads: B=1, L=16K 9.5 / 10.1,
  // 96K 10.5 / 11.35, 1M 14.6 / 14.9; B=64 ragged rows of up to 128K 18.5 / 18.5. A lone CTA has no
  // other CTA to share its row with: 1024.
  pl.threads = pl.cluster > 1 ? 512 : 1024;
  pl.list_cap = kLatencyListCap;
  pl.cand_cap = kLatencyCandCap;
  if (rows > d.sm_count) {
    // More rows than SMs: the batch fills the device by itself. One 512-thread CTA per row with
    // the list of the throughput plan, two CTAs per SM (ragged rows of up to 128K elements, 512 / 1024 threads:
    // 22.0 / 25.9 us per call at B=256, 37.2 / 42.5 at B=512; 2,048 rows of 32K 81 / 115). (The gather buffer is for
    // tunings that ask for more CTAs per row.)
    pl.cluster = 1;
    pl.threads = 512;
    pl.list_cap = kOverlapListCap1;
    pl.cand_cap = kOverlapCandCap;
  }
  if (overlap) {
    // Back-to-back calls may overlap: what counts is work per row, not the latency of one call.
    // Few CTAs per row (less cluster traffic per row), 512 threads and 70 KB (one CTA per row) or 115 KB of shared
    // memory so that two CTAs - of different calls - share an SM, and about four calls in flight.
    int ct = floor_pow2(d.sm_count / (4 * rows) > 0 ? d.sm_count / (4 * rows) : 1);
    if (ct < pl.cluster) pl.cluster = ct;
    pl.threads = 512;
    if (pl.cluster == 1) {
      pl.list_cap = kOverlapListCap1;
    } else {
      pl.list_cap = kOverlapListCap;
      pl.cand_cap = kOverlapCandCap;
    }
  }
  if (narrow && pl.cluster == 1 && pl.threads == 512 && L <= kLoneRow256) {
    // Short rows: four CTAs of 256 threads share an SM, each with some 40 KB, and the phases in which one of them has
    // little to do are the others' time. 2,048 rows, 256 / 512 threads: 4K elements 35.9 / 46.9 us, with 70 % zeros
    // 87 / 90, 6K with zeros 176 / 119 - rows that may overflow their list stay with 512 (8K of N(0,1) 45.9 / 53.8).
    pl.threads = 256;
    pl.list_cap = kLoneListCap256;
  }
  if (tn.cluster > 0) pl.cluster = tn.cluster;
  if (tn.threads > 0) pl.threads = tn.threads;
  if (tn.list_cap > 0) pl.list_cap = (tn.list_cap + 15) & ~15;
  if (tn.cand_cap > 0) pl.cand_cap = (tn.cand_cap + 15) & ~15;
  if (pl.cluster == 1) {
    lone_lists(pl, pl.list_cap);
  } else {
    pl.smem_bytes = (int)(fixed_smem_bytes(false) + (size_t)(pl.list_cap + pl.cand_cap) * 8);
  }
  return pl;
}

SelectCall basic_call(const float* score, int64_t row_stride, int32_t B, int64_t L, const int32_t* lengths,
                      const int32_t* row_starts, int32_t* out_idx, uint32_t* out_key, int32_t idx_offset,
                      uint32_t* status, void* cuda_stream) {
  SelectCall c;
  c.score = score;
  c.row_stride = row_stride;
  c.B = B;
  c.L = L;
  c.lengths = lengths;
  c.row_starts = row_starts;
  c.out_idx = out_idx;
  c.out_key = out_key;
  c.idx_offset = idx_offset;
  c.status = status;
  c.cuda_stream = cuda_stream;
  return c;
}

}  // namespace

namespace fftopk {

int launch_select(const SelectCall& c) {
  if (c.B < 0 || c.L < 0 || c.row_stride < 0 || c.k < 1 || c.k > kMaxK) return FFTOPK_EINVAL;
  if (c.B == 0) return FFTOPK_OK;
  if (!c.score || !c.lengths || !c.out_idx) return FFTOPK_EINVAL;
  const bool half_width = c.dtype != kDtypeF32;
  if ((reinterpret_cast<uintptr_t>(c.score) & (half_width ? 1u : 3u)) != 0) return FFTOPK_EINVAL;
  if (c.L > (int64_t)0x7fffffff - 8 || (int64_t)c.B * kMaxCluster > (int64_t)0x7fffffff) return FFTOPK_ERANGE;
  DeviceInfo* d = nullptr;
  int rc = device_info(&d);
  if (rc) return rc;
  const Tuning tn = tuning_snapshot();
  const bool overlap = tn.overlap != 0 && c.may_overlap;
  const bool warm = c.prev_threshold != nullptr || c.next_threshold != nullptr;
  Plan pl = make_plan(*d, tn, overlap, c.B, c.L, !half_width && !warm);
  if (half_width && pl.threads < 512) {  // (the 16-bit kernels exist for 512 and 1024 threads)
    pl.threads = 512;
    if (pl.cluster == 1) lone_lists(pl, pl.list_cap);
  }

  SelectParams p;
  p.score = c.score;
  p.row_stride = c.row_stride;
  p.L = c.L;
  p.lengths = c.lengths;
  p.row_starts = c.row_starts;
  p.out_idx = c.out_idx;
  p.out_key = c.out_key;
  p.status = c.status;
  p.B = c.B;
  p.k = c.k;
  p.idx_offset = c.idx_offset;
  p.list_cap = pl.list_cap;
  p.cand_cap = pl.cand_cap;
  p.region = pl.cluster > 1 ? gather_region(pl.cand_cap, pl.list_cap, pl.cluster) : 0;
  p.force_slow = tn.force_slow;
  p.overlap = overlap ? 1 : 0;
  // Rows that a cluster streams (shorter ones go to registers at once, and gain nothing) are asked for ahead, if all of them
  // take no more than a good part of L2; not where the launch in front is the library's own and still writes them, nor with a
  // place to start in every row. us per call in a chain whose rows lie in HBM, without / with: one row of 512K
  // 15.3 / 13.5, 1M 18.9 / 16.1, 2M 26.0 / 25.5; 4 of 300K 14.9 / 13.2, 7 of 1M 19.9 / 18.1, 20 ragged of 400K 23.6 / 20.2;
  // of 256K 10.7 / 10.7. Rows in L2 already: 1M 13.9 / 13.9. (A warm start waits for little else than the length, which
  // the request reads as well: 4 rows of 200K in L2 8.48 / 8.65, so it does not ask.)
  const int64_t row_bytes = c.L * (half_width ? 2 : 4);
  // (the rows have to be there as far as L: see rows_inside)
  p.prefetch = c.may_overlap && !overlap && !c.row_starts && row_bytes > kPrefetchRow && c.B * row_bytes <= kPrefetchBytes &&
                       rows_allocated(*d, c, half_width ? 2 : 4)
                   ? 1
                   : 0;
  p.src_page_table = c.src_page_table;
  p.src_stride = c.src_stride;
  p.cu_seqlens_q = c.cu_seqlens_q;
  p.prefill_bs = c.prefill_bs;
  p.row_offsets = c.row_offsets;
  p.cp_flag = c.cp_flag;
  p.cp_half_words = c.cp_half_words;
  p.cp_publish = c.cp_publish;
  p.cp_epoch = c.cp_epoch;
  p.prev_threshold = c.prev_threshold;
  p.next_threshold = c.next_threshold;
  p.warm_margin = c.warm_margin;
  p.cand = c.cand;
  p.cand_guess = c.cand_guess;
  if (warm && (c.k != kK || pl.threads < 512)) return FFTOPK_EINVAL;
  // (the indices of a row's given candidates lie where the list does)
  if (c.cand) pl.smem_bytes = std::max(pl.smem_bytes, (int)fixed_smem_bytes(false) + (kIdxCandCap + pl.threads) * 4);
  if ((size_t)pl.smem_bytes > (size_t)d->smem_optin) return FFTOPK_ERANGE;

  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)c.B * (unsigned)pl.cluster, 1, 1);
  cfg.blockDim = dim3((unsigned)pl.threads, 1, 1);
  cfg.dynamicSmemBytes = (size_t)pl.smem_bytes;
  cfg.stream = static_cast<cudaStream_t>(c.cuda_stream);
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)pl.cluster;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  // (every launch: see the top of select_row for what the kernel does with it)
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 2;
  int variant = c.k != kK ? kVarAnyK : kVar2048;
  if (half_width) {
    if (warm || c.src_page_table || c.cp_flag || c.cp_publish) return FFTOPK_EINVAL;
    variant = c.dtype == kDtypeF16 ? kVarF16 : kVarBF16;
  } else if (warm) {
    variant = kVarWarm;
  }
  if (c.in_front) {  // (nothing below refuses the call)
    rc = c.in_front(c.in_front_arg);
    if (rc) return rc;
  }
  const cudaError_t e = cudaLaunchKernelEx(&cfg, select_fn(pl.threads, pl.cluster == 1 ? kLoneForm : (overlap ? kTightForm : kRoomyForm), variant), p);
  if (e != cudaSuccess) return cuda_fail(e);
  return FFTOPK_OK;
}

// Single-launch context-parallel call (see select_merge2048_kernel). FFTOPK_ERANGE when the
// launch plan for (B, L) gives a row fewer CTAs than there are shards or too little shared memory
// for the merge: the caller then uses the two-launch sequence.
int launch_select_merge(const SelectCall& c, void* const* comms, int32_t G, int32_t own, int32_t b_cap, uint32_t epoch,
                        int32_t wait_ms, int32_t* out_idx) {
  if (c.B < 0 || c.L < 0 || c.row_stride < 0) return FFTOPK_EINVAL;
  if (!comms || G < 1 || own < 0 || own >= G || b_cap < 1 || c.B > b_cap || wait_ms < 0) return FFTOPK_EINVAL;
  if (G > kMaxShards) return FFTOPK_ERANGE;
  if (c.B == 0) return FFTOPK_OK;
  if (!c.score || !c.lengths || !out_idx) return FFTOPK_EINVAL;
  if ((reinterpret_cast<uintptr_t>(c.score) & 3u) != 0) return FFTOPK_EINVAL;
  if (c.L > (int64_t)0x7fffffff - 8) return FFTOPK_ERANGE;
  DeviceInfo* d = nullptr;
  int rc = device_info(&d);
  if (rc) return rc;
  const Tuning tn = tuning_snapshot();
  Plan pl = make_plan(*d, tn, false, c.B, c.L, false);
  if (pl.cluster == 1) pl.smem_bytes = (int)(fixed_smem_bytes(false) + (size_t)pl.list_cap * 8);  // (the merge's two histograms and candidates)
  const int room = pl.cluster == 1 ? pl.list_cap : pl.list_cap + pl.cand_cap;
  if (pl.cluster < G || room < G * kK || pl.threads < 512 || (size_t)pl.smem_bytes > (size_t)d->smem_optin) return FFTOPK_ERANGE;

  SelectParams p;
  memset(&p, 0, sizeof(p));
  CpFused f;
  memset(&f, 0, sizeof(f));
  for (int g = 0; g < G; ++g) {
    if (!comms[g]) return FFTOPK_EINVAL;
    f.inbox[g] = reinterpret_cast<uint4*>(static_cast<int32_t*>(comms[g]) + comm_inbox_offset(b_cap));
  }
  int32_t* own_words = static_cast<int32_t*>(comms[own]);
  f.row_epoch = reinterpret_cast<uint32_t*>(own_words + comm_rowflag_offset(b_cap));
  f.inbox_half_packets = (int64_t)(comm_inbox_half_words(b_cap) / 4);
  f.wait_ns = (unsigned long long)wait_ms * 1000000ull;
  f.out_idx = out_idx;
  f.epoch = epoch;
  f.G = G;
  f.own = own;
  f.b_cap = b_cap;
  p.score = c.score;
  p.row_stride = c.row_stride;
  p.L = c.L;
  p.lengths = c.lengths;
  p.out_idx = own_words + comm_stage_offset(b_cap);  // local selection output, pushed from there
  p.out_key = reinterpret_cast<uint32_t*>(p.out_idx + (size_t)b_cap * kK);
  p.status = c.status;
  p.B = c.B;
  p.k = kK;
  p.idx_offset = c.idx_offset;
  p.list_cap = pl.list_cap;
  p.cand_cap = pl.cand_cap;
  p.region = pl.cluster > 1 ? gather_region(pl.cand_cap, pl.list_cap, pl.cluster) : 0;
  p.force_slow = tn.force_slow;

  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)c.B * (unsigned)pl.cluster, 1, 1);
  cfg.blockDim = dim3((unsigned)pl.threads, 1, 1);
  cfg.dynamicSmemBytes = (size_t)pl.smem_bytes;
  cfg.stream = static_cast<cudaStream_t>(c.cuda_stream);
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)pl.cluster;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  const cudaError_t e = pl.threads == 1024 ? cudaLaunchKernelEx(&cfg, select_merge2048_kernel<1024>, p, f)
                                           : cudaLaunchKernelEx(&cfg, select_merge2048_kernel<512>, p, f);
  if (e != cudaSuccess) return cuda_fail(e);
  return FFTOPK_OK;
}

}  // namespace fftopk

extern "C" {

int fftopk_version(void) { return 200; }

const char* fftopk_strerror(int code) {
  switch (code) {
    case FFTOPK_OK: return "ok";
    case FFTOPK_EINVAL: return "invalid argument";
    case FFTOPK_ECUDA: return "CUDA runtime call failed";
    case FFTOPK_EDEVICE: return "device is not an sm_100-class GPU with cluster launch";
    case FFTOPK_ERANGE: return "size out of the supported range";
    default: return "unknown error";
  }
}

int fftopk_last_cuda_error(void) { return fftopk::g_last_cuda_error; }

#ifdef FFTOPK_CHECKED
// Checked builds only: the first violation recorded by the selection kernels (rec[0..3]) and by the
// merge kernel (rec[4..7]) as (site, index, limit, block); site 0 = none. Clears both records.
int fftopk_checked_read(uint32_t rec[8]) {
  const uint32_t zero[4] = {0u, 0u, 0u, 0u};
  cudaError_t e = cudaMemcpyFromSymbol(rec, fftopk::g_check_rec, sizeof(zero));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(fftopk::g_check_rec, zero, sizeof(zero));
  if (e != cudaSuccess) return fftopk::cuda_fail(e);
  return fftopk::checked_read_merge(rec + 4);
}

// Checked builds only: the rows selected since the last call, by the way they took (kRoute*). Clears the counts.
int fftopk_checked_routes(uint32_t counts[3]) {
  const uint32_t zero[3] = {0u, 0u, 0u};
  cudaError_t e = cudaMemcpyFromSymbol(counts, fftopk::g_routes, sizeof(zero));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(fftopk::g_routes, zero, sizeof(zero));
  return e == cudaSuccess ? 0 : fftopk::cuda_fail(e);
}
#endif

#ifdef FFTOPK_TRACE
int fftopk_trace_read(unsigned long long* times, int* ids, int* n) {
  cudaError_t e = cudaMemcpyFromSymbol(n, fftopk::g_trace_n, sizeof(int));
  if (e == cudaSuccess) e = cudaMemcpyFromSymbol(times, fftopk::g_trace_t, sizeof(unsigned long long) * fftopk::kTraceCap);
  if (e == cudaSuccess) e = cudaMemcpyFromSymbol(ids, fftopk::g_trace_id, sizeof(int) * fftopk::kTraceCap);
  return (int)e;
}
int fftopk_trace_clear(void) {
  const int z = 0;
  return (int)cudaMemcpyToSymbol(fftopk::g_trace_n, &z, sizeof(int));
}
#endif

uint32_t fftopk_key_of(float x) {
  uint32_t bits;
  __builtin_memcpy(&bits, &x, 4);
  return fftopk_key_from_bits(bits);
}

int fftopk_set_tuning(int32_t cluster_ctas, int32_t threads, int32_t list_cap, int32_t cand_cap,
                      int32_t force_full_histogram) {
  if (cluster_ctas > 0 && (cluster_ctas > kMaxCluster || (cluster_ctas & (cluster_ctas - 1)))) return FFTOPK_EINVAL;
  if (threads > 0 && threads != 256 && threads != 512 && threads != 1024) return FFTOPK_EINVAL;
  if (cand_cap > 0 && (cand_cap < 32 || cand_cap > 16384)) return FFTOPK_EINVAL;
  if (list_cap > 0 && (list_cap < 32 || list_cap > 16384)) return FFTOPK_EINVAL;
  std::lock_guard<std::mutex> lock(g_tuning_mu);
  g_tuning.cluster = cluster_ctas;
  g_tuning.threads = threads;
  g_tuning.list_cap = list_cap;
  g_tuning.cand_cap = cand_cap;
  g_tuning.force_slow = force_full_histogram > 0 ? 1 : 0;
  return FFTOPK_OK;
}

int fftopk_set_overlap(int32_t enable) {
  std::lock_guard<std::mutex> lock(g_tuning_mu);
  g_tuning.overlap = enable ? 1 : 0;
  return FFTOPK_OK;
}

int fftopk_plan(int32_t B, int64_t L, int32_t plan[6]) {
  if (!plan || B < 0 || L < 0) return FFTOPK_EINVAL;
  DeviceInfo* d = nullptr;
  int rc = device_info(&d);
  if (rc) return rc;
  const Tuning tn = tuning_snapshot();
  const Plan pl = make_plan(*d, tn, tn.overlap != 0, B, L, true);
  plan[0] = pl.cluster;
  plan[1] = pl.threads;
  plan[2] = pl.smem_bytes;
  plan[3] = pl.list_cap;
  plan[4] = pl.cand_cap;
  plan[5] = d->sm_count;
  return FFTOPK_OK;
}

int fftopk_select2048(const float* score, int64_t row_stride, int32_t B, int64_t L, const int32_t* lengths,
                      const int32_t* row_starts, int32_t* out_idx, uint32_t* out_key, int32_t idx_offset,
                      uint32_t* status, void* cuda_stream) {
  return launch_select(basic_call(score, row_stride, B, L, lengths, row_starts, out_idx, out_key, idx_offset, status,
                                  cuda_stream));
}

int fftopk_select_topk(const float* score, int64_t row_stride, int32_t B, int64_t L, const int32_t* lengths,
                       const int32_t* row_starts, int32_t k, int32_t* out_idx, uint32_t* out_key, int32_t idx_offset,
                       uint32_t* status, void* cuda_stream) {
  SelectCall c = basic_call(score, row_stride, B, L, lengths, row_starts, out_idx, out_key, idx_offset, status, cuda_stream);
  c.k = k;
  return launch_select(c);
}

int fftopk_select2048_warm(const float* score, int64_t row_stride, int32_t B, int64_t L, const int32_t* lengths,
                           const int32_t* row_starts, const uint32_t* prev_threshold, uint32_t margin,
                           uint32_t* next_threshold, int32_t* out_idx, uint32_t* status, void* cuda_stream) {
  if (B > 0 && !prev_threshold && !next_threshold) return FFTOPK_EINVAL;
  SelectCall c = basic_call(score, row_stride, B, L, lengths, row_starts, out_idx, nullptr, 0, status, cuda_stream);
  c.prev_threshold = prev_threshold;
  c.next_threshold = next_threshold;
  c.warm_margin = margin;
  return launch_select(c);
}

int fftopk_select2048_page_table(const float* score, int64_t row_stride, int32_t B, int64_t L,
                                 const int32_t* lengths, const int32_t* row_starts, int32_t* dst_page_table,
                                 const int32_t* src_page_table, int64_t src_stride, const int32_t* cu_seqlens_q,
                                 int32_t prefill_bs, uint32_t* status, void* cuda_stream) {
  if (B > 0 && (!src_page_table || src_stride < 0 || prefill_bs < 1 || prefill_bs > B)) return FFTOPK_EINVAL;
  SelectCall c = basic_call(score, row_stride, B, L, lengths, row_starts, dst_page_table, nullptr, 0, status, cuda_stream);
  c.src_page_table = src_page_table;
  c.src_stride = src_stride;
  c.cu_seqlens_q = cu_seqlens_q;
  c.prefill_bs = prefill_bs;
  return launch_select(c);
}

int fftopk_select2048_ragged(const float* score, int64_t row_stride, int32_t B, int64_t L, const int32_t* lengths,
                             const int32_t* row_starts, int32_t* topk_indices_ragged,
                             const int32_t* topk_indices_offset, uint32_t* status, void* cuda_stream) {
  if (B > 0 && !topk_indices_offset) return FFTOPK_EINVAL;
  SelectCall c = basic_call(score, row_stride, B, L, lengths, row_starts, topk_indices_ragged, nullptr, 0, status, cuda_stream);
  c.row_offsets = topk_indices_offset;
  return launch_select(c);
}

}  // extern "C"

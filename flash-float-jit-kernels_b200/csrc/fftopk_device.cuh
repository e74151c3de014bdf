// Device-side building blocks of the sm_100a top-2048 selector: warp/block scans that pick a
// threshold bin, the histogram update, and the single-CTA "finish" that resolves a small
// candidate list held in shared memory.
#pragma once
#include <type_traits>
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/fftopk.h"
#include "fftopk_decide.h"
#include "fftopk_key.h"
#include "fftopk_trace.cuh"

namespace fftopk {

namespace cg = cooperative_groups;

constexpr int kK = 2048;               // reference: TopK (topk_indexer_radix.cu:69)
constexpr int kMaxK = 4096;            // largest k of the general entry point (fftopk_select_topk)
constexpr int kMaxBins = 4096;         // widest digit of the distributed rounds: 12 bits
constexpr int kSup = 64;               // super-bins per histogram (each sums kMaxBins/64 bins)
constexpr int kMaxCluster = 16;        // CTAs per row (non-portable cluster size on B200)
#ifndef FFTOPK_KSMALL
#define FFTOPK_KSMALL 256
#endif
constexpr int kSmall = FFTOPK_KSMALL;            // undecided candidates that are ranked directly instead of another radix round
constexpr unsigned kFull = 0xffffffffu;
static_assert(kSampleBins <= kMaxBins, "a sample histogram fits the bins of a distributed round");

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }

// Checked build (-DFFTOPK_CHECKED): every index that the selection logic guarantees to be in
// range - an output slot below k, a candidate slot the decision step has made room for, a staged
// row index below the row length, the winner count of a finish - is tested before use. A failing
// test skips the access, raises FFTOPK_ST_CHECK in the status word and, if it is the first one,
// leaves (site, index, limit, block) in a device-side record that fftopk_checked_read() returns.
// Capacity limits that the algorithm handles by design (a full candidate list makes the row fall
// back to full histograms) are not violations. The production build compiles the tests away.
#ifdef FFTOPK_CHECKED
static __device__ unsigned int g_check_rec[4];
static __device__ __noinline__ void check_fail(int site, uint32_t idx, uint32_t limit, uint32_t* status) {
  if (atomicCAS(&g_check_rec[0], 0u, (unsigned)site) == 0u) {
    g_check_rec[1] = idx;
    g_check_rec[2] = limit;
    g_check_rec[3] = blockIdx.x;
  }
  if (status) atomicOr(status, (uint32_t)FFTOPK_ST_CHECK);
}
// ... and it counts the rows by the way they took (see kRoute*); fftopk_checked_routes() returns the counts.
static __device__ unsigned int g_routes[3];
#define FFTOPK_ROUTE(route) \
  do {                      \
    if (threadIdx.x == 0) atomicAdd(&g_routes[route], 1u); \
  } while (0)
#define FFTOPK_CHECK(site, idx, limit, status) \
  (((uint32_t)(idx) < (uint32_t)(limit)) ? true : (::fftopk::check_fail((site), (uint32_t)(idx), (uint32_t)(limit), (status)), false))
#else
#define FFTOPK_CHECK(site, idx, limit, status) true
#define FFTOPK_ROUTE(route)
#endif
// finished from the candidates of one filter pass; of these, with candidates beyond their CTAs' regions of
// the gather buffer; selected by full histograms
constexpr int kRouteHeld = 0, kRouteBeyond = 1, kRouteHistograms = 2;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory atomics with the state space spelled out. Pointers into the dynamic shared
// memory block travel through structs and function arguments here, where the compiler no longer
// knows their address space and would emit generic atomics (an order of magnitude slower on the
// shared window).
__device__ __forceinline__ void red_shared_add(uint32_t* p, uint32_t v) {
  asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t atom_shared_add(uint32_t* p, uint32_t v) {
  uint32_t old;
  asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(smem_u32(p)), "r"(v) : "memory");
  return old;
}

// The same for plain accesses, and with the address as the 32-bit shared-memory address it is: a
// pointer whose address space the compiler has lost costs 64-bit address arithmetic and a generic
// load or store. In passes that every warp of an SM makes at once (8 issue cycles per instruction with
// 32 warps) that is most of the time.
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint64_t lds64(uint32_t a) {
  uint64_t v;
  asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint2 lds64x2(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void sts64(uint32_t a, uint32_t lo, uint32_t hi) {
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"(lo), "r"(hi) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void sts_zero16(uint32_t a) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(a), "r"(0) : "memory");
}
// A peer CTA's shared memory: the address of what lies at `a` here in the CTA of rank `r`, and stores to it.
__device__ __forceinline__ uint32_t peer_smem(uint32_t a, int r) {
  uint32_t v;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(v) : "r"(a), "r"(r));
  return v;
}
__device__ __forceinline__ void st_peer32(uint32_t a, uint32_t v) { asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void st_peer64(uint32_t a, uint64_t v) { asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory"); }
__device__ __forceinline__ void red_shared_inc(uint32_t a) { asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(a) : "memory"); }

// Predicated steps of the passes over candidates, spelled out. Left to the compiler, `if (c > t) ... else
// if ...` over four candidates became a tree of branches whose lanes came together only behind the
// last of them: up to 81 paths, one after the other (2,300 cycles for counting four candidates per
// lane; 300 like this).
__device__ __forceinline__ void count_if_above(uint32_t& n, uint32_t k, uint32_t thr) {
  asm("{\n\t.reg .pred p;\n\tsetp.gt.u32 p, %1, %2;\n\t@p add.u32 %0, %0, 1;\n\t}" : "+r"(n) : "r"(k), "r"(thr));
}
__device__ __forceinline__ void count_if_above(uint32_t& n, uint64_t c, uint64_t thr) {
  asm("{\n\t.reg .pred p;\n\tsetp.gt.u64 p, %1, %2;\n\t@p add.u32 %0, %0, 1;\n\t}" : "+r"(n) : "l"(c), "l"(thr));
}
__device__ __forceinline__ void red_shared_inc_if(uint32_t a, uint32_t nonzero, uint32_t off, uint32_t span) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\tsetp.le.and.u32 p, %2, %3, p;\n\t@p red.shared.add.u32 [%0], 1;\n\t}" ::"r"(a),
      "r"(nonzero), "r"(off), "r"(span)
      : "memory");
}
__device__ __forceinline__ void st_global_if(bool on, void* a, uint32_t v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.global.u32 [%0], %1;\n\t}" ::"l"(a), "r"(v), "r"((uint32_t)on)
               : "memory");
}
// (on: a slot from the counter at `counter`, and v into slot of the array at `a`, if the array has it)
__device__ __forceinline__ uint32_t append64_if(bool on, uint32_t counter, uint32_t a, uint32_t cap, uint64_t v) {
  uint32_t slot;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .u32 at;\n\tsetp.ne.u32 p, %5, 0;\n\tmov.u32 %0, 0;\n\t@p atom.shared.add.u32 %0, [%1], 1;\n\t"
      "setp.lt.and.u32 q, %0, %3, p;\n\tmad.lo.u32 at, %0, 8, %2;\n\t@q st.shared.u64 [at], %4;\n\t}"
      : "=&r"(slot)
      : "r"(counter), "r"(a), "r"(cap), "l"(v), "r"((uint32_t)on)
      : "memory");
  return slot;
}
__device__ __forceinline__ void st_global_if_above(uint32_t k, uint32_t thr, void* a, uint32_t v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.gt.u32 p, %2, %3;\n\t@p st.global.u32 [%0], %1;\n\t}" ::"l"(a), "r"(v), "r"(k), "r"(thr)
               : "memory");
}
// (i < n: the word at `a`, else 0)
__device__ __forceinline__ uint32_t lds32_below(int i, int n, uint32_t a) {
  uint32_t v;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %2, %3;\n\tmov.u32 %0, 0;\n\t@p ld.shared.u32 %0, [%1];\n\t}"
               : "=&r"(v)
               : "r"(a), "r"(i), "r"(n)
               : "memory");
  return v;
}
__device__ __forceinline__ uint64_t lds64_below(int i, int n, uint32_t a) {
  uint64_t v;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %2, %3;\n\tmov.u64 %0, 0;\n\t@p ld.shared.u64 %0, [%1];\n\t}"
               : "=&l"(v)
               : "r"(a), "r"(i), "r"(n)
               : "memory");
  return v;
}

// What a kernel may do with its inputs before the kernel in front of it on the stream has completed: ask for them to be
// brought into L2, which is coherent, so that whatever that kernel still writes is what is read later. `hint_s32`: a
// value that may be about to change, good for nothing but the size of such a request.
__device__ __forceinline__ int32_t hint_s32(const int32_t* p) {
  int32_t v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// part i of n of the `bytes` bytes at p
__device__ __forceinline__ void prefetch_part_l2(const void* p, int64_t bytes, int i, int n) {
  const int64_t part = bytes / n;
  const uintptr_t from = (reinterpret_cast<uintptr_t>(p) + (uintptr_t)(part * i) + 15u) & ~(uintptr_t)15u;
  const uint32_t size = (uint32_t)(part > 16 ? part - 15 : 0) & ~15u;
  if (size != 0u) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(from), "r"(size) : "memory");
}

// Histogram update: a plain shared-memory reduction (no result). Measured on B200 (64K updates
// per CTA, 1024 threads): 6 to 12 updates per clock per SM whatever the bin distribution,
// all-equal bins included - the hardware combines same-address updates, and ballot / match.any
// pre-aggregation in software was 2 to 10 times slower.
__device__ __forceinline__ void hist_add(uint32_t* hist, uint32_t bin, bool valid) {
  if (valid) red_shared_add(&hist[bin], 1u);
}

// Slot allocation from a shared-memory counter (the atomic's RESULT is needed, so equal
// addresses do serialise): the lanes of a warp that are allocating together take consecutive
// slots with one atomic. May be called from divergent code.
__device__ __forceinline__ uint32_t warp_alloc(uint32_t* counter) {
  const unsigned m = __activemask();
  const int leader = __ffs(m) - 1;
  uint32_t base = 0;
  if (lane_id() == leader) base = atom_shared_add(counter, (uint32_t)__popc(m));
  base = __shfl_sync(m, base, leader);
  return base + (uint32_t)__popc(m & ((1u << lane_id()) - 1u));
}

// ---------------------------------------------------------------------------------------------
// Warp-level threshold pick over 64 counts in descending bin order. Lane l holds the counts of
// bins 2l (lo) and 2l+1 (hi). Finds the bin t with
//     above(t) < need <= above(t) + count[t],   above(t) = sum of count[j], j > t.
// This is the reference's "S[t] > k >= S[t+1]" rule (topk_indexer_radix.cu:555-566) computed with
// a shuffle suffix scan instead of eight block-wide doubling steps. Returns false if the counts
// sum to less than `need`.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ bool warp_pick64(uint32_t lo, uint32_t hi, uint32_t need, int& t, uint32_t& above,
                                            uint32_t& cnt) {
  const int lane = lane_id();
  const uint32_t s = lo + hi;
  uint32_t incl = s;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t v = __shfl_down_sync(kFull, incl, off);
    if (lane + off < 32) incl += v;
  }
  const uint32_t excl = incl - s;  // counts in lanes above this one
  const bool hit_hi = (excl < need) && (need <= excl + hi);
  const bool hit_lo = (excl + hi < need) && (need <= excl + hi + lo);
  const unsigned m = __ballot_sync(kFull, hit_hi || hit_lo);
  if (m == 0) return false;
  const int src = __ffs(m) - 1;
  t = __shfl_sync(kFull, hit_hi ? 2 * lane + 1 : 2 * lane, src);
  above = __shfl_sync(kFull, hit_hi ? excl : excl + hi, src);
  cnt = __shfl_sync(kFull, hit_hi ? hi : lo, src);
  return true;
}

__device__ __forceinline__ uint32_t warp_sum(uint32_t v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(kFull, v, off);
  return v;
}

// ---------------------------------------------------------------------------------------------
// Shared-memory control block (one per CTA; rank 0's counters are the cluster-wide ones).
// ---------------------------------------------------------------------------------------------
// Where a finish writes: the row's output, its status word, page table (NULL: none) and the offset of its indices
struct FinishTo {
  int32_t* out_idx;
  uint32_t* out_key;
  uint32_t* status;
  const int32_t* page;
  uint32_t out_base, out_slots;
  int32_t idx_offset;
  uint32_t need;  // candidates that win
};
struct Ctrl {
  uint4 fin;  // (finish) the threshold bin: smallest and largest value of the digit's field, elements above, in it
  // cluster-wide allocation counters, meaningful in rank 0 only (targets of remote atomics)
  uint32_t win_count;
  uint32_t cand_count;
  uint32_t extra_count;  // rank 0 only: candidates beyond their CTAs' regions (remote atomics)
  // published to the peers before a cluster barrier
  uint32_t pub_flag;
  // per-pass local slot counters
  uint32_t wslot;
  uint32_t cslot;
  uint32_t fslot;
  uint32_t small_n;  // (finish) undecided candidates set aside so far
  uint32_t lcount;  // entries pushed to this CTA's spill area (may exceed its capacity)
  // what the sample search leaves: the guess and the bound for the finish (keys), what to do about them
  uint32_t guess;
  uint32_t focus;
  uint32_t guess_flags;
  uint32_t need_hi;
  // result of the most recent threshold search
  int32_t t;
  uint32_t above;
  uint32_t cnt;
  int32_t sup_sel;
  uint32_t sup_above;
  uint32_t need;
  int32_t mode;
  uint32_t base_w;
  uint32_t base_c;
  uint32_t tie_prefix;
  uint32_t local_c;
  uint32_t run_total;
  // cluster-wide super-bin totals and fine-bin totals of the threshold super-bin, double-buffered
  // by search number (each search clears the buffers of the next one)
  uint32_t tot[2][kSup];
  uint32_t tot2[2][kSup];
  uint32_t totb[kSup];  // first sample round: super-bin totals of the second (finer) histogram
  uint32_t dual_b;      // ... whether the finer histogram was usable, and for which top nibble
  uint32_t dual_g;
  uint32_t wtot[32];
  uint32_t wmax[32];
  uint32_t cnt_of[kMaxCluster];  // candidates of every CTA of the cluster (each writes its own entry everywhere)
  // merge of candidate lists: this CTA's record about its shard, read by the cluster's other CTAs
  uint32_t thr_key;      // warm start: smallest key among the winners of the finish
  uint32_t merge_count;  // valid candidates
  uint32_t merge_fail;   // the bounded wait for the shard's flag ran out
  const int32_t* row_page;  // the row's page table (or NULL) and the offset of its indices
  int32_t row_idx_offset;
  uint64_t small[kSmall];
  FinishTo to;  // (finish: rows with many copies of the threshold)
#ifdef FFTOPK_CHECKED
  uint32_t* status_ptr;  // the call's status word, for checks in code that has no other way to it
#endif
};
#ifdef FFTOPK_CHECKED
#define ctrl_status(c) ((c)->status_ptr)
#endif

// What a cluster does after a threshold search (see decide_and_allocate).
enum Mode : int { kModeNext = 0, kModeGather = 1, kModeTakeAll = 2, kModeTies = 3, kModeAbort = 4, kModeFallback = 5 };

// Sum each group of nb/64 consecutive bins into sup[0..63].
template <int NT>
__device__ __forceinline__ void compute_sup(const uint32_t* hist, uint32_t* sup, int nb) {
  const int tid = threadIdx.x;
  if (nb == kMaxBins) {
    constexpr int PER = kMaxBins / NT;            // bins per thread: 4 (1024 thr), 8 (512)
    constexpr int TPS = (kMaxBins / kSup) / PER;  // threads per super-bin: 16, 8
    uint32_t s = 0;
    const uint4* h4 = reinterpret_cast<const uint4*>(hist) + tid * (PER / 4);
#pragma unroll
    for (int j = 0; j < PER / 4; ++j) {
      const uint4 v = h4[j];
      s += v.x + v.y + v.z + v.w;
    }
#pragma unroll
    for (int off = TPS / 2; off > 0; off >>= 1) s += __shfl_xor_sync(kFull, s, off);
    if ((tid % TPS) == 0) sup[tid / TPS] = s;
  } else {  // 256 bins
    if (tid < kSup) {
      const uint4 v = reinterpret_cast<const uint4*>(hist)[tid];
      sup[tid] = v.x + v.y + v.z + v.w;
    }
  }
}

// Cluster barrier; for a cluster of one CTA a block barrier does the same job for less.
__device__ __forceinline__ void cluster_sync(cg::cluster_group& cluster, int C) {
  if (C == 1) {
    __syncthreads();
  } else {
    cluster.sync();
  }
}

// What warp 0 knows after a cluster-wide threshold search.
struct Picked {
  bool ok;            // false: the histogram holds fewer than `need` elements
  int t;              // threshold bin
  uint32_t need2;     // elements still to take from bin t
  uint32_t cnt;       // cluster-wide population of bin t
  uint32_t local_w;   // this CTA's elements in bins above t
  uint32_t local_c;   // this CTA's elements in bin t
  uint32_t total;     // cluster-wide number of histogrammed elements
  int tf;             // t's position inside its super-bin (index into xch rows)
  bool fine;          // the search ran on the second, finer histogram (see cluster_pick)
  uint32_t group;     // ... whose bins all lie under this value of the key's top four bits
};

// Cluster-wide threshold search on per-CTA histograms `h` (nb bins) with super-bin sums `s`,
// both complete and published by a cluster barrier before the call. Every CTA reads its peers'
// 64 super-bin sums, then the fine bins of the threshold super-bin, over distributed shared
// memory; warp 0 picks with shuffle scans. need_of(total) maps the cluster-wide element count
// to the rank searched for. `post(picked)` runs in warp 0 (all lanes) before the closing
// barrier; the results it wants every thread to see go through `ctrl`.
// Optionally a second histogram `hb` / `sb` of the same elements on key bits [27:16] (4096 bins, 16
// times finer) comes along: it orders the elements only if they all share the key's top four
// bits, i.e. if one group of four super-bins of `h` holds everything; then the search runs on it
// (Picked::fine, ::group) and the threshold bin is a 16-bit key prefix. ctrl->totb must be zero.
// Replaces parallel_reduce_histogram + radix_prefix_sum of the reference
// (topk_indexer_radix.cu:80-107, 232-279), which reduce to rank 0 and broadcast back with three
// cluster barriers and eight block barriers per round.
template <int NT, class NeedFn, class Post>
__device__ __forceinline__ void cluster_pick(cg::cluster_group& cluster, int C, const uint32_t* h, const uint32_t* s,
                                             uint32_t* xch, Ctrl* ctrl, int& pick_no, int nb, NeedFn&& need_of,
                                             Post&& post, const uint32_t* hb = nullptr, const uint32_t* sb = nullptr) {
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int fine = nb / kSup;
  uint32_t* tot = ctrl->tot[pick_no & 1];
  uint32_t* tot2 = ctrl->tot2[pick_no & 1];
  const bool dual = hb != nullptr;
  // (A) cluster-wide super-bin totals: one remote word per thread, summed with shared-memory
  // reductions instead of a serial loop over the ranks. (Pushing the sums into the peers before
  // the cluster barrier instead - remote reductions behind a split arrive / wait barrier - was
  // measured and was not faster: the release of the extra arrive costs what the remote loads cost.)
  for (int i = tid; i < C * kSup; i += NT) {
    const uint32_t* rs = C == 1 ? s : cluster.map_shared_rank(s, i / kSup);
    red_shared_add(&tot[i % kSup], rs[i % kSup]);
    if (dual) {
      const uint32_t* rb = C == 1 ? sb : cluster.map_shared_rank(sb, i / kSup);
      red_shared_add(&ctrl->totb[i % kSup], rb[i % kSup]);
    }
  }
  __syncthreads();
  FFTOPK_MARK(40);
  // Warp 0 picks and publishes through the control block. (Letting every warp pick for itself
  // saves the two broadcast barriers but was measured slower: 32 warps running the same shuffle
  // scans get in each other's way.)
  if (warp == 0) {
    uint32_t lo = tot[2 * lane], hi = tot[2 * lane + 1];
    const uint32_t total = warp_sum(lo + hi);
    const uint32_t need = need_of(total);
    unsigned one = 0u;
    if (dual) {
      // four super-bins = 256 bins of `h` = one value of the top four key bits
      const uint32_t pair = lo + hi;
      const uint32_t grp = pair + __shfl_xor_sync(kFull, pair, 1);
      one = __ballot_sync(kFull, fine_histogram_usable(true, total, grp));
      if (one != 0u) {
        lo = ctrl->totb[2 * lane];
        hi = ctrl->totb[2 * lane + 1];
      }
    }
    uint32_t above = 0, cnt = 0;
    int ts = -1;
    const bool ok = need > 0 && warp_pick64(lo, hi, need, ts, above, cnt);
    if (lane == 0) {
      ctrl->sup_sel = ok ? ts : -1;
      ctrl->sup_above = above;
      ctrl->need = need;
      ctrl->run_total = total;
      ctrl->dual_b = one != 0u ? 1u : 0u;
      ctrl->dual_g = one != 0u ? (uint32_t)((__ffs(one) - 1) >> 1) : 0u;
    }
  }
  __syncthreads();
  FFTOPK_MARK(41);
  const int ssel = ctrl->sup_sel;
  if (dual && ctrl->dual_b != 0u) {  // (uniform) the rest of the search runs on the finer histogram
    h = hb;
    s = sb;
  }
  // (B) fine bins of the threshold super-bin: pulled from every peer, kept per rank in xch (the
  // tie path wants them) and summed into tot2
  if (ssel >= 0) {
    for (int i = tid; i < C * kSup; i += NT) {
      const int q = i / kSup, f = i % kSup;
      uint32_t v = 0;
      if (f < fine) {
        const uint32_t* rh = C == 1 ? h : cluster.map_shared_rank(h, q);
        v = rh[ssel * fine + f];
        red_shared_add(&tot2[f], v);
      }
      xch[i] = v;
    }
  }
  __syncthreads();
  FFTOPK_MARK(42);
  // the buffers of the next search: their last readers passed the barrier above long ago
  if (tid < kSup) {
    ctrl->tot[(pick_no + 1) & 1][tid] = 0u;
    ctrl->tot2[(pick_no + 1) & 1][tid] = 0u;
  }
  ++pick_no;
  if (warp == 0) {
    Picked pk;
    pk.ok = false;
    pk.t = -1;
    pk.need2 = pk.cnt = pk.local_w = pk.local_c = 0;
    pk.total = ctrl->run_total;
    pk.tf = 0;
    pk.fine = dual && ctrl->dual_b != 0u;
    pk.group = ctrl->dual_g;
    if (ssel >= 0) {
      const uint32_t lo = tot2[2 * lane], hi = tot2[2 * lane + 1];
      const uint32_t need = ctrl->need, sup_above = ctrl->sup_above;
      int tf = -1;
      uint32_t above_f = 0, cnt_t = 0;
      if (warp_pick64(lo, hi, need - sup_above, tf, above_f, cnt_t)) {
        pk.ok = true;
        pk.tf = tf;
        pk.t = ssel * fine + tf;
        pk.need2 = need - sup_above - above_f;
        pk.cnt = cnt_t;
        uint32_t lw = 0;
        lw += (2 * lane > ssel) ? s[2 * lane] : 0u;
        lw += (2 * lane + 1 > ssel) ? s[2 * lane + 1] : 0u;
        lw += (2 * lane < fine && 2 * lane > tf) ? h[ssel * fine + 2 * lane] : 0u;
        lw += (2 * lane + 1 < fine && 2 * lane + 1 > tf) ? h[ssel * fine + 2 * lane + 1] : 0u;
        pk.local_w = warp_sum(lw);
        pk.local_c = h[pk.t];
      }
    }
    post(pk);  // warp 0 only; what the other warps need goes through the control block
  }
  __syncthreads();
  FFTOPK_MARK(43);
}

// Standard decision after a search with need = what is still missing of k: either the threshold
// bin is taken whole, or its population fits rank 0's buffer and is gathered there, or
// `otherwise` (a mode) applies. Output and candidate slots are allocated with one remote atomic
// each on rank 0's counters.
// `cx` is anything with the members ctrl, ctrl0 (rank 0's control block) and cand_cap.
template <class Ctx>
__device__ __forceinline__ void decide_and_allocate(const Ctx& cx, const Picked& pk, int otherwise) {
  int md = kModeAbort;
  uint32_t base_w = 0, base_c = 0, lw = pk.local_w;
  if (pk.ok) {
    if (pk.cnt == pk.need2) {
      md = kModeTakeAll;
      lw += pk.local_c;
    } else if (pk.cnt <= (uint32_t)cx.cand_cap) {
      md = kModeGather;
    } else {
      md = otherwise;
    }
    if (lane_id() == 0) {
      base_w = atomicAdd(&cx.ctrl0->win_count, lw);
      if (md == kModeGather) base_c = atomicAdd(&cx.ctrl0->cand_count, pk.local_c);
    }
  }
  if (lane_id() == 0) {
    Ctrl* ctrl = cx.ctrl;
    ctrl->mode = md;
    ctrl->t = pk.t;
    ctrl->above = pk.need2;
    ctrl->cnt = pk.cnt;
    ctrl->base_w = base_w;
    ctrl->base_c = base_c;
    ctrl->local_c = pk.local_c;
    ctrl->wslot = 0u;
    ctrl->cslot = 0u;
  }
}

// ---------------------------------------------------------------------------------------------
// Candidate sources of the finish. A source tells a thread which candidates are its share:
// for_each(f) calls f with an array of kWalk composites at a time - loads in flight together, same trip count in
// all lanes of a warp - and 0 where there is none. Which candidates a thread sees, and in which order,
// is the same in every call.
// ---------------------------------------------------------------------------------------------

// A dense array in shared memory walked by a group of warps (`first`: this lane's first index, `step`: lanes in
// the group; first - lane is the same in all lanes of a warp)
constexpr int kWalk = 4;
template <class F>
__device__ __forceinline__ void walk(uint32_t a /* shared address */, int n, int first, int step, F&& f) {
  const int lane = lane_id();
  for (int i = first; i - lane < n; i += kWalk * step) {
    const uint32_t at = a + (uint32_t)i * 8u;
    uint64_t c[kWalk];
#pragma unroll
    for (int u = 0; u < kWalk; ++u) c[u] = lds64_below(i + u * step, n, at + (uint32_t)(u * step) * 8u);
    f(c);
  }
}

// ... and over their keys alone
template <class F>
__device__ __forceinline__ void walk_keys(uint32_t a, int n, int first, int step, F&& f) {
  const int lane = lane_id();
  for (int i = first; i - lane < n; i += kWalk * step) {
    const uint32_t at = a + (uint32_t)i * 8u + 4u;
    uint32_t k[kWalk];
#pragma unroll
    for (int u = 0; u < kWalk; ++u) k[u] = lds32_below(i + u * step, n, at + (uint32_t)(u * step) * 8u);
    f(k);
  }
}

// One dense array cand[0..n); slots equal to 0 are empty.
template <int NT>
struct DenseCands {
  uint32_t cand;  // shared address
  int n;
  __device__ __forceinline__ DenseCands(const uint64_t* c, int n_) : cand(smem_u32(c)), n(n_) {}
  template <class F>
  __device__ __forceinline__ void for_each(F&& f) const {
    walk(cand, n, (int)threadIdx.x, NT, f);
  }
  template <class F>
  __device__ __forceinline__ void for_each_key(F&& f) const {
    walk_keys(cand, n, (int)threadIdx.x, NT, f);
  }
};

// What the filter of a lone CTA leaves behind: per warp up to 32 * R candidates, their keys in registers (candidate j
// of the warp in key[j / 32] of lane j % 32; 0 where there is none) and their indices in a dense segment in shared
// memory (`wn` of them, the same in all lanes).
template <int NT, int R>
struct RegSegCands {
  uint32_t key[R];
  uint32_t seg;  // shared address of this warp's indices
  int wn;
};

// What a cluster leaves in its first CTA: one region of `region` slots per CTA, filled densely with
// count_of[r] candidates, and `extra` candidates that did not fit in front of those behind the last
// region. A region belongs to 2^lper warps (or, lper = 0, a warp to several regions).
template <int NT>
struct RegionCands {
  uint32_t cand;      // shared addresses
  uint32_t count_of;
  int region, C, extra;
  template <class W>
  __device__ __forceinline__ void each_part(W&& w) const {
    constexpr int kLogNW = NT == 1024 ? 5 : (NT == 512 ? 4 : 3);
    const int warp = threadIdx.x >> 5;
    const int lper = max(kLogNW - (31 - __clz(C)), 0);  // (NW and C are powers of two: no division)
    for (int r = warp >> lper; r < C; r += (NT / 32) >> lper)
      w(cand + (uint32_t)(r * region) * 8u, min((int)lds32(count_of + r * 4), region), (warp & ((1 << lper) - 1)) * 32 + lane_id(),
        32 << lper);
    if (extra > 0) w(cand + (uint32_t)(C * region) * 8u, extra, (int)threadIdx.x, NT);
  }
  template <class F>
  __device__ __forceinline__ void for_each(F&& f) const {
    each_part([&](uint32_t a, int n, int first, int step) { walk(a, n, first, step, f); });
  }
  template <class F>
  __device__ __forceinline__ void for_each_key(F&& f) const {
    each_part([&](uint32_t a, int n, int first, int step) { walk_keys(a, n, first, step, f); });
  }
};

// Block-wide threshold pick over kFinishBins counts (descending bin order): one thread calls
// found(bin, above, count) for the bin that holds rank `need`; nobody does if the counts sum to less. Ends
// with a barrier, which publishes what it leaves in shared memory; before() runs in thread 0 before that.
template <int NT, class Before, class Found>
__device__ __forceinline__ void block_pick(uint32_t hist /* shared address */, uint32_t need, uint32_t wtot /* shared address */,
                                           Before&& before, Found&& found) {
  constexpr int PER = (kFinishBins + NT - 1) / NT;
  constexpr int NW = NT / 32;
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  uint32_t v[PER];
  uint32_t s = 0;
  if constexpr (PER * NT == kFinishBins && PER % 2 == 0) {
#pragma unroll
    for (int j = 0; j < PER; j += 2) {
      const uint2 q = lds64x2(hist + (uint32_t)(tid * PER + j) * 4u);
      v[j] = q.x;
      v[j + 1] = q.y;
      s += q.x + q.y;
    }
  } else {
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int b = tid * PER + j;
      v[j] = (b < kFinishBins) ? lds32(hist + b * 4) : 0u;
      s += v[j];
    }
  }
  uint32_t incl = s;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t x = __shfl_down_sync(kFull, incl, off);
    if (lane + off < 32) incl += x;
  }
  if (lane == 0) sts32(wtot + warp * 4, incl);
  if (tid == 0) before();
  __syncthreads();
  const uint32_t hw = (lane > warp && lane < NW) ? lds32(wtot + lane * 4) : 0u;
  uint32_t run = __reduce_add_sync(kFull, hw) + incl - s;
  if (run < need && need <= run + s) {  // (one thread)
#pragma unroll
    for (int j = PER - 1; j >= 0; --j) {
      if (run < need && need <= run + v[j]) found((uint32_t)(tid * PER + j), run, v[j]);
      run += v[j];
    }
  }
  __syncthreads();
}

// Block-wide search over a sample histogram of kSampleBins counts (descending bin order):
// found(bin, above, count) is called by one thread for the bin of rank `need`, found_hi(bin) by one
// for the bin of rank `need_hi` (neither if the counts do not reach that rank, or the rank is 0).
// Ends with a barrier, which publishes what they leave in shared memory. Written for few
// instructions: with 32 warps on an SM each of them costs a block eight issue cycles.
template <int NT, class Found, class FoundHi>
__device__ __forceinline__ void block_pick_sample(uint32_t hist /* shared address */, uint32_t need, uint32_t need_hi,
                                                  uint32_t wtot /* shared address */,
                                                  Found&& found, FoundHi&& found_hi) {
  constexpr int PER = kSampleBins / NT;
  constexpr int NW = NT / 32;
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  uint32_t v[PER];
  uint32_t s = 0;
#pragma unroll
  for (int j = 0; j < PER / 4; ++j) {
    const uint4 q = lds128(hist + (uint32_t)(tid * PER + 4 * j) * 4u);
    v[4 * j] = q.x;
    v[4 * j + 1] = q.y;
    v[4 * j + 2] = q.z;
    v[4 * j + 3] = q.w;
    s += (q.x + q.y) + (q.z + q.w);
  }
  uint32_t incl = s;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t x = __shfl_down_sync(kFull, incl, off);
    if (lane + off < 32) incl += x;
  }
  if (lane == 0) sts32(wtot + warp * 4, incl);
  __syncthreads();
  const uint32_t w = (lane < NW && lane > warp) ? lds32(wtot + lane * 4) : 0u;
  uint32_t run = __reduce_add_sync(kFull, w) + incl - s;
  // (a thread whose bins lie wholly above or wholly below both ranks has nothing to look for)
  if ((run < need && need <= run + s) || (run < need_hi && need_hi <= run + s)) {
#pragma unroll
    for (int j = PER - 1; j >= 0; --j) {
      if (run < need && need <= run + v[j]) found((uint32_t)(tid * PER + j), run, v[j]);
      if (run < need_hi && need_hi <= run + v[j]) found_hi((uint32_t)(tid * PER + j));
      run += v[j];
    }
  }
  __syncthreads();
}

// The bin of rank `need` in the histogram of a finish round: (bin, or kNoBin if there is none; elements above it; elements in it).
constexpr uint32_t kNoBin = 0xffffffffu;
template <int NT>
__device__ __forceinline__ uint4 finish_pick(uint32_t hist /* shared address */, uint32_t need, Ctrl* ctrl) {
  const uint32_t fin = smem_u32(&ctrl->fin);
  block_pick<NT>(hist, need, smem_u32(ctrl->wtot), [&] { sts32(fin, kNoBin); },
                 [&](uint32_t bin, uint32_t above, uint32_t n) { sts128(fin, bin, above, n, 0u); });
  return lds128(fin);
}

// The output pass of a finish: candidates of which field() is above `wthr` win, those above `uthr` are undecided
// (up to kSmall, of which the `need2` best win; with all_bin there are none).
// Every warp counts its winners and gets its output slots by a sum over the warps in front of it; then it writes
// them, 32 candidates at a time, slots by ballot. (A slot-allocating atomic per warp serialised on the one
// counter - 30 cycles per warp -, and slots by thread, from a scan over the lanes, scattered every store over 32
// lines.) A threshold bin that is not taken whole holds a handful of candidates: those take an atomic.
struct FinishOut : FinishTo {
  Ctrl* ctrl;
};
// Rank by vote the `cnt` candidates set aside: warp i takes candidate i, the lanes compare it with the candidates j (32
// per step); the number of larger ones is candidate i's rank, and the best need2 go behind the
// `certain` winners. Up to 256 undecided candidates are cheaper to rank like this (at most 64
// votes per warp) than to split by another round - rows of low-precision logits have
// hundreds of exact duplicates at the threshold. (A bitonic compare-exchange network over 32
// values is a chain of 60 dependent shuffles; this is one ballot per 32 comparisons.)
template <int NT, bool kTrackMin>
__device__ __forceinline__ void rank_undecided(const FinishOut& o, uint32_t certain, uint32_t need2, uint32_t cnt) {
  const int lane = lane_id();
  __syncthreads();
  const int nchunk = ((int)cnt + 31) >> 5;
  for (int i = (int)(threadIdx.x >> 5); i < (int)cnt; i += NT / 32) {
    const uint64_t me = o.ctrl->small[i];
    uint32_t rank = 0;
    for (int ch = 0; ch < nchunk; ++ch) {
      const int j = ch * 32 + lane;
      const uint64_t other = (j < (int)cnt) ? o.ctrl->small[j] : 0ull;
      rank += (uint32_t)__popc(__ballot_sync(kFull, other > me));
    }
    if (lane == 0 && rank < need2) {
      const uint32_t pos = o.out_base + certain + rank;
      if (FFTOPK_CHECK(5, pos, o.out_slots, o.status) && pos < o.out_slots) {
        const int32_t idx = (int32_t)(~(uint32_t)me);
        o.out_idx[pos] = o.page ? __ldg(o.page + idx) : idx + o.idx_offset;
        if (o.out_key) o.out_key[pos] = (uint32_t)(me >> 32);
      }
      if constexpr (kTrackMin) atomicMin(&o.ctrl->thr_key, (uint32_t)(me >> 32));
    }
  }
}

template <int NT, bool kTrackMin, class Src, class V, class Field>
__device__ __forceinline__ void finish_output(const Src src, const FinishOut o, uint32_t need2, uint32_t cnt, bool all_bin, V wthr, V uthr,
                                              Field&& field) {
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  Ctrl* const ctrl = o.ctrl;
  const uint32_t small_s = smem_u32(ctrl->small), small_n = smem_u32(&ctrl->small_n);
  const unsigned lt = (1u << lane) - 1u;
  uint32_t n = 0u;
  if constexpr (sizeof(V) == 4) {
    src.for_each_key([&](const uint32_t (&k)[kWalk]) {
#pragma unroll
      for (int u = 0; u < kWalk; ++u) count_if_above(n, k[u], wthr);
    });
  } else {
    src.for_each([&](const uint64_t (&c)[kWalk]) {
#pragma unroll
      for (int u = 0; u < kWalk; ++u) count_if_above(n, field(c[u]), wthr);
    });
  }
  n = __reduce_add_sync(kFull, n);
  const uint32_t wsum = smem_u32(ctrl->wmax);
  if (lane == 0) sts32(wsum + warp * 4, n);
  __syncthreads();
  uint32_t wpos = o.out_base + __reduce_add_sync(kFull, lane < warp ? lds32(wsum + lane * 4) : 0u);
#ifdef FFTOPK_CHECKED
  const uint32_t set_w = __reduce_add_sync(kFull, lane < NT / 32 ? lds32(wsum + lane * 4) : 0u);  // winners found
#endif
  uint32_t win_min = 0xffffffffu;  // (kTrackMin) smallest key among the certain winners, if they are all there are
  src.for_each([&](const uint64_t (&c)[kWalk]) {
    int32_t v[kWalk];
#pragma unroll
    for (int u = 0; u < kWalk; ++u) v[u] = (int32_t)(~(uint32_t)c[u]) + o.idx_offset;
    if (o.page) {  // (the table reads in flight together)
#pragma unroll
      for (int u = 0; u < kWalk; ++u)
        if (field(c[u]) > wthr) v[u] = __ldg(o.page + (int32_t)(~(uint32_t)c[u]));
    }
    bool undecided = false;
#pragma unroll
    for (int u = 0; u < kWalk; ++u) {
      const bool w = field(c[u]) > wthr;
      const unsigned bw = __ballot_sync(kFull, w);
      const uint32_t pos = wpos + (uint32_t)__popc(bw & lt);
      const bool put = w && FFTOPK_CHECK(3, pos, o.out_slots, o.status) && pos < o.out_slots;
      st_global_if(put, o.out_idx + pos, (uint32_t)v[u]);
      if (o.out_key) st_global_if(put, o.out_key + pos, (uint32_t)(c[u] >> 32));
      wpos += (uint32_t)__popc(bw);
      undecided = undecided || (!w && field(c[u]) > uthr);
      if constexpr (kTrackMin) {
        if (all_bin) win_min = min(win_min, w ? (uint32_t)(c[u] >> 32) : 0xffffffffu);
      }
    }
    if (__any_sync(kFull, undecided)) {
#pragma unroll
      for (int u = 0; u < kWalk; ++u) {
        const uint32_t slot = append64_if(field(c[u]) > uthr && !(field(c[u]) > wthr), small_n, small_s, kSmall, c[u]);
        (void)FFTOPK_CHECK(4, slot, kSmall, o.status);
      }
    }
  });
  FFTOPK_MARK(33);
  if constexpr (kTrackMin) {
    if (all_bin) {  // (else the smallest winner is one of those that are ranked)
      win_min = __reduce_min_sync(kFull, win_min);
      if (lane == 0 && win_min != 0xffffffffu) atomicMin(&ctrl->thr_key, win_min);
    }
  }
#ifdef FFTOPK_CHECKED
  {
    // every certain winner took exactly one slot, every undecided candidate was set aside
    __syncthreads();
    const uint32_t want_w = all_bin ? o.need : o.need - need2;
    if (tid == 0) {
      if (set_w != want_w) check_fail(10, set_w, want_w, o.status);
      if (!all_bin && ctrl->small_n != cnt) check_fail(11, ctrl->small_n, cnt, o.status);
    }
  }
#endif
  if (!all_bin) rank_undecided<NT, kTrackMin>(o, o.need - need2, need2, cnt);
}

// More copies of one key than can be ranked, the threshold among them: `need` candidates are still to be taken from
// those with key `key` and - `more` of them - larger ones. Rounds over the inverted indices under the key, then the
// output. Returns false if the threshold is a key above `key` after all.
template <int NT, bool kTrackMin, class Src>
__device__ __forceinline__ bool finish_copies(const Src src, const FinishOut& o, uint32_t need, uint32_t key, bool more, int idx_bits,
                                              uint32_t* hist) {
  const int tid = threadIdx.x;
  const uint32_t hist_s = smem_u32(hist);
  uint32_t lo = inverted_index_floor(idx_bits), cap = 0xffffffffu;
  for (int round = 0; round < 8; ++round) {
    const KeyDigit dg = make_key_digit(lo, cap);
    __syncthreads();  // every thread is through with the histogram and the result of the round before
    for (int b = tid; b < kFinishBins; b += NT) hist[b] = 0u;
    __syncthreads();
    const uint32_t span = cap - lo;
    src.for_each([&](const uint64_t (&c)[kWalk]) {
#pragma unroll
      for (int u = 0; u < kWalk; ++u) {
        const uint32_t k = (uint32_t)(c[u] >> 32), v = (uint32_t)c[u];
        if (k == key && v - lo <= span) red_shared_inc(hist_s + dg.of(v) * 4u);
        if (more && k > key) red_shared_inc(hist_s + (uint32_t)(kFinishBins - 1) * 4u);
      }
    });
    __syncthreads();
    const uint4 f = finish_pick<NT>(hist_s, need, o.ctrl);
    if (f.x == kNoBin) break;
    const uint32_t cnt = f.z, need2 = need - f.y;
    if (more && f.x == (uint32_t)kFinishBins - 1u) return false;
    const uint32_t t_lo = dg.bin_low(f.x), t_hi = dg.bin_high(f.x, cap);
    if (cnt == need2 || cnt <= (uint32_t)kSmall) {
      const uint64_t k = (uint64_t)key << 32, below = (k | t_lo) - 1ull;
      finish_output<NT, kTrackMin>(src, o, need2, cnt, cnt == need2, cnt == need2 ? below : k | t_hi, below,
                                   [](uint64_t c) { return c; });
      return true;
    }
    more = false;
    lo = t_lo;
    cap = t_hi;
    need = need2;
  }
  if (tid == 0 && o.status) atomicOr(o.status, 2u);
  return true;
}

// What the rounds over the keys (finish_rounds) do when they have come down to one key. Rows with thousands of copies of one value
// do; the others should not carry the registers and instructions for them, so that is a call out of line:
//   kCopiesRest   the last thing the finish does. Kernels of 64 registers a thread spilled more around a call that the rounds go
//                 on with than for all the rest: the throughput plan's with several CTAs per row 196 bytes instead of 64, its calls
//                 3 to 9 % slower (12 rows of 250K 4.58 / 4.32 us, bf16 16 of 128K 3.95 / 3.6); the merge needed 92 registers
//                 instead of 64 (200 rows of 4 lists 49.6 / 30.4); short rows with 256 threads 39.6 / 35.8 (2,048 of 4K).
//   kCopiesBack   the rounds go on if the threshold is a larger key after all. With 128 registers a thread nothing spills,
//                 and it is the rest that costs: one row of 96K 10.54 / 10.46, 7 of 1M 18.6 / 18.4, warm 4 of 200K 9.15 / 9.02.
//                 (With the output passed through shared memory here too, one of 96K 10.54.)
//   kCopiesHere   inside the former
enum CopiesWay : int { kCopiesRest = 0, kCopiesBack = 1, kCopiesHere = 2 };
template <int NT, bool kTrackMin, int kCopies, class Src>
__device__ __forceinline__ void finish_rounds(const Src src, const FinishOut o, uint32_t need, uint32_t lo, uint32_t cap, uint32_t focus,
                                              uint32_t known_total, int idx_bits, uint32_t* hist, bool hist_clear);
// (what is passed by value comes out of the stack, into registers)
template <int NT, bool kTrackMin, class Src>
__device__ __noinline__ bool finish_copies_back(const Src passed, const FinishOut passed_out, uint32_t need, uint32_t lo, uint32_t cap,
                                                int idx_bits, uint32_t* hist) {
  const Src src = passed;
  const FinishOut o = passed_out;
  return finish_copies<NT, kTrackMin>(src, o, need, lo, cap > lo, idx_bits, hist);
}
template <int NT, bool kTrackMin, class Src>
__device__ __noinline__ void finish_copies_rest(const Src passed, Ctrl* ctrl, uint32_t need, uint32_t lo, uint32_t cap, int idx_bits,
                                                uint32_t* hist) {
  const Src src = passed;
  __syncthreads();  // (ctrl->to, left there by one thread)
  finish_rounds<NT, kTrackMin, kCopiesHere>(src, FinishOut{ctrl->to, ctrl}, need, lo, cap, lo, 0u, idx_bits, hist, false);
}

// The rounds over the keys, [lo, cap] with a focus, and the output: see cta_finish. known_total: not 0 for candidates that
// need no round.
template <int NT, bool kTrackMin, int kCopies, class Src>
__device__ __forceinline__ void finish_rounds(const Src src, const FinishOut o, uint32_t need, uint32_t lo, uint32_t cap, uint32_t focus,
                                              uint32_t known_total, int idx_bits, uint32_t* hist, bool hist_clear) {
  const int tid = threadIdx.x;
  const uint32_t hist_s = smem_u32(hist);
  // Only the threshold is determined by the rounds; nothing is written yet.
  // Outcome: the threshold bin, keys [t_lo, t_hi]. Everything above it wins; of the
  // bin itself either everything wins (all_bin) or, when it holds <= kSmall candidates, the best
  // `need2` of them, found by ranking.
  uint32_t t_lo = lo, t_hi = cap;
  uint32_t need2 = need, cnt = known_total;
  bool all_bin = false, found = false;
  if (known_total != 0u) {
    // exactly as many candidates as are wanted, or so few that they are ranked directly
    all_bin = known_total == need;
    found = true;
    __syncthreads();  // (as in a round: what the caller has read through ctrl may be overwritten from here on)
  }
  for (int round = 0; round < 8 && !found; ++round) {
    if (lo == focus) {  // one key left, or bounded by
      if constexpr (kCopies == kCopiesRest) {
        if (tid == 0) o.ctrl->to = o;
        finish_copies_rest<NT, kTrackMin>(src, o.ctrl, need, lo, cap, idx_bits, hist);
        return;
      } else if constexpr (kCopies == kCopiesBack) {
        if (finish_copies_back<NT, kTrackMin>(src, o, need, lo, cap, idx_bits, hist)) return;
      } else {
        if (finish_copies<NT, kTrackMin>(src, o, need, lo, cap > lo, idx_bits, hist)) return;
      }
      ++lo;
      focus = cap;
      hist_clear = false;
    }
    const KeyDigit dg = make_key_digit(lo, focus);
    if (!hist_clear) {
      __syncthreads();
      for (int b = tid; b < kFinishBins; b += NT) hist[b] = 0u;
      __syncthreads();
    }
    const uint32_t span = cap - lo;
    src.for_each_key([&](const uint32_t (&k)[kWalk]) {
#pragma unroll
      for (int u = 0; u < kWalk; ++u) red_shared_inc_if(hist_s + dg.of(k[u]) * 4u, k[u], k[u] - lo, span);
    });
    __syncthreads();
    FFTOPK_MARK(16);
    const uint4 f = finish_pick<NT>(hist_s, need, o.ctrl);
    FFTOPK_MARK(17);
    if (f.x == kNoBin) break;
    cnt = f.z;
    need2 = need - f.y;
    t_lo = dg.bin_low(f.x);
    t_hi = dg.bin_high(f.x, cap);
    all_bin = cnt == need2;
    found = all_bin || cnt <= (uint32_t)kSmall;
    if (!found) {
      lo = t_lo;
      cap = focus = t_hi;
      need = need2;
      hist_clear = false;
    }
  }
  FFTOPK_MARK(30);
  if (!found) {
    if (tid == 0 && o.status) atomicOr(o.status, 2u);
    return;
  }
  const uint32_t below = t_lo ? t_lo - 1u : 0u;  // (an empty slot has key 0)
  finish_output<NT, kTrackMin>(src, o, need2, cnt, all_bin, all_bin ? below : t_hi, below,
                               [](uint64_t c) { return (uint32_t)(c >> 32); });
}

// ---------------------------------------------------------------------------------------------
// Single-CTA finish. The source holds composites c = (key << 32) | ~idx in shared memory (0 =
// empty slot), all of them with keys inside [klo, kcap]; klo > kcap means "range unknown" and costs a pass
// that finds it. Writes the `need` largest composites' indices (and keys) to
// out_idx[out_base ...], in unspecified order.
//
// Replaces the reference's refinement rounds on shared-memory survivors and its CAS insertion
// tail (topk_indexer_radix.cu:686-781, 109-141, 788-850). Because the index is part of the
// composite, equal values are resolved towards the lower index by the same rounds, and the last
// <= 256 undecided candidates are ranked by votes.
//
// What bounds it is the instructions its warps issue (rank 0's 16 warps work alone on their SM, and a batch of rows
// fills every issue slot), so the rounds work on 32-bit fields: on the keys, and only when one key is left - more
// copies of the threshold than can be ranked - on the inverted indices below it. (With 64-bit
// composites as the digits' field a round cost 280 instructions per warp besides the candidates', and the output 450:
// 11,700 of the 26,200 warp instructions of a row of 8K elements.)
// `kfocus`: see FieldDigit (fftopk_decide.h).
// `idx_bits`: all indices are < 2^idx_bits, so the inverted-index bits above that are all ones.
// `page`: optional per-row table; the value written is then page[idx] instead of idx + idx_offset
// (the fused page-table transform of the reference's topk_transform_* kernels, :871-958).
// ---------------------------------------------------------------------------------------------
// `known_total`: when not 0, the number of candidates in the source; if it equals `need` they all
// win and no round is run. kTrackMin: the smallest key among the winners - the key of the
// need-th largest candidate - is left in ctrl->thr_key (atomic min; the caller presets it).
// Inlined, and the source comes by value: as a call, source and arguments went through every thread's
// stack, and beside 200 KB of shared memory L1 has no room for the stacks of 1024 threads - each access
// was a round trip to L2 (the passes over the candidates took 1.4 and 2 to 4 us instead of 0.4 and 0.7).
template <int NT, class Src, bool kTrackMin = false, int kCopies = kCopiesRest>
__device__ __forceinline__ void cta_finish(const Src src, uint32_t need, uint32_t klo, uint32_t kcap, uint32_t kfocus,
                           int idx_bits, uint32_t* hist /* >= kFinishBins words */, Ctrl* ctrl, int32_t* out_idx,
                           uint32_t* out_key, uint32_t out_base, uint32_t out_slots /* k of the row */,
                           int32_t idx_offset, uint32_t* status,
                           const int32_t* page = nullptr /* when set: out = page[idx] */, uint32_t known_total = 0u,
                           bool hist_clear = false /* `hist` is all zero already */) {
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const uint32_t hist_s = smem_u32(hist);
  if (tid == 0) ctrl->small_n = 0u;  // (every path has a block barrier before it is used)
  if (klo > kcap) {
    // Range unknown: the smallest and the largest key present bound it.
    uint32_t kmin = ~0u, kmax = 0u;
    src.for_each_key([&](const uint32_t (&k)[kWalk]) {
#pragma unroll
      for (int u = 0; u < kWalk; ++u) {
        if (k[u] != 0u) {
          kmin = min(kmin, k[u]);
          kmax = max(kmax, k[u]);
        }
      }
    });
    kmin = __reduce_min_sync(kFull, kmin);
    kmax = __reduce_max_sync(kFull, kmax);
    if (lane == 0) {
      hist[2 * warp + 0] = kmin;
      hist[2 * warp + 1] = kmax;
    }
    __syncthreads();
    const bool in = lane < NT / 32;
    klo = __reduce_min_sync(kFull, in ? hist[2 * lane + 0] : ~0u);
    kcap = __reduce_max_sync(kFull, in ? hist[2 * lane + 1] : 0u);
    if (klo > kcap) {  // no candidate at all
      if (tid == 0 && status) atomicOr(status, 2u);
      return;
    }
    kfocus = kcap;
    hist_clear = false;
    __syncthreads();  // the scratch words are about to be cleared as the histogram
    FFTOPK_MARK(31);
  }
  const bool few = known_total != 0u && known_total >= need && (known_total == need || known_total <= (uint32_t)kSmall);
  const FinishOut o{{out_idx, out_key, status, page, out_base, out_slots, idx_offset, need}, ctrl};
  finish_rounds<NT, kTrackMin, kCopies>(src, o, need, klo, kcap, kfocus < klo || kfocus > kcap ? kcap : kfocus, few ? known_total : 0u,
                                      idx_bits, hist, hist_clear);
}

// The finish of a lone CTA: the candidates' keys are in registers, round 0's histogram (`hist`, with
// make_key_digit(klo, kfocus)) is built. A batch of rows fills the issue slots, so this is written for few
// instructions: the thread that finds the bin works out the bounds, keys are compared where they are, and
// nothing but the indices is read again. Where the threshold bin holds more than can be ranked, further rounds narrow
// it to one key, and copies of that are resolved down to the last index to be taken: the keys of those behind it are
// cleared and everything that is left wins.
template <int NT, int R, bool kTrackMin>
__device__ __forceinline__ void lone_finish(RegSegCands<NT, R>& held, const FinishOut& o, uint32_t need, uint32_t klo,
                                            uint32_t kfocus, int idx_bits, uint32_t* hist) {
  static_assert(R % 4 == 0, "");
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  Ctrl* ctrl = o.ctrl;
  const uint32_t fin = smem_u32(&ctrl->fin), hist_s = smem_u32(hist), wtot = smem_u32(ctrl->wtot);
  constexpr uint32_t kMany = 0xfffffffeu;
  // fin: largest key that does not win for certain, x; undecided candidates: their keys are in (y, x]; their number (kMany:
  // too many), z; how many of them win, w
  auto pick = [&](const KeyDigit dg, uint32_t want, uint32_t cap, uint32_t most) {
    block_pick<NT>(hist_s, want, wtot, [&] { sts128(fin, 0u, 0u, kNoBin, 0u); ctrl->small_n = 0u; },
                   [&](uint32_t bin, uint32_t above, uint32_t n) {
                     const uint32_t low = dg.bin_low(bin), below = low ? low - 1u : 0u;
                     const bool all = n == want - above;
                     sts128(fin, all ? below : dg.bin_high(bin, cap), below, all ? 0u : (n <= most ? n : kMany), want - above);
                   });
    return lds128(fin);
  };
  auto clear = [&] {
    for (int b = tid; b < kFinishBins / 4; b += NT) sts_zero16(hist_s + b * 16);
    __syncthreads();
  };
  uint4 f = pick(make_key_digit(klo, kfocus), need, 0xffffffffu, (uint32_t)kSmall);
  FFTOPK_MARK(17);
  if (f.z == kMany) {  // (uniform)
    uint32_t lo = f.y + 1u, cap = f.x;
    while (lo < cap && f.z == kMany) {  // other values than one: by key again
      __syncthreads();  // (everybody has read the result)
      clear();
      const KeyDigit dg = make_key_digit(lo, cap);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        if (i * 32 >= held.wn) break;
        red_shared_inc_if(hist_s + dg.of(held.key[i]) * 4u, held.key[i], held.key[i] - lo, cap - lo);
      }
      __syncthreads();
      f = pick(dg, f.w, cap, (uint32_t)kSmall);
      lo = f.y + 1u;
      cap = f.x;
    }
    if (f.z == kMany) {  // copies of `lo`
      const uint32_t key = lo;
      uint32_t ilo = inverted_index_floor(idx_bits), icap = 0xffffffffu;
      do {  // (indices differ: a round that is down to one of them takes its bin whole)
        __syncthreads();
        clear();
        const KeyDigit dg = make_key_digit(ilo, icap);
#pragma unroll
        for (int i = 0; i < R; ++i) {
          if (i * 32 >= held.wn) break;
          if (held.key[i] == key) {
            const uint32_t v = ~lds32(held.seg + (uint32_t)(i * 32 + lane) * 4u);
            if (v - ilo <= icap - ilo) red_shared_inc(hist_s + dg.of(v) * 4u);
          }
        }
        __syncthreads();
        f = pick(dg, f.w, icap, 0u);
        ilo = f.y + 1u;
        icap = f.x;
      } while (f.z == kMany && ilo < icap);
      if (f.z == kMany) f.z = kNoBin;  // (one index many times over: not a list of the library's making)
#pragma unroll
      for (int i = 0; i < R; ++i) {
        if (i * 32 >= held.wn) break;
        if (held.key[i] == key) {
          if (~lds32(held.seg + (uint32_t)(i * 32 + lane) * 4u) < ilo) held.key[i] = 0u;
        }
      }
      if (f.z != kNoBin) f = make_uint4(key - 1u, key - 1u, 0u, 0u);
    }
  }
  if (f.z == kNoBin) {  // (uniform)
    if (tid == 0 && o.status) atomicOr(o.status, 2u);
    return;
  }
  uint32_t n = 0u;
#pragma unroll
  for (int i = 0; i < R; i += 4) {
    if (i * 32 >= held.wn) break;
#pragma unroll
    for (int u = 0; u < 4; ++u) count_if_above(n, held.key[i + u], f.x);
  }
  n = __reduce_add_sync(kFull, n);
  const uint32_t wsum = smem_u32(ctrl->wmax);
  if (lane == 0) sts32(wsum + warp * 4, n);
  __syncthreads();
  uint32_t wpos = o.out_base + __reduce_add_sync(kFull, lane < warp ? lds32(wsum + lane * 4) : 0u);
  FFTOPK_MARK(70);
  const unsigned lt = (1u << lane) - 1u;
  const uint32_t small_s = smem_u32(ctrl->small), small_n = smem_u32(&ctrl->small_n);
  uint32_t win_min = 0xffffffffu;
  auto pass = [&](auto plain) {  // (plain: indices alone, as they are)
#pragma unroll
    for (int i = 0; i < R; i += 4) {
      if (i * 32 >= held.wn) break;
      uint32_t idx[4];
      int32_t v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = (i + u) * 32 + lane;
        idx[u] = lds32_below(j, held.wn, held.seg + (uint32_t)j * 4u);
        v[u] = (int32_t)idx[u];
        if constexpr (!decltype(plain)::value) {
          if (!o.page) {
            v[u] += o.idx_offset;
          } else if (held.key[i + u] > f.x) {
            v[u] = __ldg(o.page + idx[u]);
          }
        }
      }
      uint32_t nearest = 0xffffffffu;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t k = held.key[i + u];
        const unsigned bw = __ballot_sync(kFull, k > f.x);
        const uint32_t pos = wpos + (uint32_t)__popc(bw & lt);
        if (!(k > f.x) || FFTOPK_CHECK(3, pos, o.out_slots, o.status)) {
          st_global_if_above(k, f.x, o.out_idx + pos, (uint32_t)v[u]);
          if constexpr (!decltype(plain)::value) {
            if (o.out_key) st_global_if_above(k, f.x, o.out_key + pos, k);
          }
        }
        wpos += (uint32_t)__popc(bw);
        if constexpr (kTrackMin) win_min = min(win_min, k > f.x ? k : 0xffffffffu);
        nearest = min(nearest, k - f.y - 1u);
      }
      if (__any_sync(kFull, nearest < f.x - f.y)) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint32_t k = held.key[i + u];
          const uint32_t slot =
              append64_if(k - f.y - 1u < f.x - f.y, small_n, small_s, kSmall, ((uint64_t)k << 32) | (uint64_t)(~idx[u]));
          (void)FFTOPK_CHECK(4, slot, kSmall, o.status);
        }
      }
    }
  };
  if (o.page == nullptr && o.out_key == nullptr && o.idx_offset == 0) {
    pass(std::true_type{});
  } else {
    pass(std::false_type{});
  }
  FFTOPK_MARK(33);
  if constexpr (kTrackMin) {
    if (f.z == 0u) {  // (else the smallest winner is one of those that are ranked)
      win_min = __reduce_min_sync(kFull, win_min);
      if (lane == 0 && win_min != 0xffffffffu) atomicMin(&ctrl->thr_key, win_min);
    }
  }
#ifdef FFTOPK_CHECKED
  const uint32_t set_w = __reduce_add_sync(kFull, lane < NT / 32 ? lds32(wsum + lane * 4) : 0u);
  __syncthreads();
  if (tid == 0) {
    const uint32_t want_w = f.z == 0u ? need : need - f.w;  // (undecided ones: need - f.w certain winners)
    if (set_w != want_w) check_fail(10, set_w, want_w, o.status);
    if (ctrl->small_n != f.z) check_fail(11, ctrl->small_n, f.z, o.status);
  }
#endif
  if (f.z != 0u) rank_undecided<NT, kTrackMin>(o, need - f.w, f.w, f.z);
}

}  // namespace fftopk

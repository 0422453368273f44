// engine.cu - persistent sm_100a kernels of the DynaMOSP update path.
//
// sosp_engine<Mode> runs a whole SOSP update (or an SSSP from scratch, or
// Steps 2-3 of the MOSP update) in one cooperative launch. The phases
// follow the reference algorithm (SMShovan/MOSP-CUDA src/sospUpdateGpu.cu:
// 211-519 and src/combinedGraphGpu.cu:55-121), re-planned for B200:
//
//   * all K objectives of a MOSP update share one launch and run their
//     phases and near-far iterations side by side, so the grid barriers
//     (the latency floor of a high-diameter graph) are paid once for all
//     objectives instead of K times;
//   * one grid barrier per near-far iteration: list counters rotate
//     through three slots and the far-pile minimum is folded into the
//     appends, so the threshold step needs no separate reduction pass;
//   * the barrier is a release/arrive pair on separate L2 lines with a
//     wall-clock bound (%globaltimer): a run that stalls returns
//     MOSP_ERR_TIMEOUT instead of hanging the GPU;
//   * subtree invalidation packs "ancestor or flag" into one int per
//     vertex, so a pointer-jumping step is two dependent loads;
//   * list appends are staged per CTA in shared memory and written out
//     with one reservation per list and iteration; a warp spreads the
//     edges of its items over its lanes, and rows of more than 512 edges
//     go to the whole CTA, in launches whose graph has power-law hubs
//     (rows of more than 2,048);
//   * the pull pass scans in-rows four edges per round with their loads
//     in flight together;
//   * the lowest-id parent recovery of distance-only objectives is
//     edge-balanced (equal edge slices per warp, a shuffle search for the
//     rows) and, after an update launch, runs as its own kernel
//     (recoverParents) so that L1 is not shared with the append stage;
//     with input trees declared canonical it is restricted to the vertices
//     the batch reaches (recover.cu: the unpack lists the vertices whose
//     distance changed).
//
// Result semantics (identical to the reference): words pack
// (distance << b | parent) and only strictly better words are kept
// (64-bit atomicMin), so among equal distances the lowest parent id wins;
// a vertex is expanded whenever its distance strictly decreases. The fixed
// point does not depend on the schedule, the grid size or the bucket width.
#include "engine.h"

#include <climits>

#include "device.h"

namespace mospb200 {
namespace {

// ---------------------------------------------------------------------------
// Small device helpers
// ---------------------------------------------------------------------------

__device__ __forceinline__ u64 ldRelaxed64(const u64 *p) {
  u64 v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

/// Two adjacent words, each read on its own, past L1.
__device__ __forceinline__ void ldPair(const unsigned *p, unsigned &a, unsigned &b) {
  asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(a), "=r"(b) : "l"(p) : "memory");
}

__device__ __forceinline__ void stRelaxed64(unsigned long long *p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

/// Word helpers for one objective.
struct Pk {
  int bits;
  u64 noParent;
  __device__ __forceinline__ u64 pack(u64 d, int p) const {
    return bits == 0 ? d : ((d << bits) | (p < 0 ? noParent : static_cast<u64>(p)));
  }
  __device__ __forceinline__ u64 dist(u64 w) const { return w >> bits; }
  __device__ __forceinline__ int parent(u64 w) const {
    const u64 f = w & noParent;
    return f == noParent ? -1 : static_cast<int>(f);
  }
};

__device__ __forceinline__ Pk pkOf(const ObjectiveArgs &o) {
  return Pk{o.parentBits, o.noParent};
}

/// CTA 0 records the time of a phase boundary.
__device__ __forceinline__ void markPhase(EngineControl *c, int phase) {
  if (blockIdx.x == 0 && threadIdx.x == 0) c->phaseNs[phase] = globalNs();
}

/// Reserve one slot of a list: one atomicAdd per group of lanes of the warp
/// that append to the same counter at the same time.
__device__ __forceinline__ int warpAppend(int *counter) {
  const unsigned mask = __activemask();
  const unsigned peers =
      __match_any_sync(mask, static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(counter)));
  const int leader = __ffs(peers) - 1;
  const unsigned lane = laneId();
  int base = 0;
  if (static_cast<int>(lane) == leader) base = atomicAdd(counter, __popc(peers));
  base = __shfl_sync(peers, base, leader);
  return base + __popc(peers & ((1u << lane) - 1u));
}

/// Fold d into the minimum kept (as a complement, so 0 means "none") at
/// *minC: one atomicMax per group of lanes with the same target.
__device__ __forceinline__ void warpMinInto(u64 *minC, u64 d) {
  const unsigned mask = __activemask();
  const unsigned peers =
      __match_any_sync(mask, static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(minC)));
  const unsigned hi = static_cast<unsigned>(d >> 32);
  const unsigned lo = static_cast<unsigned>(d);
  const unsigned mhi = __reduce_min_sync(peers, hi);
  const unsigned mlo = __reduce_min_sync(peers, hi == mhi ? lo : 0xffffffffu);
  if (static_cast<int>(laneId()) == __ffs(peers) - 1) {
    atomicMax(minC, ~((static_cast<u64>(mhi) << 32) | mlo));
  }
}

__device__ __forceinline__ u64 warpMinU64(u64 v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const u64 o = __shfl_xor_sync(kFull, v, off);
    v = o < v ? o : v;
  }
  return v;
}

/// Graph loads: the update and scratch modes read a graph that is
/// read-only for the whole launch (read-only path); the combined mode
/// reads a graph built earlier in the same launch (L2).
template <int Mode>
__device__ __forceinline__ int ldGraph(const int *p) {
  if constexpr (Mode == kModeCombined) {
    return __ldcg(p);
  } else {
    return __ldg(p);
  }
}

// Shared per-CTA view of the loop state (identical in every CTA).
struct LoopShared {
  long long off[kMaxK + 1];
  u64 thr[kMaxK];
  int mode[kMaxK];
  int fp[kMaxK];
  int fs[kMaxK];
  long long total;
};

enum : int { kDone = 0, kPush = 1, kSplit = 2 };

// ---------------------------------------------------------------------------
// Per-CTA staging of list appends
//
// Every append of an iteration (next near list, far piles) goes to a
// shared-memory buffer first: a shared atomic per warp group gives the slot
// and the rank within the destination list. At the end of the iteration the
// CTA reserves one range per list with a single global atomic and copies
// its entries out, so the same-address global counters see one atomic per
// CTA and list instead of one per warp group on the relaxation's critical
// path. Entries that do not fit the buffer take the direct global path.
// ---------------------------------------------------------------------------
constexpr int kStage = kStageEntriesMax;
// Long rows are expanded (push) or reduced (pull) by a whole CTA instead of
// one warp: a power-law hub row (10^5 edges) would otherwise keep one warp
// busy for the whole iteration. A launch turns this on only when its graph
// has rows of more edges than this (EngineControl::heavy, set in the first
// phase), so graphs without them take no extra CTA barriers.
constexpr int kHeavyDegDefault = 2048;  // EngineParams::heavyDeg when 0
constexpr int kHeavyCap = 128;

/// A graph with rows above this many edges runs the bulk loop; a launch
/// parameter, so the autotuner can move it.
__device__ __forceinline__ int heavyDegOf(const EngineParams &P) {
  return P.heavyDeg > 0 ? P.heavyDeg : kHeavyDegDefault;
}

/// In such a launch, rows above this many edges go to a whole CTA: a quarter of
/// the default threshold, since a warp with 2,000 edges of its own keeps the
/// grid waiting (R-MAT graph of scale 22, K = 5: update and combined loops
/// 1.32 -> 0.95 ms; of 60,001 vertices 0.24 -> 0.20 ms), while graphs with no
/// longer rows than that stay faster in the asynchronous loop.
__device__ __forceinline__ int ctaRowOf(const EngineParams &P) {
  return P.heavyDeg > 0 ? P.heavyDeg : kHeavyDegDefault / 4;
}

struct StageHeader {
  int cap;                     // entries per list partition (kStage / (2K))
  int pad;
  int count[2 * kMaxK];        // appends per list this iteration (may exceed cap)
  int start[2 * kMaxK];        // entries before this were expanded by the CTA itself
  int roundEnd[kMaxK];         // end of the near entries of the current local round
  int roundTotal;              // entries of the current local round (0: no round)
  int base[2 * kMaxK];         // global start of this CTA's range
  u64 farMin[kMaxK];           // minimum distance appended to far (plain)
  long long expanded[kMaxK];   // non-stale expansions (statistics)
  // heavy rows met by the CTA's warps, handled by the whole CTA afterwards
  // (rows beyond kHeavyCap stay with their warp)
  int heavyCount;
  int heavyK[kHeavyCap];
  int heavyU[kHeavyCap];
  int heavyBeg[kHeavyCap];
  int heavyDeg[kHeavyCap];
  u64 heavyD[kHeavyCap];       // push: the row's distance; pull: the word before the pass
  u64 heavyBest[kHeavyCap];    // pull: best word over the row, reduced by the CTA
};

struct StageEntry {
  int v;
  int meta;                    // list << 16 | rank
  u64 d;
};

/// Whether a row of deg edges goes to the whole CTA. Rows above the hub
/// threshold find the queue's second half free: a hub row left to one warp
/// costs more than many shorter ones (tree from scratch of an R-MAT graph of 1M
/// vertices 6.2 ms with any row in any place).
__device__ __forceinline__ bool takesCta(const EngineParams &P, const StageHeader &H, int deg) {
  if (deg <= ctaRowOf(P)) return false;
  return deg > heavyDegOf(P) || *const_cast<const volatile int *>(&H.heavyCount) < kHeavyCap / 2;
}

constexpr size_t kStageHeaderBytes = (sizeof(StageHeader) + 15) / 16 * 16;
constexpr size_t kStageBytes = kStageHeaderBytes + kStage * sizeof(StageEntry);

/// Dynamic shared memory of a launch with `entries` stage entries.
constexpr size_t stageBytesFor(int entries) {
  return kStageHeaderBytes + static_cast<size_t>(entries) * sizeof(StageEntry);
}

__device__ __forceinline__ StageHeader &stageHeader() {
  extern __shared__ __align__(16) unsigned char dynSmem[];
  return *reinterpret_cast<StageHeader *>(dynSmem);
}

__device__ __forceinline__ StageEntry *stageEntries() {
  extern __shared__ __align__(16) unsigned char dynSmem[];
  return reinterpret_cast<StageEntry *>(dynSmem + kStageHeaderBytes);
}

/// Destination of list l in this iteration: near list of objective l (l <
/// K) or the far pile objective l - K appends to (the current pile while it
/// pushes, the other pile while its pile is split).
struct Target {
  int *counter;
  int *v;
  u64 *d;
  u64 *minC;
};

__device__ __forceinline__ Target listTarget(const EngineParams &P, const LoopShared &L, int l,
                                             int wrSlot, int *nearWV, u64 *nearWD) {
  const int K = P.K;
  if (l < K) {
    const long long kn = static_cast<long long>(l) * P.strideNear;
    return Target{&P.ctl->nearCount[l][wrSlot], nearWV + kn, nearWD + kn, nullptr};
  }
  const int k = l - K;
  const long long ko = static_cast<long long>(k) * P.strideFar;
  if (L.mode[k] == kSplit) {
    const int s = (L.fs[k] + 1) % 3;
    return Target{&P.ctl->farCount[k][s], (L.fp[k] == 0 ? P.farL1 : P.farL0) + ko, nullptr,
                  &P.ctl->farMinC[k][s]};
  }
  const int s = L.fs[k];
  return Target{&P.ctl->farCount[k][s], (L.fp[k] == 0 ? P.farL0 : P.farL1) + ko, nullptr,
                &P.ctl->farMinC[k][s]};
}

/// A near entry (v, d) of objective k that found its near list full goes to
/// the far pile instead (once, by the in-far flag); the split after the
/// near list has run dry brings it back below the threshold. So the near
/// lists can be smaller than the worst case of one iteration.
__device__ __forceinline__ void divertToFar(const EngineParams &P, const LoopShared &L, int k, int v,
                                            u64 d) {
  if (atomicExch(P.inFar + static_cast<long long>(k) * P.stride + v, 1) != 0) return;
  const Target t = listTarget(P, L, P.K + k, 0, nullptr, nullptr);
  const int idx = warpAppend(t.counter);
  t.v[idx] = v;
  warpMinInto(t.minC, d);
}

/// Append (v, d) to list l (far lists: d only feeds the pile minimum). The
/// staging buffer is split into one partition per list; the rank within the
/// list is the slot, so a warp group needs one shared atomic.
__device__ __forceinline__ void stageAppend(const EngineParams &P, const LoopShared &L, int l,
                                            int v, u64 d, int wrSlot, int *nearWV, u64 *nearWD) {
  StageHeader &H = stageHeader();
  StageEntry *E = stageEntries();
  const unsigned lane = laneId();
  const unsigned lt = (1u << lane) - 1u;
  const unsigned mask = __activemask();
  const unsigned peers = __match_any_sync(mask, l);
  const int leader = __ffs(peers) - 1;
  int rankBase = 0;
  if (static_cast<int>(lane) == leader) rankBase = atomicAdd(&H.count[l], __popc(peers));
  rankBase = __shfl_sync(peers, rankBase, leader);
  const int rank = rankBase + __popc(peers & lt);
  if (l >= P.K) {
    // far pile minimum of this CTA (shared), reduced over the group first
    const unsigned hi = static_cast<unsigned>(d >> 32), lo = static_cast<unsigned>(d);
    const unsigned mhi = __reduce_min_sync(peers, hi);
    const unsigned mlo = __reduce_min_sync(peers, hi == mhi ? lo : 0xffffffffu);
    if (static_cast<int>(lane) == leader) {
      atomicMin(&H.farMin[l - P.K], (static_cast<u64>(mhi) << 32) | mlo);
    }
  }
  if (rank < H.cap) {
    E[l * H.cap + rank] = StageEntry{v, 0, d};
  } else {
    // partition full: this entry takes the direct global path
    const Target t = listTarget(P, L, l, wrSlot, nearWV, nearWD);
    const int idx = warpAppend(t.counter);
    if (l < P.K && idx >= P.strideNear) {
      divertToFar(P, L, l, v, d);
      return;
    }
    t.v[idx] = v;
    if (t.d != nullptr) t.d[idx] = d;
  }
}

/// End of an iteration: reserve every list's range once per CTA, copy the
/// staged entries out, fold the far minima. (The expansion counts are
/// summed per CTA and folded into the statistics after the loop.)
__device__ void flushStage(const EngineParams &P, const LoopShared &L, int wrSlot, int *nearWV,
                           u64 *nearWD) {
  StageHeader &H = stageHeader();
  StageEntry *E = stageEntries();
  const int K = P.K;
  __syncthreads();
  const int t = threadIdx.x;
  if (t < 2 * K) {
    const int staged = (H.count[t] < H.cap ? H.count[t] : H.cap) - H.start[t];
    if (staged > 0) H.base[t] = atomicAdd(listTarget(P, L, t, wrSlot, nearWV, nearWD).counter, staged);
  }
  if (t < K && H.farMin[t] != kInfWord) {
    atomicMax(listTarget(P, L, K + t, wrSlot, nearWV, nearWD).minC, ~H.farMin[t]);
  }
  __syncthreads();
  for (int l = 0; l < 2 * K; ++l) {
    const int first = H.start[l];
    const int staged = (H.count[l] < H.cap ? H.count[l] : H.cap) - first;
    if (staged <= 0) continue;
    const Target tg = listTarget(P, L, l, wrSlot, nearWV, nearWD);
    const int b = H.base[l];
    for (int i = t; i < staged; i += blockDim.x) {
      const StageEntry e = E[l * H.cap + first + i];
      if (l < K && b + i >= P.strideNear) {
        divertToFar(P, L, l, e.v, e.d);  // the near list is full
        continue;
      }
      tg.v[b + i] = e.v;
      if (tg.d != nullptr) tg.d[b + i] = e.d;
    }
  }
}

/// Edge slots a lane relaxes at once (loads and atomics overlapped).
#ifndef MOSP_EDGE_SLOTS
#define MOSP_EDGE_SLOTS 2
#endif
constexpr int kSlots = MOSP_EDGE_SLOTS;
/// A strict improvement of w's distance to d (objective k): to the next near
/// list (d below the threshold) or, once, to the far pile.
__device__ __forceinline__ void pushImproved(const EngineParams &P, const LoopShared &L, int k, int w,
                                             u64 d, int wrSlot, int *nearWV, u64 *nearWD) {
  if (d < L.thr[k]) {
    stageAppend(P, L, k, w, d, wrSlot, nearWV, nearWD);
  } else if (atomicExch(P.inFar + static_cast<long long>(k) * P.stride + w, 1) == 0) {
    stageAppend(P, L, P.K + k, w, d, wrSlot, nearWV, nearWD);
  }
}

/// Lane of the warp whose edge range holds edge slot s: the number of
/// lanes whose inclusive edge count is <= s (binary search by shuffles).
__device__ __forceinline__ int slotOwner(int incl, int s) {
  int lo = 0;
#pragma unroll
  for (int step = 16; step >= 1; step >>= 1) {
    const int probe = __shfl_sync(kFull, incl, lo + step - 1);
    if (probe <= s) lo += step;
  }
  return lo;
}

/// Relaxation of edge e out of u (objective k, distance du): atomicMin of
/// the word of its head, and the stage append of a strict improvement.
template <int Mode>
__device__ __forceinline__ void relaxEdge(const EngineParams &P, const LoopShared &L,
                                          const int *outCol, const int *const *outWk, int k,
                                          int u, u64 du, int e, int wrSlot, int *nearWV,
                                          u64 *nearWD) {
  const ObjectiveArgs &O = P.obj[k];
  const Pk pk = pkOf(O);
  const long long ko = static_cast<long long>(k) * P.stride;
  const int w = ldGraph<Mode>(outCol + e);
  const u64 nd = du + static_cast<u64>(ldGraph<Mode>(outWk[k] + e));
  if (w == P.source || nd > O.maxDist) return;
  const u64 old = atomicMin(P.packed + ko + w, pk.pack(nd, u));
  if (nd >= pk.dist(old)) return;
  pushImproved(P, L, k, w, nd, wrSlot, nearWV, nearWD);
}

/// The CTA's queued heavy rows, each expanded by all threads of the CTA.
/// Every thread of the CTA calls it; it starts with a barrier (so it also
/// serves as the barrier after the expansion that queued the rows) and,
/// when rows were queued, ends with one.
template <int Mode>
__device__ void expandHeavy(const EngineParams &P, const LoopShared &L, const int *outCol,
                            const int *const *outWk, int wrSlot, int *nearWV, u64 *nearWD) {
  StageHeader &H = stageHeader();
  __syncthreads();
  const int queued = H.heavyCount;
  if (queued == 0) return;  // the same for every thread of the CTA
  // every thread has read the count before it is reset; no warp queues a
  // row again before the last barrier below
  __syncthreads();
  if (threadIdx.x == 0) H.heavyCount = 0;
  const int count = queued < kHeavyCap ? queued : kHeavyCap;
  for (int h = 0; h < count; ++h) {
    const int k = H.heavyK[h], u = H.heavyU[h], beg = H.heavyBeg[h], end = beg + H.heavyDeg[h];
    const u64 du = H.heavyD[h];
    for (int e = beg + static_cast<int>(threadIdx.x); e < end; e += blockDim.x) {
      relaxEdge<Mode>(P, L, outCol, outWk, k, u, du, e, wrSlot, nearWV, nearWD);
    }
  }
  __syncthreads();
}

/// One warp expands up to 32 near entries, one per lane (u < 0: none):
/// the edges of all lanes are spread over the warp, two slots per lane,
/// with their loads and 64-bit atomicMin overlapped; every strict
/// improvement is staged for the next near list or the far pile. All 32
/// lanes call it.
template <int Mode>
__device__ __forceinline__ void expandWarp(const EngineParams &P, const LoopShared &L,
                                           const int *outRow, const int *outCol,
                                           const int *const *outWk, int k, int u, u64 du, int beg,
                                           int deg, int wrSlot, int *nearWV, u64 *nearWD,
                                           bool heavyOn) {
  StageHeader &H = stageHeader();
  const unsigned lane = laneId();
  {
    // statistics: one shared add per objective present in the warp
    const unsigned live = __ballot_sync(kFull, u >= 0);
    if (live != 0) {
      const unsigned peers = __match_any_sync(kFull, u >= 0 ? k : -1);
      if (u >= 0 && static_cast<int>(lane) == __ffs(peers) - 1) {
        atomicAdd(reinterpret_cast<unsigned long long *>(&H.expanded[k]),
                  static_cast<unsigned long long>(__popc(peers)));
      }
    }
  }
  if (__ballot_sync(kFull, deg > 0) == 0) return;
  // heavy rows go to the CTA's queue (expanded by the whole CTA after this
  // round of items) when the launch has any
  if (heavyOn && takesCta(P, H, deg)) {
    const int slot = atomicAdd(&H.heavyCount, 1);
    if (slot < kHeavyCap) {
      H.heavyK[slot] = k;
      H.heavyU[slot] = u;
      H.heavyBeg[slot] = beg;
      H.heavyDeg[slot] = deg;
      H.heavyD[slot] = du;
      deg = 0;
    }
  }
  // rows above 2^20 edges: whole-warp striding, one row at a time
  unsigned huge = __ballot_sync(kFull, deg > (1 << 20));
  while (huge != 0) {
    const int src = __ffs(huge) - 1;
    huge &= huge - 1;
    const int kb = __shfl_sync(kFull, k, src);
    const int ub = __shfl_sync(kFull, u, src);
    const u64 db = __shfl_sync(kFull, du, src);
    const int bb = __shfl_sync(kFull, beg, src);
    const int eb = bb + __shfl_sync(kFull, deg, src);
    const ObjectiveArgs &O = P.obj[kb];
    const Pk pk = pkOf(O);
    const long long kob = static_cast<long long>(kb) * P.stride;
    for (int e = bb + static_cast<int>(lane); e < eb; e += 32) {
      const int w = ldGraph<Mode>(outCol + e);
      const u64 nd = db + static_cast<u64>(ldGraph<Mode>(outWk[kb] + e));
      if (w == P.source || nd > O.maxDist) continue;
      const u64 old = atomicMin(P.packed + kob + w, pk.pack(nd, ub));
      if (nd >= pk.dist(old)) continue;
      pushImproved(P, L, kb, w, nd, wrSlot, nearWV, nearWD);
    }
  }
  if (deg > (1 << 20)) deg = 0;
  int incl = deg;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int o = __shfl_up_sync(kFull, incl, off);
    if (static_cast<int>(lane) >= off) incl += o;
  }
  const int edges = __shfl_sync(kFull, incl, 31);
  const int excl = incl - deg;
  constexpr int SL = kSlots;
  for (int s0 = 0; s0 < edges; s0 += 32 * SL) {
    // SL edge slots per lane, their loads and atomics overlapped
    int sl[SL], kk[SL], uu[SL], ee[SL], ww[SL], wt[SL];
    u64 dd[SL], nd[SL], old[SL];
    bool act[SL];
#pragma unroll
    for (int h = 0; h < SL; ++h) {
      sl[h] = s0 + 32 * h + static_cast<int>(lane);
      const int o = slotOwner(incl, sl[h]);
      kk[h] = __shfl_sync(kFull, k, o);
      uu[h] = __shfl_sync(kFull, u, o);
      dd[h] = __shfl_sync(kFull, du, o);
      ee[h] = __shfl_sync(kFull, beg, o) + sl[h] - __shfl_sync(kFull, excl, o);
      act[h] = sl[h] < edges;
    }
#pragma unroll
    for (int h = 0; h < SL; ++h) {
      ww[h] = act[h] ? ldGraph<Mode>(outCol + ee[h]) : 0;
      wt[h] = act[h] ? ldGraph<Mode>(outWk[kk[h]] + ee[h]) : 0;
    }
    u64 cw[SL];
#pragma unroll
    for (int h = 0; h < SL; ++h) {
      nd[h] = dd[h] + static_cast<u64>(wt[h]);
      act[h] = act[h] && ww[h] != P.source && nd[h] <= P.obj[kk[h]].maxDist;
      cw[h] = pkOf(P.obj[kk[h]]).pack(nd[h], uu[h]);
    }
    if (P.flags & kFlagPrecheck) {
      u64 cur[SL];
#pragma unroll
      for (int h = 0; h < SL; ++h) {
        cur[h] = act[h] ? __ldcg(P.packed + static_cast<long long>(kk[h]) * P.stride + ww[h]) : 0;
      }
#pragma unroll
      for (int h = 0; h < SL; ++h) act[h] = act[h] && cw[h] < cur[h];
    }
#pragma unroll
    for (int h = 0; h < SL; ++h) {
      old[h] = act[h] ? atomicMin(P.packed + static_cast<long long>(kk[h]) * P.stride + ww[h], cw[h])
                      : 0;
    }
#pragma unroll
    for (int h = 0; h < SL; ++h) {
      if (!act[h] || nd[h] >= pkOf(P.obj[kk[h]]).dist(old[h])) continue;
      pushImproved(P, L, kk[h], ww[h], nd[h], wrSlot, nearWV, nearWD);
    }
  }
}

// ---------------------------------------------------------------------------
// Near-far loop shared by every mode
//
// Near lists carry (vertex, distance) pairs: an entry is stale when the
// vertex's word has a smaller distance by the time it is read, and is then
// skipped (a newer entry exists). Every strict improvement appends exactly
// one entry, so no claim atomic is needed and a list never holds more
// entries than the relaxations of one iteration (<= m) plus the far pile
// (<= n). Far piles keep one entry per vertex (inFar flag).
// ---------------------------------------------------------------------------
template <int Mode>
__device__ bool nearFarLoop(const EngineParams &P, const int *outRow,
                            const int *outCol, const int *const *outWk,
                            Sync &epoch, u64 *deltaOverride, int genBase) {
  __shared__ LoopShared L;
  StageHeader &H = stageHeader();
  EngineControl *c = P.ctl;
  const int K = P.K;
  const unsigned lane = laneId();
  const int warp = threadIdx.x >> 5;
  const long long gwarp = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + warp;
  const long long nwarps = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);

  // Per-objective loop state, held by lane k of warp 0 (same in every CTA).
  u64 thr = 0;
  int fp = 0, fs = 0;
  int iters = 0, epochs = 0;
  u64 delta = 1;
  if (warp == 0 && static_cast<int>(lane) < K) {
    delta = P.obj[lane].delta;
    if (deltaOverride != nullptr && lane == 0) delta = *deltaOverride;
  }

  if (threadIdx.x < kMaxK) H.expanded[threadIdx.x] = 0;
  // set before the grid barrier that precedes the loop, the same for all
  const bool heavyOn = __ldcg(&c->heavy) != 0;
  int it = 0;
  unsigned long long profNs[2] = {0, 0};
  long long profIters[2] = {0, 0}, profItems[2] = {0, 0};
  unsigned long long part[5] = {0, 0, 0, 0, 0};
  unsigned long long tDecided = 0, tWorked = 0;
  for (;; ++it) {
    const int rdSlot = it % 3, wrSlot = (it + 1) % 3, clrSlot = (it + 2) % 3;
    const unsigned long long itStart = globalNs();
    if (threadIdx.x < 2 * kMaxK) {
      H.count[threadIdx.x] = 0;
      H.start[threadIdx.x] = 0;
    }
    if (threadIdx.x < kMaxK) H.farMin[threadIdx.x] = kInfWord;
    if (threadIdx.x == 0) {
      H.cap = P.stageEntries / (2 * K);
      H.heavyCount = 0;
    }
    if (warp == 0) {
      const int k = static_cast<int>(lane);
      const bool act = k < K;
      int mode = kDone;
      long long items = 0;
      if (act) {
        // (a count past the list's capacity counts entries diverted to far)
        const int nc = static_cast<int>(
            min(static_cast<long long>(__ldcg(&c->nearCount[k][rdSlot])), P.strideNear));
        if (nc > 0) {
          mode = kPush;
          items = nc;
        } else {
          const int fc = __ldcg(&c->farCount[k][fs]);
          if (fc > 0) {
            mode = kSplit;
            items = fc;
            const u64 mnC = __ldcg(&c->farMinC[k][fs]);
            u64 lo = thr;
            if (mnC != 0) {
              const u64 mn = ~mnC;
              lo = mn > thr ? mn : thr;
            }
            thr = (lo > kInfWord - delta) ? kInfWord - 1 : lo + delta;
          }
        }
      }
      long long incl = items;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const long long o = __shfl_up_sync(kFull, incl, off);
        if (static_cast<int>(lane) >= off) incl += o;
      }
      if (act) {
        L.off[k] = incl - items;
        L.thr[k] = thr;
        L.mode[k] = mode;
        L.fp[k] = fp;
        L.fs[k] = fs;
      }
      const long long total = __shfl_sync(kFull, incl, 31);
      if (lane == 0) L.total = total;
      if (act) {
        if (blockIdx.x == 0) {
          c->nearCount[k][clrSlot] = 0;
          if (mode == kSplit) {
            c->farCount[k][(fs + 2) % 3] = 0;
            c->farMinC[k][(fs + 2) % 3] = 0;
          }
        }
        if (mode == kPush) {
          ++iters;
        } else if (mode == kSplit) {
          ++epochs;
          fp ^= 1;           // takes effect after this iteration
          fs = (fs + 1) % 3;
        }
      }
    }
    __syncthreads();
    const long long total = L.total;
    if (total == 0) break;
    if (blockIdx.x == 0 && threadIdx.x == 0) tDecided = globalNs();

    const int *nearRV = (it & 1) ? P.nearV1 : P.nearV0;
    const u64 *nearRD = (it & 1) ? P.nearD1 : P.nearD0;
    int *nearWV = (it & 1) ? P.nearV0 : P.nearV1;
    u64 *nearWD = (it & 1) ? P.nearD0 : P.nearD1;

    // items per warp: ceil(total / warps), between 8 and 32, so that an
    // iteration is spread over every warp of the grid rather than over
    // total / 32 of them (the edges of a warp's items still spread over
    // all 32 lanes)
    //
    // A narrow iteration (at most P.narrowItems items, e.g. a deep graph's
    // thin wavefront or the tail of an epoch) goes to CTA 0 alone, which
    // then keeps expanding the entries it produces (up to P.narrowRounds
    // CTA-local rounds, each a __syncthreads instead of a grid barrier)
    // while the other CTAs go straight to the barrier.
    const bool narrow = total <= P.narrowItems;
    const long long myWarp = narrow ? warp : gwarp;
    const long long allWarps = narrow ? static_cast<long long>(blockDim.x >> 5) : nwarps;
    long long chunk = (total + allWarps - 1) / allWarps;
    chunk = chunk < 8 ? 8 : (chunk > 32 ? 32 : chunk);
    const long long myEnd = (narrow && blockIdx.x != 0) ? 0 : total;
    for (long long base = myWarp * chunk; base < myEnd; base += allWarps * chunk) {
      const long long j = base + lane;
      const bool valid = static_cast<long long>(lane) < chunk && j < total;
      int k = 0;
      if (valid) {
        while (k + 1 < K && L.off[k + 1] <= j) ++k;
      }
      const int mode = valid ? L.mode[k] : kDone;
      const long long i = valid ? j - L.off[k] : 0;
      const long long ko = static_cast<long long>(k) * P.stride;

      if (mode == kSplit) {
        // far pile entry: to the near list below the new threshold
        const int v = __ldcg((L.fp[k] == 0 ? P.farL0 : P.farL1) +
                             static_cast<long long>(k) * P.strideFar + i);
        const u64 word = __ldcg(P.packed + ko + v);
        const u64 d = word == kInfWord ? kInfWord : pkOf(P.obj[k]).dist(word);
        if (d < L.thr[k]) {
          P.inFar[ko + v] = 0;
          stageAppend(P, L, k, v, d, wrSlot, nearWV, nearWD);
        } else {
          stageAppend(P, L, K + k, v, d, wrSlot, nearWV, nearWD);
        }
      }

      // push: one non-stale near entry per lane, edges spread over the warp
      int u = -1, beg = 0, deg = 0;
      u64 du = 0;
      if (mode == kPush) {
        const long long kn = static_cast<long long>(k) * P.strideNear;
        // A stale entry (the word has dropped below its tag since) is
        // expanded with its tag: its offers are strictly larger than the
        // ones of the newer entry, so they never win a word. Skipping the
        // check saves a dependent load on every expansion.
        u = __ldcg(nearRV + kn + i);
        du = __ldcg(nearRD + kn + i);
        beg = ldGraph<Mode>(outRow + u);
        deg = ldGraph<Mode>(outRow + u + 1) - beg;
      }
      expandWarp<Mode>(P, L, outRow, outCol, outWk, k, u, du, beg, deg, wrSlot, nearWV, nearWD,
                       heavyOn);
    }
    if (heavyOn) expandHeavy<Mode>(P, L, outCol, outWk, wrSlot, nearWV, nearWD);
    // Local rounds: the CTA expands the near entries it has just staged
    // itself, up to P.localRounds times while its partitions are at most
    // half full, so a frontier advances several hops per grid barrier. An
    // entry expanded here is not flushed; the last round's appends are.
    // (Relaxations are monotone atomicMin, so expanding an entry earlier
    // than the next iteration would cannot change the fixed point.)
    const int rounds = narrow ? (blockIdx.x == 0 ? P.narrowRounds : 0) : P.localRounds;
    for (int r = 0; r < rounds; ++r) {
      __syncthreads();
      if (threadIdx.x == 0) {
        int tot = 0;
        bool room = true;
        for (int q = 0; q < K; ++q) {
          const int end = H.count[q] < H.cap ? H.count[q] : H.cap;
          H.roundEnd[q] = end;
          tot += end - H.start[q];
          room = room && H.count[q] <= H.cap / 2;
        }
        H.roundTotal = room ? tot : 0;
      }
      __syncthreads();
      const int tot = H.roundTotal;
      if (tot == 0) break;
      for (int b0 = warp * 32; b0 < tot; b0 += (blockDim.x >> 5) * 32) {
        const int j = b0 + static_cast<int>(lane);
        int kq = 0, uq = -1, begq = 0, degq = 0;
        u64 dq = 0;
        if (j < tot) {
          int rem = j;
          while (rem >= H.roundEnd[kq] - H.start[kq]) {
            rem -= H.roundEnd[kq] - H.start[kq];
            ++kq;
          }
          const StageEntry e = stageEntries()[kq * H.cap + H.start[kq] + rem];
          uq = e.v;
          dq = e.d;
          begq = ldGraph<Mode>(outRow + uq);
          degq = ldGraph<Mode>(outRow + uq + 1) - begq;
        }
        expandWarp<Mode>(P, L, outRow, outCol, outWk, kq, uq, dq, begq, degq, wrSlot, nearWV, nearWD,
                         heavyOn);
      }
      if (heavyOn) {
        expandHeavy<Mode>(P, L, outCol, outWk, wrSlot, nearWV, nearWD);
      } else {
        __syncthreads();
      }
      if (threadIdx.x < K) H.start[threadIdx.x] = H.roundEnd[threadIdx.x];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) tWorked = globalNs();
    __syncthreads();
    unsigned long long tAll = 0, tFlushed = 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) tAll = globalNs();
    flushStage(P, L, wrSlot, nearWV, nearWD);
    if (blockIdx.x == 0 && threadIdx.x == 0) tFlushed = globalNs();
    if (!gridSync(c, epoch)) return false;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      bool split = false;
      for (int k = 0; k < K; ++k) split |= L.mode[k] == kSplit;
      const unsigned long long tEnd = globalNs();
      profNs[split ? 0 : 1] += tEnd - itStart;
      profIters[split ? 0 : 1] += 1;
      profItems[split ? 0 : 1] += total;
      if (!split) {
        part[0] += tDecided - itStart;
        part[1] += tWorked - tDecided;
        part[2] += tAll - tWorked;
        part[3] += tFlushed - tAll;
        part[4] += tEnd - tFlushed;
      }
    }
  }

  if (threadIdx.x < K && H.expanded[threadIdx.x] != 0) {
    atomicAdd(reinterpret_cast<unsigned long long *>(&c->pushes[threadIdx.x]),
              static_cast<unsigned long long>(H.expanded[threadIdx.x]));
  }
  if (blockIdx.x == 0 && warp == 0 && static_cast<int>(lane) < K) {
    c->iterations[lane] = iters;
    c->epochs[lane] = epochs;
    if (lane == 0) {
      c->finalGen = genBase + 1 + it;
      *P.genPtr = genBase + 1 + it;
      for (int q = 0; q < 2; ++q) {
        c->loopNs[q] = profNs[q];
        c->loopIters[q] = profIters[q];
        c->loopItems[q] = profItems[q];
      }
      for (int q = 0; q < 5; ++q) c->iterSplitNs[q] = part[q];
    }
  }
  return true;
}

// ---------------------------------------------------------------------------
// Asynchronous near-far loop
//
// The bulk loop above pays a grid barrier per iteration and waits in every
// iteration for the slowest warp of the grid. Here a phase splits the far
// piles and expands the near entries with no barrier until the phase has run
// dry; only a new threshold per objective needs the grid to agree.
// Relaxations are the same monotone 64-bit atomicMin, so the fixed point,
// i.e. every word, is the one the bulk loop reaches.
//
// What bounds the loop is the number of hops of the deepest path times the
// latency of a hop, from the improvement of a vertex to the improvement of
// its neighbours (thin wavefronts: about 2,000 hops of a few hundred entries
// each on a grid road network of 500,000 vertices). So a hop stays inside
// one warp, or at least inside one CTA:
//
//   * a CTA takes an equal, contiguous share of the far piles. An entry
//     below the new threshold is expanded on the spot, the others go to the
//     warp's far buffer;
//   * a warp with few entries gives each a group of lanes and goes on with
//     what they improve, hop after hop (chase, chaseRecords). What is more
//     than it can hold goes by mail to a warp of the CTA that has nothing to
//     do (slots and an mbarrier of its own, on which it waits without
//     polling: 31 polling warps took half of the issue slots), or to the
//     CTA's ring of near entries in shared memory;
//   * with many entries, warps take up to 32 at a time from the ring and push
//     what improves back to it;
//   * a CTA whose ring holds more than kDonate entries while others have run
//     dry, or more than kRingSpill in any case, sends its pushes to a global
//     spill queue, from which dry CTAs claim up to 1,024 entries at a time. A
//     push that finds its shard full goes to the far pile.
//
// Row records (one 32-byte sector with a vertex's first four edges) make the
// loads of a hop one round trip to L2 that runs beside the atomicMin.
//
// Measured on a B200 against one grid-wide sharded queue with a claim, a slot
// and two counters per hop: a hop of a bare chain 0.59 us; tree from scratch
// of a 497,700-vertex road network 10.05 -> 2.33 ms, update of a million
// vertices with local detours (K = 3) 28.7 -> 7.6 ms, combined graph of
// 249,500 vertices (K = 6) 5.26 -> 1.25 ms, update of 2M vertices with
// long-range insertions (wide phases) 2.49 -> 2.17 ms; tree from scratch of 2M
// random vertices of degree 10 1.15 -> 1.05 ms, but the combined launch of such
// a graph (K = 3) 0.51 -> 0.78 ms.
//
// A vertex enters the far pile when an atomicMin takes it from infinity (or,
// in an update, from its tree distance) to a distance past the threshold;
// while its word stays past the threshold it is in the pile already, so the
// far append needs no flag.
//
// End of a phase: EngineControl::asyncPending counts the CTAs that still work
// on their share and the spilled entries that are not settled. A warp adds
// its finished entries to the CTA's `settled` count when it runs out of work,
// after its far buffer is flushed; the warp that makes the counts meet
// settles the CTA's share and its claimed entries with one atomic. The phase
// is over when asyncPending is zero, which an idle warp of every CTA polls.
// No grid barrier separates the phases: this counter and those of the far
// piles and the spill queue rotate through three slots, so a CTA that enters
// a phase early touches none that a late one reads.
// ---------------------------------------------------------------------------
constexpr unsigned long long kEmptySlot = ~0ULL;
constexpr unsigned kTagSat = 0xFFFFFFFEu;  // distances >= this are not carried in the entry
constexpr unsigned kOverflow = 0x80000000u;  // far-pile entry of an overflowed push
constexpr int kWarps = kThreads / 32;
constexpr unsigned kRingMask = kRing - 1;
// a push finds the ring at most this full, plus 128 entries of each of the
// other warps that passed the check at the same time, plus a claim
constexpr unsigned kRingSpill = kRing / 4;
// Ring entries above which a CTA feeds dry ones: kDonate in updates with row
// records, else kDonateLeast. Tree from scratch of random graphs, 500,000
// vertices of degree 6, 300,000 of 18, 100,000 of 66, us: 455, 627, 1103 with
// 512; 419, 522, 819 with 128; 441, 502, 638 with 64. Combined graph of 2M road
// vertices 650 with 512, 601 with 64. But their update with long-range changes
// is 3 % slower with 128 than with 512.
constexpr unsigned kDonate = 512;
constexpr unsigned kDonateLeast = 64;
constexpr unsigned kSliceFirst = 1024;  // ring entries above which the share waits
// entries claimed from the spill queue at a time (256: tree from scratch of 2M
// random vertices of degree 10 1.36 ms, 1,024 1.18), and read at a time
constexpr int kClaim = 1024;
constexpr int kFetch = 256;
// A claim of so many entries says that the phase is wide. In a graph without
// records the CTA's warps then take all they can carry and give each entry a
// lane, which keeps the order breadth-first (combined graph of 2M random
// vertices, 2.7 edges each: loop 661 -> 532 us; with records it makes road
// networks slower, update of 2M vertices 1135 -> 1174).
constexpr unsigned kBacklog = 64;
constexpr int kOctBatch = 4;         // entries of a batch that is expanded by octets of lanes
constexpr int kOctDeg = 32;          // longest row of such a batch
constexpr int kQuadBatch = 8;        // the same with row records (four lanes each)
constexpr int kChaseRing = 64;       // ring entries above which a warp keeps no entries of its own
// What a batch of the loop reads: the CSR; row records for few entries and the
// CSR for full batches; row records for all. An update's full batches read the
// CSR, those of a launch from scratch the records, whatever their size: loops
// of road networks with records and with the CSR in full batches, us:
//   update, long-range changes (wide phases), 5, 28, 95 and 180 MB of records:
//     K = 1 332/310, 555/506, 980/818, 1385/1110; K = 3 286/283, 539/485,
//     880/735; 64 networks, K = 3, 117 MB 1102/957
//   update, short detours (narrow phases), 5, 28, 95 MB: K = 3 706/703,
//     2390/2363, 5105/5056
//   combined graph, 3, 30, 100 and 180 MB: wide 310/340, 411/443, 535/549,
//     663/669; narrow 633/636, 1505/1510, 4659/4674, 6026/6050
//   tree from scratch, 3, 15, 60, 176 MB: 925/922, 2282/2290, 5104/5111,
//     9732/9750
enum : int { kCsrOnly = 0, kThinRecords = 1, kRecords = 2 };
// The records are used where at most one row in kLongRows is longer than one:
// a batch with such a row has loaded its records for nothing. Tree from
// scratch and update with short changes, 302,500 vertices, with records and
// without, us: grids, 0.5% of the rows longer 1702/2268, 3661/4830; random
// graphs, 0% 657/783, 1832/2097; 4.7% 822/689, 1525/1437; 17% 880/683,
// 1433/1222.
constexpr long long kLongRows = 50;
constexpr unsigned kThinShare = 64;  // far-pile entries per CTA up to which a phase is wider
constexpr unsigned kSpinLimit = 1u << 24;
#ifndef MOSP_EDGE_SLOTS_ASYNC
#define MOSP_EDGE_SLOTS_ASYNC 3
#endif
// three slots per lane cover the ~90 edges of 32 road vertices in one pass
constexpr int kSlotsAsync = MOSP_EDGE_SLOTS_ASYNC;
static_assert(kRingSpill + kWarps * 128 + kClaim <= kRing, "ring reservations fit");
static_assert(kMail == kQuadBatch, "a mail is a batch");

/// What an expansion needs of its objective.
struct alignas(16) AsyncObj {
  u64 *packed;
  const int4 *rec;   // row records (two int4 per vertex) or null
  u64 thrWord;       // words below it have a distance below the threshold
  u64 mostWord;      // the largest word of a distance within the bound
  unsigned scale;    // 1 << bits
  unsigned mask;     // the word's parent field: the low `bits` bits
  int bits;
  int pad;
  const int *outW;
  const long long *dist;  // update: the distances of the input tree
  u64 thr;
  u64 prev;          // the last phase's threshold
};

/// An entry on its way from lane to lane: a head, the word it took and its
/// row record.
struct alignas(16) HopSlot {
  u64 word;
  int v, k;
  int4 cols, wts;
};

/// A CTA's state of the asynchronous loop (shared memory). head and tail are
/// the ring's positions, cur the entries taken of the CTA's share of the far
/// piles, mailed the entries sent by mail, settled the finished entries of
/// all three; dry when settled == tail + mailed + share. lock guards the
/// change between busy and dry.
struct AsyncCta {
  unsigned head, tail, cur, settled;
  unsigned share;    // entries of the CTA's share of this phase
  unsigned owed;     // entries claimed from the spill queue (and the phase's own share: 1)
  unsigned mailed;
  unsigned idle;     // warps that wait for mail
  int dry;
  int lock;
  int over;          // the phase is over
  int full;          // the last claim found a backlog (kBacklog)
  int abort;         // the launch stops
  long long base;    // first far-pile index of the share
  // statistics: rounds, those of a phase from the CTA's first claim of spilled
  // entries on (fed; at round fedFrom), entries
  int fed;
  unsigned rounds, fedRounds, fedFrom, items, taken;
  unsigned expanded[kMaxK];
  int mail[kWarps];  // entries in a warp's mail
  u64 bar[kWarps];   // its mbarrier
  int K;
  unsigned donateAt;  // ring entries above which the CTA feeds dry ones
  unsigned phase;
  unsigned long long deadline;
  AsyncObj obj[kMaxK];
  LoopShared L;
  HopSlot hop[kWarps][kQuadBatch];   // a warp's entries of the next hop
  HopSlot mailbox[kWarps][kMail];
};
static_assert(sizeof(AsyncCta) <= kAsyncCtaBytes, "kAsyncCtaBytes");

__device__ __forceinline__ u64 *asyncRing() { return reinterpret_cast<u64 *>(stageEntries()); }

/// The warp's buffer of far appends (distance << 32 | v << 5 | k).
__device__ __forceinline__ u64 *asyncFarBuffer() {
  return asyncRing() + kRing + (threadIdx.x >> 5) * kFarBuf;
}

/// The CTA's state, after the far buffers in the dynamic shared memory.
__device__ __forceinline__ AsyncCta &asyncCta() {
  return *reinterpret_cast<AsyncCta *>(asyncRing() + kRing + kWarps * kFarBuf);
}

__device__ __forceinline__ unsigned ldShared(const unsigned *p) {
  return *reinterpret_cast<const volatile unsigned *>(p);
}
__device__ __forceinline__ int ldShared(const int *p) {
  return *reinterpret_cast<const volatile int *>(p);
}
__device__ __forceinline__ u64 ldShared(const u64 *p) {
  return *reinterpret_cast<const volatile u64 *>(p);
}
__device__ __forceinline__ void stShared(u64 *p, u64 v) { *reinterpret_cast<volatile u64 *>(p) = v; }
__device__ __forceinline__ void stShared(int *p, int v) { *reinterpret_cast<volatile int *>(p) = v; }

__device__ __forceinline__ void barInit(u64 *bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(bar)))
               : "memory");
}

/// One arrival completes the phase the warp waits for (release: the mail).
__device__ __forceinline__ void barArrive(u64 *bar) {
  asm volatile("{ .reg .b64 s; mbarrier.arrive.release.cta.shared::cta.b64 s, [%0]; }" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(bar)))
               : "memory");
}

/// Waits for the phase of parity `parity` for a few microseconds at most.
__device__ __forceinline__ bool barTryWait(u64 *bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{ .reg .pred p; mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2, %3; "
      "selp.u32 %0, 1, 0, p; }"
      : "=r"(done)
      : "r"(static_cast<unsigned>(__cvta_generic_to_shared(bar))), "r"(parity), "r"(4000u)
      : "memory");
  return done != 0;
}

/// A bounded wait ran out (or the deadline passed): the launch stops.
__device__ __noinline__ void asyncAbort(const EngineParams &P) {
  AsyncCta &C = asyncCta();
  atomicCAS(&P.ctl->status, 0, MOSP_ERR_TIMEOUT);
  stShared(&C.abort, 1);
}

/// Whether the launch has to stop (a warp with work looks now and then, so
/// that a run ends by its deadline whether it stalls or keeps iterating).
/// All lanes call it.
__device__ __noinline__ bool asyncStop(const EngineParams &P) {
  AsyncCta &C = asyncCta();
  int stop = 0;
  if (laneId() == 0) {
    stop = ldShared(&C.abort);
    if (stop == 0 && (ldVolatile(&P.ctl->status) != 0 || globalNs() > C.deadline)) {
      asyncAbort(P);
      stop = 1;
    }
  }
  return __shfl_sync(kFull, stop, 0) != 0;
}

/// Takes an idle warp out of the idle set (lane 0): its number or -1.
__device__ __forceinline__ int takeIdle() {
  AsyncCta &C = asyncCta();
  unsigned m = ldShared(&C.idle);
  while (m != 0) {
    const int w = __ffs(m) - 1;
    m = atomicAnd(&C.idle, ~(1u << w));
    if ((m >> w) & 1u) return w;
  }
  return -1;
}

/// Sends up to `count` idle warps to the ring (lane 0).
__device__ __noinline__ void wakeIdle(int count) {
  AsyncCta &C = asyncCta();
  const unsigned idle = ldShared(&C.idle);
  unsigned rest = idle;
  for (; count > 0; --count) rest &= rest - 1u;
  unsigned wake = idle ^ rest;
  // (one that is no longer idle has been sent elsewhere and looks here next)
  if (wake != 0) wake &= atomicAnd(&C.idle, ~wake);
  for (; wake != 0; wake &= wake - 1u) {
    const int w = __ffs(wake) - 1;
    C.mail[w] = 0;
    barArrive(&C.bar[w]);
  }
}

/// Wakes every idle warp, a lane per warp. All lanes call it.
__device__ __forceinline__ void wakeAll() {
  AsyncCta &C = asyncCta();
  const unsigned lane = laneId();
  unsigned m = 0;
  if (lane == 0) m = atomicExch(&C.idle, 0u);
  m = __shfl_sync(kFull, m, 0);
  if ((m >> lane) & 1u) {
    C.mail[lane] = 0;
    barArrive(&C.bar[lane]);
  }
  __syncwarp();
}

/// The warp's far buffer to the piles: one reservation per objective and 32
/// entries, the pile minimum into the CTA's. All lanes call it.
__device__ __noinline__ void flushFarEntries(const EngineParams &P, int count) {
  const LoopShared &L = asyncCta().L;
  StageHeader &H = stageHeader();
  const int lane = static_cast<int>(laneId());
  const u64 *buf = asyncFarBuffer();
  __syncwarp();
#pragma unroll 1
  for (int i0 = 0; i0 < count; i0 += 32) {
    const bool have = i0 + lane < count;
    const u64 e = have ? buf[i0 + lane] : 0;
    const int k = have ? static_cast<int>(e & 31u) : -1;
    const unsigned peers = __match_any_sync(kFull, k);
    const unsigned least = __reduce_min_sync(peers, static_cast<unsigned>(e >> 32));
    const int leader = __ffs(peers) - 1;
    const Target t = listTarget(P, L, P.K + (k < 0 ? 0 : k), 0, nullptr, nullptr);
    int at = 0;
    if (have && lane == leader) {
      // (a distance that does not fit the tag went to the minimum on its own)
      if (least < kTagSat) atomicMin(&H.farMin[k], static_cast<u64>(least));
      at = atomicAdd(t.counter, __popc(peers));
    }
    at = __shfl_sync(kFull, at, leader);
    if (have) t.v[at + __popc(peers & ((1u << lane) - 1u))] = static_cast<int>(static_cast<unsigned>(e) >> 5);
  }
  __syncwarp();
}

/// Append (w, d) of objective k to the warp's far buffer in the lanes with
/// `want`; flushes first when the buffer could overflow. All lanes call it.
__device__ __forceinline__ void farAppend(const EngineParams &P, int &farCount, bool want, int k, int w,
                                          u64 d) {
  const unsigned mask = __ballot_sync(kFull, want);
  if (mask == 0) return;
  if (farCount > kFarBuf - 32) {
    flushFarEntries(P, farCount);
    farCount = 0;
  }
  if (want) {
    const unsigned tag = d < kTagSat ? static_cast<unsigned>(d) : kTagSat;
    if (tag == kTagSat) atomicMin(&stageHeader().farMin[k], d);
    asyncFarBuffer()[farCount + __popc(mask & ((1u << laneId()) - 1u))] =
        (static_cast<u64>(tag) << 32) | ((static_cast<unsigned>(w) << 5) | static_cast<unsigned>(k));
  }
  farCount += __popc(mask);
}

/// Whether a vertex x whose word went from `old` to a distance past the
/// threshold is not in the far pile yet: it comes from infinity or, in an
/// update, from the distance of its input tree.
template <int Mode>
__device__ __forceinline__ bool newInFar(const AsyncObj &O, u64 old, int x) {
  if (old == kInfWord) return true;
  if constexpr (Mode == kModeUpdate) {
    return __ldcg(O.dist + x) == static_cast<long long>(old >> O.bits);
  } else {
    return false;
  }
}

/// Room for `count` near entries of the warp in the spill queue: counted in
/// asyncPending before their slots can be claimed (the reservation releases
/// the count). The shard, and the first entry's position in it, which may lie
/// past its capacity (spillWrite). All lanes call it.
__device__ __noinline__ unsigned spillReserve(const EngineParams &P, int count, int &shard) {
  AsyncCta &C = asyncCta();
  // the shards take turns, a different one for each CTA
  const int s = static_cast<int>((blockIdx.x * 5u + (threadIdx.x >> 5) + (ldShared(&C.settled) >> 5)) %
                                 static_cast<unsigned>(P.aqShards));
  const int target = __shfl_sync(kFull, s, 0);
  unsigned base = 0;
  if (laneId() == 0) {
    atomicAdd(&P.ctl->asyncPending[C.phase % 3], static_cast<unsigned>(count));
    AsyncShard *A = P.aqCtr + C.phase % 3 * P.aqShards + target;
    asm volatile("atom.add.release.gpu.global.u32 %0, [%1], %2;" : "=r"(base) : "l"(&A->reserved), "r"(count) : "memory");
    // the ones past the capacity are not queued
    const unsigned end = base + static_cast<unsigned>(count);
    if (end > P.aqShardCap) {
      atomicSub(&P.ctl->asyncPending[C.phase % 3], end - (base > P.aqShardCap ? base : P.aqShardCap));
    }
  }
  shard = target;
  return __shfl_sync(kFull, base, 0);
}

/// A near entry to its reserved place. Past the shard's capacity its vertex
/// goes to the far pile, once (by its flag), marked so that the split expands
/// it.
__device__ __forceinline__ void spillWrite(const EngineParams &P, int shard, unsigned idx, u64 entry) {
  if (idx < P.aqShardCap) {
    if (static_cast<unsigned>(entry >> 32) == kTagSat) __threadfence();  // the word before the entry
    stRelaxed64(P.aqSlots + static_cast<long long>(shard) * P.aqShardCap + idx, entry);
    return;
  }
  const int k = static_cast<int>(entry & 31u);
  const int v = static_cast<int>(static_cast<unsigned>(entry) >> 5);
  __threadfence();  // the word before the flag
  if (atomicExch(P.inFar + static_cast<long long>(k) * P.stride + v, 1) == 0) {
    const Target t = listTarget(P, asyncCta().L, P.K + k, 0, nullptr, nullptr);
    t.v[atomicAdd(t.counter, 1)] = static_cast<int>(static_cast<unsigned>(v) | kOverflow);
  }
}

/// Near entries of the lanes in `mask` to the spill queue. All lanes call it.
__device__ __noinline__ void spillNear(const EngineParams &P, unsigned mask, u64 entry) {
  int shard;
  const unsigned at = spillReserve(P, __popc(mask), shard);
  if ((mask >> laneId()) & 1u) spillWrite(P, shard, at + __popc(mask & ((1u << laneId()) - 1u)), entry);
}

/// Write an entry to a reserved ring slot. The slot is empty unless the warp
/// that claimed its last entry has not read it yet.
__device__ __forceinline__ void ringWrite(const EngineParams &P, unsigned pos, u64 entry) {
  AsyncCta &C = asyncCta();
  u64 *slot = asyncRing() + (pos & kRingMask);
  unsigned spin = 0;
  while (ldShared(slot) != kEmptySlot) {
    if (++spin > kSpinLimit || ((spin & 1023u) == 0 && ldShared(&C.abort) != 0)) {
      asyncAbort(P);
      break;
    }
  }
  if (static_cast<unsigned>(entry >> 32) == kTagSat) __threadfence();  // the word before the entry
  stShared(slot, entry);
}

/// Room in the ring for `count` entries (lane 0): reserved at `at`, or false
/// when the CTA spills.
__device__ __forceinline__ bool ringReserve(bool donate, int count, unsigned &at) {
  AsyncCta &C = asyncCta();
  const unsigned held = ldShared(&C.tail) - ldShared(&C.head);
  if (held > kRingSpill || (donate && held > C.donateAt)) return false;
  at = atomicAdd(&C.tail, static_cast<unsigned>(count));
  __threadfence_block();  // the entries before the look at the idle warps
  if (ldShared(&C.idle) != 0) wakeIdle(1 + (count >> 3));
  return true;
}

/// Near entries of N edges per lane (ballot[h]: the lanes whose edge h has one)
/// to the CTA's ring or the spill queue, one reservation for the warp. All
/// lanes call it.
template <int N>
__device__ __forceinline__ void nearPush(const EngineParams &P, const unsigned (&ballot)[N], bool donate,
                                         const u64 (&entry)[N]) {
  const unsigned lane = laneId();
  int count = 0;
#pragma unroll
  for (int h = 0; h < N; ++h) count += __popc(ballot[h]);
  if (count == 0) return;
  unsigned at = 0;
  int room = 0, shard = 0;
  if (lane == 0) room = ringReserve(donate, count, at);
  room = __shfl_sync(kFull, room, 0);
  at = room ? __shfl_sync(kFull, at, 0) : spillReserve(P, count, shard);
#pragma unroll
  for (int h = 0; h < N; ++h) {
    if ((ballot[h] >> lane) & 1u) {
      const unsigned idx = at + __popc(ballot[h] & ((1u << lane) - 1u));
      if (room) {
        ringWrite(P, idx, entry[h]);
      } else {
        spillWrite(P, shard, idx, entry[h]);
      }
    }
    at += __popc(ballot[h]);
  }
}

/// The same for one edge per lane. (The way to the queue is a function of its
/// own, which keeps the registers of this one few.)
__device__ __noinline__ void ringPush(const EngineParams &P, unsigned mask, bool donate, u64 entry) {
  const unsigned lane = laneId();
  unsigned at = 0;
  int room = 0;
  if (lane == 0) room = ringReserve(donate, __popc(mask), at);
  room = __shfl_sync(kFull, room, 0);
  at = __shfl_sync(kFull, at, 0);
  if (!room) {
    spillNear(P, mask, entry);
  } else if ((mask >> lane) & 1u) {
    ringWrite(P, at + __popc(mask & ((1u << lane) - 1u)), entry);
  }
}

__device__ __forceinline__ u64 nearEntry(int k, int w, u64 d) {
  const unsigned tag = d < kTagSat ? static_cast<unsigned>(d) : kTagSat;
  return (static_cast<u64>(tag) << 32) | ((static_cast<unsigned>(w) << 5) | static_cast<unsigned>(k));
}

/// The offer of edge weight w by v at distance d is offerBase + w * scale,
/// with v in the parent field (runNearFar sees to it that a distance within
/// the bound plus any weight fits the word).
__device__ __forceinline__ u64 offerBase(const AsyncObj &O, u64 d, int v) {
  return O.bits == 0 ? d : (d << O.bits) | static_cast<u64>(static_cast<unsigned>(v));
}

/// The offer base of a head x that took word `word`.
__device__ __forceinline__ u64 nextBase(u64 word, int x, unsigned mask) {
  const unsigned lo = (static_cast<unsigned>(word) & ~mask) | (static_cast<unsigned>(x) & mask);
  return (word & 0xffffffff00000000ULL) | lo;
}

/// Improvements of one edge per lane (x of objective k from word `old` to
/// cw): near ones to the ring, new far ones to the far buffer. All lanes.
template <int Mode>
__device__ __forceinline__ void pushEdges(const EngineParams &P, const AsyncObj &O, bool donate,
                                          int &farCount, int k, int x, u64 cw, u64 old) {
  const bool imp = old > (cw | O.mask);
  const bool near = imp && cw < O.thrWord;
  const unsigned mask = __ballot_sync(kFull, near);
  if (mask != 0) ringPush(P, mask, donate, nearEntry(k, x, cw >> O.bits));
  const bool far = imp && !near && newInFar<Mode>(O, old, x);
  farAppend(P, farCount, far, k, x, cw >> O.bits);
}

/// Lane 0 of the warp that settled the CTA's last entry: if the CTA is still
/// dry under the lock (the fetching warp may have brought new entries),
/// settle its share and claimed entries.
__device__ __noinline__ void asyncDry(const EngineParams &P, unsigned phase) {
  AsyncCta &C = asyncCta();
  const LoopShared &L = C.L;
  EngineControl *c = P.ctl;
  StageHeader &H = stageHeader();
  unsigned spin = 0;
  while (atomicCAS(&C.lock, 0, 1) != 0) {
    if (++spin > kSpinLimit || ((spin & 1023u) == 0 && ldShared(&C.abort) != 0)) {
      asyncAbort(P);
      return;
    }
  }
  __threadfence_block();
  if (C.dry == 0 && ldShared(&C.settled) == ldShared(&C.tail) + ldShared(&C.mailed) + C.share) {
#pragma unroll 1
    for (int k = 0; k < P.K; ++k) {
      if (H.farMin[k] != kInfWord) {
        atomicMax(listTarget(P, L, P.K + k, 0, nullptr, nullptr).minC, ~H.farMin[k]);
        H.farMin[k] = kInfWord;
      }
    }
    C.dry = 1;
    const unsigned done = C.owed;
    C.owed = 0;
    atomicAdd(&c->asyncHungry[phase % 3], 1);
    // release: what the CTA's warps wrote; acquire-free, the others poll
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(&c->asyncPending[phase % 3]),
                 "r"(0u - done)
                 : "memory");
  }
  __threadfence_block();
  atomicExch(&C.lock, 0);
}

/// The idle turn of warp 0: the end of the phase, or entries of the spill
/// queue for the CTA's ring. All lanes call it.
__device__ __noinline__ void asyncFetch(const EngineParams &P, unsigned phase) {
  AsyncCta &C = asyncCta();
  EngineControl *c = P.ctl;
  const int lane = static_cast<int>(laneId());
  const int S = P.aqShards;
  unsigned left = 1;
  unsigned head = 0, tail = 0;
  AsyncShard *shards = P.aqCtr + phase % 3 * S;
  // (relaxed polls: an acquire would empty L1 at every turn)
  if (lane < S) ldPair(&shards[lane].claimed, head, tail);
  if (lane == 31) left = *reinterpret_cast<volatile unsigned *>(&c->asyncPending[phase % 3]);
  if (__shfl_sync(kFull, left, 31) == 0) {
    if (lane == 0) {
      __threadfence();
      stShared(&C.over, 1);
      __threadfence_block();  // over before the look at the idle warps
    }
    __syncwarp();
    wakeAll();
    return;
  }
  const unsigned cap = P.aqShardCap;
  if (tail > cap) tail = cap;
  const unsigned have = __ballot_sync(kFull, lane < S && tail > head);
  if (have == 0) return;
  // the first shard with entries from this CTA's own on
  const unsigned own = blockIdx.x % S;
  const unsigned later = have >> own << own;
  const int s = __ffs(later != 0 ? later : have) - 1;
  head = __shfl_sync(kFull, head, s);
  tail = __shfl_sync(kFull, tail, s);
  const unsigned n = tail - head < kClaim ? tail - head : kClaim;
  unsigned r0 = 0;
  int got = 0;
  if (lane == 0 && atomicCAS(&C.lock, 0, 1) == 0) {
    __threadfence_block();
    if (ldShared(&C.tail) - ldShared(&C.head) <= kDonate &&
        atomicCAS(&shards[s].claimed, head, head + n) == head) {
      __threadfence();  // acquire: the producers' counts and slots
      C.owed += n;
      C.full = n >= kBacklog;
      C.taken += n;
      if (C.fed == 0) {
        C.fed = 1;
        C.fedFrom = ldShared(&C.rounds);
      }
      r0 = atomicAdd(&C.tail, n);
      if (C.dry != 0) {
        C.dry = 0;
        atomicSub(&c->asyncHungry[phase % 3], 1);
      }
      got = 1;
    }
    __threadfence_block();
    atomicExch(&C.lock, 0);
  }
  if (__shfl_sync(kFull, got, 0) == 0) return;
  r0 = __shfl_sync(kFull, r0, 0);
  u64 *slots = P.aqSlots + static_cast<long long>(s) * cap + head;
  for (unsigned j0 = 0; j0 < n; j0 += kFetch) {
    u64 e[kFetch / 32];
#pragma unroll
    for (int i = 0; i < kFetch / 32; ++i) {
      const unsigned j = j0 + static_cast<unsigned>(i * 32 + lane);
      e[i] = j < n ? ldRelaxed64(slots + j) : 0;
    }
#pragma unroll
    for (int i = 0; i < kFetch / 32; ++i) {
      const unsigned j = j0 + static_cast<unsigned>(i * 32 + lane);
      if (j >= n) continue;
      // the producer reserved the slot and is about to write it
      for (unsigned spin = 0; e[i] == kEmptySlot; e[i] = ldRelaxed64(slots + j)) {
        if (++spin > (kSpinLimit >> 4) || ((spin & 1023u) == 0 && ldShared(&C.abort) != 0)) {
          asyncAbort(P);
          break;
        }
      }
      stRelaxed64(slots + j, kEmptySlot);
      ringWrite(P, r0 + j, e[i]);
    }
  }
  __syncwarp();
  if (n > 128) {
    wakeAll();
  } else if (lane == 0) {
    wakeIdle(static_cast<int>(n >> 3));
  }
}

/// Graph loads of the asynchronous loop. The combined mode's graph was
/// written earlier in the same launch and is read-only since the last grid
/// barrier, so plain loads may keep it in L1.
template <int Mode>
__device__ __forceinline__ int ldLoop(const int *p) {
  if constexpr (Mode == kModeCombined) {
    return *p;
  } else {
    return __ldg(p);
  }
}

/// Graphs without row records, thin wavefronts: up to four entries (one per
/// octet of lanes; rows of at most kOctDeg edges, beg == end for none),
/// expanded hop after hop by the same warp for as long as they improve
/// something below the threshold. The row pointers of the heads are loaded
/// while the atomicMin is on its way.
template <int Mode>
__device__ __forceinline__ void chase(const EngineParams &P, const int *outRow, const int *outCol,
                                      bool donate, int &farCount, int k, int v, u64 du, int beg, int end) {
  AsyncCta &C = asyncCta();
  const unsigned lane = laneId();
  u64 base = offerBase(C.obj[k], du, v);
  for (unsigned hops = 1;; ++hops) {
    if ((hops & 4095u) == 0 && asyncStop(P)) return;
    const AsyncObj &O = C.obj[k];
    int e = beg + static_cast<int>(lane & 7u);
    int x, rb = 0, re = 0;
    u64 cw, old;
    while (true) {
      const bool in = e < end;
      x = in ? ldLoop<Mode>(outCol + e) : P.source;
      cw = base + static_cast<u64>(static_cast<unsigned>(in ? ldLoop<Mode>(O.outW + e) : 0)) * O.scale;
      old = 0;
      if (x != P.source && cw <= O.mostWord) {
        old = atomicMin(O.packed + x, cw);
        rb = ldLoop<Mode>(outRow + x);
        re = ldLoop<Mode>(outRow + x + 1);
      }
      e += 8;
      if (!__any_sync(kFull, e < end)) break;
      pushEdges<Mode>(P, O, donate, farCount, k, x, cw, old);
    }
    const bool imp = old > (cw | O.mask);
    const bool near = imp && cw < O.thrWord;
    const unsigned nearMask = __ballot_sync(kFull, near);
    farAppend(P, farCount, imp && !near && newInFar<Mode>(O, old, x), k, x, cw >> O.bits);
    if (nearMask == 0) return;
    unsigned keep = __ballot_sync(kFull, near && re - rb <= kOctDeg);
    if (keep != nearMask || __popc(keep) > kOctBatch) {
      // a CTA with work for all its warps keeps the breadth-first order
      const int busy =
          __shfl_sync(kFull, static_cast<int>(ldShared(&C.tail) - ldShared(&C.head)), 0) > kChaseRing;
      const bool mine = (keep >> lane) & 1u;
      const bool give = near && (busy || !mine || __popc(keep & ((1u << lane) - 1u)) >= kOctBatch);
      const unsigned mask = __ballot_sync(kFull, give);
      if (mask != 0) ringPush(P, mask, donate, nearEntry(k, x, cw >> O.bits));
      if (busy) return;
    }
    // octet q goes on with the q-th of them
    HopSlot *slots = C.hop[threadIdx.x >> 5];
    const int rank = __popc(keep & ((1u << lane) - 1u));
    const int count = __popc(keep);
    if (((keep >> lane) & 1u) && rank < kOctBatch) {
      slots[rank].word = cw;
      slots[rank].v = x;
      slots[rank].k = k;
    }
    const int src = rank < kOctBatch && ((keep >> lane) & 1u) ? rank : -1;
    __syncwarp();
    const int q = static_cast<int>(lane >> 3);
    const bool on = q < count;
    // the row of the q-th comes from the lane that loaded it
    int from = 0;
#pragma unroll
    for (int i = 0; i < kOctBatch; ++i) {
      const unsigned who = __ballot_sync(kFull, src == i);
      if (i == q && who != 0) from = __ffs(who) - 1;
    }
    beg = __shfl_sync(kFull, rb, from);
    end = __shfl_sync(kFull, re, from);
    if (on) {
      v = slots[q].v;
      k = slots[q].k;
      base = nextBase(slots[q].word, v, C.obj[k].mask);
      if ((lane & 7u) == 0) atomicAdd(&C.expanded[k], 1u);
    } else {
      end = beg;
    }
    __syncwarp();
  }
}

/// The rows of the lanes' entries (this lane's: edges [beg, end) of v at
/// distance du in objective k; beg == end for none) as one flat range of
/// edges, three per lane and turn. All lanes call it.
template <int Mode>
__device__ __forceinline__ void expandRows(const EngineParams &P, const int *outCol, bool donate,
                                           int &farCount, int k, int v, u64 du, int beg, int end) {
  AsyncCta &C = asyncCta();
  const unsigned lane = laneId();
  const u64 base = offerBase(C.obj[k], du, v);
  int deg = end - beg;
  // a row of more than 2^20 edges goes to the whole warp by itself
  unsigned huge = __ballot_sync(kFull, deg > (1 << 20));
  while (huge != 0) {
    const int src = __ffs(huge) - 1;
    huge &= huge - 1;
    const int kb = __shfl_sync(kFull, k, src);
    const u64 ob = __shfl_sync(kFull, base, src);
    const int bb = __shfl_sync(kFull, beg, src);
    const int eb = __shfl_sync(kFull, end, src);
    const AsyncObj &O = C.obj[kb];
    for (int e0 = bb; e0 < eb; e0 += 32) {
      const int e = e0 + static_cast<int>(lane);
      const int x = e < eb ? ldLoop<Mode>(outCol + e) : P.source;
      const u64 cw =
          ob + static_cast<u64>(static_cast<unsigned>(e < eb ? ldLoop<Mode>(O.outW + e) : 0)) * O.scale;
      const u64 old = x != P.source && cw <= O.mostWord ? atomicMin(O.packed + x, cw) : 0;
      pushEdges<Mode>(P, O, donate, farCount, kb, x, cw, old);
    }
  }
  if (deg > (1 << 20)) deg = 0;
  int incl = deg;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int o = __shfl_up_sync(kFull, incl, off);
    if (static_cast<int>(lane) >= off) incl += o;
  }
  const int edges = __shfl_sync(kFull, incl, 31);
  const int first = beg - (incl - deg);
  constexpr int SL = kSlotsAsync;
  for (int s0 = 0; s0 < edges; s0 += 32 * SL) {
    int kk[SL], ww[SL];
    u64 cw[SL], old[SL];
#pragma unroll
    for (int h = 0; h < SL; ++h) {
      const int sl = s0 + 32 * h + static_cast<int>(lane);
      const int o = slotOwner(incl, sl);
      kk[h] = __shfl_sync(kFull, k, o);
      cw[h] = __shfl_sync(kFull, base, o);
      const int e = __shfl_sync(kFull, first, o) + sl;
      ww[h] = P.source;
      if (sl < edges) {
        const AsyncObj &O = C.obj[kk[h]];
        ww[h] = ldLoop<Mode>(outCol + e);
        cw[h] += static_cast<u64>(static_cast<unsigned>(ldLoop<Mode>(O.outW + e))) * O.scale;
      }
    }
#pragma unroll
    for (int h = 0; h < SL; ++h) {
      const AsyncObj &O = C.obj[kk[h]];
      old[h] = ww[h] != P.source && cw[h] <= O.mostWord ? atomicMin(O.packed + ww[h], cw[h]) : 0;
    }
#pragma unroll
    for (int h = 0; h < SL; ++h) pushEdges<Mode>(P, C.obj[kk[h]], donate, farCount, kk[h], ww[h], cw[h], old[h]);
  }
}

/// Thin wavefronts of a graph with row records: up to eight entries, four
/// lanes each (lane sub of the quad takes the record's edge sub), expanded
/// hop after hop by the same warp for as long as they improve something
/// below the threshold. The record of a head is requested before its
/// atomicMin, so a hop is one round trip to L2 and a short run of
/// instructions (a lone warp issues them one after another, so they count
/// as much as the round trip): words are compared without unpacking them,
/// and the next hop's entries pass through slots in shared memory. More than
/// eight go to an idle warp by mail, or to the ring.
template <int Mode>
__device__ __noinline__ int chaseRecords(const EngineParams &P, bool donate, int farCount, int k, int v,
                                         u64 base, int x, int t) {
  AsyncCta &C = asyncCta();
  const unsigned lane = laneId();
  const int sub = static_cast<int>(lane & 3u);
  const int q = static_cast<int>(lane >> 2);
  HopSlot *slots = C.hop[threadIdx.x >> 5];
  const AsyncObj *O = &C.obj[k];
  u64 *packed = O->packed;
  const int4 *rec = O->rec;
  u64 thrWord = O->thrWord, mostWord = O->mostWord;
  unsigned scale = O->scale, mask = O->mask;
  const bool oneK = Mode != kModeUpdate || C.K == 1;
  // expansions, counted here where there is one objective: an atomicAdd to
  // shared memory per hop costs 70 ns of it on a bare chain
  unsigned done = 0;
  for (unsigned hops = 1;; ++hops) {
    // (one verdict for the warp: lanes may read the clock and the flag
    // differently, and one that left alone would keep the others waiting at
    // the next ballot)
    if ((hops & 4095u) == 0 && __any_sync(kFull, ldShared(&C.abort) != 0 || globalNs() > C.deadline)) {
      atomicCAS(&P.ctl->status, 0, MOSP_ERR_TIMEOUT);
      stShared(&C.abort, 1);
      break;
    }
    const u64 cw = static_cast<u64>(static_cast<unsigned>(t)) * scale + base;
    u64 old = 0;
    int4 cols, wts;
    if (x >= 0 && cw <= mostWord) {
      // (volatile, so that they are requested before the atomicMin)
      asm volatile("ld.global.v4.s32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(cols.x), "=r"(cols.y), "=r"(cols.z), "=r"(cols.w)
                   : "l"(rec + 2LL * x));
      asm volatile("ld.global.v4.s32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(wts.x), "=r"(wts.y), "=r"(wts.z), "=r"(wts.w)
                   : "l"(rec + 2LL * x + 1));
      old = atomicMin(packed + x, cw);
    }
    const bool imp = old > (cw | mask);
    const bool near = imp && cw < thrWord;
    // a head whose row is longer than its record goes to the ring, for a batch
    // by rows: its quad would load the rest of a long row one edge after
    // another (R-MAT graph of 4,547 vertices, rows up to 2,000 edges: 885 ->
    // 338 us per update)
    const bool more = near && cols.w == kMoreEdges;
    const unsigned keep = __ballot_sync(kFull, near && !more);
    // (the update has something for the far pile in most hops: one ballot less)
    if (Mode == kModeUpdate || __any_sync(kFull, imp && (more || !near))) {
      const unsigned longer = __ballot_sync(kFull, more);
      if (longer != 0) ringPush(P, longer, donate, nearEntry(k, x, cw >> O->bits));
      farAppend(P, farCount, imp && !near && newInFar<Mode>(*O, old, x), k, x, cw >> O->bits);
    }
    if (keep == 0) break;
    const int count = __popc(keep);
    const int rank = __popc(keep & ((1u << lane) - 1u));
    if (count > kQuadBatch) {
      // the next eight by mail to an idle warp
      int w = -1, busy = 0;
      if (lane == 0) {
        w = takeIdle();
        busy = w < 0 && ldShared(&C.tail) - ldShared(&C.head) > kChaseRing;
      }
      w = __shfl_sync(kFull, w, 0);
      busy = __shfl_sync(kFull, busy, 0);
      int kept = kQuadBatch;
      if (w >= 0) {
        if (near && !more && rank >= kQuadBatch && rank < 2 * kQuadBatch) {
          C.mailbox[w][rank - kQuadBatch] = HopSlot{cw, x, k, cols, wts};
        }
        __syncwarp();
        if (lane == 0) {
          const int sent = count - kQuadBatch < kMail ? count - kQuadBatch : kMail;
          atomicAdd(&C.mailed, static_cast<unsigned>(sent));
          C.mail[w] = sent;
          barArrive(&C.bar[w]);
        }
        kept = 2 * kQuadBatch;
      }
      // a CTA with work for all its warps keeps the breadth-first order
      const unsigned give = __ballot_sync(kFull, near && !more && (busy || rank >= kept));
      if (give != 0) ringPush(P, give, donate, nearEntry(k, x, cw >> O->bits));
      if (busy) break;
    }
    // quad q goes on with the q-th of them
    if (near && !more && rank < kQuadBatch) slots[rank] = HopSlot{cw, x, k, cols, wts};
    __syncwarp();
    x = -1;
    if (Mode != kModeUpdate) done += count < kQuadBatch ? count : kQuadBatch;
    if (q < count) {
      const HopSlot &h = slots[q];
      v = h.v;
      if (!oneK) {
        k = h.k;
        O = &C.obj[k];
        packed = O->packed;
        rec = O->rec;
        thrWord = O->thrWord;
        mostWord = O->mostWord;
        scale = O->scale;
        mask = O->mask;
      }
      x = reinterpret_cast<const int *>(&h.cols)[sub];
      t = reinterpret_cast<const int *>(&h.wts)[sub];
      base = nextBase(h.word, v, mask);
      if (Mode == kModeUpdate && sub == 0) atomicAdd(&C.expanded[k], 1u);
    }
    __syncwarp();
  }
  if (Mode != kModeUpdate && lane == 0 && done != 0) atomicAdd(&C.expanded[0], done);
  return farCount;
}

/// One entry per lane of a graph with row records: its word and its record
/// arrive together, its edges' atomicMin go out together, the improvements
/// of the warp take one reservation of the ring.
template <int Mode>
__device__ __noinline__ int expandRecords(const EngineParams &P, bool donate, int farCount, int k, int v,
                                          u64 base, bool live, int4 cols, int4 wts) {
  AsyncCta &C = asyncCta();
  const unsigned lane = laneId();
  const AsyncObj &O = C.obj[k];
  const unsigned scale = O.scale;
  const u64 most = live ? O.mostWord : 0;  // 0: nothing passes
  const u64 thrWord = O.thrWord;
  const int x[4] = {cols.x, cols.y, cols.z, cols.w};
  const u64 cw[4] = {static_cast<u64>(static_cast<unsigned>(wts.x)) * scale + base,
                     static_cast<u64>(static_cast<unsigned>(wts.y)) * scale + base,
                     static_cast<u64>(static_cast<unsigned>(wts.z)) * scale + base,
                     static_cast<u64>(static_cast<unsigned>(wts.w)) * scale + base};
  u64 old[4];
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    old[h] = 0;
    if (x[h] >= 0 && cw[h] <= most) old[h] = atomicMin(O.packed + x[h], cw[h]);
  }
  unsigned far = 0;  // bit h: this lane's edge h
  unsigned ballot[4];
  u64 entry[4];
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const bool imp = old[h] > (cw[h] | O.mask);
    const bool nr = imp && cw[h] < thrWord;
    far |= static_cast<unsigned>(imp && !nr && newInFar<Mode>(O, old[h], x[h])) << h;
    ballot[h] = __ballot_sync(kFull, nr);
    entry[h] = nearEntry(k, x[h], cw[h] >> O.bits);
  }
  nearPush<4>(P, ballot, donate, entry);
  if (__any_sync(kFull, far != 0)) {
#pragma unroll
    for (int h = 0; h < 4; ++h) farAppend(P, farCount, (far >> h) & 1u, k, x[h], cw[h] >> O.bits);
  }
  return farCount;
}

/// An idle warp's wait (warps other than 0): the entries that came by mail,
/// 0 when it has to look around again. All lanes call it.
__device__ __forceinline__ int asyncWait(const EngineParams &P, const Sync &sync, unsigned &parity) {
  AsyncCta &C = asyncCta();
  const int warp = static_cast<int>(threadIdx.x >> 5);
  int mail = 0;
  if (laneId() == 0) {
    atomicOr(&C.idle, 1u << warp);
    __threadfence_block();
    // what came between the last look and the idle bit
    bool wait = true;
    if (ldShared(&C.over) != 0 || ldShared(&C.abort) != 0 || ldShared(&C.tail) != ldShared(&C.head)) {
      // (a cleared bit means that a signal is on its way)
      wait = ((atomicAnd(&C.idle, ~(1u << warp)) >> warp) & 1u) == 0;
    }
    if (wait) {
      unsigned turns = 0;
      bool came = true;
      while (!barTryWait(&C.bar[warp], parity)) {
        ++turns;
        if ((turns & 255u) == 0 && globalNs() > sync.deadline + 1000000000ULL) asyncAbort(P);
        if (ldShared(&C.abort) != 0) {
          came = false;
          break;
        }
      }
      parity ^= 1u;
      // (who gives up has no mail: its count and slots may hold anything)
      if (came) mail = ldShared(&C.mail[warp]);
    }
  }
  parity = __shfl_sync(kFull, parity, 0);
  return __shfl_sync(kFull, mail, 0);
}

/// One phase for one warp: entries of the CTA's share and ring until the
/// phase is over (true) or the launch stops (false).
template <int Mode, int Kind>
__device__ __forceinline__ bool asyncConsume(const EngineParams &P, const int *outRow, const int *outCol,
                                             unsigned phase, const Sync &sync, unsigned &parity) {
  AsyncCta &C = asyncCta();
  const LoopShared &L = C.L;
  EngineControl *c = P.ctl;
  unsigned owed = 0;    // finished entries not yet added to the CTA's count
  int farCount = 0;     // entries in the warp's far buffer
  bool donate = false;  // other CTAs have run dry
  constexpr bool Rec = Kind != kCsrOnly;
  constexpr bool wideRecords = Kind == kRecords;
  const unsigned lane = laneId();
  const int warp = threadIdx.x >> 5;
  unsigned spins = 0, rounds = 0;
  while (true) {
    // ---- a batch of the ring, or of the share while the ring is short ----
    unsigned what = 0, at = 0;  // what: source << 8 | entries, donate in bit 16
    if (lane == 0) {
      while (true) {
        const unsigned h = ldShared(&C.head);
        const unsigned held = ldShared(&C.tail) - h;
        const unsigned cur = ldShared(&C.cur);
        if (cur < C.share && held <= kSliceFirst) {
          const unsigned left = C.share - cur;
          const unsigned n = left >= 1024 ? 32u : (left + 31u) >> 5;
          at = atomicAdd(&C.cur, n);
          if (at >= C.share) continue;
          what = (2u << 8) | (C.share - at < n ? C.share - at : n);
          break;
        }
        if (held == 0) break;
        const bool full = !Rec && ldShared(&C.full) != 0;
        const unsigned n = held >= 128 || (full && held >= 32) ? 32u : full ? held : (held + 3u) >> 2;
        if (atomicCAS(&C.head, h, h + n) != h) continue;
        if (full) what = 1u << 17;
        at = h;
        what |= (1u << 8) | n;
        if (held > C.donateAt) what |= 1u << 16;
        break;
      }
    }
    what = __shfl_sync(kFull, what, 0);
    int k = 0, v = 0;
    if (what == 0) {
      // ---- idle: settle what is done, then wait ---------------------------
      if (owed != 0) {
        if (farCount > 0) flushFarEntries(P, farCount);
        farCount = 0;
        if (lane == 0) {
          __threadfence_block();
          const unsigned now = atomicAdd(&C.settled, owed) + owed;
          __threadfence_block();
          if (now == ldShared(&C.tail) + ldShared(&C.mailed) + C.share) asyncDry(P, phase);
        }
        owed = 0;
        __syncwarp();
        continue;
      }
      int stop = 0;
      if (lane == 0) stop = ldShared(&C.abort) != 0 ? 2 : ldShared(&C.over);
      stop = __shfl_sync(kFull, stop, 0);
      if (stop == 2) return false;
      if (stop == 1) return true;
      if (warp == 0) {
        asyncFetch(P, phase);
        if ((++spins & 63u) == 0 && lane == 0 &&
            (ldVolatile(&c->status) != 0 || globalNs() > sync.deadline)) {
          asyncAbort(P);
        }
        __nanosleep(40);
        __syncwarp();
        continue;
      }
      const int mail = asyncWait(P, sync, parity);
      if constexpr (Rec) {
        if (mail > 0) {
          __syncwarp();  // lane 0's wait orders the mail for the others too
          owed += mail;
          const int q = static_cast<int>(lane >> 2);
          u64 base = 0;
          int x = -1, t = 0;
          if (q < mail) {
            const HopSlot &h = C.mailbox[warp][q];
            k = h.k;
            v = h.v;
            base = nextBase(h.word, v, C.obj[k].mask);
            x = reinterpret_cast<const int *>(&h.cols)[lane & 3u];
            t = reinterpret_cast<const int *>(&h.wts)[lane & 3u];
            if ((lane & 3u) == 0) atomicAdd(&C.expanded[k], 1u);
          }
          // (every lane's edge goes into the first hop's ballot, so the slots
          // are read before lane 0 can call the warp idle again)
          farCount = chaseRecords<Mode>(P, donate, farCount, k, v, base, x, t);
        }
      }
      continue;
    }
    at = __shfl_sync(kFull, at, 0);
    spins = 0;
    if ((++rounds & 1023u) == 0 && asyncStop(P)) return false;
    const bool fromRing = ((what >> 8) & 3u) == 1u;
    const unsigned n = what & 63u;
    // other CTAs have run dry (read with the entries' loads)
    int hungry = 0;
    if (lane == 0) {
      if (((what >> 16) & 1u) != 0) hungry = ldVolatile(&c->asyncHungry[phase % 3]);
      atomicAdd(&C.rounds, 1u);
      atomicAdd(&C.items, n);
    }
    owed += n;
    // few entries: a group of lanes each, expanded hop after hop
    constexpr unsigned kGroup = Rec ? 4 : 8;
    const bool thin = n <= 32 / kGroup && (what >> 17) == 0;
    const unsigned mine = thin ? lane / kGroup : lane;
    const bool lead = !thin || lane % kGroup == 0;
    const bool have = mine < n;
    unsigned tag = kTagSat;
    bool marked = false;
    if (fromRing) {
      u64 *slot = asyncRing() + ((at + mine) & kRingMask);
      u64 e = kEmptySlot;
      if (have) {
        unsigned spin = 0;
        while ((e = ldShared(slot)) == kEmptySlot) {  // reserved, about to be written
          if (++spin > kSpinLimit || ((spin & 1023u) == 0 && ldShared(&C.abort) != 0)) {
            asyncAbort(P);
            e = 0;
            break;
          }
        }
        k = static_cast<int>(e & 31u);
        v = static_cast<int>(static_cast<unsigned>(e) >> 5);
        tag = static_cast<unsigned>(e >> 32);
      }
      __syncwarp();
      if (have && lead) stShared(slot, kEmptySlot);
    } else if (have) {
      const long long j = C.base + at + mine;
      while (k + 1 < P.K && L.off[k + 1] <= j) ++k;
      const unsigned raw = static_cast<unsigned>(
          __ldcg((L.fp[k] == 0 ? P.farL0 : P.farL1) + static_cast<long long>(k) * P.strideFar +
                 (j - L.off[k])));
      v = static_cast<int>(raw & ~kOverflow);
      marked = (raw & kOverflow) != 0;
      if (marked || phase == 0) {
        // the flag is cleared before the word is read, so a push that still
        // finds it set is covered by the distance read here
        if (lead) atomicExch(P.inFar + static_cast<long long>(k) * P.stride + v, 0);
        __threadfence();
      }
    }
    if (!fromRing) __syncwarp();
    u64 word = kInfWord;
    int beg = 0, end = 0;
    // the entry's row record (thin: the lane's edge of it)
    const bool records = Rec && (thin || wideRecords);
    int4 cols = make_int4(-1, -1, -1, -1), wts = make_int4(0, 0, 0, 0);
    if (have) {
      word = __ldcg(C.obj[k].packed + v);
      if (records) {
        const int4 *r = C.obj[k].rec + 2LL * v;
        if (thin) {
          cols.x = reinterpret_cast<const int *>(r)[lane & 3u];
          wts.x = reinterpret_cast<const int *>(r)[4 + (lane & 3u)];
        } else {
          cols = r[0];
          wts = r[1];
        }
      } else {
        beg = ldLoop<Mode>(outRow + v);
        end = ldLoop<Mode>(outRow + v + 1);
      }
    }
    // A ring entry is stale when its vertex has improved since (the newer
    // distance has its own entry); else it is expanded with its tag, which
    // also covers a word read that is older than the entry. A pile entry
    // below the last phase's threshold was expanded when it got there.
    const AsyncObj &O = C.obj[k];
    const u64 d = word == kInfWord ? kInfWord : word >> O.bits;
    bool live = false;
    u64 du = d;
    if (fromRing) {
      if (tag < kTagSat) {
        live = have && d >= tag;
        du = tag;
      } else {
        live = have && d != kInfWord;
      }
    } else {
      const bool near = d < O.thr;
      live = have && near && (marked || d >= O.prev);
      farAppend(P, farCount, have && !near && lead, k, v, d);
    }
    if (live && lead) atomicAdd(&C.expanded[k], 1u);
    donate = __shfl_sync(kFull, hungry, 0) > 0;
    bool rows = !records;
    if constexpr (Rec) {
      // a row longer than its record: this batch by rows
      if (records && __any_sync(kFull, live && (thin ? cols.x : cols.w) == kMoreEdges)) {
        rows = true;
        if (live) {
          beg = ldLoop<Mode>(outRow + v);
          end = ldLoop<Mode>(outRow + v + 1);
        }
      }
    }
    if (Rec && !rows) {
      const u64 base = offerBase(O, du, v);
      if (thin) {
        farCount = chaseRecords<Mode>(P, donate, farCount, k, v, base, live ? cols.x : -1, wts.x);
        continue;
      }
      if constexpr (wideRecords) {
        farCount = expandRecords<Mode>(P, donate, farCount, k, v, base, live, cols, wts);
        continue;
      }
    }
    if (!live) end = beg;
    if constexpr (!Rec) {
      if (thin && !__any_sync(kFull, end - beg > kOctDeg)) {
        chase<Mode>(P, outRow, outCol, donate, farCount, k, v, du, beg, end);
        continue;
      }
    }
    expandRows<Mode>(P, outCol, donate, farCount, k, v, du, beg, lead ? end : beg);
  }
}

template <int Mode, int Kind>
__device__ __noinline__ bool asyncNearFar(const EngineParams &P, const int *outRow, const int *outCol,
                                          const int *const *outWk, Sync &epoch, u64 *deltaOverride,
                                          int genBase) {
  AsyncCta &C = asyncCta();
  LoopShared &L = C.L;
  StageHeader &H = stageHeader();
  EngineControl *c = P.ctl;
  const int K = P.K;
  const unsigned lane = laneId();
  const int warp = threadIdx.x >> 5;
  const Sync sync = epoch;

  // per-objective state, held by lane k of warp 0 (the same in every CTA)
  u64 thr = 0;
  int fp = 0, fs = 0, phasesK = 0;
  u64 delta = 1;
  if (warp == 0 && static_cast<int>(lane) < K) {
    delta = P.obj[lane].delta;
    if (deltaOverride != nullptr && lane == 0) delta = *deltaOverride;
    const ObjectiveArgs &O = P.obj[lane];
    AsyncObj &A = C.obj[lane];
    A.packed = P.packed + lane * P.stride;
    A.rec = P.rec == nullptr ? nullptr : P.rec + 2 * lane * P.stride;
    A.outW = outWk[lane];
    A.dist = O.dist;
    A.bits = O.parentBits;
    A.scale = 1u << O.parentBits;
    A.mask = A.scale - 1u;
    A.mostWord = (O.maxDist << O.parentBits) | A.mask;
    A.thr = 0;
  }
  if (threadIdx.x < kMaxK) C.expanded[threadIdx.x] = 0;
  if (threadIdx.x < kWarps) barInit(&C.bar[threadIdx.x]);
  if (threadIdx.x == 0) {
    C.lock = 0;
    C.abort = 0;
    C.idle = 0;
    C.fed = 0;
    C.rounds = C.fedRounds = C.items = C.taken = 0;
    C.K = K;
    C.donateAt = Kind == kThinRecords ? kDonate : kDonateLeast;
    C.deadline = sync.deadline;
  }
  for (int i = threadIdx.x; i < kRing; i += blockDim.x) asyncRing()[i] = kEmptySlot;
  unsigned parity = 0;
  const unsigned long long t0 = globalNs();
  unsigned long long tPhase = t0;
  unsigned phase = 0;
  for (;; ++phase) {
    if (threadIdx.x < kMaxK) H.farMin[threadIdx.x] = kInfWord;
    if (warp == 0) {
      const int k = static_cast<int>(lane);
      const bool act = k < K;
      int mode = kDone;
      long long items = 0;
      u64 least = 0;
      if (act) {
        const int fc = __ldcg(&c->farCount[k][fs]);
        const u64 mnC = __ldcg(&c->farMinC[k][fs]);
        C.obj[k].prev = thr;
        if (fc > 0) {
          mode = kSplit;
          items = fc;
          if (mnC != 0) least = ~mnC;
        }
      }
      long long incl = items;
      for (int off = 1; off < K; off <<= 1) {
        const long long o = __shfl_up_sync(kFull, incl, off);
        if (static_cast<int>(lane) >= off) incl += o;
      }
      const long long total = __shfl_sync(kFull, incl, K - 1);
      if (mode == kSplit) {
        // Thin phases (few entries per CTA) are twice as wide: they pay for
        // their start and end more than for entries expanded again. Twice
        // the width everywhere: loop from scratch of a 497,700-vertex road
        // network 2.90 -> 2.50 ms (1,500 entries per phase), combined graph
        // of 249,500 vertices 1.47 -> 1.29 ms, but the update of 2M vertices
        // with 1.2M entries per phase 1.20 -> 1.30 ms; four times: 2.71,
        // 1.38 and 1.25 ms. Not so the first phase of a graph without
        // records, where a root may reach most of a graph of small diameter
        // (tree from scratch of 2M random vertices of degree 10: 10.2M
        // entries in 2.64 ms, with the single width 4.6M in 1.36).
        const bool thin = total <= static_cast<long long>(kThinShare) * gridDim.x && (phase > 0 || Kind != kCsrOnly);
        const u64 width = thin ? 2 * delta : delta;
        const u64 lo = least > thr ? least : thr;
        thr = lo > kInfWord - width ? kInfWord - 1 : lo + width;
      }
      if (act) {
        L.off[k] = incl - items;
        L.thr[k] = thr;
        AsyncObj &A = C.obj[k];
        A.thr = thr;
        A.thrWord = thr > (kInfWord >> A.bits) ? kInfWord : thr << A.bits;
        L.mode[k] = mode;
        L.fp[k] = fp;
        L.fs[k] = fs;
      }
      if (lane == 0) {
        // this CTA's share: an equal, contiguous range of the piles
        const long long per = (total + gridDim.x - 1) / gridDim.x;
        const long long lo = per * blockIdx.x < total ? per * blockIdx.x : total;
        const long long hi = lo + per < total ? lo + per : total;
        L.total = total;
        C.base = lo;
        C.share = static_cast<unsigned>(hi - lo);
        C.head = C.tail = C.cur = C.settled = C.mailed = 0;
        C.owed = 1;
        C.dry = 0;
        C.over = 0;
        C.full = 0;
        if (C.fed != 0) C.fedRounds += C.rounds - C.fedFrom;
        C.fed = 0;
        C.phase = phase;
        if (blockIdx.x == 0) {
          // the counters of the next phase (last looked at before this one)
          c->asyncPending[(phase + 1) % 3] = gridDim.x;
          c->asyncHungry[(phase + 1) % 3] = 0;
        }
        if (globalNs() > sync.deadline) {
          atomicCAS(&c->status, 0, MOSP_ERR_TIMEOUT);
          L.total = -1;  // the launch stops
        }
      }
      if (blockIdx.x == 0 && static_cast<int>(lane) < P.aqShards) {
        AsyncShard &A = P.aqCtr[(phase + 1) % 3 * P.aqShards + lane];
        A.claimed = A.reserved = 0;
      }
      if (act && mode == kSplit) {
        if (blockIdx.x == 0) {
          // the slot the next phase appends to (last read a phase ago)
          c->farCount[k][(fs + 2) % 3] = 0;
          c->farMinC[k][(fs + 2) % 3] = 0;
        }
        ++phasesK;
        fp ^= 1;
        fs = (fs + 1) % 3;
      }
    }
    __syncthreads();
    if (L.total < 0) return false;
    if (L.total == 0) break;
    if (threadIdx.x == 0 && C.share == 0) asyncDry(P, phase);
    const bool ok = asyncConsume<Mode, Kind>(P, outRow, outCol, phase, sync, parity);
    if (__syncthreads_or(!ok)) return false;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      // phase durations (the first four, then the rest summed)
      const unsigned long long now = globalNs();
      c->iterSplitNs[phase < 4 ? phase : 4] += now - tPhase;
      tPhase = now;
    }
  }
  if (threadIdx.x == 0 && C.rounds != 0) {
    atomicAdd(reinterpret_cast<unsigned long long *>(&c->loopIters[1]),
              static_cast<unsigned long long>(C.rounds));
    atomicAdd(reinterpret_cast<unsigned long long *>(&c->loopNs[1]),
              static_cast<unsigned long long>(C.rounds - C.fedRounds));
    atomicAdd(reinterpret_cast<unsigned long long *>(&c->loopItems[0]),
              static_cast<unsigned long long>(C.taken));
    atomicAdd(reinterpret_cast<unsigned long long *>(&c->loopItems[1]),
              static_cast<unsigned long long>(C.items - C.taken));
  }
  if (threadIdx.x < K && C.expanded[threadIdx.x] != 0) {
    atomicAdd(reinterpret_cast<unsigned long long *>(&c->pushes[threadIdx.x]),
              static_cast<unsigned long long>(C.expanded[threadIdx.x]));
  }
  if (blockIdx.x == 0 && warp == 0 && static_cast<int>(lane) < K) {
    c->iterations[lane] = phasesK;
    c->epochs[lane] = phasesK;
    if (lane == 0) {
      c->finalGen = genBase + 1;
      *P.genPtr = genBase + 1;
      c->loopNs[0] = globalNs() - t0;
      c->loopIters[0] = phase;
    }
  }
  return true;
}

/// Lowest-id tight parent of every vertex of the distance-only objectives
/// (parent INT_MAX after the unpack, -1 for roots and unreached vertices);
/// thread tid of T.
template <int Mode>
__device__ void recoverTightParents(const EngineParams &P, const int *outRow, const int *outCol,
                                    const int *const *outWk, long long tid, long long T) {
  const int n = P.n, K = P.K;
  // Lowest-id tight parent of every vertex of a distance-only objective:
  // every edge (u, x) with d(u) + w = d(x) offers u to x by atomicMin, so
  // the result does not depend on which thread checks which edge.
  // Edge-balanced: warp w takes the w-th equal slice of the edge array and
  // its lanes read two windows of 32 consecutive edges at a time
  // (coalesced), so hub rows and hub-dense id ranges of power-law graphs
  // cost no more than any other slice. The warp finds the source rows of
  // its edges from the ends of the next 32 rows (one coalesced load) by a
  // 5-step shuffle search, moving on 32 rows at a time through runs of
  // empty rows. The row search and the head loads are shared by all
  // distance-only objectives, whose loads then go out together.
  const unsigned lane = laneId();
  const long long gwarp = tid >> 5;
  const long long nwarps = T >> 5;
  const long long m = ldGraph<Mode>(outRow + n);
  const long long wb = m * gwarp / nwarps, we = m * (gwarp + 1) / nwarps;
  if (wb >= we) return;  // warp-uniform
  // the row of the slice's first edge: the last r with rowPtr[r] <= wb
  int lo = 0, hi = n;
  while (hi - lo > 1) {
    const int mid = lo + ((hi - lo) >> 1);
    if (ldGraph<Mode>(outRow + mid) <= wb) lo = mid; else hi = mid;
  }
  int r0 = lo;  // no edge of the rest of the slice lies in a row before r0
  for (long long e0 = wb; e0 < we; e0 += 64) {
    const int ea = static_cast<int>(e0 + lane);
    const int eb = static_cast<int>(e0 + 32 + lane);
    const bool la = e0 + lane < we, lb = e0 + 32 + lane < we;
    const int xa = la ? ldGraph<Mode>(outCol + ea) : 0;
    const int xb = lb ? ldGraph<Mode>(outCol + eb) : 0;
    int rowA = la ? -1 : 0, rowB = lb ? -1 : 0;
    // at most ceil((n - r0) / 32) windows: the window holding row n - 1
    // ends every search, since rows past n count as ending at INT_MAX
    for (int base = r0; base < n; base += 32) {
      const int rr = base + static_cast<int>(lane);
      const int end = rr < n ? ldGraph<Mode>(outRow + rr + 1) : INT_MAX;
      // pos = how many of the window's rows end at or before the edge
      int posA = 0, posB = 0;
#pragma unroll
      for (int step = 16; step >= 1; step >>= 1) {
        const int probeA = __shfl_sync(kFull, end, posA + step - 1);
        const int probeB = __shfl_sync(kFull, end, posB + step - 1);
        if (probeA <= ea) posA += step;
        if (probeB <= eb) posB += step;
      }
      const int lastEnd = __shfl_sync(kFull, end, 31);
      if (rowA < 0 && ea < lastEnd) rowA = base + posA;
      if (rowB < 0 && eb < lastEnd) rowB = base + posB;
      if (__all_sync(kFull, rowA >= 0 && rowB >= 0)) break;
    }
    // lane 31 of the second window holds the largest row; when it is past
    // the slice the loop ends here anyway
    r0 = __shfl_sync(kFull, rowB, 31);
    const bool ca = la && rowA >= 0 && !isRoot(P.source, P.sources, P.nSources, xa);
    const bool cb = lb && rowB >= 0 && !isRoot(P.source, P.sources, P.nSources, xb);
    for (int k = 0; k < K; ++k) {
      const ObjectiveArgs &O = P.obj[k];
      if (O.parentBits > 0) continue;  // the same for every thread
      const long long ko = static_cast<long long>(k) * P.stride;
      const int *w = outWk[k];
      u64 da = kInfWord, db = kInfWord, pa = 0, pb = 0;
      int wa = 0, wbt = 0;
      if (ca) {
        da = __ldcg(P.packed + ko + rowA);
        pa = __ldcg(P.packed + ko + xa);
        wa = ldGraph<Mode>(w + ea);
      }
      if (cb) {
        db = __ldcg(P.packed + ko + rowB);
        pb = __ldcg(P.packed + ko + xb);
        wbt = ldGraph<Mode>(w + eb);
      }
      if (da != kInfWord && da + static_cast<u64>(wa) == pa) atomicMin(O.parent + xa, rowA);
      if (db != kInfWord && db + static_cast<u64>(wbt) == pb) atomicMin(O.parent + xb, rowB);
    }
  }
}

/// The distance-only objectives of a launch, in order: their number.
__device__ int fallbackObjectives(const EngineParams &P, int *which) {
  int count = 0;
  for (int k = 0; k < P.K; ++k) {
    if (P.obj[k].parentBits == 0) which[count++] = k;
  }
  return count;
}

// ---------------------------------------------------------------------------
// Unpack words into (distance, parent); distance-only objectives recover
// the lowest-id tight parent (reference src/sospUpdateGpu.cu:478-512).
// ---------------------------------------------------------------------------
template <int Mode>
__device__ bool unpackResults(const EngineParams &P, const int *outRow,
                              const int *outCol, const int *const *outWk,
                              Sync &epoch) {
  const int n = P.n, K = P.K;
  const long long tid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long T = static_cast<long long>(gridDim.x) * blockDim.x;
  const bool restricted = Mode == kModeUpdate && P.recMark != nullptr && P.recChangedList != nullptr &&
                          (P.flags & (kFlagCanonical | kFlagHostRecovery)) ==
                              (kFlagCanonical | kFlagHostRecovery);
  bool anyFallback = false;
  for (int k = 0; k < K; ++k) {
    const ObjectiveArgs &O = P.obj[k];
    const Pk pk = pkOf(O);
    const long long ko = static_cast<long long>(k) * P.stride;
    if (O.parentBits > 0) {
      // four words per thread (v, v + T, v + 2T, v + 3T), loaded together
      for (long long v0 = tid; v0 < n; v0 += 4 * T) {
        u64 word[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const long long v = v0 + q * T;
          word[q] = v < n ? __ldcg(P.packed + ko + v) : kInfWord;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const long long v = v0 + q * T;
          if (v >= n) break;
          if (word[q] == kInfWord) {
            O.dist[v] = kDistInf;
            O.parent[v] = -1;
          } else {
            O.dist[v] = static_cast<long long>(pk.dist(word[q]));
            O.parent[v] = pk.parent(word[q]);
          }
        }
      }
    } else if (restricted) {
      // restricted recovery (recover.cu): the input parents stay; the mark
      // byte says whether the distance changed, and the changed vertices
      // are listed (one reservation per warp)
      anyFallback = true;
      unsigned char *mark = P.recMark + ko;
      int *changed = P.recChangedList + ko;
      const int lane = static_cast<int>(laneId());
      for (long long v0 = tid - lane; v0 < n; v0 += T) {  // the same v0 in the whole warp
        const long long v = v0 + lane;
        bool chg = false;
        if (v < n) {
          const u64 word = __ldcg(P.packed + ko + v);
          const long long d = word == kInfWord ? kDistInf : static_cast<long long>(word);
          chg = O.dist[v] != d;
          mark[v] = chg ? kRecChanged : 0;
          O.dist[v] = d;
          if (word == kInfWord || isRoot(P.source, P.sources, P.nSources, static_cast<int>(v))) {
            O.parent[v] = -1;
          }
        }
        const unsigned bal = __ballot_sync(kFull, chg);
        if (bal != 0) {
          int at = 0;
          if (lane == __ffs(bal) - 1) at = atomicAdd(&P.ctl->recChanged[k], __popc(bal));
          at = __shfl_sync(kFull, at, __ffs(bal) - 1);
          if (chg) changed[at + __popc(bal & ((1u << lane) - 1))] = static_cast<int>(v);
        }
      }
    } else if (Mode == kModeUpdate && P.recDist != nullptr) {
      anyFallback = true;  // below, all of them together
    } else {
      anyFallback = true;
      for (long long v = tid; v < n; v += T) {
        const u64 word = __ldcg(P.packed + ko + v);
        O.dist[v] = word == kInfWord ? kDistInf : static_cast<long long>(word);
        O.parent[v] = (word == kInfWord || isRoot(P.source, P.sources, P.nSources, static_cast<int>(v)))
                          ? -1
                          : INT_MAX;
      }
    }
  }
  if (Mode == kModeUpdate && anyFallback && !restricted && P.recDist != nullptr) {
    // a vertex's distances side by side for recoverParents32
    __shared__ int sFall[kMaxK];
    __shared__ int sCount;
    if (threadIdx.x == 0) sCount = fallbackObjectives(P, sFall);
    __syncthreads();
    const int count = sCount;
    const int vec = count <= 4 ? 1 : 2;
    bool wide = false;
    for (int g0 = 0; g0 < count; g0 += 8) {
      int4 *out = P.recDist + static_cast<long long>(g0 / 8) * 2 * n;
      for (long long v = tid; v < n; v += T) {
        const bool root = isRoot(P.source, P.sources, P.nSources, static_cast<int>(v));
        unsigned d32[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          d32[j] = ~0u;
          if (g0 + j >= count) continue;
          const int k = sFall[g0 + j];
          const ObjectiveArgs &O = P.obj[k];
          const u64 word = __ldcg(P.packed + static_cast<long long>(k) * P.stride + v);
          O.dist[v] = word == kInfWord ? kDistInf : static_cast<long long>(word);
          O.parent[v] = word == kInfWord || root ? -1 : INT_MAX;
          if (word != kInfWord) {
            wide |= word >= (1ULL << 31);
            d32[j] = static_cast<unsigned>(word);
          }
        }
        out[vec * v] = make_int4(d32[0], d32[1], d32[2], d32[3]);
        if (vec == 2) out[2 * v + 1] = make_int4(d32[4], d32[5], d32[6], d32[7]);
      }
    }
    if (wide) P.ctl->recWide = 1;
  }
  if (!anyFallback || (P.flags & kFlagHostRecovery) != 0) return true;
  if (!gridSync(P.ctl, epoch)) return false;
  recoverTightParents<Mode>(P, outRow, outCol, outWk, tid, T);
  return true;
}

/// Exclusive scan in[0, len) -> out[0, len) (and copy -> cursor) across the
/// grid; two phases separated by one grid barrier. Returns the total.
__device__ bool gridExclusiveScan(const int *in, int *out, int *cursor, long long len,
                                  long long *blockSums, EngineControl *c,
                                  Sync &epoch, long long *grandTotal) {
  const long long chunk = (len + gridDim.x - 1) / gridDim.x;
  const long long lo = static_cast<long long>(blockIdx.x) * chunk;
  const long long hi = lo + chunk < len ? lo + chunk : len;
  long long local = 0;
  for (long long i = lo + threadIdx.x; i < hi; i += blockDim.x) local += __ldcg(in + i);
  const long long sum = blockSum(local);
  if (threadIdx.x == 0) blockSums[blockIdx.x] = sum;
  if (!gridSync(c, epoch)) return false;
  long long before = 0, all = 0;
  for (int b = threadIdx.x; b < static_cast<int>(gridDim.x); b += blockDim.x) {
    const long long s = __ldcg(blockSums + b);
    all += s;
    if (b < static_cast<int>(blockIdx.x)) before += s;
  }
  before = blockSum(before);
  all = blockSum(all);
  long long carry = before;
  for (long long t = lo; t < hi; t += blockDim.x) {
    const long long i = t + threadIdx.x;
    const long long x = i < hi ? __ldcg(in + i) : 0;
    long long tileTotal;
    const long long incl = blockInclusiveScan(x, &tileTotal);
    if (i < hi) {
      out[i] = static_cast<int>(carry + incl - x);
      if (cursor != nullptr) cursor[i] = static_cast<int>(carry + incl - x);
    }
    carry += tileTotal;
  }
  *grandTotal = all;
  return true;
}

// ---------------------------------------------------------------------------
// Combined graph edge of parent k of v (reference
// src/combinedGraphGpu.cu:55-75): edge (p, v) is attributed to the first
// tree whose parent of v is p; its weight is base - sum of the preference
// terms of every tree with that parent.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool combinedEdge(const EngineParams &P, int v, int k,
                                             int &p, int &weight) {
  const long long n = P.n;
  p = __ldg(P.combParents + k * n + v);
  if (p < 0) return false;
  for (int j = 0; j < k; ++j) {
    if (__ldg(P.combParents + j * n + v) == p) return false;
  }
  weight = P.combBase - P.prefTerms[k];
  for (int j = k + 1; j < P.combK; ++j) {
    if (__ldg(P.combParents + j * n + v) == p) weight -= P.prefTerms[j];
  }
  return true;
}

template <int Mode>
__device__ void scratchOrCombined(const EngineParams &P, Sync &epoch, int genBase,
                                  const int **sOutWk);

/// The invalidated vertices of objective k: their words to infinity and into
/// the candidate list. A warp takes 32 x Words vertices at a time, whose loads
/// are in flight together, keeps their verdicts as one word per lane and
/// reserves its part of the list with one atomic. Against a contiguous range
/// per CTA, compacted by block scans in a second pass over it: 2M vertices,
/// K = 3 0.056 -> 0.033 ms; 4.2M, K = 5 0.168 -> 0.081; with Words = 16 for
/// 93,300, K = 3 too few warps have work, 0.012 -> 0.017.
template <int Words>
__device__ __forceinline__ void collectInvalid(const EngineParams &P, int k, long long gwarp, long long nwarps) {
  EngineControl *c = P.ctl;
  const int n = P.n;
  const unsigned lane = laneId();
  const long long ko = static_cast<long long>(k) * P.stride;
  for (long long b = gwarp * (32 * Words); b < n; b += nwarps * (32 * Words)) {
    int val[Words];
#pragma unroll
    for (int j = 0; j < Words; ++j) {
      const long long v = b + 32 * j + lane;
      val[j] = v < n ? __ldcg(P.val + ko + v) : -1;
    }
    unsigned mine = 0;  // lane j: the verdicts of vertices b + 32 j ...
#pragma unroll
    for (int j = 0; j < Words; ++j) {
      const unsigned inv = __ballot_sync(kFull, val[j] == -2);
      if (static_cast<int>(lane) == j) mine = inv;
    }
    int incl = __popc(mine);
#pragma unroll
    for (int off = 1; off < Words; off <<= 1) {
      const int o = __shfl_up_sync(kFull, incl, off);
      if (static_cast<int>(lane) >= off) incl += o;
    }
    const int found = __shfl_sync(kFull, incl, Words - 1);
    if (found == 0) continue;
    int base = 0;
    if (lane == 0) {
      base = atomicAdd(&c->candCount[k], found);
      atomicAdd(&c->invalidated[k], found);
    }
    base = __shfl_sync(kFull, base, 0) + incl - __popc(mine);
#pragma unroll
    for (int j = 0; j < Words; ++j) {
      const unsigned inv = __shfl_sync(kFull, mine, j);
      const int at = __shfl_sync(kFull, base, j) + __popc(inv & ((1u << lane) - 1u));
      if ((inv >> lane) & 1u) {
        const long long v = b + 32 * j + lane;
        P.packed[ko + v] = kInfWord;
        P.cand[ko + at] = static_cast<int>(v);
      }
    }
  }
}

/// Row records for the asynchronous loop, one 32-byte sector per objective
/// and vertex: the heads of its first four edges (-1: none, or the source,
/// which nothing improves) and their weights. A row of more than four edges
/// holds kMoreEdges in place of the fourth; the rest stays in the CSR.
/// Thread tid of T.
template <int Mode>
__device__ void buildRecords(const EngineParams &P, const int *outRow, const int *outCol,
                             const int *const *outWk, long long tid, long long T) {
  int longer = 0;
  for (long long v = tid; v < P.n; v += T) {
    const int b = ldLoop<Mode>(outRow + v);
    const int deg = ldLoop<Mode>(outRow + v + 1) - b;
    int c[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) c[q] = q < deg ? ldLoop<Mode>(outCol + b + q) : -1;
#pragma unroll
    for (int q = 0; q < 4; ++q) c[q] = c[q] == P.source ? -1 : c[q];
    if (deg > 4) {
      c[3] = kMoreEdges;
      ++longer;
    }
    for (int k = 0; k < P.K; ++k) {
      int w[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) w[q] = q < deg ? ldLoop<Mode>(outWk[k] + b + q) : 0;
      int4 *r = P.rec + 2 * (static_cast<long long>(k) * P.stride + v);
      r[0] = make_int4(c[0], c[1], c[2], c[3]);
      r[1] = make_int4(w[0], w[1], w[2], w[3]);
    }
  }
  __syncwarp();
  longer = __reduce_add_sync(kFull, longer);
  if (laneId() == 0 && longer > 0) atomicAdd(&P.ctl->longRows, longer);
}

/// The near-far loop of a launch: asynchronous when the launch asks for it
/// and the graph has no hub rows (which the bulk loop hands to whole CTAs),
/// with row records where the launch made them (rec) and they hold nearly all
/// rows; the same decision in every CTA (the hub flag and the count of longer
/// rows are final before a barrier).
template <int Mode>
__device__ bool runNearFar(const EngineParams &P, const int *outRow, const int *outCol,
                           const int *const *outWk, Sync &epoch, u64 *deltaOverride, int genBase,
                           bool rec) {
  // the asynchronous loop adds a weight to a packed word without a check: a
  // bound within 2^31 of what the word holds goes to the bulk loop
  bool fits = true;
  for (int k = 0; k < P.K; ++k) {
    fits = fits && P.obj[k].maxDist + (1ULL << 31) <= (kInfWord >> P.obj[k].parentBits);
  }
  const bool async = fits && (P.flags & kFlagAsync) != 0 && P.aqSlots != nullptr && P.aqShards > 0 &&
                     P.aqShards <= kAsyncShards && P.n <= (1 << 27) &&
                     P.stageEntries >= kStageEntriesAsync &&
                     __ldcg(&P.ctl->heavy) == 0;
  if (async && rec && kLongRows * __ldcg(&P.ctl->longRows) <= P.n) {
    constexpr int Kind = Mode == kModeUpdate ? kThinRecords : kRecords;
    return asyncNearFar<Mode, Kind>(P, outRow, outCol, outWk, epoch, deltaOverride, genBase);
  }
  if (async) return asyncNearFar<Mode, kCsrOnly>(P, outRow, outCol, outWk, epoch, deltaOverride, genBase);
  return nearFarLoop<Mode>(P, outRow, outCol, outWk, epoch, deltaOverride, genBase);
}

// ---------------------------------------------------------------------------
// The engine kernel
// ---------------------------------------------------------------------------
/// Pull pass: the best word that the in-edges e = first, first + step, ...
/// (< end) offer to their head (objective with args O at offset ko), folded
/// into `best`. Four edges per round with their loads in flight together
/// (the column and weight loads, then the four tail words), so a long
/// in-row is not one chain of dependent loads per edge.
__device__ __forceinline__ u64 pullBest(const EngineParams &P, const ObjectiveArgs &O,
                                        const Pk &pk, long long ko, int first, int end,
                                        int step, u64 best) {
  for (long long e0 = first; e0 < end; e0 += 4LL * step) {
    int u[4], w[4];
    u64 wd[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const long long e = e0 + static_cast<long long>(q) * step;
      u[q] = e < end ? __ldg(P.inCol + e) : -1;
      w[q] = e < end ? __ldg(O.inW + e) : 0;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) wd[q] = u[q] >= 0 ? __ldcg(P.packed + ko + u[q]) : kInfWord;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (wd[q] == kInfWord) continue;
      const u64 nd = pk.dist(wd[q]) + static_cast<u64>(w[q]);
      if (nd <= O.maxDist) {
        const u64 cw = pk.pack(nd, u[q]);
        best = cw < best ? cw : best;
      }
    }
  }
  return best;
}

/// The push direction of the pass before the near-far loop, for objective
/// k: every valid (finite, not invalidated) vertex offers its distance plus
/// the edge weight along each out-edge; strict improvements go to far pile
/// 0 once (in-far flag). Warp gwarp of nwarps; a lane per short row, the
/// whole warp per row of more than kLaneRowMax edges.
__device__ void pushFromValid(const EngineParams &P, int k, const int *w, long long gwarp,
                              long long nwarps) {
  EngineControl *c = P.ctl;
  const ObjectiveArgs &O = P.obj[k];
  const Pk pk = pkOf(O);
  const long long ko = static_cast<long long>(k) * P.stride;
  const unsigned lane = laneId();
  auto relax = [&](int u, u64 du, int e) {
    const int x = __ldg(P.outCol + e);
    const u64 nd = du + static_cast<u64>(__ldg(w + e));
    if (x == P.source || nd > O.maxDist) return;
    const u64 old = atomicMin(P.packed + ko + x, pk.pack(nd, u));
    if (nd >= pk.dist(old)) return;
    if (atomicExch(P.inFar + ko + x, 1) == 0) {
      const int idx = warpAppend(&c->farCount[k][0]);
      P.farL0[static_cast<long long>(k) * P.strideFar + idx] = x;
      warpMinInto(&c->farMinC[k][0], nd);
    }
  };
  for (long long base = gwarp * 32; base < P.n; base += nwarps * 32) {
    const long long v = base + lane;
    u64 word = kInfWord;
    int beg = 0, end = 0;
    if (v < P.n) {
      word = __ldcg(P.packed + ko + v);
      if (word != kInfWord) {
        beg = __ldg(P.outRow + v);
        end = __ldg(P.outRow + v + 1);
      }
    }
    const u64 dv = word == kInfWord ? 0 : pk.dist(word);
    const int deg = end - beg;
    if (deg <= kLaneRowMax) {
      for (int e = beg; e < end; ++e) relax(static_cast<int>(v), dv, e);
    }
    unsigned big = __ballot_sync(kFull, deg > kLaneRowMax);
    while (big != 0) {
      const int src = __ffs(big) - 1;
      big &= big - 1;
      const int ub = static_cast<int>(__shfl_sync(kFull, v, src));
      const u64 db = __shfl_sync(kFull, dv, src);
      const int bb = __shfl_sync(kFull, beg, src);
      const int eb = __shfl_sync(kFull, end, src);
      for (int e = bb + static_cast<int>(lane); e < eb; e += 32) relax(ub, db, e);
    }
  }
}

template <int Mode>
__global__ void __launch_bounds__(kThreads, 1) sospEngine(const __grid_constant__ EngineParams P) {
  EngineControl *c = P.ctl;
  const int n = P.n, K = P.K;
  const long long tid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long T = static_cast<long long>(gridDim.x) * blockDim.x;
  const unsigned lane = laneId();
  const int warp = threadIdx.x >> 5;
  Sync epoch = startSync(P.timeoutNs);
  // Stamp generations of this launch start after the previous launch's.
  const int genBase = __ldcg(P.genPtr) + 1;

  __shared__ const int *sOutWk[kMaxK];
  if (threadIdx.x < kMaxK) {
    sOutWk[threadIdx.x] =
        static_cast<int>(threadIdx.x) < K ? P.obj[threadIdx.x].outW : nullptr;
  }
  const int *outRow = P.outRow;
  const int *outCol = P.outCol;

  markPhase(c, kPhaseStart);
  // the asynchronous loop's spill queue starts empty and every CTA owes its
  // share of the first phase (every mode passes a grid barrier before its
  // near-far loop)
  if ((P.flags & kFlagAsync) != 0 && P.aqCtr != nullptr) {
    for (long long i = tid; i < P.aqShards; i += T) P.aqCtr[i].claimed = P.aqCtr[i].reserved = 0;
    if (tid == 0) c->asyncPending[0] = gridDim.x;
  }
  if constexpr (Mode == kModeUpdate) {
    // ---- Heavy rows: does the graph have rows for whole-CTA handling? -----
    const int heavyDeg = heavyDegOf(P);
    bool heavyRow = false;  // one store at the end, so the loads run ahead
    for (long long v = tid; v < n; v += T) {
      heavyRow |= __ldg(outRow + v + 1) - __ldg(outRow + v) > heavyDeg ||
                  __ldg(P.inRow + v + 1) - __ldg(P.inRow + v) > heavyDeg;
    }
    if (heavyRow) c->heavy = 1;
    // ---- Pack the old trees; ancestors (reference :234-252) ---------------
    // four vertices per thread (v, v + T, v + 2T, v + 3T): their loads are
    // issued before any of their stores
    bool badParent = false, badDist = false;
    for (int k = 0; k < K; ++k) {
      const ObjectiveArgs &O = P.obj[k];
      const Pk pk = pkOf(O);
      const long long ko = static_cast<long long>(k) * P.stride;
      for (long long v0 = tid; v0 < n; v0 += 4 * T) {
        long long d[4];
        int p[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const long long v = v0 + q * T;
          d[q] = v < n ? O.dist[v] : kDistInf;
          p[q] = v < n ? O.parent[v] : -1;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const long long v = v0 + q * T;
          if (v >= n) break;
          if (p[q] < -1 || p[q] >= n) {
            badParent = true;
            p[q] = -1;
          }
          u64 word;
          if (d[q] >= kDistInf / 2) {
            word = kInfWord;
          } else if (d[q] < 0 || static_cast<u64>(d[q]) > O.maxDist) {
            badDist = true;
            word = kInfWord;
          } else {
            word = pk.pack(static_cast<u64>(d[q]), p[q]);
          }
          P.packed[ko + v] = word;
          P.val[ko + v] = p[q];  // >= 0: ancestor; -1: none; -2: invalidated
        }
      }
    }
    if (badParent) c->invalid = 1;
    if (badDist) c->overflow = 1;
    __syncthreads();  // sOutWk
    if (P.rec != nullptr) buildRecords<Mode>(P, outRow, outCol, sOutWk, tid, T);
    if (!gridSync(c, epoch)) return;
    markPhase(c, kPhasePacked);

    // ---- Roots: heads of changed tree edges -------------------------------
    long long changes = 0;
    for (int k = 0; k < K; ++k) {
      const ObjectiveArgs &O = P.obj[k];
      const long long ko = static_cast<long long>(k) * P.stride;
      changes += O.nChanged;
      for (long long i = tid; i < O.nChanged; i += T) {
        const int v = O.chTo[i], u = O.chFrom[i];
        if (v < 0 || v >= n || u < 0 || u >= n) {
          c->invalid = 1;
          continue;
        }
        if (O.parent[v] == u) P.val[ko + v] = -2;
      }
    }
    if (!gridSync(c, epoch)) return;
    markPhase(c, kPhaseRoots);

    // ---- Subtree invalidation by pointer jumping (reference :254-291) -----
    // val[v] >= 0: no root on the tree path from v up to (excluding)
    // val[v]; -1: no root above v at all; -2: a root is v or an ancestor.
    // Every value another thread can observe keeps this invariant, so the
    // updates are made in place.
    if (changes > 0) {
      for (int round = 0; round < P.maxRounds; ++round) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
          c->jumpActive[(round + 1) % 3] = 0;
          c->rounds = round + 1;
        }
        int jumping = 0;
        for (int k = 0; k < K; ++k) {
          if (P.obj[k].nChanged == 0) continue;
          int *val = P.val + static_cast<long long>(k) * P.stride;
          // up to four jumps per round, each along the pointers the other
          // vertices have already lengthened, so a round covers more than
          // twice the distance and fewer rounds (and full scans) are needed
          // four vertices per thread (v, v + T, v + 2T, v + 3T) with their
          // chains of dependent loads in flight together
          for (long long v0 = tid; v0 < n; v0 += 4 * T) {
            int a[4], b[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const long long v = v0 + q * T;
              a[q] = v < n ? __ldcg(val + v) : -1;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) b[q] = a[q] >= 0 ? __ldcg(val + a[q]) : -1;
#pragma unroll
            for (int hop = 1; hop < 4; ++hop) {
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                if (a[q] >= 0 && b[q] >= 0) {
                  a[q] = b[q];
                  b[q] = __ldcg(val + a[q]);
                }
              }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              if (a[q] < 0) continue;  // no ancestor pointer (or past n)
              val[v0 + q * T] = b[q];
              jumping |= b[q] >= 0;
            }
          }
        }
        if (__syncthreads_or(jumping) && threadIdx.x == 0) {
          atomicOr(&c->jumpActive[round % 3], 1);
        }
        if (!gridSync(c, epoch)) return;
        if (__ldcg(&c->jumpActive[round % 3]) == 0) break;
        if (round + 1 == P.maxRounds && blockIdx.x == 0 && threadIdx.x == 0) {
          c->invalid = 1;  // the parent arrays are not a forest
        }
      }
    }

    markPhase(c, kPhaseJumped);
    // ---- Invalidate; candidates = invalidated + insert heads (:293-313) ---
    // (512 vertices at a time pay once every fourth warp has some)
    for (int k = 0; k < K; ++k) {
      if (n >= 4 * T) {
        collectInvalid<16>(P, k, tid >> 5, T >> 5);
      } else {
        collectInvalid<2>(P, k, tid >> 5, T >> 5);
      }
    }
    for (int k = 0; k < K; ++k) {
      const long long ko = static_cast<long long>(k) * P.stride;
      for (long long i = tid; i < P.nHeads; i += T) {
        const int v = P.heads[i];
        if (v < 0 || v >= n) {
          c->invalid = 1;
          continue;
        }
        if (isRoot(P.source, P.sources, P.nSources, v) || __ldcg(P.val + ko + v) == -2) continue;
        if (atomicExch(P.stamp + ko + v, genBase) != genBase) {
          const int idx = warpAppend(&c->candCount[k]);
          P.cand[ko + idx] = v;
        }
      }
    }
    if (!gridSync(c, epoch)) return;
    markPhase(c, kPhaseCandidates);

    // ---- Pull pass over in-edges (reference :315-344) ----------------------
    // The improved candidates form far pile 0; the first iteration of the
    // loop sets the threshold to their minimum + delta and splits them.
    //
    // Direction per objective: when more than half of the vertices were
    // invalidated, the few valid vertices push along all their out-edges
    // instead (pushFromValid below). That makes the same offers to the
    // invalidated vertices (their valid in-neighbours) and to the insert
    // heads (every inserted edge leaves a valid or an invalidated vertex, and
    // the latter is re-expanded in the loop anyway), for the out-edges of the
    // valid part instead of the in-edges of the invalidated part.
    __shared__ int sPush[kMaxK];
    if (threadIdx.x < kMaxK) {
      sPush[threadIdx.x] = static_cast<int>(threadIdx.x) < K && (P.flags & kFlagPullOnly) == 0 &&
                           2LL * __ldcg(&c->invalidated[threadIdx.x]) > n;
    }
    __syncthreads();
    {
      __shared__ long long sOff[kMaxK + 1];
      if (warp == 0) {
        const long long cnt =
            static_cast<int>(lane) < K && !sPush[lane] ? __ldcg(&c->candCount[lane]) : 0;
        long long incl = cnt;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const long long o = __shfl_up_sync(kFull, incl, off);
          if (static_cast<int>(lane) >= off) incl += o;
        }
        sOff[lane] = incl - cnt;
        if (lane == 31) sOff[kMaxK] = incl;
      }
      StageHeader &H = stageHeader();
      StageEntry *E = stageEntries();
      if (threadIdx.x < kMaxK) {
        H.count[threadIdx.x] = 0;
        H.farMin[threadIdx.x] = kInfWord;
      }
      if (threadIdx.x == 0) {
        H.cap = P.stageEntries / K;
        H.heavyCount = 0;
      }
      __syncthreads();
      const long long total = sOff[kMaxK];
      // set in the first phase, the same for every thread of the grid
      const bool heavyOn = __ldcg(&c->heavy) != 0;
      // Improved candidates go to far pile 0. With a partition of at least
      // one tile per objective (K * blockDim <= stage entries) the appends are
      // staged per CTA and written out with one reservation per objective
      // when a partition could fill up and at the end; otherwise each warp
      // appends to the global pile directly.
      const bool staged = K * static_cast<int>(blockDim.x) <= P.stageEntries;
      auto flushPull = [&]() {
        __syncthreads();
        if (threadIdx.x < K && H.count[threadIdx.x] > 0) {
          H.base[threadIdx.x] = atomicAdd(&c->farCount[threadIdx.x][0], H.count[threadIdx.x]);
          atomicMax(&c->farMinC[threadIdx.x][0], ~H.farMin[threadIdx.x]);
        }
        __syncthreads();
        for (int k = 0; k < K; ++k) {
          const int cnt = H.count[k];
          const long long ko = static_cast<long long>(k) * P.strideFar;
          for (int q = threadIdx.x; q < cnt; q += blockDim.x) {
            P.farL0[ko + H.base[k] + q] = E[k * H.cap + q].v;
          }
        }
        __syncthreads();
        if (threadIdx.x < kMaxK) {
          H.count[threadIdx.x] = 0;
          H.farMin[threadIdx.x] = kInfWord;
        }
        __syncthreads();
      };
      // The tiles of all CTAs are interleaved, so that few candidates spread
      // over the grid: by single candidates where the graph has hubs, whose
      // in-rows then meet different CTAs, else by 32, whose loads are one line.
      // Pull phase by CTA tiles, by 32 and by ones, us: R-MAT of 262,144
      // vertices, K = 4: 848 candidates 36, 28, 18; 52,582: 61, 46, 40; scale
      // 22, K = 5, 270,959: 121, 120, 115; road networks: 64 of 20,020
      // vertices, 1.3M candidates: 61, 50, 83; 640,000 vertices, 413,402: 46,
      // 43, 54; 93,300 vertices, 83,544: 9.9, 9.4, 11.1.
      const unsigned groupBits = heavyOn ? 0 : 5;
      const long long tileStride = static_cast<long long>(gridDim.x) * blockDim.x;
      for (long long tile = static_cast<long long>(blockIdx.x) * blockDim.x;
           tile - static_cast<long long>(blockIdx.x) * blockDim.x < total; tile += tileStride) {
        const long long j = tile - static_cast<long long>(blockIdx.x) * blockDim.x +
                            ((static_cast<long long>(threadIdx.x >> groupBits) * gridDim.x + blockIdx.x) << groupBits) +
                            (threadIdx.x & ((1u << groupBits) - 1u));
        const bool valid = j < total;
        int k = 0;
        if (valid) {
          while (k + 1 < K && sOff[k + 1] <= j) ++k;
        }
        const long long ko = static_cast<long long>(k) * P.stride;
        const ObjectiveArgs &O = P.obj[k];
        const Pk pk = pkOf(O);
        int v = -1, beg = 0, end = 0;
        u64 cur = kInfWord;
        if (valid) {
          v = __ldcg(P.cand + ko + (j - sOff[k]));
          cur = __ldcg(P.packed + ko + v);
          beg = __ldg(P.inRow + v);
          end = __ldg(P.inRow + v + 1);
        }
        // heavy in-rows are reduced by the whole CTA after the tile
        if (heavyOn && takesCta(P, H, end - beg)) {
          const int slot = atomicAdd(&H.heavyCount, 1);
          if (slot < kHeavyCap) {
            H.heavyK[slot] = k;
            H.heavyU[slot] = v;
            H.heavyBeg[slot] = beg;
            H.heavyDeg[slot] = end - beg;
            H.heavyD[slot] = cur;
            end = beg;
          }
        }
        u64 best = cur;
        const int deg = end - beg;
        unsigned big = __ballot_sync(kFull, deg > kLaneRowMax);
        if (deg <= kLaneRowMax) best = pullBest(P, O, pk, ko, beg, end, 1, best);
        while (big != 0) {
          const int src = __ffs(big) - 1;
          big &= big - 1;
          const int kb = __shfl_sync(kFull, k, src);
          const int bb = __shfl_sync(kFull, beg, src);
          const int eb = __shfl_sync(kFull, end, src);
          const ObjectiveArgs &Ob = P.obj[kb];
          const Pk pb = pkOf(Ob);
          const long long kob = static_cast<long long>(kb) * P.stride;
          u64 part = pullBest(P, Ob, pb, kob, bb + static_cast<int>(lane), eb, 32, kInfWord);
          part = warpMinU64(part);
          if (static_cast<int>(lane) == src) best = part < best ? part : best;
        }
        if (valid && best < cur) {
          // only this thread writes the word of v during the pull pass
          P.packed[ko + v] = best;
          if (pk.dist(best) < (cur == kInfWord ? kInfWord : pk.dist(cur))) {
            P.inFar[ko + v] = 1;
            if (!staged) {
              const int idx = warpAppend(&c->farCount[k][0]);
              P.farL0[static_cast<long long>(k) * P.strideFar + idx] = v;
              warpMinInto(&c->farMinC[k][0], pk.dist(best));
            } else {
              const unsigned peers = __match_any_sync(__activemask(), k);
              const int leader = __ffs(peers) - 1;
              int rb = 0;
              if (static_cast<int>(lane) == leader) rb = atomicAdd(&H.count[k], __popc(peers));
              rb = __shfl_sync(peers, rb, leader);
              E[k * H.cap + rb + __popc(peers & ((1u << lane) - 1u))].v = v;
              const u64 d = pk.dist(best);
              const unsigned hi = static_cast<unsigned>(d >> 32), lo = static_cast<unsigned>(d);
              const unsigned mhi = __reduce_min_sync(peers, hi);
              const unsigned mlo = __reduce_min_sync(peers, hi == mhi ? lo : 0xffffffffu);
              if (static_cast<int>(lane) == leader) {
                atomicMin(&H.farMin[k], (static_cast<u64>(mhi) << 32) | mlo);
              }
            }
          }
        }
        if (heavyOn) {
          // the tile's heavy in-rows: every thread of the CTA takes a share
          // of each row, the partial minima meet in shared memory, and one
          // thread per row writes the word and appends an improved vertex
          // to the global far pile (as the unstaged path does)
          __syncthreads();
          const int queued = H.heavyCount;
          if (queued > 0) {  // the same for every thread of the CTA
            const int count = queued < kHeavyCap ? queued : kHeavyCap;
            if (static_cast<int>(threadIdx.x) < count) H.heavyBest[threadIdx.x] = kInfWord;
            __syncthreads();
            if (threadIdx.x == 0) H.heavyCount = 0;
            for (int h = 0; h < count; ++h) {
              const int kh = H.heavyK[h], eh = H.heavyBeg[h] + H.heavyDeg[h];
              const ObjectiveArgs &Oh = P.obj[kh];
              const Pk ph = pkOf(Oh);
              const long long koh = static_cast<long long>(kh) * P.stride;
              u64 part = pullBest(P, Oh, ph, koh, H.heavyBeg[h] + static_cast<int>(threadIdx.x), eh,
                                  static_cast<int>(blockDim.x), kInfWord);
              part = warpMinU64(part);
              if (lane == 0 && part != kInfWord) atomicMin(&H.heavyBest[h], part);
            }
            __syncthreads();
            if (static_cast<int>(threadIdx.x) < count) {
              const int h = threadIdx.x;
              const int kh = H.heavyK[h], vh = H.heavyU[h];
              const Pk ph = pkOf(P.obj[kh]);
              const long long koh = static_cast<long long>(kh) * P.stride;
              const u64 curh = H.heavyD[h], besth = H.heavyBest[h];
              if (besth < curh) {
                // only this thread writes the word of vh during the pull pass
                P.packed[koh + vh] = besth;
                if (ph.dist(besth) < (curh == kInfWord ? kInfWord : ph.dist(curh))) {
                  P.inFar[koh + vh] = 1;
                  const int idx = atomicAdd(&c->farCount[kh][0], 1);
                  P.farL0[static_cast<long long>(kh) * P.strideFar + idx] = vh;
                  atomicMax(&c->farMinC[kh][0], ~ph.dist(besth));
                }
              }
            }
          }
          // every thread has read the queue (and the rows are done) before
          // the next tile queues rows again
          __syncthreads();
        }
        if (!staged) continue;
        // a tile appends at most blockDim entries: flush before a partition
        // could overflow
        __syncthreads();
        if (__syncthreads_or(threadIdx.x < static_cast<unsigned>(K) &&
                             H.count[threadIdx.x] > H.cap - static_cast<int>(blockDim.x))) {
          flushPull();
        }
      }
      if (staged) flushPull();
    }
    for (int k = 0; k < K; ++k) {
      if (sPush[k]) pushFromValid(P, k, sOutWk[k], tid >> 5, T >> 5);
    }
    if (!gridSync(c, epoch)) return;
    markPhase(c, kPhasePulled);
    if (!runNearFar<Mode>(P, outRow, outCol, sOutWk, epoch, nullptr, genBase, P.rec != nullptr)) return;
    markPhase(c, kPhaseLoop);
    unpackResults<Mode>(P, outRow, outCol, sOutWk, epoch);
    if (!gridSync(c, epoch)) return;
    markPhase(c, kPhaseEnd);
  } else {
    scratchOrCombined<Mode>(P, epoch, genBase, sOutWk);
  }
}

/// Steps 2-3 (combined mode) and the SSSP from scratch (both modes).
/// The combined edges into v of every tree at once, for combK <= 8: the K
/// parents are loaded once (combinedEdge reloads them per tree); has[k],
/// p[k] and w[k] are what combinedEdge(P, v, k, ...) gives.
__device__ __forceinline__ void combinedEdges8(const EngineParams &P, int v, int (&p)[8],
                                               int (&w)[8], bool (&has)[8]) {
  const long long n = P.n;
#pragma unroll
  for (int k = 0; k < 8; ++k) p[k] = k < P.combK ? __ldg(P.combParents + k * n + v) : -1;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    bool first = p[k] >= 0;
#pragma unroll
    for (int j = 0; j < k; ++j) first = first && p[j] != p[k];
    int weight = P.combBase - P.prefTerms[k];
#pragma unroll
    for (int j = k + 1; j < 8; ++j) {
      if (p[j] == p[k]) weight -= P.prefTerms[j];  // trees past combK hold -1
    }
    has[k] = first;
    w[k] = weight;
  }
}

template <int Mode>
__device__ void scratchOrCombined(const EngineParams &P, Sync &epoch, int genBase,
                                  const int **sOutWk) {
  EngineControl *c = P.ctl;
  const int n = P.n, K = P.K;
  const long long tid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long T = static_cast<long long>(gridDim.x) * blockDim.x;
  const unsigned lane = laneId();
  __shared__ u64 sCombDelta;
  const int *outRow = P.outRow;
  const int *outCol = P.outCol;

  if constexpr (Mode == kModeCombined) {
    // ---- Step 2: combined graph, count / scan / fill (reference
    // src/combinedGraphGpu.cu:80-121, 281-300), then Step 3 below --------
    for (long long v = tid; v <= n; v += T) P.combDeg[v] = 0;
    if (!gridSync(c, epoch)) return;
    // four vertices per thread (v, v + T, v + 2T, v + 3T) in the count and
    // fill passes, so their parent loads and atomics are in flight together
    unsigned long long edges = 0, wsum = 0;
    bool badParent = false;
    const bool regs = P.combK <= 8;  // the same for every thread
    for (long long v = tid; regs && v < n; v += T) {
      if (isRoot(P.source, P.sources, P.nSources, static_cast<int>(v))) continue;
      int p[8], w[8];
      bool has[8];
      combinedEdges8(P, static_cast<int>(v), p, w, has);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (!has[k]) continue;
        if (p[k] >= n) {
          badParent = true;
          continue;
        }
        atomicAdd(P.combDeg + p[k], 1);
        ++edges;
        wsum += static_cast<unsigned long long>(w[k]);
      }
    }
    for (long long v0 = tid; !regs && v0 < n; v0 += 4 * T) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const long long v = v0 + q * T;
        if (v >= n || isRoot(P.source, P.sources, P.nSources, static_cast<int>(v))) continue;
        for (int k = 0; k < P.combK; ++k) {
          int p, w;
          if (combinedEdge(P, static_cast<int>(v), k, p, w)) {
            if (p >= n) {
              badParent = true;
              continue;
            }
            atomicAdd(P.combDeg + p, 1);
            ++edges;
            wsum += static_cast<unsigned long long>(w);
          }
        }
      }
    }
    if (badParent) c->invalid = 1;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      edges += __shfl_down_sync(kFull, edges, off);
      wsum += __shfl_down_sync(kFull, wsum, off);
    }
    if (lane == 0 && edges > 0) {
      atomicAdd(&c->sums[0], edges);
      atomicAdd(&c->sums[1], wsum);
    }
    if (!gridSync(c, epoch)) return;
    long long totalEdges = 0;
    if (__ldcg(&c->invalid) != 0) return;
    // row starts; the degree array becomes the fill cursor (each CTA reads
    // and rewrites only its own chunk)
    if (!gridExclusiveScan(P.combDeg, P.combRow, P.combDeg, static_cast<long long>(n) + 1,
                           P.blockSums, c, epoch, &totalEdges)) {
      return;
    }
    if (!gridSync(c, epoch)) return;
    for (long long v = tid; regs && v < n; v += T) {
      if (isRoot(P.source, P.sources, P.nSources, static_cast<int>(v))) continue;
      int p[8], w[8];
      bool has[8];
      combinedEdges8(P, static_cast<int>(v), p, w, has);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (!has[k]) continue;
        const int pos = atomicAdd(P.combDeg + p[k], 1);
        P.combCol[pos] = static_cast<int>(v);
        P.combW[pos] = w[k];
      }
    }
    for (long long v0 = tid; !regs && v0 < n; v0 += 4 * T) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const long long v = v0 + q * T;
        if (v >= n || isRoot(P.source, P.sources, P.nSources, static_cast<int>(v))) continue;
        for (int k = 0; k < P.combK; ++k) {
          int p, w;
          if (combinedEdge(P, static_cast<int>(v), k, p, w)) {
            const int pos = atomicAdd(P.combDeg + p, 1);
            P.combCol[pos] = static_cast<int>(v);
            P.combW[pos] = w;
          }
        }
      }
    }
    if (threadIdx.x == 0) {
      // Default bucket width of the combined graph (reference
      // src/combinedGraphGpu.cu:310-312 and :607-616 of sospUpdateGpu.cu).
      u64 d = static_cast<u64>(P.combDelta);
      if (P.combDelta <= 0) {
        const double e = static_cast<double>(__ldcg(&c->sums[0]));
        const double ws = static_cast<double>(__ldcg(&c->sums[1]));
        long long dd = 1;
        if (e > 0 && n > 0) {
          dd = static_cast<long long>(32.0 * (ws / e) / (e / static_cast<double>(n)));
          if (dd < 1) dd = 1;
        }
        d = static_cast<u64>(dd);
      }
      sCombDelta = d;
    }
    outRow = P.combRow;
    outCol = P.combCol;
    if (threadIdx.x == 0) sOutWk[0] = P.combW;
    markPhase(c, kPhasePacked);
    // fall through to the SSSP from scratch
  }

  if constexpr (Mode == kModeScratch) {
    // The caller's CSR is checked before any access that it indexes: row
    // offsets monotone from 0 to m, every column in [0, n). A malformed graph
    // ends the launch with `invalid` set, before the relaxations.
    if (tid == 0 && (__ldg(outRow) != 0 || __ldg(outRow + n) != P.m)) c->invalid = 1;
    for (long long v = tid; v < n; v += T) {
      if (__ldg(outRow + v + 1) < __ldg(outRow + v)) c->invalid = 1;
    }
    for (long long e = tid; e < P.m; e += T) {
      const int x = __ldg(outCol + e);
      if (x < 0 || x >= n) c->invalid = 1;
    }
    if (!gridSync(c, epoch)) return;
    if (__ldcg(&c->invalid) != 0) return;
  }

  // ---- SSSP from scratch: only the source (the roots) is finite ------------
  bool heavyRow = false;  // one store at the end, so the loads run ahead
  for (long long v = tid; v < n; v += T) {
    heavyRow |= ldGraph<Mode>(outRow + v + 1) - ldGraph<Mode>(outRow + v) > heavyDegOf(P);
  }
  if (heavyRow) c->heavy = 1;
  __syncthreads();  // sOutWk
  // (of the combined graph only the kernel knows the edge count)
  bool rec = P.rec != nullptr;
  if constexpr (Mode == kModeCombined) {
    rec = rec && recordsPay(n, static_cast<long long>(__ldcg(&c->sums[0])));
    if (rec && !gridSync(c, epoch)) return;  // the rows are filled
  }
  if (rec) buildRecords<Mode>(P, outRow, outCol, sOutWk, tid, T);
  for (int k = 0; k < K; ++k) {
    const Pk pk = pkOf(P.obj[k]);
    const long long ko = static_cast<long long>(k) * P.stride;
    for (long long v = tid; v < n; v += T) {
      P.packed[ko + v] =
          isRoot(P.source, P.sources, P.nSources, static_cast<int>(v)) ? pk.pack(0, -1) : kInfWord;
    }
    const int roots = P.nSources > 1 ? P.nSources : 1;
    for (long long i = tid; i < roots; i += T) {
      const int r = P.nSources > 1 ? P.sources[i] : P.source;
      P.inFar[ko + r] = 1;
      P.farL0[static_cast<long long>(k) * P.strideFar + i] = r;
    }
    if (tid == 0) {
      c->farCount[k][0] = roots;
      c->farMinC[k][0] = ~0ULL;  // minimum 0
    }
  }
  if (!gridSync(c, epoch)) return;
  markPhase(c, kPhasePulled);
  u64 *deltaOverride = nullptr;
  if constexpr (Mode == kModeCombined) deltaOverride = &sCombDelta;
  if (!runNearFar<Mode>(P, outRow, outCol, sOutWk, epoch, deltaOverride, genBase, rec)) return;
  markPhase(c, kPhaseLoop);
  unpackResults<Mode>(P, outRow, outCol, sOutWk, epoch);
  if (!gridSync(c, epoch)) return;
  markPhase(c, kPhaseEnd);
}

// ---------------------------------------------------------------------------
// Device graph: objective-major weights and the reverse CSR (reference
// src/deviceGraph.cu:28-63, 87-135), one cooperative launch.
//
// Bound by the scattered traffic of the transposition: one returning atomic
// per edge (its rank among the edges into its head, kept, so that the fill
// needs no second atomic) and K + 1 scattered stores. Both passes are
// balanced over edges. (With rows dealt to warps, the
// one that held the low ids of an R-MAT graph walked most of its hubs: 3.9M
// edges, K = 4: 4.13 -> 0.36 ms; 16.1M, K = 3: 11.2 -> 1.8 ms; road network
// of 5.6M edges, K = 3: 0.24 -> 0.20 ms.)
//
// Once the reverse arrays outgrow L2, every scattered 4-byte store is a
// 32-byte sector read and written in HBM, K + 1 times per edge. There the
// scatter writes one number per edge, whose array stays in L2 for longer, and
// a second pass gathers the edge's K adjacent weights and stores in order:
// 3.9M edges, K = 4: 0.36 -> 0.30 ms; 16.1M, K = 3: 1.74 -> 0.95; 65M, K = 5:
// 18.3 -> 8.8. The rule's line: R-MAT graphs with K = 3 take 0.163 and 0.174 ms
// (direct, by order) at 31 MB of reverse arrays, 0.317 and 0.290 at 63 MB;
// 16.1M edges with K = 1 0.744 and 0.741; road networks, whose stores stay
// close, are the same within 2 % on either side.
// ---------------------------------------------------------------------------
constexpr long long kScatterBytes = 48LL << 20;

/// Ranked: B.rank is there.
template <bool Ranked>
__global__ void __launch_bounds__(kThreads, 1) buildGraph(const __grid_constant__ BuildParams B) {
  EngineControl *c = B.ctl;
  const int n = B.n, m = B.m, K = B.K;
  const long long tid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long T = static_cast<long long>(gridDim.x) * blockDim.x;
  const unsigned lane = laneId();
  const long long nwarps = T >> 5;
  Sync epoch = startSync(B.timeoutNs);

  // validate the row offsets; clear the degree counts
  bool bad = tid == 0 && (__ldg(B.outRow) != 0 || __ldg(B.outRow + n) != m);
  for (long long v = tid; v <= n; v += T) {
    bad |= v < n && __ldg(B.outRow + v + 1) < __ldg(B.outRow + v);
    B.cursor[v] = 0;
  }
  if (bad) c->invalid = 1;
  if (!gridSync(c, epoch)) return;

  // validate the heads; count them, keeping each edge's rank; split the
  // weights. Four edges per thread, so their atomics are in flight together.
  bad = false;
  for (long long e0 = tid; e0 < m; e0 += 4 * T) {
    int x[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const long long e = e0 + q * T;
      x[q] = e < m ? __ldg(B.outCol + e) : -1;
      if (e < m && (x[q] < 0 || x[q] >= n)) {
        bad = true;
        x[q] = -1;
      }
    }
    int r[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) r[q] = x[q] >= 0 ? atomicAdd(B.cursor + x[q], 1) : 0;
    for (int k = 0; k < K; ++k) {
      int w[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const long long e = e0 + q * T;
        w[q] = e < m ? __ldg(B.edgeMajorW + e * K + k) : 0;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const long long e = e0 + q * T;
        if (e < m) B.outW[static_cast<long long>(k) * m + e] = w[q];
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const long long e = e0 + q * T;
      if (Ranked && e < m) B.rank[e] = r[q];
    }
  }
  if (bad) c->invalid = 1;
  if (!gridSync(c, epoch)) return;
  if (__ldcg(&c->invalid) != 0) return;
  long long total = 0;
  if (!gridExclusiveScan(B.cursor, B.inRow, Ranked ? nullptr : B.cursor, static_cast<long long>(n) + 1, B.blockSums, c,
                         epoch, &total)) {
    return;
  }
  if (!gridSync(c, epoch)) return;

  // fill: edge e of row u goes to position rank[e] of its head's row, or
  // (byOrder) leaves its number there, and its row in place of the rank;
  // without ranks to the next position, by a second atomic
  const bool byOrder = Ranked && K > 1 && 4LL * m * (K + 1) > kScatterBytes;
  EdgeChunks chunks(m, tid >> 5, nwarps, &c->chunkNext);
  long long wb, we;
  int r0;
  while (chunks.take(B.outRow, n, wb, we, r0)) {
    for (long long e0 = wb; e0 < we; e0 += 32) {
      const long long e = e0 + lane;
      const bool in = e < we;
      const int x = in ? __ldg(B.outCol + e) : 0;
      int pos = 0;
      if constexpr (Ranked) {
        pos = in ? __ldcg(B.inRow + x) + __ldcg(B.rank + e) : 0;
      } else {
        pos = in ? atomicAdd(B.cursor + x, 1) : 0;
      }
      const int row = edgeRow(B.outRow, n, e, in, r0);
      if (!in) continue;
      if (byOrder) {
        B.inCol[pos] = static_cast<int>(e);
        B.rank[e] = row;
        continue;
      }
      B.inCol[pos] = row;
      for (int k = 0; k < K; ++k) {
        B.inW[static_cast<long long>(k) * m + pos] = __ldg(B.edgeMajorW + e * K + k);
      }
    }
  }
  if (!byOrder) return;
  if (!gridSync(c, epoch)) return;
  // the reverse rows in order, four edges per thread in flight
  for (long long i0 = tid; i0 < m; i0 += 4 * T) {
    int e[4], row[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) e[q] = i0 + q * T < m ? __ldcg(B.inCol + i0 + q * T) : 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) row[q] = __ldcg(B.rank + e[q]);
    for (int k = 0; k < K; ++k) {
      int w[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) w[q] = __ldg(B.edgeMajorW + static_cast<long long>(e[q]) * K + k);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (i0 + q * T < m) B.inW[static_cast<long long>(k) * m + i0 + q * T] = w[q];
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (i0 + q * T < m) B.inCol[i0 + q * T] = row[q];
    }
  }
}

// ---------------------------------------------------------------------------
// MOSP path costs: sums of the original weights along the MOSP tree by
// pointer jumping with double buffering (replaces the host BFS of
// reference src/combinedGraphGpu.cu:161-208; same edge rule: the first
// occurrence of v in row p).
// ---------------------------------------------------------------------------
__device__ __forceinline__ long long satAdd(long long a, long long b) {
  if (a >= kDistInf / 2 || b >= kDistInf / 2) return kDistInf;
  const long long s = a + b;
  return s >= kDistInf / 2 ? kDistInf : s;
}

__global__ void __launch_bounds__(kThreads, 1) pathCosts(const __grid_constant__ CostParams C) {
  EngineControl *c = C.ctl;
  const int n = C.n, KG = C.KG;
  const long long tid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long T = static_cast<long long>(gridDim.x) * blockDim.x;
  const unsigned lane = laneId();
  const long long nwarps = T >> 5;
  Sync epoch = startSync(C.timeoutNs);

  for (long long v = tid; v < n; v += T) C.edgeOf[v] = INT_MAX;
  if (!gridSync(c, epoch)) return;
  // first occurrence of the tree edge (parent[v], v): lowest e in row p
  {
    const long long m = __ldg(C.outRow + n);
    EdgeChunks chunks(m, tid >> 5, nwarps, &c->chunkNext);
    long long wb, we;
    int r0;
    while (chunks.take(C.outRow, n, wb, we, r0)) {
      for (long long e0 = wb; e0 < we; e0 += 32) {
        const bool valid = e0 + lane < we;
        const int e = static_cast<int>(e0 + lane);
        const int x = valid ? __ldg(C.outCol + e) : 0;
        const bool known = valid && static_cast<unsigned>(x) < static_cast<unsigned>(n);
        const int p = known ? __ldg(C.parent + x) : -1;
        const int row = edgeRow(C.outRow, n, e, valid, r0);
        if (known && p == row && row >= 0 && !isRoot(C.source, C.sources, C.nSources, x)) {
          atomicMin(C.edgeOf + x, e);
        }
      }
    }
  }
  if (!gridSync(c, epoch)) return;
  for (long long v = tid; v < n; v += T) {
    const int p = __ldg(C.parent + v);
    long long *acc = C.acc0 + v * KG;
    if (isRoot(C.source, C.sources, C.nSources, static_cast<int>(v))) {
      C.anc0[v] = -1;
      for (int k = 0; k < KG; ++k) acc[k] = 0;
    } else if (p < 0 || p >= n) {
      if (p >= n) c->invalid = 1;
      C.anc0[v] = -1;
      for (int k = 0; k < KG; ++k) acc[k] = kDistInf;
    } else {
      const int e = __ldcg(C.edgeOf + v);
      if (e == INT_MAX) {
        c->invalid = 1;  // the tree edge is not in the graph
        C.anc0[v] = -1;
        for (int k = 0; k < KG; ++k) acc[k] = kDistInf;
      } else {
        C.anc0[v] = p;
        for (int k = 0; k < KG; ++k) {
          acc[k] = __ldg(C.outW + static_cast<long long>(k) * C.m + e);
        }
      }
    }
  }
  if (!gridSync(c, epoch)) return;
  int round = 0;
  for (;; ++round) {
    const int *ancR = (round & 1) ? C.anc1 : C.anc0;
    int *ancW = (round & 1) ? C.anc0 : C.anc1;
    const long long *accR = (round & 1) ? C.acc1 : C.acc0;
    long long *accW = (round & 1) ? C.acc0 : C.acc1;
    if (blockIdx.x == 0 && threadIdx.x == 0) c->jumpActive[(round + 1) % 3] = 0;
    int active = 0;
    for (long long v = tid; v < n; v += T) {
      const int a = __ldcg(ancR + v);
      if (a >= 0) {
        const int b = __ldcg(ancR + a);
        for (int k = 0; k < KG; ++k) {
          accW[v * KG + k] = satAdd(__ldcg(accR + v * KG + k), __ldcg(accR + static_cast<long long>(a) * KG + k));
        }
        ancW[v] = b;
        active |= b >= 0;
      } else {
        for (int k = 0; k < KG; ++k) accW[v * KG + k] = __ldcg(accR + v * KG + k);
        ancW[v] = a;
      }
    }
    if (__syncthreads_or(active) && threadIdx.x == 0) atomicOr(&c->jumpActive[round % 3], 1);
    if (!gridSync(c, epoch)) return;
    if (__ldcg(&c->jumpActive[round % 3]) == 0 || round > 64) break;
  }
  const long long *accF = (round & 1) ? C.acc0 : C.acc1;
  for (long long i = tid; i < static_cast<long long>(n) * KG; i += T) {
    const long long x = __ldcg(accF + i);
    C.costs[i] = x >= kDistInf / 2 ? kDistInf : x;
  }
}

// ---------------------------------------------------------------------------
// Failure-path probe: every CTA but the first waits at a barrier that the
// first never reaches; the bounded wait must end with MOSP_ERR_TIMEOUT.
// ---------------------------------------------------------------------------
__global__ void barrierProbe(EngineControl *c, long long timeoutNs) {
  Sync epoch = startSync(timeoutNs);
  if (blockIdx.x == 0) return;
  gridSync(c, epoch);
}

/// Cost of the grid barrier alone: `rounds` barriers back to back; with
/// `reads`, every CTA also reads two control words after each barrier (the
/// loop's decision step). CTA 0 records the elapsed device time.
__global__ void barrierCost(EngineControl *c, int rounds, int reads, long long timeoutNs) {
  Sync epoch = startSync(timeoutNs);
  const unsigned long long t0 = globalNs();
  for (int r = 0; r < rounds; ++r) {
    if (reads && threadIdx.x < 32) {
      const int a = __ldcg(&c->nearCount[threadIdx.x & 7][r % 3]);
      const int b = __ldcg(&c->farCount[threadIdx.x & 7][r % 3]);
      if (a == 12345 && b == 678) c->invalid = 0;
    }
    if (!gridSync(c, epoch)) return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) c->phaseNs[0] = globalNs() - t0;
}

/// The parent recovery of an update launch that ran with kFlagHostRecovery,
/// as a kernel of its own: no shared-memory stage, so L1 keeps its full
/// size for the graph reads.
__global__ void __launch_bounds__(256) recoverParents(const __grid_constant__ EngineParams P) {
  __shared__ const int *sOutWk[kMaxK];
  if (P.recDist != nullptr && __ldcg(&P.ctl->recWide) == 0) return;  // recoverParents32 did it
  if (threadIdx.x < kMaxK) {
    sOutWk[threadIdx.x] =
        static_cast<int>(threadIdx.x) < P.K ? P.obj[threadIdx.x].outW : nullptr;
  }
  __syncthreads();
  const long long tid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long T = static_cast<long long>(gridDim.x) * blockDim.x;
  recoverTightParents<kModeUpdate>(P, P.outRow, P.outCol, sOutWk, tid, T);
}

/// The same recovery with the distances of up to 4 V objectives side by side
/// in 32 bits (every finite one is below 2^31, so a sum with a weight is
/// exact): edge (u, x) gathers one sector for x where the objectives' own
/// arrays take one each, and warps take chunks on demand. Bound by the
/// gathers (a wavefront of L1 per edge) and the streams of heads and weights,
/// which are read past L2's lasting part to leave it to the distances: 65M
/// edges of an R-MAT graph of scale 22, K = 5: 2.89 -> 1.07 ms (2.05 with
/// equal slices).
template <int V>
__global__ void __launch_bounds__(256) recoverParents32(const __grid_constant__ EngineParams P) {
  __shared__ int sFall[kMaxK];
  __shared__ int sCount;
  if (__ldcg(&P.ctl->recWide) != 0) return;
  if (threadIdx.x == 0) sCount = fallbackObjectives(P, sFall);
  __syncthreads();
  const int n = P.n;
  const unsigned lane = laneId();
  const long long m = __ldg(P.outRow + n);
  const long long tid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  EdgeChunks chunks(m, tid >> 5, (static_cast<long long>(gridDim.x) * blockDim.x) >> 5, &P.ctl->chunkNext);
  long long wb, we;
  int first;
  while (chunks.take(P.outRow, n, wb, we, first)) {
    for (int g0 = 0; g0 < sCount; g0 += 4 * V) {
      const int4 *dist = P.recDist + static_cast<long long>(g0 / 8) * 2 * n;
      const int count = sCount - g0 < 4 * V ? sCount - g0 : 4 * V;
      int r0 = first;
      for (long long e0 = wb; e0 < we; e0 += 32) {
        const long long e = e0 + lane;
        const bool in = e < we;
        const int x = in ? __ldcs(P.outCol + e) : 0;
        int4 dx[V];
#pragma unroll
        for (int i = 0; i < V; ++i) dx[i] = __ldg(dist + static_cast<long long>(V) * x + i);
        int w[4 * V];
#pragma unroll
        for (int j = 0; j < 4 * V; ++j) {
          w[j] = in && j < count ? __ldcs(P.obj[sFall[g0 + j]].outW + e) : 0;
        }
        const int row = edgeRow(P.outRow, n, e, in, r0);
        if (!in || row < 0) continue;
        int4 du[V];
#pragma unroll
        for (int i = 0; i < V; ++i) du[i] = __ldg(dist + static_cast<long long>(V) * row + i);
#pragma unroll
        for (int j = 0; j < 4 * V; ++j) {
          if (j >= count) break;
          const int4 a = du[j / 4], b = dx[j / 4];
          const unsigned from =
              static_cast<unsigned>(j % 4 == 0 ? a.x : j % 4 == 1 ? a.y : j % 4 == 2 ? a.z : a.w);
          const unsigned to =
              static_cast<unsigned>(j % 4 == 0 ? b.x : j % 4 == 1 ? b.y : j % 4 == 2 ? b.z : b.w);
          // (roots hold parent -1, which no id lowers; ~0 is no sum)
          if (from != ~0u && from + static_cast<unsigned>(w[j]) == to) {
            atomicMin(P.obj[sFall[g0 + j]].parent + x, row);
          }
        }
      }
    }
  }
}

template <typename Kernel>
cudaError_t ctasFor(Kernel kernel, int sms, int ctasPerSm, int &ctas, size_t smem = 0) {
  int perSm = 0;
  if (smem > 0) {
    cudaError_t a = cudaFuncSetAttribute(reinterpret_cast<const void *>(kernel),
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem));
    if (a != cudaSuccess) return a;
  }
  cudaError_t err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kernel, kThreads, smem);
  if (err != cudaSuccess) return err;
  if (perSm < 1) return cudaErrorInvalidConfiguration;
  if (ctasPerSm > 0 && ctasPerSm < perSm) perSm = ctasPerSm;
  ctas = perSm * sms;
  return cudaSuccess;
}

}  // namespace

cudaError_t queryLaunchShape(int ctasPerSm, LaunchShape &shape) {
  int device = 0, sms = 0, coop = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err == cudaSuccess) err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (err == cudaSuccess) err = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device);
  if (err != cudaSuccess) return err;
  if (!coop) return cudaErrorNotSupported;
  int a = 0, b = 0, d = 0, e = 0;
  if ((err = ctasFor(sospEngine<kModeUpdate>, sms, ctasPerSm, a, kStageBytes)) != cudaSuccess) return err;
  if ((err = ctasFor(sospEngine<kModeScratch>, sms, ctasPerSm, b, kStageBytes)) != cudaSuccess) return err;
  if ((err = ctasFor(sospEngine<kModeCombined>, sms, ctasPerSm, d, kStageBytes)) != cudaSuccess) return err;
  shape.engineCtas = a < b ? (a < d ? a : d) : (b < d ? b : d);
  if ((err = ctasFor(buildGraph<true>, sms, ctasPerSm, e)) != cudaSuccess) return err;
  if ((err = ctasFor(buildGraph<false>, sms, ctasPerSm, a)) != cudaSuccess) return err;
  shape.buildCtas = a < e ? a : e;
  if ((err = ctasFor(pathCosts, sms, ctasPerSm, e)) != cudaSuccess) return err;
  shape.costCtas = e;
  return applyFusedShape(sms, ctasPerSm, shape.applyCtas);
}

cudaError_t launchEngine(const EngineParams &p, int ctas, cudaStream_t s) {
  void *args[] = {const_cast<EngineParams *>(&p)};
  const void *fn = nullptr;
  switch (p.mode) {
    case kModeUpdate: fn = reinterpret_cast<const void *>(sospEngine<kModeUpdate>); break;
    case kModeScratch: fn = reinterpret_cast<const void *>(sospEngine<kModeScratch>); break;
    default: fn = reinterpret_cast<const void *>(sospEngine<kModeCombined>); break;
  }
  return cudaLaunchCooperativeKernel(fn, dim3(ctas), dim3(kThreads), args,
                                     stageBytesFor(p.stageEntries), s);
}

bool needsHostRecovery(const EngineParams &p) {
  if (p.mode != kModeUpdate) return false;
  for (int k = 0; k < p.K; ++k) {
    if (p.obj[k].parentBits == 0) return true;
  }
  return false;
}

cudaError_t launchRecovery(const EngineParams &p, cudaStream_t s) {
  int device = 0, sms = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err == cudaSuccess) err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (err != cudaSuccess) return err;
  if ((p.flags & kFlagCanonical) != 0 && p.recMark != nullptr) {
    return launchRestrictedRecovery(p, sms, s);
  }
  if (p.recDist != nullptr) {
    int count = 0;
    for (int k = 0; k < p.K; ++k) count += p.obj[k].parentBits == 0;
    if (count <= 4) {
      recoverParents32<1><<<sms * 8, 256, 0, s>>>(p);
    } else {
      recoverParents32<2><<<sms * 8, 256, 0, s>>>(p);
    }
    if ((err = cudaGetLastError()) != cudaSuccess) return err;
  }
  recoverParents<<<sms * 8, 256, 0, s>>>(p);
  return cudaGetLastError();
}

cudaError_t launchEngineEx(const EngineParams &p, int ctas, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = stageBytesFor(p.stageEntries);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  switch (p.mode) {
    case kModeUpdate: return cudaLaunchKernelEx(&cfg, sospEngine<kModeUpdate>, p);
    case kModeScratch: return cudaLaunchKernelEx(&cfg, sospEngine<kModeScratch>, p);
    default: return cudaLaunchKernelEx(&cfg, sospEngine<kModeCombined>, p);
  }
}

cudaError_t launchBuild(const BuildParams &p, int ctas, cudaStream_t s) {
  void *args[] = {const_cast<BuildParams *>(&p)};
  const void *fn = p.rank != nullptr ? reinterpret_cast<const void *>(buildGraph<true>)
                                     : reinterpret_cast<const void *>(buildGraph<false>);
  return cudaLaunchCooperativeKernel(fn, dim3(ctas), dim3(kThreads), args, 0, s);
}

cudaError_t launchCosts(const CostParams &p, int ctas, cudaStream_t s) {
  void *args[] = {const_cast<CostParams *>(&p)};
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(pathCosts), dim3(ctas),
                                     dim3(kThreads), args, 0, s);
}

cudaError_t launchBarrierCost(EngineControl *ctl, int rounds, int reads, long long timeoutNs,
                              int ctas, cudaStream_t s) {
  void *args[] = {&ctl, &rounds, &reads, &timeoutNs};
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(barrierCost), dim3(ctas),
                                     dim3(kThreads), args, 0, s);
}

cudaError_t launchBarrierProbe(EngineControl *ctl, long long timeoutNs, int ctas,
                               cudaStream_t s) {
  void *args[] = {&ctl, &timeoutNs};
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(barrierProbe), dim3(ctas),
                                     dim3(kThreads), args, 0, s);
}

}  // namespace mospb200

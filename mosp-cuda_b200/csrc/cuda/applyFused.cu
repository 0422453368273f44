// applyFused.cu - Step 1 on the GPU in one cooperative launch, for batches of
// up to kFusedBatch changes (larger ones: the sorted form in apply.cu, which
// states the semantics both follow).
//
// The sorted form pays for its launches: two radix sorts and half a dozen
// scans are some 75 launches and four read-backs. Here the changes of a (u,v)
// group meet in a hash table instead of a sort, and every per-group quantity
// of the rules does not depend on the order in which they arrive:
//   deletions and insertions of the group: counts;
//   its first and last insertion: minimum and maximum of file positions;
//   occurrences of v in row u and the first one: count and minimum over the
//   row's edges.
// Order matters in two places. A live edge moves by the edges appended less
// those removed before it, in whatever row: each block of 32 edges has the sum
// up to its first edge (a scan of the groups' changes) and bits for the changes
// inside it. Only a block with several edges appended at one place goes by its
// rows. The place of an appended edge is the number of appended groups of its
// row with an earlier first insertion: counted over the row's own list, or,
// where a row takes more than a sixteenth of a batch of more than 8,192
// insertions, over bits by file position (200,000 edges appended to one row:
// 1.16 ms, by lists alone 8.8, sorted form 6.3). Either costs the square of the
// insertions into one row, which sets kFusedBatch. Like the sorted form, one
// lane walks the row of a group that touches more than one of its parallel
// edges, from the first of them to the last it touches, 16 heads at a time (two
// edges 100,000 apart: 2.0 ms, head by head 11.4, sorted form 9.3; 1,000
// deletions of one edge: 0.11 ms, with an atomic each 0.56, sorted form 0.43).
//
// The copy is one pass over all edges: a warp takes 128 of them, which need no
// row, and moves their heads and their 128 K weights as one consecutive range
// each, so loads and stores coalesce whatever K is, eight weights per lane in
// flight; the weight statistics are taken from the same loads. Bound by HBM:
// the graph read and written once (2.6 TB/s of both on 65M edges; searching
// the rows of 32 edges at a time instead, 1.4).
//
// Measured on a B200, sorted form and this one: 50,000 changes on a road
// network of 5.56M edges, K = 3 (178 MB read and written): 578 -> 145 us;
// 24 changes on 4,200 edges: 307 -> 78 us; 20,000 on an R-MAT graph of 3.9M
// edges, K = 4: 2112 -> 171 us; 60,000 on one of 65M, K = 5: 12.8 -> 1.2 ms.
#include <cuda_runtime.h>

#include <algorithm>

#include "device.h"

namespace mospb200 {
namespace {

constexpr u64 kNoKey = ~0ULL;
constexpr int kLaneRow = 16;  // touched rows of at most so many edges are searched by one lane,
constexpr int kPiece = 64;    // longer ones in pieces of so many by a warp each
constexpr int kWalk = 16;     // heads in flight on the walk to a group's next parallel edge
constexpr int kCopyThreads = 256;
constexpr int kCopyEdges = 128;  // edges a warp of the copy takes at a time
constexpr int kTurns = 8;        // turns of its weights in flight
constexpr int kMarkRows = 16;    // rows with bits of their own: more than one in so many of the insertions,
constexpr int kMarkLeast = 8192;  // in batches of more than so many
constexpr unsigned kByRows = ~0U;  // Block::app: more than one edge appended at one place
constexpr int kNoMove = INT_MIN;
constexpr int kMaxCtas = 2048;
constexpr int kCounts = 5;  // FusedScratch::counts

/// What moves 32 consecutive edges of the old graph.
struct alignas(16) Block {
  int shift;      // how far the first one moves (the scan of its changes)
  unsigned dead;  // edges that go: those behind them move one less
  unsigned app;   // edges before which one is appended: they move one more
  unsigned other;  // edges that take an insertion's weights
};

struct FusedScratch {
  // groups: a hash table of `slots` (a power of two, at least twice the batch)
  u64 *key;  // u << 32 | v
  int *cD, *cI, *firstIns, *lastIns, *occ, *first;
  unsigned *bits;
  unsigned slots;
  unsigned *filter;  // filterBits bits, set where a group hashes: 16 or more per group for up to
                     // 65,536 changes, no fewer than 4 past that (128 KB: what L1 holds)
  unsigned filterBits;
  int *entrySlot;  // slot of batch entry j (deletions first)
  // touched rows, in no order
  int *rows, *nApp, *segApp, *curApp;
  int *markOf;      // of a row that many edges are appended to: its bits, else -1
  unsigned *marks;  // kMarkRows rows of markWords: a bit per insertion whose group appends
  int markWords;    // (a multiple of 4; 0: no such rows)
  u64 *pieces;     // of the longer touched rows: vertex << 32 | piece
  Block *block;    // per 32 edges, and one behind them
  int *app;        // insertions that append, by row segment
  int2 *other;     // edges that take an insertion's weights: edge, slot
  // per vertex: touched row + 1 (0: none), and its change of degree
  int *rowSlot, *delta;
  int *counts;     // touched rows, pieces, appended, edges with an insertion's weights, rows with bits
  long long *blockSums;  // of the CTAs: degree changes, then (moveSums) block moves
  long long *moveSums;
  FusedResult *result;
};

/// The 64-bit finaliser of MurmurHash3 (public domain), to spread the ids.
__device__ __forceinline__ unsigned hashOf(u64 key) {
  key ^= key >> 33;
  key *= 0xff51afd7ed558ccdULL;
  key ^= key >> 33;
  key *= 0xc4ceb9fe1a85ec53ULL;
  key ^= key >> 33;
  return static_cast<unsigned>(key);
}

/// The filter bit of a key with this hash.
__device__ __forceinline__ unsigned filterBit(const FusedScratch &S, unsigned hash) {
  return (hash >> 9) & (S.filterBits - 1);
}

/// Edges b, b + step, ... (< end) of touched row u: occurrences of their
/// groups. Four at a time, their loads and probes in flight together. (Edges
/// past the end of a row count up to 2^31 + 127: unsigned.)
__device__ __forceinline__ void countOccurrences(const ApplyParams &P, const FusedScratch &S, int u, unsigned b,
                                                 unsigned end, unsigned step) {
  for (unsigned e0 = b; e0 < end; e0 += 4 * step) {
    u64 key[4], at[4];
    unsigned s[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const unsigned e = e0 + q * step;
      key[q] = (static_cast<u64>(static_cast<unsigned>(u)) << 32) |
               static_cast<unsigned>(e < end ? __ldg(P.col + e) : -1);
      s[q] = hashOf(key[q]);
    }
    // most edges of a touched row are in no group: the filter says so from L1
    // (a plain load: nothing writes it after the barrier before this phase)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const unsigned f = filterBit(S, s[q]);
      at[q] = e0 + q * step < end && ((S.filter[f >> 5] >> (f & 31u)) & 1u) ? 0 : kNoKey;
      s[q] &= S.slots - 1;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (at[q] == 0) at[q] = __ldcg(S.key + s[q]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      while (at[q] != key[q] && at[q] != kNoKey) {
        s[q] = (s[q] + 1) & (S.slots - 1);
        at[q] = __ldcg(S.key + s[q]);
      }
      if (at[q] == kNoKey) continue;
      const unsigned e = e0 + q * step;
      atomicAdd(S.occ + s[q], 1);
      atomicMin(S.first + s[q], static_cast<int>(e));
    }
  }
}

/// Sum of x over the lanes before this one; the warp's sum in `total`.
__device__ __forceinline__ int warpExclusive(int x, int &total) {
  int incl = x;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int o = __shfl_up_sync(kFull, incl, off);
    if (static_cast<int>(laneId()) >= off) incl += o;
  }
  total = __shfl_sync(kFull, incl, 31);
  return incl - x;
}

/// Room for x entries per lane behind one counter, one atomic for the warp.
/// All lanes call it.
__device__ __forceinline__ int warpReserve(int *counter, int x) {
  int total;
  const int before = warpExclusive(x, total);
  int base = 0;
  if (laneId() == 0 && total > 0) base = atomicAdd(counter, total);
  return __shfl_sync(kFull, base, 0) + before;
}

/// One group of the batch: the change of its row's degree, the edges it
/// removes and appends as moves of the edges behind them, the list size of
/// its row, its weight-increase mask, and the edge (other) that takes its last
/// insertion's weights.
__device__ __forceinline__ void resolveGroup(const ApplyParams &P, const FusedScratch &S, int s, u64 key,
                                             int &other) {
  const int u = static_cast<int>(key >> 32), v = static_cast<int>(key);
  const int occ = __ldcg(S.occ + s), cD = __ldcg(S.cD + s), cI = __ldcg(S.cI + s);
  const int removed = occ < cD ? occ : cD;
  const int appended = occ <= cD && cI > 0 ? 1 : 0;
  if (appended) {
    const int r = __ldcg(S.rowSlot + u) - 1;
    atomicAdd(S.nApp + r, 1);
    const unsigned e = __ldg(P.row + u + 1);
    atomicAdd(&S.block[(e + 31) >> 5].shift, 1);
    if ((e & 31) != 0) {
      const unsigned bit = 1u << (e & 31);
      if (atomicOr(&S.block[e >> 5].app, bit) & bit) atomicOr(&S.block[e >> 5].app, kByRows);
    }
  }
  if (appended != removed) atomicAdd(S.delta + u, appended - removed);
  // the first `removed` occurrences go; the next one takes the weights
  const int seen = removed + (cI > 0 && occ > cD ? 1 : 0);
  const unsigned end = static_cast<unsigned>(__ldg(P.row + u + 1));
  unsigned e0 = static_cast<unsigned>(__ldcg(S.first + s));
  for (int i = 0; i < seen && e0 < end; e0 += kWalk) {
    int head[kWalk];
#pragma unroll
    for (int q = 0; q < kWalk; ++q) head[q] = e0 + q < end && (q == 0 || seen > 1) ? __ldg(P.col + e0 + q) : -1;
    unsigned hits = 0;
#pragma unroll
    for (int q = 0; q < kWalk; ++q) hits |= (head[q] == v ? 1u : 0u) << q;
    unsigned gone = hits;
    for (int left = __popc(hits); left > removed - i; --left) gone &= ~(0x80000000u >> __clz(gone));
    if (gone != 0) {
      // (the block of e0 and the next one)
      const u64 dead = static_cast<u64>(gone) << (e0 & 31u);
      Block *b = S.block + (e0 >> 5);
      const unsigned lo = static_cast<unsigned>(dead), hi = static_cast<unsigned>(dead >> 32);
      if (lo != 0) {
        atomicOr(&b[0].dead, lo);
        atomicAdd(&b[1].shift, -__popc(lo));
      }
      if (hi != 0) {
        atomicOr(&b[1].dead, hi);
        atomicAdd(&b[2].shift, -__popc(hi));
      }
      i += __popc(gone);
    }
    if (hits != gone && i < seen) {
      other = static_cast<int>(e0) + __ffs(hits ^ gone) - 1;
      atomicOr(&S.block[other >> 5].other, 1u << (other & 31));
      ++i;
    }
  }
  if (cI > 0 && occ > 0) {
    const int *wn = P.insW + static_cast<long long>(__ldcg(S.lastIns + s)) * P.K;
    const int *wo = P.w + static_cast<long long>(__ldcg(S.first + s)) * P.K;
    unsigned bits = 0;
    for (int k = 0; k < P.K; ++k) bits |= (wn[k] > wo[k] ? 1u : 0u) << k;
    S.bits[s] = bits;
  }
}

__global__ void __launch_bounds__(kThreads, 1)
applyFused(const __grid_constant__ ApplyParams P, const __grid_constant__ FusedScratch S, EngineControl *c,
           long long timeoutNs) {
  const int n = static_cast<int>(P.n), m = static_cast<int>(P.m);
  const long long tid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long T = static_cast<long long>(gridDim.x) * blockDim.x;
  const unsigned lane = laneId();
  const int B = P.nDel + P.nIns;
  Sync epoch = startSync(timeoutNs);

  // ---- clear ---------------------------------------------------------------
  for (long long v = tid; v < n + 4; v += T) {
    S.rowSlot[v] = 0;
    S.delta[v] = 0;
  }
  for (long long s = tid; s < S.slots; s += T) {
    S.key[s] = kNoKey;
    S.cD[s] = S.cI[s] = S.occ[s] = 0;
    S.firstIns[s] = S.first[s] = INT_MAX;
    S.lastIns[s] = -1;
    S.bits[s] = 0;
  }
  for (long long i = tid; i <= (m + 31LL) / 32; i += T) S.block[i] = Block{0, 0, 0, 0};
  for (long long i = tid; i < S.filterBits / 32; i += T) S.filter[i] = 0;
  for (long long i = tid; i < static_cast<long long>(kMarkRows) * S.markWords; i += T) S.marks[i] = 0;
  for (long long r = tid; r < B; r += T) S.nApp[r] = S.curApp[r] = 0;
  if (tid < kCounts) S.counts[tid] = 0;
  if (tid < kMaxK) {
    S.result->maxWeight[tid] = 1;
    S.result->weightSum[tid] = 0;
  }
  if (!gridSync(c, epoch)) return;

  // ---- groups and touched rows ---------------------------------------------
  for (long long j0 = tid - lane; j0 < B; j0 += T) {  // the same j0 in the whole warp
    const long long j = j0 + lane;
    const bool del = j < P.nDel;
    const int i = static_cast<int>(del ? j : j - P.nDel);
    int u = -1, v = -1;
    if (j < B) {
      u = del ? P.delFrom[i] : P.insFrom[i];
      v = del ? P.delTo[i] : P.insTo[i];
      if (u < 0 || u >= n || v < 0 || v >= n) {
        c->invalid = 1;
        u = -1;
      }
    }
    bool newRow = false;
    if (u >= 0) {
      const u64 key = (static_cast<u64>(static_cast<unsigned>(u)) << 32) | static_cast<unsigned>(v);
      const unsigned hash = hashOf(key), f = filterBit(S, hash);
      atomicOr(S.filter + (f >> 5), 1u << (f & 31u));
      unsigned s = hash & (S.slots - 1);
      while (true) {
        const u64 old = atomicCAS(S.key + s, kNoKey, key);
        if (old == kNoKey || old == key) break;
        s = (s + 1) & (S.slots - 1);
      }
      S.entrySlot[j] = static_cast<int>(s);
      if (del) {
        atomicAdd(S.cD + s, 1);
      } else {
        atomicAdd(S.cI + s, 1);
        atomicMin(S.firstIns + s, i);
        atomicMax(S.lastIns + s, i);
      }
      newRow = atomicCAS(S.rowSlot + u, 0, -1) == 0;
    }
    const int r = warpReserve(S.counts + 0, newRow ? 1 : 0);
    const int deg = newRow ? __ldg(P.row + u + 1) - __ldg(P.row + u) : 0;
    const int mine = deg > kLaneRow ? static_cast<int>((deg + kPiece - 1u) / kPiece) : 0;
    const int at = warpReserve(S.counts + 1, mine);
    if (newRow) {
      S.rows[r] = u;
      S.rowSlot[u] = r + 1;
      for (int p = 0; p < mine; ++p) S.pieces[at + p] = (static_cast<u64>(u) << 32) | static_cast<unsigned>(p);
    }
  }
  if (!gridSync(c, epoch)) return;
  if (__ldcg(&c->invalid) != 0) return;

  // ---- occurrences: a lane per short touched row (a lane of every warp
  // before a second one of any), a warp per piece of a longer one
  const int R = __ldcg(S.counts + 0);
  const long long warps = T >> 5;
  for (long long r = (tid >> 5) + lane * warps; r < R; r += T) {
    const int u = __ldcg(S.rows + r);
    const int b = __ldg(P.row + u), end = __ldg(P.row + u + 1);
    if (end - b <= kLaneRow) countOccurrences(P, S, u, b, end, 1);
  }
  const int pieces = __ldcg(S.counts + 1);
  for (long long i = tid >> 5; i < pieces; i += warps) {
    const u64 piece = __ldcg(S.pieces + i);
    const int u = static_cast<int>(piece >> 32);
    const int b = __ldg(P.row + u) + static_cast<int>(piece) * kPiece;
    const int end = __ldg(P.row + u + 1);
    countOccurrences(P, S, u, b + lane, end - b < kPiece ? end : b + kPiece, 32);
  }
  if (!gridSync(c, epoch)) return;

  // ---- groups resolved: degrees, what moves edges, list sizes, weight-
  // increase masks
  for (long long s0 = tid - lane; s0 < S.slots; s0 += T) {
    const long long s = s0 + lane;
    const u64 key = s < S.slots ? __ldcg(S.key + s) : kNoKey;
    int other = -1;  // the group's edge that takes the last insertion's weights
    if (key != kNoKey) resolveGroup(P, S, static_cast<int>(s), key, other);
    const int at = warpReserve(S.counts + 3, other >= 0 ? 1 : 0);
    if (other >= 0) S.other[at] = make_int2(other, static_cast<int>(s));
  }
  if (!gridSync(c, epoch)) return;
  // ---- row segments of the lists; masks; sums of the degree changes --------
  for (long long q0 = tid - lane; q0 < R; q0 += T) {
    const long long r = q0 + lane;
    const int count = r < R ? __ldcg(S.nApp + r) : 0;
    const int a = warpReserve(S.counts + 2, count);
    if (r < R) {
      S.segApp[r] = a;
      S.markOf[r] = S.markWords > 0 && count > P.nIns / kMarkRows ? atomicAdd(S.counts + 4, 1) : -1;
    }
  }
  for (long long i = tid; i < P.nIns; i += T) P.mask[i] = __ldcg(S.bits + S.entrySlot[P.nDel + i]);
  // (a CTA's range in whole groups of four vertices)
  const long long per = ((static_cast<long long>(n) + gridDim.x - 1) / gridDim.x + 3) / 4 * 4;
  const long long lo = per * blockIdx.x < n ? per * blockIdx.x : n;
  const long long hi = lo + per < n ? lo + per : n;
  // (and of the blocks)
  const long long blocks = (m + 31LL) / 32;
  const long long bPer = (blocks + gridDim.x - 1) / gridDim.x;
  const long long bLo = bPer * blockIdx.x < blocks ? bPer * blockIdx.x : blocks;
  const long long bHi = bLo + bPer < blocks ? bLo + bPer : blocks;
  {
    long long local = 0;
    for (long long v = lo + 4LL * threadIdx.x; v < hi; v += 4LL * blockDim.x) {
      const int4 d = __ldcg(reinterpret_cast<const int4 *>(S.delta + v));  // (zeros past n)
      local += d.x + d.y + d.z + d.w;
    }
    const long long sum = blockSum(local);
    local = 0;
    for (long long b = bLo + threadIdx.x; b < bHi; b += blockDim.x) local += __ldcg(&S.block[b].shift);
    const long long moves = blockSum(local);
    if (threadIdx.x == 0) {
      S.blockSums[blockIdx.x] = sum;
      S.moveSums[blockIdx.x] = moves;
    }
  }
  if (!gridSync(c, epoch)) return;

  // ---- lists; new row offsets ----------------------------------------------
  for (long long s = tid; s < S.slots; s += T) {
    const u64 key = __ldcg(S.key + s);
    if (key == kNoKey) continue;
    const int occ = __ldcg(S.occ + s), cD = __ldcg(S.cD + s);
    if (occ <= cD && __ldcg(S.cI + s) > 0) {
      const int r = __ldcg(S.rowSlot + static_cast<int>(key >> 32)) - 1;
      const int i = __ldcg(S.firstIns + s), segment = __ldcg(S.segApp + r), bits = __ldcg(S.markOf + r);
      S.app[segment + atomicAdd(S.curApp + r, 1)] = i;
      if (bits >= 0) atomicOr(S.marks + static_cast<long long>(bits) * S.markWords + (i >> 5), 1u << (i & 31));
    }
  }
  {
    long long before = 0, all = 0;
    for (int b = threadIdx.x; b < static_cast<int>(gridDim.x); b += blockDim.x) {
      const long long x = __ldcg(S.blockSums + b);
      all += x;
      if (b < static_cast<int>(blockIdx.x)) before += x;
    }
    long long carry = blockSum(before);
    all = blockSum(all);
    for (long long t = lo; t < hi; t += 4LL * blockDim.x) {
      const long long v = t + 4LL * threadIdx.x;
      int4 d = make_int4(0, 0, 0, 0);
      if (v < hi) d = __ldcg(reinterpret_cast<const int4 *>(S.delta + v));
      const long long x = d.x + d.y + d.z + d.w;
      long long tile;
      long long run = carry + blockInclusiveScan(x, &tile) - x;
      const int step[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (v + q < hi) P.newRow[v + q] = static_cast<int>(__ldg(P.row + v + q) + run);
        run += step[q];
      }
      carry += tile;
    }
    if (tid == 0) {
      P.newRow[n] = static_cast<int>(m + all);
      S.result->newM = static_cast<int>(m + all);
    }
  }
  // ---- where the blocks of the copy begin -----------------------------------
  {
    long long before = 0;
    for (int b = threadIdx.x; b < static_cast<int>(blockIdx.x); b += blockDim.x) before += __ldcg(S.moveSums + b);
    long long carry = blockSum(before);
    for (long long t = bLo; t < bHi; t += blockDim.x) {
      const long long b = t + threadIdx.x;
      long long tile;
      const long long incl = carry + blockInclusiveScan(b < bHi ? __ldcg(&S.block[b].shift) : 0, &tile);
      if (b < bHi) S.block[b].shift = static_cast<int>(incl);
      carry += tile;
    }
  }
}

/// How far edge e of row u moves, where its block is one that goes by rows.
__device__ __forceinline__ int moveByRow(const ApplyParams &P, const Block &B, int u, int e) {
  const int e0 = e & ~31, start = __ldg(P.row + u);
  unsigned gone = B.dead & ((1u << (e & 31)) - 1u);
  if (start <= e0) return B.shift - __popc(gone);
  gone &= ~((1u << (start - e0)) - 1u);
  return __ldcg(P.newRow + u) - start - __popc(gone);
}

/// The same for a block with at most one appended edge at each place.
__device__ __forceinline__ int moveByBits(const Block &B, int bit) {
  return B.shift - __popc(B.dead & ((1u << bit) - 1u)) + __popc(B.app & ((2u << bit) - 1u));
}

/// The copy: every edge to its new place, appended edges behind their rows.
/// A launch of its own: small CTAs, so that one that has run out of edges makes
/// room, and its own share of the registers for the loads in flight (the call on
/// 5.56M edges, K = 3: 217 us with the rows of 32 edges searched, 160 without).
__global__ void __launch_bounds__(kCopyThreads, 4)
copyFused(const __grid_constant__ ApplyParams P, const __grid_constant__ FusedScratch S, EngineControl *c,
          int stats) {
  __shared__ unsigned long long sSum[kMaxK];
  __shared__ int sMax[kMaxK];
  __shared__ int sMove[kCopyThreads / 32][kCopyEdges];
  if (__ldcg(&c->status) != 0 || __ldcg(&c->invalid) != 0) return;
  const int n = static_cast<int>(P.n), m = static_cast<int>(P.m), K = P.K;
  const long long tid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long T = static_cast<long long>(gridDim.x) * blockDim.x;
  const unsigned lane = laneId();
  if (threadIdx.x < kMaxK) {
    sSum[threadIdx.x] = 0;
    sMax[threadIdx.x] = 1;
  }
  __syncthreads();
  // Lanes 0 .. span - 1 (a multiple of K) move the weights, so a lane always
  // holds the same objective and its statistics stay in two registers.
  const int span = 32 / K * K;
  const int myK = static_cast<int>(lane) % K;
  long long sum = 0;
  int most = 1;
  const int step = span / K;                      // edges a turn moves
  const int ownEdge = static_cast<int>(lane) / K;  // this lane's among them
  int *moves = sMove[threadIdx.x >> 5];
  for (long long e0 = (tid >> 5) * kCopyEdges; e0 < m; e0 += (T >> 5) * kCopyEdges) {
    const int edges = static_cast<int>(m - e0 < kCopyEdges ? m - e0 : kCopyEdges);
    const int *src = P.w + e0 * K;
    const int ints = static_cast<int>(lane) < span ? edges * K : 0;
    int w[kTurns];
#pragma unroll
    for (int q = 0; q < kTurns; ++q) {
      const int i = q * span + static_cast<int>(lane);
      w[q] = i < ints ? __ldg(src + i) : 0;
    }
    int col[kCopyEdges / 32];
    Block B[kCopyEdges / 32];
#pragma unroll
    for (int j = 0; j < kCopyEdges / 32; ++j) {
      const int i = 32 * j + static_cast<int>(lane);
      col[j] = i < edges ? __ldg(P.col + e0 + i) : 0;
      const int4 b = 32 * j < edges ? __ldcg(reinterpret_cast<const int4 *>(S.block + (e0 >> 5) + j))
                                    : make_int4(0, 0, 0, 0);
      B[j] = Block{b.x, static_cast<unsigned>(b.y), static_cast<unsigned>(b.z), static_cast<unsigned>(b.w)};
    }
#pragma unroll
    for (int j = 0; j < kCopyEdges / 32; ++j) {
      const int i = 32 * j + static_cast<int>(lane);
      const long long e = e0 + i;
      int move = moveByBits(B[j], static_cast<int>(lane));
      if (B[j].app == kByRows) {
        // (the same for the whole warp; 32 j < edges, as the rest is zero)
        int r0 = chunkRow(P.row, n, e0 + 32 * j);
        const int u = edgeRow(P.row, n, e, i < edges, r0);
        move = i < edges ? moveByRow(P, B[j], u, static_cast<int>(e)) : 0;
      }
      const bool stays = i < edges && ((B[j].dead >> lane) & 1u) == 0;
      if (stays) P.newCol[e + move] = col[j];
      moves[i] = stays && ((B[j].other >> lane) & 1u) == 0 ? move * K : kNoMove;
    }
    __syncwarp();
    int *dst = P.newW + e0 * K;
    for (int t = 0; t * step < edges; t += kTurns) {
#pragma unroll
      for (int q = 0; q < kTurns; ++q) {
        const int i = (t + q) * span + static_cast<int>(lane);
        if (i < ints) {
          sum += w[q];
          most = w[q] > most ? w[q] : most;
          const int move = moves[(t + q) * step + ownEdge];
          if (move != kNoMove) dst[i + static_cast<long long>(move)] = w[q];
        }
      }
      if ((t + kTurns) * step < edges) {
#pragma unroll
        for (int q = 0; q < kTurns; ++q) {
          const int i = (t + kTurns + q) * span + static_cast<int>(lane);
          w[q] = i < ints ? __ldg(src + i) : 0;
        }
      }
    }
    __syncwarp();
  }
  // the insertions' weights of edges that stay
  const int others = __ldcg(S.counts + 3);
  for (long long a = tid; a < others; a += T) {
    const int2 o = __ldcg(S.other + a);
    const int4 b = __ldcg(reinterpret_cast<const int4 *>(S.block + (o.x >> 5)));
    const Block B{b.x, static_cast<unsigned>(b.y), static_cast<unsigned>(b.z), static_cast<unsigned>(b.w)};
    const int u = static_cast<int>(__ldcg(S.key + o.y) >> 32);
    const long long to = o.x + (B.app == kByRows ? moveByRow(P, B, u, o.x) : moveByBits(B, o.x & 31));
    const long long last = __ldcg(S.lastIns + o.y);
    for (int k = 0; k < K; ++k) P.newW[to * K + k] = __ldg(P.insW + last * K + k);
  }
  // appended edges, at the end of their row in the order of their groups'
  // first insertions
  const int appended = __ldcg(S.counts + 2);
  for (long long a = tid; a < appended; a += T) {
    const int i = __ldcg(S.app + a);
    const int u = __ldg(P.insFrom + i);
    const int r = __ldcg(S.rowSlot + u) - 1;
    const int count = __ldcg(S.nApp + r), segment = __ldcg(S.segApp + r), bits = __ldcg(S.markOf + r);
    int rank = 0;
    if (bits >= 0) {
      const unsigned *marks = S.marks + static_cast<long long>(bits) * S.markWords;
      for (int x = 0; x < i >> 7; ++x) {
        const uint4 b = __ldg(reinterpret_cast<const uint4 *>(marks) + x);
        rank += __popc(b.x) + __popc(b.y) + __popc(b.z) + __popc(b.w);
      }
      for (int x = i >> 7 << 2; x < i >> 5; ++x) rank += __popc(__ldg(marks + x));
      rank += __popc(__ldg(marks + (i >> 5)) & ((1u << (i & 31)) - 1u));
    } else {
      const int *list = S.app + segment;
      for (int x = 0; x < count; ++x) rank += __ldcg(list + x) < i;
    }
    const int to = __ldcg(P.newRow + u + 1) - count + rank;
    P.newCol[to] = __ldg(P.insTo + i);
    const long long last = __ldcg(S.lastIns + S.entrySlot[P.nDel + i]);
    for (int k = 0; k < K; ++k) P.newW[static_cast<long long>(to) * K + k] = __ldg(P.insW + last * K + k);
  }
  if (!stats) return;
  // the largest weight covers the insertions too
  if (static_cast<int>(lane) < span) {
    const long long all = static_cast<long long>(P.nIns) * K;
    const long long warps = T >> 5;
    for (long long i = (tid >> 5) * span + lane; i < all; i += warps * span) {
      const int w = __ldg(P.insW + i);
      most = w > most ? w : most;
    }
    atomicAdd(&sSum[myK], static_cast<unsigned long long>(sum));
    atomicMax(&sMax[myK], most);
  }
  __syncthreads();
  if (threadIdx.x < K) {
    atomicAdd(reinterpret_cast<unsigned long long *>(&S.result->weightSum[threadIdx.x]), sSum[threadIdx.x]);
    atomicMax(&S.result->maxWeight[threadIdx.x], static_cast<long long>(sMax[threadIdx.x]));
  }
}

unsigned slotsFor(long long B) {
  unsigned s = 64;
  while (s < 2 * B) s *= 2;
  return s;
}

template <typename X>
X *carve(unsigned char *&p, long long count) {
  X *r = reinterpret_cast<X *>(p);
  p += (static_cast<long long>(sizeof(X)) * (count > 0 ? count : 1) + 255) / 256 * 256;
  return r;
}

unsigned char *layout(unsigned char *p, long long n, long long m, long long nIns, long long nDel,
                      FusedScratch &S) {
  const long long B = nIns + nDel;
  S.slots = slotsFor(B);
  S.result = carve<FusedResult>(p, 1);
  S.counts = carve<int>(p, kCounts);
  S.key = carve<u64>(p, S.slots);
  for (int **x : {&S.cD, &S.cI, &S.firstIns, &S.lastIns, &S.occ, &S.first}) *x = carve<int>(p, S.slots);
  S.bits = carve<unsigned>(p, S.slots);
  S.filterBits = std::min(8 * S.slots, 1u << 20);
  S.filter = carve<unsigned>(p, S.filterBits / 32);
  for (int **x : {&S.entrySlot, &S.rows, &S.nApp, &S.segApp, &S.curApp, &S.markOf}) {
    *x = carve<int>(p, B);
  }
  S.pieces = carve<u64>(p, m / kPiece + B);
  S.block = carve<Block>(p, (m + 31) / 32 + 1);
  S.moveSums = carve<long long>(p, kMaxCtas);
  S.app = carve<int>(p, nIns);
  S.markWords = nIns > kMarkLeast ? static_cast<int>((nIns + 127) / 128 * 4) : 0;
  S.marks = carve<unsigned>(p, static_cast<long long>(kMarkRows) * S.markWords);
  S.other = carve<int2>(p, nIns);
  S.rowSlot = carve<int>(p, n + 4);
  S.delta = carve<int>(p, n + 4);
  return p;
}

}  // namespace

size_t applyFusedBytes(long long n, long long m, long long nIns, long long nDel) {
  FusedScratch S;
  unsigned char *base = reinterpret_cast<unsigned char *>(static_cast<uintptr_t>(256));
  return static_cast<size_t>(layout(base, n, m, nIns, nDel, S) - base) + 256;
}

cudaError_t applyFusedShape(int sms, int ctasPerSm, int &ctas) {
  int perSm = 0;
  cudaError_t err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, applyFused, kThreads, 0);
  if (err != cudaSuccess) return err;
  if (perSm < 1) return cudaErrorInvalidConfiguration;
  if (ctasPerSm > 0 && ctasPerSm < perSm) perSm = ctasPerSm;
  ctas = std::min(perSm * sms, kMaxCtas);
  return cudaSuccess;
}

cudaError_t applyBatchFused(const ApplyParams &P, void *scratch, EngineControl *ctl, long long *blockSums,
                            long long timeoutNs, int ctas, bool stats, FusedResult *pinned,
                            EngineControl *pinnedCtl, cudaStream_t s) {
  FusedScratch S;
  layout(static_cast<unsigned char *>(scratch), P.n, P.m, P.nIns, P.nDel, S);
  S.blockSums = blockSums;
  ApplyParams p = P;
  cudaError_t err = cudaMemsetAsync(ctl, 0, sizeof(EngineControl), s);
  if (err != cudaSuccess) return err;
  void *args[] = {&p, &S, &ctl, &timeoutNs};
  err = cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(applyFused), dim3(ctas), dim3(kThreads), args,
                                    0, s);
  if (err == cudaSuccess) {
    const long long want = (std::max(P.m, static_cast<long long>(P.nIns)) + kCopyThreads - 1) / kCopyThreads;
    const int grid = static_cast<int>(std::min(std::max(want, 1LL), 4LL * ctas));
    copyFused<<<grid, kCopyThreads, 0, s>>>(P, S, ctl, stats ? 1 : 0);
    err = cudaGetLastError();
  }
  if (err == cudaSuccess) {
    err = cudaMemcpyAsync(pinned, S.result, sizeof(FusedResult), cudaMemcpyDeviceToHost, s);
  }
  if (err == cudaSuccess) {
    err = cudaMemcpyAsync(pinnedCtl, ctl, sizeof(EngineControl), cudaMemcpyDeviceToHost, s);
  }
  if (err == cudaSuccess) err = cudaStreamSynchronize(s);
  return err;
}

}  // namespace mospb200

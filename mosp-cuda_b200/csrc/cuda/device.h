// device.h - device helpers shared by the persistent kernels (engine.cu,
// apply.cu): the bounded grid barrier, block scans, and passes over all edges
// of a CSR with their rows. Every translation unit has its own copy.
#pragma once

#include <climits>

#include "engine.h"

namespace mospb200 {
namespace {

constexpr unsigned kFull = 0xffffffffu;


__device__ __forceinline__ unsigned laneId() { return threadIdx.x & 31u; }

__device__ __forceinline__ unsigned long long globalNs() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned ldAcquire(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void stRelease(unsigned *p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ int ldVolatile(const int *p) {
  return *reinterpret_cast<const volatile int *>(p);
}

/// Barrier bookkeeping of one CTA: the barrier epoch and the wall-clock
/// deadline (%globaltimer) of the whole launch.
struct Sync {
  unsigned epoch;
  unsigned long long deadline;
};

__device__ __forceinline__ Sync startSync(long long timeoutNs) {
  return Sync{0u, globalNs() + static_cast<unsigned long long>(timeoutNs)};
}

/// Software grid barrier. Thread 0 of every CTA arrives on `arrive`; the
/// last arrival publishes the epoch on `release`, which the others poll
/// (acquire). The launch has one wall-clock deadline: a CTA that reaches a
/// barrier after it marks the run MOSP_ERR_TIMEOUT and returns false
/// without arriving, so the others cannot pass this barrier; a CTA that
/// waits past it, or sees the status set while it waits (checked every 32
/// polls, off the path of a release that arrives in time), does the same.
/// A CTA that passed a barrier before the status was set returns false at
/// the next one (the deadline has passed by then), and the kernel must
/// return. So a run ends by the deadline whether it stalls or keeps
/// iterating.
__device__ bool gridSync(EngineControl *c, Sync &sync) {
  __shared__ int sOk;
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned epoch = ++sync.epoch;
    int ok = 1;
    if (globalNs() > sync.deadline) {
      atomicCAS(&c->status, 0, MOSP_ERR_TIMEOUT);
      ok = 0;
    } else {
      __threadfence();
      const unsigned prev = atomicAdd(&c->arrive, 1u);
      if (prev + 1u == epoch * gridDim.x) {
        stRelease(&c->release, epoch);
      } else {
        unsigned spin = 0;
        while (static_cast<int>(ldAcquire(&c->release) - epoch) < 0) {
          if ((++spin & 31u) == 0) {
            if (ldVolatile(&c->status) != 0) {
              ok = 0;
              break;
            }
            if (globalNs() > sync.deadline) {
              atomicCAS(&c->status, 0, MOSP_ERR_TIMEOUT);
              ok = 0;
              break;
            }
          }
        }
      }
      __threadfence();
    }
    sOk = ok;
  }
  __syncthreads();
  return sOk != 0;
}

// ---------------------------------------------------------------------------
// Block-level scan helpers (combined-graph and reverse-CSR builds)
// ---------------------------------------------------------------------------

/// Inclusive scan of one value per thread over the CTA; *total = CTA sum.
__device__ long long blockInclusiveScan(long long x, long long *total) {
  __shared__ long long warpSums[kThreads / 32];
  const unsigned lane = laneId();
  const int warp = threadIdx.x >> 5;
  long long v = x;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const long long o = __shfl_up_sync(kFull, v, off);
    if (static_cast<int>(lane) >= off) v += o;
  }
  if (lane == 31) warpSums[warp] = v;
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    long long s = static_cast<int>(lane) < nw ? warpSums[lane] : 0;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const long long o = __shfl_up_sync(kFull, s, off);
      if (static_cast<int>(lane) >= off) s += o;
    }
    if (static_cast<int>(lane) < nw) warpSums[lane] = s;
  }
  __syncthreads();
  const long long prefix = warp > 0 ? warpSums[warp - 1] : 0;
  *total = warpSums[(blockDim.x >> 5) - 1];
  __syncthreads();
  return prefix + v;
}

/// Sum of one value per thread over the CTA (every thread gets it).
__device__ long long blockSum(long long x) {
  long long total;
  blockInclusiveScan(x, &total);
  return total;
}

// ---------------------------------------------------------------------------
// Passes over all edges with their rows (device-graph fill, tree edges of the
// path costs, parent recovery): warps take chunks of the edge array on
// demand, find the row of a chunk's first edge by binary search and the rows
// of 32 edges at a time by a shuffle search over row ends. Equal slices
// per warp would leave half of the grid idle on power-law graphs: where rows
// are short a slice takes several times as long.
// ---------------------------------------------------------------------------
/// The last row that starts at or before edge e: 32 probes a step, so five
/// dependent loads for a million rows where halving takes twenty. All lanes
/// call it.
__device__ __forceinline__ int chunkRow(const int *outRow, int n, long long e) {
  int row = 0;
  for (int hi = n; hi - row > 1;) {
    const int mid = row + static_cast<int>(static_cast<long long>(hi - row) * (laneId() + 1) / 33);
    const int below = __popc(__ballot_sync(kFull, __ldg(outRow + mid) <= e));
    const int lo = __shfl_sync(kFull, mid, below > 0 ? below - 1 : 0);
    const int up = __shfl_sync(kFull, mid, below < 32 ? below : 31);
    if (below < 32) hi = up;
    if (below > 0) row = lo;
  }
  return row;
}

struct EdgeChunks {
  long long size, m, nwarps;
  long long mine;  // the warp's first chunk; the others come off the counter
  unsigned *next;  // zero at the start of the pass

  /// About eight chunks per warp, of at least 256 edges (a chunk pays for a
  /// binary search); fewer edges than that: one chunk per warp.
  __device__ __forceinline__ EdgeChunks(long long edges, long long gwarp, long long warps, unsigned *counter)
      : m(edges), nwarps(warps), mine(gwarp), next(counter) {
    size = (m / (8 * nwarps) + 31) / 32 * 32;
    if (size < 256) size = 256;
    if (size > 4096) size = 4096;
    if (size * nwarps > m) size = (m + 32 * nwarps - 1) / (32 * nwarps) * 32;
  }
  /// The warp's next chunk [wb, we) and the row of its first edge: false
  /// when there is none. All lanes call it.
  __device__ __forceinline__ bool take(const int *outRow, int n, long long &wb, long long &we, int &row) {
    long long i = mine;
    mine = -1;
    if (i < 0) {
      if (size * nwarps >= m) return false;
      unsigned a = 0;
      if (laneId() == 0) a = atomicAdd(next, 1u);
      i = nwarps + __shfl_sync(kFull, a, 0);
    }
    wb = size * i;
    we = wb + size < m ? wb + size : m;
    if (wb >= we) return false;
    row = chunkRow(outRow, n, wb);
    return true;
  }
};

/// The row of this lane's edge (`in`: it has one) of 32 consecutive edges, none
/// of which lies in a row before r0; r0 moves on to the last one's. The
/// window holding row n - 1 ends the search: rows past n count as ending at
/// INT_MAX. All lanes call it.
__device__ __forceinline__ int edgeRow(const int *outRow, int n, long long e, bool in, int &r0) {
  int row = in ? -1 : r0;
  for (int base = r0; base < n; base += 32) {
    const unsigned rr = base + laneId();  // (past INT_MAX for the last rows)
    const int end = rr < static_cast<unsigned>(n) ? __ldg(outRow + rr + 1) : INT_MAX;
    int at = 0;  // rows of the window that end at or before the edge
#pragma unroll
    for (int step = 16; step >= 1; step >>= 1) {
      if (__shfl_sync(kFull, end, at + step - 1) <= e) at += step;
    }
    // every lane takes part in the shuffles, found or not
    const int lastEnd = __shfl_sync(kFull, end, 31);
    if (row < 0 && e < lastEnd) row = base + at;
    if (__all_sync(kFull, row >= 0)) break;
  }
  r0 = __shfl_sync(kFull, row, 31);  // the largest; past the chunk the caller ends
  return row;
}

}  // namespace
}  // namespace mospb200

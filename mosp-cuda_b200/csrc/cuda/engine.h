// engine.h - shared host/device definitions of the sm_100a MOSP engine.
//
// The engine is a set of persistent kernels (one CTA group resident per SM,
// launched cooperatively so that every CTA is co-resident) whose phases are
// separated by a software grid barrier with a bounded wait. All state a
// phase hands to the next one lives in the workspace (device memory) or in
// the control block; per-launch arguments travel as one __grid_constant__
// parameter block, so a launch needs no host-to-device copy and can be
// queued back to back with the next one.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "mosp_b200.h"

namespace mospb200 {

using u64 = unsigned long long;

constexpr int kThreads = 1024;                // threads per CTA
constexpr int kMaxK = MOSP_MAX_OBJECTIVES;    // objectives per launch
constexpr u64 kInfWord = ~0ULL;               // packed INF (all ones)
constexpr long long kDistInf = MOSP_DISTANCE_INF;
constexpr int kLaneRowMax = 32;               // rows above: warp-cooperative
#ifndef MOSP_STAGE_ENTRIES
#define MOSP_STAGE_ENTRIES 8192
#endif
// entries of the per-CTA append stage of a bulk near-far launch (16 bytes
// each, dynamic shared memory); asynchronous launches take fewer
constexpr int kStageEntriesMax = MOSP_STAGE_ENTRIES;
// entries of an asynchronous launch: the CTA's ring of near entries (8 bytes
// each), the far buffers of its 32 warps (128 entries of 8 bytes) and its
// state (AsyncCta in engine.cu)
constexpr int kRing = 8192;
constexpr int kFarBuf = 128;
constexpr int kMail = 8;
constexpr int kAsyncCtaBytes = 30 * 1024;
constexpr int kStageEntriesAsync = (kRing + kThreads / 32 * kFarBuf) / 2 + kAsyncCtaBytes / 16;

enum EngineMode : int { kModeUpdate = 0, kModeScratch = 1, kModeCombined = 2 };

/// Per-objective arguments of one engine launch.
struct ObjectiveArgs {
  const int *outW;       // out-edge weights of this objective [m]
  const int *inW;        // in-edge weights of this objective [m]
  long long *dist;       // tree in/out [n]
  int *parent;           // tree in/out [n]
  const int *chFrom;     // deleted / weight-increased edges
  const int *chTo;
  int nChanged;
  int parentBits;        // 0: distance-only words
  u64 noParent;          // all-ones parent field
  u64 maxDist;           // (n - 1) * maxWeight: no candidate above it
  u64 delta;             // near-far bucket width (> 0)
};

/// Control block of one launch: barrier, status and the per-objective list
/// counters. Counters that change from one iteration to the next live in
/// rings of three slots (read slot i, write slot i+1, clear slot i+2), so
/// one grid barrier per iteration suffices.
struct alignas(128) EngineControl {
  unsigned arrive;       // barrier arrivals (monotone)
  unsigned pad0[31];
  unsigned release;      // barrier epoch released by the last arrival
  unsigned pad1[31];
  // asynchronous near-far, one slot per phase modulo three: CTAs that still
  // work on their share of the phase plus entries of the spill queue that are
  // not settled; CTAs that have run dry
  unsigned asyncPending[3];
  unsigned pad3[29];
  int asyncHungry[3];
  unsigned pad4[29];
  int status;            // 0 or MOSP_ERR_TIMEOUT (run aborted)
  int overflow;          // an input distance does not fit the packing
  int invalid;           // malformed input (ids out of range, cycles)
  int rounds;            // pointer-jumping rounds
  int jumpActive[4];
  int finalGen;          // last stamp generation used
  int heavy;             // the graph has rows of more than kHeavyDeg edges
  int pad2[2];
  unsigned long long sums[2];  // combined graph: edges, weight sum
  int candCount[kMaxK];
  int invalidated[kMaxK];
  int nearCount[kMaxK][4];
  int farCount[kMaxK][4];
  u64 farMinC[kMaxK][4];       // complement of the far-pile minimum
  int iterations[kMaxK];
  int epochs[kMaxK];
  long long pushes[kMaxK];
  // %globaltimer at the phase boundaries, written by CTA 0 (see kPhase*)
  unsigned long long phaseNs[8];
  // near-far loop profile. Bulk loop (written by CTA 0): time and items of
  // iterations that split a far pile ([0]) and of pure push iterations
  // ([1]). Asynchronous loop: loopNs[0] its time, loopIters[0] its phases,
  // loopIters[1] warp rounds, loopNs[1] of which before the CTA took spilled
  // entries in its phase, loopItems entries taken from the spill queue ([0])
  // and from the CTAs' own rings and far-pile shares ([1])
  unsigned long long loopNs[2];
  long long loopIters[2];
  long long loopItems[2];
  // bulk loop: time (ns) of CTA 0 summed over the push iterations: decision
  // step, thread 0's own items, waiting for the CTA's other warps, list
  // flush, grid barrier. Asynchronous loop: durations of phases 0-3 and of
  // the rest
  unsigned long long iterSplitNs[5];
  // restricted parent recovery (kFlagCanonical): vertices in the changed
  // and scan lists of each objective, and chunks in the two chunk lists
  int recChanged[kMaxK];
  int recScan[kMaxK];
  int recChunks[2];
  int recWide;        // full parent recovery: a distance of 2^31 or more (recDist is not used)
  int longRows;       // rows longer than a row record
  unsigned chunkNext; // next chunk of a pass over all edges (at most one per launch)
};

// EngineParams::flags (tuning switches; results do not depend on them)
enum : int {
  kFlagPrecheck = 1,     // read the word before the atomicMin of a relaxation
  kFlagHostRecovery = 2, // leave the lowest-id parent recovery of distance-only
                         // objectives to recoverParents, launched right after
  kFlagAsync = 4,        // asynchronous near-far loop (one grid barrier per far-pile
                         // split instead of one per iteration) when the graph has
                         // no hub rows
  kFlagPullOnly = 8,     // always pull into the candidates (never push from the
                         // valid vertices)
                         // (16 is free: the asynchronous loop always goes on
                         // inside its warps)
  kFlagCanonical = 32    // the input trees follow the lowest-id tie rule: with
                         // kFlagHostRecovery, distance-only objectives recover
                         // parents only where the batch can change them
                         // (recover.cu); the same result as the full recovery
                         // for such inputs
};

// Mark bytes of the restricted parent recovery (EngineParams::recMark, one
// per objective and vertex): the update launch writes kRecChanged where a
// distance-only objective's distance changed; kRecScan marks the vertices
// whose in-row is scanned again.
enum : unsigned char { kRecChanged = 1, kRecScan = 2 };

/// Positions of one shard of the asynchronous loop's spill queue: entries
/// claimed by consumers and reserved by producers, side by side, so that one
/// load sees both. Words of their own, as a claim is a compare-and-swap: in one
/// word for both it failed whenever a producer came between (tree from scratch
/// of 2M random vertices of degree 10: 6.2 ms so, 2.6 with two words).
struct alignas(128) AsyncShard {
  unsigned claimed, reserved;
  unsigned pad[30];
};
constexpr int kAsyncShards = 16;  // shards of the spill queue

// Row records of the asynchronous loop: the edges of a row, side by side with
// their weights, in one 32-byte sector per objective and vertex.
constexpr int kMoreEdges = -2;   // fourth head of a record: the row has more than four edges

/// A far pile of the asynchronous loop holds a vertex at most this often:
/// once as it leaves infinity or its valid tree distance, once more when an
/// invalidated vertex passes its old distance, and once by overflow of the
/// spill queue (flagged).
constexpr int kFarCopies = 3;

/// Whether a launch makes row records: graphs of at most 3.5 edges per
/// vertex, most of which have few longer rows. Grids of 302,500 vertices, K = 3,
/// with records and without, pass in us: 2 edges per vertex, update with
/// long-range changes 1102/1356, with short ones 4012/5585, tree from scratch
/// 2434/3409; 2.8: 1047/1092, 3661/4830, 1702/2268; 3.4: 1067/1070, 3965/5207,
/// 1826/2377; 4: 1182/1202, 4167/5280, 1919/2470; 5: 1385/1215, 7389/5079,
/// 5035/2497 (every row is longer). A random graph of 3.4 has 17% longer rows,
/// where the records are not used; making them takes 10 us of a pass of 700.
__host__ __device__ inline bool recordsPay(long long n, long long m) { return 2 * m <= 7 * n; }

// Phase boundaries recorded in EngineControl::phaseNs.
enum : int {
  kPhaseStart = 0,     // kernel start
  kPhasePacked = 1,    // old trees packed (update) / graph built (combined)
  kPhaseRoots = 2,     // roots marked
  kPhaseJumped = 3,    // subtrees flagged by pointer jumping
  kPhaseCandidates = 4,
  kPhasePulled = 5,    // pull pass done; near-far loop starts
  kPhaseLoop = 6,      // near-far loop done
  kPhaseEnd = 7        // results written
};

/// Parameters of one engine launch (passed by value, < 4 KB).
struct EngineParams {
  int n, m, K, source;
  // A batched run (independent instances stored as one disjoint union)
  // has one root per instance: `sources` holds them sorted, `source` is the
  // first. nSources <= 1 means the single root `source`.
  const int *sources;
  int nSources;
  int mode, maxRounds, nHeads, flags;
  int localRounds;  // CTA-local expansion rounds per near-far iteration (0: none)
  int narrowItems;  // iterations with at most this many items run on CTA 0 alone
  int narrowRounds; // CTA-local rounds of such an iteration
  long long timeoutNs;
  int *genPtr;                 // stamp generation, advanced by every launch
  const int *outRow, *outCol, *inRow, *inCol;
  const int *heads;
  // workspace lists: objective k uses [k * stride, (k + 1) * stride) of the
  // per-vertex arrays and [k * strideNear, ...) of the near lists
  u64 *packed;
  int *val, *stamp, *inFar, *cand;
  int *farL0, *farL1;
  int *nearV0, *nearV1;        // near lists: vertices
  u64 *nearD0, *nearD1;        // near lists: distance when appended
  long long stride, strideNear;
  long long strideFar;         // far piles: objective k from k * strideFar
  // spill queue of the asynchronous loop (kFlagAsync): aqShards shards of
  // aqShardCap slots, every slot ~0 (empty) between launches
  u64 *aqSlots;
  AsyncShard *aqCtr;
  unsigned aqShardCap;
  int aqShards;
  int4 *rec;                   // row records (two int4 per vertex; objective k from
                               // 2 * k * stride) or null: the launch uses none
  int stageEntries;            // entries of the per-CTA append stage (dynamic shared memory)
  int heavyDeg;                // a row above this many edges: bulk loop, longer rows by whole
                               // CTAs (0: 2,048 for the loop, 512 for the rows)
  EngineControl *ctl;
  // combined graph (Steps 2-3)
  const int *combParents;      // K trees, objective-major
  int *combDeg, *combRow, *combCol, *combW;
  long long *blockSums;
  int combK, combBase;
  long long combDelta;         // > 0: fixed width; else default
  int prefTerms[kMaxK];        // L / Pref_i
  // restricted parent recovery (kFlagCanonical): mark bytes [k * stride +
  // v]; per objective the list of vertices whose distance changed
  // (recChanged + k * stride) and of the other vertices whose in-row is
  // scanned (recScanList + k * stride); chunks of rows of more than
  // kRecLightRow edges: out-rows of changed vertices in [0, recChunkCap) of
  // recChunkList, in-rows to scan in [recChunkCap, 2 recChunkCap)
  unsigned char *recMark;
  int *recChangedList;
  int *recScanList;
  u64 *recChunkList;
  int recChunkCap;
  // full parent recovery: the distances of the distance-only objectives side
  // by side in 32 bits (~0: unreached), written by the unpack, or null. Up to
  // four of them: one int4 per vertex; else groups of eight, two int4 per
  // vertex and group, group g from g * 2 * n
  int4 *recDist;
  ObjectiveArgs obj[kMaxK];
};
static_assert(sizeof(EngineParams) <= 4096, "kernel parameter block limit");

// rows of the restricted recovery up to this many edges are handled by the
// warp of their vertex; longer rows go to a chunk list in chunks of
// 2 kRecLightRow edges, one warp per chunk (so each chunk list needs at
// most K (m / kRecLightRow + 1) entries, and no warp walks more than
// 32 kRecLightRow edges of its own vertices)
constexpr int kRecLightRow = 64;

/// Parameters of the device-graph build.
struct BuildParams {
  int n, m, K;
  long long timeoutNs;
  const int *outRow, *outCol, *edgeMajorW;
  int *outW, *inRow, *inCol, *inW;
  int *cursor;  // in-degrees [n + 1]
  int *rank;    // edge e among the edges into its head [m], or null: no room
  long long *blockSums;
  EngineControl *ctl;
};

/// Parameters of the MOSP path-cost kernel.
struct CostParams {
  int n, m, KG, source;
  const int *sources;  // sorted roots of a batched run (nSources > 1), else unused
  int nSources;
  long long timeoutNs;
  const int *outRow, *outCol, *outW;  // outW: KG objective-major columns
  const int *parent;
  int *edgeOf;
  int *anc0, *anc1;
  long long *acc0, *acc1;
  long long *costs;
  EngineControl *ctl;
};

// Host-side launchers (engine.cu). Each returns a cudaError_t of the
// launch; device-side errors are reported through the control block.
struct LaunchShape {
  int engineCtas, buildCtas, costCtas, applyCtas;
};
cudaError_t queryLaunchShape(int ctasPerSm, LaunchShape &shape);
cudaError_t launchEngine(const EngineParams &p, int ctas, cudaStream_t s);
/// The same cooperative launch through cudaLaunchKernelEx with the
/// cooperative attribute, the form a CUDA graph can capture.
cudaError_t launchEngineEx(const EngineParams &p, int ctas, cudaStream_t s);

/// An update launch with a distance-only objective: its parent recovery
/// runs as a kernel of its own (all of L1 for the graph reads, where the
/// update launch gives most of the SM's on-chip memory to its stage).
bool needsHostRecovery(const EngineParams &p);

/// The lowest-id tight parent recovery of the distance-only objectives of
/// update launch `p` (which ran with kFlagHostRecovery), on stream s: over
/// all edges, or (kFlagCanonical) only where the batch can change a parent.
cudaError_t launchRecovery(const EngineParams &p, cudaStream_t s);
/// The restricted recovery (recover.cu): four launches on stream s.
cudaError_t launchRestrictedRecovery(const EngineParams &p, int sms, cudaStream_t s);
cudaError_t launchBuild(const BuildParams &p, int ctas, cudaStream_t s);
cudaError_t launchCosts(const CostParams &p, int ctas, cudaStream_t s);
cudaError_t launchBarrierProbe(EngineControl *ctl, long long timeoutNs,
                               int ctas, cudaStream_t s);
cudaError_t launchBarrierCost(EngineControl *ctl, int rounds, int reads,
                              long long timeoutNs, int ctas, cudaStream_t s);

// ---------------------------------------------------------------------------
// Step 1 on the GPU (apply.cu): a change batch applied to a device CSR
// ---------------------------------------------------------------------------
struct ApplyParams {
  long long n, m;
  int K;
  const int *row, *col, *w;  // original out-CSR, edge-major weights w[e*K+k]
  int nIns, nDel;
  const int *insFrom, *insTo, *insW, *delFrom, *delTo;
  int *newRow, *newCol, *newW;  // updated out-CSR (capacity m + nIns edges)
  unsigned *mask;               // nIns weight-increase masks
  // set by applyBatchGpu
  int vbits, ibits;
  const int *sortedVals;
};

/// Per (u,v) group of the sorted batch.
struct ApplyGroups {
  int *start;  // first entry of each group (+ end sentinel)
  int *u, *v, *cD, *cI, *firstIns, *lastIns, *occ, *first;
};

/// Rows with at least one change.
struct ApplyRows {
  int *row, *gs, *deg, *off;
};

enum ApplyCounter : int {
  kApplyInvalid = 0,
  kApplyEntries,
  kApplyGroups,
  kApplyRows,
  kApplyAppended,
  kApplyCounters
};

/// Scratch bytes of applyBatchGpu for these sizes.
size_t applyScratchBytes(long long n, long long m, long long nIns, long long nDel);
/// Runs Step 1 on stream `s` and waits for it. hostCounters receives the
/// kApplyCounters device counters followed by the new edge count; when
/// hostStats is non-null it receives per objective the largest weight of
/// the original edges and insertions (at least 1), then the weight sums of
/// the original edges (2K values).
cudaError_t applyBatchGpu(ApplyParams P, void *scratch, int sms, cudaStream_t s, int *hostCounters,
                          long long *hostStats);

// Step 1 in one cooperative launch (applyFused.cu), for batches of up to this
// many changes
constexpr long long kFusedBatch = 1 << 18;

/// What a fused Step 1 leaves for the host.
struct FusedResult {
  int newM;
  int pad;
  long long maxWeight[kMaxK];
  long long weightSum[kMaxK];
};
size_t applyFusedBytes(long long n, long long m, long long nIns, long long nDel);
cudaError_t applyFusedShape(int sms, int ctasPerSm, int &ctas);
/// Runs Step 1 on stream `s` with `ctas` CTAs and waits for it; the result
/// and the control block come back in the pinned buffers (the result is valid
/// if the control block's status and invalid are zero).
cudaError_t applyBatchFused(const ApplyParams &P, void *scratch, EngineControl *ctl, long long *blockSums,
                            long long timeoutNs, int ctas, bool stats, FusedResult *pinned,
                            EngineControl *pinnedCtl, cudaStream_t s);

/// Whether v is a root: the source, or one of the sorted batched roots.
__device__ __forceinline__ bool isRoot(int source, const int *sources, int nSources, int v) {
  if (v == source) return true;
  if (nSources <= 1) return false;
  int lo = 0, hi = nSources;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    const int s = sources[mid];
    if (s == v) return true;
    if (s < v) lo = mid + 1; else hi = mid;
  }
  return false;
}

/// Sets the calling thread's last-error message of the C ABI
/// (mosp_last_error) and returns `status`.
int recordFailure(int status, const char *message);

}  // namespace mospb200

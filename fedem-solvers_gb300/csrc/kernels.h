// kernels.h -- launch wrappers of the batched FEDEM Newton engine kernels.
#pragma once

#include <cuda_runtime.h>

#include <functional>
#include <string>

#include "engine_dev.cuh"

namespace fgpu {

// Refused launches.  The launch wrappers return nothing: the first launch of a host
// thread that the runtime refuses is kept until the thread's next takeLaunchError(),
// which every call that enqueues kernels asks before it reports success (and, at its
// start, to begin afresh).  Until then the thread launches nothing more: no kernel runs
// on what a missing one should have written.  The runtime's own last error is cleared,
// so that it does not turn up in another batch's call.
inline thread_local cudaError_t t_launchError = cudaSuccess;
inline void noteLaunch(cudaError_t e) {
  if (e == cudaSuccess) return;
  cudaGetLastError();
  if (t_launchError == cudaSuccess) t_launchError = e;
}
inline cudaError_t takeLaunchError() {
  const cudaError_t e = t_launchError;
  t_launchError = cudaSuccess;
  return e;
}
// Test hook: the t_refuseLaunch-th launch of this host thread from now asks for more
// shared memory than any device has, which the runtime refuses (0: off).
inline thread_local int t_refuseLaunch = 0;
inline size_t launchShared(size_t smem) {
  return t_refuseLaunch > 0 && --t_refuseLaunch == 0 ? (size_t)1 << 30 : smem;
}

// Programmatic dependent launch.  Every kernel of the engine is launched with
// programmatic stream serialization (pdlLaunch) and calls pdlEntry() first:
// it waits until the previous kernel of its stream has completed and its
// memory is visible (griddepcontrol.wait), then lets the next kernel's blocks
// be scheduled (griddepcontrol.launch_dependents), which then wait the same
// way.  Ordering and results are those of plain stream order; only the launch
// of each kernel overlaps the end of the one before.
#ifdef __CUDACC__
__device__ __forceinline__ void pdlEntry() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// One launch (none after one that the runtime refused, see above, or of an empty grid).
template <typename... KArgs, typename... Args>
inline void launchWith(cudaLaunchAttribute* attrs, int nAttrs, void (*kernel)(KArgs...), dim3 grid, dim3 block,
                       size_t smem, cudaStream_t s, Args... args) {
  if (t_launchError != cudaSuccess || grid.x == 0) return;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = launchShared(smem);
  cfg.stream = s;
  cfg.attrs = attrs;
  cfg.numAttrs = nAttrs;
  noteLaunch(cudaLaunchKernelEx(&cfg, kernel, args...));
}

template <typename... KArgs, typename... Args>
inline void pdlLaunch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                      Args... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  launchWith(attr, 1, kernel, grid, block, smem, s, args...);
}

// Dynamic shared memory a launch may ask for.  The limit is an attribute of the
// function, shared by every batch and host thread of the process: a kernel that can
// need more than the default 48 KB always gets this one value, since a limit set to one
// batch's need could be lowered under another batch's launch, or captured graph.
constexpr int kMaxDynamicShared = 220 * 1024;
template <typename K>
inline cudaError_t allowBigShared(K kernel) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicShared);
}
#endif

// element pass modes
enum ElemMode : int {
  EM_PRED = 0,         // predictor: velocities from dk/ak, no position update
  EM_INC = 1,          // after an increment: corotation, deformation, forces
  EM_STATIC_INIT = 2,  // static, initial frame kept (linInc = 1)
  EM_STATIC = 3,       // static after an increment (corotated update)
  EM_FINAL = 4         // final static update: corotation, zero velocities, no vld
};

// --- element_kernels.cu ----------------------------------------------------
// Seeding of the backward work queues by the step-start kernels: for each
// solve q of the iteration, queue q receives the roots of the active models
// and ctr[4 q + 2] their number of chains (ctr[4 q] and ctr[4 q + 1] are the
// take and fill positions); nq = 0 seeds nothing.
struct BackwardSeed {
  int nq = 0;      // queues (solves per iteration)
  int stride = 0;  // slots per queue
  int maxRoots = 0;  // largest number of entries a model has in one of the queues
  // per model: the tops of the cascades' subtrees (fronts whose parent is not the
  // cascades', or roots) in roots[rootOff[m]..rootOff[m+1]), and its number
  // of chains
  const int* rootOff = nullptr;
  const int* roots = nullptr;
  const int* slotCnt = nullptr;
  int* queue = nullptr;
  int* ctr = nullptr;
  // the same for the queues of the trees on thread blocks (chunks in the place of
  // fronts); strideT = 0: none
  int strideT = 0;
  const int* rootOffT = nullptr;
  const int* rootsT = nullptr;
  const int* slotCntT = nullptr;
  int* queueT = nullptr;
  int* ctrT = nullptr;
};
// parts that each of `queues` queues of a model is cut into when `warps` warps seed
// them, a part per warp (no queues: nothing to seed)
inline __host__ __device__ int seedParts(int warps, int queues) {
  return queues <= 0 ? 0 : warps > queues ? warps / queues : 1;
}
// What the last kernel of an iteration does beside the step end: the iteration's
// counters and backward queues reset for the next one (in place of memset nodes),
// and a report into host memory, its serial number last, that the host can follow
// without a copy or a synchronisation.
constexpr int kIterationsAhead = 6;
// reports in turn, more than iterations in flight: one is not overwritten while it is read
constexpr int kReports = 8;
static_assert(kIterationsAhead < kReports, "a report would be overwritten before it is read");
// every so many iterations one is timed, farther apart than iterations in flight: its
// events are read before the next timed one records them
constexpr int kTimedEvery = 7;
static_assert(kIterationsAhead < kTimedEvery, "phase events would be recorded again before they are read");
struct IterationReport {
  long long serial;    // iterations finished since the counters' last reset by the host
  long long elements;  // elements of the models that took part
  int active;          // models that took part
  int remaining;       // models with another iteration to do
  int more;            // of them, models with a further step after the one they are in (or about to start)
  int far;             // of them, models with kIterationsAhead - 1 further steps or more
};
struct IterationEnd {
  int* ctr = nullptr;  // counters to zero
  int ctrInts = 0;
  int* queue = nullptr;  // queue slots to empty (-1)
  int queueInts = 0;
  const int* active = nullptr;          // (inside ctr)
  const long long* elements = nullptr;  // (inside ctr)
  int* tally = nullptr;                 // remaining, more (counted by the convergence test), kept: active of
                                        // the last iteration; far; then the serial number
  IterationReport* host = nullptr;      // pinned host memory, kReports
};
void launchBeginStep(const DevData& d, int* activeCount, long long* activeEl, const BackwardSeed& seed,
                     cudaStream_t s);
void launchPredictDofs(const DevData& d, cudaStream_t s);
void launchElements(const DevData& d, int mode, cudaStream_t s);
void launchResidual(const DevData& d, cudaStream_t s);
void launchBuildElementNewton(const DevData& d, cudaStream_t s);
void launchRotateElementNewton(const DevData& d, cudaStream_t s);
void launchCsrGather(const DevData& d, cudaStream_t s);
void launchIncrement(const DevData& d, cudaStream_t s);
void launchNormsControl(const DevData& d, const IterationEnd& e, cudaStream_t s);
// the same in two parts: the per-chunk partial norms (reading the increments
// and the residual only), then the convergence test and the step end
void launchNormsPartial(const DevData& d, cudaStream_t s);
void launchControlStepEnd(const DevData& d, const IterationEnd& e, cudaStream_t s);
// static equilibrium helpers
void launchStaticBegin(const DevData& d, int* activeCount, const BackwardSeed& seed, cudaStream_t s);
void launchSeedBackward(const DevData& d, const BackwardSeed& seed, cudaStream_t s);
void launchStaticResidual(const DevData& d, cudaStream_t s);
void launchStaticNorm(const DevData& d, cudaStream_t s);
void launchStaticIncrement(const DevData& d, cudaStream_t s);
void launchStaticFinish(const DevData& d, cudaStream_t s);

// --- joint_kernels.cu: master-slave joints ----------------------------------
// per joint: joint variables incremented (EM_INC, EM_STATIC), dependent triad
// placed, constraint coefficients rebuilt; same model gating as the element pass
void launchJoints(const DevData& d, int mode, cudaStream_t s);
// expanded Newton matrices of the elements with a dependent triad (tangent models)
void launchExpandElements(const DevData& d, cudaStream_t s);
// expanded forces of those elements after an element pass of this mode
void launchExpandForces(const DevData& d, int mode, cudaStream_t s);

// reduced parts (part_kernels.cu): the element pass, the Newton matrices and
// the end-of-step copy of the deformation; preparePartKernels sets the shared
// memory the batch's largest part needs (0, or < 0 on error)
int preparePartKernels(const DevData& d);
void launchParts(const DevData& d, int mode, cudaStream_t s);
void launchPartsNewton(const DevData& d, cudaStream_t s);
void launchPartsStepEnd(const DevData& d, cudaStream_t s);

// --- front_cascade.cu: one launch per phase over all fronts of all models ----
// Large fronts: the blocks of a launch work through waves; tasks[wave * grid +
// block] is the block's front in that wave (f < 0: none), the front's ordinal
// among the large ones, the block's rank and the number of blocks on the front.
struct LargeTask {
  int f, li, rank, G;
};
struct LargePlan {
  const LargeTask* tasks = nullptr;
  int nWaves = 0, grid = 0;
  bool wide = false;             // some level has more fronts than SMs: several blocks per SM
  const int* expect = nullptr;   // per large front: signals of its large children's blocks
  const int* parent = nullptr;   // per large front: its (large) parent's ordinal, or -1
  // inverse row maps: inv[invOff[li] + c * nrow + i] = update row of child c at row i, or -1
  const int* inv = nullptr;
  const int64_t* invOff = nullptr;
  // the children's update-vector entries of each row, in child order:
  // gSrc[gOff[gRow[li] + i]] .. up to gOff[gRow[li] + i + 1]
  const int* gOff = nullptr;
  const int* gSrc = nullptr;
  const int* gRow = nullptr;
  // original entries of each pivot column: asmCol[asmColOff[li] + j] .. [+ j + 1]
  // (offsets from the front's first entry), and each pivot's diagonal entry
  // (index into the assembled values)
  const int* asmCol = nullptr;
  const int* asmColOff = nullptr;
  const int* diagAsm = nullptr;
  const int* diagOff = nullptr;
  // pivot blocks of 32: the fronts and their parts of them, each front's first one,
  // and their inverses (2048 values each; see front_large.cu)
  int nInvBlk = 0;
  const int* invFront = nullptr;
  const int* invPart = nullptr;
  const int* invBlk = nullptr;
  void* inverse = nullptr;
  int maxRow = 0;                // largest large front (rows)
  int64_t stageCap = 0;          // values of L a block of the solves can stage
  int *done = nullptr, *bar = nullptr, *err = nullptr;
  long long spinLimit = 0;
};
// Small-front trees cut into chunks of at most `warps` fronts (front_cascade.cu,
// kTree): fronts chunks[c].off .. + n with their levels inside the chunk
// (children below their parents), ascending.
struct TreeChunk {
  int off, n, levels, model;
  int parent, parentNeed;  // the chunk of the root's parent front (-1: none) and that chunk's child chunks
  int kidOff, nKids;       // child chunks
};
struct TreePlan {
  const TreeChunk* chunks = nullptr;
  const int* fronts = nullptr;
  const unsigned char* level = nullptr;
  const int* kids = nullptr;
  const int* start = nullptr;  // chunks without child chunks, longest root path first
  int nStart = 0;
  int nChunks = 0;
  int warps = 0;  // fronts per chunk at most, and warps per block (0: no such trees)
};
struct PersistentPlan {
  TreePlan tree;
  const int* leaves;  // fronts without children, longest root path first (factorisation)
  int nLeaves;
  // forward-elimination tasks, longest root path first: a leaf, or a front
  // whose children are all leaves with bit 30 set (a group, eliminated by one
  // warp)
  const int* tasks;
  int nTasks;
  int maxRow;         // largest front of the batch (rows)
  int maxNpiv;        // largest pivot block of the batch
  int maxAsm;         // largest number of original entries of one front
  int maxSeg;         // largest children update segment of one front (packed lower values)
  // per-front counters, each followed by the launch's leaf counter: one set for
  // the factorisation, one per refinement forward elimination (nfrontTot + 1
  // apart); zeroed with the other iteration counters at the iteration start
  int *cntFactor, *cntForward, *errFlag;
  // backward work queues, one per solve of the iteration (nLeaves slots apart),
  // and their counters (4 per queue), seeded by the step-start kernels; the
  // fronts whose leaf children are solved inline
  const unsigned char* bwInline;
  int *bwQueue, *bwCtr;
  // polls of a bounded wait in the back substitution before it gives up and
  // sets errFlag (about 1-2 s at the default)
  long long spinLimit = 1LL << 23;
  // large fronts (more than kLargeFrontRows rows, and all their ancestors;
  // front_large.cu): their number, the plans of the factorisation for the four
  // shares of the GPU's blocks (largeCluster 2, 4, 8, 16) and of the solves
  // (large[4]), and their counters (nLarge each: factorisation signals and
  // barriers, then per solve forward signals, backward signals, backward
  // barriers), zeroed with the other iteration counters
  int nLarge = 0;
  LargePlan large[5];
  int* cntLarge = nullptr;
  // the trees' counters (nChunks + 1 per solve: child chunks done, then the start
  // counter), queues (tree.nStart slots per solve) and queue counters (4 per solve)
  int *cntTree = nullptr, *treeQueue = nullptr, *treeCtr = nullptr;
  // Launch shapes, picked per batch by the engine's autotuner.  No choice
  // changes a result bit: tasks are taken dynamically, and each front's
  // arithmetic is the same whichever warp or block does it.
  int factorPanel = 0;     // small-front panel factorisation: 0 shuffles, 1 register-blocked
                           // (blocks of 8), 2 register-blocked (blocks of 4, fronts up to 32 rows)
  int forwardWarps = 8;    // warps per block of the forward-elimination cascade
  int backwardWarps = 8;   // warps per block of the back-substitution queue
  int largeCluster = 16;   // sixteenths of the GPU's SMs the large-front factorisation runs on (2, 4, 8 or 16)
};
// fronts with more rows than this are factored and solved by several thread
// blocks each (front_large.cu); smaller ones by one warp each in shared memory.
// 8 steps of the space-frame tower with the line at 96 / 64 / 48 rows: FP64 16.1 /
// 15.6 / 13.8 ms, mixed 14.7 / 14.1 / 13.0; 20 steps of 16 reduced parts, FP64 (80
// row leaf fronts): 24.4 / 19.9 / 19.0 ms.  Batches, an iteration in microseconds at
// 96 / 64 / 48, FP64 (mixed): 4 such towers 1168 / 1008 / 1005 (767 / 773 / 660), 16
// frames of 6 x 3 737 / 672 / 662 (606 / 506 / 565), 128 of 3 x 2 713 / 560 / 529 (601 /
// 493 / 467), 16 chains of 16 parts 371 / 287 / 287 (303 / 291 / 291).  Chains of 8 parts
// of 32 DOFs, whose largest fronts have 60 rows, are better off at 64: 64 of them 205 / 204
// / 220 (197 / 197 / 273).  Fronts of beam chains (up to 30 rows) stay below it: there the
// trees' parallelism suffices.
constexpr int kLargeFrontRows = 48;
// the large-front kernels: factorisation (tangent models), forward elimination
// of rhs and back substitution (active models; before the warp queue's small
// fronts) of solve `sweep` of the iteration
void launchLargeFactor(const DevData& d, const PersistentPlan& p, bool fp32, cudaStream_t s);
void launchLargeForward(const DevData& d, const PersistentPlan& p, bool fp32, const double* rhs, int sweep,
                        cudaStream_t s);
void launchLargeBackward(const DevData& d, const PersistentPlan& p, bool fp32, int sweep, bool last, cudaStream_t s);
// blocks per SM of the large fronts' factorisation, or of their solves with so many bytes
// of shared memory a block (0: not one fits); wide: more than one, see LargePlan
int largeBlocksPerSm(bool fp32, bool solve, bool wide, size_t smem);
size_t largeSolveShared(int maxRow, int64_t stage, size_t elemBytes);
// values of L a block of the large-front solves stages for a front shared by G blocks
int64_t largeSolveStage(int nr, int np, int G, size_t elemBytes);
// The trees on thread blocks take all small fronts of a batch of at most kTreeAllLeaves
// leaf fronts, or the levels from a height on (treeTopHeight, -1: none; lowest: the number
// of subtrees' lowest fronts from a height on) of one of at most kTreeTopLeaves, where
// the cut into chunks pays; else the cascades do.
constexpr int kTreeAllLeaves = 8192, kTreeTopLeaves = 32768;
int treeTopHeight(int maxHeight, const std::function<long long(int)>& lowest);
bool treesPay(int nChunks, long long nFronts, int warps, int fromHeight);
// their warps per block (and fronts per chunk) for nLeaves leaf fronts (0: the upper
// levels of a larger batch) and fronts of at most maxRow rows; 0: too few fit
int treeWarps(int nLeaves, int maxRow, bool fp32);
// values of one front's L block the solve kernels stage in shared memory
int stagingCapacity(const PersistentPlan& p, size_t elemBytes);
// The first solve's back substitution run by the factorisation's own launch
// (its warps serve the solve's queue once every leaf is taken); queue null:
// not fused.  Batches without large fronts only.
struct FusedBackward {
  int* queue = nullptr;
  int* ctr = nullptr;
  const unsigned char* bwInline = nullptr;
  int* errFlag = nullptr;
  long long spinLimit = 0;
  int acc = 0, finalize = 0, capL = 0;
};
// whether the factorisation's launch can run the first back substitution: no
// large fronts, and every front's L block fits the warp's staging area (the
// fused solve reads L through L2 into shared memory)
bool fusableBackward(const PersistentPlan& p, bool fp32);
// factorisation of the models with a tangent update fused with the forward
// elimination of rhs for every active model (first solve of an iteration);
// withBackward: the back substitution of that solve too (lastSweep: it is the
// iteration's last solve), in place of launchBackward for sweep 0
void launchFactorForwardCascade(const DevData& d, const PersistentPlan& p, bool fp32, const double* rhs,
                                cudaStream_t s, bool withBackward = false, bool lastSweep = false);
// forward elimination of the right-hand side rhs (FP64, rounded to the solve precision)
// (withBackward, trees on thread blocks only: the back substitution of that
// sweep too, in place of launchBackward; lastSweep: it is the iteration's last)
void launchForwardCascade(const DevData& d, const PersistentPlan& p, bool fp32, const double* rhs, int sweep,
                          cudaStream_t s, bool withBackward = false, bool lastSweep = false);
// back substitution; stores the solution in del (FP64 solve) or accumulates it in xref
// (FP32 refinement sweep `sweep`; the last sweep also copies xref to del)
// (treeDone: the trees' part already ran)
void launchBackward(const DevData& d, const PersistentPlan& p, bool fp32, int sweep, bool last, cudaStream_t s,
                    bool treeDone = false);
// One warp of the back-substitution queue kernel on a private queue (4 ints of
// counters at ctr, the slots at queue), waiting at most `spins` polls: with an
// empty slot 0 and a slot total of 1 the wait runs out and sets p.errFlag.
void launchBackwardWaitProbe(const DevData& d, const PersistentPlan& p, int* queue, int* ctr, long long spins,
                             cudaStream_t s);
// One warp of the fused factorisation without leaves on a private queue whose
// slot 0 holds a root of an active model and private counters cnt (zeroed,
// nfrontTot + 1): the root's release never comes, so the bounded wait runs out
// after `spins` polls and sets p.errFlag.
void launchRootWaitProbe(const DevData& d, const PersistentPlan& p, int* queue, int* ctr, int* cnt, long long spins,
                         cudaStream_t s);
// prescribed deflections (step start), their predictor right-hand side (after the
// element Newton matrices), and the restart state of pure linear quasi-static steps
void launchMotions(const DevData& d, cudaStream_t s);
void launchLoads(const DevData& d, cudaStream_t s);
void launchMotionRhs(const DevData& d, cudaStream_t s);
void launchQsRestore(const DevData& d, cudaStream_t s);
// synthetic, diagonally dominant original entries of every front (the
// autotuner's timing probe, before the first iteration gathers the real ones)
void launchProbeEntries(const DevData& d, bool fp32, cudaStream_t s);
// results database of the primary response (results.cu): per model a ring of
// kRecordRing records (step, time, triad positions, superelement frames and
// generalized DOFs, as doubles) in buf, written at each completed step
struct RecordPlan {
  double* buf = nullptr;       // the rings, model after model
  long long* off = nullptr;    // per model: first value of its ring
  int* vals = nullptr;         // per model: values per record (2 + data)
  int* triRec = nullptr;       // per triad (global): offset of its values in its model's record
  int* elRec = nullptr;        // per model: offset of its beam frames (12 per element)
  int* partFirst = nullptr;    // per model, + 1: first reduced part (global)
  int* partRec = nullptr;      // per part: offset of its frame and generalized DOFs
  long long* count = nullptr;  // per model: records written so far
  int ring = 0;
};
constexpr int kRecordRing = 8;
// all: a record of every model's current state; otherwise of the models whose
// step has just completed
void launchRecordStep(const DevData& d, const RecordPlan& r, bool all, cudaStream_t s);
// FP64 refinement residual r = b - A x (front_kernels.cu)
void launchRefineResidual(const DevData& d, cudaStream_t s);

// Convergence norms of model m recomputed into a fixed scratch array compiled
// into the library (no device allocation); blocks until the 18 values are in
// out18 (host).  c0/nc: the model's first norm chunk and chunk count; dev: the
// batch's device (made current for the launch).
int normsNoAlloc(const DevData& d, int m, int c0, int nc, int dev, cudaStream_t s, double* out18, std::string& err);

// One block of the trees, or of a large-front solve, that waits at most `spins` polls for
// what nothing gives: an empty queue slot 0 or (root) the elimination of the root in it;
// the large children of a task's front or (backward) the second of its blocks.
void launchTreeWaitProbe(const DevData& d, const PersistentPlan& p, bool fp32, int* queue, int* ctr, int* cnt,
                         bool root, long long spins, cudaStream_t s);
void launchLargeWaitProbe(const DevData& d, const PersistentPlan& p, bool fp32, const LargeTask* task, int* done,
                          int* bar, bool backward, long long spins, cudaStream_t s);

}  // namespace fgpu

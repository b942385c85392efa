// front_cascade.cu -- one-launch multifrontal factorisation and solves over
// the assembly trees of all models, without co-residency assumptions.
//
// Factor and forward solve run bottom-up as a cascade: warps start at the
// leaves; a front's counter is incremented (release) when one of its children
// is done, and the warp whose increment completes the count goes on with the
// parent itself.  Nothing ever waits, so the launch is correct whatever the
// residency (several engines may run concurrently on their own streams).
// The backward solve runs top-down through a work queue of fronts whose
// parents are solved (kBackwardQueue); a warp waits only for a queue slot to
// be filled, by warps that are running and never wait themselves, so the wait
// ends whatever the residency.  Each wait is still bounded and sets errFlag
// when it runs out.
// Batches of few or deep trees, up to 32,768 leaf fronts, pay the cascades' latency per
// tree level, not their work; there whole subtrees go to thread blocks, a warp per front
// (kTree; treesPay).
// The forward and backward solves stage each front's L block in shared memory
// first (one burst of loads instead of one load latency per pivot).
//
// These kernels replace the factor and solve of the absent SAM/SPR solver that
// the reference calls from csSolve (src/vpmCommon/vpmLinAlg/
// solExtensionModule.f90:153-505: SPRFC1/SPRFC3, SPRFS1/SPRBS1).  Semantics
// kept: LDL^T without pivoting, a pivot counts as singular when
// |d_k| <= tolFactorize * |a_kk| (error -3), negative pivots are counted.
// Fronts are dense column-major nrow x nrow tiles in shared memory (lower
// triangle used), pivots first; children's contributions are added in child
// order, so every sum has a fixed order (no atomics on floating-point data).
// Mixed precision: FP32 factor and correction solves; the FP64 refinement
// residual is in front_kernels.cu.

#include <algorithm>
#include <atomic>

#include "kernels.h"
#include "pivot.cuh"

namespace fgpu {
namespace {


// Partial LDL^T of a front, blocked: the pivot panel (all rows, the np
// pivot columns) is factored right-looking within the panel, one row per lane;
// the update matrix (the Schur complement of the update block) is then formed
// in one rank-np pass over its lower triangle, one entry per lane, and stored
// packed column by column at Uout.  F afterwards holds D on the diagonal and
// the unit L below it in the panel; the unscaled panel values of the update
// rows (L d) are kept in the unused upper triangle (row k, column i) for the
// rank-np pass.
// Panel factorisations of the small fronts, all with the same arithmetic in
// the same order (so the same factor to the last bit), picked per batch by the
// engine's autotuner: pivot by pivot with the multipliers passed by shuffles
// and the rows kept in shared memory (few registers, high occupancy), or
// register-blocked (fewer instructions and shared-memory accesses, more
// registers) in blocks of 8 or 4 pivots.
constexpr int kPanelShuffle = 0;
constexpr int kPanelRegisters = 1;   // blocks of 8 pivots, fronts up to 64 rows
constexpr int kPanelRegisters4 = 2;  // blocks of 4 pivots, one row per lane (fronts up to 32 rows)

// pivot by pivot: rows lane and lane + 32 in shared memory; the multipliers of
// the pivot rows (lanes below np) are passed by shuffles, one barrier per pivot
template <typename T>
__device__ void panelShuffle(T* F, const T* diag0, int nr, int np, int lane, int& neg, bool& sing) {
  const int i0 = lane, i1 = lane + 32;
  for (int k = 0; k < np; ++k) {
    const T dk = F[k + nr * k];
    const bool bad = !absGreater(dk, diag0[k]);
    sing |= bad;
    if (negative(dk)) ++neg;
    const T inv = bad ? T(0) : T(1) / dk;
    const bool r0 = i0 > k && i0 < nr, r1 = i1 > k && i1 < nr;
    const T f0 = r0 ? F[i0 + nr * k] : T(0), f1 = r1 ? F[i1 + nr * k] : T(0);
    const T l0 = f0 * inv, l1 = nr > 32 ? f1 * inv : T(0);
    for (int j = k + 1; j < np; ++j) {
      const T lj = __shfl_sync(0xffffffffu, l0, j);
      if (r0 && j <= i0) F[i0 + nr * j] -= f0 * lj;
      if (r1) F[i1 + nr * j] -= f1 * lj;
    }
    if (r0) {
      if (i0 >= np) F[k + nr * i0] = f0;
      F[i0 + nr * k] = l0;
    }
    if (r1) {
      if (i1 >= np) F[k + nr * i1] = f1;
      F[i1 + nr * k] = l1;
    }
    __syncwarp();
  }
}

// register-blocked in blocks of PB pivots (TWO: a second row per lane, fronts
// of up to 64 rows; else at most 32 rows)
template <typename T, int PB, bool TWO>
__device__ void panelRegisters(T* F, const T* diag0, int nr, int np, int lane, int& neg, bool& sing) {
  // Register-blocked panel: lane r owns rows r and r + 32; the pivot columns
  // are taken PB at a time.  Inside a block the row values sit in
  // registers and each multiplier l_jk is passed by a shuffle from the lane
  // owning row j; the block's columns are then stored (l_ik below the
  // diagonal, the unscaled value of an update row in its upper position),
  // and the later pivot columns receive the block's updates all at once,
  // l_jk read from shared memory (one broadcast load per value).  Every
  // entry receives the same multiply-subtracts in the same order as in a
  // right-looking elimination one pivot at a time, so the factor is the same
  // to the last bit, with a fraction of the shared-memory traffic and no
  // barrier per pivot.
  const int i0 = lane, i1 = lane + 32;
  const bool two = TWO && nr > 32;     // warp-uniform: a second row per lane
  const bool h1 = two && i1 < nr;      // row i1 exists (it is below every pivot: np <= 32)
  for (int k0 = 0; k0 < np; k0 += PB) {
    const int kb = min(PB, np - k0);
    const bool h0 = i0 >= k0 && i0 < nr;
    T a0[PB], a1[PB];
#pragma unroll
    for (int kk = 0; kk < PB; ++kk) {
      a0[kk] = (kk < kb && h0) ? F[i0 + nr * (k0 + kk)] : T(0);
      a1[kk] = (kk < kb && h1) ? F[i1 + nr * (k0 + kk)] : T(0);
    }
#pragma unroll
    for (int kk = 0; kk < PB; ++kk) {
      if (kk >= kb) break;  // warp-uniform
      const int k = k0 + kk;
      const T dk = __shfl_sync(0xffffffffu, a0[kk], k);  // row k < 32 is lane k's first row
      const bool bad = !absGreater(dk, diag0[k]);
      sing |= bad;
      if (negative(dk)) ++neg;
      const T inv = bad ? T(0) : T(1) / dk;
      const bool r0 = i0 > k && i0 < nr;
      const T f0 = r0 ? a0[kk] : T(0), f1 = h1 ? a1[kk] : T(0);
      const T l0 = f0 * inv, l1 = two ? f1 * inv : T(0);
#pragma unroll
      for (int jj = kk + 1; jj < PB; ++jj) {
        if (jj >= kb) break;
        const T lj = __shfl_sync(0xffffffffu, l0, k0 + jj);
        if (r0 && k0 + jj <= i0) a0[jj] -= f0 * lj;
        if (h1) a1[jj] -= f1 * lj;
      }
      if (i0 == k) F[k + nr * k] = dk;
      if (r0) {
        F[i0 + nr * k] = l0;
        if (i0 >= np) F[k + nr * i0] = f0;
        a0[kk] = f0;
      }
      if (h1) {
        F[i1 + nr * k] = l1;
        if (i1 >= np) F[k + nr * i1] = f1;
        a1[kk] = f1;
      }
    }
    __syncwarp();
    // the later pivot columns j (row i >= j): C(i, j) -= f_i,k l_j,k over the block's k in order
    for (int j = k0 + kb; j < np; ++j) {
      T lj[PB];
#pragma unroll
      for (int kk = 0; kk < PB; ++kk) lj[kk] = kk < kb ? F[j + nr * (k0 + kk)] : T(0);
      if (i0 >= j && i0 < nr) {
        T c = F[i0 + nr * j];
#pragma unroll
        for (int kk = 0; kk < PB; ++kk)
          if (kk < kb) c -= a0[kk] * lj[kk];
        F[i0 + nr * j] = c;
      }
      if (h1) {
        T c = F[i1 + nr * j];
#pragma unroll
        for (int kk = 0; kk < PB; ++kk)
          if (kk < kb) c -= a1[kk] * lj[kk];
        F[i1 + nr * j] = c;
      }
    }
    __syncwarp();
  }
}

template <typename T, int PANEL>
__device__ void factorBlocked(T* F, T* lcol, const T* diag0, int nr, int np, int lane, int& neg, bool& sing, T* Uout) {
  if (np <= 32 && nr <= 64) {
    if constexpr (PANEL == kPanelRegisters) {
      panelRegisters<T, 8, true>(F, diag0, nr, np, lane, neg, sing);
    } else if constexpr (PANEL == kPanelRegisters4) {
      if (nr <= 32) panelRegisters<T, 4, false>(F, diag0, nr, np, lane, neg, sing);
      else panelShuffle<T>(F, diag0, nr, np, lane, neg, sing);
    } else {
      panelShuffle<T>(F, diag0, nr, np, lane, neg, sing);
    }
  } else {
    for (int k = 0; k < np; ++k) {
      const T dk = F[k + nr * k];
      const bool bad = !absGreater(dk, diag0[k]);
      sing |= bad;
      if (negative(dk)) ++neg;
      const T inv = bad ? T(0) : T(1) / dk;
      for (int i = k + 1 + lane; i < nr; i += 32) lcol[i] = F[i + nr * k] * inv;
      __syncwarp();
      for (int i = k + 1 + lane; i < nr; i += 32) {
        const T fik = F[i + nr * k];
        const int je = i < np - 1 ? i : np - 1;
        for (int j = k + 1; j <= je; ++j) F[i + nr * j] -= fik * lcol[j];
        if (i >= np) F[k + nr * i] = fik;
        F[i + nr * k] = lcol[i];
      }
      __syncwarp();
    }
  }
  // update matrix, lower triangle packed column by column: entry e = lane + 32 q
  // is (row np + b + t, column np + b)
  const int nu = nr - np;
  int b = 0, t = lane;
  while (b < nu && t >= nu - b) { t -= nu - b; ++b; }
  for (int e = lane; b < nu; e += 32) {
    const int i = np + b + t, j = np + b;
    T v = F[i + nr * j];
    for (int k = 0; k < np; ++k) v -= F[k + nr * i] * F[j + nr * k];
    Uout[e] = v;
    t += 32;
    while (b < nu && t >= nu - b) { t -= nu - b; ++b; }
  }
  __syncwarp();
}

// extend-add of N entries per lane, entry u of lane l the (32 u + l)-th of the front's
// children segment (pos: child << 20 | position, or -1 past its end).  The segment holds
// the children in order, so 32 entries are of one child, or of two or a few at a seam:
// they are added child by child, positions of one child being distinct.  (One pass over
// all N per child took twice the instructions, half of them without an active lane.)
template <typename T, int N>
__device__ __forceinline__ void extendAdd(T* F, const int* pos, const T* val) {
#pragma unroll
  for (int u = 0; u < N; ++u) {
    unsigned left = __ballot_sync(0xffffffffu, pos[u] >= 0);
    while (left) {
      const int c = __shfl_sync(0xffffffffu, pos[u], __ffs(left) - 1) >> 20;
      const bool on = pos[u] >= 0 && (pos[u] >> 20) == c;
      if (on) F[pos[u] & 0xfffff] += val[u];
      __syncwarp();
      left &= ~__ballot_sync(0xffffffffu, on);
    }
  }
}

// partial LDL^T of front f in shared memory (F: maxRow^2, lcol/diag0: maxRow).
// The original entries (front-ordered copy of the CSR values) and the
// children's packed update matrices are contiguous per front and loaded
// kFrontBatch per lane before use; the rank-1 updates run one row per lane.
constexpr int kFrontBatch = 4;
// Uout: the front's packed update matrix (its place in the parent's
// segment); segIn: the front's own children segment
template <typename T, int PANEL>
__device__ void factorOneFront(const DevData& d, int f, T* F, T* lcol, T* diag0, const T* asmVal, T* Lbase,
                               T* Uout, const T* segIn, double tolFact, int lane) {
  const int m = d.fModel[f];
  const int nr = d.fNrow[f], np = d.fNpiv[f];
  const int64_t ao = d.fAsmOff[f], so = d.fSegOff[f];
  const int na = d.fNasm[f], ns = d.fSegLen[f];
  for (int k = lane; k < nr * nr; k += 32) F[k] = T(0);
  for (int k0 = 0; k0 < na; k0 += 32 * kFrontBatch) {
    T val[kFrontBatch];
    int pos[kFrontBatch];
#pragma unroll
    for (int u = 0; u < kFrontBatch; ++u) {
      const int k = k0 + 32 * u + lane;
      pos[u] = k < na ? __ldg(d.asmPos + ao + k) : -1;
      val[u] = k < na ? __ldg(asmVal + ao + k) : T(0);
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < kFrontBatch; ++u)
      if (pos[u] >= 0) F[pos[u]] = val[u];
  }
  __syncwarp();
  // a pivot counts as singular when |d_k| <= tolFactorize * |a_kk|
  for (int k = lane; k < np; k += 32) diag0[k] = singularBound(F[k + nr * k], (T)tolFact);
  __syncwarp();
  // extend-add of the children's update matrices, child by child
  for (int k0 = 0; k0 < ns; k0 += 32 * kFrontBatch) {
    T val[kFrontBatch];
    int pc[kFrontBatch];
#pragma unroll
    for (int u = 0; u < kFrontBatch; ++u) {
      const int k = k0 + 32 * u + lane;
      pc[u] = k < ns ? __ldg(d.segPos + so + k) : -1;
      val[u] = k < ns ? __ldcg(segIn + k) : T(0);
    }
    extendAdd<T, kFrontBatch>(F, pc, val);
  }
  int neg = 0;
  bool sing = false;
  factorBlocked<T, PANEL>(F, lcol, diag0, nr, np, lane, neg, sing, Uout);
  T* Lout = Lbase + d.fLOff[f];
  for (int k = lane; k < nr * np; k += 32) Lout[k] = F[k];
  if (lane == 0) {
    if (neg) atomicAdd(&d.m.negPiv[m], neg);
    if (sing) atomicOr(&d.m.status[m], SS_SINGULAR);
  }
}

// forward elimination of front f: v = [b_p; 0] + children's updates, y = L11^-1 v_p,
// w = v_u - L21 y; X(pivots) = D^-1 y
// copies the nr x np block L of a front into the warp's staging area Ls when
// it fits (capL values), else returns the global block
// asynchronous global -> shared copies of single elements (cp.async): every
// copy of a block is in flight at once and none occupies a register
template <typename T>
__device__ inline void copyAsync(T* dstShared, const T* srcGlobal) {
  static_assert(sizeof(T) == 4 || sizeof(T) == 8, "4- or 8-byte elements");
  const unsigned dst = (unsigned)__cvta_generic_to_shared(dstShared);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(dst), "l"(srcGlobal), "n"(sizeof(T)));
}
__device__ inline void copyAsyncWait() {
  asm volatile("cp.async.commit_group;\n" ::);
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// copies the L block into Ls (callers wait with copyAsyncWait and __syncwarp
// before reading Ls); returns the global block when it does not fit
template <typename T>
__device__ inline const T* stageL(const T* Lg, int cnt, T* Ls, int capL, int lane) {
  if (cnt > capL) return Lg;
  for (int k = lane; k < cnt; k += 32) copyAsync(Ls + k, Lg + k);
  return Ls;
}

template <typename T>
__device__ void forwardOneFront(const DevData& d, int f, T* v, T* Ls, int capL, const T* Lbase, const double* rhs,
                                T* X, T* W, int lane, const T* Lres = nullptr) {
  const int nr = d.fNrow[f], np = d.fNpiv[f], nu = nr - np;
  const int* rows = d.frontRows + d.fRowOff[f];
  // the factor block first (independent loads; or the front just factored in
  // shared memory), then the right-hand side of the pivot rows rounded to the
  // solve precision
  const T* L = Lres ? Lres : stageL(Lbase + d.fLOff[f], nr * np, Ls, capL, lane);
  for (int r = lane; r < nr; r += 32) v[r] = r < np ? (T)rhs[__ldg(rows + r)] : T(0);
  copyAsyncWait();
  __syncwarp();
  const int nc = d.fNchild[f];
  const int64_t co = d.fChildOff[f];
  for (int c = 0; c < nc; ++c) {
    const int ch = d.childList[co + c];
    const int cu = d.fNrow[ch] - d.fNpiv[ch];
    const T* wc = W + d.fWOff[ch];
    const int* rel = d.relIndex + d.fRelOff[ch];
    for (int a = lane; a < cu; a += 32) v[__ldg(rel + a)] += __ldcg(wc + a);
    __syncwarp();
  }
  for (int k = 0; k < np; ++k) {
    const T yk = v[k];
    __syncwarp();
    for (int i = k + 1 + lane; i < nr; i += 32) v[i] -= L[i + (size_t)nr * k] * yk;
    __syncwarp();
  }
  for (int r = lane; r < np; r += 32) X[rows[r]] = v[r] / L[r + (size_t)nr * r];
  T* wo = W + d.fWOff[f];
  for (int a = lane; a < nu; a += 32) wo[a] = v[np + a];
}

// Forward elimination with few dependent memory round trips (fronts of at most
// 64 rows and 64 child update rows): the front's descriptors, then its L block
// (asynchronous copies), row list and child gather list together, then the
// right-hand side and the children's update values together.

// Wout: where the front's update vector goes; Win: the children's update
// vectors concatenated in child order in shared memory (their gather list
// order), or null to read them from W
// Descriptors a solve of front f reads, loaded together in one round of
// independent loads (every lane the same address: broadcasts).  The caller
// loads them early, the parent's climb data right after (ParentLink), so that
// neither costs a round trip of its own later.
struct SolveDesc {
  int f, nr, np, cg0, ncg, nch, parent;
  int64_t lOff, rowOff, wOff;
};
__device__ inline SolveDesc solveDesc(const DevData& d, int f) {
  SolveDesc q;
  q.f = f;
  q.nr = d.fNrow[f];
  q.np = d.fNpiv[f];
  q.cg0 = d.cgOff[f];
  q.ncg = d.cgOff[f + 1] - q.cg0;
  q.nch = d.fNchild[f];
  q.parent = d.fParent[f];
  q.lOff = d.fLOff[f];
  q.rowOff = d.fRowOff[f];
  q.wOff = d.fWOff[f];
  return q;
}

// the arithmetic of a forward elimination (fronts of at most 64 rows and 64
// child update rows) on loaded values: lane r has rows and child entries r, r + 32
template <typename T>
__device__ void forwardRun(const SolveDesc& q, const int* row, const int* dst, const int* src, const double* b,
                           const T* wv, T* v, const T* L, T* X, int lane, T* Wout) {
  const int nr = q.nr, np = q.np, nch = q.nch;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int r = lane + 32 * u;
    if (r < nr) v[r] = r < np ? (T)b[u] : T(0);
  }
  __syncwarp();
  for (int c = 0; c < nch; ++c) {
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (src[u] >= 0 && (dst[u] >> 16) == c) v[dst[u] & 0xffff] += wv[u];
    __syncwarp();
  }
  // the elimination with the rows in registers (lane r: rows r and r + 32), the
  // pivot value of each step passed by a shuffle: no barrier between steps
  T v0 = lane < nr ? v[lane] : T(0), v1 = lane + 32 < nr ? v[lane + 32] : T(0);
  if (nr <= 32) {
    for (int k = 0; k < np; ++k) {
      const T yk = __shfl_sync(0xffffffffu, v0, k);
      if (lane > k && lane < nr) v0 -= L[lane + (size_t)nr * k] * yk;
    }
  } else {
    for (int k = 0; k < np; ++k) {
      const T yk = __shfl_sync(0xffffffffu, k < 32 ? v0 : v1, k & 31);
      const T* Lk = L + (size_t)nr * k;
      if (lane > k && lane < nr) v0 -= Lk[lane] * yk;
      if (lane + 32 > k && lane + 32 < nr) v1 -= Lk[lane + 32] * yk;
    }
  }
  if (lane >= np && lane < nr) Wout[lane - np] = v0;
  if (lane + 32 >= np && lane + 32 < nr) Wout[lane + 32 - np] = v1;
  if (lane < np) X[row[0]] = v0 / L[lane + (size_t)nr * lane];
  if (lane + 32 < np) X[row[1]] = v1 / L[(lane + 32) + (size_t)nr * (lane + 32)];
}

template <typename T>
__device__ bool forwardOneFrontFast(const DevData& d, const SolveDesc& q, T* v, T* Ls, int capL, const T* Lbase,
                                    const double* rhs, T* X, const T* W, int lane, const T* Lres, T* Wout,
                                    const T* Win = nullptr) {
  const int nr = q.nr, np = q.np;
  const int cg0 = q.cg0, ncg = q.ncg, nch = q.nch;
  const int cnt = nr * np;
  if (nr > 64 || ncg > 64 || (!Lres && cnt > capL)) return false;
  const int* rows = d.frontRows + q.rowOff;
  // second round of loads: independent loads (the L block asynchronously into shared memory)
  if (!Lres) {
    const T* Lg = Lbase + q.lOff;
    for (int k = lane; k < cnt; k += 32) copyAsync(Ls + k, Lg + k);
  }
  int row[2], src[2], dst[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int r = lane + 32 * u;
    row[u] = r < np ? __ldg(rows + r) : -1;
    src[u] = r < ncg ? __ldg(d.cgSrc + cg0 + r) : -1;
    dst[u] = r < ncg ? __ldg(d.cgDst + cg0 + r) : 0;
  }
  // third round of loads: values through the indices
  double b[2];
  T wv[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    b[u] = row[u] >= 0 ? rhs[row[u]] : 0.0;
    wv[u] = src[u] < 0 ? T(0) : Win ? Win[lane + 32 * u] : __ldcg(W + src[u]);
  }
  if (!Lres) copyAsyncWait();
  forwardRun<T>(q, row, dst, src, b, wv, v, Lres ? Lres : Ls, X, lane, Wout);
  return true;
}

// After a front is done: release its data and count it at the parent; true
// if this warp completed the parent's count (and must go on with the parent),
// false otherwise (also for a large parent: the large-front kernels take it up
// afterwards).  The parent's id, size class and child count (ParentLink) are
// loaded while the front is still being processed, so the climb itself is one
// atomic.  The warp barrier orders every lane's stores before lane 0's counter
// update, a release-acquire RMW at GPU scope (no full fence): the warp that
// completes the count acquires the children's stores, and its barrier passes
// them on to its other lanes.
struct ParentLink {
  int p, nch;
  bool large;
};
__device__ inline ParentLink parentLink(const DevData& d, int p) {
  ParentLink l{p, 0, true};
  if (p >= 0) {
    l.large = d.fLarge[p] != 0;
    l.nch = d.fNchild[p];
  }
  return l;
}
__device__ inline bool climb(const ParentLink& l, int* cnt, int lane) {
  __syncwarp();
  int go = 0;
  if (lane == 0 && l.p >= 0 && !l.large) {
    int old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;\n" : "=r"(old) : "l"(cnt + l.p) : "memory");
    go = old == l.nch - 1;
  }
  go = __shfl_sync(0xffffffffu, go, 0);
  __syncwarp();
  return go != 0;
}

// A root's elimination is complete: its counter gets kRootDone added with
// release semantics (after the warp barrier that orders every lane's stores),
// which the fused back substitution acquires before it solves the root.
constexpr int kRootDone = 1 << 24;
__device__ inline void releaseRoot(int* cnt, int f, int lane) {
  __syncwarp();
  if (lane == 0) asm volatile("red.release.gpu.global.add.s32 [%0], %1;\n" ::"l"(cnt + f), "r"(kRootDone) : "memory");
  __syncwarp();
}
__device__ inline int acquireCount(const int* c) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];\n" : "=r"(v) : "l"(c) : "memory");
  return v;
}

// Leaves are taken in their stored order (longest root paths first) from a
// launch-wide counter, cnt[nfrontTot]; lane 0 asks for the next leaf before
// the current one is processed, so the request's latency is hidden.
__device__ inline int requestLeaf(int* next, int lane) { return lane == 0 ? atomicAdd(next, 1) : 0; }

// Forward-elimination tasks are single leaves or groups: a group is a front
// whose children are all leaves (kGroupBit set in the task), eliminated by one
// warp -- the children first, their update vectors kept in shared memory, then
// the front itself -- so that inside a group nothing goes through global
// memory or a counter.  After a task the warp climbs as from a leaf.  (The
// factorisation keeps one task per leaf: there the leaves are the most
// expensive fronts, and factoring siblings one after the other lengthens the
// critical path more than the saved climbs shorten it.)
constexpr int kGroupBit = 1 << 30;

// factorisation (models with a tangent update) fused with the forward
// elimination of the first solve (all active models): one climb per front, and
// the forward elimination reads L from the front still in shared memory
template <typename T>
__device__ void backwardQueueLoop(const DevData& d, int maxRow, int capL, const T* Lbase, T* X, int* queue, int* ctr,
                                  const unsigned char* bwInline, int* errFlag, int acc, int finalize,
                                  long long spinLimit, T* xs, T* Ls, int lane, const int* rootDone);
template <typename T, int PANEL>
__global__ void kFactorForwardCascade(DevData d, const int* __restrict__ leaves, int nLeaves, int maxRow,
                                      const T* asmVal, T* Lbase, T* Ubase, double tolFact, const double* rhs, T* X,
                                      T* Wv, int* cnt, FusedBackward fb) {
  pdlEntry();
  extern __shared__ __align__(16) unsigned char smraw[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int capL = maxRow * maxRow;  // F doubles as the staging area of L
  T* F = reinterpret_cast<T*>(smraw) + (size_t)w * ((size_t)maxRow * maxRow + 3 * maxRow);
  T* lcol = F + (size_t)maxRow * maxRow;
  T* diag0 = lcol + maxRow;
  T* v = diag0 + maxRow;
  int* const next = cnt + d.nfrontTot;
  int idx = __shfl_sync(0xffffffffu, requestLeaf(next, lane), 0);
  while (idx < nLeaves) {
    const int pending = requestLeaf(next, lane);
    int f = leaves[idx];
    const int fl = d.m.flags[d.fModel[f]];
    const bool factor = fl & FL_TANGENT;
    while ((fl & FL_ACTIVE) && f >= 0) {
      const SolveDesc q = solveDesc(d, f);
      const ParentLink pl = parentLink(d, q.parent);
      const T* Lres = nullptr;
      if (factor) {
        factorOneFront<T, PANEL>(d, f, F, lcol, diag0, asmVal, Lbase, Ubase + d.fUOff[f], Ubase + d.fSegOff[f],
                                 tolFact, lane);
        __syncwarp();
        Lres = F;
      }
      if (!forwardOneFrontFast<T>(d, q, v, F, capL, Lbase, rhs, X, Wv, lane, Lres, Wv + q.wOff))
        forwardOneFront<T>(d, f, v, F, capL, Lbase, rhs, X, Wv, lane, Lres);
      if (fb.queue && q.parent < 0) releaseRoot(cnt, f, lane);
      f = climb(pl, cnt, lane) ? q.parent : -1;
    }
    idx = __shfl_sync(0xffffffffu, pending, 0);
  }
  // Fused first back substitution: once every leaf is taken, the warp serves
  // the back-substitution queue.  Every front still to be eliminated belongs to
  // a running warp that never waits, so a root the queue hands out completes;
  // the warp waits for it (bounded) before solving it.
  if (fb.queue)
    backwardQueueLoop<T>(d, maxRow, fb.capL, Lbase, X, fb.queue, fb.ctr, fb.bwInline, fb.errFlag, fb.acc, fb.finalize,
                         fb.spinLimit, v, F, lane, cnt);
}

template <typename T>
__global__ void kForwardCascade(DevData d, const int* __restrict__ tasks, int nTasks, int maxRow, int capL,
                                const T* Lbase, const double* rhs, T* X, T* W, int* cnt) {
  pdlEntry();
  extern __shared__ __align__(16) unsigned char smraw[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T* v = reinterpret_cast<T*>(smraw) + (size_t)w * (maxRow + capL + 64);
  T* Ls = v + maxRow;
  T* wsm = Ls + capL;
  int* const next = cnt + d.nfrontTot;
  int idx = __shfl_sync(0xffffffffu, requestLeaf(next, lane), 0);
  while (idx < nTasks) {
    const int pending = requestLeaf(next, lane);
    const int task = tasks[idx];
    int f = task & ~kGroupBit;
    const bool active = d.m.flags[d.fModel[f]] & FL_ACTIVE;
    if (!active) f = -1;
    SolveDesc q;
    if (f >= 0) q = solveDesc(d, f);
    if (f >= 0 && (task & kGroupBit)) {
      const ParentLink pl = parentLink(d, q.parent);
      const int* ch = d.childList + d.fChildOff[f];
      int wo = 0;
      SolveDesc cq = solveDesc(d, ch[0]);
      for (int c = 0; c < q.nch; ++c) {
        // the next child's descriptors are loaded while this one is eliminated
        const SolveDesc nq = solveDesc(d, ch[c + 1 < q.nch ? c + 1 : c]);
        forwardOneFrontFast<T>(d, cq, v, Ls, capL, Lbase, rhs, X, W, lane, nullptr, wsm + wo);
        wo += cq.nr - cq.np;
        __syncwarp();
        cq = nq;
      }
      forwardOneFrontFast<T>(d, q, v, Ls, capL, Lbase, rhs, X, W, lane, nullptr, W + q.wOff, wsm);
      f = climb(pl, cnt, lane) ? q.parent : -1;
      if (f >= 0) q = solveDesc(d, f);
    }
    while (f >= 0) {
      // the parent's climb data and descriptors are loaded ahead of this
      // front's elimination; they are used only if this warp goes on to it
      const ParentLink pl = parentLink(d, q.parent);
      const SolveDesc pq = solveDesc(d, q.parent >= 0 ? q.parent : f);
      if (!forwardOneFrontFast<T>(d, q, v, Ls, capL, Lbase, rhs, X, W, lane, nullptr, W + q.wOff))
        forwardOneFront<T>(d, f, v, Ls, capL, Lbase, rhs, X, W, lane);
      f = climb(pl, cnt, lane) ? q.parent : -1;
      q = pq;
    }
    idx = __shfl_sync(0xffffffffu, pending, 0);
  }
}

// backward substitution of front f (parent values already in X): the update
// rows' contribution for every pivot at once (one lane per pivot), then the
// unit triangle column by column; writes the pivot values to X
// accumulation of the solved pivot values: ACC_SET del = x (FP64 solve), ACC_FIRST
// xref = x, ACC_ADD xref += x (FP32 refinement sweeps); finalize: del = xref
enum { ACC_SET = 0, ACC_FIRST = 1, ACC_ADD = 2 };

// Descriptors of a back substitution, loaded together: the front's, and with
// them those of its first child (the front the warp goes on to), so that the
// next front starts without a descriptor round trip.
struct BackDesc {
  int f, nr, np, nch;
  bool inl;  // children all leaves, solved by this warp
  int64_t lOff, rowOff, childOff;
};
__device__ inline BackDesc backDesc(const DevData& d, const unsigned char* bwInline, int f) {
  BackDesc q;
  q.f = f;
  q.nr = d.fNrow[f];
  q.np = d.fNpiv[f];
  q.nch = d.fNchild[f];
  q.inl = bwInline[f] != 0;
  q.lOff = d.fLOff[f];
  q.rowOff = d.fRowOff[f];
  q.childOff = d.fChildOff[f];
  return q;
}

// l2Only: L was written in the same launch (fused back substitution), so it
// is staged through L2 loads; an L1 line filled earlier in the launch by a
// neighbouring front's solve could hold its old values (fusableBackward
// guarantees that every block fits the staging area)
// the arithmetic of a back substitution: xs holds the front's solution values
// (pivots: the eliminated right-hand side), L its block; stores the pivots'
template <typename T>
__device__ void backwardSolve(const DevData& d, const int* rows, int nr, int np, T* xs, const T* L, T* X, int acc,
                              bool finalize, int lane) {
  if (np <= 32) {
    // one pivot per lane in a register; the back substitution passes each
    // solved value by a shuffle (no barrier between steps).  The update rows' share
    // is split over 4 groups of 8 lanes (up to 8 pivots) or 2 of 16: a front of 6
    // pivots and 12 update rows takes 3 multiply-subtracts and 2 additions one after
    // the other in place of 12
    const int width = np <= 8 ? 8 : np <= 16 ? 16 : 32;
    const int p = lane & (width - 1);
    T a = lane < np ? xs[lane] : T(0);
    if (p < np)
      for (int i = np + lane / width; i < nr; i += 32 / width) a -= L[i + (size_t)nr * p] * xs[i];
    for (int o = width; o < 32; o <<= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    for (int j = np - 1; j > 0; --j) {
      const T xj = __shfl_sync(0xffffffffu, a, j);
      if (lane < j) a -= L[j + (size_t)nr * lane] * xj;
    }
    if (lane < np) xs[lane] = a;
    __syncwarp();
  } else {
    for (int k = lane; k < np; k += 32) {
      T a = xs[k];
      for (int i = np; i < nr; ++i) a -= L[i + (size_t)nr * k] * xs[i];
      xs[k] = a;
    }
    __syncwarp();
    for (int j = np - 1; j > 0; --j) {
      const T xj = xs[j];
      for (int k = lane; k < j; k += 32) xs[k] -= L[j + (size_t)nr * k] * xj;
      __syncwarp();
    }
  }
  for (int r = lane; r < np; r += 32) {
    const int row = rows[r];
    const T x = xs[r];
    X[row] = x;
    if (acc == ACC_SET) {
      d.del[row] = (double)x;
    } else {
      const double xr = acc == ACC_FIRST ? (double)x : d.xref[row] + (double)x;
      d.xref[row] = xr;
      if (finalize) d.del[row] = xr;
    }
  }
}

template <typename T>
__device__ void backwardOneFront(const DevData& d, const BackDesc& q, T* xs, T* Ls, int capL, const T* Lbase, T* X,
                                 int acc, bool finalize, int lane, bool l2Only = false) {
  const int nr = q.nr, np = q.np;
  const int* rows = d.frontRows + q.rowOff;
  const T* L;
  if (l2Only) {
    const T* Lg = Lbase + q.lOff;
    const int cnt = nr * np;
    if (cnt > capL) {
      L = Lg;
    } else {
      for (int k = lane; k < cnt; k += 32) Ls[k] = __ldcg(Lg + k);
      L = Ls;
    }
  } else {
    L = stageL(Lbase + q.lOff, nr * np, Ls, capL, lane);
  }
  for (int r = lane; r < nr; r += 32) xs[r] = __ldcg(X + __ldg(rows + r));
  copyAsyncWait();
  __syncwarp();
  backwardSolve<T>(d, rows, nr, np, xs, L, X, acc, finalize, lane);
}

// Top-down work queue.  The step-start kernel puts the roots of the active
// models in the first queue slots and sets the slot total to their number of
// chains; a warp takes the next slot, waits until a front is stored there,
// solves it and goes on with its first child, storing the other children in
// fresh slots, until it reaches a leaf; a front whose children are all leaves
// (bwInline) has them solved by the same warp, one after the other, which ends
// the chain.  Every chain ends at a distinct leaf or such front, so the slots
// are exactly the chains of the active models: a warp whose slot number
// reaches the total is done.  A front is stored only after its parent is
// solved (fence, then the slot write; the taker fences after reading it).  A
// waiting warp holds no front, and every stored slot below the one it waits
// for is held by a running warp that solves without waiting, so each wait
// ends; it is still bounded and sets errFlag when it runs out.
// ctr: [0] next slot to take, [1] next free slot, [2] slot total.
// rootDone: the fused factorisation's counters (a root may still be in
// elimination in the same launch), or null when the roots are complete
template <typename T>
__device__ void backwardQueueLoop(const DevData& d, int maxRow, int capL, const T* Lbase, T* X, int* queue, int* ctr,
                                  const unsigned char* bwInline, int* errFlag, int acc, int finalize,
                                  long long spinLimit, T* xs, T* Ls, int lane, const int* rootDone) {
  const int total = *(volatile const int*)(ctr + 2);
  for (;;) {
    const int slot = __shfl_sync(0xffffffffu, lane == 0 ? atomicAdd(ctr, 1) : 0, 0);
    if (slot >= total) break;
    int f = -1, ok = 1;
    if (lane == 0) {
      long long spins = 0;
      while ((f = *(volatile const int*)(queue + slot)) < 0) {
        __nanosleep(32);
        if (++spins > spinLimit) {
          atomicOr(errFlag, 1);
          ok = 0;
          break;
        }
      }
      __threadfence();
      // a root of an active model: wait until its elimination is released
      if (ok && rootDone && d.fParent[f] < 0 && (d.m.flags[d.fModel[f]] & FL_ACTIVE)) {
        while (acquireCount(rootDone + f) < kRootDone) {
          __nanosleep(32);
          if (++spins > spinLimit) {
            atomicOr(errFlag, 1);
            ok = 0;
            break;
          }
        }
      }
    }
    f = __shfl_sync(0xffffffffu, f, 0);
    ok = __shfl_sync(0xffffffffu, ok, 0);
    __syncwarp();
    if (!ok) break;
    BackDesc q = backDesc(d, bwInline, f);
    while (f >= 0) {
      // the first child and its descriptors are loaded ahead of this front's solve
      const int* ch = d.childList + q.childOff;
      const int c0 = q.nch > 0 ? ch[0] : -1;
      const BackDesc cq = backDesc(d, bwInline, c0 >= 0 ? c0 : f);
      backwardOneFront<T>(d, q, xs, Ls, capL, Lbase, X, acc, finalize != 0, lane, rootDone != nullptr);
      __threadfence();
      __syncwarp();
      const int nch = q.nch;
      int next = -1;
      if (nch > 0) {
        if (q.inl) {
          // children that are all leaves: solved here, one after the other
          BackDesc lq = cq;
          for (int c = 0; c < nch; ++c) {
            const BackDesc nq = backDesc(d, bwInline, ch[c + 1 < nch ? c + 1 : c]);
            backwardOneFront<T>(d, lq, xs, Ls, capL, Lbase, X, acc, finalize != 0, lane, rootDone != nullptr);
            __syncwarp();
            lq = nq;
          }
        } else {
          next = c0;
          if (lane == 0 && nch > 1) {
            const int base = atomicAdd(ctr + 1, nch - 1);
            for (int k = 1; k < nch; ++k) atomicExch(queue + base + k - 1, ch[k]);
          }
        }
      }
      __syncwarp();
      f = next;
      q = cq;
    }
  }
}

template <typename T>
__global__ void kBackwardQueue(DevData d, int maxRow, int capL, const T* Lbase, T* X, int* queue, int* ctr,
                               const unsigned char* __restrict__ bwInline, int* errFlag, int acc, int finalize,
                               long long spinLimit) {
  pdlEntry();
  extern __shared__ __align__(16) unsigned char smraw[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T* xs = reinterpret_cast<T*>(smraw) + (size_t)w * (maxRow + capL);
  T* Ls = xs + maxRow;
  backwardQueueLoop<T>(d, maxRow, capL, Lbase, X, queue, ctr, bwInline, errFlag, acc, finalize, spinLimit, xs, Ls,
                       lane, nullptr);
}

// ---- trees on thread blocks ----------------------------------------------------
// Batches of few small fronts (a single model, a few models) are bound by the
// latency of their assembly trees: in the cascades every level costs a front's
// loads in four dependent rounds and a release-acquire through L2 (about 9 us a
// level in the factorisation, 4 us in the solves, on a chain of 3,826 beams).
// Here the host cuts the trees into chunks, connected pieces of at most as many
// fronts as a block has warps, and a block takes a chunk with one warp per front:
// every warp loads all that does not depend on its children (descriptors,
// original entries, extend-add map, right-hand side, or the factor block) at
// the chunk's start, then the levels follow one another at block barriers.
// Between chunks the cascades' protocol applies, a chunk in the place of a
// front: the block that completes a parent chunk's count goes on with it;
// the back substitution is handed down through the queue, a block holding one
// chunk at a time and going on with its first child chunk.  The arithmetic of
// every front is that of the cascades (the same device functions), so both give
// the same bits and the choice is the launch's alone.

// loads of a front's forward elimination that do not depend on its children
template <typename T>
struct ForwardIn {
  int row[2], src[2], dst[2];
  double b[2];
};

template <typename T, int PANEL>
__global__ void __launch_bounds__(512, 1) kTree(DevData d, TreePlan tp, int maxRow, const T* asmVal, T* Lbase, T* Ubase,
                                              double tolFact, const double* rhs, T* X, T* Wv, int* cnt,
                                              FusedBackward fb, int up, int mayFactor) {
  pdlEntry();
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ int shNext;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  T* F = reinterpret_cast<T*>(smraw) + (size_t)w * ((size_t)maxRow * maxRow + 3 * maxRow);
  T* lcol = F + (size_t)maxRow * maxRow;
  T* diag0 = lcol + maxRow;
  T* v = diag0 + maxRow;
  if (up) {
    int* const start = cnt + tp.nChunks;
    auto take = [&]() {
      const int i = atomicAdd(start, 1);
      return i < tp.nStart ? tp.start[i] : -1;
    };
    if (tid == 0) shNext = take();
    __syncthreads();
    int c = shNext;
    while (c >= 0) {
      const TreeChunk ch = tp.chunks[c];
      const int fl = d.m.flags[ch.model];
      const bool active = fl & FL_ACTIVE, factor = mayFactor && (fl & FL_TANGENT);
      if (active) {
        const bool mine = w < ch.n;
        const int f = mine ? tp.fronts[ch.off + w] : -1;
        const int level = mine ? tp.level[ch.off + w] : -1;
        SolveDesc q{};
        ForwardIn<T> in;
        constexpr int kSeg = 8;  // extend-add entries per lane loaded ahead
        int sp[kSeg];
        int ns = 0;
        const T* segIn = nullptr;
        const int* segPos = nullptr;
        bool fast = false;
        if (mine) {
          q = solveDesc(d, f);
          const int nr = q.nr, np = q.np;
          fast = nr <= 64 && q.ncg <= 64;
          if (factor) {
            const int64_t ao = d.fAsmOff[f], so = d.fSegOff[f];
            const int na = d.fNasm[f];
            ns = d.fSegLen[f];
            segIn = Ubase + so;
            segPos = d.segPos + so;
#pragma unroll
            for (int u = 0; u < kSeg; ++u) {
              const int k = lane + 32 * u;
              sp[u] = k < ns ? __ldg(segPos + k) : -1;
            }
            for (int k = lane; k < nr * nr; k += 32) F[k] = T(0);
            for (int k0 = 0; k0 < na; k0 += 32 * kFrontBatch) {
              T val[kFrontBatch];
              int pos[kFrontBatch];
#pragma unroll
              for (int u = 0; u < kFrontBatch; ++u) {
                const int k = k0 + 32 * u + lane;
                pos[u] = k < na ? __ldg(d.asmPos + ao + k) : -1;
                val[u] = k < na ? __ldg(asmVal + ao + k) : T(0);
              }
              __syncwarp();
#pragma unroll
              for (int u = 0; u < kFrontBatch; ++u)
                if (pos[u] >= 0) F[pos[u]] = val[u];
            }
            __syncwarp();
            for (int k = lane; k < np; k += 32) diag0[k] = singularBound(F[k + nr * k], (T)tolFact);
          } else {
            const T* Lg = Lbase + q.lOff;
            for (int k = lane; k < nr * np; k += 32) copyAsync(F + k, Lg + k);
          }
          if (fast) {
            const int* rows = d.frontRows + q.rowOff;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int r = lane + 32 * u;
              in.row[u] = r < np ? __ldg(rows + r) : -1;
              in.src[u] = r < q.ncg ? __ldg(d.cgSrc + q.cg0 + r) : -1;
              in.dst[u] = r < q.ncg ? __ldg(d.cgDst + q.cg0 + r) : 0;
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) in.b[u] = in.row[u] >= 0 ? rhs[in.row[u]] : 0.0;
          }
          if (!factor) copyAsyncWait();
          __syncwarp();
        }
        for (int l = 0; l < ch.levels; ++l) {
          if (level == l) {
            const int nr = q.nr, np = q.np;
            T wv[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) wv[u] = fast && in.src[u] >= 0 ? __ldcg(Wv + in.src[u]) : T(0);
            if (factor) {
              // extend-add of the children's update matrices, child by child
              T sv[kSeg];
#pragma unroll
              for (int u = 0; u < kSeg; ++u) sv[u] = sp[u] >= 0 ? __ldcg(segIn + lane + 32 * u) : T(0);
              extendAdd<T, kSeg>(F, sp, sv);
              for (int k0 = 32 * kSeg; k0 < ns; k0 += 32 * kFrontBatch) {
                T val[kFrontBatch];
                int pc[kFrontBatch];
#pragma unroll
                for (int u = 0; u < kFrontBatch; ++u) {
                  const int k = k0 + 32 * u + lane;
                  pc[u] = k < ns ? __ldg(segPos + k) : -1;
                  val[u] = k < ns ? __ldcg(segIn + k) : T(0);
                }
                extendAdd<T, kFrontBatch>(F, pc, val);
              }
              int neg = 0;
              bool sing = false;
              factorBlocked<T, PANEL>(F, lcol, diag0, nr, np, lane, neg, sing, Ubase + d.fUOff[f]);
              if (lane == 0) {
                if (neg) atomicAdd(&d.m.negPiv[ch.model], neg);
                if (sing) atomicOr(&d.m.status[ch.model], SS_SINGULAR);
              }
            }
            if (fast) forwardRun<T>(q, in.row, in.dst, in.src, in.b, wv, v, F, X, lane, Wv + q.wOff);
            else forwardOneFront<T>(d, f, v, F, 0, Lbase, rhs, X, Wv, lane, F);
            if (factor) {
              T* Lout = Lbase + q.lOff;
              for (int k = lane; k < nr * np; k += 32) Lout[k] = F[k];
            }
          }
          __syncthreads();
        }
      }
      __syncthreads();
      if (tid == 0) {
        int nx = -1;
        if (active) {
          if (ch.parent >= 0) {
            int old;
            asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;\n" : "=r"(old) : "l"(cnt + ch.parent) : "memory");
            if (old == ch.parentNeed - 1) nx = ch.parent;
          } else if (fb.queue) {
            asm volatile("red.release.gpu.global.add.s32 [%0], %1;\n" ::"l"(cnt + c), "r"(kRootDone) : "memory");
          }
        }
        shNext = nx >= 0 ? nx : take();
      }
      __syncthreads();
      c = shNext;
    }
  }
  if (!fb.queue) return;
  // back substitution: the queue of kBackwardQueue with chunks in the place of
  // fronts.  With the elimination in the same launch (up), the roots' done marks
  // are waited for, and L, written in this launch, is read through L2.
  const int total = *(volatile const int*)(fb.ctr + 2);
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      int c = -1;
      const int slot = atomicAdd(fb.ctr, 1);
      if (slot < total) {
        long long spins = 0;
        bool ok = true;
        while ((c = *(volatile const int*)(fb.queue + slot)) < 0) {
          __nanosleep(20);
          if (++spins > fb.spinLimit) {
            atomicOr(fb.errFlag, 1);
            ok = false;
            break;
          }
        }
        __threadfence();
        if (ok && up && tp.chunks[c].parent < 0 && (d.m.flags[tp.chunks[c].model] & FL_ACTIVE)) {
          while (acquireCount(cnt + c) < kRootDone) {
            __nanosleep(20);
            if (++spins > fb.spinLimit) {
              atomicOr(fb.errFlag, 1);
              ok = false;
              break;
            }
          }
        }
        if (!ok) c = -1;
      }
      shNext = c;
    }
    __syncthreads();
    int c = shNext;
    if (c < 0) break;
    while (c >= 0) {
      const TreeChunk ch = tp.chunks[c];
      const bool mine = w < ch.n;
      const int f = mine ? tp.fronts[ch.off + w] : -1;
      const int level = mine ? tp.level[ch.off + w] : -1;
      const int* rows = nullptr;
      int nr = 0, np = 0, rr[3];
      if (mine) {
        nr = d.fNrow[f];
        np = d.fNpiv[f];
        rows = d.frontRows + d.fRowOff[f];
        const T* Lg = Lbase + d.fLOff[f];
#pragma unroll
        for (int u = 0; u < 3; ++u) rr[u] = lane + 32 * u < nr ? __ldg(rows + lane + 32 * u) : -1;
        if (up && mayFactor) {
          for (int k = lane; k < nr * np; k += 32) F[k] = __ldcg(Lg + k);
        } else {
          for (int k = lane; k < nr * np; k += 32) copyAsync(F + k, Lg + k);
          copyAsyncWait();
        }
        __syncwarp();
      }
      for (int l = ch.levels - 1; l >= 0; --l) {
        if (level == l) {
#pragma unroll
          for (int u = 0; u < 3; ++u)
            if (rr[u] >= 0) v[lane + 32 * u] = __ldcg(X + rr[u]);
          for (int r = lane + 96; r < nr; r += 32) v[r] = __ldcg(X + __ldg(rows + r));
          __syncwarp();
          backwardSolve<T>(d, rows, nr, np, v, F, X, fb.acc, fb.finalize != 0, lane);
        }
        __syncthreads();
      }
      if (tid == 0) {
        int nx = -1;
        if (ch.nKids > 0) {
          nx = tp.kids[ch.kidOff];
          if (ch.nKids > 1) {
            __threadfence();
            const int base = atomicAdd(fb.ctr + 1, ch.nKids - 1);
            for (int k = 1; k < ch.nKids; ++k) atomicExch(fb.queue + base + k - 1, tp.kids[ch.kidOff + k]);
          }
        }
        shNext = nx;
      }
      __syncthreads();
      c = shNext;
      __syncthreads();
    }
  }
}

int smCountCached() {
  // engines may be built on several host threads at once
  static std::atomic<int> cached{0};
  int n = cached.load(std::memory_order_relaxed);
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 1;
    cached.store(n, std::memory_order_relaxed);
  }
  return n;
}

template <typename K>
int occupancyBlocks(K kernel, int threads, size_t smem, int needed) {
  int perSm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kernel, threads, smem) != cudaSuccess || perSm < 1)
    perSm = 1;
  int cap = perSm * smCountCached();
  return needed < cap ? (needed > 0 ? needed : 1) : cap;
}

// one launch of a factor cascade kernel (either panel variant)
template <typename T>
void factorCascade(void (*kernel)(DevData, const int*, int, int, const T*, T*, T*, double, const double*, T*, T*,
                                  int*, FusedBackward),
                   int wpb, size_t sm, const DevData& d, const PersistentPlan& p, const T* asmVal, T* L, T* U,
                   double tol, const double* rhs, T* X, T* W, const FusedBackward& fb, cudaStream_t s) {
  if (sm > 48 * 1024) allowBigShared(kernel);
  const int blocks = occupancyBlocks(kernel, 32 * wpb, sm, (p.nLeaves + wpb - 1) / wpb);
  pdlLaunch(kernel, blocks, 32 * wpb, sm, s, d, p.leaves, p.nLeaves, p.maxRow, asmVal, L, U, tol, rhs, X, W, p.cntFactor,
            fb);
}

// subtrees' lowest fronts from which a larger batch's upper levels go to the trees
constexpr long long kTreeTops = 1500;

size_t treeWarpValues(int maxRow) { return (size_t)maxRow * maxRow + 3 * (size_t)maxRow; }

// one launch of the trees on thread blocks (kTree)
template <typename T>
void treeLaunch(const DevData& d, const PersistentPlan& p, const T* asmVal, T* L, T* U, const double* rhs, T* X, T* W,
                int* cnt, const FusedBackward& fb, bool up, bool mayFactor, cudaStream_t s) {
  const auto kernel = !mayFactor || p.factorPanel == kPanelShuffle ? kTree<T, kPanelShuffle>
                      : p.factorPanel == kPanelRegisters           ? kTree<T, kPanelRegisters>
                                                                   : kTree<T, kPanelRegisters4>;
  const int threads = 32 * p.tree.warps;
  const size_t sm = p.tree.warps * treeWarpValues(p.maxRow) * sizeof(T);
  if (sm > 48 * 1024) allowBigShared(kernel);
  const int blocks = occupancyBlocks(kernel, threads, sm, p.tree.nStart);
  pdlLaunch(kernel, blocks, threads, sm, s, d, p.tree, p.maxRow, asmVal, L, U, 1.0e-12, rhs, X, W, cnt, fb, up ? 1 : 0,
            mayFactor ? 1 : 0);
}

void treeLaunch(const DevData& d, const PersistentPlan& p, bool fp32, const double* rhs, int* cnt,
                const FusedBackward& fb, bool up, bool mayFactor, cudaStream_t s) {
  if (fp32)
    treeLaunch<float>(d, p, d.asmVal32, d.L32, d.U32, rhs, d.x32, d.w32, cnt, fb, up, mayFactor, s);
  else
    treeLaunch<double>(d, p, d.asmVal64, d.L64, d.U64, rhs, d.x64, d.w64, cnt, fb, up, mayFactor, s);
}

// the back substitution of solve `sweep` (launchBackward's arguments), the
// cascades' or the trees'
FusedBackward backwardOf(const PersistentPlan& p, bool fp32, int sweep, bool last, bool tree) {
  FusedBackward fb;
  fb.queue = tree ? p.treeQueue + (size_t)sweep * p.tree.nStart : p.bwQueue + (size_t)sweep * p.nLeaves;
  fb.ctr = (tree ? p.treeCtr : p.bwCtr) + 4 * sweep;
  fb.bwInline = p.bwInline;
  fb.errFlag = p.errFlag;
  fb.spinLimit = p.spinLimit;
  fb.acc = !fp32 ? ACC_SET : (sweep == 0 ? ACC_FIRST : ACC_ADD);
  fb.finalize = (fp32 && last) ? 1 : 0;
  return fb;
}

int factorWarpsPerBlock(size_t perWarpBytes) {
  int w = (int)(96 * 1024 / (perWarpBytes > 0 ? perWarpBytes : 1));
  return w > 8 ? 8 : (w < 1 ? 1 : w);
}

// Synthetic original entries for the autotuner's timing probe: a dominant
// diagonal and small off-diagonal values of alternating sign (pivots stay
// positive and far from singular, like a Newton matrix's), one thread per front.
template <typename T>
__global__ void kProbeEntries(DevData d, T* asmVal) {
  pdlEntry();
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= d.nfrontTot) return;
  const int nr = d.fNrow[f], na = d.fNasm[f];
  const int64_t ao = d.fAsmOff[f];
  for (int k = 0; k < na; ++k) {
    const int pos = d.asmPos[ao + k];
    const int i = pos % nr, j = pos / nr;
    asmVal[ao + k] = i == j ? T(4 + nr) : (((i + j) & 1) ? T(0.01) : T(-0.01));
  }
}

// the cascades' factorisation with the first forward elimination (and the back
// substitution fb, if any)
void factorForwardCascade(const DevData& d, const PersistentPlan& p, bool fp32, const double* rhs,
                          const FusedBackward& fb, cudaStream_t s) {
  const double tol = 1.0e-12;
  const size_t perWarp = (size_t)p.maxRow * p.maxRow + 3 * p.maxRow;
  if (fp32) {
    const int wpb = factorWarpsPerBlock(perWarp * sizeof(float));
    const size_t sm = (size_t)wpb * perWarp * sizeof(float);
    if (p.factorPanel == kPanelRegisters)
      factorCascade(kFactorForwardCascade<float, kPanelRegisters>, wpb, sm, d, p, d.asmVal32, d.L32, d.U32, tol, rhs,
                    d.x32, d.w32, fb, s);
    else if (p.factorPanel == kPanelRegisters4)
      factorCascade(kFactorForwardCascade<float, kPanelRegisters4>, wpb, sm, d, p, d.asmVal32, d.L32, d.U32, tol,
                    rhs, d.x32, d.w32, fb, s);
    else
      factorCascade(kFactorForwardCascade<float, kPanelShuffle>, wpb, sm, d, p, d.asmVal32, d.L32, d.U32, tol, rhs,
                    d.x32, d.w32, fb, s);
  } else {
    const int wpb = factorWarpsPerBlock(perWarp * sizeof(double));
    const size_t sm = (size_t)wpb * perWarp * sizeof(double);
    if (p.factorPanel == kPanelRegisters)
      factorCascade(kFactorForwardCascade<double, kPanelRegisters>, wpb, sm, d, p, d.asmVal64, d.L64, d.U64, tol,
                    rhs, d.x64, d.w64, fb, s);
    else if (p.factorPanel == kPanelRegisters4)
      factorCascade(kFactorForwardCascade<double, kPanelRegisters4>, wpb, sm, d, p, d.asmVal64, d.L64, d.U64, tol,
                    rhs, d.x64, d.w64, fb, s);
    else
      factorCascade(kFactorForwardCascade<double, kPanelShuffle>, wpb, sm, d, p, d.asmVal64, d.L64, d.U64, tol, rhs,
                    d.x64, d.w64, fb, s);
  }
}


// the cascades' forward elimination of a refinement solve
void forwardCascade(const DevData& d, const PersistentPlan& p, bool fp32, const double* rhs, int sweep,
                    cudaStream_t s) {
  const int wpb = p.forwardWarps;
  int* cnt = p.cntForward + (size_t)(sweep - 1) * ((size_t)d.nfrontTot + 1);
  if (fp32) {
    const int capL = stagingCapacity(p, sizeof(float));
    const size_t sm = (size_t)wpb * (p.maxRow + capL + 64) * sizeof(float);
    if (sm > 48 * 1024) allowBigShared(kForwardCascade<float>);
    const int blocks = occupancyBlocks(kForwardCascade<float>, 32 * wpb, sm, (p.nTasks + wpb - 1) / wpb);
    pdlLaunch(kForwardCascade<float>, blocks, 32 * wpb, sm, s, d, p.tasks, p.nTasks, p.maxRow, capL, d.L32, rhs, d.x32,
                                                       d.w32, cnt);
  } else {
    const int capL = stagingCapacity(p, sizeof(double));
    const size_t sm = (size_t)wpb * (p.maxRow + capL + 64) * sizeof(double);
    if (sm > 48 * 1024) allowBigShared(kForwardCascade<double>);
    const int blocks = occupancyBlocks(kForwardCascade<double>, 32 * wpb, sm, (p.nTasks + wpb - 1) / wpb);
    pdlLaunch(kForwardCascade<double>, blocks, 32 * wpb, sm, s, d, p.tasks, p.nTasks, p.maxRow, capL, d.L64, rhs, d.x64,
                                                         d.w64, cnt);
  }
}

}  // namespace

void launchProbeEntries(const DevData& d, bool fp32, cudaStream_t s) {
  if (d.nfrontTot <= 0) return;
  const int blocks = (d.nfrontTot + 127) / 128;
  if (fp32) pdlLaunch(kProbeEntries<float>, blocks, 128, 0, s, d, d.asmVal32);
  else pdlLaunch(kProbeEntries<double>, blocks, 128, 0, s, d, d.asmVal64);
}

void launchFactorForwardCascade(const DevData& d, const PersistentPlan& p, bool fp32, const double* rhs,
                                cudaStream_t s, bool withBackward, bool lastSweep) {
  // the cascades below the trees first; the back substitution of the trees is part
  // of their launch, the cascades' follows on its own
  if (p.tree.warps > 0) {
    if (p.nLeaves > 0) factorForwardCascade(d, p, fp32, rhs, FusedBackward{}, s);
    treeLaunch(d, p, fp32, rhs, p.cntTree, withBackward ? backwardOf(p, fp32, 0, lastSweep, true) : FusedBackward{},
               true, true, s);
    return;
  }
  if (p.nLeaves <= 0) return;
  FusedBackward fb;
  if (withBackward) {
    // (its solve vector and L staging reuse the warp's v and F areas)
    fb = backwardOf(p, fp32, 0, lastSweep, false);
    fb.capL = stagingCapacity(p, fp32 ? sizeof(float) : sizeof(double));
  }
  factorForwardCascade(d, p, fp32, rhs, fb, s);
}

// staging capacity (values) of one front's L block per warp
int stagingCapacity(const PersistentPlan& p, size_t elemBytes) {
  long long want = (long long)p.maxRow * p.maxNpiv;
  long long cap = (long long)(12 * 1024 / elemBytes);
  return (int)(want < cap ? want : cap);
}

// The line between the trees on thread blocks and the cascades (iteration in
// microseconds on batches of chains, written models x beams; FP64, mixed in brackets).
// A block takes one chunk at a time whatever its fronts, so many chunks of few fronts
// each leave most of its warps idle: 4,000 x 1 (one front a chunk) 420 (569) on trees
// against 184 (210) on cascades, 1,000 x 8 209 (244) / 136 (153), 300 x 12 127 (144) /
// 112 (128), 128 frames of 3 x 2 with 736 chunks 557 (582) / 526 (469).  Few chunks, or
// well filled ones, spare the cascades' latency per tree level: 1 x 20 72 (84) / 84
// (102), 64 chains of 8 reduced parts with 192 chunks 219 (275) / 264 (267), 150 x 20
// with 246 chunks of 8 fronts 122 (133) / 122 (140), 64 x 150 with 556 of 11 183 (197) /
// 228 (232).
//   With more than 4,096 leaf fronts two blocks of 8 warps share an SM better than one
// of 16, as long as the chunks are few enough: 300 x 40 with 1,572 chunks 196 (210) /
// 219 (224); 1,000 x 12 with 1,832 187 (211) / 187 (197); 128 x 150 with 2,057 253
// (273) / 251 (276).
//   Otherwise the cascades take the fronts up to the height above which at most
// kTreeTops subtrees begin, and the trees the levels from there, where the cascades run
// out of fronts: 5 x 4,000 336 (339) / 404 (422), 30 x 600 with 259 chunks 318 (311) /
// 353 (349), 100 x 300 with 248 375 (364) / 366 (392), but 250 x 100 with 413 265 (284) /
// 245 (275).  (1,500 subtrees: with 300, 600 or 3,000 up to 9 % slower.)  Above 32,768
// leaf fronts other models' fronts fill the cascades' upper levels (64,000: 675 / 689,
// FP64 727 / 749).
int treeTopHeight(int maxHeight, const std::function<long long(int)>& lowest) {
  for (int h = 1; h + 2 <= maxHeight; ++h)
    if (lowest(h) <= kTreeTops) return h;
  return -1;
}

bool treesPay(int nChunks, long long nFronts, int warps, int fromHeight) {
  if (fromHeight > 0) return nChunks <= 300;
  if (warps > 8) return nChunks <= 200 || 2 * nFronts >= (long long)warps * nChunks;
  return nChunks <= 1800;
}

int treeWarps(int nLeaves, int maxRow, bool fp32) {
  const int fit = (int)(200 * 1024 / (treeWarpValues(maxRow) * (fp32 ? sizeof(float) : sizeof(double))));
  const int w = std::min(nLeaves <= 4096 ? 16 : 8, fit);
  return w >= 3 ? w : 0;
}

bool fusableBackward(const PersistentPlan& p, bool fp32) {
  if (p.tree.warps > 0) return p.nLarge == 0;
  return p.nLeaves > 0 && p.nLarge == 0 &&
         (long long)stagingCapacity(p, fp32 ? sizeof(float) : sizeof(double)) >= (long long)p.maxRow * p.maxNpiv;
}

void launchForwardCascade(const DevData& d, const PersistentPlan& p, bool fp32, const double* rhs, int sweep,
                          cudaStream_t s, bool withBackward, bool lastSweep) {
  if (p.nTasks > 0) forwardCascade(d, p, fp32, rhs, sweep, s);
  if (p.tree.warps > 0)
    treeLaunch(d, p, fp32, rhs, p.cntTree + (size_t)sweep * (p.tree.nChunks + 1),
               withBackward ? backwardOf(p, fp32, sweep, lastSweep, true) : FusedBackward{}, true, false, s);
}

void launchBackward(const DevData& d, const PersistentPlan& p, bool fp32, int sweep, bool last, cudaStream_t s,
                    bool treeDone) {
  const int acc = !fp32 ? ACC_SET : (sweep == 0 ? ACC_FIRST : ACC_ADD);
  const int fin = (fp32 && last) ? 1 : 0;
  if (p.tree.warps > 0 && !treeDone)
    treeLaunch(d, p, fp32, nullptr, p.cntTree, backwardOf(p, fp32, sweep, last, true), false, false, s);
  if (p.nLeaves <= 0) return;
  const int wpb = p.backwardWarps;
  int* queue = p.bwQueue + (size_t)sweep * p.nLeaves;
  int* ctr = p.bwCtr + 4 * sweep;
  const int needed = (p.nLeaves + wpb - 1) / wpb;
  if (fp32) {
    const int capL = stagingCapacity(p, sizeof(float));
    const size_t sm = (size_t)wpb * (p.maxRow + capL) * sizeof(float);
    if (sm > 48 * 1024) allowBigShared(kBackwardQueue<float>);
    const int blocks = occupancyBlocks(kBackwardQueue<float>, 32 * wpb, sm, needed);
    pdlLaunch(kBackwardQueue<float>, blocks, 32 * wpb, sm, s, d, p.maxRow, capL, d.L32, d.x32, queue, ctr, p.bwInline,
                                                      p.errFlag, acc, fin, p.spinLimit);
  } else {
    const int capL = stagingCapacity(p, sizeof(double));
    const size_t sm = (size_t)wpb * (p.maxRow + capL) * sizeof(double);
    if (sm > 48 * 1024) allowBigShared(kBackwardQueue<double>);
    const int blocks = occupancyBlocks(kBackwardQueue<double>, 32 * wpb, sm, needed);
    pdlLaunch(kBackwardQueue<double>, blocks, 32 * wpb, sm, s, d, p.maxRow, capL, d.L64, d.x64, queue, ctr, p.bwInline,
                                                        p.errFlag, acc, fin, p.spinLimit);
  }
}

void launchBackwardWaitProbe(const DevData& d, const PersistentPlan& p, int* queue, int* ctr, long long spins,
                             cudaStream_t s) {
  // one warp; it waits on slot 0 and touches no front (the wait gives up first)
  const int capL = stagingCapacity(p, sizeof(double));
  const size_t sm = (size_t)(p.maxRow + capL) * sizeof(double);
  if (sm > 48 * 1024) allowBigShared(kBackwardQueue<double>);
  pdlLaunch(kBackwardQueue<double>, 1, 32, sm, s, d, p.maxRow, capL, d.L64, d.x64, queue, ctr, p.bwInline, p.errFlag,
                                           ACC_SET, 0, spins);
}

void launchRootWaitProbe(const DevData& d, const PersistentPlan& p, int* queue, int* ctr, int* cnt, long long spins,
                         cudaStream_t s) {
  // one warp of the fused factorisation with no leaf: it goes straight to the
  // back substitution, takes slot 0 (a root) and waits for a release that no
  // elimination makes (cnt is zero); the wait gives up before any front is touched
  const size_t perWarp = (size_t)p.maxRow * p.maxRow + 3 * p.maxRow;
  const size_t sm = perWarp * sizeof(double);
  FusedBackward fb;
  fb.queue = queue;
  fb.ctr = ctr;
  fb.bwInline = p.bwInline;
  fb.errFlag = p.errFlag;
  fb.spinLimit = spins;
  fb.acc = ACC_SET;
  fb.capL = stagingCapacity(p, sizeof(double));
  if (sm > 48 * 1024) allowBigShared(kFactorForwardCascade<double, kPanelShuffle>);
  pdlLaunch(kFactorForwardCascade<double, kPanelShuffle>, 1, 32, sm, s, d, p.leaves, 0, p.maxRow,
            (const double*)d.asmVal64, d.L64, d.U64, 1.0e-12, (const double*)d.del, d.x64, d.w64, cnt, fb);
}

void launchTreeWaitProbe(const DevData& d, const PersistentPlan& p, bool fp32, int* queue, int* ctr, int* cnt,
                         bool root, long long spins, cudaStream_t s) {
  // one block of the trees without a chunk to eliminate takes queue slot 0: it is empty,
  // or holds a root whose elimination nothing releases (cnt is zero); the wait gives up
  // before any front is touched
  PersistentPlan one = p;
  one.tree.nStart = 0;
  FusedBackward fb = backwardOf(p, fp32, 0, true, true);
  fb.queue = queue;
  fb.ctr = ctr;
  fb.spinLimit = spins;
  treeLaunch(d, one, fp32, d.del, cnt, fb, root, false, s);
}

}  // namespace fgpu

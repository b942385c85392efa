// front_large.cu -- multifrontal factorisation and solves of the large fronts
// (more rows than one warp's shared-memory front holds).
//
// Large fronts are marked upward-closed on the host (every ancestor of a large
// front is large), so the warp kernels of front_cascade.cu finish every small
// subtree first and these kernels take the tops of the assembly trees.  Each
// of the three passes (factorisation, forward elimination, back substitution)
// is one cooperative launch of at most one block per SM.  The host lays the
// fronts out in waves (fronts of one tree level, their blocks shared out by
// work); a block walks its column of that table, so it always knows its next
// front, its rank and the number of blocks working on it (LargeTask).  A front
// starts when its large children (its parent, in the back substitution) have
// signalled, and its blocks meet at barriers of their own; all blocks are
// resident (cooperative launch), each wait is bounded and sets errFlag when it
// runs out, after which every block runs to its end without waiting.
//
// Why whole-GPU fronts: a GB300 SM sub-core issues one FP64 instruction per 64
// cycles whatever its active lanes, so one front's update on one cluster sets
// the pace (space-frame tower, 15 fronts deep, FP64: 4.3 ms on clusters of 16
// blocks that factored each panel redundantly; the split here is by entry, so
// every sub-core of the GPU takes an equal share of a panel's update).
//
// A large front is factored in place in its outputs: its pivot columns in its
// L block (nrow x npiv, column-major) and its trailing lower triangle in its
// packed update matrix (column by column, inside the parent's segment), so no
// workspace is needed.  Blocked right-looking LDL^T in panels of 32 pivots:
//   every block factors the panel's diagonal block itself (the same arithmetic,
//     so the same values; cheaper than a broadcast);
//   the rows below it are shared out, one warp per row, one lane per column;
//   after a barrier the trailing triangle is updated, C -= L_p D_p L_p^T, in
//     16 x 16 blocks, a warp each (FP32 fronts: mma.sync TF32 products on the
//     tensor cores in the 3xTF32 split) or a warp per half (FP64 fronts).
// Every entry's arithmetic is the same whichever block or warp does it, so the
// result does not depend on the number of blocks.  Semantics as the warp
// kernels and the reference's SPRFC1/SPRFS1/SPRBS1 seam
// (solExtensionModule.f90:153-505): no pivoting, a pivot is singular when
// |d_k| <= tolFactorize |a_kk|, negative pivots counted, children's update
// matrices added in child order (fixed summation order).
// Front data written in the same launch are read through L2 (__ldcg).

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "kernels.h"
#include "pivot.cuh"

namespace fgpu {
namespace {

constexpr int kLT = 256;  // threads per block
constexpr int kLW = kLT / 32;
constexpr int kPanel = 32;  // pivots per panel

// lower-triangle entry (ii >= jj) of an nu x nu matrix packed column by column
__device__ inline int64_t packedAt(int ii, int jj, int nu) {
  return (int64_t)jj * nu - (int64_t)jj * (jj - 1) / 2 + (ii - jj);
}

template <typename T>
struct Front {
  T* L;  // nr x np, column-major
  T* U;  // packed lower triangle of the trailing nu x nu block
  int nr, np, nu;
  __device__ T* at(int i, int j) const {  // i >= j
    return j < np ? L + i + (int64_t)nr * j : U + packedAt(i - np, j - np, nu);
  }
};

template <typename T>
__device__ inline T ld(const T* p) {
  return __ldcg(p);
}
template <typename T>
__device__ inline void st(T* p, T v) {
  __stcg(p, v);
}

// ---- waits ------------------------------------------------------------------
// Waits until *c >= target, bounded; every thread of the block calls it and
// afterwards sees what the signalling blocks wrote (through L2).  Once a wait
// has run out (here or in another block) it returns at once: `dead` stays set.
struct WaitState {
  int* err;
  long long limit;
  bool dead;
};
__device__ inline int acquireCount(const int* c) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];\n" : "=r"(v) : "l"(c) : "memory");
  return v;
}
__device__ inline void signalCount(int* c) {
  asm volatile("red.release.gpu.global.add.s32 [%0], 1;\n" ::"l"(c) : "memory");
}
__device__ inline void waitCount(const int* c, int target, WaitState& ws) {
  bool out = false;
  if (threadIdx.x == 0 && !ws.dead) {
    long long spins = 0;
    while (acquireCount(c) < target) {
      ++spins;
      if (spins > 256) __nanosleep(32);
      if (spins > ws.limit || ((spins & 1023) == 0 && *(volatile const int*)ws.err)) {
        atomicOr(ws.err, 1);
        out = true;
        break;
      }
    }
  }
  if (__syncthreads_or(out)) ws.dead = true;
}
// barrier of the G blocks of one front (phase: 1, 2, ... per front)
__device__ inline void groupBarrier(int* bar, int G, int phase, WaitState& ws) {
  if (G == 1) {
    __syncthreads();
    return;
  }
  __syncthreads();
  if (threadIdx.x == 0) signalCount(bar);
  waitCount(bar, G * phase, ws);
}

// ---- FP32 trailing blocks on the tensor cores ---------------------------------
// mma.sync m16n8k8 TF32 products with FP32 accumulation in the 3xTF32 split
// (x = hi + lo, both TF32; a b = hi hi + hi lo + lo hi), which keeps the FP32
// accuracy of the update.  Fragment layouts of m16n8k8.row.col: lane = 4 g + t
// holds A(g, t), A(g + 8, t), A(g, t + 4), A(g + 8, t + 4); B(t, g), B(t + 4, g);
// C(g, 2t), C(g, 2t + 1), C(g + 8, 2t), C(g + 8, 2t + 1).
__device__ inline uint32_t tf32Of(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}

__device__ inline void split3(float x, uint32_t& hi, uint32_t& lo) {
  hi = tf32Of(x);
  lo = tf32Of(x - __uint_as_float(hi));
}

__device__ inline void mmaTf32(float* c, const uint32_t* a, const uint32_t* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// shared memory of the factorisation: the panel's factored diagonal block
// (Lt[k][i] = l_ik), its pivots, their reciprocals and singularity thresholds
// (two panels'), the elimination's column buffers, and per warp the staged
// operand rows of one trailing block (k-major: 16 rows, and 16 or 8 columns)
template <typename T>
struct FactorShared {
  T Lt[kPanel][kPanel];
  T d[kPanel], dinv[kPanel], diag0[2][kPanel];
  T ubuf[2][kPanel], uk[2][kPanel];
  T A[kLW][kPanel][16 + (sizeof(T) == 4 ? 4 : 0)];
  T B[kLW][kPanel][std::is_same<T, float>::value ? 20 : 8];
};

// Partial LDL^T of the kb x kb diagonal block (lower triangle in s.Lt[col][row],
// unscaled; diag0: the singularity thresholds) by warps 0 to 3, one row per
// lane, in steps with one barrier each.  In step k warp 0 applies the update of
// pivot k - 1 to column k, takes its pivot and scales it; warps 1 to 3, which own
// the later columns c = 3 q + w - 1, meanwhile apply pivot k - 1 to them, column
// k + 1 first, which they pass on.  The chain of a pivot (a multiply-subtract, a
// reciprocal, a product) so has a sub-core's FP64 pipe to itself: with the
// columns on all four warps and every warp computing the reciprocal a block took
// 26,300 cycles in FP64.
template <typename T>
__device__ void factorDiagonal(FactorShared<T>& s, const T* diag0, int kb, int& neg, bool& sing) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (w == 0) {
    T u = lane < kb ? s.Lt[0][lane] : T(0), l = T(0);
    for (int k = 0; k < kb; ++k) {
      if (k > 0) {
        const T uk = __shfl_sync(0xffffffffu, u, k);  // pivot k - 1's unscaled value of row k
        asm volatile("bar.sync 1, 128;" ::: "memory");
        u = s.ubuf[k & 1][lane] - l * uk;
      }
      const T dk = __shfl_sync(0xffffffffu, u, k);
      const bool bad = !absGreater(dk, diag0[k]);
      const T inv = bad ? T(0) : T(1) / dk;
      if (negative(dk)) ++neg;
      sing |= bad;
      l = u * inv;
      // for the others' step k + 1 (and the panel): l below the diagonal, u
      s.Lt[k][lane] = lane > k ? l : T(0);
      s.uk[k & 1][lane] = u;
      if (lane == 0) {
        s.d[k] = dk;
        s.dinv[k] = inv;
      }
    }
  } else if (w < 4) {
    // columns c = 3 q + w - 1 (c >= 1); a[q] holds the row's value of column c
    T a[11];
#pragma unroll
    for (int q = 0; q < 11; ++q) {
      const int c = 3 * q + w - 1;
      a[q] = (c > 0 && c < kb && lane < kb && lane >= c) ? s.Lt[c][lane] : T(0);
      if (c == 1) s.ubuf[1][lane] = a[q];
    }
#pragma unroll
    for (int k = 1; k < kPanel; ++k) {  // step k: pivot k - 1 applied to columns above k
      if (k >= kb) break;
      asm volatile("bar.sync 1, 128;" ::: "memory");
      const T l = s.Lt[k - 1][lane];
      const T* u = s.uk[(k - 1) & 1];
#pragma unroll
      for (int q = 0; q < 11; ++q) {
        const int c = 3 * q + w - 1;
        if (3 * q + 2 > k && c > k && c < kb) {
          a[q] -= l * u[c];
          if (c == k + 1) s.ubuf[(k + 1) & 1][lane] = a[q];
        }
      }
    }
  }
  __syncthreads();
}

// one warp's 16 x 8 half of the trailing block (rows r0.., columns c0..; front
// indices), FP64: lane = 8 lc + lr has rows lr, lr + 8 and columns lc, lc + 4
__device__ inline void trailingBlock(const Front<double>& F, FactorShared<double>& s, int k0, int kb, int r0, int c0) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nr = F.nr;
  double va[16], vb[8];
#pragma unroll
  for (int t = 0; t < 16; ++t) {
    const int r = r0 + (lane & 15), k = 2 * t + (lane >> 4);
    va[t] = (r < nr && k < kb) ? ld(F.L + r + (int64_t)nr * (k0 + k)) : 0.0;
  }
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const int c = c0 + (lane & 7), k = 4 * t + (lane >> 3);
    vb[t] = (c < nr && k < kb) ? ld(F.L + c + (int64_t)nr * (k0 + k)) : 0.0;
  }
  const int lr = lane & 7, lc = lane >> 3;
  double* dst[2][2];
  double cur[2][2];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const int r = r0 + lr + 8 * a, c = c0 + lc + 4 * b;
      dst[a][b] = (r < nr && r >= c) ? F.at(r, c) : nullptr;
      cur[a][b] = dst[a][b] ? ld(dst[a][b]) : 0.0;
    }
  __syncwarp();
#pragma unroll
  for (int t = 0; t < 16; ++t) s.A[w][2 * t + (lane >> 4)][lane & 15] = va[t];
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const int k = 4 * t + (lane >> 3);
    s.B[w][k][lane & 7] = k < kb ? vb[t] * s.d[k] : 0.0;
  }
  __syncwarp();
  double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll 8
  for (int k = 0; k < kb; ++k) {
    const double a0 = s.A[w][k][lr], a1 = s.A[w][k][lr + 8], b0 = s.B[w][k][lc], b1 = s.B[w][k][lc + 4];
    acc[0][0] += a0 * b0;
    acc[0][1] += a0 * b1;
    acc[1][0] += a1 * b0;
    acc[1][1] += a1 * b1;
  }
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b)
      if (dst[a][b]) st(dst[a][b], cur[a][b] - acc[a][b]);
}

// one warp's 16 x 16 trailing block, FP32 on the tensor cores
__device__ inline void trailingBlock(const Front<float>& F, FactorShared<float>& s, int k0, int kb, int r0, int c0) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nr = F.nr;
  float va[16], vb[16];
#pragma unroll
  for (int t = 0; t < 16; ++t) {
    const int r = r0 + (lane & 15), c = c0 + (lane & 15), k = 2 * t + (lane >> 4);
    va[t] = (r < nr && k < kb) ? ld(F.L + r + (int64_t)nr * (k0 + k)) : 0.0f;
    vb[t] = (c < nr && k < kb) ? ld(F.L + c + (int64_t)nr * (k0 + k)) : 0.0f;
  }
  const int g = lane >> 2, t4 = lane & 3;
  float* dst[2][4];
  float cur[2][4];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = r0 + g + 8 * (q >> 1), c = c0 + 8 * j + 2 * t4 + (q & 1);
      dst[j][q] = (r < nr && c < nr && r >= c) ? F.at(r, c) : nullptr;
      cur[j][q] = dst[j][q] ? ld(dst[j][q]) : 0.0f;
    }
  __syncwarp();
#pragma unroll
  for (int t = 0; t < 16; ++t) {
    const int k = 2 * t + (lane >> 4);
    s.A[w][k][lane & 15] = va[t];
    s.B[w][k][lane & 15] = k < kb ? vb[t] * s.d[k] : 0.0f;
  }
  __syncwarp();
  float acc[2][4];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[j][q] = 0.0f;
#pragma unroll
  for (int kk = 0; kk < kPanel; kk += 8) {
    if (kk >= kb) break;
    uint32_t ah[4], al[4];
    split3(s.A[w][kk + t4][g], ah[0], al[0]);
    split3(s.A[w][kk + t4][g + 8], ah[1], al[1]);
    split3(s.A[w][kk + t4 + 4][g], ah[2], al[2]);
    split3(s.A[w][kk + t4 + 4][g + 8], ah[3], al[3]);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      uint32_t bh[2], bl[2];
      split3(s.B[w][kk + t4][8 * j + g], bh[0], bl[0]);
      split3(s.B[w][kk + t4 + 4][8 * j + g], bh[1], bl[1]);
      mmaTf32(acc[j], al, bh);
      mmaTf32(acc[j], ah, bl);
      mmaTf32(acc[j], ah, bh);
    }
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (dst[j][q]) st(dst[j][q], cur[j][q] - acc[j][q]);
}

// Assembly of front f: entry (i, j) = the children's contributions in child
// order, then the original entry.  Pulled by target through the children's
// inverse row maps, so nothing waits between children: a warp takes 128 rows
// of one column at a time.
template <typename T>
__device__ void assembleLarge(const DevData& d, const LargePlan& lp, const LargeTask& t, const Front<T>& F,
                              const T* asmVal, const T* Ubase) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nr = F.nr, np = F.np, f = t.f;
  const int nch = d.fNchild[f];
  const int* chl = d.childList + d.fChildOff[f];
  const int* inv = lp.inv + lp.invOff[t.li];
  const int64_t ao = d.fAsmOff[f];
  const int* colPtr = lp.asmCol + lp.asmColOff[t.li];
  const int nrb = (nr + 127) >> 7;
  for (int u = t.rank + t.G * w; u < nr * nrb; u += t.G * kLW) {
    const int j = u / nrb, i0 = (u - j * nrb) << 7;
    if (i0 + 127 < j) continue;
    const int k0 = j < np ? __ldg(colPtr + j) : 0, k1 = j < np ? __ldg(colPtr + j + 1) : 0;
    T v[4] = {T(0), T(0), T(0), T(0)};
    for (int c0 = 0; c0 < nch; c0 += 32) {
      // lane c: child c0 + c's update row at row j and the start of its column,
      // shifted so that [row] addresses it; then the children that have row j, in order
      int b = -1;
      long long off = 0;
      if (c0 + lane < nch) {
        b = __ldg(inv + (int64_t)(c0 + lane) * nr + j);
        const int ch = __ldg(chl + c0 + lane);
        const int cu = __ldg(d.fNrow + ch) - __ldg(d.fNpiv + ch);
        off = __ldg(d.fUOff + ch) + ((int64_t)b * cu - (int64_t)b * (b - 1) / 2 - b);
      }
      for (unsigned m = __ballot_sync(0xffffffffu, b >= 0); m; m &= m - 1) {
        const int c = __ffs(m) - 1;
        const int* ic = inv + (int64_t)(c0 + c) * nr;
        const T* U = Ubase + __shfl_sync(0xffffffffu, off, c);
        int a[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = i0 + 32 * q + lane;
          a[q] = (i < nr && i >= j) ? __ldg(ic + i) : -1;
        }
        T x[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) x[q] = a[q] >= 0 ? ld(U + a[q]) : T(0);
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] += x[q];
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = i0 + 32 * q + lane;
      if (i < nr && i >= j) st(F.at(i, j), v[q]);
    }
    __syncwarp();
    for (int k = k0 + lane; k < k1; k += 32) {
      const int i = __ldg(d.asmPos + ao + k) - nr * j;
      if (i >= i0 && i < i0 + 128) {
        T* q = F.L + i + (int64_t)nr * j;
        st(q, ld(q) + ld(asmVal + ao + k));
      }
    }
  }
}

// Assembly and blocked partial LDL^T of large front t.f by its G blocks
template <typename T>
__device__ void factorLarge(const DevData& d, const LargePlan& lp, const LargeTask& t, const T* asmVal, T* Lbase,
                            T* Ubase, double tolFact, FactorShared<T>& s, WaitState& ws) {
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int f = t.f, G = t.G;
  const Front<T> F{Lbase + d.fLOff[f], Ubase + d.fUOff[f], d.fNrow[f], d.fNpiv[f], d.fNrow[f] - d.fNpiv[f]};
  const int nr = F.nr, np = F.np;
  int* bar = lp.bar + t.li;
  const int gw = t.rank + G * w, nw = G * kLW;  // warps numbered across the blocks first: one per sub-core
  // a pivot is singular when |d_k| <= tolFactorize |a_kk| (the original entry);
  // the thresholds of a panel are loaded ahead of it
  auto threshold = [&](int k) {
    return singularBound(ld(asmVal + __ldg(lp.diagAsm + lp.diagOff[t.li] + k)), (T)tolFact);
  };
  if (tid < min(kPanel, np)) s.diag0[0][tid] = threshold(tid);
  assembleLarge<T>(d, lp, t, F, asmVal, Ubase);
  int phase = 0, neg = 0;
  bool sing = false;
  for (int k0 = 0; k0 < np; k0 += kPanel) {
    groupBarrier(bar, G, ++phase, ws);  // the panel's columns complete (assembly, earlier trailing updates)
    const int kb = min(kPanel, np - k0);
    T* diag0 = s.diag0[(k0 / kPanel) & 1];
    for (int q = tid; q < kPanel * kPanel; q += kLT) {
      const int c = q >> 5, r = q & 31;
      if (c < kb && r < kb && r >= c) s.Lt[c][r] = ld(F.L + (k0 + r) + (int64_t)nr * (k0 + c));
    }
    // this warp's first row below the block, loaded beside the block's factorisation
    const int rBelow = k0 + kb;
    T a0 = T(0);
    if (rBelow + gw < nr && lane < kb) a0 = ld(F.L + (rBelow + gw) + (int64_t)nr * (k0 + lane));
    __syncthreads();
    factorDiagonal<T>(s, diag0, kb, neg, sing);
    // rows below the block: lane j holds column j; for k in order a_j -= a_k l_jk, then l_j = a_j / d_j
    const T di = lane < kb ? s.dinv[lane] : T(0);
    for (int r = rBelow + gw; r < nr; r += nw) {
      T a = a0;
      if (r + nw < nr && lane < kb) a0 = ld(F.L + (r + nw) + (int64_t)nr * (k0 + lane));
      for (int k = 0; k < kb - 1; ++k) {
        const T x = __shfl_sync(0xffffffffu, a, k);
        a -= x * s.Lt[k][lane];  // zero at and above the diagonal
      }
      if (lane < kb) st(F.L + r + (int64_t)nr * (k0 + lane), a * di);
    }
    groupBarrier(bar, G, ++phase, ws);  // the panel's rows complete
    // every block has read the unfactored diagonal block by now
    if (t.rank == 0)
      for (int q = tid; q < kPanel * kPanel; q += kLT) {
        const int c = q >> 5, r = q & 31;
        if (c < kb && r < kb && r >= c) st(F.L + (k0 + r) + (int64_t)nr * (k0 + c), r == c ? s.d[c] : s.Lt[c][r]);
      }
    const int nt = nr - rBelow;
    if (nt <= 0) break;
    if (tid < min(kPanel, np - rBelow)) s.diag0[(rBelow / kPanel) & 1][tid] = threshold(rBelow + tid);
    // trailing lower triangle in 16 x 16 blocks (row block rb >= column block cb)
    constexpr int kHalves = std::is_same<T, float>::value ? 1 : 2;
    const int nb = (nt + 15) >> 4, ntask = kHalves * (nb * (nb + 1) / 2);
    for (int task = gw; task < ntask; task += nw) {
      const int blk = task / kHalves, half = task % kHalves;
      int rb = (int)((sqrtf(8.0f * (float)blk + 1.0f) - 1.0f) * 0.5f);
      while ((rb + 1) * (rb + 2) / 2 <= blk) ++rb;
      while (rb * (rb + 1) / 2 > blk) --rb;
      const int cb = blk - rb * (rb + 1) / 2;
      const int c0 = rBelow + 16 * cb + 8 * half;
      if (c0 < nr) trailingBlock(F, s, k0, kb, rBelow + 16 * rb, c0);
    }
  }
  if (tid == 0 && t.rank == 0) {
    const int m = d.fModel[f];
    if (neg) atomicAdd(&d.m.negPiv[m], neg);
    if (sing) atomicOr(&d.m.status[m], SS_SINGULAR);
  }
}

// The waves of this block whose front's model has all of `want` in its flags,
// as a mask in shared memory (kLT waves from `base`): one round of loads, so
// that an iteration with nothing to do passes its waves at once.
__device__ inline void scanWaves(const DevData& d, const LargePlan& lp, int base, int want, unsigned char* todo) {
  const int wv = base + threadIdx.x;
  bool on = false;
  if (wv < lp.nWaves) {
    const int f = lp.tasks[(int64_t)wv * gridDim.x + blockIdx.x].f;
    on = f >= 0 && (d.m.flags[d.fModel[f]] & want) == want;
  }
  todo[threadIdx.x] = on ? 1 : 0;
  __syncthreads();
}

template <typename T, int PER_SM>
__global__ void __launch_bounds__(kLT, PER_SM) kLargeFactor(DevData d, LargePlan lp, const T* asmVal, T* Lbase, T* Ubase,
                                                     double tolFact) {
  pdlEntry();
  extern __shared__ __align__(16) unsigned char smraw[];
  FactorShared<T>& s = *reinterpret_cast<FactorShared<T>*>(smraw);
  WaitState ws{lp.err, lp.spinLimit, false};
  __shared__ unsigned char todo[kLT];
  for (int wv = 0; wv < lp.nWaves; ++wv) {
    if (wv % kLT == 0) scanWaves(d, lp, wv, FL_ACTIVE | FL_TANGENT, todo);
    if (!todo[wv % kLT]) {
      if (wv % kLT == kLT - 1) __syncthreads();
      continue;
    }
    const LargeTask t = lp.tasks[(int64_t)wv * gridDim.x + blockIdx.x];
    const int need = lp.expect[t.li];
    if (need > 0) waitCount(lp.done + t.li, need, ws);
    factorLarge<T>(d, lp, t, asmVal, Lbase, Ubase, tolFact, s, ws);
    __syncthreads();
    const int par = lp.parent[t.li];
    if (threadIdx.x == 0 && par >= 0) signalCount(lp.done + par);
  }
}

// ---- solves -----------------------------------------------------------------
// asynchronous global -> shared copies of single elements
template <typename T>
__device__ inline void copyAsync(T* dstShared, const T* srcGlobal) {
  const unsigned dst = (unsigned)__cvta_generic_to_shared(dstShared);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(dst), "l"(srcGlobal), "n"(sizeof(T)));
}
__device__ inline void copyAsyncWait() {
  asm volatile("cp.async.commit_group;\n" ::);
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// values of L a block of the solves stages in shared memory: the pivot block
// (np columns, an odd number of rows apart so that the back substitution's
// reads across columns hit different banks) and its share of the rows below
// (forward) or of the columns (backward)
__host__ __device__ inline int64_t forwardStage(int nr, int np, int G) {
  return (int64_t)np * (np | 1) + (int64_t)((nr - np + G - 1) / G) * np;
}
__host__ __device__ inline int64_t backwardStage(int nr, int np, int G) {
  return (int64_t)np * (np | 1) + (int64_t)((np + G - 1) / G) * (nr - np);
}

// ---- inverses of the pivot blocks ----------------------------------------------
// The solves multiply by the inverse of each 32 x 32 unit lower pivot block instead
// of substituting through it: 32 dependent steps of a shuffle and a multiply-add
// (3,000 cycles in FP64) become one product shared by four warps (850).  The space-
// frame tower's solves, 17 fronts deep, spent more than half their time there.
// inverse + 2048 blk: the block's inverse column by column (entry (i, k) at
// 32 k + i), then row by row (1024 + 32 i + k); identity beyond a short block.
// this lane's (row or column `lane`) eight values 8 h .. 8 h + 7
template <typename T>
__device__ inline void loadInverse(T* li, const T* inv, int h, int lane) {
#pragma unroll
  for (int q = 0; q < 8; ++q) li[q] = ld(inv + 32 * (8 * h + q) + lane);
}

// One block of 128 threads per pivot block (of a model that factored): the 8 x 8
// diagonal blocks by substitution, then twice the size from the halves,
// [A 0; B C]^-1 = [A' 0; -C' B A' C'].
template <typename T>
__global__ void __launch_bounds__(128) kLargeInverse(DevData d, LargePlan lp, const T* Lbase) {
  pdlEntry();
  __shared__ T L[32][33], V[32][33], M[16][17];  // [row][column]
  const int f = lp.invFront[blockIdx.x], k0 = 32 * lp.invPart[blockIdx.x];
  const int fl = d.m.flags[d.fModel[f]];
  if (!(fl & FL_ACTIVE) || !(fl & FL_TANGENT)) return;
  const int nr = d.fNrow[f], kb = min(32, d.fNpiv[f] - k0);
  const T* Lf = Lbase + d.fLOff[f] + k0 + (int64_t)nr * k0;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  for (int q = tid; q < 1024; q += 128) {
    const int i = q & 31, k = q >> 5;
    L[i][k] = (i > k && i < kb) ? ld(Lf + i + (int64_t)nr * k) : T(0);
    V[i][k] = T(0);
  }
  __syncthreads();
  if (lane < 8) {  // column `lane` of the inverse of diagonal block w
    T x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      T a = T(0);
#pragma unroll
      for (int k = 0; k < i; ++k) a += L[8 * w + i][8 * w + k] * x[k];
      x[i] = i == lane ? T(1) : (i > lane ? -a : T(0));
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) V[8 * w + i][8 * w + lane] = x[i];
  }
  __syncthreads();
  {  // 16: one entry of each product per thread
    const int p = tid >> 6, i = (tid >> 3) & 7, k = tid & 7, o = 16 * p;
    T a = T(0);
#pragma unroll
    for (int j = 0; j < 8; ++j) a += L[o + 8 + i][o + j] * V[o + j][o + k];
    M[8 * p + i][k] = a;
    __syncthreads();
    a = T(0);
#pragma unroll
    for (int j = 0; j < 8; ++j) a += V[o + 8 + i][o + 8 + j] * M[8 * p + j][k];
    V[o + 8 + i][o + k] = -a;
  }
  __syncthreads();
  {  // 32: two entries of each product per thread
    const int i = tid >> 3, k = tid & 7;
    T a = T(0), b = T(0);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      a += L[16 + i][j] * V[j][k];
      b += L[16 + i][j] * V[j][k + 8];
    }
    __syncthreads();
    M[i][k] = a;
    M[i][k + 8] = b;
    __syncthreads();
    a = b = T(0);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      a += V[16 + i][16 + j] * M[j][k];
      b += V[16 + i][16 + j] * M[j][k + 8];
    }
    V[16 + i][k] = -a;
    V[16 + i][k + 8] = -b;
  }
  __syncthreads();
  T* out = static_cast<T*>(lp.inverse) + 2048 * (int64_t)blockIdx.x;
  for (int q = tid; q < 1024; q += 128) {
    out[q] = V[q & 31][q >> 5];
    out[1024 + q] = V[q >> 5][q & 31];
  }
}

// Forward elimination of front t.f, y = L11^-1 v_p, w = v_u - L21 y, by its G
// blocks: each solves the pivot block itself (no barrier) and takes a slice of
// the rows below it.  L does not depend on the children: it is staged in shared
// memory while the block waits for them.  Rows below: a warp takes 32 rows and
// a quarter of the pivots (a sub-core issues one FP64 instruction per 64
// cycles, so the pivots are shared out too); the quarters are added in order.
template <typename T>
__device__ void forwardLarge(const DevData& d, const LargePlan& lp, const LargeTask& t, const T* Lbase,
                             const double* rhs, T* X, T* W, T* v, T* part, T* Ls, WaitState& ws) {
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int f = t.f, nr = d.fNrow[f], np = d.fNpiv[f], nu = nr - np;
  const int share = (nu + t.G - 1) / t.G, r0 = np + t.rank * share, r1 = min(nr, r0 + share), ns = max(0, r1 - r0);
  const T* L = Lbase + d.fLOff[f];
  const int* rows = d.frontRows + d.fRowOff[f];
  // pivot block at Ls[i + lds k], rows r0..r1-1 at Lr[(i - r0) + ns k]
  const bool staged = forwardStage(nr, np, t.G) <= lp.stageCap;
  const int lds = np | 1;
  T* Lr = Ls + (int64_t)np * lds;
  __syncthreads();  // the previous front's reads of the staging area are done
  if (staged) {
    for (int k = w; k < np; k += kLW) {
      for (int i = k + lane; i < np; i += 32) copyAsync(Ls + i + lds * k, L + i + (int64_t)nr * k);
      for (int i = lane; i < ns; i += 32) copyAsync(Lr + i + ns * k, L + r0 + i + (int64_t)nr * k);
    }
  }
  const T* Lp = staged ? Ls : L;
  const int ldp = staged ? lds : nr;
  const T* Lq = staged ? Lr : L + r0;
  const int ldq = staged ? ns : nr;
  T li[8];  // this lane's share of a pivot block's inverse
  const T* linv = static_cast<const T*>(lp.inverse) + 2048 * (int64_t)lp.invBlk[t.li];
  if (w < 4) loadInverse(li, linv, w, lane);
  // the right-hand side of the pivot rows, and where the children's
  // contributions to the pivot rows and to this block's rows come from (in
  // child order), before the wait; their values after it
  const int* gOff = lp.gOff + lp.gRow[t.li];
  const int nv = np + ns;
  int p0 = 0, p1 = 0, src[4] = {0, 0, 0, 0};
  T x = T(0);
  if (tid < nv) {
    const int r = tid < np ? tid : r0 + tid - np;
    p0 = __ldg(gOff + r);
    p1 = __ldg(gOff + r + 1);
    if (tid < np) x = (T)rhs[__ldg(rows + r)];
#pragma unroll
    for (int q = 0; q < 4; ++q) src[q] = p0 + q < p1 ? __ldg(lp.gSrc + p0 + q) : -1;
  }
  const int need = lp.expect[t.li];
  if (need > 0) waitCount(lp.done + t.li, need, ws);
  for (int q0 = tid; q0 < nv; q0 += kLT) {
    if (q0 != tid) {
      const int r = q0 < np ? q0 : r0 + q0 - np;
      p0 = __ldg(gOff + r);
      p1 = __ldg(gOff + r + 1);
      x = q0 < np ? (T)rhs[__ldg(rows + r)] : T(0);
#pragma unroll
      for (int q = 0; q < 4; ++q) src[q] = p0 + q < p1 ? __ldg(lp.gSrc + p0 + q) : -1;
    }
    T c[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) c[q] = src[q] >= 0 && p0 + q < p1 ? ld(W + src[q]) : T(0);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (p0 + q < p1) x += c[q];
    for (int p = p0 + 4; p < p1; ++p) x += ld(W + __ldg(lp.gSrc + p));
    v[q0] = x;
  }
  if (staged) copyAsyncWait();
  __syncthreads();
  for (int b0 = 0; b0 < np; b0 += 32) {
    const int bs = min(32, np - b0);
    // the block's pivots: inverse times right-hand side, a quarter of the columns
    // per warp (the next block's inverse is loaded meanwhile)
    if (w < 4) {
      T a = T(0);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (8 * w + q < bs) a += li[q] * v[b0 + 8 * w + q];
      part[tid] = a;
      if (b0 + 32 < np) loadInverse(li, linv + 2048 * (b0 / 32 + 1), w, lane);
    }
    __syncthreads();
    if (w == 0 && lane < bs) v[b0 + lane] = ((part[lane] + part[32 + lane]) + part[64 + lane]) + part[96 + lane];
    __syncthreads();
    // the later pivot rows: four lanes a row, each a quarter of the block's pivots
    const int left = np - b0 - bs;
    for (int q = tid; q < ((4 * left + 31) & ~31); q += kLT) {
      const int i = b0 + bs + (q >> 2), h = q & 3;
      T a = T(0);
      if (i < np)
        for (int k = 8 * h; k < min(bs, 8 * h + 8); ++k) a += Lp[i + (int64_t)ldp * (b0 + k)] * v[b0 + k];
      T sum = __shfl_sync(0xffffffffu, a, lane & ~3);
#pragma unroll
      for (int o = 1; o < 4; ++o) sum += __shfl_sync(0xffffffffu, a, (lane & ~3) + o);
      if (h == 0 && i < np) v[i] -= sum;
    }
    __syncthreads();
  }
  if (t.rank == 0)
    for (int r = tid; r < np; r += kLT) st(X + __ldg(rows + r), v[r] / Lp[r + (int64_t)ldp * r]);
  // rows below: quarter h of the pivots of 32 rows per warp, two row groups at a time
  const int qn = (np + 3) >> 2;
  T* wo = W + d.fWOff[f] + (r0 - np);
  for (int g0 = 0; g0 < ns; g0 += 64) {
    const int g = g0 + 32 * (w >> 2), h = w & 3, i = g + lane;
    T a = T(0);
    if (i < ns) {
      const int ke = min(np, (h + 1) * qn);
#pragma unroll 8
      for (int k = h * qn; k < ke; ++k) a += Lq[i + (int64_t)ldq * k] * v[k];
    }
    part[tid] = a;
    __syncthreads();
    if (h == 0 && i < ns) {
      T sum = a;
#pragma unroll
      for (int o = 1; o < 4; ++o) sum += part[tid + 32 * o];
      st(wo + i, v[np + i] - sum);
    }
    __syncthreads();
  }
}

template <typename T, int PER_SM>
__global__ void __launch_bounds__(kLT, PER_SM) kLargeForward(DevData d, LargePlan lp, const T* Lbase, const double* rhs, T* X,
                                                      T* W) {
  pdlEntry();
  extern __shared__ __align__(16) unsigned char smraw[];
  T* v = reinterpret_cast<T*>(smraw);
  T* part = v + lp.maxRow;
  T* Ls = part + kLT;
  WaitState ws{lp.err, lp.spinLimit, false};
  __shared__ unsigned char todo[kLT];
  for (int wv = 0; wv < lp.nWaves; ++wv) {
    if (wv % kLT == 0) scanWaves(d, lp, wv, FL_ACTIVE, todo);
    if (!todo[wv % kLT]) {
      if (wv % kLT == kLT - 1) __syncthreads();
      continue;
    }
    const LargeTask t = lp.tasks[(int64_t)wv * gridDim.x + blockIdx.x];
    forwardLarge<T>(d, lp, t, Lbase, rhs, X, W, v, part, Ls, ws);
    __syncthreads();
    const int par = lp.parent[t.li];
    if (threadIdx.x == 0 && par >= 0) signalCount(lp.done + par);
  }
}

// Back substitution of front t.f, x_p = L11^-T (v_p - L21^T x_u), waves taken
// from the last: its blocks share out the pivot columns (a warp per column),
// block 0 then solves the pivot block and signals the children.  L is staged
// while the block waits for the parent.
template <typename T>
__device__ void backwardLarge(const DevData& d, const LargePlan& lp, const LargeTask& t, const T* Lbase, T* X, int acc,
                              int finalize, T* xs, T* part, T* Ls, WaitState& ws) {
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int f = t.f, nr = d.fNrow[f], np = d.fNpiv[f], nu = nr - np;
  const T* L = Lbase + d.fLOff[f];
  const int* rows = d.frontRows + d.fRowOff[f];
  const int cshare = (np + t.G - 1) / t.G, k0 = t.rank * cshare, k1 = min(np, k0 + cshare), nc = max(0, k1 - k0);
  const bool staged = backwardStage(nr, np, t.G) <= lp.stageCap;
  const int lds = np | 1;
  T* Lc = Ls + (t.rank == 0 ? (int64_t)np * lds : 0);  // columns k0..k1-1 below the pivot block, nu values each
  __syncthreads();
  if (staged) {
    for (int k = w; k < nc; k += kLW)
      for (int i = lane; i < nu; i += 32) copyAsync(Lc + i + nu * k, L + np + i + (int64_t)nr * (k0 + k));
    if (t.rank == 0)
      for (int k = w; k < np; k += kLW)
        for (int i = k + 1 + lane; i < np; i += 32) copyAsync(Ls + i + lds * k, L + i + (int64_t)nr * k);
  }
  const T* Lq = staged ? Lc : L + np + (int64_t)nr * k0;
  const int ldq = staged ? nu : nr;
  // row indices and this warp's first pivot value before the wait
  const int par = lp.parent[t.li];
  int row[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) row[q] = np + tid + kLT * q < nr ? __ldg(rows + np + tid + kLT * q) : -1;
  const int rowk = w < nc ? __ldg(rows + k0 + w) : 0, rowp = tid < np ? __ldg(rows + tid) : 0;
  const T yk = w < nc ? ld(X + rowk) : T(0);
  // (block 0) the last pivot block's inverse, row by row
  T li[8];
  const T* linv = static_cast<const T*>(lp.inverse) + 2048 * (int64_t)lp.invBlk[t.li] + 1024;
  if (t.rank == 0 && w < 4) loadInverse(li, linv + 2048 * ((np - 1) / 32), w, lane);
  if (par >= 0) waitCount(lp.done + par, 1, ws);
#pragma unroll
  for (int q = 0; q < 2; ++q)
    if (row[q] >= 0) xs[np + tid + kLT * q] = ld(X + row[q]);
  for (int r = np + tid + 2 * kLT; r < nr; r += kLT) xs[r] = ld(X + __ldg(rows + r));
  if (staged) copyAsyncWait();
  __syncthreads();
  for (int k = w; k < nc; k += kLW) {
    T a = T(0);
#pragma unroll 4
    for (int i = lane; i < nu; i += 32) a += Lq[i + (int64_t)ldq * k] * xs[np + i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if (lane == 0) {
      if (k == w) {
        st(X + rowk, yk - a);
      } else {
        T* q = X + __ldg(rows + k0 + k);
        st(q, ld(q) - a);
      }
    }
  }
  __syncthreads();
  if (t.rank != 0) {
    if (tid == 0) signalCount(lp.bar + t.li);
    return;
  }
  if (t.G > 1) waitCount(lp.bar + t.li, t.G - 1, ws);
  for (int r = tid; r < np; r += kLT) xs[r] = ld(X + (r == tid ? rowp : __ldg(rows + r)));
  __syncthreads();
  const T* Lp = staged ? Ls : L;
  const int ldp = staged ? lds : nr;
  // the unit upper triangle L11^T, the factorisation's blocks of 32 pivots from the
  // last: the transposed inverse of the block times its values, then the pivots
  // above it are updated
  for (int bEnd = np; bEnd > 0; bEnd = (bEnd - 1) & ~31) {
    const int b0 = (bEnd - 1) & ~31, bs = bEnd - b0;
    if (w < 4) {
      T a = T(0);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (8 * w + q < bs) a += li[q] * xs[b0 + 8 * w + q];
      part[tid] = a;
      if (b0 > 0) loadInverse(li, linv + 2048 * (b0 / 32 - 1), w, lane);
    }
    __syncthreads();
    if (w == 0 && lane < bs) xs[b0 + lane] = ((part[lane] + part[32 + lane]) + part[64 + lane]) + part[96 + lane];
    __syncthreads();
    // pivots above the block: four lanes a pivot, each a quarter of the block's rows
    for (int q = tid; q < ((4 * b0 + 31) & ~31); q += kLT) {
      const int k = q >> 2, h = q & 3;
      T a = T(0);
      if (k < b0)
        for (int j = 8 * h; j < min(bs, 8 * h + 8); ++j) a += Lp[b0 + j + (int64_t)ldp * k] * xs[b0 + j];
      T sum = __shfl_sync(0xffffffffu, a, lane & ~3);
#pragma unroll
      for (int o = 1; o < 4; ++o) sum += __shfl_sync(0xffffffffu, a, (lane & ~3) + o);
      if (h == 0 && k < b0) xs[k] -= sum;
    }
    __syncthreads();
  }
  for (int r = tid; r < np; r += kLT) st(X + __ldg(rows + r), xs[r]);
  __syncthreads();
  if (tid == 0) signalCount(lp.done + t.li);
  for (int r = tid; r < np; r += kLT) {
    const int row = __ldg(rows + r);
    const T x = xs[r];
    if (acc == 0) {
      d.del[row] = (double)x;
    } else {
      const double xr = acc == 1 ? (double)x : d.xref[row] + (double)x;
      d.xref[row] = xr;
      if (finalize) d.del[row] = xr;
    }
  }
}

template <typename T, int PER_SM>
__global__ void __launch_bounds__(kLT, PER_SM) kLargeBackward(DevData d, LargePlan lp, const T* Lbase, T* X, int acc,
                                                       int finalize) {
  pdlEntry();
  extern __shared__ __align__(16) unsigned char smraw[];
  T* xs = reinterpret_cast<T*>(smraw);
  T* part = xs + lp.maxRow;
  T* Ls = part + kLT;
  WaitState ws{lp.err, lp.spinLimit, false};
  __shared__ unsigned char todo[kLT];
  for (int wv = lp.nWaves - 1; wv >= 0; --wv) {
    if (wv == lp.nWaves - 1 || wv % kLT == kLT - 1) {
      __syncthreads();
      scanWaves(d, lp, wv - wv % kLT, FL_ACTIVE, todo);
    }
    if (!todo[wv % kLT]) continue;
    const LargeTask t = lp.tasks[(int64_t)wv * gridDim.x + blockIdx.x];
    backwardLarge<T>(d, lp, t, Lbase, X, acc, finalize, xs, part, Ls, ws);
  }
}

// cooperative launch (all blocks resident), ordered like any launch of the stream
template <typename... KArgs, typename... Args>
void coopLaunch(void (*kernel)(KArgs...), int grid, size_t smem, cudaStream_t s, Args... args) {
  allowBigShared(kernel);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  launchWith(attr, 1, kernel, dim3(grid), dim3(kLT), smem, s, args...);
}

// blocks per SM of the kernels for plans with levels of more fronts than SMs
// (registers: 80 and 64 a thread, the factorisation's with 50 to 110 bytes spilled)
constexpr int kWideFactor = 3, kWideSolve = 4;

template <typename T>
size_t solveShared(const LargePlan& lp) {
  return largeSolveShared(lp.maxRow, lp.stageCap, sizeof(T));
}

}  // namespace

// Blocks of a cooperative launch must all be resident: as many per SM as the device holds
// of each kernel at once, one, or (wide: batches of many fronts, see Engine::upload) up to
// kWideFactor and kWideSolve.
int largeBlocksPerSm(bool fp32, bool solve, bool wide, size_t smem) {
  auto resident = [&](auto kernel, size_t bytes, int most) {
    int n = 0;
    if (allowBigShared(kernel) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kLT, bytes) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return std::min(n, most);
  };
  auto of = [&](auto zero) {
    using T = decltype(zero);
    const size_t fs = sizeof(FactorShared<T>);
    if (!solve)
      return wide ? resident(kLargeFactor<T, kWideFactor>, fs, kWideFactor) : resident(kLargeFactor<T, 1>, fs, 1);
    return wide ? std::min(resident(kLargeForward<T, kWideSolve>, smem, kWideSolve),
                           resident(kLargeBackward<T, kWideSolve>, smem, kWideSolve))
                : std::min(resident(kLargeForward<T, 1>, smem, 1), resident(kLargeBackward<T, 1>, smem, 1));
  };
  return fp32 ? of(0.0f) : of(0.0);
}

size_t largeSolveShared(int maxRow, int64_t stage, size_t elemBytes) { return (maxRow + kLT + stage) * elemBytes; }

// at most about 200 KB of staged L per block
int64_t largeSolveStage(int nr, int np, int G, size_t elemBytes) {
  const int64_t want = std::max(forwardStage(nr, np, G), backwardStage(nr, np, G));
  return std::min<int64_t>(want, (int64_t)(200 * 1024 / elemBytes));
}

namespace {
template <typename T>
void factorLaunch(const DevData& d, const LargePlan& lp, const T* asmVal, T* L, T* U, cudaStream_t s) {
  coopLaunch(lp.wide ? kLargeFactor<T, kWideFactor> : kLargeFactor<T, 1>, lp.grid, sizeof(FactorShared<T>), s, d, lp,
             asmVal, L, U, 1.0e-12);
  // the inverses of the pivot blocks, for the solves
  pdlLaunch(kLargeInverse<T>, lp.nInvBlk, 128, 0, s, d, lp, (const T*)L);
}
template <typename T>
void forwardLaunch(const DevData& d, const LargePlan& lp, const T* L, const double* rhs, T* X, T* W, cudaStream_t s) {
  coopLaunch(lp.wide ? kLargeForward<T, kWideSolve> : kLargeForward<T, 1>, lp.grid, solveShared<T>(lp), s, d, lp, L,
             rhs, X, W);
}
template <typename T>
void backwardLaunch(const DevData& d, const LargePlan& lp, const T* L, T* X, int acc, int fin, cudaStream_t s) {
  coopLaunch(lp.wide ? kLargeBackward<T, kWideSolve> : kLargeBackward<T, 1>, lp.grid, solveShared<T>(lp), s, d, lp, L,
             X, acc, fin);
}
}  // namespace

void launchLargeFactor(const DevData& d, const PersistentPlan& p, bool fp32, cudaStream_t s) {
  if (p.nLarge <= 0) return;
  int shape = 0;
  for (int k = 0; k < 4; ++k)
    if (p.largeCluster == (2 << k)) shape = k;
  LargePlan lp = p.large[shape];
  lp.spinLimit = p.spinLimit;
  lp.done = p.cntLarge;
  lp.bar = p.cntLarge + p.nLarge;
  if (fp32) factorLaunch<float>(d, lp, d.asmVal32, d.L32, d.U32, s);
  else factorLaunch<double>(d, lp, d.asmVal64, d.L64, d.U64, s);
}

void launchLargeForward(const DevData& d, const PersistentPlan& p, bool fp32, const double* rhs, int sweep,
                        cudaStream_t s) {
  if (p.nLarge <= 0) return;
  LargePlan lp = p.large[4];
  lp.spinLimit = p.spinLimit;
  lp.done = p.cntLarge + (size_t)(2 + 3 * sweep) * p.nLarge;
  if (fp32) forwardLaunch<float>(d, lp, d.L32, rhs, d.x32, d.w32, s);
  else forwardLaunch<double>(d, lp, d.L64, rhs, d.x64, d.w64, s);
}

void launchLargeBackward(const DevData& d, const PersistentPlan& p, bool fp32, int sweep, bool last, cudaStream_t s) {
  if (p.nLarge <= 0) return;
  const int acc = !fp32 ? 0 : (sweep == 0 ? 1 : 2);
  const int fin = (fp32 && last) ? 1 : 0;
  LargePlan lp = p.large[4];
  lp.spinLimit = p.spinLimit;
  lp.done = p.cntLarge + (size_t)(3 + 3 * sweep) * p.nLarge;
  lp.bar = p.cntLarge + (size_t)(4 + 3 * sweep) * p.nLarge;
  if (fp32) backwardLaunch<float>(d, lp, d.L32, d.x32, acc, fin, s);
  else backwardLaunch<double>(d, lp, d.L64, d.x64, acc, fin, s);
}

void launchLargeWaitProbe(const DevData& d, const PersistentPlan& p, bool fp32, const LargeTask* task, int* done,
                          int* bar, bool backward, long long spins, cudaStream_t s) {
  // one block with one front: the forward elimination waits for children that nothing
  // signals, the back substitution of a root for the second block of the front; each goes
  // on to its end on what is there (the solve vectors and update vectors, which the next
  // solve rewrites)
  LargePlan lp = p.large[4];
  lp.spinLimit = spins;
  lp.tasks = task;
  lp.nWaves = lp.grid = 1;
  lp.done = done;
  lp.bar = bar;
  if (backward) {
    if (fp32) backwardLaunch<float>(d, lp, d.L32, d.x32, 1, 0, s);
    else backwardLaunch<double>(d, lp, d.L64, d.x64, 0, 0, s);
  } else if (fp32) {
    forwardLaunch<float>(d, lp, d.L32, d.del, d.x32, d.w32, s);
  } else {
    forwardLaunch<double>(d, lp, d.L64, d.del, d.x64, d.w64, s);
  }
}

}  // namespace fgpu

// front_kernels.cu -- FP64 refinement residual of the mixed-precision solves.
//
// The multifrontal factorisation and the triangular solves replace the factor
// and solve of the absent SAM/SPR solver that the reference calls from csSolve
// (src/vpmCommon/vpmLinAlg/solExtensionModule.f90:153-505); they live in
// front_cascade.cu.  With FP32 fronts, each further solve of a Newton
// iteration corrects the accumulated FP64 solution x with the residual
// r = b - A x of the FP64 Newton matrix computed here.

#include "kernels.h"

namespace fgpu {
namespace {

constexpr int TPB = 256;
inline int blocksFor(long long n, int tpb = TPB) { return (int)((n + tpb - 1) / tpb); }

// r = b - A x with the FP64 Newton matrix (full symmetric CSR), one row per thread.
// Bound by HBM (12 bytes an entry, read once) with the FP64 pipe close behind (one
// instruction an entry), if enough loads are in flight: entry by entry 256 chains
// (1,020,000 rows of 18) took 35.7 us, six entries' loads at a time 30.2.  (Copying a
// warp's rows into shared memory by whole lines first: 73 us, too few warps left.)
constexpr int kRefineBatch = 6;
__global__ void kRefineResidual(DevData d) {
  pdlEntry();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.neqTot) return;
  // the row's extent is read with the model index, before the activity test
  const int64_t kb = d.rowPtr[i], ke = d.rowPtr[i + 1];
  if (!(d.m.flags[d.eqModel[i]] & FL_ACTIVE)) return;
  // kRefineBatch entries at a time, their loads independent of each other
  double s = 0.0;
  for (int64_t k = kb; k < ke; k += kRefineBatch) {
    double v[kRefineBatch], x[kRefineBatch];
    int c[kRefineBatch];
#pragma unroll
    for (int u = 0; u < kRefineBatch; ++u) {
      const bool in = k + u < ke;
      c[u] = in ? d.colInd[k + u] : 0;
      v[u] = in ? d.csrVal[k + u] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kRefineBatch; ++u) x[u] = d.xref[c[u]];
#pragma unroll
    for (int u = 0; u < kRefineBatch; ++u)
      if (k + u < ke) s += v[u] * x[u];
  }
  d.rref[i] = d.del[i] - s;
}

}  // namespace

void launchRefineResidual(const DevData& d, cudaStream_t s) {
  if (d.neqTot > 0) pdlLaunch(kRefineResidual, blocksFor(d.neqTot), TPB, 0, s, d);
}

}  // namespace fgpu

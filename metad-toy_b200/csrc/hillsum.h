// hillsum.h -- the exact FP64 hill sum over a batch of CV points (hillsum.cu).
#pragma once

#include <cuda_runtime.h>

namespace mtd {

// Doubles per packed hill: [c0 c1 c2 c3 w 1/(2 sigma^2) 1/sigma^2 80 sigma^2]
// (centres beyond D are zero).  A hill with r^2 above the last entry
// contributes below w e^-40 (4e-18 w) and is skipped.
constexpr int kHillRec = 8;

// V (npts) and, when dV is not null, dV/ds (rows of gs doubles, the first D
// written, all gs when gs is 4) at npts device points (rows of ps >= D
// doubles), enqueued on st.  [lo, hi] is the box that the points are expected
// in: it shapes the spatial order only, points outside are as good.  `scratch`
// (hillsum_scratch bytes, any contents; small sums need none) is in use until the
// call has run; without it (null) the sum is one kernel that leaves out fewer
// hills, with the same results.
size_t hillsum_scratch(int npts, int nh);
cudaError_t hillsum_batch(int D, const double *lo, const double *hi, int npts, const double *pts, int ps, int nh,
                          const double *hills, double *V, double *dV, int gs, void *scratch, cudaStream_t st);

}  // namespace mtd

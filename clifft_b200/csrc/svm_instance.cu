// One instance of the interpreter kernel (svm_kernel.cuh) per translation
// unit: the build compiles this file once for every row of CGPU_INSTANCES
// (svm_dispatch.h) with CGPU_NAME, CGPU_REAL, CGPU_G, CGPU_NW and CGPU_DENSE
// set, so the instances compile in parallel.
#include "svm_dispatch.h"
#include "svm_kernel.cuh"

namespace cgpu {
KernelFn CGPU_NAME() { return svm_sample_kernel<CGPU_REAL, CGPU_G, CGPU_NW, CGPU_DENSE != 0>; }
}  // namespace cgpu

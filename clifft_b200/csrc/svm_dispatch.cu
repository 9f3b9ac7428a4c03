// Kernel table over the instances that svm_instance.cu compiles to.
#include "svm_dispatch.h"

#include <type_traits>

namespace cgpu {

#define CGPU_DECLARE(name, real, g, nw, dense) KernelFn name();
CGPU_INSTANCES(CGPU_DECLARE)
#undef CGPU_DECLARE

KernelFn find_kernel(bool fp64, int G, int nw, bool dense) {
    const int width = nw <= 1 ? 1 : 4;
#define CGPU_MATCH(name, real, g, w, d) \
    if (fp64 == std::is_same<real, double>::value && G == g && width == w && dense == (d != 0)) return name();
    CGPU_INSTANCES(CGPU_MATCH)
#undef CGPU_MATCH
    return nullptr;
}

}  // namespace cgpu

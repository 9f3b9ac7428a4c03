// Kernel table shared by the host code and the kernel instances.
#pragma once

namespace cgpu {

struct DevProg;
struct KParams;
using KernelFn = void (*)(const DevProg, const KParams);

// Every kernel instance: X(name, statevector type, G, NW, dense).
// G = lanes per shot (1, 2, 4, 8, 16, 32), 0 for one CTA per shot, -1 for
// one CTA per shot whose last warp moves the fused blocks' tiles, -2 for a
// team of such CTAs per shot; NW = frame
// words (1, or 2..4 served by the 4-word kernel); dense: with the tensor-core
// dense blocks. The build reads this list (one translation unit per row).
#define CGPU_INSTANCES(X)            \
    X(f32_g1_n1, float, 1, 1, 0)     \
    X(f32_g2_n1, float, 2, 1, 0)     \
    X(f32_g4_n1, float, 4, 1, 0)     \
    X(f32_g8_n1, float, 8, 1, 0)     \
    X(f32_g16_n1, float, 16, 1, 0)   \
    X(f32_g32_n1, float, 32, 1, 0)   \
    X(f32_cta_n1, float, 0, 1, 0)    \
    X(f32_ws_n1, float, -1, 1, 0)    \
    X(f32_g1_n4, float, 1, 4, 0)     \
    X(f32_g2_n4, float, 2, 4, 0)     \
    X(f32_g4_n4, float, 4, 4, 0)     \
    X(f32_g8_n4, float, 8, 4, 0)     \
    X(f32_g16_n4, float, 16, 4, 0)   \
    X(f32_g32_n4, float, 32, 4, 0)   \
    X(f32_cta_n4, float, 0, 4, 0)    \
    X(f32_ws_n4, float, -1, 4, 0)    \
    X(f64_g1_n1, double, 1, 1, 0)    \
    X(f64_g2_n1, double, 2, 1, 0)    \
    X(f64_g4_n1, double, 4, 1, 0)    \
    X(f64_g8_n1, double, 8, 1, 0)    \
    X(f64_g16_n1, double, 16, 1, 0)  \
    X(f64_g32_n1, double, 32, 1, 0)  \
    X(f64_cta_n1, double, 0, 1, 0)   \
    X(f64_ws_n1, double, -1, 1, 0)   \
    X(f64_g1_n4, double, 1, 4, 0)    \
    X(f64_g2_n4, double, 2, 4, 0)    \
    X(f64_g4_n4, double, 4, 4, 0)    \
    X(f64_g8_n4, double, 8, 4, 0)    \
    X(f64_g16_n4, double, 16, 4, 0)  \
    X(f64_g32_n4, double, 32, 4, 0)  \
    X(f64_cta_n4, double, 0, 4, 0)   \
    X(f64_ws_n4, double, -1, 4, 0)   \
    X(f32_team_n1, float, -2, 1, 0)  \
    X(f32_team_n4, float, -2, 4, 0)  \
    X(f64_team_n1, double, -2, 1, 0) \
    X(f64_team_n4, double, -2, 4, 0) \
    X(f32_cta_n1_dense, float, 0, 1, 1) \
    X(f32_cta_n4_dense, float, 0, 4, 1) \
    X(f32_ws_n1_dense, float, -1, 1, 1) \
    X(f32_ws_n4_dense, float, -1, 4, 1)

// The instance for a precision (fp64: complex double statevectors), group
// width and frame width; nullptr when there is none.
KernelFn find_kernel(bool fp64, int G, int nw, bool dense = false);

}  // namespace cgpu

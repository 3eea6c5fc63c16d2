// Test shim: the parts of the GPU physics routines (ziran2020_gb300/csrc/physics.cuh, compiled here as host C++) whose
// arithmetic precision the CPU tests look at.
#include "../../ziran2020_gb300/csrc/physics.cuh"

using namespace zr;

extern "C" {
double shim_newton_scale(double J) { return newton_scale(J); }
double shim_gradient_share(float s, float g0, float g1, float g2) { return gradient_share(s, g0, g1, g2); }
double shim_diagonal_share(float diag, float p) { return diagonal_share(diag, p); }
}

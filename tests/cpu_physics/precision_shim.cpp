// Test shim: the parts of the GPU physics routines (ziran2020_gb300/csrc/physics.cuh, compiled here as host C++) whose
// arithmetic precision the CPU tests look at.
#include "../../ziran2020_gb300/csrc/physics.cuh"

using namespace zr;

extern "C" {
double shim_newton_scale(double J) { return newton_scale(J); }
}

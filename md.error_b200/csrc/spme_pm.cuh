// Particle-mesh steps of the SPME chain (spme_pm.cu).
#pragma once
#include "device_common.cuh"

// dynamic shared memory of the order's kernels
int pm_prepare(int prec, int order);
// charges of the system onto the (cleared) real mesh Q
int pm_spread(md_system* sys, const int K[3], int order, void* Q, Recorder* rec);
// forces from the convolved mesh G: method 0 ik (Real4 per point), 1 analytic;
// store: into `force` instead of adding
int pm_gather(md_system* sys, const int K[3], int order, int method, const void* G, double4a* force, int store,
              Recorder* rec);
// dE/dq [N] and dE/dr [N][3] (either may be null), caller's atom order
int pm_gather_adjoint(md_system* sys, const int K[3], int order, const void* G, double* dq, double* dr, Recorder* rec);

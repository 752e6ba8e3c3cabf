// Transform passes of the SPME chain for meshes whose x and y sizes are equal
// (spme_plane.cu).
#pragma once
#include "device_common.cuh"

struct PlaneChain {
  int n, K2, method;     // method 0 ik, 1 analytic, 2 adjoint
  void* Q;               // real mesh, cleared behind the first pass
  void* C;               // four half meshes of complex values
  void* G;               // convolved mesh: Real4 per point (ik) or one Real
  const double* bm;      // per-axis |b(m)|^2
  const void* tw_n;      // twiddles of the x and y axes, and of z
  const void* tw_z;
  double beta;
  double* partials;
  int with_stats, merge;
  int back;              // 0: the adjoint ends with the k-space step (energy and dE/dbeta alone)
  double *energy, *dbeta;  // adjoint: device results (may be null)
};

// whether the chain's transforms run by planes
bool plane_chain_ok(int prec, const int K[3]);
int plane_prepare(int prec, const int K[3], int method);
// z forward, plane, z backward (with back)
int plane_chain(md_system* sys, const PlaneChain& p, Recorder* rec);

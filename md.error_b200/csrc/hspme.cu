// SPME (ik differentiation) with a piecewise cubic Hermite interpolation basis,
// and the hand-written adjoints that give the gradients of its energy and of a
// force-error functional with respect to the charges, the positions and the
// basis coefficients, for a batch of candidate bases, in FP64 on the GPU.
//
// The basis is optiBasis's symmetric Hermite basis (optiBasis/Hermite.py:6-130,
// optiBasis/HatComput.py:155-300): phi(x) = p(|x|) on |x| < CC grid units, p
// the cubic Hermite interpolant on nbin bins of width h = CC/nbin with value 1
// and slope 0 at 0 and the candidate's values v_j and slopes d_j at the other
// knots (coefficients [v_1..v_n, d_1..d_n], n = nbin, or nbin - 1 when bound0:
// value and slope 0 at CC).  The SPME it defines (RE/src/EleRecBSpline.cpp:
// 393-536 with the B-spline replaced by phi):
//   u_i,d   = K_d frac(r_i,d / L_d),  W_i(k) = prod_d phi(u_i,d - k_d)
//   Q(k)    = sum_i q_i W_i(k)                         (periodic in k)
//   Qh(m)   = sum_k Q(k) exp(-2 pi i m.k / K)
//   G(m)    = exp(-pi^2 |m|^2 / beta^2) / (pi V |m|^2) prod_d 1 / b_d(m_d)^2,
//             |m|^2 = sum_d (m_d / L_d)^2, G(0) = 0,
//             b_d(m)  = sum_{k integer} phi(k) exp(-2 pi i m k / K_d)   (real)
//   E       = 1/2 sum_m G(m) |Qh(m)|^2
//   phi_pot = IFFT(G Qh) (unnormalised: E = 1/2 sum_k Q phi_pot by Parseval)
//   F_i     = -q_i sum_k W_i(k) grad phi_pot(k),  grad phi_pot by ik:
//             IFFT(i 2 pi m_a/L_a G Qh) (the Nyquist term of axis a zeroed)
// b_d is the interpolation factor of SPME (1/|b(m)|^2 of calB,
// EleRecBSpline.cpp:729-796, is prod over the integer samples of the spline);
// with phi a (scaled) even-order cardinal B-spline this is the reference SPME.
//
// Adjoints (R = 2 (F - F_ref) / N the residual of the force-error functional
// L = 1/N sum_i |F_i - F_ref,i|^2, B_a = -sum_i q_i R_i,a W_i the residuals
// spread on the mesh, E_a = IFFT(i 2 pi m_a/L_a G Qh) the ik field):
//   dE/dq_i = sum_k W_i phi_pot,  dE/dr_i = q_i sum_k grad W_i phi_pot,
//   dE/dc   = sum_i q_i sum_k dW_i/dc phi_pot - sum_d sum_m P_d(m) db_d(m)/dc / b_d(m),
//             P_d(m_d) = sum over the other two indices of G |Qh|^2;
//   dL/dq_i = R_i . g_i + sum_k W_i Lam,   g_i = -sum_k W_i grad phi_pot,
//   dL/dr_i = -q_i sum_a R_i,a sum_k grad W_i E_a + q_i sum_k grad W_i Lam,
//   dL/dc   = -sum_i q_i sum_k dW_i/dc (R_i . E(k)) + sum_i q_i sum_k dW_i/dc Lam
//             - 2 sum_d sum_m H_d(m) db_d(m)/dc / b_d(m),
//   Lam     = -Re IFFT(sum_a i 2 pi m_a/L_a G Bh_a),
//   H_d     = marginals of Re(sum_a conj(Bh_a) i 2 pi m_a/L_a Qh) G
// (all inverse transforms unnormalised).
// Candidates go through in batches of up to four, one launch per step.  All
// meshes are real, so the FP64 grid transforms (dft.cu) carry two fields of a
// candidate each where it has two, as the real and imaginary parts: (E_0, E_1)
// and (E_2, kap phi_pot) back, (B_0, B_1) forward -- 9 complex transforms per
// candidate for both functionals where one per mesh takes 14 -- and read and write
// real grids where it has one.  Two candidates
// never share a transform: the rounding of one (or its infinities) would reach
// the other, 4 to 10 times the error in the gradient of the smaller.  Spread
// and gather give a warp to an atom with lanes along its
// stencil rows; the gather leaves the scalar field of the stencil in shared
// memory and contracts it by axis, which yields dE/dq, dE/dr and the
// coefficient sums together (for the force error all three need only the
// scalar Lam - R.E).  Sums over blocks and the marginals are block reductions
// in a fixed order.  Bound: FP64 mesh atomics in the spread, latency and L2
// reads in the gather.  8 candidates of order-6 support, 20,736 charges, 64^3,
// energy and force error with every gradient: 1.8 ms, 11.8 ms when each
// candidate ran by itself with serial finishing sums and atomic marginals.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>
#include "device_common.cuh"

int dft3_grid(double2* data, const int n[3], int sign, int batch, cudaStream_t stream);
int dft3_from_real(const double* re, const double* im, int n_im, double2* out, const int n[3], int batch,
                   cudaStream_t stream);
int dft3_to_real(double2* data, int n_c, double* outr, const int n[3], int batch, cudaStream_t stream);

namespace {

constexpr int HS_MAX_S = 16;      // stencil points per axis (2 ceil(CC))
constexpr int HS_MAX_NBIN = 64;
constexpr int HS_MAX_COEF = 2 * HS_MAX_NBIN;
constexpr int HS_BATCH = 4;  // candidates per launch (two where four would not stay in L2)
constexpr int HS_ATOMS = 4;  // atoms per warp of the spread and the gather
constexpr int HS_COPIES = 8; // of a warp's coefficient sums: four lanes each

struct HsGeom {
  int K[3];
  double L[3];
  double beta, CC, h;
  double kap;  // of E_2 + i kap phi (k_hs_kspace_fwd), a power of two
  int nbin, nk, ncoef, S, half;  // half = ceil(CC)
  long Kt;
};

// cubic Hermite polynomials and their derivatives in t
__device__ __forceinline__ void herm(double t, double v[4], double dv[4]) {
  v[0] = (1 + 2 * t) * (1 - t) * (1 - t);  // h00
  v[1] = t * (1 - t) * (1 - t);            // h10
  v[2] = t * t * (3 - 2 * t);              // h01
  v[3] = t * t * (t - 1);                  // h11
  dv[0] = 6 * t * (t - 1);
  dv[1] = (3 * t - 1) * (t - 1);
  dv[2] = 6 * t * (1 - t);
  dv[3] = t * (3 * t - 2);
}

// knot value / slope of the candidate c (knot 0: 1, 0; knots past nk: 0, 0)
__device__ __forceinline__ double knot_v(const HsGeom& g, const double* c, int j) {
  return j == 0 ? 1.0 : (j <= g.nk ? c[j - 1] : 0.0);
}
__device__ __forceinline__ double knot_d(const HsGeom& g, const double* c, int j) {
  return (j == 0 || j > g.nk) ? 0.0 : c[g.nk + j - 1];
}

// phi(x), phi'(x) and the (at most four) coefficients with a nonzero
// derivative dphi(x)/dc_b: index idx[t] (-1: none) and value dc[t]
struct PhiEval {
  double v, dv;
  int idx[4];
  double dc[4];
};

__device__ __forceinline__ PhiEval phi_eval(const HsGeom& g, const double* c, double x) {
  PhiEval e;
  e.v = 0.0;
  e.dv = 0.0;
  for (int t = 0; t < 4; ++t) { e.idx[t] = -1; e.dc[t] = 0.0; }
  const double ax = fabs(x);
  if (!(ax < g.CC)) return e;
  int j = (int)(ax / g.h);
  if (j >= g.nbin) j = g.nbin - 1;
  const double t = ax / g.h - j;
  double hv[4], hd[4];
  herm(t, hv, hd);
  const double V0 = knot_v(g, c, j), D0 = knot_d(g, c, j), V1 = knot_v(g, c, j + 1), D1 = knot_d(g, c, j + 1);
  const double p = hv[0] * V0 + hv[1] * g.h * D0 + hv[2] * V1 + hv[3] * g.h * D1;
  const double dp = (hd[0] * V0 + hd[1] * g.h * D0 + hd[2] * V1 + hd[3] * g.h * D1) / g.h;
  const double sg = x < 0 ? -1.0 : 1.0;
  e.v = p;
  e.dv = sg * dp;
  // dp/dv_j = h00, dp/dd_j = h10 h, dp/dv_{j+1} = h01, dp/dd_{j+1} = h11 h
  if (j >= 1 && j <= g.nk) { e.idx[0] = j - 1; e.dc[0] = hv[0]; e.idx[1] = g.nk + j - 1; e.dc[1] = hv[1] * g.h; }
  if (j + 1 <= g.nk) { e.idx[2] = j; e.dc[2] = hv[2]; e.idx[3] = g.nk + j; e.dc[3] = hv[3] * g.h; }
  return e;
}

__device__ __forceinline__ int wrap(int k, int K) {
  k %= K;
  return k < 0 ? k + K : k;
}

// warps per block: the larger stencils' scalar field fills shared memory
__host__ __device__ constexpr int hs_warps(int S) { return S <= 8 ? 4 : 1; }

// An atom's stencil in shared memory, evaluated by its warp: the weights phi
// and phi' and the wrapped mesh offsets of the 3 S one-dimensional points.
template <int S>
struct HsStencil {
  double v[3][S], dv[3][S];
  int off[3][S];
};

template <int S>
__device__ __forceinline__ PhiEval hs_entry(const HsGeom& g, const double* c, const double* r, int t, HsStencil<S>& st) {
  const int d = t / S, j = t - d * S;
  double f = r[d] / g.L[d];
  f -= floor(f);
  const double u = g.K[d] * f;
  const int k = (int)floor(u) - g.half + 1 + j;
  const PhiEval e = phi_eval(g, c, u - (double)k);
  st.v[d][j] = e.v;
  st.dv[d][j] = e.dv;
  st.off[d][j] = wrap(k, g.K[d]) * (d == 0 ? g.K[1] * g.K[2] : d == 1 ? g.K[2] : 1);
  return e;
}

__device__ __forceinline__ double hs_block_sum(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += sh[w];
  return s;  // thread 0
}

// b_d(m) and db_d(m)/dc_b: one thread per (axis, m), a candidate per blockIdx.z
__global__ void k_hs_factor(HsGeom g, const double* __restrict__ c, double* __restrict__ bfac,
                            double* __restrict__ dbfac, int Kmax) {
  const int d = blockIdx.y;
  c += (long)blockIdx.z * g.ncoef;
  bfac += (long)blockIdx.z * 3 * Kmax;
  dbfac += (long)blockIdx.z * 3 * g.ncoef * Kmax;
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= g.K[d]) return;
  double b = 0.0;
  double db[HS_MAX_COEF];
  for (int t = 0; t < g.ncoef; ++t) db[t] = 0.0;
  for (int k = -g.half; k <= g.half; ++k) {
    const PhiEval e = phi_eval(g, c, (double)k);
    double s, cs;
    sincospi(2.0 * (double)((long)m * (long)(k < 0 ? k + g.K[d] : k) % g.K[d]) / g.K[d], &s, &cs);
    b += e.v * cs;  // phi even: the imaginary parts cancel
    for (int t = 0; t < 4; ++t)
      if (e.idx[t] >= 0) db[e.idx[t]] += e.dc[t] * cs;
  }
  bfac[d * Kmax + m] = b;
  for (int t = 0; t < g.ncoef; ++t) dbfac[((long)d * g.ncoef + t) * Kmax + m] = db[t];
}

// Spread, a candidate per blockIdx.y, a warp per atom with lanes along its
// stencil rows, onto real meshes (a row of 6 points is then two or three 32-byte
// sectors an instruction; as parts of complex meshes it was four, and the atomics
// are what bounds this).  MODE 0: Q += q_i W_i into grid c of im; MODE 1:
// B_a -= q_i R_i,a W_i, B_0 and B_2 into grids c and nb + c of re, B_1 into im.
template <int S, int MODE>
__global__ void __launch_bounds__(32 * hs_warps(S))
k_hs_spread(HsGeom g, int N, const double* __restrict__ q, const double* __restrict__ r,
            const double* __restrict__ coeffs, const double* __restrict__ R, double* __restrict__ re,
            double* __restrict__ im) {
  constexpr int RP = 32 / S, NR = S * S, NI = (NR + RP - 1) / RP, W = hs_warps(S);
  __shared__ HsStencil<S> sst[W];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, cand = blockIdx.y;
  HsStencil<S>& st = sst[warp];
  const double* c = coeffs + (long)cand * g.ncoef;
  const int k = lane / S, z = lane - k * S;
  double* m0 = (MODE == 0 ? im : re) + (long)cand * g.Kt;
  double* m2 = re + (long)(gridDim.y + cand) * g.Kt;
  double* m1 = im + (long)cand * g.Kt;
  for (int n = 0; n < HS_ATOMS; ++n) {
    const int i = (blockIdx.x * W + warp) * HS_ATOMS + n;
    if (i >= N) return;  // the whole warp
    __syncwarp();
    for (int t = lane; t < 3 * S; t += 32) hs_entry<S>(g, c, r + 3 * (long)i, t, st);
    __syncwarp();
    if (k >= RP) continue;
    double a[3];
    a[0] = q[i];
    if (MODE == 1) {
      const double* Ri = R + 3 * ((long)cand * N + i);
      a[1] = -a[0] * Ri[1];
      a[2] = -a[0] * Ri[2];
      a[0] = -a[0] * Ri[0];
    }
    const double wz = st.v[2][z];
    const int oz = st.off[2][z];
#pragma unroll 4
    for (int j = 0; j < NI; ++j) {
      const int row = j * RP + k;
      if (row >= NR) break;
      const int x = row / S, y = row - x * S;
      const double w = st.v[0][x] * st.v[1][y] * wz;
      if (w == 0.0) continue;
      const int p = st.off[0][x] + st.off[1][y] + oz;
      atomicAdd(m0 + p, a[0] * w);
      if (MODE == 1) {
        atomicAdd(m1 + p, a[1] * w);
        atomicAdd(m2 + p, a[2] * w);
      }
    }
  }
}

struct HsPoint {
  int m[3];
  double k[3];  // 2 pi m_a / L_a, zero at the axis' own Nyquist index
  double G;     // e^{-pi^2 |m|^2 / beta^2} / (pi V |m|^2), without the interpolation factors
  long q;       // index of -m
};

__device__ __forceinline__ HsPoint hs_point(const HsGeom& g, long p) {
  HsPoint h;
  // (a grid has 1,024^3 points at most; 32-bit divisions are several times faster)
  const unsigned t = (unsigned)p / g.K[2], x = t / g.K[1];
  h.m[2] = (int)((unsigned)p - t * g.K[2]);
  h.m[1] = (int)(t - x * g.K[1]);
  h.m[0] = (int)x;
  double m2 = 0.0;
  h.q = 0;
  for (int d = 0; d < 3; ++d) {
    const int md = h.m[d] <= g.K[d] / 2 ? h.m[d] : h.m[d] - g.K[d];
    const double mv = md / g.L[d];
    m2 += mv * mv;
    h.k[d] = (g.K[d] % 2 == 0) && h.m[d] == g.K[d] / 2 ? 0.0 : 2.0 * M_PI * mv;
    h.q = h.q * g.K[d] + (h.m[d] ? g.K[d] - h.m[d] : 0);
  }
  const double V = g.L[0] * g.L[1] * g.L[2];
  h.G = m2 == 0.0 ? 0.0 : exp(-M_PI * M_PI * m2 / (g.beta * g.beta)) / (M_PI * V * m2);
  return h;
}

__device__ __forceinline__ double hs_factor2(const HsPoint& h, const double* bfac, int Kmax) {
  const double b = bfac[h.m[0]] * bfac[Kmax + h.m[1]] * bfac[2 * Kmax + h.m[2]];
  return h.G / (b * b);
}

// spectra of the two real meshes packed as a complex one: z = Z(m), y = Z(-m)
__device__ __forceinline__ double2 hs_first(double2 z, double2 y) { return make_double2(0.5 * (z.x + y.x), 0.5 * (z.y - y.y)); }
__device__ __forceinline__ double2 hs_second(double2 z, double2 y) { return make_double2(0.5 * (z.y + y.y), 0.5 * (y.x - z.x)); }

// k space of the forward pass, a point per thread, nb candidates: with
// g = G Qh, F[c] = transform of E_0 + i E_1 = (i k_0 - k_1) g; energy pass
// (loss = 0) F[nb + c] = E_2 + i kap phi = i (k_2 + kap) g; force error (loss = 1)
// F[nb + c] = E_2 = i k_2 g.  w[c] = G |Qh|^2 (or null).
// A transform rounds to its larger part, and a field is a potential over a
// length: kap, near sqrt(2 pi beta / L) (the ratio of the two in a disordered
// system, whose modes reach from 2 pi / L to about beta), keeps the parts alike
// in any unit of length.  With kap = 1 the forces along z of a box 10^4 times as
// long were off by 3e-12, and dE/dq of one 10^4 times as short by 1e-12.
__global__ void __launch_bounds__(256)
k_hs_kspace_fwd(HsGeom g, int nb, int loss, const double2* __restrict__ Z, const double* __restrict__ bfac, int Kmax,
                double2* __restrict__ F, double* __restrict__ w) {
  const long p = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (p >= g.Kt) return;
  const HsPoint h = hs_point(g, p);
  const double k2 = loss ? h.k[2] : h.k[2] + g.kap;
  for (int c = 0; c < nb; ++c) {
    const double2 Q = Z[c * g.Kt + p];
    const double G = hs_factor2(h, bfac + (long)c * 3 * Kmax, Kmax);
    const double2 a = make_double2(G * Q.x, G * Q.y);
    F[c * g.Kt + p] = make_double2(-h.k[0] * a.y - h.k[1] * a.x, h.k[0] * a.x - h.k[1] * a.y);
    F[(nb + c) * g.Kt + p] = make_double2(-k2 * a.y, k2 * a.x);
    if (w) w[c * g.Kt + p] = G * (Q.x * Q.x + Q.y * Q.y);
  }
}

// k space of the loss adjoint: Lam = -sum_a i k_a G Bh_a in place of Bh_2,
// w[c] = Re(sum_a conj(Bh_a) i k_a Qh) G
__global__ void __launch_bounds__(256)
k_hs_kspace_adj(HsGeom g, int nb, const double2* __restrict__ Z, const double2* __restrict__ Y, double2* Y2,
                const double* __restrict__ bfac, int Kmax, double* __restrict__ w) {
  const long p = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (p >= g.Kt) return;
  const HsPoint h = hs_point(g, p);
  for (int c = 0; c < nb; ++c) {
    const long o = c * g.Kt;
    const double2 Q = Z[o + p], zb = Y[o + p], yb = Y[o + h.q];
    const double2 b[3] = {hs_first(zb, yb), hs_second(zb, yb), Y2[o + p]};
    const double G = hs_factor2(h, bfac + (long)c * 3 * Kmax, Kmax);
    double2 a = make_double2(0.0, 0.0);
    double v = 0.0;
    for (int d = 0; d < 3; ++d) {
      a.x += h.k[d] * G * b[d].y;  // -i k G b
      a.y -= h.k[d] * G * b[d].x;
      v += h.k[d] * (-b[d].x * Q.y + b[d].y * Q.x);  // Re(conj(b) i k Q)
    }
    if (w) w[o + p] = v * G;
    Y2[o + p] = a;
  }
}

// marginals of w[c]: block (m, d, c) sums the plane m_d = m
__global__ void __launch_bounds__(256)
k_hs_marginal(HsGeom g, const double* __restrict__ w, int Kmax, double* __restrict__ marg) {
  __shared__ double sh[8];
  const int m = blockIdx.x, d = blockIdx.y, c = blockIdx.z;
  if (m >= g.K[d]) return;
  const double* wc = w + c * g.Kt;
  const int n1 = d == 0 ? g.K[1] : g.K[0], n2 = d == 2 ? g.K[1] : g.K[2];  // the other two axes
  const long s0 = d == 0 ? (long)g.K[1] * g.K[2] : d == 1 ? g.K[2] : 1;   // strides
  const long s1 = d == 0 ? g.K[2] : (long)g.K[1] * g.K[2], s2 = d == 2 ? g.K[2] : 1;
  double v = 0.0;
  for (int t = threadIdx.x; t < n1 * n2; t += 256) v += wc[m * s0 + (t / n2) * s1 + (t % n2) * s2];
  v = hs_block_sum(v, sh);
  if (threadIdx.x == 0) marg[(c * 3 + d) * (long)Kmax + m] = v;
}

struct HsOut {
  double *F, *dq, *dr;  // [nb][N][3], [nb][N], [nb][N][3]; null where not asked
  double* cpart;        // [nb][blocks][ncoef]
};

// Gather, a candidate per blockIdx.y, a warp per atom.
//   MODE 0 (energy): f1 = (E_0, E_1), f2 = (E_2, kap phi): F_i, dE/dq_i, dE/dr_i and
//     the coefficient partials of the scalar phi
//   MODE 1 (loss): E_2 from the real grid e2: F_i, the residual R_i = 2 (F_i - Fref_i) / N
//     and the block's part of the loss
//   MODE 2 (loss adjoint): dL/dq_i, dL/dr_i and the coefficient partials of the
//     scalar Lam - R_i.E (dL/dr_i = q_i sum grad W_i (Lam - R_i.E), and so for dq, dc)
// Per atom the lanes read the field along the stencil rows and leave the scalar
// s(a, b, c) in shared memory; u(a, b) = sum_c w s, then lane (d, j) forms
// T[d][j] = sum over the other two axes of w w s, whose products with the
// weights, their derivatives and their coefficient derivatives are the results.
template <int S, int MODE>
__global__ void __launch_bounds__(32 * hs_warps(S))
k_hs_gather(HsGeom g, int N, const double* __restrict__ q, const double* __restrict__ r,
            const double* __restrict__ coeffs, const double2* __restrict__ f1, const double2* __restrict__ f2,
            const double* __restrict__ e2, const double* __restrict__ lam, const double* __restrict__ fref, double* __restrict__ R,
            double* __restrict__ lpart, HsOut out) {
  constexpr int RP = 32 / S, NR = S * S, NI = (NR + RP - 1) / RP, W = hs_warps(S), LD = S + 1;
  __shared__ HsStencil<S> sst[W];
  __shared__ double ss[W][MODE == 1 ? 1 : NR * LD], su[W][MODE == 1 ? 1 : NR], sp[W][MODE == 1 ? 1 : 32 + 4 * S];
  // the four coefficient terms of each one-dimensional point, and a warp's sums of
  // them, HS_COPIES copies of [ncoef]
  __shared__ double sv[W][MODE == 1 ? 1 : 12 * S], sl[W];
  __shared__ int si[W][MODE == 1 ? 1 : 12 * S];
  extern __shared__ double hs_csum[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, cand = blockIdx.y;
  if (MODE != 1) {
    if (out.cpart)
      for (int t = threadIdx.x; t < W * HS_COPIES * g.ncoef; t += blockDim.x) hs_csum[t] = 0.0;
    __syncthreads();
  }
  HsStencil<S>& st = sst[warp];
  const double* c = coeffs + (long)cand * g.ncoef;
  const int k = lane / S, z = lane - k * S;
  const double2* e01 = f1 + (long)cand * g.Kt;
  const double2* e2p = f2 + (long)cand * g.Kt;
  const double *e2r = e2 + (long)cand * g.Kt, *lm = lam + (long)cand * g.Kt;
  const double kinv = 1.0 / g.kap;  // exact
  double loss = 0.0;
  for (int n = 0; n < HS_ATOMS; ++n) {
    const int i = (blockIdx.x * W + warp) * HS_ATOMS + n;
    if (i >= N) break;  // the whole warp
    __syncwarp();
    PhiEval e;
    if (lane < 3 * S) e = hs_entry<S>(g, c, r + 3 * (long)i, lane, st);
    if (3 * S > 32 && lane + 32 < 3 * S) hs_entry<S>(g, c, r + 3 * (long)i, lane + 32, st);
    __syncwarp();
    const double qi = q[i];
    const long ia = (long)cand * N + i;
    double Ri[3] = {0.0, 0.0, 0.0};
    if (MODE == 2)
      for (int d = 0; d < 3; ++d) Ri[d] = R[3 * ia + d];
    double Ef[3] = {0.0, 0.0, 0.0}, t2 = 0.0;
    if (k < RP) {
      const int oz = st.off[2][z];
#pragma unroll 4
      for (int j = 0; j < NI; ++j) {
        const int row = j * RP + k;
        if (row >= NR) break;
        const int x = row / S, y = row - x * S, p = st.off[0][x] + st.off[1][y] + oz;
        const double wxy = st.v[0][x] * st.v[1][y];
        const double2 a = e01[p], b = MODE == 0 ? e2p[p] : make_double2(e2r[p], 0.0);
        if (MODE == 2) {
          const double s = lm[p] - (Ri[0] * a.x + Ri[1] * a.y + Ri[2] * b.x);
          ss[warp][row * LD + z] = s;
          t2 += wxy * s;
        } else {
          Ef[0] += wxy * a.x;
          Ef[1] += wxy * a.y;
          Ef[2] += wxy * b.x;
          if (MODE == 0) {
            const double s = b.y * kinv;
            ss[warp][row * LD + z] = s;
            t2 += wxy * s;
          }
        }
      }
      if (MODE != 2) {
        const double wz = st.v[2][z];
        for (int d = 0; d < 3; ++d) Ef[d] *= wz;
      }
    }
    if (MODE != 2) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        for (int d = 0; d < 3; ++d) Ef[d] += __shfl_xor_sync(0xffffffffu, Ef[d], o);
      if (lane < 3) {
        const double F = -qi * (lane == 0 ? Ef[0] : lane == 1 ? Ef[1] : Ef[2]);
        if (out.F) out.F[3 * ia + lane] = F;
        if (MODE == 1) {
          const double dF = F - fref[3 * (long)i + lane];
          R[3 * ia + lane] = 2.0 * dF / N;
          loss += dF * dF / N;
        }
      }
    }
    if (MODE == 1) continue;
    sp[warp][lane] = t2;
    __syncwarp();
    for (int row = lane; row < NR; row += 32) {
      double u = 0.0;
#pragma unroll
      for (int j = 0; j < S; ++j) u += st.v[2][j] * ss[warp][row * LD + j];
      su[warp][row] = u;
    }
    __syncwarp();
    for (int t = lane; t < 3 * S; t += 32) {
      const int d = t / S, j = t - d * S;
      double T = 0.0;
      if (d == 0) {
#pragma unroll
        for (int b = 0; b < S; ++b) T += st.v[1][b] * su[warp][j * S + b];
      } else if (d == 1) {
#pragma unroll
        for (int a = 0; a < S; ++a) T += st.v[0][a] * su[warp][a * S + j];
      } else {
#pragma unroll
        for (int a = 0; a < RP; ++a) T += sp[warp][a * S + j];
      }
      sp[warp][32 + t] = st.dv[d][j] * T;
      if (d == 0) sp[warp][32 + 3 * S + j] = st.v[0][j] * T;
      if (out.cpart) {
        // which coefficients the weight depends on
        const double tv = qi * T;
        if (t >= 32) {
          HsStencil<S>& same = st;  // re-evaluated: the same values are stored again
          e = hs_entry<S>(g, c, r + 3 * (long)i, t, same);
        }
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          sv[warp][4 * t + b] = tv * e.dc[b];
          si[warp][4 * t + b] = e.idx[b];
        }
      }
    }
    __syncwarp();
    if (out.cpart) {
      // four lanes to a point, whose four coefficients differ, eight points at a
      // time, each into its own copy: no two lanes meet (shared FP64 atomics, as
      // before, retry where they do: 161 us a batch of four then, 145 now)
      double* acc = hs_csum + (warp * HS_COPIES + (lane >> 2)) * g.ncoef;
#pragma unroll
      for (int t0 = 0; t0 < 12 * S; t0 += 32) {
        const int t = t0 + lane;
        if (t < 12 * S && si[warp][t] >= 0) acc[si[warp][t]] += sv[warp][t];
        __syncwarp();
      }
    }
    if (lane < 4) {
      double v = 0.0;
#pragma unroll
      for (int j = 0; j < S; ++j) v += sp[warp][32 + lane * S + j];
      if (lane < 3) {
        if (out.dr) out.dr[3 * ia + lane] = qi * v * g.K[lane] / g.L[lane];
      } else if (out.dq) {
        out.dq[ia] = v;
      }
    }
  }
  if (MODE == 1) {
    for (int o = 2; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
    if (lane == 0) sl[warp] = loss;
    __syncthreads();
    if (threadIdx.x == 0) {
      double v = 0.0;
      for (int w = 0; w < W; ++w) v += sl[w];
      lpart[(long)cand * gridDim.x + blockIdx.x] = v;
    }
  } else if (out.cpart) {
    __syncthreads();
    for (int t = threadIdx.x; t < g.ncoef; t += blockDim.x) {
      double v = 0.0;
      for (int w = 0; w < W * HS_COPIES; ++w) v += hs_csum[w * g.ncoef + t];
      out.cpart[((long)cand * gridDim.x + blockIdx.x) * g.ncoef + t] = v;
    }
  }
}

// Block (t, c): coefficient t's gradient of candidate c, the gather's block
// partials plus the interpolation factor term -wfac sum_d sum_m marg_d(m) db_d(m)/dc / b_d(m);
// t = ncoef: the energy, half the sum of a marginal, or the loss from its parts
__global__ void __launch_bounds__(128)
k_hs_finish(HsGeom g, const double* __restrict__ cpart, int nblk, const double* __restrict__ marg,
            const double* __restrict__ bfac, const double* __restrict__ dbfac, int Kmax, double wfac,
            double* __restrict__ out, const double* __restrict__ lpart, double* __restrict__ scalar) {
  __shared__ double sh[4];
  const int t = blockIdx.x, c = blockIdx.y;
  double s = 0.0;
  if (t < g.ncoef) {
    if (!out) return;
    for (int b = threadIdx.x; b < nblk; b += 128) s += cpart[((long)c * nblk + b) * g.ncoef + t];
    double f = 0.0;
    for (int d = 0; d < 3; ++d)
      for (int m = threadIdx.x; m < g.K[d]; m += 128)
        f += marg[(c * 3 + d) * (long)Kmax + m] * dbfac[(((long)c * 3 + d) * g.ncoef + t) * Kmax + m] /
             bfac[(c * 3 + d) * (long)Kmax + m];
    s = hs_block_sum(s - wfac * f, sh);
    if (threadIdx.x == 0) out[(long)c * g.ncoef + t] = s;
    return;
  }
  if (!scalar) return;
  if (lpart)
    for (int b = threadIdx.x; b < nblk; b += 128) s += lpart[(long)c * nblk + b];
  else
    for (int m = threadIdx.x; m < g.K[0]; m += 128) s += 0.5 * marg[c * 3 * (long)Kmax + m];
  s = hs_block_sum(s, sh);
  if (threadIdx.x == 0) scalar[c] = s;
}

}  // namespace

struct md_hspme {
  int device = 0;
  int N = 0;
  HsGeom g;
  int Kmax = 0;
  int B = HS_BATCH;          // candidates per batch
  int nab = 0;               // blocks of the spread and the gather
  double2* Z = nullptr;      // [B][Kt] charge meshes, transformed in place
  double2* F = nullptr;      // [2B][Kt] fields; B_0 and B_2 of the loss as [2B][Kt] real grids in its second half
  double2* Y = nullptr;      // [2B][Kt] transforms of the residual meshes, then Lam in place of B_2
  double* e2 = nullptr;      // [B][Kt] the loss's E_2
  double* w = nullptr;       // [B][Kt] the spread Q or B_1, then the summand of the marginals, then the loss's Lam
  double* bfac = nullptr;    // [B][3][Kmax]
  double* dbfac = nullptr;   // [B][3][ncoef][Kmax]
  double* marg = nullptr;    // [B][3][Kmax]
  double* cpart = nullptr;   // [B][nab][ncoef]
  double* lpart = nullptr;   // [B][nab]
  double* R = nullptr;       // [B][N][3] residual weights
  void* slab = nullptr;      // the memory of all of these
};

static void hs_free(md_hspme* h) {
  if (h->slab) cudaFree(h->slab);
  h->slab = nullptr;
}

// Workspace for batches of B candidates, from one allocation: an object per mesh
// and box is made in a loop over them, and eleven of them were most of its cost.
static bool hs_alloc(md_hspme* h, long B) {
  const size_t Kt = h->g.Kt, nco = std::max(h->g.ncoef, 1), b = B;
  const struct { void** p; size_t doubles; } part[] = {
      {(void**)&h->Z, 2 * b * Kt},          {(void**)&h->F, 4 * b * Kt},
      {(void**)&h->Y, 4 * b * Kt},          {(void**)&h->e2, b * Kt},
      {(void**)&h->w, b * Kt},              {(void**)&h->bfac, b * 3 * h->Kmax},
      {(void**)&h->dbfac, b * 3 * nco * h->Kmax}, {(void**)&h->marg, b * 3 * h->Kmax},
      {(void**)&h->cpart, b * h->nab * nco}, {(void**)&h->lpart, b * h->nab},
      {(void**)&h->R, b * 3 * h->N}};
  size_t bytes = 0;
  for (const auto& q : part) bytes += (q.doubles * sizeof(double) + 255) & ~(size_t)255;
  if (cudaMalloc(&h->slab, bytes) != cudaSuccess) {
    h->slab = nullptr;
    return false;
  }
  char* at = (char*)h->slab;
  for (const auto& q : part) {
    *q.p = at;
    at += (q.doubles * sizeof(double) + 255) & ~(size_t)255;
  }
  return true;
}

// stencil widths 2 ceil(CC)
#define HS_WIDTHS(X) X(2) X(4) X(6) X(8) X(10) X(12) X(14) X(16)

static int hs_gather_prepare(int S);

extern "C" int md_hspme_create(md_hspme** out, int natoms, const int K[3], const double L[3], double beta, double CC,
                               int nbin, int bound0, int device) {
  if (!out || natoms < 1 || !K || !L || !(beta > 0) || !(CC > 0) || nbin < 1 || nbin > HS_MAX_NBIN) {
    md_set_error("md_hspme_create: bad arguments");
    return MD_ERR_BADARG;
  }
  const int half = (int)ceil(CC - 1e-12);
  if (2 * half > HS_MAX_S) { md_set_error("md_hspme_create: support CC %g wider than %d grid points", CC, HS_MAX_S); return MD_ERR_BADARG; }
  for (int d = 0; d < 3; ++d)
    if (K[d] < 2 * half + 1 || K[d] > 1024 || !(L[d] > 0)) {
      md_set_error("md_hspme_create: mesh %d or box %g out of range on axis %d", K[d], L[d], d);
      return MD_ERR_BADARG;
    }
  MD_CUDA(cudaSetDevice(device));
  if (int r = hs_gather_prepare(2 * half)) return r;
  md_hspme* h = new md_hspme();
  h->device = device;
  h->N = natoms;
  HsGeom& g = h->g;
  for (int d = 0; d < 3; ++d) { g.K[d] = K[d]; g.L[d] = L[d]; }
  g.beta = beta;
  g.CC = CC;
  g.nbin = nbin;
  g.h = CC / nbin;
  g.nk = bound0 ? nbin - 1 : nbin;
  g.ncoef = 2 * g.nk;
  g.half = half;
  g.S = 2 * half;
  g.Kt = (long)K[0] * K[1] * K[2];
  g.kap = exp2(rint(0.5 * log2(2.0 * M_PI * beta / cbrt(L[0] * L[1] * L[2]))));
  h->Kmax = std::max(K[0], std::max(K[1], K[2]));
  const int per = HS_ATOMS * hs_warps(g.S);
  h->nab = (natoms + per - 1) / per;
  // the meshes of a batch (96 bytes per point and candidate) stay in the 126 MB
  // L2 with four candidates up to 64^3; fewer where memory holds no more
  h->B = g.Kt * 96 * HS_BATCH <= (96L << 20) ? HS_BATCH : 2;
  while (!hs_alloc(h, h->B)) {
    const cudaError_t e = cudaGetLastError();
    hs_free(h);
    if (e != cudaErrorMemoryAllocation || h->B == 1) {
      delete h;
      return md_cuda_fail(e, "md_hspme_create");
    }
    h->B /= 2;
  }
  *out = h;
  return MD_OK;
}

extern "C" int md_hspme_destroy(md_hspme* h) {
  if (!h) return MD_OK;
  cudaSetDevice(h->device);
  hs_free(h);
  delete h;
  return MD_OK;
}

extern "C" int md_hspme_num_coeffs(md_hspme* h, int* out) {
  if (!h || !out) return MD_ERR_BADARG;
  *out = h->g.ncoef;
  return MD_OK;
}

template <int MODE>
static int hs_spread(md_hspme* h, int nb, const double* q, const double* r, const double* c, cudaStream_t s) {
  double* re = reinterpret_cast<double*>(h->F + (long)nb * h->g.Kt);
  switch (h->g.S) {
#define HS_CASE(W)                                                                                               \
  case W:                                                                                                        \
    k_hs_spread<W, MODE><<<dim3(h->nab, nb), 32 * hs_warps(W), 0, s>>>(h->g, h->N, q, r, c, h->R, re, h->w);       \
    break;
    HS_WIDTHS(HS_CASE)
#undef HS_CASE
  }
  MD_CHECK_LAUNCH("hspme spread");
  return MD_OK;
}

// a block's coefficient sums
static constexpr size_t hs_csum_bytes(int S, int ncoef) { return sizeof(double) * hs_warps(S) * HS_COPIES * ncoef; }

// The gathers may take the sums of any coefficient count: the limit belongs to
// the kernel, not to a handle, so one of fewer coefficients must not lower it
// between another's setting and launch.
static int hs_gather_prepare(int S) {
  const void* f[2] = {nullptr, nullptr};
  switch (S) {
#define HS_CASE(W)                            \
  case W:                                     \
    f[0] = (const void*)k_hs_gather<W, 0>;    \
    f[1] = (const void*)k_hs_gather<W, 2>;    \
    break;
    HS_WIDTHS(HS_CASE)
#undef HS_CASE
  }
  for (const void* k : f) {
    if (!k) continue;  // a support of no width has no stencil
    MD_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hs_csum_bytes(S, HS_MAX_COEF)));
  }
  return MD_OK;
}

template <int MODE>
static int hs_gather(md_hspme* h, int nb, const double* q, const double* r, const double* c, const double* fref,
                     const HsOut& out, cudaStream_t s) {
  const double2* f2 = h->F + (long)nb * h->g.Kt;
  switch (h->g.S) {
#define HS_CASE(W)                                                                                               \
  case W:                                                                                                        \
    k_hs_gather<W, MODE><<<dim3(h->nab, nb), 32 * hs_warps(W), out.cpart ? hs_csum_bytes(W, h->g.ncoef) : 0, s>>>( \
        h->g, h->N, q, r, c, h->F, f2, h->e2, h->w, fref, h->R, h->lpart, out);                                    \
    break;
    HS_WIDTHS(HS_CASE)
#undef HS_CASE
  }
  MD_CHECK_LAUNCH("hspme gather");
  return MD_OK;
}

static int hs_marginals(md_hspme* h, int nb, int axes, cudaStream_t s) {
  k_hs_marginal<<<dim3(axes == 1 ? h->g.K[0] : h->Kmax, axes, nb), 256, 0, s>>>(h->g, h->w, h->Kmax, h->marg);
  MD_CHECK_LAUNCH("hspme marginals");
  return MD_OK;
}

// forward pass of nb candidates: factors, spread, transform, k space and the
// inverse transforms of the fields (loss: as the force error wants them)
static int hs_forward(md_hspme* h, int nb, const double* q, const double* r, const double* c, bool loss, bool want_w,
                      cudaStream_t s) {
  HsGeom& g = h->g;
  k_hs_factor<<<dim3((h->Kmax + 63) / 64, 3, nb), 64, 0, s>>>(g, c, h->bfac, h->dbfac, h->Kmax);
  MD_CHECK_LAUNCH("hspme factor");
  MD_CUDA(cudaMemsetAsync(h->w, 0, sizeof(double) * nb * g.Kt, s));
  if (int e = hs_spread<0>(h, nb, q, r, c, s)) return e;
  if (int e = dft3_from_real(h->w, nullptr, 0, h->Z, g.K, nb, s)) return e;
  k_hs_kspace_fwd<<<(unsigned)((g.Kt + 255) / 256), 256, 0, s>>>(g, nb, loss ? 1 : 0, h->Z, h->bfac, h->Kmax, h->F,
                                                                 want_w ? h->w : nullptr);
  MD_CHECK_LAUNCH("hspme kspace");
  return loss ? dft3_to_real(h->F, nb, h->e2, g.K, 2 * nb, s) : dft3_grid(h->F, g.K, +1, 2 * nb, s);
}

extern "C" int md_hspme_energy(md_hspme* h, const double* q, const double* r, const double* coeffs, int C,
                               double* energy, double* forces, double* dE_dq, double* dE_dr, double* dE_dc,
                               void* stream) {
  if (!h || !q || !r || !coeffs || C < 1 || !energy) { md_set_error("md_hspme_energy: bad arguments"); return MD_ERR_BADARG; }
  MD_CUDA(cudaSetDevice(h->device));
  cudaStream_t s = (cudaStream_t)stream;
  HsGeom& g = h->g;
  const long N = h->N;
  for (int b = 0; b < C; b += h->B) {
    const int nb = std::min(h->B, C - b);
    const double* c = coeffs + (long)b * g.ncoef;
    if (int e = hs_forward(h, nb, q, r, c, false, true, s)) return e;
    if (int e = hs_marginals(h, nb, dE_dc ? 3 : 1, s)) return e;
    if (forces || dE_dq || dE_dr || dE_dc) {
      HsOut o = {forces ? forces + 3 * N * b : nullptr, dE_dq ? dE_dq + N * b : nullptr,
                 dE_dr ? dE_dr + 3 * N * b : nullptr, dE_dc ? h->cpart : nullptr};
      if (int e = hs_gather<0>(h, nb, q, r, c, nullptr, o, s)) return e;
    }
    // the factor term of dE/dc: 1/2 sum G|Qh|^2 (-2 db/b) = -sum P db / b
    k_hs_finish<<<dim3(g.ncoef + 1, nb), 128, 0, s>>>(g, h->cpart, h->nab, h->marg, h->bfac, h->dbfac, h->Kmax, 1.0,
                                                      dE_dc ? dE_dc + (long)g.ncoef * b : nullptr, nullptr, energy + b);
    MD_CHECK_LAUNCH("hspme finish");
  }
  return MD_OK;
}

extern "C" int md_hspme_force_error(md_hspme* h, const double* q, const double* r, const double* coeffs, int C,
                                    const double* fref, double* loss, double* dL_dq, double* dL_dr, double* dL_dc,
                                    void* stream) {
  if (!h || !q || !r || !coeffs || C < 1 || !fref || !loss) {
    md_set_error("md_hspme_force_error: bad arguments");
    return MD_ERR_BADARG;
  }
  MD_CUDA(cudaSetDevice(h->device));
  cudaStream_t s = (cudaStream_t)stream;
  HsGeom& g = h->g;
  const long N = h->N, Kt = g.Kt;
  const bool grads = dL_dq || dL_dr || dL_dc;
  for (int b = 0; b < C; b += h->B) {
    const int nb = std::min(h->B, C - b);
    const double* c = coeffs + (long)b * g.ncoef;
    if (int e = hs_forward(h, nb, q, r, c, true, false, s)) return e;
    if (int e = hs_gather<1>(h, nb, q, r, c, fref, HsOut{}, s)) return e;
    if (grads) {
      // adjoint: residuals spread, transformed, Lam and the factor marginals
      double2 *Y2 = h->Y + nb * Kt, *B02 = h->F + nb * Kt;
      MD_CUDA(cudaMemsetAsync(B02, 0, sizeof(double) * 2 * nb * Kt, s));
      MD_CUDA(cudaMemsetAsync(h->w, 0, sizeof(double) * nb * Kt, s));
      if (int e = hs_spread<1>(h, nb, q, r, c, s)) return e;
      if (int e = dft3_from_real((const double*)B02, h->w, nb, h->Y, g.K, 2 * nb, s)) return e;
      k_hs_kspace_adj<<<(unsigned)((Kt + 255) / 256), 256, 0, s>>>(g, nb, h->Z, h->Y, Y2, h->bfac, h->Kmax,
                                                                   dL_dc ? h->w : nullptr);
      MD_CHECK_LAUNCH("hspme adjoint kspace");
      if (dL_dc)
        if (int e = hs_marginals(h, nb, 3, s)) return e;
      if (int e = dft3_to_real(Y2, 0, h->w, g.K, nb, s)) return e;
      HsOut o = {nullptr, dL_dq ? dL_dq + N * b : nullptr, dL_dr ? dL_dr + 3 * N * b : nullptr,
                 dL_dc ? h->cpart : nullptr};
      if (int e = hs_gather<2>(h, nb, q, r, c, nullptr, o, s)) return e;
    }
    // factor term of dL/dc through G: sum_m H(m) dG/dc = -2 sum_d sum_m H_d db/b
    k_hs_finish<<<dim3(g.ncoef + 1, nb), 128, 0, s>>>(g, h->cpart, h->nab, h->marg, h->bfac, h->dbfac, h->Kmax, 2.0,
                                                      dL_dc ? dL_dc + (long)g.ncoef * b : nullptr, h->lpart, loss + b);
    MD_CHECK_LAUNCH("hspme finish");
  }
  return MD_OK;
}

// Exact reciprocal Ewald sum in FP64.
// Reference: ElectrostaticInteraction_rec_ES (longRange.hetero/profile.test/
// template/tools/real.error/src/EleRecES.cpp:49-144):
//   S(m) = sum_i q_i exp(2 pi i m.r_i) for every m of the |m_d| <= K_d/2 box
//   (calPotential), E = sum_m ex(m) |S|^2 / (2 pi V), ex = e^{-pi^2 m^2/beta^2} / m^2,
//   F_i = sum_m (2/V) ex(m) (S_r q_i sin - S_i q_i cos) m (applyInteraction).
//
// The phase factors by axis, e^{2 pi i m.r} = e_0(m_0) e_1(m_1) e_2(m_2), so
// both sums are contractions over tables of sum_d (K_d/2 + 1) values per atom
// instead of a sincos per (mode, atom).  A "row" is a pair (m_0 >= 0, m_1),
// a "column" an m_2 >= 0: the modes -m_0 follow from S(-m) = conj S(m), and
// +-m_2 share the four products of A = q e_0 e_1 with e_2 = c + i s:
//   S(+-) = (sum A_r c -+ sum A_i s) + i (+-sum A_r s + sum A_i c).
// Bound: FP64 arithmetic, 4 FMA per (row, column, atom) for S and 8 for the
// forces.  4,000 charges and 33^3 modes: 460 M FMA, 25 us at 64 FMA per SM
// and clock; this takes 0.18 ms (S 93 us, forces 53); one thread per atom walking
// every mode with a sincos and an exp each, as before, 25.8 ms (32 blocks on the
// chip and a serial chain).
#include <algorithm>
#include <cmath>
#include "device_common.cuh"

namespace {

constexpr int EW_CHUNK = 65536;  // atoms per pass: bounds the tables (16 B x sum_d (K_d/2 + 1) each)
constexpr int EW_T = 16;         // rows and columns of an S tile
constexpr int EW_A = 32;         // atoms staged at a time
constexpr int EW_ROWS = 8;       // rows a thread of the force kernel holds in registers
constexpr int EW_COLS = 64;      // columns of their coefficients staged at a time

struct EwGeom {
  int M[3];
  int nrow, ncol, n1;  // n1 = 2 M_1 + 1 rows per m_0
};

// e_d(m) = exp(2 pi i m x_d / L_d), m = 0..M_d, of the chunk's atoms; the
// product m x_d / L_d is reduced to its fraction exactly (fma) before sincospi
__global__ void __launch_bounds__(256)
k_ew_tables(int N, int i0, int nc, const double4a* __restrict__ pos, const float4* __restrict__ posf, EwGeom g,
            const DevState* __restrict__ st, double2* __restrict__ tab) {
  const int k = blockIdx.y * blockDim.x + threadIdx.x;
  int m = blockIdx.x, d = 0;
  if (k >= nc) return;
  while (m > g.M[d]) { m -= g.M[d] + 1; ++d; }
  const int i = i0 + k;
  double x;
  if (pos) x = d == 0 ? pos[i].x : d == 1 ? pos[i].y : pos[i].z;
  else x = d == 0 ? posf[i].x : d == 1 ? posf[i].y : posf[i].z;
  const double u = x * st->Li[d], p = m * u;
  const double f = (p - rint(p)) + fma((double)m, u, -p);
  double s, c;
  sincospi(2.0 * f, &s, &c);
  tab[(size_t)blockIdx.x * nc + k] = make_double2(c, s);
}

// One 16 x 16 tile of (row, column) sums over this block's share of the
// chunk's atoms; 64 threads with a 2 x 2 micro-tile and four sums per entry.
// The atoms are split over blockIdx.z so that a few tiles still fill the
// chip; the parts are added up in a fixed order by k_ew_coef.
__global__ void __launch_bounds__(64)
k_ew_sk(int i0, int nc, const double4a* __restrict__ pos, const float4* __restrict__ posf, EwGeom g,
        const double2* __restrict__ tab, int per, int accumulate, double* __restrict__ part) {
  __shared__ double2 A[EW_A][EW_T], B[EW_A][EW_T];
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
  const int ct = (g.ncol + EW_T - 1) / EW_T;  // tiles along blockIdx.x, the one index that reaches any count
  const int r0 = (int)(blockIdx.x / ct) * EW_T, c0 = (int)(blockIdx.x % ct) * EW_T;
  const int a0 = blockIdx.z * per, a1 = min(nc, a0 + per);
  const double2* e0 = tab;
  const double2* e1 = e0 + (size_t)(g.M[0] + 1) * nc;
  const double2* e2 = e1 + (size_t)(g.M[1] + 1) * nc;
  double s[2][2][4] = {};
  for (int a = a0; a < a1; a += EW_A) {
    __syncthreads();
    for (int t = threadIdx.x; t < EW_A * EW_T; t += 64) {
      const int at = t % EW_A, w = t / EW_A, k = a + at;  // lanes along the atoms: coalesced table reads
      double2 va = make_double2(0.0, 0.0), vb = va;
      if (k < a1) {
        const int r = r0 + w, c = c0 + w;
        if (r < g.nrow) {
          const int m0 = r / g.n1, m1 = r - m0 * g.n1 - g.M[1];
          const double2 x = e0[(size_t)m0 * nc + k];
          double2 y = e1[(size_t)abs(m1) * nc + k];
          if (m1 < 0) y.y = -y.y;
          const double q = pos ? pos[i0 + k].w : (double)posf[i0 + k].w;
          va = make_double2(q * (x.x * y.x - x.y * y.y), q * (x.x * y.y + x.y * y.x));
        }
        if (c < g.ncol) vb = e2[(size_t)c * nc + k];
      }
      A[at][w] = va;
      B[at][w] = vb;
    }
    __syncthreads();
#pragma unroll 4
    for (int at = 0; at < EW_A; ++at) {
      const double2 x[2] = {A[at][ty], A[at][ty + 8]}, y[2] = {B[at][tx], B[at][tx + 8]};
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          s[i][j][0] = fma(x[i].x, y[j].x, s[i][j][0]);
          s[i][j][1] = fma(x[i].y, y[j].y, s[i][j][1]);
          s[i][j][2] = fma(x[i].x, y[j].y, s[i][j][2]);
          s[i][j][3] = fma(x[i].y, y[j].x, s[i][j][3]);
        }
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int r = r0 + ty + 8 * i, c = c0 + tx + 8 * j;
      if (r >= g.nrow || c >= g.ncol) continue;
      double* p = part + (((size_t)blockIdx.z * g.nrow + r) * g.ncol + c) * 4;
#pragma unroll
      for (int q = 0; q < 4; ++q) p[q] = accumulate ? p[q] + s[i][j][q] : s[i][j][q];
    }
}

// S of each (row, +-column), the energy, and the force coefficients
// D(m) = w (2/V) ex(m) S(m) (w = 2 for m_0 > 0, whose mirror modes are not
// enumerated) as P = D(+) + D(-), M = D(+) - D(-)
__global__ void __launch_bounds__(256)
k_ew_coef(EwGeom g, double beta, int nsplit, const double* __restrict__ part, DevState* st, double4a* __restrict__ coef,
          double* partials, double* energy) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  double e[1] = {0.0};
  if (t < g.nrow * g.ncol) {
    const int r = t / g.ncol, m2 = t - r * g.ncol, m0 = r / g.n1, m1 = r - m0 * g.n1 - g.M[1];
    double s[4] = {0, 0, 0, 0};
    for (int z = 0; z < nsplit; ++z)
      for (int q = 0; q < 4; ++q) s[q] += part[((size_t)z * g.nrow * g.ncol + t) * 4 + q];
    const double2 sp = make_double2(s[0] - s[1], s[2] + s[3]), sm = make_double2(s[0] + s[1], s[3] - s[2]);
    const double V = st->L[0] * st->L[1] * st->L[2], sc = M_PI * M_PI / (beta * beta);
    const double x = m0 * st->Li[0], y = m1 * st->Li[1], z = m2 * st->Li[2], mm = x * x + y * y + z * z;
    const double ex = mm != 0.0 ? exp(-sc * mm) / mm : 0.0, w = m0 > 0 ? 2.0 : 1.0, f = w * 2.0 / V * ex;
    e[0] = w * ex * (sp.x * sp.x + sp.y * sp.y) / (2.0 * M_PI * V);
    double4a c = {f * sp.x, f * sp.y, f * sp.x, f * sp.y};
    if (m2 > 0) {
      e[0] += w * ex * (sm.x * sm.x + sm.y * sm.y) / (2.0 * M_PI * V);
      c = double4a{f * (sp.x + sm.x), f * (sp.y + sm.y), f * (sp.x - sm.x), f * (sp.y - sm.y)};
    }
    coef[t] = c;
  }
  block_reduce_finish<1>(e, partials, &st->red_counter[RED_MISC], energy, true);
}

// Forces of one thread's atom over this block's rows, EW_ROWS at a time: per
// column the atom's e_2 is read once and meets the rows' coefficients from
// shared memory (a broadcast), T0 = sum_{+-m_2} conj(D) e_2 and
// T1 = sum m_2 conj(D) e_2; then F += Im(q e_0 e_1 (m_0 T0, m_1 T0, T1)).
// Rows are split over blockIdx.y; the parts are added in order by k_ew_sum.
__global__ void __launch_bounds__(128)
k_ew_force(int i0, int nc, const double4a* __restrict__ pos, const float4* __restrict__ posf, EwGeom g,
           const double2* __restrict__ tab, const double4a* __restrict__ coef, int rows_per,
           const DevState* __restrict__ st, double* __restrict__ fpart) {
  __shared__ double4a D[EW_COLS * EW_ROWS];
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = k < nc;
  const int ka = live ? k : nc - 1;
  const double2* e0 = tab + ka;
  const double2* e1 = e0 + (size_t)(g.M[0] + 1) * nc;
  const double2* e2 = e1 + (size_t)(g.M[1] + 1) * nc;
  const int rb = blockIdx.y * rows_per, re = min(g.nrow, rb + rows_per);
  double fx = 0.0, fy = 0.0, fz = 0.0;
  for (int r0 = rb; r0 < re; r0 += EW_ROWS) {
    double2 T0[EW_ROWS], T1[EW_ROWS];
#pragma unroll
    for (int j = 0; j < EW_ROWS; ++j) T0[j] = T1[j] = make_double2(0.0, 0.0);
    for (int c0 = 0; c0 < g.ncol; c0 += EW_COLS) {
      const int nc0 = min(EW_COLS, g.ncol - c0);
      __syncthreads();
      for (int t = threadIdx.x; t < nc0 * EW_ROWS; t += blockDim.x) {
        const int r = r0 + t % EW_ROWS, c = c0 + t / EW_ROWS;
        D[t] = r < re ? coef[(size_t)r * g.ncol + c] : double4a{0, 0, 0, 0};
      }
      __syncthreads();
      for (int c = 0; c < nc0; ++c) {
        const double2 e = e2[(size_t)(c0 + c) * nc];
        const double mc = (c0 + c) * e.x, ms = (c0 + c) * e.y;
#pragma unroll
        for (int j = 0; j < EW_ROWS; ++j) {
          const double4a d = D[c * EW_ROWS + j];  // P, M
          T0[j].x += e.x * d.x + e.y * d.w;
          T0[j].y += e.y * d.z - e.x * d.y;
          T1[j].x += mc * d.z + ms * d.y;
          T1[j].y += ms * d.x - mc * d.w;
        }
      }
    }
#pragma unroll
    for (int j = 0; j < EW_ROWS; ++j) {
      const int r = r0 + j;
      if (r >= re) break;
      const int m0 = r / g.n1, m1 = r - m0 * g.n1 - g.M[1];
      const double2 x = e0[(size_t)m0 * nc];
      double2 y = e1[(size_t)abs(m1) * nc];
      if (m1 < 0) y.y = -y.y;
      const double2 a = make_double2(x.x * y.x - x.y * y.y, x.x * y.y + x.y * y.x);
      const double t0 = a.x * T0[j].y + a.y * T0[j].x;
      fx += m0 * t0;
      fy += m1 * t0;
      fz += a.x * T1[j].y + a.y * T1[j].x;
    }
  }
  if (!live) return;
  const double q = pos ? pos[i0 + k].w : (double)posf[i0 + k].w;
  double* f = fpart + (size_t)blockIdx.y * 3 * nc + k;
  f[0] = q * fx * st->Li[0];
  f[nc] = q * fy * st->Li[1];
  f[2 * (size_t)nc] = q * fz * st->Li[2];
}

__global__ void __launch_bounds__(256)
k_ew_sum(int i0, int nc, int nsplit, const double* __restrict__ fpart, double4a* __restrict__ force) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nc) return;
  double f[3] = {0, 0, 0};
  for (int z = 0; z < nsplit; ++z)
    for (int d = 0; d < 3; ++d) f[d] += fpart[((size_t)z * 3 + d) * nc + k];
  double4a v = force[i0 + k];
  v.x += f[0]; v.y += f[1]; v.z += f[2];
  force[i0 + k] = v;
}

}  // namespace

extern "C" int md_ewald_exact(md_system* sys, const int K[3], double beta, double* energy, int add_forces) {
  if (!sys || !K || !(beta > 0)) return MD_ERR_BADARG;
  EwGeom g;
  for (int d = 0; d < 3; ++d) g.M[d] = K[d] / 2;
  g.n1 = 2 * g.M[1] + 1;
  if (g.M[0] < 0 || g.M[1] < 0 || g.M[2] < 0 || (double)(g.M[0] + 1) * g.n1 * (g.M[2] + 1) > 2.0e9) {
    md_set_error("md_ewald_exact: mode box %d x %d x %d out of range", K[0], K[1], K[2]);
    return MD_ERR_BADARG;
  }
  g.nrow = (g.M[0] + 1) * g.n1;
  g.ncol = g.M[2] + 1;
  const int N = sys->N, nmax = std::min(N, EW_CHUNK), nm = g.nrow * g.ncol, ntab = g.M[0] + g.M[1] + g.M[2] + 3;
  // enough blocks for a few per SM: the S sum split over atoms, the forces over rows
  const int tiles = ceil_div(g.nrow, EW_T) * ceil_div(g.ncol, EW_T);
  const int ss = std::max(1, std::min(ceil_div(nmax, 2 * EW_A), ceil_div(148 * 16, tiles)));
  const int per = ceil_div(ceil_div(nmax, ss), EW_A) * EW_A, ns = ceil_div(nmax, per);
  const int fs = std::max(1, std::min(ceil_div(g.nrow, EW_ROWS), ceil_div(148 * 8, ceil_div(nmax, 128))));
  const int rows_per = ceil_div(ceil_div(g.nrow, fs), EW_ROWS) * EW_ROWS, nf = ceil_div(g.nrow, rows_per);
  const int nbc = ceil_div(nm, 256);
  const size_t b_coef = sizeof(double4a) * (size_t)nm, b_tab = sizeof(double2) * (size_t)ntab * nmax,
               b_part = sizeof(double) * 4 * (size_t)ns * nm, b_f = sizeof(double) * 3 * (size_t)nf * nmax,
               b_red = sizeof(double) * ((size_t)nbc + 4);
  SysScratch buf;
  if (int r = buf.take(sys, b_coef + b_tab + b_part + b_f + b_red)) return r;
  char* p = (char*)buf.p;
  double4a* coef = (double4a*)p;
  double2* tab = (double2*)(p += b_coef);
  double* part = (double*)(p += b_tab);
  double* fpart = (double*)(p += b_part);
  double* e = (double*)(p += b_f);
  double* red = e + 4;
  cudaStream_t s = sys->stream;
  const bool f64 = sys->prec == MD_PREC_FP64;
  const double4a* pos = f64 ? (const double4a*)sys->pos : nullptr;
  const float4* posf = f64 ? nullptr : (const float4*)sys->pos;
  auto tables = [&](int i0, int nc) {
    k_ew_tables<<<dim3(ntab, ceil_div(nc, 256)), 256, 0, s>>>(N, i0, nc, pos, posf, g, sys->st, tab);
  };
  for (int i0 = 0; i0 < N; i0 += EW_CHUNK) {
    const int nc = std::min(EW_CHUNK, N - i0);
    tables(i0, nc);
    k_ew_sk<<<dim3(tiles, 1, ns), 64, 0, s>>>(i0, nc, pos, posf, g, tab, per, i0 > 0, part);
  }
  k_ew_coef<<<nbc, 256, 0, s>>>(g, beta, ns, part, sys->st, coef, red, e);
  MD_CHECK_LAUNCH("ewald sk");
  if (add_forces) {
    for (int i0 = 0; i0 < N; i0 += EW_CHUNK) {
      const int nc = std::min(EW_CHUNK, N - i0);
      if (N > EW_CHUNK) tables(i0, nc);
      k_ew_force<<<dim3(ceil_div(nc, 128), nf), 128, 0, s>>>(i0, nc, pos, posf, g, tab, coef, rows_per, sys->st,
                                                            fpart);
      k_ew_sum<<<ceil_div(nc, 256), 256, 0, s>>>(i0, nc, nf, fpart, sys->force);
    }
    MD_CHECK_LAUNCH("ewald force");
  }
  double h = 0;
  MD_CUDA(cudaMemcpyAsync(&h, e, sizeof(double), cudaMemcpyDeviceToHost, s));
  MD_CUDA(cudaStreamSynchronize(s));
  if (energy) *energy = h;
  return MD_OK;
}

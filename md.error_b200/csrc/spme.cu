// Smooth particle-mesh Ewald (reciprocal part).
// Reference (RE = longRange.hetero/profile.test/template/tools/real.error):
//   calQ spread                      RE/src/EleRecBSpline.cpp:541-619
//   calB / calPsiFPhiF (ik)          RE/src/EleRecBSpline.cpp:729-877
//   applyInteractionCalPotential ik  RE/src/EleRecBSpline.cpp:393-536
//   analytic differentiation         RE/src/EleRecFBSpline.cpp:771-907, 1146-1195
//
// Chain of one force evaluation (each step one kernel):
//   spread      lanes along the stencil rows, mesh atomics; dense large systems
//               through a shared-memory tile (spme_pm.cu)
// then, where the x and y sizes are equal and a plane fits an SM, three passes by
// planes (spme_plane.cu); on other meshes
//   z pass      R2C along z (real lines -> half-complex lines)
//   y pass      forward C2C along y
//   x pass      forward C2C along x, k-space step (energy and virial in FP64,
//               influence multiply; ik: the three products i(-2 pi m_d) psi Q^,
//               analytic: psi Q^ / 2) and the inverse C2C along x, fused
//   y pass      inverse C2C along y (all products)
//   z pass      C2R along z with the Hermitian completion of an r2c half
//               spectrum (the FFTW c2r convention the reference relies on);
//               for ik the three meshes are written interleaved, one Real4
//               per mesh point
//   gather      a warp per atom, lanes along its stencil rows (spme_pm.cu)
// The FFT passes are radix-8 Stockham transforms of whole lines in shared
// memory; a block holds several lines adjacent in memory so that strided
// axes load coalesced.  Mixed precision: mesh, FFT and gather in FP32,
// energy/virial and force accumulation in FP64.  Power-of-two mesh sizes.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>
#include "device_common.cuh"
#include "fft_lines.cuh"
#include "spme_plane.cuh"
#include "spme_pm.cuh"

struct md_spme {
  md_system* sys = nullptr;
  int K[3] = {0, 0, 0};
  int K2h = 0;
  int order = 6;
  int method = 0;  // 0 ik, 1 analytic
  double beta = 1.0;
  size_t nreal = 0, nhalf = 0;
  void* Q = nullptr;      // real mesh
  void* C = nullptr;      // complex half meshes: [0] Q^, [1..3] products
  void* G = nullptr;      // convolved real mesh(es): ik Real4 (x, y, z, 0) per point; analytic and adjoint one Real
  void* psi = nullptr;    // influence function on the half spectrum (ik normalisation)
  void* tw[3] = {nullptr, nullptr, nullptr};  // per-axis forward twiddles exp(-2 pi i m / K_d)
  double* bm = nullptr;   // per-axis |b(m)|^2 (k_spme_bmod)
  double4a* frec = nullptr;   // reciprocal forces of a concurrent evaluation (stored, not added)
  double* partials = nullptr; // block partials of the x pass (its own: it may run beside other reductions)
  int max_blocks = 0;
  bool planes = false;        // equal x and y sizes: the transforms run by planes (spme_plane.cu)
  double* d_box_tab = nullptr;  // box psi was computed for (device; 0 = never)
};

// ---------------------------------------------------------------- B-spline weights
// M_n(f + j), j = 0..n-1 (and derivatives) by the recursion
// M_k(u) = (u M_{k-1}(u) + (k - u) M_{k-1}(u - 1)) / (k - 1)  (Essmann et al. 1995)
template <class R>
__device__ __forceinline__ void bspline_w(int n, R f, R* w, R* dw) {
  w[0] = f;
  w[1] = R(1) - f;
  for (int j = 2; j < n; ++j) w[j] = R(0);
  for (int k = 3; k <= n; ++k) {
    if (k == n && dw) {
      for (int j = 0; j < n; ++j) dw[j] = (j < n - 1 ? w[j] : R(0)) - (j > 0 ? w[j - 1] : R(0));
    }
    const R inv = R(1) / R(k - 1);
    for (int j = k - 1; j >= 0; --j) {
      const R u = f + R(j);
      const R a = (j < k - 1) ? w[j] : R(0);
      const R b = (j > 0) ? w[j - 1] : R(0);
      w[j] = (u * a + (R(k) - u) * b) * inv;
    }
  }
  if (n == 2 && dw) { dw[0] = R(1); dw[1] = R(-1); }
}

// ---------------------------------------------------------------- FFT passes (fft_lines.cuh)
// One transform pass over lines of one axis.
//   MODE 0: real lines along z (contiguous) -> half-complex lines (n/2+1);
//           the input lines are cleared after they are read
//   MODE 1: complex lines of the half spectrum; line L starts at
//           (L / inner) * outer + L % inner, elements `stride` apart; lines
//           adjacent in memory share a block, so loads coalesce across lines
//   MODE 2: half-complex z lines -> real lines (Hermitian completion, the
//           FFTW c2r convention the reference relies on)
// blockIdx.y selects the batch (in_bs / out_bs apart).  OUT4 (MODE 2): the
// three batches of a line are transformed side by side in one block, by
// three groups of FFT_THREADS threads, and written interleaved, one Real4
// (x, y, z, 0) per mesh point.
template <class R, int LOGN, int MODE, int SIGN, int OUT4>
__global__ void __launch_bounds__(FFT_THREADS * (OUT4 ? 2 : 1))
k_fftp(const void* in, void* out, const typename C2<R>::T* __restrict__ twg, long nlines, long stride, long inner,
       long outer, long in_bs, long out_bs) {
  typedef typename C2<R>::T T2;
  typedef FftGeom<LOGN> G;
  // OUT4: the three Hermitian spectra become the x, y, z of one real
  // 4-vector mesh; group 0 inverts A + iB (the x and y spectra: both results
  // real, they come back as the real and imaginary parts), group 1 the z
  constexpr int n = G::n, LPB = G::LPB, LS = G::LS, NG = OUT4 ? 2 : 1, nh = n / 2 + 1;
  extern __shared__ __align__(16) unsigned char fft_smem[];
  T2* tw = reinterpret_cast<T2*>(fft_smem);
  T2* X = tw + n;
  long* lo = reinterpret_cast<long*>(X + NG * LPB * LS);
  load_tw<R, SIGN>(tw, twg, n);
  // MODE 0: the real lines 2L and 2L + 1 go in as the real and imaginary
  // parts of complex line L, and their half spectra are separated after the
  // transform: A_k = (Z_k + conj Z_{n-k}) / 2, B_k = (Z_k - conj Z_{n-k}) / 2i
  const long nlc = MODE == 0 ? (nlines + 1) / 2 : nlines;  // complex lines
  const long line0 = (long)blockIdx.x * LPB;
  if (threadIdx.x < LPB) {
    const long L = line0 + threadIdx.x;
    lo[threadIdx.x] = MODE == 1 ? (L / inner) * outer + L % inner : L;
  }
  __syncthreads();
  const int grp = NG > 1 ? (int)threadIdx.x / FFT_THREADS : 0;
  const int gt = NG > 1 ? (int)threadIdx.x % FFT_THREADS : (int)threadIdx.x;
  const long batch = OUT4 ? 2 * grp : blockIdx.y;
  T2* Xb = X + grp * LPB * LS;
  {
    // all loads of a thread are issued before any shared-memory store (and,
    // in MODE 0, before the mesh is cleared), so they are in flight together
    T2 vv[G::EPT];
#pragma unroll
    for (int s = 0; s < G::EPT; ++s) {
      const int e = gt + s * FFT_THREADS;
      int l, k;
      if (MODE == 1) { l = e % LPB; k = e / LPB; }
      else { l = e >> LOGN; k = e & (n - 1); }
      const long L = line0 + l;
      T2 v;
      v.x = R(0);
      v.y = R(0);
      if (L < nlc) {
        if (MODE == 0) {
          const R* src = reinterpret_cast<const R*>(in) + batch * in_bs;
          v.x = src[2 * L * n + k];
          if (2 * L + 1 < nlines) v.y = src[(2 * L + 1) * n + k];
        } else if (MODE == 1) {
          v = reinterpret_cast<const T2*>(in)[batch * in_bs + lo[l] + k * stride];
        } else {
          const T2* src = reinterpret_cast<const T2*>(in) + batch * in_bs + L * nh;
          if (k < nh) v = src[k];
          else { const T2 u = src[n - k]; v.x = u.x; v.y = -u.y; }
          if (OUT4 && grp == 0) {
            // + i B, B the spectrum of the next batch.  A real transform
            // ignores the imaginary parts at k = 0 and n/2 (the mirrored half
            // carries the rest); they are dropped here, or they would cross
            // into the other result
            const T2* srb = src + in_bs;
            T2 b;
            if (k < nh) b = srb[k];
            else { const T2 u = srb[n - k]; b.x = u.x; b.y = -u.y; }
            if (k == 0 || k == n / 2) { v.y = R(0); b.y = R(0); }
            v.x -= b.y;
            v.y += b.x;
          }
        }
      }
      vv[s] = v;
    }
#pragma unroll
    for (int s = 0; s < G::EPT; ++s) {
      const int e = gt + s * FFT_THREADS;
      int l, k;
      if (MODE == 1) { l = e % LPB; k = e / LPB; }
      else { l = e >> LOGN; k = e & (n - 1); }
      if (MODE == 0) {
        // the real mesh is consumed: cleared for the next spread
        const long L = line0 + l;
        R* src = reinterpret_cast<R*>(const_cast<void*>(in)) + batch * in_bs;
        if (L < nlc) src[2 * L * n + k] = R(0);
        if (2 * L + 1 < nlines) src[(2 * L + 1) * n + k] = R(0);
      }
      Xb[l * LS + fft_pad<R>(k)] = vv[s];
    }
  }
  __syncthreads();
  fft_stages<R, LOGN, 0, SIGN>(Xb + (gt / G::TPL) * LS, tw, gt % G::TPL);
  if (OUT4) {
    typedef typename V4<R>::T R4;
    for (int e = threadIdx.x; e < LPB * n; e += NG * FFT_THREADS) {
      const int l2 = e >> LOGN, k = e & (n - 1);
      const long L = line0 + l2;
      if (L >= nlines) continue;
      R4 o;
      const T2 xy = X[l2 * LS + fft_pad<R>(k)];
      o.x = xy.x;
      o.y = xy.y;
      o.z = X[LPB * LS + l2 * LS + fft_pad<R>(k)].x;
      o.w = R(0);
      reinterpret_cast<R4*>(out)[L * n + k] = o;
    }
    return;
  }
  for (int e = threadIdx.x; e < LPB * n; e += FFT_THREADS) {
    int l2, k;
    if (MODE == 1) { l2 = e % LPB; k = e / LPB; }
    else { l2 = e >> LOGN; k = e & (n - 1); }
    const long L = line0 + l2;
    if (L >= nlc) continue;
    const T2 v = X[l2 * LS + fft_pad<R>(k)];
    if (MODE == 0) {
      if (k < nh) {
        const T2 w = X[l2 * LS + fft_pad<R>((n - k) & (n - 1))];
        T2 a, b;
        a.x = R(0.5) * (v.x + w.x);
        a.y = R(0.5) * (v.y - w.y);
        b.x = R(0.5) * (v.y + w.y);
        b.y = R(0.5) * (w.x - v.x);
        T2* dst = reinterpret_cast<T2*>(out) + batch * out_bs;
        dst[2 * L * nh + k] = a;
        if (2 * L + 1 < nlines) dst[(2 * L + 1) * nh + k] = b;
      }
    } else if (MODE == 1) {
      reinterpret_cast<T2*>(out)[batch * out_bs + lo[l2] + k * stride] = v;
    } else {
      reinterpret_cast<R*>(out)[batch * out_bs + L * n + k] = v.x;
    }
  }
}

template <class R>
static size_t fftp_smem(int logn, int nbuf) {
  const int n = 1 << logn, tpl = n >= 8 ? n / 8 : 1, lpb = FFT_THREADS / tpl;
  return sizeof(typename C2<R>::T) * ((size_t)n + (size_t)nbuf * lpb * fft_line_stride(n)) + sizeof(long) * lpb;
}

// Forward transform along x, the k-space step and the inverse transform(s)
// along x, in one pass over the x lines (y, kz fixed) of the half spectrum:
//   psi(m) = exp(-pi^2 m^2 / beta^2) / m^2 |b0(i)|^2 |b1(j)|^2 |b2(k)|^2 / (pi V)
//     (calB / calPsiFPhiF), evaluated in FP64 from the per-axis |b|^2
//     tables for the current box, so an NPT box change needs no extra pass,
//   E = 1/2 sum_m psi |Q^|^2 and the diagonal virial (FP64, with_stats),
//   ik (METHOD 0): the three products phi_d = i (-2 pi m_d) psi Q^,
//   (merge = 0: the sums stay in DevState::scratch for a later merge)
//   analytic (METHOD 1): psi Q^ / 2 (FBSpline normalisation),
// each transformed back along x and written to C[1 + d].  Groups of
// FFT_THREADS threads: group 0 runs the forward transform and the k-space
// step (group 1 meets the same barriers), then for ik group 0 inverts phi_x
// and group 1 inverts psi Q^,
// whose transform times -2 pi i m_y and -2 pi i m_z (constant along the
// line) gives phi_y and phi_z.  The last block merges the energy and the
// virial into the statistics slots.
template <class R, int LOGN, int METHOD>
__global__ void __launch_bounds__(FFT_THREADS * (METHOD == 0 ? 3 : 1))
k_fft_x_kspace(typename C2<R>::T* C, const typename C2<R>::T* __restrict__ twg, const double* __restrict__ bm, int K1,
               int K2, double beta, DevState* st, double* partials, int with_stats, int merge) {
  typedef typename C2<R>::T T2;
  typedef FftGeom<LOGN> G;
  // ik: group 0 transforms -2 pi i m_x psi Q^ back; m_y and m_z are constant
  // along an x line, so group 1 transforms psi Q^ once and its result, times
  // -2 pi i m_y and -2 pi i m_z, gives the other two products
  constexpr int n = G::n, LPB = G::LPB, LS = G::LS, EPT = G::EPT, NG = METHOD == 0 ? 2 : 1;
  const int K2h = K2 / 2 + 1;
  const long nlines = (long)K1 * K2h, stride = nlines;
  const size_t nhalf = (size_t)n * nlines;
  extern __shared__ __align__(16) unsigned char fft_smem[];
  T2* twf = reinterpret_cast<T2*>(fft_smem);
  T2* twi = twf + n;
  T2* X = twi + n;
  T2* Y = X + LPB * LS;  // NG buffers
  R* PS = reinterpret_cast<R*>(Y + NG * LPB * LS);
  // psi = exp(-pi^2 m^2 / beta^2) / m^2 * B(m) / (pi V) factors by axis: the
  // x factors exp(-sc m_x^2) b_x(i) for the n points of a line and, per line
  // (j, k), exp(-sc (m_y^2 + m_z^2)) b_y(j) b_z(k) / (pi V) and m_y^2 + m_z^2,
  // worked out once per block (FP64), leaving one reciprocal per point
  double* EX = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(PS + LPB * LS) + 7) & ~(uintptr_t)7);
  double* EJK = EX + n;
  double* MJK = EJK + LPB;
  int* lj = reinterpret_cast<int*>(MJK + LPB);
  int* lk = lj + LPB;
  load_tw<R, -1>(twf, twg, n);
  load_tw<R, 1>(twi, twg, n);
  const long line0 = (long)blockIdx.x * LPB;
  const double sc = M_PI * M_PI / (beta * beta);
  if (threadIdx.x < LPB) {
    const long L = line0 + threadIdx.x;
    const int j = (int)(L / K2h), k = (int)(L % K2h);
    lj[threadIdx.x] = j;
    lk[threadIdx.x] = k;
    const int jp = j <= K1 / 2 ? j : j - K1;
    const double my = jp * st->Li[1], mz = k * st->Li[2], mjk = my * my + mz * mz;
    const double V = st->L[0] * st->L[1] * st->L[2];
    MJK[threadIdx.x] = mjk;
    EJK[threadIdx.x] = exp(-sc * mjk) * (bm[n + j] * bm[n + K1 + k]) / (M_PI * V);
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int ip = i <= n / 2 ? i : i - n;
    const double mx = ip * st->Li[0];
    EX[i] = exp(-sc * mx * mx) * bm[i];
  }
  const int grp = NG > 1 ? (int)threadIdx.x / FFT_THREADS : 0;
  const int gt = NG > 1 ? (int)threadIdx.x % FFT_THREADS : (int)threadIdx.x;
  if (grp == 0) {
    T2 vv[EPT];
#pragma unroll
    for (int s = 0; s < EPT; ++s) {
      const int e = gt + s * FFT_THREADS, l = e % LPB, i = e / LPB;
      const long L = line0 + l;
      vv[s].x = R(0);
      vv[s].y = R(0);
      if (L < nlines) vv[s] = C[L + i * stride];
    }
#pragma unroll
    for (int s = 0; s < EPT; ++s) {
      const int e = gt + s * FFT_THREADS;
      X[(e % LPB) * LS + fft_pad<R>(e / LPB)] = vv[s];
    }
  }
  __syncthreads();
  const int l = gt / G::TPL, tl = gt % G::TPL;
  if (grp == 0) fft_stages<R, LOGN, 0, -1>(X + l * LS, twf, tl);
  else fft_stage_barriers<LOGN, 0>();
  double v[4] = {0, 0, 0, 0};
  if (grp == 0) {
#pragma unroll
    for (int s = 0; s < EPT; ++s) {
      const int e = gt + s * FFT_THREADS, le = e % LPB, i = e / LPB;
      const long L = line0 + le;
      const int j = lj[le], k = lk[le];
      const int ip = i <= n / 2 ? i : i - n, jp = j <= K1 / 2 ? j : j - K1;
      const double mx = ip * st->Li[0];
      const double mm = mx * mx + MJK[le];
      const bool live = L < nlines && (ip || jp || k);
      const double inv = live ? 1.0 / mm : 0.0;
      const R ps = live ? (R)(EX[i] * EJK[le] * inv) : R(0);
      PS[le * LS + i] = ps;
      if (with_stats && live) {
        // E = 1/2 sum_m |Q^|^2 psi over the full spectrum: interior z planes count twice
        const T2 q = X[le * LS + fft_pad<R>(i)];
        const double wgt = (k == 0 || (2 * k == K2)) ? 1.0 : 2.0;
        const double e2 = 0.5 * wgt * ((double)q.x * q.x + (double)q.y * q.y) * (double)ps;
        // f = 2 (1 + pi^2 m^2 / beta^2) / m^2
        const double f = 2.0 * inv + 2.0 * sc;
        const double m[3] = {mx, jp * st->Li[1], k * st->Li[2]};
        v[0] += e2;
        // pressure tensor V P_aa = sum_m E_m (1 - f m_a^2); the virial slots hold W_aa = -V P_aa
#pragma unroll
        for (int d = 0; d < 3; ++d) v[1 + d] += -e2 * (1.0 - f * m[d] * m[d]);
      }
    }
  }
  __syncthreads();
  T2* Yg = Y + grp * LPB * LS;
#pragma unroll
  for (int s = 0; s < EPT; ++s) {
    const int e = gt + s * FFT_THREADS, le = e % LPB, i = e / LPB;
    const T2 q = X[le * LS + fft_pad<R>(i)];
    const R ps = PS[le * LS + i];
    T2 g;
    if (METHOD == 0 && grp == 0) {
      // phi_x = i (-2 pi m_x) psi Q^, m_x = i' / L_x (signed index)
      const int ix = i <= n / 2 ? i : i - n;
      const R c = (R)(-2.0 * M_PI * (ix * st->Li[0])) * ps;
      g.x = -q.y * c;
      g.y = q.x * c;
    } else if (METHOD == 0) {
      g.x = q.x * ps;
      g.y = q.y * ps;
    } else {
      g.x = q.x * (R(0.5) * ps);
      g.y = q.y * (R(0.5) * ps);
    }
    Yg[le * LS + fft_pad<R>(i)] = g;
  }
  __syncthreads();
  fft_stages<R, LOGN, 0, 1>(Yg + l * LS, twi, tl);
  if (METHOD == 0 && grp == 1) {
    // phi_y and phi_z = i (-2 pi m_d) times the transform of psi Q^
    T2* outy = C + 2 * nhalf;
    T2* outz = C + 3 * nhalf;
    for (int e = gt; e < LPB * n; e += FFT_THREADS) {
      const int le = e % LPB, i = e / LPB;
      const long L = line0 + le;
      if (L >= nlines) continue;
      const int jp = lj[le] <= K1 / 2 ? lj[le] : lj[le] - K1;
      const R cy = (R)(-2.0 * M_PI * (jp * st->Li[1])), cz = (R)(-2.0 * M_PI * (lk[le] * st->Li[2]));
      const T2 v = Yg[le * LS + fft_pad<R>(i)];
      T2 a, b;
      a.x = -v.y * cy;
      a.y = v.x * cy;
      b.x = -v.y * cz;
      b.y = v.x * cz;
      outy[L + i * stride] = a;
      outz[L + i * stride] = b;
    }
  } else {
    T2* out = C + (1 + grp) * nhalf;
    for (int e = gt; e < LPB * n; e += FFT_THREADS) {
      const int le = e % LPB, i = e / LPB;
      const long L = line0 + le;
      if (L < nlines) out[L + i * stride] = Yg[le * LS + fft_pad<R>(i)];
    }
  }
  if (with_stats && block_reduce_finish<4>(v, partials, &st->red_counter[RED_SPME], st->scratch, true) && merge) {
    // reciprocal energy into its slot, its diagonal virial added to the virial slots
    st->stats[MD_STAT_ELEC_REC] = st->scratch[0];
    for (int d = 0; d < 3; ++d) st->stats[MD_STAT_VIRIAL_XX + d] += st->scratch[1 + d];
  }
}

template <class R>
static size_t fftx_smem(int logn, int method) {
  const int n = 1 << logn, tpl = n >= 8 ? n / 8 : 1, lpb = FFT_THREADS / tpl, ng = method == 0 ? 2 : 1;
  return sizeof(typename C2<R>::T) * (2 * (size_t)n + (1 + (size_t)ng) * lpb * fft_line_stride(n)) +
         sizeof(R) * (size_t)lpb * fft_line_stride(n) + 8 + sizeof(double) * ((size_t)n + 2 * lpb) + 2 * sizeof(int) * lpb;
}

// per-axis forward twiddle table exp(-2 pi i m / n), m < n, from FP64
template <class R>
__global__ void k_fft_twiddles(int n, typename C2<R>::T* tw) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= n) return;
  double s, c;
  sincospi(2.0 * m / n, &s, &c);
  tw[m].x = (R)c;
  tw[m].y = (R)(-s);
}

// ---------------------------------------------------------------- influence
__device__ __forceinline__ double bmod_d(int n, int K, int m) {
  // |b(m)|^2 = 1 / |sum_{k=0}^{n-2} M_n(k+1) exp(2 pi i m k / K)|^2 (calB)
  double w[16];
  bspline_w<double>(n, 0.0, w, nullptr);  // w[j] = M_n(j)
  double re = 0, im = 0;
  for (int k = 0; k < n - 1; ++k) {
    double s, c;
    sincospi(2.0 * (double)((long)m * k % K) / K, &s, &c);
    re += w[k + 1] * c;
    im += w[k + 1] * s;
  }
  return 1.0 / (re * re + im * im);
}

// psi is recomputed only when the box differs from `tab`, the box it was last
// computed for (NPT); the comparison is made on the device so that no host
// round trip is needed, and `tab` is updated by k_spme_box_tab afterwards.
// The force chain evaluates psi inside its x pass; this stored copy serves
// the adjoint and md_spme_get_influence.
template <class R>
__global__ void k_spme_influence(int K0, int K1, int K2, int n, double beta, const DevState* st, R* psi,
                                 const double* tab) {
  const int K2h = K2 / 2 + 1;
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (t >= (long)K0 * K1 * K2h) return;
  if (st->L[0] == tab[0] && st->L[1] == tab[1] && st->L[2] == tab[2]) return;
  const int k = (int)(t % K2h), j = (int)((t / K2h) % K1), i = (int)(t / ((long)K2h * K1));
  const int ip = i <= K0 / 2 ? i : i - K0, jp = j <= K1 / 2 ? j : j - K1, kp = k;
  if (!ip && !jp && !kp) { psi[t] = R(0); return; }
  const double V = st->L[0] * st->L[1] * st->L[2];
  const double m0 = ip * st->Li[0], m1 = jp * st->Li[1], m2 = kp * st->Li[2];
  const double mm = m0 * m0 + m1 * m1 + m2 * m2;
  const double B = bmod_d(n, K0, i) * bmod_d(n, K1, j) * bmod_d(n, K2, k);
  const double sc = M_PI * M_PI / beta / beta;
  psi[t] = (R)(exp(-sc * mm) / mm * B / (M_PI * V));
}

__global__ void k_spme_box_tab(const DevState* st, double* tab) {
  for (int d = 0; d < 3; ++d) tab[d] = st->L[d];
}

// per-axis |b_d(m)|^2 tables, concatenated: [0, K0) | [0, K1) | [0, K2/2+1)
__global__ void k_spme_bmod(int K0, int K1, int K2, int n, double* bm) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < K0) bm[t] = bmod_d(n, K0, t);
  else if (t < K0 + K1) bm[t] = bmod_d(n, K1, t - K0);
  else if (t < K0 + K1 + K2 / 2 + 1) bm[t] = bmod_d(n, K2, t - K0 - K1);
}

// ---------------------------------------------------------------- adjoint
// The reciprocal energy is the quadratic form E = 1/2 sum_m psi(m) |Q^(m)|^2
// = 1/2 sum_k Q(k) Phi(k) with Phi = IFFT(psi Q^) (unnormalised transforms),
// Q(k) = sum_i q_i theta_i(k), theta_i(k) = prod_d M_n(u_id - k_d), u = K x / L.
// Hence
//   dE/dq_i      = sum_k theta_i(k) Phi(k)                      (potential)
//   dE/dx_id     = q_i sum_k d theta_i(k)/du_d Phi(k) K_d / L_d  (exact gradient,
//                  the analytic-differentiation force with its sign flipped)
//   dE/dpsi(m)   = 1/2 |Q^(m)|^2
//   dE/dbeta     = sum_m 1/2 |Q^(m)|^2 psi(m) 2 pi^2 |m|^2 / beta^3
// The adjoint recomputes the spread mesh and its transform instead of
// keeping them from an earlier forward call.
template <class R>
__global__ void __launch_bounds__(256)
k_spme_adj_kspace(int K0, int K1, int K2, double beta, const R* __restrict__ psi, typename C2<R>::T* __restrict__ C,
                  size_t nhalf, DevState* st, double* partials, double* __restrict__ dpsi) {
  typedef typename C2<R>::T T2;
  const int K2h = K2 / 2 + 1;
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  double v[2] = {0, 0};
  if (t < (long)nhalf) {
    const int k = (int)(t % K2h), j = (int)((t / K2h) % K1), i = (int)(t / ((long)K2h * K1));
    const int ip = i <= K0 / 2 ? i : i - K0, jp = j <= K1 / 2 ? j : j - K1, kp = k;
    const T2 q = C[t];
    const R ps = psi[t];
    T2 g;
    g.x = q.x * ps;
    g.y = q.y * ps;
    C[nhalf + t] = g;
    // interior z planes of the half spectrum stand for two full-spectrum modes
    const double wgt = (k == 0 || (2 * k == K2)) ? 1.0 : 2.0;
    const double q2 = 0.5 * wgt * ((double)q.x * q.x + (double)q.y * q.y);
    if (dpsi) dpsi[t] = (ip || jp || kp) ? q2 : 0.0;
    if (ip || jp || kp) {
      const double m0 = ip * st->Li[0], m1 = jp * st->Li[1], m2 = kp * st->Li[2];
      const double mm = m0 * m0 + m1 * m1 + m2 * m2;
      v[0] = q2 * (double)ps;
      v[1] = v[0] * 2.0 * M_PI * M_PI * mm / (beta * beta * beta);
    }
  }
  block_reduce_finish<2>(v, partials, &st->red_counter[RED_SPME], st->scratch, true);
}

// ---------------------------------------------------------------- self-force correction
// SelfCorr (RE/src/SelfCorr.cpp:99-220), analytic differentiation, |k| <= 3:
//   c_d(k) = sum_{m != 0} f(m) (-2) g_d(m_d, k) (-4 pi k K_d / L_d),
//   f(m) = e^{-pi^2 |m|^2 / beta^2} / |m|^2 / (2 pi V)
//   g_d(m, k) = (u + 2 pi k)^-n / sum_{l=-3..3} (u + 2 pi l)^-n, u = 2 pi m / K_d
//   (0 at the Nyquist index of an even K_d);
//   F_id -= sum_{k=1..3} c_d(k) q_i^2 sin(2 pi k K_d x_id / L_d).
// g_d depends on m_d alone, so the K^3 sum is regrouped per axis: W_d(i) is
// the sum of f over the other two indices (one block per (i, d)), then the
// nine c_d(k) are 1-D sums.
__global__ void __launch_bounds__(256)
k_selfcorr_weights(int K0, int K1, int K2, double beta, const DevState* st, double* W /* [3][Kmax] */, int Kmax) {
  const int d = blockIdx.y, i = blockIdx.x;
  const int K[3] = {K0, K1, K2};
  if (i >= K[d]) return;
  const int a = (d + 1) % 3, b = (d + 2) % 3;
  int p[3];
  p[d] = i > (K[d] >> 1) ? i - K[d] : i;
  const double V = st->L[0] * st->L[1] * st->L[2];
  const double t = M_PI / beta, scal = 1.0 / (2.0 * M_PI * V);
  double acc = 0.0;
  for (int e = threadIdx.x; e < K[a] * K[b]; e += blockDim.x) {
    const int ia = e / K[b], ib = e % K[b];
    p[a] = ia > (K[a] >> 1) ? ia - K[a] : ia;
    p[b] = ib > (K[b] >> 1) ? ib - K[b] : ib;
    const double m0 = p[0] * st->Li[0], m1 = p[1] * st->Li[1], m2 = p[2] * st->Li[2];
    const double mm = m0 * m0 + m1 * m1 + m2 * m2;
    if (mm == 0.0) continue;
    acc += exp(-t * t * mm) / mm * scal;
  }
  __shared__ double sh[8];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += sh[w];
    W[d * Kmax + i] = s;
  }
}

__device__ __forceinline__ double ipow_dev(double x, int n) {
  double r = 1.0;
  for (int k = 0; k < n; ++k) r *= x;
  return r;
}

// one warp per (d, k), k = 1..3: c[d][k]
__global__ void k_selfcorr_coef(int K0, int K1, int K2, int order, const DevState* st, const double* W, int Kmax,
                                double* coef /* [3][4] */) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (w >= 9) return;
  const int d = w / 3, kk = 1 + w % 3;
  const int K[3] = {K0, K1, K2};
  double acc = 0.0;
  for (int i = lane; i < K[d]; i += 32) {
    if (i == (K[d] >> 1) && (K[d] % 2 == 0)) continue;
    const int p = i > (K[d] >> 1) ? i - K[d] : i;
    const double u = 2.0 * M_PI * p / K[d];
    double s = 1.0 / ipow_dev(u, order), up = u, un = u;
    for (int l = 0; l < 3; ++l) {
      up += 2.0 * M_PI;
      un -= 2.0 * M_PI;
      s += 1.0 / ipow_dev(up, order);
      s += 1.0 / ipow_dev(un, order);
    }
    const double g = 1.0 / ipow_dev(u + 2.0 * M_PI * kk, order) / s;
    acc += W[d * Kmax + i] * (-2.0 * g) * (-4.0) * M_PI * kk * (double)K[d] * st->Li[d];
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) coef[d * 4 + kk] = acc;
}

template <class R>
__global__ void __launch_bounds__(256)
k_selfcorr_apply(int N, const typename V4<R>::T* __restrict__ pos, int K0, int K1, int K2, const DevState* st,
                 const double* __restrict__ coef, double4a* __restrict__ force) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const typename V4<R>::T p = pos[i];
  const double q2 = (double)p.w * (double)p.w;
  const double x[3] = {(double)p.x, (double)p.y, (double)p.z};
  const int K[3] = {K0, K1, K2};
  double f[3] = {0, 0, 0};
  for (int d = 0; d < 3; ++d)
    for (int kk = 1; kk <= 3; ++kk)
      f[d] -= coef[d * 4 + kk] * q2 * sinpi(2.0 * kk * K[d] * st->Li[d] * x[d]);
  double4a F = force[i];
  F.x += f[0]; F.y += f[1]; F.z += f[2];
  force[i] = F;
}

// ---------------------------------------------------------------- host
template <class R, int LOGN>
static const void* fftp_fn_n(int mode, int sign, int out4) {
  if (mode == 0) return (const void*)k_fftp<R, LOGN, 0, -1, 0>;
  if (mode == 1) return sign < 0 ? (const void*)k_fftp<R, LOGN, 1, -1, 0> : (const void*)k_fftp<R, LOGN, 1, 1, 0>;
  return out4 ? (const void*)k_fftp<R, LOGN, 2, 1, 1> : (const void*)k_fftp<R, LOGN, 2, 1, 0>;
}

// line lengths 4 .. 1024
#define FFT_LOGNS(X) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10)

template <class R>
static const void* fftp_fn(int logn, int mode, int sign, int out4) {
  switch (logn) {
#define FFT_CASE(L) case L: return fftp_fn_n<R, L>(mode, sign, out4);
    FFT_LOGNS(FFT_CASE)
#undef FFT_CASE
  }
  return nullptr;
}

template <class R>
static const void* fftx_fn(int logn, int method) {
  switch (logn) {
#define FFT_CASE(L) \
  case L: return method == 0 ? (const void*)k_fft_x_kspace<R, L, 0> : (const void*)k_fft_x_kspace<R, L, 1>;
    FFT_LOGNS(FFT_CASE)
#undef FFT_CASE
  }
  return nullptr;
}

static int ilog2i(int k) {
  int l = 0;
  while ((1 << l) < k) ++l;
  return l;
}
static int fft_lpb(int n) { return FFT_THREADS / (n >= 8 ? n / 8 : 1); }

// one transform pass: mode 0 R2C z, 1 C2C along `axis` (0 x, 1 y), 2 C2R z
// (out4: the three batches interleaved into Real4)
template <class R>
static int fft_launch(md_spme* s, Recorder* rec, const void* in, void* out, int mode, int axis, int sign, int batch,
                      int out4) {
  const int K0 = s->K[0], K1 = s->K[1], K2 = s->K[2], K2h = s->K2h;
  int n;
  long nlines, stride = 1, inner = 1, outer = 0, in_bs = 0, out_bs = 0;
  if (mode == 0 || mode == 2) {
    axis = 2;
    n = K2; nlines = (long)K0 * K1;
    in_bs = (long)s->nhalf; out_bs = (long)s->nreal;
  } else if (axis == 1) {
    n = K1; nlines = (long)K0 * K2h; stride = K2h; inner = K2h; outer = (long)K1 * K2h;
    in_bs = out_bs = (long)s->nhalf;
  } else {
    n = K0; nlines = (long)K1 * K2h; stride = (long)K1 * K2h; inner = (long)K1 * K2h; outer = 0;
    in_bs = out_bs = (long)s->nhalf;
  }
  const int logn = ilog2i(n), lpb = fft_lpb(n);
  const size_t smem = fftp_smem<R>(logn, out4 ? 2 : 1);
  const long nlc = mode == 0 ? (nlines + 1) / 2 : nlines;  // R2C: two real lines per complex transform
  dim3 grid((unsigned)((nlc + lpb - 1) / lpb), out4 ? 1 : batch);
  const void* twg = s->tw[axis];
  void* a[] = {&in, &out, &twg, &nlines, &stride, &inner, &outer, &in_bs, &out_bs};
  return rec_launch(rec, fftp_fn<R>(logn, mode, sign, out4), grid, dim3(FFT_THREADS * (out4 ? 2 : 1)), smem, a);
}

// dynamic shared memory above the default 48 KB needs the opt-in attribute
static int smem_optin(const void* fn, size_t bytes) {
  if (bytes > 48 * 1024) MD_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return MD_OK;
}

template <class R>
static int spme_prepare(md_spme* s) {
  typedef typename C2<R>::T T2;
  cudaStream_t str = s->sys->stream;
  // the real mesh starts cleared; every z pass clears it again after reading
  MD_CUDA(cudaMemsetAsync(s->Q, 0, sizeof(R) * s->nreal, str));
  MD_CUDA(cudaMalloc(&s->frec, sizeof(double4a) * s->sys->N));
  // blocks of the x pass, or a plane each
  s->max_blocks = std::max(ceil_div((long)s->K[1] * s->K2h, fft_lpb(s->K[0])), s->K2h);
  MD_CUDA(cudaMalloc(&s->partials, sizeof(double) * 4 * s->max_blocks));
  const int nbm = s->K[0] + s->K[1] + s->K2h;
  MD_CUDA(cudaMalloc(&s->bm, sizeof(double) * nbm));
  k_spme_bmod<<<ceil_div(nbm, 256), 256, 0, str>>>(s->K[0], s->K[1], s->K[2], s->order, s->bm);
  MD_CHECK_LAUNCH("spme bmod");
  for (int d = 0; d < 3; ++d) {
    MD_CUDA(cudaMalloc(&s->tw[d], sizeof(T2) * s->K[d]));
    k_fft_twiddles<R><<<ceil_div(s->K[d], 256), 256, 0, str>>>(s->K[d], (T2*)s->tw[d]);
    MD_CHECK_LAUNCH("fft twiddles");
  }
  const int l0 = ilog2i(s->K[0]), l1 = ilog2i(s->K[1]), l2 = ilog2i(s->K[2]);
  if (int r = pm_prepare(s->sys->prec, s->order)) return r;
  s->planes = plane_chain_ok(s->sys->prec, s->K);
  if (s->planes)
    if (int r = plane_prepare(s->sys->prec, s->K, s->method)) return r;
  if (int r = smem_optin(fftp_fn<R>(l2, 0, -1, 0), fftp_smem<R>(l2, 1))) return r;
  if (int r = smem_optin(fftp_fn<R>(l2, 2, 1, 0), fftp_smem<R>(l2, 1))) return r;
  if (int r = smem_optin(fftp_fn<R>(l2, 2, 1, 1), fftp_smem<R>(l2, 2))) return r;
  for (int sg = -1; sg <= 1; sg += 2) {
    if (int r = smem_optin(fftp_fn<R>(l1, 1, sg, 0), fftp_smem<R>(l1, 1))) return r;
    if (int r = smem_optin(fftp_fn<R>(l0, 1, sg, 0), fftp_smem<R>(l0, 1))) return r;
  }
  if (int r = smem_optin(fftx_fn<R>(l0, s->method), fftx_smem<R>(l0, s->method))) return r;
  return MD_OK;
}

// stored influence function psi, refreshed only when the box changed
// (adjoint and md_spme_get_influence; the force chain evaluates psi in its
// x pass)
template <class R>
static int influence_launch(md_spme* s, Recorder* rec) {
  int K0 = s->K[0], K1 = s->K[1], K2 = s->K[2], n = s->order;
  R* psi = (R*)s->psi;
  DevState* st = s->sys->st;
  double beta = s->beta;
  {
    void* a[] = {&K0, &K1, &K2, &n, &beta, &st, &psi, &s->d_box_tab};
    if (int r = rec_launch(rec, (const void*)k_spme_influence<R>, dim3((unsigned)((s->nhalf + 255) / 256)),
                           dim3(256), 0, a)) return r;
  }
  void* a[] = {&st, &s->d_box_tab};
  return rec_launch(rec, (const void*)k_spme_box_tab, dim3(1), dim3(1), 0, a);
}

// spread and the forward transform along z (which clears the real mesh for
// the next spread), y and (with_x) x: C[0] = Q^ on the half spectrum.  Every
// launch goes through the recorder, so the chain is either run on the stream
// or recorded into the step graph of the simulation driver.
template <class R>
static int spme_forward_mesh(md_spme* s, Recorder* rec, bool with_x) {
  typedef typename C2<R>::T T2;
  R* Q = (R*)s->Q;
  T2* C = (T2*)s->C;
  if (int r = pm_spread(s->sys, s->K, s->order, Q, rec)) return r;
  if (int r = fft_launch<R>(s, rec, Q, C, 0, 2, -1, 1, 0)) return r;
  if (int r = fft_launch<R>(s, rec, C, C, 1, 1, -1, 1, 0)) return r;
  if (with_x)
    if (int r = fft_launch<R>(s, rec, C, C, 1, 0, -1, 1, 0)) return r;
  return MD_OK;
}

static PlaneChain plane_args(md_spme* s, int method) {
  PlaneChain p;
  p.n = s->K[0];
  p.K2 = s->K[2];
  p.method = method;
  p.Q = s->Q;
  p.C = s->C;
  p.G = s->G;
  p.bm = s->bm;
  p.tw_n = s->tw[0];
  p.tw_z = s->tw[2];
  p.beta = s->beta;
  p.partials = s->partials;
  p.with_stats = 1;
  p.merge = 0;
  p.back = 1;
  p.energy = p.dbeta = nullptr;
  return p;
}

template <class R>
static int spme_run(md_spme* s, bool with_stats, Recorder* rec, bool concurrent) {
  typedef typename C2<R>::T T2;
  md_system* sys = s->sys;
  int K1 = s->K[1], K2 = s->K[2], method = s->method;
  T2* C = (T2*)s->C;
  DevState* st = sys->st;
  if (s->planes) {
    PlaneChain p = plane_args(s, method);
    p.with_stats = with_stats ? 1 : 0;
    p.merge = concurrent ? 0 : 1;
    if (int r = pm_spread(sys, s->K, s->order, s->Q, rec)) return r;
    if (int r = plane_chain(sys, p, rec)) return r;
    return pm_gather(sys, s->K, s->order, method, s->G, concurrent ? s->frec : sys->force, concurrent ? 1 : 0, rec);
  }
  if (int r = spme_forward_mesh<R>(s, rec, false)) return r;
  const int l0 = ilog2i(s->K[0]);
  const int nb = ceil_div((long)K1 * s->K2h, fft_lpb(s->K[0]));
  if (with_stats && nb > s->max_blocks) { md_set_error("partials buffer too small for the mesh"); return MD_ERR_BADARG; }
  {
    double beta = s->beta;
    const void* twg = s->tw[0];
    int ws = with_stats ? 1 : 0, merge = concurrent ? 0 : 1;
    void* a[] = {&C, &twg, &s->bm, &K1, &K2, &beta, &st, &s->partials, &ws, &merge};
    if (int r = rec_launch(rec, fftx_fn<R>(l0, method), dim3(nb), dim3(FFT_THREADS * (method == 0 ? 2 : 1)),
                           fftx_smem<R>(l0, method), a)) return r;
  }
  const int nconv = method == 0 ? 3 : 1;
  T2* Cp = C + s->nhalf;
  if (int r = fft_launch<R>(s, rec, Cp, Cp, 1, 1, +1, nconv, 0)) return r;
  if (int r = fft_launch<R>(s, rec, Cp, s->G, 2, 2, +1, nconv, method == 0 ? 1 : 0)) return r;
  return pm_gather(sys, s->K, s->order, method, s->G, concurrent ? s->frec : sys->force, concurrent ? 1 : 0, rec);
}

bool spme_belongs_to(const md_spme* s, const md_system* sys) { return s && s->sys == sys; }

// the chain of one SPME force evaluation, recorded (driver) or launched
int spme_apply_impl(md_spme* s, bool with_stats, Recorder* rec, bool concurrent) {
  return s->sys->prec == MD_PREC_FP64 ? spme_run<double>(s, with_stats, rec, concurrent)
                                      : spme_run<float>(s, with_stats, rec, concurrent);
}

const double4a* spme_force_buffer(const md_spme* s) { return s->frec; }

// energy and gradient: recompute the mesh and its transform, influence
// multiply (energy, dE/dbeta, dE/dpsi), one inverse transform to Phi, gather
__global__ void k_adj_out(const DevState* st, double* energy, double* dbeta) {
  if (energy) *energy = st->scratch[0];
  if (dbeta) *dbeta = st->scratch[1];
}

// dev = true: energy, dq, dr, dbeta are device pointers the results are left
// in (no host copy, no wait); dpsi must then be NULL
template <class R>
static int spme_energy_grad(md_spme* s, double* energy, double* dq, double* dr, double* dbeta, double* dpsi,
                            bool dev = false) {
  typedef typename C2<R>::T T2;
  md_system* sys = s->sys;
  cudaStream_t st_ = sys->stream;
  const int K0 = s->K[0], K1 = s->K[1], K2 = s->K[2];
  T2* C = (T2*)s->C;
  const int nb = (int)((s->nhalf + 255) / 256);
  if (nb > sys->max_partial_blocks) { md_set_error("partials buffer too small for the mesh"); return MD_ERR_BADARG; }
  // device outputs: dq [N], dr [N][3], dpsi [nhalf] (FP64, caller's atom order)
  const size_t nq = dq ? (size_t)sys->N : 0, nr = dr ? 3 * (size_t)sys->N : 0, np = dpsi ? s->nhalf : 0;
  double* d = nullptr;
  if (!dev && nq + nr + np) MD_CUDA(cudaMallocAsync((void**)&d, sizeof(double) * (nq + nr + np), st_));
  double* d_q = dev ? dq : (dq ? d : nullptr);
  double* d_r = dev ? dr : (dr ? d + nq : nullptr);
  double* d_p = dev ? nullptr : (dpsi ? d + nq + nr : nullptr);
  Recorder rec;
  rec.stream = st_;
  const bool planes = s->planes && !dpsi;
  if (planes) {
    // energy and dE/dbeta leave the plane pass for their device outputs
    PlaneChain p = plane_args(s, 2);
    p.back = dq || dr;
    if (dev) {
      p.energy = energy;
      p.dbeta = dbeta;
    }
    if (int r = pm_spread(sys, s->K, s->order, s->Q, &rec)) return r;
    if (int r = plane_chain(sys, p, &rec)) return r;
    if (dq || dr)
      if (int r = pm_gather_adjoint(sys, s->K, s->order, s->G, d_q, d_r, &rec)) return r;
    if (dev) return MD_OK;
  }
  if (!planes) {
    if (int r = influence_launch<R>(s, &rec)) return r;
    if (int r = spme_forward_mesh<R>(s, &rec, true)) return r;
    k_spme_adj_kspace<R><<<nb, 256, 0, st_>>>(K0, K1, K2, s->beta, (const R*)s->psi, C, s->nhalf, sys->st,
                                               sys->partials, d_p);
    MD_CHECK_LAUNCH("spme adjoint kspace");
    if (dq || dr) {
      T2* Cp = C + s->nhalf;
      if (int r = fft_launch<R>(s, &rec, Cp, Cp, 1, 0, +1, 1, 0)) return r;
      if (int r = fft_launch<R>(s, &rec, Cp, Cp, 1, 1, +1, 1, 0)) return r;
      if (int r = fft_launch<R>(s, &rec, Cp, s->G, 2, 2, +1, 1, 0)) return r;
      if (int r = pm_gather_adjoint(sys, s->K, s->order, s->G, d_q, d_r, &rec)) return r;
    }
  }
  if (dev) {
    k_adj_out<<<1, 1, 0, st_>>>(sys->st, energy, dbeta);
    MD_CHECK_LAUNCH("spme adjoint out");
    return MD_OK;
  }
  double red[2];
  MD_CUDA(cudaMemcpyAsync(red, sys->st->scratch, sizeof(red), cudaMemcpyDeviceToHost, st_));
  if (dq) MD_CUDA(cudaMemcpyAsync(dq, d_q, sizeof(double) * nq, cudaMemcpyDeviceToHost, st_));
  if (dr) MD_CUDA(cudaMemcpyAsync(dr, d_r, sizeof(double) * nr, cudaMemcpyDeviceToHost, st_));
  if (dpsi) MD_CUDA(cudaMemcpyAsync(dpsi, d_p, sizeof(double) * np, cudaMemcpyDeviceToHost, st_));
  if (d) MD_CUDA(cudaFreeAsync(d, st_));
  MD_CUDA(cudaStreamSynchronize(st_));
  if (energy) *energy = red[0];
  if (dbeta) *dbeta = red[1];
  return MD_OK;
}

static bool pow2(int k) { return k >= 2 && (k & (k - 1)) == 0; }

extern "C" int md_spme_create(md_spme** out, md_system* sys, const int K[3], int order, double beta, int method) {
  if (!out || !sys || !K || order < 2 || order > 14 || !(beta > 0) || (method != 0 && method != 1)) {
    md_set_error("md_spme_create: bad arguments");
    return MD_ERR_BADARG;
  }
  for (int d = 0; d < 3; ++d)
    if (!pow2(K[d]) || K[d] > 1024 || K[d] <= order) {
      md_set_error("md_spme_create: mesh sizes must be powers of two in (order, 1024]");
      return MD_ERR_BADARG;
    }
  md_spme* s = new md_spme();
  s->sys = sys;
  for (int d = 0; d < 3; ++d) s->K[d] = K[d];
  s->K2h = K[2] / 2 + 1;
  s->order = order;
  s->beta = beta;
  s->method = method;
  s->nreal = (size_t)K[0] * K[1] * K[2];
  s->nhalf = (size_t)K[0] * K[1] * s->K2h;
  const size_t rs = sys->real_size();
  // G: ik Real4 per mesh point (the adjoint's single mesh fits as well)
  bool ok = cudaMalloc(&s->Q, rs * s->nreal) == cudaSuccess &&
            cudaMalloc(&s->C, 2 * rs * s->nhalf * 4) == cudaSuccess &&
            cudaMalloc(&s->G, sys->r4_size() * s->nreal) == cudaSuccess &&
            cudaMalloc(&s->psi, rs * s->nhalf) == cudaSuccess &&
            cudaMalloc(&s->d_box_tab, sizeof(double) * 3) == cudaSuccess &&
            cudaMemsetAsync(s->d_box_tab, 0, sizeof(double) * 3, sys->stream) == cudaSuccess;
  if (!ok) {
    md_cuda_fail(cudaGetLastError(), "md_spme_create");
    md_spme_destroy(s);
    return MD_ERR_CUDA;
  }
  if (int r = sys->prec == MD_PREC_FP64 ? spme_prepare<double>(s) : spme_prepare<float>(s)) {
    md_spme_destroy(s);
    return r;
  }
  *out = s;
  return MD_OK;
}

extern "C" int md_spme_destroy(md_spme* s) {
  if (!s) return MD_OK;
  void* p[] = {s->Q, s->C, s->G, s->psi, s->d_box_tab, s->tw[0], s->tw[1], s->tw[2], s->bm, s->frec, s->partials};
  for (void* q : p) if (q) cudaFree(q);
  delete s;
  return MD_OK;
}

extern "C" int md_spme_apply(md_spme* s, md_system* sys, int with_stats) {
  if (!s || !sys || sys != s->sys) { md_set_error("md_spme_apply: bad arguments"); return MD_ERR_BADARG; }
  Recorder rec;
  rec.stream = sys->stream;
  return spme_apply_impl(s, with_stats != 0, &rec);
}

// the same with DEVICE outputs (energy and dE_dbeta one double each, dE_dq [N],
// dE_dr [N][3], caller's atom order), asynchronous on the system's stream
extern "C" int md_spme_energy_grad_device(md_spme* s, md_system* sys, double* energy, double* dE_dq, double* dE_dr,
                                          double* dE_dbeta) {
  if (!s || !sys || sys != s->sys) { md_set_error("md_spme_energy_grad_device: bad arguments"); return MD_ERR_BADARG; }
  return sys->prec == MD_PREC_FP64 ? spme_energy_grad<double>(s, energy, dE_dq, dE_dr, dE_dbeta, nullptr, true)
                                   : spme_energy_grad<float>(s, energy, dE_dq, dE_dr, dE_dbeta, nullptr, true);
}

extern "C" int md_spme_energy_grad(md_spme* s, md_system* sys, double* energy, double* dE_dq, double* dE_dr,
                                   double* dE_dbeta, double* dE_dpsi) {
  if (!s || !sys || sys != s->sys) { md_set_error("md_spme_energy_grad: bad arguments"); return MD_ERR_BADARG; }
  return sys->prec == MD_PREC_FP64 ? spme_energy_grad<double>(s, energy, dE_dq, dE_dr, dE_dbeta, dE_dpsi)
                                   : spme_energy_grad<float>(s, energy, dE_dq, dE_dr, dE_dbeta, dE_dpsi);
}

__global__ void k_mesh_out(size_t n, const float* a, const double* b, double* out);

extern "C" int md_spme_self_correction(md_spme* s, md_system* sys) {
  if (!s || !sys || sys != s->sys) { md_set_error("md_spme_self_correction: bad arguments"); return MD_ERR_BADARG; }
  const int Kmax = std::max(s->K[0], std::max(s->K[1], s->K[2]));
  double* d = nullptr;
  MD_CUDA(cudaMallocAsync((void**)&d, sizeof(double) * (3 * Kmax + 12), sys->stream));
  k_selfcorr_weights<<<dim3(Kmax, 3), 256, 0, sys->stream>>>(s->K[0], s->K[1], s->K[2], s->beta, sys->st, d, Kmax);
  MD_CHECK_LAUNCH("selfcorr weights");
  k_selfcorr_coef<<<1, 9 * 32, 0, sys->stream>>>(s->K[0], s->K[1], s->K[2], s->order, sys->st, d, Kmax,
                                                 d + 3 * Kmax);
  MD_CHECK_LAUNCH("selfcorr coef");
  const int nb = ceil_div(sys->N, 256);
  if (sys->prec == MD_PREC_FP64)
    k_selfcorr_apply<double><<<nb, 256, 0, sys->stream>>>(sys->N, (const double4a*)sys->pos, s->K[0], s->K[1],
                                                           s->K[2], sys->st, d + 3 * Kmax, sys->force);
  else
    k_selfcorr_apply<float><<<nb, 256, 0, sys->stream>>>(sys->N, (const float4*)sys->pos, s->K[0], s->K[1],
                                                         s->K[2], sys->st, d + 3 * Kmax, sys->force);
  MD_CHECK_LAUNCH("selfcorr apply");
  MD_CUDA(cudaFreeAsync(d, sys->stream));
  return MD_OK;
}

extern "C" int md_spme_get_influence(md_spme* s, double* psi) {
  if (!s || !psi) return MD_ERR_BADARG;
  md_system* sys = s->sys;
  Recorder rec;
  rec.stream = sys->stream;
  if (int r = sys->prec == MD_PREC_FP64 ? influence_launch<double>(s, &rec) : influence_launch<float>(s, &rec))
    return r;
  double* d = nullptr;
  MD_CUDA(cudaMallocAsync((void**)&d, sizeof(double) * s->nhalf, sys->stream));
  const bool f = sys->prec != MD_PREC_FP64;
  k_mesh_out<<<(unsigned)((s->nhalf + 255) / 256), 256, 0, sys->stream>>>(
      s->nhalf, f ? (const float*)s->psi : nullptr, f ? nullptr : (const double*)s->psi, d);
  MD_CHECK_LAUNCH("influence out");
  MD_CUDA(cudaMemcpyAsync(psi, d, sizeof(double) * s->nhalf, cudaMemcpyDeviceToHost, sys->stream));
  MD_CUDA(cudaFreeAsync(d, sys->stream));
  MD_CUDA(cudaStreamSynchronize(sys->stream));
  return MD_OK;
}

__global__ void k_mesh_out(size_t n, const float* a, const double* b, double* out) {
  size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (t < n) out[t] = a ? (double)a[t] : b[t];
}

// the charge mesh of the current positions: spread onto the cleared mesh,
// copied out, and cleared again for the next force evaluation
extern "C" int md_spme_get_mesh(md_spme* s, double* Q) {
  if (!s || !Q) return MD_ERR_BADARG;
  md_system* sys = s->sys;
  Recorder rec;
  rec.stream = sys->stream;
  const bool f = sys->prec != MD_PREC_FP64;
  if (int r = pm_spread(sys, s->K, s->order, s->Q, &rec)) return r;
  double* d = nullptr;
  MD_CUDA(cudaMallocAsync((void**)&d, sizeof(double) * s->nreal, sys->stream));
  k_mesh_out<<<(unsigned)((s->nreal + 255) / 256), 256, 0, sys->stream>>>(
      s->nreal, f ? (const float*)s->Q : nullptr, f ? nullptr : (const double*)s->Q, d);
  MD_CHECK_LAUNCH("mesh out");
  MD_CUDA(cudaMemsetAsync(s->Q, 0, sys->real_size() * s->nreal, sys->stream));
  MD_CUDA(cudaMemcpyAsync(Q, d, sizeof(double) * s->nreal, cudaMemcpyDeviceToHost, sys->stream));
  MD_CUDA(cudaFreeAsync(d, sys->stream));
  MD_CUDA(cudaStreamSynchronize(sys->stream));
  return MD_OK;
}

__global__ void k_self_energy(int N, const float4* pf, const double4a* pd, int prec, double beta, DevState* st,
                              double* partials) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double v[1] = {0};
  if (i < N) {
    const double q = prec == MD_PREC_FP64 ? pd[i].w : (double)pf[i].w;
    v[0] = -beta / sqrt(M_PI) * q * q;
  }
  block_reduce_finish<1>(v, partials, &st->red_counter[RED_MISC], &st->stats[MD_STAT_ELEC_SELF], true);
}

extern "C" int md_ewald_self_energy(md_system* sys, double beta, double* out) {
  if (!sys || !(beta > 0)) return MD_ERR_BADARG;
  k_self_energy<<<ceil_div(sys->N, 256), 256, 0, sys->stream>>>(sys->N, (float4*)sys->pos, (double4a*)sys->pos,
                                                                 sys->prec, beta, sys->st, sys->partials);
  MD_CHECK_LAUNCH("self energy");
  if (out) {
    DevState hs;
    if (int r = sys->read_state(hs)) return r;
    *out = hs.stats[MD_STAT_ELEC_SELF];
  }
  return MD_OK;
}

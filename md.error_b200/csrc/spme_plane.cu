// The SPME chain's transforms for meshes with equal power-of-two x and y sizes
// n (16 to 128 in binary32, to 64 in binary64), in three passes:
//   z forward   real lines -> half spectra, written transposed, [k_z][x][y]
//   plane       one block per k_z holds the n x n plane in shared memory:
//               forward along y and x, the k-space step (psi, energy and
//               virial in FP64), and the inverse transforms of all products
//   z backward  half spectra -> real lines, the mesh [x][y][z]
// against one pass over memory per axis and direction (spme.cu, which keeps
// the other meshes): the half spectrum is read once and each product written
// once between the two z passes.  ik writes three products, phi_x, phi_y and
// P = xy-inverse of psi Q^, from seven sets of line transforms: m_y is constant
// along x, so phi_y and P share the inverse along x, and m_z is constant in
// the plane, so the z pass forms phi_z = -2 pi i m_z P from P itself.
//
// Lines of a plane are transformed in place in two stages, n = A 8 (A = n / 8):
// forward by decimation in frequency, which leaves frequency k1 + A k2 at
// position 8 k1 + k2, inverse by decimation in time from that order, so no
// stage reorders and a stage costs one barrier.  Lanes of a warp hold the same
// butterfly of different lines: twiddles are broadcasts, and with the odd row
// stride n + 1 neither direction has bank conflicts.  Bound: shared-memory
// bandwidth (four accesses per point and set) and FP64 issue in the k-space
// step; a 128 x 128 plane fills an SM (131 KB), so its blocks do not overlap.
// Transforms and k space, ik, binary32: 128x128x512 372 us as passes per axis,
// 207 by planes (z 25, plane 97, z back 85); 64^3 28 and 18; binary64 64^3 99 and
// 50 with spread and gather.  Binary64 planes of 128 x 128 do not fit an SM and
// keep the passes; so do axes of unequal size.
#include <algorithm>
#include "fft_lines.cuh"
#include "spme_plane.cuh"

namespace {

template <class R, int SIGN>
__device__ __forceinline__ void dft16(typename C2<R>::T (&v)[16]) {
  typedef typename C2<R>::T T2;
  // r = 4 r1 + r2, k = k1 + 4 k2
#pragma unroll
  for (int r2 = 0; r2 < 4; ++r2) dft4<SIGN>(v[r2], v[4 + r2], v[8 + r2], v[12 + r2]);
  const R c1 = R(0.92387953251128675613), s1 = R(0.38268343236508977173), h = R(0.70710678118654752440);
  const R cs[10] = {1, c1, h, s1, 0, -s1, -h, -c1, -1, -c1}, sn[10] = {0, s1, h, c1, 1, c1, h, s1, 0, -s1};
#pragma unroll
  for (int k1 = 1; k1 < 4; ++k1)
#pragma unroll
    for (int r2 = 1; r2 < 4; ++r2) {
      T2 w;
      w.x = cs[k1 * r2];
      w.y = SIGN > 0 ? sn[k1 * r2] : -sn[k1 * r2];
      v[4 * k1 + r2] = cmul(v[4 * k1 + r2], w);
    }
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) dft4<SIGN>(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);
  T2 o[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) o[k] = v[4 * (k & 3) + (k >> 2)];
#pragma unroll
  for (int k = 0; k < 16; ++k) v[k] = o[k];
}

template <class R, int RR, int SIGN>
__device__ __forceinline__ void dft_any(typename C2<R>::T (&v)[RR]) {
  if constexpr (RR == 16) dft16<R, SIGN>(v);
  else dft_reg<R, RR, SIGN>(v);
}

template <int LOGN>
struct PlaneGeom {
  static constexpr int n = 1 << LOGN, A = n / 8, LS = n + 1;
  static constexpr int T = LOGN <= 5 ? 128 : 512;  // threads per plane
  static constexpr int EPT = n * n / T;
};

// point p of line l: along y (DIR 0) or x (DIR 1)
template <int LS, int DIR>
__device__ __forceinline__ int plane_at(int l, int p) { return DIR == 0 ? l * LS + p : p * LS + l; }

// A-point transforms over the points j + 8 r of every line (r = 0..A-1)
template <class R, int LOGN, int DIR, int SIGN, bool TWIDDLE>
__device__ __forceinline__ void plane_stage_a(typename C2<R>::T* X, const typename C2<R>::T* tw) {
  typedef PlaneGeom<LOGN> P;
  typedef typename C2<R>::T T2;
  constexpr int n = P::n, A = P::A;
#pragma unroll 1  // one 16-point transform's registers at a time
  for (int t0 = 0; t0 < 8 * n; t0 += P::T) {
    const int t = t0 + threadIdx.x;
    if (8 * n % P::T != 0 && t >= 8 * n) break;
    const int l = t & (n - 1), j = t >> LOGN;
    T2 v[A];
#pragma unroll
    for (int r = 0; r < A; ++r) v[r] = X[plane_at<P::LS, DIR>(l, j + 8 * r)];
    dft_any<R, A, SIGN>(v);
#pragma unroll
    for (int r = 0; r < A; ++r) {
      if (TWIDDLE && r > 0) {
        T2 w = tw[j * r];
        if (SIGN > 0) w.y = -w.y;
        v[r] = cmul(v[r], w);
      }
      X[plane_at<P::LS, DIR>(l, j + 8 * r)] = v[r];
    }
  }
  __syncthreads();
}

// 8-point transforms over the points 8 k1 + j of every line (j = 0..7)
template <class R, int LOGN, int DIR, int SIGN, bool TWIDDLE>
__device__ __forceinline__ void plane_stage_b(typename C2<R>::T* X, const typename C2<R>::T* tw) {
  typedef PlaneGeom<LOGN> P;
  typedef typename C2<R>::T T2;
  constexpr int n = P::n, A = P::A;
#pragma unroll 1
  for (int t0 = 0; t0 < A * n; t0 += P::T) {
    const int t = t0 + threadIdx.x;
    if (A * n % P::T != 0 && t >= A * n) break;
    const int l = t & (n - 1), k1 = t >> LOGN;
    T2 v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = X[plane_at<P::LS, DIR>(l, 8 * k1 + j)];
    dft_reg<R, 8, SIGN>(v);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (TWIDDLE && j > 0) {
        T2 w = tw[j * k1];
        if (SIGN > 0) w.y = -w.y;
        v[j] = cmul(v[j], w);
      }
      X[plane_at<P::LS, DIR>(l, 8 * k1 + j)] = v[j];
    }
  }
  __syncthreads();
}

template <class R, int LOGN, int DIR>
__device__ __forceinline__ void plane_forward(typename C2<R>::T* X, const typename C2<R>::T* tw) {
  plane_stage_a<R, LOGN, DIR, -1, true>(X, tw);
  plane_stage_b<R, LOGN, DIR, -1, false>(X, tw);
}
template <class R, int LOGN, int DIR>
__device__ __forceinline__ void plane_inverse(typename C2<R>::T* X, const typename C2<R>::T* tw) {
  plane_stage_b<R, LOGN, DIR, 1, true>(X, tw);
  plane_stage_a<R, LOGN, DIR, 1, false>(X, tw);
}

template <class R, int LOGN>
constexpr size_t plane_smem() {
  typedef PlaneGeom<LOGN> P;
  return sizeof(double) * 4 * P::n + sizeof(typename C2<R>::T) * (P::n + (size_t)P::n * P::LS);
}

// METHOD 0: C[1] = -2 pi i m_x psi Q^, C[2] = -2 pi i m_y psi Q^, C[3] = psi Q^;
// 1: C[1] = psi Q^ / 2 (FBSpline normalisation); 2: C[1] = psi Q^; each
// transformed back along x and y (2: only with back).  psi = exp(-pi^2 m^2 / beta^2) / m^2
// |b0|^2 |b1|^2 |b2|^2 / (pi V) (calB / calPsiFPhiF) from factors per axis, for the
// current box.  The energy E = 1/2 sum psi |Q^|^2 with the diagonal virial
// (METHODS 0, 1) or dE/dbeta (2) is reduced in FP64.
template <class R, int LOGN, int METHOD>
__global__ void __launch_bounds__(PlaneGeom<LOGN>::T)
k_spme_plane(typename C2<R>::T* C, const typename C2<R>::T* __restrict__ twg, const double* __restrict__ bm, int K2,
             double beta, DevState* st, double* partials, int with_stats, int merge, int back, double* energy, double* dbeta) {
  typedef PlaneGeom<LOGN> P;
  typedef typename C2<R>::T T2;
  constexpr int n = P::n, T = P::T, EPT = P::EPT, NS = METHOD == 0 ? EPT : 1;
  // ik with fewer planes than half the SMs: two blocks per plane, one for phi_x
  // (and the sums), one for phi_y and P
  const bool first = blockIdx.y == 0, second = gridDim.y == 1 || blockIdx.y == 1;
  with_stats = with_stats && first;
  extern __shared__ __align__(16) unsigned char pl_smem[];
  double* EX = reinterpret_cast<double*>(pl_smem);  // by position: factor and m of the frequency there
  double *MX = EX + n, *EY = MX + n, *MY = EY + n;
  T2* tw = reinterpret_cast<T2*>(MY + n);
  T2* X = tw + n;
  const int kz = blockIdx.x;
  const size_t nhalf = (size_t)n * n * (K2 / 2 + 1), base = (size_t)kz * n * n;
  const double sc = M_PI * M_PI / (beta * beta), V = st->L[0] * st->L[1] * st->L[2], mz = kz * st->Li[2];
#pragma unroll
  for (int s = 0; s < EPT; ++s) {
    const int e = threadIdx.x + s * T;
    X[(e >> LOGN) * P::LS + (e & (n - 1))] = C[base + e];
  }
  for (int t = threadIdx.x; t < 2 * n; t += T) {
    const int d = t >> LOGN, p = t & (n - 1), k = (p >> 3) + P::A * (p & 7), kc = k <= n / 2 ? k : k - n;
    const double m = kc * st->Li[d];
    (d ? MY : MX)[p] = m;
    (d ? EY : EX)[p] = exp(-sc * m * m) * bm[d * n + k];
  }
  for (int t = threadIdx.x; t < n; t += T) tw[t] = twg[t];
  const double ez = exp(-sc * mz * mz) * bm[2 * n + kz] / (M_PI * V);
  __syncthreads();
  plane_forward<R, LOGN, 0>(X, tw);
  plane_forward<R, LOGN, 1>(X, tw);
  // interior z planes of the half spectrum stand for two modes
  const double wgt = (kz == 0 || 2 * kz == K2) ? 0.5 : 1.0;
  double v[METHOD == 2 ? 2 : 4] = {};
  T2 S[NS];  // psi Q^, for the second product
#pragma unroll
  for (int s = 0; s < EPT; ++s) {
    const int e = threadIdx.x + s * T, px = e >> LOGN, py = e & (n - 1);
    T2* x = X + px * P::LS + py;
    const T2 q = *x;
    const double mx = MX[px], my = MY[py], mm = mx * mx + my * my + mz * mz;
    const double inv = mm != 0.0 ? 1.0 / mm : 0.0;
    const R ps = (R)(EX[px] * EY[py] * ez * inv);
    if (with_stats) {
      const double e2 = wgt * ((double)q.x * q.x + (double)q.y * q.y) * (double)ps;
      v[0] += e2;
      if constexpr (METHOD == 2) {
        v[1] += e2 * 2.0 * M_PI * M_PI * mm / (beta * beta * beta);
      } else {
        // pressure tensor V P_aa = sum_m E_m (1 - f m_a^2), f = 2 (1 + pi^2 m^2 / beta^2) / m^2;
        // the virial slots hold W_aa = -V P_aa
        const double f = 2.0 * inv + 2.0 * sc;
        if (mm != 0.0) {
          v[1] -= e2 * (1.0 - f * mx * mx);
          v[2] -= e2 * (1.0 - f * my * my);
          v[3] -= e2 * (1.0 - f * mz * mz);
        }
      }
    }
    T2 g;
    g.x = q.x * ps;
    g.y = q.y * ps;
    if constexpr (METHOD == 0) {
      S[s] = g;
      const R c = (R)(-2.0 * M_PI * mx);
      x->x = -g.y * c;
      x->y = g.x * c;
    } else if constexpr (METHOD == 1) {
      x->x = R(0.5) * g.x;
      x->y = R(0.5) * g.y;
    } else {
      *x = g;
    }
  }
  __syncthreads();
  if (first && (METHOD != 2 || back)) {
    plane_inverse<R, LOGN, 1>(X, tw);
    plane_inverse<R, LOGN, 0>(X, tw);
#pragma unroll
    for (int s = 0; s < EPT; ++s) {
      const int e = threadIdx.x + s * T;
      C[nhalf + base + e] = X[(e >> LOGN) * P::LS + (e & (n - 1))];
    }
  }
  if (METHOD == 0 && second) {
    __syncthreads();
#pragma unroll
    for (int s = 0; s < EPT; ++s) {
      const int e = threadIdx.x + s * T;
      X[(e >> LOGN) * P::LS + (e & (n - 1))] = S[s];
    }
    __syncthreads();
    plane_inverse<R, LOGN, 1>(X, tw);
    // along y the products are still in frequency order: phi_y from a copy
#pragma unroll
    for (int s = 0; s < EPT; ++s) {
      const int e = threadIdx.x + s * T;
      S[s] = X[(e >> LOGN) * P::LS + (e & (n - 1))];
    }
    __syncthreads();
    plane_inverse<R, LOGN, 0>(X, tw);
#pragma unroll
    for (int s = 0; s < EPT; ++s) {
      const int e = threadIdx.x + s * T, py = e & (n - 1);
      T2* x = X + (e >> LOGN) * P::LS + py;
      C[3 * nhalf + base + e] = *x;
      const R c = (R)(-2.0 * M_PI * MY[py]);
      x->x = -S[s].y * c;
      x->y = S[s].x * c;
    }
    __syncthreads();
    plane_inverse<R, LOGN, 0>(X, tw);
#pragma unroll
    for (int s = 0; s < EPT; ++s) {
      const int e = threadIdx.x + s * T;
      C[2 * nhalf + base + e] = X[(e >> LOGN) * P::LS + (e & (n - 1))];
    }
  }
  if (!with_stats) return;
  if constexpr (METHOD == 2) {
    if (block_reduce_finish<2>(v, partials, &st->red_counter[RED_SPME], st->scratch, true)) {
      if (energy) *energy = st->scratch[0];
      if (dbeta) *dbeta = st->scratch[1];
    }
  } else if (block_reduce_finish<4>(v, partials, &st->red_counter[RED_SPME], st->scratch, true) && merge) {
    // reciprocal energy into its slot, its diagonal virial added to the virial slots
    st->stats[MD_STAT_ELEC_REC] = st->scratch[0];
    for (int d = 0; d < 3; ++d) st->stats[MD_STAT_VIRIAL_XX + d] += st->scratch[1 + d];
  }
}

// complex lines of a z pass block: 1,024 points, 2,048 from 512 on, so that the
// transposed accesses still cover whole 32-byte sectors
template <int LOGN>
struct ZGeom {
  static constexpr int n = 1 << LOGN, TPL = n >= 8 ? n / 8 : 1, LS = fft_line_stride(n), nh = n / 2 + 1;
  static constexpr int NC = (LOGN >= 9 ? 512 : 128) / TPL;  // complex lines
  static constexpr int T = NC * TPL;
  // ik backward: LR real lines as LR + LR / 2 complex ones
  static constexpr int LR = LOGN >= 7 ? (LOGN == 10 ? 2 : 256 / TPL) : LOGN >= 5 ? 128 / TPL : 64;
  static constexpr int TB = LR * 3 / 2 * TPL;
};

// pairs of values at an even index
template <class R>
struct alignas(4 * sizeof(R) > 16 ? 16 : 4 * sizeof(R)) Pair {
  typename C2<R>::T a, b;
};

// real lines 2l and 2l + 1 as the real and imaginary parts of one complex
// line, separated after the transform; the half spectra go to [k][line]
template <class R, int LOGN>
__global__ void __launch_bounds__(ZGeom<LOGN>::T)
k_spme_z_forward(R* __restrict__ Q, typename C2<R>::T* __restrict__ out, const typename C2<R>::T* __restrict__ twg,
                 long nlines) {
  typedef ZGeom<LOGN> Z;
  typedef typename C2<R>::T T2;
  constexpr int n = Z::n, NC = Z::NC, LS = Z::LS, EPT = NC * n / Z::T;
  extern __shared__ __align__(16) unsigned char z_smem[];
  T2* tw = reinterpret_cast<T2*>(z_smem);
  T2* X = tw + n;
  const long c0 = (long)blockIdx.x * NC;
  R* src = Q + 2 * c0 * n;
  T2 v[EPT];
#pragma unroll
  for (int s = 0; s < EPT; ++s) {
    const int e = threadIdx.x + s * Z::T, l = e >> LOGN, k = e & (n - 1);
    v[s].x = src[(2 * l) * n + k];
    v[s].y = src[(2 * l + 1) * n + k];
  }
  load_tw<R, -1>(tw, twg, n);
#pragma unroll
  for (int s = 0; s < EPT; ++s) {
    const int e = threadIdx.x + s * Z::T, l = e >> LOGN, k = e & (n - 1);
    X[l * LS + fft_pad<R>(k)] = v[s];
    src[(2 * l) * n + k] = R(0);  // the mesh is consumed: cleared for the next spread
    src[(2 * l + 1) * n + k] = R(0);
  }
  __syncthreads();
  fft_stages<R, LOGN, 0, -1>(X + (threadIdx.x / Z::TPL) * LS, tw, threadIdx.x % Z::TPL);
  for (int e = threadIdx.x; e < NC * Z::nh; e += Z::T) {
    const int l = e % NC, k = e / NC;
    const T2 z = X[l * LS + fft_pad<R>(k)], w = X[l * LS + fft_pad<R>((n - k) & (n - 1))];
    Pair<R> o;
    o.a.x = R(0.5) * (z.x + w.x);
    o.a.y = R(0.5) * (z.y - w.y);
    o.b.x = R(0.5) * (z.y + w.y);
    o.b.y = R(0.5) * (w.x - z.x);
    *reinterpret_cast<Pair<R>*>(out + k * nlines + 2 * (c0 + l)) = o;
  }
}

// sets points k and n - k of the complex line whose real and imaginary parts
// are the real lines with half spectra a and b; a real transform ignores the
// imaginary parts at k = 0 and n / 2, which would cross into the other line
template <class R, int LOGN>
__device__ __forceinline__ void set_pair(typename C2<R>::T* x, int k, typename C2<R>::T a, typename C2<R>::T b) {
  constexpr int n = 1 << LOGN;
  typename C2<R>::T z;
  if (k == 0 || k == n / 2) {
    z.x = a.x;
    z.y = b.x;
    x[fft_pad<R>(k)] = z;
    return;
  }
  z.x = a.x - b.y;
  z.y = a.y + b.x;
  x[fft_pad<R>(k)] = z;
  z.x = a.x + b.y;
  z.y = b.x - a.y;
  x[fft_pad<R>(n - k)] = z;
}

// ik: phi_x + i phi_y of each line, and phi_z = -2 pi i m_z P of two lines as one
template <class R, int LOGN>
__global__ void __launch_bounds__(ZGeom<LOGN>::TB)
k_spme_z_backward_ik(const typename C2<R>::T* __restrict__ in, typename V4<R>::T* __restrict__ out,
                     const typename C2<R>::T* __restrict__ twg, long nlines, const DevState* __restrict__ st) {
  typedef ZGeom<LOGN> Z;
  typedef typename C2<R>::T T2;
  constexpr int n = Z::n, LR = Z::LR, LS = Z::LS;
  extern __shared__ __align__(16) unsigned char z_smem[];
  T2* tw = reinterpret_cast<T2*>(z_smem);
  T2* X = tw + n;
  load_tw<R, 1>(tw, twg, n);
  const long l0 = (long)blockIdx.x * LR;
  const size_t nhalf = (size_t)nlines * Z::nh;
  const double li = st->Li[2];
#pragma unroll 2
  for (int e = threadIdx.x; e < LR / 2 * Z::nh; e += Z::TB) {
    const int q = e % (LR / 2), k = e / (LR / 2);
    const T2* src = in + k * nlines + l0 + 2 * q;
    const Pair<R> a = *reinterpret_cast<const Pair<R>*>(src);
    const Pair<R> b = *reinterpret_cast<const Pair<R>*>(src + nhalf);
    Pair<R> p = *reinterpret_cast<const Pair<R>*>(src + 2 * nhalf);
    const R c = (R)(-2.0 * M_PI * (k * li));
    T2 s, t;
    s.x = -p.a.y * c;
    s.y = p.a.x * c;
    t.x = -p.b.y * c;
    t.y = p.b.x * c;
    set_pair<R, LOGN>(X + (2 * q) * LS, k, a.a, b.a);
    set_pair<R, LOGN>(X + (2 * q + 1) * LS, k, a.b, b.b);
    set_pair<R, LOGN>(X + (LR + q) * LS, k, s, t);
  }
  __syncthreads();
  fft_stages<R, LOGN, 0, 1>(X + (threadIdx.x / Z::TPL) * LS, tw, threadIdx.x % Z::TPL);
  for (int e = threadIdx.x; e < LR * n; e += Z::TB) {
    const int l = e >> LOGN, k = e & (n - 1);
    const T2 xy = X[l * LS + fft_pad<R>(k)], z = X[(LR + (l >> 1)) * LS + fft_pad<R>(k)];
    typename V4<R>::T o;
    o.x = xy.x;
    o.y = xy.y;
    o.z = (l & 1) ? z.y : z.x;
    o.w = R(0);
    out[l0 * n + e] = o;
  }
}

// one real mesh: two lines as one complex line
template <class R, int LOGN>
__global__ void __launch_bounds__(ZGeom<LOGN>::T)
k_spme_z_backward(const typename C2<R>::T* __restrict__ in, R* __restrict__ out,
                  const typename C2<R>::T* __restrict__ twg, long nlines) {
  typedef ZGeom<LOGN> Z;
  typedef typename C2<R>::T T2;
  constexpr int n = Z::n, NC = Z::NC, LS = Z::LS;
  extern __shared__ __align__(16) unsigned char z_smem[];
  T2* tw = reinterpret_cast<T2*>(z_smem);
  T2* X = tw + n;
  load_tw<R, 1>(tw, twg, n);
  const long c0 = (long)blockIdx.x * NC;
#pragma unroll 4
  for (int e = threadIdx.x; e < NC * Z::nh; e += Z::T) {
    const int q = e % NC, k = e / NC;
    const Pair<R> a = *reinterpret_cast<const Pair<R>*>(in + k * nlines + 2 * (c0 + q));
    set_pair<R, LOGN>(X + q * LS, k, a.a, a.b);
  }
  __syncthreads();
  fft_stages<R, LOGN, 0, 1>(X + (threadIdx.x / Z::TPL) * LS, tw, threadIdx.x % Z::TPL);
  for (int e = threadIdx.x; e < 2 * NC * n; e += Z::T) {
    const int l = e >> LOGN, k = e & (n - 1);
    const T2 z = X[(l >> 1) * LS + fft_pad<R>(k)];
    out[2 * c0 * n + e] = (l & 1) ? z.y : z.x;
  }
}

struct Kernel {
  const void* f;
  int threads, lines;  // lines: real lines per block (z passes)
  size_t smem;
};

template <class R, int LOGN>
Kernel z_kernel_n(int dir, int ik) {
  typedef ZGeom<LOGN> Z;
  const size_t el = sizeof(typename C2<R>::T);
  if (dir > 0 && ik)
    return {(const void*)k_spme_z_backward_ik<R, LOGN>, Z::TB, Z::LR, el * (Z::n + (size_t)Z::LR * 3 / 2 * Z::LS)};
  const size_t smem = el * (Z::n + (size_t)Z::NC * Z::LS);
  if (dir > 0) return {(const void*)k_spme_z_backward<R, LOGN>, Z::T, 2 * Z::NC, smem};
  return {(const void*)k_spme_z_forward<R, LOGN>, Z::T, 2 * Z::NC, smem};
}

int log2i(int k) {
  int l = 0;
  while ((1 << l) < k) ++l;
  return l;
}

template <class R>
Kernel z_kernel(int K2, int dir, int ik) {
  switch (log2i(K2)) {
#define Z_CASE(L) case L: return z_kernel_n<R, L>(dir, ik);
    Z_CASE(2) Z_CASE(3) Z_CASE(4) Z_CASE(5) Z_CASE(6) Z_CASE(7) Z_CASE(8) Z_CASE(9) Z_CASE(10)
#undef Z_CASE
  }
  return {nullptr, 0, 1, 0};
}

template <class R, int LOGN>
Kernel plane_kernel_n(int method) {
  const void* f = method == 0 ? (const void*)k_spme_plane<R, LOGN, 0>
                              : method == 1 ? (const void*)k_spme_plane<R, LOGN, 1> : (const void*)k_spme_plane<R, LOGN, 2>;
  return {f, PlaneGeom<LOGN>::T, 0, plane_smem<R, LOGN>()};
}

Kernel plane_kernel(int prec, int n, int method) {
  if (prec == MD_PREC_FP64) switch (n) {
    case 16: return plane_kernel_n<double, 4>(method);
    case 32: return plane_kernel_n<double, 5>(method);
    case 64: return plane_kernel_n<double, 6>(method);
  }
  else switch (n) {
    case 16: return plane_kernel_n<float, 4>(method);
    case 32: return plane_kernel_n<float, 5>(method);
    case 64: return plane_kernel_n<float, 6>(method);
    case 128: return plane_kernel_n<float, 7>(method);
  }
  return {nullptr, 0, 0, 0};
}

Kernel z_pass(int prec, int K2, int dir, int ik) {
  return prec == MD_PREC_FP64 ? z_kernel<double>(K2, dir, ik) : z_kernel<float>(K2, dir, ik);
}

}  // namespace

bool plane_chain_ok(int prec, const int K[3]) {
  return K[0] == K[1] && plane_kernel(prec, K[0], 0).f && z_pass(prec, K[2], -1, 0).f;
}

int plane_prepare(int prec, const int K[3], int method) {
  const int methods[2] = {method, 2};
  for (int m : methods) {
    const Kernel k[3] = {plane_kernel(prec, K[0], m), z_pass(prec, K[2], -1, 0), z_pass(prec, K[2], 1, m == 0)};
    for (const Kernel& q : k)
      if (q.smem > 48 * 1024)
        MD_CUDA(cudaFuncSetAttribute(q.f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)q.smem));
  }
  return MD_OK;
}

int plane_chain(md_system* sys, const PlaneChain& p, Recorder* rec) {
  const int prec = sys->prec, ik = p.method == 0;
  const size_t el = prec == MD_PREC_FP64 ? sizeof(double2) : sizeof(float2);
  long nlines = (long)p.n * p.n;
  DevState* st = sys->st;
  PlaneChain a = p;
  void* c1 = (char*)p.C + el * (size_t)nlines * (p.K2 / 2 + 1);
  {
    const Kernel k = z_pass(prec, p.K2, -1, 0);
    void* args[] = {&a.Q, &a.C, &a.tw_z, &nlines};
    if (int r = rec_launch(rec, k.f, dim3((unsigned)(nlines / k.lines)), dim3(k.threads), k.smem, args)) return r;
  }
  {
    const Kernel k = plane_kernel(prec, p.n, p.method);
    void* args[] = {&a.C, &a.tw_n, &a.bm, &a.K2, &a.beta, &st, &a.partials, &a.with_stats, &a.merge, &a.back, &a.energy, &a.dbeta};
    // two blocks a plane while all of them fit one an SM (whole forces, one / two blocks:
    // 128 x 128 x 128, 65 planes, 81 / 66 us, x 256, 129 planes, 118 / 128; binary64 64 x 64 x 128
    // 52 / 46, x 256 66 / 70)
    const int planes = p.K2 / 2 + 1;
    if (int r = rec_launch(rec, k.f, dim3(planes, ik && 2 * planes <= 148 ? 2 : 1), dim3(k.threads), k.smem, args))
      return r;
  }
  if (!p.back) return MD_OK;
  const Kernel k = z_pass(prec, p.K2, 1, ik);
  void* args[] = {&c1, &a.G, &a.tw_z, &nlines, &st};
  return rec_launch(rec, k.f, dim3((unsigned)(nlines / k.lines)), dim3(k.threads), k.smem, args);
}

// Batched FP64 transforms of complex grids [n0][n1][n2], unnormalised, any
// sizes up to 1024 per axis, one pass per axis.
//
// Power-of-two axes: radix-8 Stockham lines in shared memory (fft_lines.cuh),
// 1,024 points per block of 128 threads; lines adjacent in memory share a
// block, so strided axes load coalesced.  Bound: latency of two or three
// shared-memory exchanges per pass; the radix-2 line per block it replaces
// made log2 n of them and loaded strided axes 16 bytes at a time (64^3 grids:
// 21 us a pass of one before, 5.7 us of three and 10 us of eight now).
//
// Other sizes (the odd bin grids of AdaptRCut): a length p is summed over the
// (p-1)/2 pairs x_j +- x_{p-j}, which gives outputs k and p-k together from
// 4 real products per pair where the direct sum takes 16; composite lengths
// n = n1 n2 with a prime n1 <= 11 take two such stages (Cooley-Tukey).  Lanes
// hold different lines, so a twiddle is one broadcast and six outputs share
// each loaded pair.  Bound: shared-memory bandwidth and FP64 issue (six grids of
// 41 x 41 x 161: 31 us along the 41-point axes, 38 along the other).
#include <algorithm>
#include "fft_lines.cuh"

namespace {

// line L of an axis of n points: elements `inner` apart from (L / inner) n inner + L % inner.
// At most 2^20 lines a grid, so 32 bits hold any L; a 64-bit division here cost more
// than the transform (one per point read and written).
__device__ __forceinline__ size_t line_base(unsigned L, int n, unsigned inner) {
  const unsigned q = L / inner;
  return (size_t)q * n * inner + (L - q * inner);
}

// Where a pass reads and writes its grids (element p of all grids end to end):
// complex in and out; or, first pass of real grids, (re[p], im[p]) with im = 0
// from element n_im on; or, last pass, the real parts alone from element n_c on,
// to outr[p - n_c].
struct DftIo {
  const double2* in = nullptr;
  double2* out = nullptr;
  const double *re = nullptr, *im = nullptr;
  long n_im = 0;
  double* outr = nullptr;
  long n_c = 0;
};
enum { IO_PLAIN = 0, IO_REAL_IN = 1, IO_REAL_OUT = 2 };

template <int IO>
__device__ __forceinline__ double2 io_load(const DftIo& io, size_t p) {
  if (IO != IO_REAL_IN) return io.in[p];
  return make_double2(io.re[p], (long)p < io.n_im ? io.im[p] : 0.0);
}
template <int IO>
__device__ __forceinline__ void io_store(const DftIo& io, size_t p, double2 v) {
  if (IO == IO_REAL_OUT && (long)p >= io.n_c) io.outr[p - io.n_c] = v.x;
  else io.out[p] = v;
}

template <int LOGN, int IO>
__global__ void __launch_bounds__(FFT_THREADS)
k_fft_grid(DftIo io, unsigned nlines, unsigned inner, int sign) {
  typedef FftGeom<LOGN> G;
  constexpr int n = G::n, LPB = G::LPB, LS = G::LS, EPT = G::EPT;
  extern __shared__ __align__(16) unsigned char fg_smem[];
  double2* tw = reinterpret_cast<double2*>(fg_smem);
  double2* X = tw + n;
  for (int m = threadIdx.x; m < n; m += FFT_THREADS) {
    double s, c;
    sincospi(2.0 * m / n, &s, &c);
    tw[m] = make_double2(c, sign * s);
  }
  // element s of the thread: line l of the block, point k of it, element p of the
  // grids (a thread's elements of a strided axis lie on one line: LPB divides
  // the threads)
  const unsigned line0 = blockIdx.x * LPB;
  const size_t first = inner > 1 ? line_base(line0 + threadIdx.x % LPB, n, inner) : 0;
  auto element = [&](int s, int& l, int& k, size_t& p) -> bool {
    const int e = threadIdx.x + s * FFT_THREADS;
    l = inner > 1 ? e % LPB : e >> LOGN;
    k = inner > 1 ? e / LPB : e & (n - 1);
    p = inner > 1 ? first + (size_t)k * inner : (size_t)line0 * n + e;
    return line0 + l < nlines;
  };
  double2 v[EPT];
#pragma unroll
  for (int s = 0; s < EPT; ++s) {
    int l, k;
    size_t p;
    v[s] = element(s, l, k, p) ? io_load<IO>(io, p) : make_double2(0.0, 0.0);
  }
#pragma unroll
  for (int s = 0; s < EPT; ++s) {
    int l, k;
    size_t p;
    element(s, l, k, p);
    X[l * LS + fft_pad<double>(k)] = v[s];
  }
  __syncthreads();
  double2* x = X + (threadIdx.x / G::TPL) * LS;
  if (sign < 0) fft_stages<double, LOGN, 0, -1>(x, tw, threadIdx.x % G::TPL);
  else fft_stages<double, LOGN, 0, 1>(x, tw, threadIdx.x % G::TPL);
#pragma unroll
  for (int s = 0; s < EPT; ++s) {
    int l, k;
    size_t p;
    if (element(s, l, k, p)) io_store<IO>(io, p, X[l * LS + fft_pad<double>(k)]);
  }
}

template <int LOGN, int IO>
int fft_grid_launch(const DftIo& io, long nlines, long inner, int sign, cudaStream_t s) {
  typedef FftGeom<LOGN> G;
  const size_t smem = sizeof(double2) * (G::n + (size_t)G::LPB * G::LS);
  k_fft_grid<LOGN, IO><<<(unsigned)((nlines + G::LPB - 1) / G::LPB), FFT_THREADS, smem, s>>>(io, nlines, inner, sign);
  MD_CHECK_LAUNCH("fft axis");
  return MD_OK;
}

constexpr int DA_THREADS = 128;
constexpr int DA_KB = 6;  // output pairs (k, p - k) a thread forms at a time

// the pair sums of outputs k0 .. k0 + DA_KB - 1 (<= p / 2) of the length-p
// transform whose point j sits at x[j * xs]: A_k = sum_j a_j cos, B_k = sum_j b_j sin,
// X_k = x_0 + A_k + i B_k, X_{p-k} = x_0 + A_k - i B_k; tw holds (cos, sin) of
// 2 pi m / n, st = n / p.  ready: x already holds a_j at j and b_j at p - j.
template <bool READY>
__device__ __forceinline__ void pair_sums(const double2* x, int xs, int p, int k0, const double2* tw, int n, int st,
                                          double2 (&A)[DA_KB], double2 (&B)[DA_KB]) {
  int m[DA_KB], dm[DA_KB];
  const double2 x0 = x[0];
#pragma unroll
  for (int q = 0; q < DA_KB; ++q) {
    A[q] = x0;
    B[q] = make_double2(0.0, 0.0);
    dm[q] = min(k0 + q, p / 2) * st;
    m[q] = 0;
  }
  const int h = (p - 1) / 2;
  for (int j = 1; j <= h; ++j) {
    double2 a = x[(size_t)j * xs], b = x[(size_t)(p - j) * xs];
    if (!READY) {
      const double2 t = a;
      a = make_double2(t.x + b.x, t.y + b.y);
      b = make_double2(t.x - b.x, t.y - b.y);
    }
#pragma unroll
    for (int q = 0; q < DA_KB; ++q) {
      m[q] += dm[q];
      if (m[q] >= n) m[q] -= n;
      const double2 w = tw[m[q]];
      A[q].x = fma(a.x, w.x, A[q].x);
      A[q].y = fma(a.y, w.x, A[q].y);
      B[q].x = fma(-b.y, w.y, B[q].x);
      B[q].y = fma(b.x, w.y, B[q].y);
    }
  }
  if ((p & 1) == 0) {  // the unpaired middle point
    const double2 c = x[(size_t)(p / 2) * xs];
#pragma unroll
    for (int q = 0; q < DA_KB; ++q) {
      const double sg = ((k0 + q) & 1) ? -1.0 : 1.0;
      A[q].x += sg * c.x;
      A[q].y += sg * c.y;
    }
  }
}

// LN lines per block, one per lane; n = n1 n2 (n1 = 1: a single stage of length n)
template <int LN, int IO>
__global__ void __launch_bounds__(DA_THREADS)
k_dft_any(DftIo io, unsigned nlines, unsigned inner, int n, int n1, int sign) {
  extern __shared__ __align__(16) unsigned char da_smem[];
  constexpr int LS = LN + 1, NG = DA_THREADS / LN;
  double2* tw = reinterpret_cast<double2*>(da_smem);  // (cos, sign sin) of 2 pi m / n
  double2* x = tw + n;                                // [n][LS]
  const int n2 = n / n1;
  const unsigned line0 = blockIdx.x * LN;
  for (int m = threadIdx.x; m < n; m += DA_THREADS) {
    double s, c;
    sincospi(2.0 * m / n, &s, &c);
    tw[m] = make_double2(c, sign * s);
  }
  const int l = threadIdx.x % LN, g = threadIdx.x / LN;
  const bool live = line0 + l < nlines;
  const size_t dst = live ? line_base(line0 + l, n, inner) : 0;
  if (inner > 1) {  // the thread's line, a point in NG
    for (int j = g; j < n; j += NG)
      x[j * LS + l] = live ? io_load<IO>(io, dst + (size_t)j * inner) : make_double2(0.0, 0.0);
  } else {  // whole lines end to end
    const size_t p0 = (size_t)line0 * n;
    for (int t = threadIdx.x; t < n * LN; t += DA_THREADS) {
      const int q = t / n;
      x[(t - q * n) * LS + q] = line0 + q < nlines ? io_load<IO>(io, p0 + t) : make_double2(0.0, 0.0);
    }
  }
  __syncthreads();
  double2 A[DA_KB], B[DA_KB];
  if (n1 > 1) {
    // stage 1, in place: a thread holds all outputs of a length-n1 transform
    // (n1 <= 11: k <= 5), times W_n^{j2 k1}
    for (int j2 = g; j2 < n2; j2 += NG) {
      double2* c = x + j2 * LS + l;
      pair_sums<false>(c, n2 * LS, n1, 0, tw, n, n2, A, B);
#pragma unroll
      for (int q = 0; q < DA_KB; ++q) {
        if (q > n1 / 2) break;
        const double2 w = tw[j2 * q];  // (j2 < n2, q < n1: below n)
        const double2 u = make_double2(A[q].x + B[q].x, A[q].y + B[q].y);
        c[(size_t)q * n2 * LS] = make_double2(u.x * w.x - u.y * w.y, u.x * w.y + u.y * w.x);
        if (q > 0 && 2 * q < n1) {
          const int k = n1 - q;
          const double2 z = tw[j2 * k];
          const double2 v = make_double2(A[q].x - B[q].x, A[q].y - B[q].y);
          c[(size_t)k * n2 * LS] = make_double2(v.x * z.x - v.y * z.y, v.x * z.y + v.y * z.x);
        }
      }
    }
    __syncthreads();
  }
  // the last stage: n1 transforms of length n2 (point j2 of transform k1 at
  // row k1 n2 + j2); pairs first, in place, then the outputs
  const int h = (n2 - 1) / 2;
  for (int t = threadIdx.x; t < n1 * h * LN; t += DA_THREADS) {
    const int ll = t % LN, r = t / LN, k1 = r / h, j = 1 + r - k1 * h;
    double2* a = x + (k1 * n2 + j) * LS + ll;
    double2* b = x + (k1 * n2 + n2 - j) * LS + ll;
    const double2 u = *a, v = *b;
    *a = make_double2(u.x + v.x, u.y + v.y);
    *b = make_double2(u.x - v.x, u.y - v.y);
  }
  __syncthreads();
  const int nk = n2 / 2 + 1, nt = (nk + DA_KB - 1) / DA_KB;
  for (int t = g; t < n1 * nt; t += NG) {
    const int k1 = t / nt, k0 = (t - k1 * nt) * DA_KB;
    pair_sums<true>(x + k1 * n2 * LS + l, LS, n2, k0, tw, n, n1, A, B);
    if (!live) continue;
#pragma unroll
    for (int q = 0; q < DA_KB; ++q) {
      const int k2 = k0 + q;
      if (k2 >= nk) break;
      io_store<IO>(io, dst + (size_t)(k1 + n1 * k2) * inner, make_double2(A[q].x + B[q].x, A[q].y + B[q].y));
      if (k2 > 0 && 2 * k2 < n2)
        io_store<IO>(io, dst + (size_t)(k1 + n1 * (n2 - k2)) * inner, make_double2(A[q].x - B[q].x, A[q].y - B[q].y));
    }
  }
}

template <int LN, int IO>
int dft_any_launch(const DftIo& io, long nlines, long inner, int n, int n1, int sign, cudaStream_t s) {
  const size_t smem = sizeof(double2) * (n + (size_t)n * (LN + 1));
  if (smem > 48 * 1024)
    MD_CUDA(cudaFuncSetAttribute(k_dft_any<LN, IO>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
  k_dft_any<LN, IO><<<(unsigned)((nlines + LN - 1) / LN), DA_THREADS, smem, s>>>(io, nlines, inner, n, n1, sign);
  MD_CHECK_LAUNCH("dft axis");
  return MD_OK;
}

template <int IO>
int dft_pass(const DftIo& io, const int n[3], int axis, int sign, int batch, cudaStream_t s) {
  const int na = n[axis];
  const long inner = axis == 2 ? 1 : axis == 1 ? n[2] : (long)n[1] * n[2];
  const long nlines = (long)n[0] * n[1] * n[2] / na * batch;
  switch (na) {
#define FFT_CASE(L) case 1 << L: return fft_grid_launch<L, IO>(io, nlines, inner, sign, s);
    FFT_CASE(1) FFT_CASE(2) FFT_CASE(3) FFT_CASE(4) FFT_CASE(5) FFT_CASE(6) FFT_CASE(7) FFT_CASE(8) FFT_CASE(9) FFT_CASE(10)
#undef FFT_CASE
  }
  int n1 = 1;  // the smallest prime factor when it is at most 11 and proper
  for (int f = 2; f <= 11 && f < na; ++f)
    if (na % f == 0) { n1 = f; break; }
  // lines per block: all lanes of a warp where several blocks' lines still fit
  // on an SM (41 points: 23 KB, 161 points: 46 KB of the 228 KB)
  if (na <= 96) return dft_any_launch<32, IO>(io, nlines, inner, na, n1, sign, s);
  if (na <= 192) return dft_any_launch<16, IO>(io, nlines, inner, na, n1, sign, s);
  if (na <= 384) return dft_any_launch<8, IO>(io, nlines, inner, na, n1, sign, s);
  return dft_any_launch<4, IO>(io, nlines, inner, na, n1, sign, s);
}

}  // namespace

// one pass (sign -1 forward, +1 backward) over `batch` consecutive grids along
// `axis`; in may equal out
int dft3_axis(const double2* in, double2* out, const int n[3], int axis, int sign, int batch, cudaStream_t s) {
  DftIo io;
  io.in = in;
  io.out = out;
  return dft_pass<IO_PLAIN>(io, n, axis, sign, batch, s);
}

// unnormalised 3D transform of `batch` consecutive grids, in place
int dft3_grid(double2* data, const int n[3], int sign, int batch, cudaStream_t s) {
  for (int axis = 2; axis >= 0; --axis)
    if (int r = dft3_axis(data, data, n, axis, sign, batch, s)) return r;
  return MD_OK;
}

// forward transforms out of the `batch` real grids re, the first n_im of them
// with the grids im as imaginary parts
int dft3_from_real(const double* re, const double* im, int n_im, double2* out, const int n[3], int batch,
                   cudaStream_t s) {
  DftIo io;
  io.re = re;
  io.im = im;
  io.n_im = (long)n_im * n[0] * n[1] * n[2];
  io.out = out;
  if (int r = dft_pass<IO_REAL_IN>(io, n, 2, -1, batch, s)) return r;
  for (int axis = 1; axis >= 0; --axis)
    if (int r = dft3_axis(out, out, n, axis, -1, batch, s)) return r;
  return MD_OK;
}

// backward transforms of `batch` grids, the first n_c in place, of the others
// the real parts to outr
int dft3_to_real(double2* data, int n_c, double* outr, const int n[3], int batch, cudaStream_t s) {
  for (int axis = 2; axis >= 1; --axis)
    if (int r = dft3_axis(data, data, n, axis, +1, batch, s)) return r;
  DftIo io;
  io.in = data;
  io.out = data;
  io.outr = outr;
  io.n_c = (long)n_c * n[0] * n[1] * n[2];
  return dft_pass<IO_REAL_OUT>(io, n, 0, +1, batch, s);
}

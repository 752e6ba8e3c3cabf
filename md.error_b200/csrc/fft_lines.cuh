// Line transforms in shared memory, shared by the SPME passes (spme.cu) and
// the FP64 grid transforms (dft.cu, errmap.cu).
#pragma once
#include "device_common.cuh"

template <class R> struct C2;
template <> struct C2<float> { typedef float2 T; };
template <> struct C2<double> { typedef double2 T; };

// ---------------------------------------------------------------- FFT
// Stockham transform of whole lines in shared memory, in the formulation of
// Govindaraju et al. (SC'08): with Ns the length already transformed, stage
// (radix R) takes butterfly j < n/R, reads its R inputs at stride n/R,
// multiplies input r by W_n^{r k n/(Ns R)} (k = j mod Ns), applies an R-point
// DFT in registers and writes output r to (j / Ns) Ns R + k + r Ns.  Stages
// of radix 8, then one of radix 4 or 2, cover n = 2^LOGN and leave the line
// in natural order.  One stage reads all its inputs, synchronises and then
// writes, so a single buffer per line suffices.  A block of FFT_THREADS
// threads holds FFT_THREADS / TPL lines (TPL = n/8 threads per line); twiddles
// come from a per-axis table computed once in FP64 (conjugated for the inverse
// transform).  Element i of a line sits at fft_pad(i): the outputs of a radix-8
// stage are 8 apart from lane to lane (and, the next 64, from eighth to ninth
// lane), which fall on one bank where they lie in order (8-way conflicts).
// binary64: one element of padding per 8.  binary32: a permutation within each
// 16 elements; padding would split every aligned run over two wavefronts.
constexpr int FFT_THREADS = 128;

template <class T2>
__device__ __forceinline__ T2 cmul(T2 a, T2 b) {
  T2 r;
  r.x = a.x * b.x - a.y * b.y;
  r.y = a.x * b.y + a.y * b.x;
  return r;
}
template <class T2>
__device__ __forceinline__ T2 c_add(T2 a, T2 b) {
  T2 r;
  r.x = a.x + b.x;
  r.y = a.y + b.y;
  return r;
}
template <class T2>
__device__ __forceinline__ T2 c_sub(T2 a, T2 b) {
  T2 r;
  r.x = a.x - b.x;
  r.y = a.y - b.y;
  return r;
}
// a * (SIGN i)
template <int SIGN, class T2>
__device__ __forceinline__ T2 c_mul_si(T2 a) {
  T2 r;
  r.x = SIGN > 0 ? -a.y : a.y;
  r.y = SIGN > 0 ? a.x : -a.x;
  return r;
}

// X_s = sum_r v_r exp(SIGN 2 pi i r s / 4)
template <int SIGN, class T2>
__device__ __forceinline__ void dft4(T2& v0, T2& v1, T2& v2, T2& v3) {
  const T2 s0 = c_add(v0, v2), d0 = c_sub(v0, v2), s1 = c_add(v1, v3), d1 = c_mul_si<SIGN>(c_sub(v1, v3));
  v0 = c_add(s0, s1);
  v2 = c_sub(s0, s1);
  v1 = c_add(d0, d1);
  v3 = c_sub(d0, d1);
}

template <class R, int RR, int SIGN>
__device__ __forceinline__ void dft_reg(typename C2<R>::T (&v)[RR]) {
  typedef typename C2<R>::T T2;
  if constexpr (RR == 2) {
    const T2 a = v[0];
    v[0] = c_add(a, v[1]);
    v[1] = c_sub(a, v[1]);
  } else if constexpr (RR == 4) {
    dft4<SIGN>(v[0], v[1], v[2], v[3]);
  } else {
    // radix 8 = two radix-4 DFTs of the even and odd inputs, odd ones
    // multiplied by W^k, W = exp(SIGN 2 pi i / 8)
    T2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    dft4<SIGN>(e0, e1, e2, e3);
    dft4<SIGN>(o0, o1, o2, o3);
    const R h = R(0.70710678118654752440);  // 1/sqrt(2)
    T2 t;
    t.x = (SIGN > 0 ? o1.x - o1.y : o1.x + o1.y) * h;
    t.y = (SIGN > 0 ? o1.y + o1.x : o1.y - o1.x) * h;
    o1 = t;
    o2 = c_mul_si<SIGN>(o2);
    t.x = (SIGN > 0 ? -o3.x - o3.y : -o3.x + o3.y) * h;
    t.y = (SIGN > 0 ? -o3.y + o3.x : -o3.y - o3.x) * h;
    o3 = t;
    v[0] = c_add(e0, o0);
    v[4] = c_sub(e0, o0);
    v[1] = c_add(e1, o1);
    v[5] = c_sub(e1, o1);
    v[2] = c_add(e2, o2);
    v[6] = c_sub(e2, o2);
    v[3] = c_add(e3, o3);
    v[7] = c_sub(e3, o3);
  }
}

template <class R>
__host__ __device__ __forceinline__ constexpr int fft_pad(int i) {
  return sizeof(R) == 4 ? i ^ ((i >> 4) & 7) ^ (((i >> 6) & 1) << 3) : i + (i >> 3);
}
// lines shorter than 256 share a warp: odd, so that accesses across lines fall
// on different banks; longer ones pair up in the real passes (2 modulo 8)
__host__ __device__ __forceinline__ constexpr int fft_line_stride(int n) { return n < 256 ? n + (n >> 3) + 1 : n + (n >> 3) + 2; }

template <int LOGN>
struct FftGeom {
  static constexpr int n = 1 << LOGN;
  static constexpr int TPL = n >= 8 ? n / 8 : 1;  // threads per line
  static constexpr int LPB = FFT_THREADS / TPL;   // lines per block
  static constexpr int LS = fft_line_stride(n);   // padded line stride
  static constexpr int EPT = LPB * n / FFT_THREADS;  // elements per thread
};

// the stages from Ns = 2^LOGNS on, for the line x of this thread (lane tl of
// the line's TPL threads); every thread of the block takes part
template <class R, int LOGN, int LOGNS, int SIGN>
__device__ __forceinline__ void fft_stages(typename C2<R>::T* x, const typename C2<R>::T* tw, int tl) {
  typedef typename C2<R>::T T2;
  constexpr int n = 1 << LOGN, TPL = FftGeom<LOGN>::TPL;
  constexpr int LR = (LOGN - LOGNS) >= 3 ? 3 : (LOGN - LOGNS);
  constexpr int RR = 1 << LR, NS = 1 << LOGNS, NBF = n / RR, BPT = NBF / TPL;
  static_assert(BPT >= 1, "at least one butterfly per thread");
  T2 v[BPT][RR];
#pragma unroll
  for (int q = 0; q < BPT; ++q) {
    const int j = tl + q * TPL;
#pragma unroll
    for (int r = 0; r < RR; ++r) v[q][r] = x[fft_pad<R>(j + r * NBF)];
    if constexpr (LOGNS > 0) {
      const int k = j & (NS - 1);
#pragma unroll
      for (int r = 1; r < RR; ++r) v[q][r] = cmul(v[q][r], tw[(r * k) << (LOGN - LOGNS - LR)]);
    }
    dft_reg<R, RR, SIGN>(v[q]);
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < BPT; ++q) {
    const int j = tl + q * TPL;
    const int d = ((j >> LOGNS) << (LOGNS + LR)) + (j & (NS - 1));
#pragma unroll
    for (int r = 0; r < RR; ++r) x[fft_pad<R>(d + r * NS)] = v[q][r];
  }
  __syncthreads();
  if constexpr (LOGNS + LR < LOGN) fft_stages<R, LOGN, LOGNS + LR, SIGN>(x, tw, tl);
}

// the block barriers of fft_stages<R, LOGN, LOGNS, *> without the work: a
// group with nothing to transform meets the others' barriers
template <int LOGN, int LOGNS>
__device__ __forceinline__ void fft_stage_barriers() {
  constexpr int LR = (LOGN - LOGNS) >= 3 ? 3 : (LOGN - LOGNS);
  __syncthreads();
  __syncthreads();
  if constexpr (LOGNS + LR < LOGN) fft_stage_barriers<LOGN, LOGNS + LR>();
}

template <class R, int SIGN>
__device__ __forceinline__ void load_tw(typename C2<R>::T* tw, const typename C2<R>::T* __restrict__ twg, int n) {
  for (int m = threadIdx.x; m < n; m += blockDim.x) {
    typename C2<R>::T w = twg[m];
    if (SIGN > 0) w.y = -w.y;
    tw[m] = w;
  }
}

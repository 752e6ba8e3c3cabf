// Particle-mesh steps of the SPME chain: charges onto the mesh and the mesh
// back to the atoms (B-spline weights, orders 2..14).
// Reference (RE = longRange.hetero/profile.test/template/tools/real.error):
//   calQ spread                      RE/src/EleRecBSpline.cpp:541-619
//   force gather, ik                 RE/src/EleRecBSpline.cpp:393-536
//   force gather, analytic           RE/src/EleRecFBSpline.cpp:1146-1195
//
// In all of them the lanes of a warp lie along the rows of an atom's stencil:
// with order n, lane = (row k, point c), 32 / n rows of n consecutive z points
// per instruction, so one access touches a few contiguous row pieces.  Lane
// (k, c) keeps its c, hence its z weight, over the whole stencil.
#include <climits>
#include "spme_pm.cuh"

namespace {

// K is a power of two: the product with 1/K rounds as the quotient, and the mask
// takes b = K to 0.  It also keeps every base inside the mesh: a binary64 NaN
// (a coordinate that is none) becomes the lowest int, from which the extent of a
// staged region would come out negative and its reads outside the block's memory.
template <class R>
__device__ __forceinline__ void grid_coord(R x, R Linv, int K, int& base, R& frac) {
  const R kinv = sizeof(R) == 4 ? (R)__int_as_float((127 - (31 - __clz(K))) << 23)
                                : (R)__hiloint2double((1023 - (31 - __clz(K))) << 20, 0);
  R u = R(K) * x * Linv;
  u -= floor_r(u * kinv) * R(K);
  R b = floor_r(u);
  frac = u - b;
  base = (int)b & (K - 1);
}

// M_n(f + j), j = 0..n-1, and derivatives (D) by the recursion
// M_k(u) = (u M_{k-1}(u) + (k - u) M_{k-1}(u - 1)) / (k - 1) (Essmann et al. 1995),
// the order a compile-time constant so that the arrays stay in registers
template <class R, int NO, bool D>
__device__ __forceinline__ void bsp_t(R f, R (&w)[NO], R (&dw)[NO]) {
  w[0] = f;
  w[1] = R(1) - f;
#pragma unroll
  for (int j = 2; j < NO; ++j) w[j] = R(0);
#pragma unroll
  for (int k = 3; k <= NO; ++k) {
    if (D && k == NO) {
#pragma unroll
      for (int j = 0; j < NO; ++j) dw[j] = (j < NO - 1 ? w[j] : R(0)) - (j > 0 ? w[j - 1] : R(0));
    }
    const R inv = R(1) / R(k - 1);
#pragma unroll
    for (int j = k - 1; j >= 0; --j) {
      const R u = f + R(j);
      const R a = (j < k - 1) ? w[j] : R(0);
      const R b = (j > 0) ? w[j - 1] : R(0);
      w[j] = (u * a + (R(k) - u) * b) * inv;
    }
  }
  if (D && NO == 2) { dw[0] = R(1); dw[1] = R(-1); }
}

#define SPME_ORDERS(X) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14)

// ---------------------------------------------------------------- spread
// Large dense systems in binary32 (spread_by_tile).  A block of two warps
// takes 32 consecutive charges (cell order, hence compact in space) and adds
// their stencils to a shared-memory tile without atomics: each warp owns every
// other x plane of the tile and takes the charges one at a time, whose points
// are distinct, with plain loads and stores.  (Shared atomics run as a retry
// loop; 64 charges per block of 256 threads with them took 415 us for
// 1,048,576 charges on 128 x 128 x 512 at order 6, bound by the shared-memory
// pipe at 76 wavefronts per charge; this takes 232 us,
// that pipe at 95 %.)  Weights are read for
// four charges at once (they lie along the charges), and the tile's row
// stride is +-n modulo the banks, so that the 32 / n rows of an instruction
// fall on consecutive banks.  The tile is then added to the mesh with one
// 4-wide atomic per 4 z points, skipping empty groups.  Each charge's stencil
// base is taken in the periodic image closest to the block's first charge, so
// that a block next to a periodic face still has a compact tile.  The tile's z
// origin and extent are multiples of 4 (K2 is a power of two >= 4, so a group
// never wraps).  A block whose tile does not fit adds every point with a
// global atomic.
constexpr int SPREAD_CHARGES = 32, SPREAD_LD = SPREAD_CHARGES + 4;  // + 4: the rows' weights on different banks
constexpr int SPREAD_THREADS = 64;

template <class T> struct alignas(16) Vec4 { T v[4]; };

// rows r0 .. of the stencils of the block's charges onto this warp's planes:
// row rho of a charge is plane a0 + 2 (rho / n), a0 its first plane of the
// warp's parity, and y point rho % n; NJ rows per lane
template <int NO, int NJ>
__device__ __forceinline__ void spread_rows(float* tile, const float (*sw)[NO + 1][SPREAD_LD], const int* sbase, int na4,
                                            int ie1, int irs, int r0, int warp, int lane) {
  constexpr int RP = 32 / NO, NR = ((NO + 1) / 2) * NO;
  // lanes beyond the RP rows, and rows beyond the last, repeat a point of the
  // same instruction with the same value, so that no access is predicated
  const int k = lane / NO % RP, c = lane % NO;
  int off[NJ], ia[NJ], ib[NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int row = min(r0 + j * RP + k, NR - 1);
    const int i = row / NO, b = row - i * NO;
    ia[j] = 2 * i * SPREAD_LD;
    ib[j] = b * SPREAD_LD;
    off[j] = -(2 * i * ie1 + b) * irs - c;
  }
#pragma unroll 1
  for (int g = 0; g < na4; g += 4) {
    const Vec4<float> wz = *reinterpret_cast<const Vec4<float>*>(&sw[2][c][g]);
    const Vec4<int> bs = *reinterpret_cast<const Vec4<int>*>(&sbase[g]);
    float wyz[NJ][4];
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const Vec4<float> wy = *reinterpret_cast<const Vec4<float>*>(&sw[1][0][g + ib[j]]);
#pragma unroll
      for (int u = 0; u < 4; ++u) wyz[j][u] = wy.v[u] * wz.v[u];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int a0 = (bs.v[u] ^ warp) & 1;  // bit 0: parity of the base's x plane
      float* t = tile + (bs.v[u] >> 1) - a0 * ie1 * irs;
      const float* wx = &sw[0][a0][g + u];
      float v[NJ], w[NJ];
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        v[j] = t[off[j]];
        w[j] = wx[ia[j]];
      }
#pragma unroll
      for (int j = 0; j < NJ; ++j) t[off[j]] = v[j] + w[j] * wyz[j][u];
      __syncwarp();  // the next charge's points may be these
    }
  }
}

template <int NO>
__global__ void __launch_bounds__(SPREAD_THREADS)
k_spme_spread_t(int N, const float4* __restrict__ pos, int K0, int K1, int K2,
                const DevState* __restrict__ st, float* __restrict__ Q, int tile_cap) {
  constexpr int A = SPREAD_CHARGES;
  extern __shared__ __align__(32) unsigned char sp_smem[];
  float* tile = reinterpret_cast<float*>(sp_smem);
  // z weights carry the charge; plane NO of an odd order has weight zero
  __shared__ __align__(32) float sw[3][NO + 1][SPREAD_LD];
  __shared__ int sb[3][SPREAD_CHARGES], sq[SPREAD_CHARGES], red[2][6];
  __shared__ __align__(16) int sbase[SPREAD_CHARGES];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i0 = blockIdx.x * A, na = min(A, N - i0), na4 = (na + 3) & ~3;
  if (threadIdx.x < 12) red[threadIdx.x / 6][threadIdx.x % 6] = threadIdx.x % 6 < 3 ? INT_MAX : INT_MIN;
  __syncthreads();
  // one (charge, axis) per thread; A is a multiple of 32, so an axis per warp
  for (int t = threadIdx.x; t < 3 * A; t += SPREAD_THREADS) {
    const int d = t / A, at = t - d * A;
    const float4 p = pos[i0 + min(at, na - 1)];
    const float q = at < na ? p.w : 0.f;
    const float x = d == 0 ? p.x : d == 1 ? p.y : p.z;
    int b;
    float f, w[NO], dw[NO];
    grid_coord<float>(x, (float)st->Li[d], d == 0 ? K0 : d == 1 ? K1 : K2, b, f);
    bsp_t<float, NO, false>(f, w, dw);
#pragma unroll
    for (int j = 0; j < NO; ++j) sw[d][j][at] = d == 2 ? w[j] * q : w[j];
    if (d == 0) {
      sw[0][NO][at] = 0.f;
      sq[at] = q != 0.f;
    }
    sb[d][at] = b;
  }
  __syncthreads();
  // images nearest the first charge, and the box of the charged ones
  for (int t = threadIdx.x; t < 3 * A; t += SPREAD_THREADS) {
    const int d = t / A, at = t - d * A, Kd = d == 0 ? K0 : d == 1 ? K1 : K2;
    int b = sb[d][at];
    const int dv = b - sb[d][0];
    if (2 * dv > Kd) b -= Kd;
    else if (2 * dv < -Kd) b += Kd;
    const bool on = sq[at] != 0;
    if (at > 0) sb[d][at] = b;  // the first charge's own stays as it is
    const int l = __reduce_min_sync(0xffffffffu, on ? b : INT_MAX);
    const int h = __reduce_max_sync(0xffffffffu, on ? b : INT_MIN);
    if (lane == 0) {
      red[warp][d] = min(red[warp][d], l);
      red[warp][3 + d] = max(red[warp][3 + d], h);
    }
  }
  __syncthreads();
  int lo[3], hi[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    lo[d] = min(red[0][d], red[1][d]);
    hi[d] = max(red[0][3 + d], red[1][3 + d]);
  }
  if (lo[0] > hi[0]) return;  // no charge in this block
  const int o0 = lo[0] - (NO - 1) - (NO & 1), o1 = lo[1] - (NO - 1), o2 = (lo[2] - (NO - 1)) & ~3;
  const long e0 = hi[0] - o0 + 1, e1 = hi[1] - o1 + 1, e2 = (hi[2] - o2 + 4) & ~3;
  constexpr int M = 32;  // banks
  const long rs = e2 + min((NO - (int)e2) & (M - 1), (-NO - (int)e2) & (M - 1));
  if (e0 * e1 * rs <= tile_cap) {
    const int ie1 = (int)e1, irs = (int)rs, tsz = (int)(e0 * e1 * rs);
    const Vec4<float> zero = {{0.f, 0.f, 0.f, 0.f}};
#pragma unroll 4
    for (int e = 4 * threadIdx.x; e < tsz; e += 4 * SPREAD_THREADS)
      *reinterpret_cast<Vec4<float>*>(tile + e) = zero;  // the capacity is a multiple of 4
    // tile index of each charge's base point and the parity of its x plane
    for (int at = threadIdx.x; at < na4; at += SPREAD_THREADS) {
      const bool no = sq[at] == 0;  // no charge: its zeros go where the box's corner is
      const int x = (no ? lo[0] : sb[0][at]) - o0, y = (no ? lo[1] : sb[1][at]) - o1, z = (no ? lo[2] : sb[2][at]) - o2;
      sbase[at] = 2 * ((x * ie1 + y) * irs + z) + (x & 1);
    }
    __syncthreads();
    constexpr int RP = 32 / NO, NR = ((NO + 1) / 2) * NO, NI = (NR + RP - 1) / RP, JC = 8;
    if constexpr (NI <= JC) {
      spread_rows<NO, NI>(tile, sw, sbase, na4, ie1, irs, 0, warp, lane);
    } else {
#pragma unroll 1
      for (int j = 0; j < NI / JC; ++j)
        spread_rows<NO, JC>(tile, sw, sbase, na4, ie1, irs, j * JC * RP, warp, lane);
      if constexpr (NI % JC != 0)
        spread_rows<NO, NI % JC>(tile, sw, sbase, na4, ie1, irs, NI / JC * JC * RP, warp, lane);
    }
    __syncthreads();
    // the tile onto the mesh: lanes along z in groups of 4 points, the threads'
    // rows of one x plane per pass
    const int g2 = (int)(e2 >> 2), ie0 = (int)e0;
    const int lpr = min(g2, SPREAD_THREADS), rpw = SPREAD_THREADS / lpr;
    const int r_lane = threadIdx.x / lpr, z_lane = threadIdx.x - r_lane * lpr;
    if (r_lane >= rpw) return;
    for (int z4 = z_lane; z4 < g2; z4 += lpr) {
      const int gz = (o2 + 4 * z4) & (K2 - 1);
      int x = 0, y = r_lane;
      while (y >= ie1) { y -= ie1; ++x; }
#pragma unroll 4
      while (x < ie0) {
        const float* t = tile + (x * ie1 + y) * irs + 4 * z4;
        const float v0 = t[0], v1 = t[1], v2 = t[2], v3 = t[3];
        const int m = (((o0 + x) & (K0 - 1)) * K1 + ((o1 + y) & (K1 - 1))) * K2 + gz;  // at most 2^30 points
        if (v0 != 0.f || v1 != 0.f || v2 != 0.f || v3 != 0.f) 
          atomicAdd(reinterpret_cast<float4*>(Q + m), make_float4(v0, v1, v2, v3));
        y += rpw;
        while (y >= ie1) { y -= ie1; ++x; }
      }
    }
  } else {
    constexpr int RP = 32 / NO, NR = NO * NO;
    if (lane >= RP * NO) return;
    const int k = lane / NO, c = lane - k * NO;
    for (int at = warp; at < na; at += SPREAD_THREADS / 32) {
      if (!sq[at]) continue;
      const float wz = sw[2][c][at];
      const int gz = (sb[2][at] - c) & (K2 - 1);
      for (int row = k; row < NR; row += RP) {
        const int a = row / NO, b = row - a * NO;
        const size_t g = (size_t)((sb[0][at] - a) & (K0 - 1)) * K1 + ((sb[1][at] - b) & (K1 - 1));
        atomicAdd(Q + g * K2 + gz, sw[0][a][at] * sw[1][b][at] * wz);
      }
    }
  }
}

// Everywhere else straight onto the mesh: a warp per PMG_ATOMS charges, every
// stencil point one atomic, the 32 / n rows of an instruction contiguous
// pieces.  Bound: the L2's atomic rate (about 0.75 T additions a second).
// Against tiles with shared atomics (us): 20,736 charges on 64^3 9.4 from 13.8
// in binary32, 12.9 from 24.4 in binary64; 65,536 on 128 x 128 x 512 23 from 47 and
// 30 from 74.
constexpr int PMG_ATOMS = 8, PMG_WARPS = 4;

template <class R, int NO>
__global__ void __launch_bounds__(32 * PMG_WARPS)
k_spme_spread_direct(int N, const typename V4<R>::T* __restrict__ pos, int K0, int K1, int K2,
                     const DevState* __restrict__ st, R* __restrict__ Q) {
  constexpr int RP = 32 / NO, NR = NO * NO, NI = (NR + RP - 1) / RP;
  __shared__ R sw[PMG_WARPS][3][PMG_ATOMS][NO];
  __shared__ int sb[PMG_WARPS][3][PMG_ATOMS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i0 = (blockIdx.x * PMG_WARPS + warp) * PMG_ATOMS;
  if (i0 >= N) return;
  const int na = min(PMG_ATOMS, N - i0);
  for (int t = lane; t < 3 * PMG_ATOMS; t += 32) {
    const int d = t / PMG_ATOMS, at = t - d * PMG_ATOMS;
    const typename V4<R>::T p = pos[i0 + min(at, na - 1)];
    int b;
    R f, w[NO], dw[NO];
    grid_coord<R>(d == 0 ? p.x : d == 1 ? p.y : p.z, (R)st->Li[d], d == 0 ? K0 : d == 1 ? K1 : K2, b, f);
    bsp_t<R, NO, false>(f, w, dw);
    sb[warp][d][at] = b;
#pragma unroll
    for (int j = 0; j < NO; ++j) sw[warp][d][at][j] = d == 2 ? w[j] * p.w : w[j];  // z weights carry the charge
  }
  __syncwarp();
  const int k = lane / NO, c = lane - k * NO;
  if (k >= RP) return;
  for (int at = 0; at < na; ++at) {
    const R wz = sw[warp][2][at][c];
    const int b0 = sb[warp][0][at], b1 = sb[warp][1][at], gz = (sb[warp][2][at] - c) & (K2 - 1);
#pragma unroll 8
    for (int j = 0; j < NI; ++j) {
      const int row = j * RP + k;
      if (row >= NR) break;
      const int a = row / NO, b = row - a * NO;
      const R v = sw[warp][0][at][a] * sw[warp][1][at][b] * wz;
      if (v != R(0)) atomicAdd(Q + (((b0 - a) & (K0 - 1)) * K1 + ((b1 - b) & (K1 - 1))) * K2 + gz, v);
    }
  }
}

// ---------------------------------------------------------------- gather, forces
// A warp takes PMG_ATOMS atoms, four at a time, and reads the mesh directly:
// the rows of one instruction are contiguous pieces of n points.  A lane sums
// its rows in the working precision, the lanes are added in FP64 with the four
// atoms' sums folded into one butterfly.  The weights of the warp's atoms are
// worked out once, one lane per (atom, axis), into shared memory.  Bound: L2
// reads where neighbouring atoms share little (ik, 65,536 charges on
// 128 x 128 x 512: 62 us for 270 MB of sectors), else latency.  Against staging
// each block's mesh region in shared memory (us): 20,736 charges on 64^3 14.6
// from 22.4 (ik), 11.6 from 25.1 (analytic); in binary64 15.5 from 37.7.  Orders 11
// to 14 put two rows to an instruction and go plane by plane (whole forces,
// 1,000,000 charges on 128^3 at order 14: 5.3 ms analytic and 6.3 ik, 8.1 and 8.2 with
// every row's weights read anew, 6.5 and 14.3 by staged regions).
//   MODE 0: ik, the three convolved meshes interleaved, one Real4 per point
//   MODE 1: analytic differentiation of the single convolved mesh
// store: force is a separate buffer that receives every atom's reciprocal
// force (zero for neutral atoms) instead of accumulating it.
template <class R, int NO, int MODE>
__global__ void __launch_bounds__(32 * PMG_WARPS)
k_spme_gather_t(int N, const typename V4<R>::T* __restrict__ pos, int K0, int K1, int K2,
                const DevState* __restrict__ st, const void* __restrict__ Gv, double4a* __restrict__ force, int store) {
  typedef typename V4<R>::T R4;
  constexpr int RP = 32 / NO, NR = NO * NO, NI = (NR + RP - 1) / RP;
  constexpr int ND = MODE == 0 ? 1 : 2;
  __shared__ R sw[PMG_WARPS][3][PMG_ATOMS][NO][ND];  // weights (and derivatives)
  __shared__ int sb[PMG_WARPS][3][PMG_ATOMS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i0 = (blockIdx.x * PMG_WARPS + warp) * PMG_ATOMS;
  if (i0 >= N) return;
  const int K[3] = {K0, K1, K2};
  R qa = R(0);  // charge of atom `lane` of the warp
  if (lane < PMG_ATOMS && i0 + lane < N) qa = pos[i0 + lane].w;
  for (int t = lane; t < 3 * PMG_ATOMS; t += 32) {
    const int d = t / PMG_ATOMS, at = t - d * PMG_ATOMS;
    const R4 p = pos[min(i0 + at, N - 1)];
    const R x = d == 0 ? p.x : d == 1 ? p.y : p.z;
    const int Kd = d == 0 ? K0 : d == 1 ? K1 : K2;
    int b;
    R f, w[NO], dw[NO];
    grid_coord<R>(x, (R)st->Li[d], Kd, b, f);
    bsp_t<R, NO, MODE != 0>(f, w, dw);
    sb[warp][d][at] = b;
#pragma unroll
    for (int j = 0; j < NO; ++j) {
      sw[warp][d][at][j][0] = w[j];
      if (ND == 2) sw[warp][d][at][j][ND - 1] = dw[j];
    }
  }
  __syncwarp();
  const unsigned charged = __ballot_sync(0xffffffffu, qa != R(0));
  const int k = lane / NO, c = lane - k * NO;
  const bool in = k < RP;
  double4a mine = {0.0, 0.0, 0.0, 0.0};  // sums of atom `lane` of the warp
#pragma unroll 1
  for (int g = 0; g < PMG_ATOMS; g += 4) {
    if (!((charged >> g) & 15u)) continue;
    double v[4][3];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int at = g + u;
      R s0 = R(0), s1 = R(0), s2 = R(0);
      if (((charged >> at) & 1u) && in) {
        const int b0 = sb[warp][0][at], b1 = sb[warp][1][at], gz = (sb[warp][2][at] - c) & (K2 - 1);
        const R wz = sw[warp][2][at][c][0];
        if constexpr (RP == 2) {
          // orders 11 to 14, two rows an instruction: the rows of a plane share its weights
#pragma unroll 1
          for (int a = 0; a < NO; ++a) {
            const size_t plane = (size_t)((b0 - a) & (K0 - 1)) * K1;
            R t0 = R(0), t1 = R(0), t2 = R(0);  // over the plane's rows: m w_b each, or m w_b and m w'_b
#pragma unroll
            for (int b = 0; b < NO; b += 2) {
              if (NO % 2 && b + k >= NO) break;
              const size_t at_mesh = (plane + ((b1 - b - k) & (K1 - 1))) * K2 + gz;
              const R wb = sw[warp][1][at][b + k][0];
              if constexpr (MODE == 0) {
                const R4 m = reinterpret_cast<const R4*>(Gv)[at_mesh];
                t0 += m.x * wb;
                t1 += m.y * wb;
                t2 += m.z * wb;
              } else {
                const R m = reinterpret_cast<const R*>(Gv)[at_mesh];
                t0 += m * wb;
                t1 += m * sw[warp][1][at][b + k][ND - 1];
              }
            }
            const R wa = sw[warp][0][at][a][0];
            if constexpr (MODE == 0) {
              s0 += wa * t0;
              s1 += wa * t1;
              s2 += wa * t2;
            } else {
              s0 += sw[warp][0][at][a][ND - 1] * t0;
              s1 += wa * t1;
              s2 += wa * t0;
            }
          }
        } else {
#pragma unroll 8
          for (int j = 0; j < NI; ++j) {
            const int row = j * RP + k;
            if (row < NR) {
              const int a = row / NO, b = row - a * NO;
              const size_t at_mesh = ((size_t)((b0 - a) & (K0 - 1)) * K1 + ((b1 - b) & (K1 - 1))) * K2 + gz;
              const R wa = sw[warp][0][at][a][0], wb = sw[warp][1][at][b][0];
              if constexpr (MODE == 0) {
                const R4 m = reinterpret_cast<const R4*>(Gv)[at_mesh];
                const R w = wa * wb;
                s0 += m.x * w;
                s1 += m.y * w;
                s2 += m.z * w;
              } else {
                const R m = reinterpret_cast<const R*>(Gv)[at_mesh];
                const R da = sw[warp][0][at][a][ND - 1], db = sw[warp][1][at][b][ND - 1];
                s0 += m * (da * wb);
                s1 += m * (wa * db);
                s2 += m * (wa * wb);
              }
            }
          }
        }
        if constexpr (MODE == 0) {
          s0 *= wz;
          s1 *= wz;
          s2 *= wz;
        } else {
          s0 *= -wz;
          s1 *= -wz;
          s2 *= -sw[warp][2][at][c][ND - 1];
        }
      }
      v[u][0] = (double)s0;
      v[u][1] = (double)s1;
      v[u][2] = (double)s2;
    }
    // four atoms' sums over the lanes: two folding steps leave each group of
    // 8 lanes with one atom, three more add it up
    double h[2][3], f[3];
    const bool up = lane & 16, up2 = lane & 8;
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const double keep = up ? v[u + 2][d] : v[u][d], give = up ? v[u][d] : v[u + 2][d];
        h[u][d] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
      }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double keep = up2 ? h[1][d] : h[0][d], give = up2 ? h[0][d] : h[1][d];
      f[d] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) f[d] += __shfl_xor_sync(0xffffffffu, f[d], o);
    }
    // lanes 8u .. 8u + 7 hold atom u; lane g + u takes it
    const int src = ((lane - g) & 3) * 8;
    const double f0 = __shfl_sync(0xffffffffu, f[0], src), f1 = __shfl_sync(0xffffffffu, f[1], src),
                 f2 = __shfl_sync(0xffffffffu, f[2], src);
    if (lane >= g && lane < g + 4) {
      mine.x = f0;
      mine.y = f1;
      mine.z = f2;
    }
  }
  const int i = i0 + lane;
  if (lane >= PMG_ATOMS || i >= N) return;
  double4a f = {0.0, 0.0, 0.0, 0.0};
  if (qa == R(0)) {
    if (store) force[i] = f;
    return;
  }
  if (!store) f = force[i];
  const double q = (double)qa;
  if (MODE == 0) {
    f.x += q * mine.x;
    f.y += q * mine.y;
    f.z += q * mine.z;
  } else {
    f.x += 2.0 * q * mine.x * K0 * st->Li[0];
    f.y += 2.0 * q * mine.y * K1 * st->Li[1];
    f.z += 2.0 * q * mine.z * K2 * st->Li[2];
  }
  force[i] = f;
}

// ---------------------------------------------------------------- gather, adjoint
// Potential dE/dq_i and exact position gradient dE/dx_i from the mesh Phi, in
// FP64 sums, in the caller's atom order.  A block of 32 atoms x LPA lanes
// stages the mesh region of its stencils in FP64 (one conversion per staged
// point instead of four per stencil point); lane a takes the stencil plane
// b0 - a and factors it by axis: per row the sums over c with the z weights
// and their derivatives, per plane the sums over the rows.  Per stencil point
// that is one shared load and two FMA (the four products per point it
// replaces needed 864 conversions an atom).  The weights are worked out once
// per (atom, axis).  1,048,576 charges, order 6: 887 -> 334 us, now bound by
// shared-memory wavefronts (76 %) and the staging latency; 20,736 in binary64:
// 31 -> 15 us.  A block whose region does not fit reads the mesh.
__host__ __device__ constexpr int gather_lanes(int order) { return order <= 4 ? 4 : (order <= 8 ? 8 : 16); }
constexpr int ADJ_ATOMS = 32;
constexpr int ADJ_TILE_BYTES = 44 * 1024;

template <class R, int NO>
__global__ void __launch_bounds__(ADJ_ATOMS * gather_lanes(NO), NO <= 6 ? 4 : 1)
k_spme_gather_adj(int N, const typename V4<R>::T* __restrict__ pos, const int* __restrict__ id, int K0, int K1, int K2,
                  const DevState* __restrict__ st, const R* __restrict__ G, double* __restrict__ dq,
                  double* __restrict__ dr, int tile_cap) {
  typedef typename V4<R>::T R4;
  constexpr int LPA = gather_lanes(NO), NT = ADJ_ATOMS * LPA;
  extern __shared__ __align__(16) unsigned char adj_smem[];
  double* tile = reinterpret_cast<double*>(adj_smem);
  __shared__ double2 sw[3][ADJ_ATOMS][NO];  // weight, derivative
  __shared__ int sb[3][ADJ_ATOMS], sbox[6];
  const int i0 = blockIdx.x * ADJ_ATOMS, na = min(ADJ_ATOMS, N - i0);
  for (int t = threadIdx.x; t < 3 * ADJ_ATOMS; t += NT) {
    const int d = t / ADJ_ATOMS, at = t - d * ADJ_ATOMS;  // one axis per warp
    int b = INT_MAX;
    const int Kd = d == 0 ? K0 : d == 1 ? K1 : K2;
    if (at < na) {
      const R4 p = pos[i0 + at], p0 = pos[i0];
      const R x = d == 0 ? p.x : d == 1 ? p.y : p.z, x0 = d == 0 ? p0.x : d == 1 ? p0.y : p0.z;
      int r;
      R f, fr, w[NO], dw[NO];
      grid_coord<R>(x, (R)st->Li[d], Kd, b, f);
      grid_coord<R>(x0, (R)st->Li[d], Kd, r, fr);
      const int dv = b - r;
      if (2 * dv > Kd) b -= Kd;
      else if (2 * dv < -Kd) b += Kd;
      bsp_t<R, NO, true>(f, w, dw);
#pragma unroll
      for (int j = 0; j < NO; ++j) sw[d][at][j] = make_double2((double)w[j], (double)dw[j]);
      sb[d][at] = b;
    }
    const int mn = __reduce_min_sync(0xffffffffu, b), mx = __reduce_max_sync(0xffffffffu, b == INT_MAX ? INT_MIN : b);
    if ((threadIdx.x & 31) == 0) {
      sbox[d] = mn;
      sbox[3 + d] = mx;
    }
  }
  __syncthreads();
  const int o0 = sbox[0] - (NO - 1), o1 = sbox[1] - (NO - 1), o2 = sbox[2] - (NO - 1);
  const long e0 = sbox[3] - o0 + 1, e1 = sbox[4] - o1 + 1, e2 = sbox[5] - o2 + 1;
  // odd plane stride: the planes of an atom fall on different banks
  const long ps = (e1 * e2) | 1;
  const bool staged = e0 * ps <= tile_cap;
  if (staged) {
    // 16 lanes along a row, two rows in flight per lane
    const int nrow = (int)(e0 * e1), ie1 = (int)e1, ie2 = (int)e2, ips = (int)ps;
    constexpr int RG = NT / 16;
    const int r0 = threadIdx.x >> 4, z0 = threadIdx.x & 15;
    int y = r0 % ie1, xx = r0 / ie1;
    for (int row = r0; row < nrow; row += 2 * RG) {
      const int xa = xx, ya = y;
      y += RG;
      while (y >= ie1) { y -= ie1; ++xx; }
      const bool two = row + RG < nrow;
      const R* ga = G + ((size_t)((o0 + xa) & (K0 - 1)) * K1 + ((o1 + ya) & (K1 - 1))) * K2;
      const R* gb = G + ((size_t)((o0 + xx) & (K0 - 1)) * K1 + ((o1 + y) & (K1 - 1))) * K2;
      double *ta = tile + xa * ips + ya * ie2, *tb = tile + xx * ips + y * ie2;
      y += RG;
      while (y >= ie1) { y -= ie1; ++xx; }
      for (int z = z0; z < ie2; z += 16) {
        const int gz = (o2 + z) & (K2 - 1);
        const R va = ga[gz], vb = two ? gb[gz] : R(0);
        ta[z] = (double)va;
        if (two) tb[z] = (double)vb;
      }
    }
    __syncthreads();
  }
  const int at = threadIdx.x / LPA, a = threadIdx.x & (LPA - 1);
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  if (at < na && a < NO) {
    double2 wz[NO];
#pragma unroll
    for (int c = 0; c < NO; ++c) wz[c] = sw[2][at][c];
    const int b0 = sb[0][at], b1 = sb[1][at], b2 = sb[2][at];
    double t0 = 0.0, t1 = 0.0, t2 = 0.0;  // sum over rows of w r0, w' r0, w r1
    const double* tp = tile + (b0 - a - o0) * (int)ps + (b1 - o1) * (int)e2 + (b2 - o2);
    const R* gp = G + (size_t)((b0 - a) & (K0 - 1)) * K1 * K2;
#pragma unroll 2
    for (int b = 0; b < NO; ++b) {
      double r0 = 0.0, r1 = 0.0;
      if (staged) {
        const double* tr = tp - b * (int)e2;
#pragma unroll
        for (int c = 0; c < NO; ++c) {
          const double g = tr[-c];
          r0 = fma(g, wz[c].x, r0);
          r1 = fma(g, wz[c].y, r1);
        }
      } else {
        const R* gr = gp + (size_t)((b1 - b) & (K1 - 1)) * K2;
#pragma unroll
        for (int c = 0; c < NO; ++c) {
          const double g = (double)gr[(b2 - c) & (K2 - 1)];
          r0 = fma(g, wz[c].x, r0);
          r1 = fma(g, wz[c].y, r1);
        }
      }
      const double2 wb = sw[1][at][b];
      t0 = fma(wb.x, r0, t0);
      t1 = fma(wb.y, r0, t1);
      t2 = fma(wb.x, r1, t2);
    }
    const double2 wa = sw[0][at][a];
    s[0] = wa.x * t0;
    s[1] = wa.y * t0;
    s[2] = wa.x * t1;
    s[3] = wa.x * t2;
  }
#pragma unroll
  for (int o = LPA / 2; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < 4; ++q) s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
  if (at >= na || a != 0) return;
  const int i = i0 + at, o = id[i];  // results in the caller's atom order
  if (dq) dq[o] = s[0];
  if (dr) {
    const double q = (double)pos[i].w;
    dr[3 * o] = q * s[1] * K0 * st->Li[0];
    dr[3 * o + 1] = q * s[2] * K1 * st->Li[1];
    dr[3 * o + 2] = q * s[3] * K2 * st->Li[2];
  }
}

const void* spread_tile_fn(int order) {
  switch (order) {
#define ORDER_CASE(NO) case NO: return (const void*)k_spme_spread_t<NO>;
    SPME_ORDERS(ORDER_CASE)
#undef ORDER_CASE
  }
  return nullptr;
}

template <class R>
const void* spread_direct_fn(int order) {
  switch (order) {
#define ORDER_CASE(NO) case NO: return (const void*)k_spme_spread_direct<R, NO>;
    SPME_ORDERS(ORDER_CASE)
#undef ORDER_CASE
  }
  return nullptr;
}

template <class R>
const void* gather_fn(int order, int mode) {
  switch (order) {
#define ORDER_CASE(NO)                                                           \
  case NO:                                                                       \
    return mode == 0 ? (const void*)k_spme_gather_t<R, NO, 0>                    \
                     : (mode == 1 ? (const void*)k_spme_gather_t<R, NO, 1> : (const void*)k_spme_gather_adj<R, NO>);
    SPME_ORDERS(ORDER_CASE)
#undef ORDER_CASE
  }
  return nullptr;
}

// The tile pays where many charges share its margins: binary32, 200,000 charges and
// more on at most 10 mesh points per charge (forces by analytic differentiation, us,
// direct / tile of 32 charges at order 6 and 8: 1,000,000 charges on 8.4 points each
// 709 / 669 and 1,177 / 1,027, on 16.8 994 / 1,073 and 1,459 / 1,463; 400,000 on 5.2 290 /
// 272 and 486 / 394, on 10.5 309 / 307 and 500 / 474, on 21 360 / 421 and 554 / 553; 200,000 on
// 5.2 171 / 164 and 274 / 228, on 10.5 175 / 180 and 275 / 265; at order 4 the two are within
// 4 % of each other there).  16 KB hold the stencils of 32 charges in cell order at
// these densities.
constexpr int SPREAD_TILE_MIN = 200000, SPREAD_TILE_PPC = 10, SPREAD_TILE_BYTES = 16 * 1024;
bool spread_by_tile(int prec, int N, const int K[3]) {
  return prec == MD_PREC_MIXED && N >= SPREAD_TILE_MIN && (double)K[0] * K[1] * K[2] / N <= SPREAD_TILE_PPC;
}

}  // namespace

int pm_prepare(int prec, int order) {
  const void* g = prec == MD_PREC_FP64 ? gather_fn<double>(order, 2) : gather_fn<float>(order, 2);
  MD_CUDA(cudaFuncSetAttribute(g, cudaFuncAttributeMaxDynamicSharedMemorySize, ADJ_TILE_BYTES));
  return MD_OK;
}

int pm_spread(md_system* sys, const int K[3], int order, void* Q, Recorder* rec) {
  int K0 = K[0], K1 = K[1], K2 = K[2], N = sys->N;
  DevState* st = sys->st;
  const void* pos = sys->pos;
  if (spread_by_tile(sys->prec, N, K)) {
    int cap = SPREAD_TILE_BYTES / (int)sizeof(float);
    void* a[] = {&N, &pos, &K0, &K1, &K2, &st, &Q, &cap};
    return rec_launch(rec, spread_tile_fn(order), dim3(ceil_div(N, SPREAD_CHARGES)), dim3(SPREAD_THREADS),
                      SPREAD_TILE_BYTES, a);
  }
  void* a[] = {&N, &pos, &K0, &K1, &K2, &st, &Q};
  return rec_launch(rec, sys->prec == MD_PREC_FP64 ? spread_direct_fn<double>(order) : spread_direct_fn<float>(order),
                    dim3(ceil_div(N, PMG_ATOMS * PMG_WARPS)), dim3(32 * PMG_WARPS), 0, a);
}

int pm_gather(md_system* sys, const int K[3], int order, int method, const void* G, double4a* force, int store,
              Recorder* rec) {
  int K0 = K[0], K1 = K[1], K2 = K[2], N = sys->N;
  DevState* st = sys->st;
  const void* pos = sys->pos;
  void* a[] = {&N, &pos, &K0, &K1, &K2, &st, &G, &force, &store};
  return rec_launch(rec, sys->prec == MD_PREC_FP64 ? gather_fn<double>(order, method) : gather_fn<float>(order, method),
                    dim3(ceil_div(N, PMG_ATOMS * PMG_WARPS)), dim3(32 * PMG_WARPS), 0, a);
}

int pm_gather_adjoint(md_system* sys, const int K[3], int order, const void* G, double* dq, double* dr, Recorder* rec) {
  int K0 = K[0], K1 = K[1], K2 = K[2], N = sys->N, cap = ADJ_TILE_BYTES / (int)sizeof(double);
  DevState* st = sys->st;
  const void* pos = sys->pos;
  void* a[] = {&N, &pos, &sys->id, &K0, &K1, &K2, &st, &G, &dq, &dr, &cap};
  return rec_launch(rec, sys->prec == MD_PREC_FP64 ? gather_fn<double>(order, 2) : gather_fn<float>(order, 2),
                    dim3(ceil_div(N, ADJ_ATOMS)), dim3(ADJ_ATOMS * gather_lanes(order)), ADJ_TILE_BYTES, a);
}

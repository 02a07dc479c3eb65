// Kernels of the residual L(U) and of the SSP-RK3 step around it.
//
// Data layout.  The caller's state is a strided 3-D array (i, j, channel)
// addressed as p[i*s0 + j*s1 + k*s2] -- the reference's (nx+6, ny+6, C) C-order
// array (s0 = (ny+6)*C, s1 = C, s2 = 1) or the solver's structure-of-arrays
// planes (s0 = ny+6, s1 = 1, s2 = plane).  j is the contiguous axis and maps to
// threadIdx.x.  Intermediate face data live in workspace planes of one
// component each (`Planes`), so every warp load and store is a contiguous run.
//
// Residual pipeline for one direction (x shown; y swaps the roles of i and j):
//   pass1   (m-5) x n   faces x columns : normal WENO5 (char or cons) -> q_l, q_r
//   pass2   (m-5) x (n-6) faces        : transverse 2-point Gauss WENO of q_l,
//           q_r, Euler fluxes of the four Gauss states, face averages (the FAST
//           HLLE takes their doubles, the Gauss-point sums), then the HLLE
//           flux, or HLLC + HLLE + mean pressure for the sensor blend
//   blend   (sensor blend only)        : pressure-gradient weight, F
//   residual (m-6) x (n-6) cells       : -(dF/dx + dG/dy), optionally fused
//           with the SSP-RK3 stage combination.
#pragma once

#include "euler_math.cuh"
#include "step_ctl.h"

namespace weno {
inline namespace WENO_TU_NS {

template <class T>
struct CView {
  const T* p;
  int64_t s0, s1, s2;
  __device__ __forceinline__ T at(int64_t i, int64_t j, int k) const { return p[i * s0 + j * s1 + k * s2]; }
};

// A set of planes: component k, element (r, c) at p[k*ps + r*ld + c].
template <class T>
struct Planes {
  T* p;
  int64_t ps, ld;
  __device__ __forceinline__ T& at(int k, int64_t r, int64_t c) const { return p[k * ps + r * ld + c]; }
};

// The (row, column) of this thread in a rows x cols index space: of a 2-D grid of
// (32, 4) blocks, or with one-row blocks of the flattened space (launch_impl.cuh
// says which is launched when).  False past the end.
__device__ __forceinline__ bool locate(int64_t rows, int64_t cols, int64_t& row, int64_t& col) {
  if (blockDim.y == 1) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= rows * cols) return false;
    if (rows * cols < ((int64_t)1 << 32)) {
      const uint32_t q = (uint32_t)e / (uint32_t)cols;
      row = q;
      col = (uint32_t)e - q * (uint32_t)cols;
    } else {
      row = e / cols;
      col = e - row * cols;
    }
    return true;
  }
  col = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  row = (int64_t)blockIdx.y * blockDim.y + threadIdx.y;
  return row < rows && col < cols;
}

// ---------------------------------------------------------------------------
// Pass 1 (weno.rs:390-454 characteristic, weno.rs:654-717 component-wise)
// ---------------------------------------------------------------------------
// What the df64 pass 1 leaves in plane 0 of q_l for a face that k_pass1_marked has
// to reconstruct: a NaN no arithmetic produces.
constexpr uint32_t kDf64Marker = 0x7fc0df64u;

// Resident blocks per SM that pass 1 is compiled for (4 warps each).  FP64: 4, at
// 128 registers (at three blocks the FAST 2048^2 step took 2.6 % longer, exact ones
// of 300 x 310 2.6 % and of 2000 x 1500 0.3 %); FP32: 8, at 64 (6: 2.7 % longer, 7:
// 1 %, 9 spills: 1.6 %); df64: 4 (3: 2 % longer).
template <class T>
constexpr int kPass1Blocks = is_native_f64<T> ? 4 : (is_f32<T> ? 8 : 4);

// Pass 1, one face per thread.  FP64 is bound by its pipe, so what counts is FP64
// instructions per face: FAST, characteristic, 214 with the weights on the FP32 pipe
// (447 with FP64 weights), a 2048^2 sweep 1.57 ms for 3.66, the pipe 91.5 % busy and
// HBM at 3 %.  FP32 and df64 are bound by issue slots.
template <class T, bool FAST, bool Y, bool CHAR>
__global__ void __launch_bounds__(128, kPass1Blocks<T>) k_pass1(CView<T> u, int64_t rows, int64_t cols, T gamma, Planes<T> PL,
                                                Planes<T> PR, T weps) {
  int64_t row, col;
  if (!locate(rows, cols, row, col)) return;
  T c[6][4];
#pragma unroll
  for (int s = 0; s < 6; ++s)
#pragma unroll
    for (int k = 0; k < 4; ++k) c[s][k] = Y ? u.at(row, col + s, k) : u.at(row + s, col, k);
  T ql[4], qr[4];
  if constexpr (std::is_same<T, df64>::value) {
    // df64 has the float exponent range: a face whose stencil holds a tiny
    // density or a huge value (near vacuum the characteristic projection scales
    // by 1/(rho*c)) is left to k_pass1_marked, in native double: with that code
    // in this kernel its registers would bind every face (168 where 128, with 64 bytes
    // of spills in the characteristic form, serve without it).
    bool safe = true;
#pragma unroll
    for (int s = 0; s < 6; ++s) {
      safe = safe && c[s][0].hi > 1e-6f;
#pragma unroll
      for (int k = 0; k < 4; ++k) safe = safe && fabsf(c[s][k].hi) < 1e15f;
    }
    if (!safe) {
      PL.at(0, row, col) = df64(__uint_as_float(kDf64Marker), 0.0f);
      return;
    }
    pass1_face<T, FAST, Y, CHAR>(c, gamma, ql, qr, weps);
  } else {
    pass1_face<T, FAST, Y, CHAR>(c, gamma, ql, qr, weps);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    PL.at(k, row, col) = ql[k];
    PR.at(k, row, col) = qr[k];
  }
}

// The faces k_pass1<df64> marked, in native double.
template <bool Y, bool CHAR>
__global__ void __launch_bounds__(128) k_pass1_marked(CView<df64> u, int64_t rows, int64_t cols, df64 gamma,
                                                       Planes<df64> PL, Planes<df64> PR, df64 weps) {
  int64_t row, col;
  if (!locate(rows, cols, row, col)) return;
  if (__float_as_uint(PL.at(0, row, col).hi) != kDf64Marker) return;
  f64 c[6][4], l[4], r[4];
#pragma unroll
  for (int s = 0; s < 6; ++s)
#pragma unroll
    for (int k = 0; k < 4; ++k) c[s][k] = f64((double)(Y ? u.at(row, col + s, k) : u.at(row + s, col, k)));
  pass1_face<f64, true, Y, CHAR>(c, f64((double)gamma), l, r, f64((double)weps));
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    PL.at(k, row, col) = df64(l[k].v);
    PR.at(k, row, col) = df64(r[k].v);
  }
}

// Component-wise pass 1, one cell per thread: the cell's indicators serve the
// state at its right face (q_l there) and at its left face (q_r there), so every
// stencil's are formed once instead of on two faces.  Thread t of a sweep owns
// the cell t + 2, the left one of face t and the right one of face t - 1.  Bound as
// k_pass1; with the float-pair weights the 2048^2 FAST FP64 component-wise step (all
// kernels) takes 14.8 ms for 35.9, the exact one 50.2 ms.
template <class T, bool FAST, bool Y>
__global__ void __launch_bounds__(128) k_pass1_cells(CView<T> u, int64_t rows, int64_t cols, Planes<T> PL,
                                                      Planes<T> PR, T weps) {
  int64_t row, col;
  if (!locate(Y ? rows : rows + 1, Y ? cols + 1 : cols, row, col)) return;
  const bool has_l = Y ? col < cols : row < rows, has_r = Y ? col > 0 : row > 0;
  const int64_t rr = Y ? row : row - 1, rc = Y ? col - 1 : col;
  constexpr int STEP = is_f32<T> ? 2 : 1;
#pragma unroll(is_f32<T> ? 2 : 1)
  for (int k = 0; k < 4; k += STEP) {
    if constexpr (is_f32<T>) {
      f32x2 v[5], l, r;
#pragma unroll
      for (int s = 0; s < 5; ++s)
        v[s] = Y ? f32x2(u.at(row, col + s, k), u.at(row, col + s, k + 1))
                 : f32x2(u.at(row + s, col, k), u.at(row + s, col, k + 1));
      weno5_cell_fast<f32x2>(v, f32x2(weps), r, l);
      if (has_l) {
        PL.at(k, row, col) = l.v.x;
        PL.at(k + 1, row, col) = l.v.y;
      }
      if (has_r) {
        PR.at(k, rr, rc) = r.v.x;
        PR.at(k + 1, rr, rc) = r.v.y;
      }
    } else {
      T v[5], l, r;
#pragma unroll
      for (int s = 0; s < 5; ++s) v[s] = Y ? u.at(row, col + s, k) : u.at(row + s, col, k);
      if constexpr (FAST) weno5_cell_fast<T>(v, weps, r, l);
      else weno5_cell_exact<T>(v, weps, r, l);
      if (has_l) PL.at(k, row, col) = l;
      if (has_r) PR.at(k, rr, rc) = r;
    }
  }
}

// ---------------------------------------------------------------------------
// Pass 2 (weno.rs:460-501 / :587-631) + Riemann solver (riemann.rs)
// ---------------------------------------------------------------------------
enum Pass2Out : int {
  P2_STATES = 0,  // q_l, f_l, q_r, f_r as four dense (rows, cols, 4) arrays
  P2_HLLE = 1,    // HLLE flux planes F[4]
  P2_BLEND = 2,   // HLLC planes Fc[4], HLLE planes Fe[4], mean pressure plane
};

struct Pass2Dst {
  void* a;  // P2_STATES: q_l ; P2_HLLE: F planes ; P2_BLEND: Fc planes
  void* b;  // P2_STATES: f_l ;                      P2_BLEND: Fe planes
  void* c;  // P2_STATES: q_r ;                      P2_BLEND: pbar plane
  void* d;  // P2_STATES: f_r
  int64_t ps, ld;
};

template <class T, bool FAST, bool Y>
__device__ __forceinline__ void gq_face(const Planes<T>& P, int64_t row, int64_t col, T q1[4], T q2[4], T weps) {
#pragma unroll(kFieldUnroll<T>)
  for (int k = 0; k < 4; ++k) {
    T s[5], a, b;
#pragma unroll
    for (int t = 0; t < 5; ++t) s[t] = Y ? P.at(k, row + 1 + t, col) : P.at(k, row, col + 1 + t);
    weno5_gq_pair<T, FAST>(s[0], s[1], s[2], s[3], s[4], a, b, weps);
    put4(q1, k, a);
    put4(q2, k, b);
  }
}

// The Riemann solver and the stores of one pass-2 face (row, col).
// S = 2 (FAST, P2_HLLE): the states and fluxes are twice the face averages.
template <class T, bool FAST, bool Y, int OUT, int S = 1>
__device__ __forceinline__ void pass2_emit(const T ql[4], const T fl[4], const T qr[4], const T fr[4], T gamma,
                                           const Pass2Dst& dst, int64_t row, int64_t col, int64_t cols) {
  static_assert(S == 1 || OUT == P2_HLLE, "doubled states feed the HLLE flux only");
  const int64_t e = row * dst.ld + col;
  if constexpr (OUT == P2_STATES) {
    const int64_t o = (row * cols + col) * 4;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      static_cast<T*>(dst.a)[o + k] = ql[k];
      static_cast<T*>(dst.b)[o + k] = fl[k];
      static_cast<T*>(dst.c)[o + k] = qr[k];
      static_cast<T*>(dst.d)[o + k] = fr[k];
    }
  } else {
    const RiemannPre<T, FAST, Y> r = riemann_pre<T, FAST, Y, S>(ql, qr, gamma);
    T F[4];
    hlle_flux<T, FAST, Y, S>(r, ql, fl, qr, fr, F);
    if constexpr (OUT == P2_HLLE) {
#pragma unroll
      for (int k = 0; k < 4; ++k) static_cast<T*>(dst.a)[k * dst.ps + e] = F[k];
    } else {
      T G[4];
      hllc_flux<T, FAST, Y>(r, ql, fl, qr, fr, G);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        static_cast<T*>(dst.a)[k * dst.ps + e] = G[k];
        static_cast<T*>(dst.b)[k * dst.ps + e] = F[k];
      }
      // con2primi pressure of q_l and q_r is the clamped p of the solver
      // preamble (utils.rs:28 == riemann.rs:33-36).
      static_cast<T*>(dst.c)[e] = T(0.5) * (r.p_l + r.p_r);
    }
  }
}

template <class T, bool FAST, bool Y, int OUT>
__global__ void __launch_bounds__(128) k_pass2(Planes<T> PL, Planes<T> PR, int64_t rows, int64_t cols, T gamma,
                                                Pass2Dst dst, T weps) {
  int64_t row, col;
  if (!locate(rows, cols, row, col)) return;
  T ql[4], qr[4], fl[4], fr[4];
#pragma unroll(is_f32<T> ? 2 : 1)
  for (int side = 0; side < 2; ++side) {
    T a1[4], a2[4], f1[4], f2[4];
    const Planes<T> P{side ? PR.p : PL.p, PL.ps, PL.ld};
    gq_face<T, FAST, Y>(P, row, col, a1, a2, weps);
    euler_flux_pair<T, FAST, Y>(a1, a2, gamma, f1, f2);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const T f = mul_pow2<-1>(T(f1[k] + f2[k])), q = mul_pow2<-1>(T(a1[k] + a2[k]));
      fl[k] = side ? fl[k] : f;
      ql[k] = side ? ql[k] : q;
      fr[k] = f;
      qr[k] = q;
    }
  }
  pass2_emit<T, FAST, Y, OUT>(ql, fl, qr, fr, gamma, dst, row, col, cols);
}

// Face-averaged states and fluxes of two neighbouring faces (along the
// transverse direction) from one side's pass-1 planes, FAST arithmetic.  SUM:
// twice the averages (the Gauss-point sums), for the doubled-state HLLE.
template <class T, bool Y, bool SUM = false>
__device__ __forceinline__ void gq_side_two(const Planes<T>& P, int64_t row, int64_t col, T gamma, T weps, T qA[4],
                                            T fA[4], T qB[4], T fB[4]) {
  T a1A[4], a2A[4], a1B[4], a2B[4];
  if constexpr (is_f32<T>) {
    // components (0,1) and (2,3) as packed pairs on the FP32x2 instructions
#pragma unroll
    for (int k = 0; k < 4; k += 2) {
      f32x2 v[6];
#pragma unroll
      for (int t = 0; t < 6; ++t)
        v[t] = Y ? f32x2(P.at(k, row + 1 + t, col), P.at(k + 1, row + 1 + t, col))
                 : f32x2(P.at(k, row, col + 1 + t), P.at(k + 1, row, col + 1 + t));
      f32x2 raA, rbA, raB, rbB;
      weno5_gq_two<f32x2>(v[0], v[1], v[2], v[3], v[4], v[5], f32x2(weps), raA, rbA, raB, rbB);
      a1A[k] = raA.v.x, a1A[k + 1] = raA.v.y, a2A[k] = rbA.v.x, a2A[k + 1] = rbA.v.y;
      a1B[k] = raB.v.x, a1B[k + 1] = raB.v.y, a2B[k] = rbB.v.x, a2B[k + 1] = rbB.v.y;
    }
  } else {
#pragma unroll(kFieldUnroll<T>)
    for (int k = 0; k < 4; ++k) {
      T v[6], pA, mA, pB, mB;
#pragma unroll
      for (int t = 0; t < 6; ++t) v[t] = Y ? P.at(k, row + 1 + t, col) : P.at(k, row, col + 1 + t);
      weno5_gq_two<T>(v[0], v[1], v[2], v[3], v[4], v[5], weps, pA, mA, pB, mB);
      put4(a1A, k, pA);
      put4(a2A, k, mA);
      put4(a1B, k, pB);
      put4(a2B, k, mB);
    }
  }
  euler_flux_sum<T, Y>(a1A, a2A, gamma, fA);
  euler_flux_sum<T, Y>(a1B, a2B, gamma, fB);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    qA[k] = a1A[k] + a2A[k];
    qB[k] = a1B[k] + a2B[k];
    if constexpr (!SUM) {
      fA[k] = half(fA[k]);
      qA[k] = half(qA[k]);
      fB[k] = half(fB[k]);
      qB[k] = half(qB[k]);
    }
  }
}

// Resident blocks per SM that k_pass2_two is compiled for.  The FP64 blend takes 136
// registers in the x sweep unbounded, three blocks; at four (128) two component-wise
// blend steps of 1024 x 1030 take 9.42-9.56 ms for 9.73-9.82, characteristic ones of
// 2000 x 700 16.68 for 17.04.  The others fit four (FP64) or seven to eight (FP32) as
// they are, and slow down with a bound: FP64 HLLE by 0.5 % at 4, FP32 by 0.1-0.8 % at 8
// and 3 % at 9.
template <class T, int OUT>
constexpr int kPass2Blocks = is_native_f64<T> && OUT == P2_BLEND ? 4 : 0;

// FAST pass 2 with two faces per thread along the transverse direction
// (columns for the x sweep, rows for the y sweep): the six transverse values
// of each component serve both faces, whose Gauss-point reconstructions share
// their first and second differences.  FP64: 220 instructions of the pipe per face
// with the weights on the FP32 pipe (453 with FP64 weights), a 2048^2 HLLE sweep
// 1.72 ms for 3.74, the pipe 84-86 % busy.
template <class T, bool Y, int OUT>
__global__ void __launch_bounds__(128, kPass2Blocks<T, OUT>) k_pass2_two(Planes<T> PL, Planes<T> PR, int64_t rows, int64_t cols, T gamma,
                                                    Pass2Dst dst, T weps) {
  int64_t row, col;
  if (!locate(Y ? (rows + 1) / 2 : rows, Y ? cols : (cols + 1) / 2, row, col)) return;
  if constexpr (Y) row *= 2;
  else col *= 2;
  const bool two = Y ? (row + 1 < rows) : (col + 1 < cols);
  // the HLLE flux takes the Gauss-point sums (twice the face averages)
  constexpr bool SUM = OUT == P2_HLLE;
  constexpr int S = SUM ? 2 : 1;
  T qlA[4], flA[4], qlB[4], flB[4], qrA[4], frA[4], qrB[4], frB[4];
  if constexpr (is_native_f64<T>) {
#pragma unroll 1
    for (int side = 0; side < 2; ++side) {  // one copy of the code, left then right
      const Planes<T> P{side ? PR.p : PL.p, PL.ps, PL.ld};
      gq_side_two<T, Y, SUM>(P, row, col, gamma, weps, qrA, frA, qrB, frB);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        qlA[k] = side ? qlA[k] : qrA[k];
        flA[k] = side ? flA[k] : frA[k];
        qlB[k] = side ? qlB[k] : qrB[k];
        flB[k] = side ? flB[k] : frB[k];
      }
    }
  } else {
    gq_side_two<T, Y, SUM>(PL, row, col, gamma, weps, qlA, flA, qlB, flB);
    gq_side_two<T, Y, SUM>(PR, row, col, gamma, weps, qrA, frA, qrB, frB);
  }
  if constexpr (is_native_f64<T>) {
#pragma unroll 1
    for (int face = 0; face < (two ? 2 : 1); ++face) {
      pass2_emit<T, true, Y, OUT, S>(qlA, flA, qrA, frA, gamma, dst, Y ? row + face : row, Y ? col : col + face, cols);
#pragma unroll
      for (int k = 0; k < 4; ++k) qlA[k] = qlB[k], flA[k] = flB[k], qrA[k] = qrB[k], frA[k] = frB[k];
    }
  } else {
    pass2_emit<T, true, Y, OUT, S>(qlA, flA, qrA, frA, gamma, dst, row, col, cols);
    if (two)
      pass2_emit<T, true, Y, OUT, S>(qlB, flB, qrB, frB, gamma, dst, Y ? row + 1 : row, Y ? col : col + 1, cols);
  }
}

// ---------------------------------------------------------------------------
// Small FP64 grids: four lanes per face.  With fewer than about four warps per SM
// (the line is in launch_api.h) the one-thread-per-face kernels wait for their own
// chain of dependent operations (an FP64 one takes 64 cycles: a 64 x 64 residual spent
// 50 us in each of four passes); a quad shares the fields of a face among its lanes, which costs a third
// more FP64 instructions (the averages, repeated on four lanes) and leaves a
// chain about a sixth as long.  The faces' values are those of k_pass1 / k_pass2 /
// k_pass2_two operation by operation.
// ---------------------------------------------------------------------------
// The face (row, col) and component of this lane; lanes past the end work on the
// last face and store nothing.
__device__ __forceinline__ bool locate_quad(unsigned block, int64_t rows, int64_t cols, int64_t& row, int64_t& col,
                                            int& k) {
  int64_t e = ((int64_t)block * blockDim.x + threadIdx.x) >> 2;
  k = threadIdx.x & 3;
  const bool in = e < rows * cols;
  if (!in) e = rows * cols - 1;
  row = e / cols;
  col = e - row * cols;
  return in;
}

template <bool FAST, bool Y, bool CHAR>
__device__ __forceinline__ void pass1_quad(unsigned block, const CView<f64>& u, int64_t rows, int64_t cols, f64 gamma,
                                           const Planes<f64>& PL, const Planes<f64>& PR, f64 weps) {
  int64_t row, col;
  int k;
  const bool in = locate_quad(block, rows, cols, row, col, k);
  f64 c[6][4], l, r;
#pragma unroll
  for (int s = 0; s < 6; ++s)
#pragma unroll
    for (int j = 0; j < 4; ++j) c[s][j] = Y ? u.at(row, col + s, j) : u.at(row + s, col, j);
  pass1_face_quad<f64, FAST, Y, CHAR>(c, k, gamma, l, r, weps);
  if (!in) return;
  PL.at(k, row, col) = l;
  PR.at(k, row, col) = r;
}

// Pass 1 of an (m, n) array: the first nbx blocks the x faces, the others the y
// faces (either may be none), so that one launch covers both sweeps.
template <bool FAST, bool CHAR>
__global__ void __launch_bounds__(32) k_pass1_quad(CView<f64> u, int64_t m, int64_t n, unsigned nbx, f64 gamma,
                                                    Planes<f64> PLx, Planes<f64> PRx, Planes<f64> PLy,
                                                    Planes<f64> PRy, f64 weps) {
  if (blockIdx.x < nbx) pass1_quad<FAST, false, CHAR>(blockIdx.x, u, m - 5, n, gamma, PLx, PRx, weps);
  else pass1_quad<FAST, true, CHAR>(blockIdx.x - nbx, u, m, n - 5, gamma, PLy, PRy, weps);
}

template <bool FAST, bool Y, int OUT>
__device__ __forceinline__ void pass2_quad(unsigned block, const Planes<f64>& PL, const Planes<f64>& PR, int64_t rows,
                                           int64_t cols, f64 gamma, const Pass2Dst& dst, f64 weps) {
  int64_t row, col;
  int k;
  const bool in = locate_quad(block, rows, cols, row, col, k);
  constexpr bool SUM = FAST && OUT == P2_HLLE;
  constexpr int S = SUM ? 2 : 1;
  f64 ql[4], fl[4], qr[4], fr[4];
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    const Planes<f64> P{side ? PR.p : PL.p, PL.ps, PL.ld};
    f64 s[5], a, b, a1[4], a2[4];
#pragma unroll
    for (int t = 0; t < 5; ++t) s[t] = Y ? P.at(k, row + 1 + t, col) : P.at(k, row, col + 1 + t);
    weno5_gq_pair<f64, FAST, 3>(s[0], s[1], s[2], s[3], s[4], a, b, weps);
    quad_gather(a, a1);
    quad_gather(b, a2);
    f64 f[4];
    if constexpr (FAST) {
      euler_flux_sum<f64, Y>(a1, a2, gamma, f);
    } else {
      f64 f1[4], f2[4];
      euler_flux_pair<f64, false, Y>(a1, a2, gamma, f1, f2);
#pragma unroll
      for (int j = 0; j < 4; ++j) f[j] = f1[j] + f2[j];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const f64 q = SUM ? a1[j] + a2[j] : half(a1[j] + a2[j]);
      const f64 g = SUM ? f[j] : half(f[j]);
      ql[j] = side ? ql[j] : q;
      fl[j] = side ? fl[j] : g;
      qr[j] = q;
      fr[j] = g;
    }
  }
  const int64_t e = row * dst.ld + col;
  if constexpr (OUT == P2_STATES) {
    if (!in) return;
    const int64_t o = (row * cols + col) * 4 + k;
    static_cast<f64*>(dst.a)[o] = pick4(ql, k);
    static_cast<f64*>(dst.b)[o] = pick4(fl, k);
    static_cast<f64*>(dst.c)[o] = pick4(qr, k);
    static_cast<f64*>(dst.d)[o] = pick4(fr, k);
  } else {
    const RiemannPre<f64, FAST, Y> r = riemann_pre<f64, FAST, Y, S>(ql, qr, gamma);
    f64 F[4];
    hlle_flux<f64, FAST, Y, S>(r, ql, fl, qr, fr, F);
    if constexpr (OUT == P2_HLLE) {
      if (in) static_cast<f64*>(dst.a)[k * dst.ps + e] = pick4(F, k);
    } else {
      f64 G[4];
      hllc_flux<f64, FAST, Y>(r, ql, fl, qr, fr, G);
      if (!in) return;
      static_cast<f64*>(dst.a)[k * dst.ps + e] = pick4(G, k);
      static_cast<f64*>(dst.b)[k * dst.ps + e] = pick4(F, k);
      if (k == 0) static_cast<f64*>(dst.c)[e] = f64(0.5) * (r.p_l + r.p_r);
    }
  }
}

// Pass 2 of the same: (m-5) x (n-6) x faces, then (m-6) x (n-5) y faces.
template <bool FAST, int OUT>
__global__ void __launch_bounds__(32) k_pass2_quad(Planes<f64> PLx, Planes<f64> PRx, Planes<f64> PLy, Planes<f64> PRy,
                                                    int64_t m, int64_t n, unsigned nbx, f64 gamma, Pass2Dst dx,
                                                    Pass2Dst dy, f64 weps) {
  if (blockIdx.x < nbx) pass2_quad<FAST, false, OUT>(blockIdx.x, PLx, PRx, m - 5, n - 6, gamma, dx, weps);
  else pass2_quad<FAST, true, OUT>(blockIdx.x - nbx, PLy, PRy, m - 6, n - 5, gamma, dy, weps);
}

// Riemann solver on caller-provided dense (rows, cols, 4) face arrays
// (hllc_x_rs_py & co, lib.rs:54-132).  KIND 0: HLLC -> out dense;
// KIND 1: HLLE -> out dense; KIND 2: HLLC, HLLE and mean pressure -> planes
// for k_blend.
template <class T, bool FAST, bool Y, int KIND>
__global__ void __launch_bounds__(128) k_riemann(const T* QL, const T* FL, const T* QR, const T* FR, int64_t rows,
                                                  int64_t cols, T gamma, T* out, Planes<T> Fc, Planes<T> Fe,
                                                  Planes<T> Pbar) {
  int64_t row, col;
  if (!locate(rows, cols, row, col)) return;
  const int64_t o = (row * cols + col) * 4;
  T ql[4], qr[4], fl[4], fr[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    ql[k] = QL[o + k]; fl[k] = FL[o + k]; qr[k] = QR[o + k]; fr[k] = FR[o + k];
  }
  const RiemannPre<T, FAST, Y> r = riemann_pre<T, FAST, Y>(ql, qr, gamma);
  T F[4];
  if constexpr (KIND == 0) {
    hllc_flux<T, FAST, Y>(r, ql, fl, qr, fr, F);
#pragma unroll
    for (int k = 0; k < 4; ++k) out[o + k] = F[k];
  } else if constexpr (KIND == 1) {
    hlle_flux<T, FAST, Y>(r, ql, fl, qr, fr, F);
#pragma unroll
    for (int k = 0; k < 4; ++k) out[o + k] = F[k];
  } else {
    T G[4];
    hllc_flux<T, FAST, Y>(r, ql, fl, qr, fr, G);
    hlle_flux<T, FAST, Y>(r, ql, fl, qr, fr, F);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      Fc.at(k, row, col) = G[k];
      Fe.at(k, row, col) = F[k];
    }
    Pbar.at(0, row, col) = T(0.5) * (r.p_l + r.p_r);
  }
}

// ---------------------------------------------------------------------------
// Sensor blend (riemann.rs:352-410 shock_sensor_grad_p and riemann.rs:412-448).
// The derivative spacing is 1/min(rows, cols) of the face array, with one-sided
// differences (still divided by 2*dx) on its edges.  rows, cols >= 2.
// Output: planes (DENSE = false) or a dense (rows, cols, 4) array.
// ---------------------------------------------------------------------------
template <class T, bool FAST>
__device__ __forceinline__ T blend_weight(const Planes<T>& Pbar, int64_t rows, int64_t cols, int64_t row, int64_t col,
                                          T jp_lo, T jp_hi) {
  const int64_t min_dim = rows < cols ? rows : cols;
  const T dx = T(1.0) / T((double)min_dim);
  const T two_dx = T(2.0) * dx;
  const int64_t ra = row == 0 ? 0 : (row == rows - 1 ? rows - 2 : row - 1);
  const int64_t rb = row == 0 ? 1 : (row == rows - 1 ? rows - 1 : row + 1);
  const int64_t ca = col == 0 ? 0 : (col == cols - 1 ? cols - 2 : col - 1);
  const int64_t cb = col == 0 ? 1 : (col == cols - 1 ? cols - 1 : col + 1);
  const T p = Pbar.at(0, row, col);
  const T dpdx = qdiv<T, FAST>(Pbar.at(0, rb, col) - Pbar.at(0, ra, col), two_dx);
  const T dpdy = qdiv<T, FAST>(Pbar.at(0, row, cb) - Pbar.at(0, row, ca), two_dx);
  return sensor_weight<T, FAST>(dpdx, dpdy, p, jp_lo, jp_hi);
}

template <class T, bool FAST, bool DENSE>
__global__ void __launch_bounds__(128) k_blend(Planes<T> Fc, Planes<T> Fe, Planes<T> Pbar, int64_t rows,
                                                int64_t cols, T jp_lo, T jp_hi, T* out, Planes<T> Fout) {
  int64_t row, col;
  if (!locate(rows, cols, row, col)) return;
  const T w = blend_weight<T, FAST>(Pbar, rows, cols, row, col, jp_lo, jp_hi);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const T f = w * Fc.at(k, row, col) + (T(1.0) - w) * Fe.at(k, row, col);
    if constexpr (DENSE) out[(row * cols + col) * 4 + k] = f;
    else Fout.at(k, row, col) = f;
  }
}

// ---------------------------------------------------------------------------
// Residual (riemann.rs:513-540) fused with the SSP-RK3 stage combination of
// Rie_prob_2d_rs.py:183-202 in numpy's evaluation order:
//   STAGE 0: out[i,j,k] dense = L                       (l_local_py)
//   STAGE 1: q1 = q + dt*L
//   STAGE 2: q2 = (0.75*q + 0.25*q1) + (0.25*dt)*L
//   STAGE 3: qn = ((1/3)*q + (2/3)*q2) + ((2/3)*dt)*L
// Fx planes are (m-5) x (n-6) faces, Fy planes (m-6) x (n-5).
// ---------------------------------------------------------------------------

// What a stage does with the residual L of cell (row, col).
template <class T, int STAGE>
__device__ __forceinline__ void residual_store(const T L[4], int64_t row, int64_t col, int64_t cols, T* out,
                                               const Planes<T>& Qn, const Planes<T>& Qs, const Planes<T>& Qo,
                                               const StepCtl* ctl) {
  if constexpr (STAGE == 0) {
#pragma unroll
    for (int k = 0; k < 4; ++k) out[(row * cols + col) * 4 + k] = L[k];
  } else {
    const double dt = ctl->dt;
    const int64_t r = row + 3, c = col + 3;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const T qn = Qn.at(k, r, c);
      T v;
      if constexpr (STAGE == 1) {
        v = qn + T(dt) * L[k];
      } else if constexpr (STAGE == 2) {
        v = T(0.75) * qn + T(0.25) * Qs.at(k, r, c) + T(0.25 * dt) * L[k];
      } else {
        v = T(1.0 / 3.0) * qn + T(2.0 / 3.0) * Qs.at(k, r, c) + T((2.0 / 3.0) * dt) * L[k];
      }
      Qo.at(k, r, c) = v;
    }
  }
}

template <class T, bool FAST, int STAGE>
__global__ void __launch_bounds__(128) k_residual(Planes<T> Fx, Planes<T> Fy, int64_t rows, int64_t cols, T dx,
                                                   T* out, Planes<T> Qn, Planes<T> Qs, Planes<T> Qo,
                                                   const StepCtl* ctl) {
  int64_t row, col;
  if (!locate(rows, cols, row, col)) return;
  if constexpr (STAGE > 0) {
    if (!ctl->active) return;
  }
  T L[4];
  if constexpr (FAST) {
    // one reciprocal instead of eight divides (riemann.rs:527 divides both
    // differences by the same dx)
    const T idx = qrcp<T, FAST>(dx);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      L[k] = -((Fx.at(k, row + 1, col) - Fx.at(k, row, col)) + (Fy.at(k, row, col + 1) - Fy.at(k, row, col))) * idx;
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const T dfdx = (Fx.at(k, row + 1, col) - Fx.at(k, row, col)) / dx;
      const T dgdy = (Fy.at(k, row, col + 1) - Fy.at(k, row, col)) / dx;
      L[k] = -(dfdx + dgdy);
    }
  }
  residual_store<T, STAGE>(L, row, col, cols, out, Qn, Qs, Qo, ctl);
}

// The same with the sensor blend of the four faces of the cell in place of k_blend
// (planes 0..3 HLLC, 4..7 HLLE, 8 the mean pressure).  FP32 only: each weight is
// formed on two cells, which costs less than the 13 planes that k_blend reads and
// writes per direction (17 us per launch at 2049 x 512, a quarter of the stage);
// in FP64 the second weight would cost more than the planes.
template <int STAGE>
__global__ void __launch_bounds__(128) k_residual_blend(Planes<float> Fx, Planes<float> Fy, int64_t rows, int64_t cols,
                                                         float dx, float jp_lo, float jp_hi, Planes<float> Qn,
                                                         Planes<float> Qs, Planes<float> Qo, const StepCtl* ctl) {
  int64_t row, col;
  if (!locate(rows, cols, row, col)) return;
  if (!ctl->active) return;
  const Planes<float> Px{Fx.p + 8 * Fx.ps, Fx.ps, Fx.ld}, Py{Fy.p + 8 * Fy.ps, Fy.ps, Fy.ld};
  const float xa = blend_weight<float, true>(Px, rows + 1, cols, row, col, jp_lo, jp_hi);
  const float xb = blend_weight<float, true>(Px, rows + 1, cols, row + 1, col, jp_lo, jp_hi);
  const float ya = blend_weight<float, true>(Py, rows, cols + 1, row, col, jp_lo, jp_hi);
  const float yb = blend_weight<float, true>(Py, rows, cols + 1, row, col + 1, jp_lo, jp_hi);
  const float idx = qrcp<float, true>(dx);
  float L[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float fa = xa * Fx.at(k, row, col) + (1.0f - xa) * Fx.at(4 + k, row, col);
    const float fb = xb * Fx.at(k, row + 1, col) + (1.0f - xb) * Fx.at(4 + k, row + 1, col);
    const float ga = ya * Fy.at(k, row, col) + (1.0f - ya) * Fy.at(4 + k, row, col);
    const float gb = yb * Fy.at(k, row, col + 1) + (1.0f - yb) * Fy.at(4 + k, row, col + 1);
    L[k] = -((fb - fa) + (gb - ga)) * idx;
  }
  residual_store<float, STAGE>(L, row, col, cols, nullptr, Qn, Qs, Qo, ctl);
}

// ---------------------------------------------------------------------------
// Boundary fills, in place, on NC channels of a strided array (the solver's
// 4 conserved planes, or the driver's 8-channel array).  Each ghost value
// depends only on interior values, so the fill is one pointwise pass.
// Requires nx, ny >= 3.
// ---------------------------------------------------------------------------
template <class T>
struct S3 {
  T* p;
  int64_t s0, s1, s2;
  __device__ __forceinline__ T& at(int64_t i, int64_t j, int k) const { return p[i * s0 + j * s1 + k * s2]; }
};

// Rie_prob_2d_rs.py:123-152 apply_bc_zero_gradient: ghost g <- 5-g on the low
// side and the mirror about the last interior cell on the high side; the
// corners end up mirrored in both directions.
__device__ __forceinline__ int64_t mirror_idx(int64_t i, int64_t M) {
  if (i < 3) return 5 - i;
  if (i >= M - 3) return 2 * M - 7 - i;
  return i;
}

// Ghost cell number e of an M x N array (M, N >= 6): three rows at each end, then
// three columns at each end of the rows between.  The fills launch one thread per
// ghost cell (over all cells they took 22 us at 2048 x 2048, 12 times as long).
__host__ __device__ __forceinline__ int64_t ghost_count(int64_t M, int64_t N) { return 6 * N + 6 * (M - 6); }
__device__ __forceinline__ bool ghost_cell(int64_t M, int64_t N, int64_t& i, int64_t& j) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ghost_count(M, N)) return false;
  if (e < 6 * N) {
    const int64_t r = e / N;
    j = e - r * N;
    i = r < 3 ? r : M - 6 + r;
  } else {
    const int64_t f = e - 6 * N, r = f / 6, c = f - 6 * r;
    i = 3 + r;
    j = c < 3 ? c : N - 6 + c;
  }
  return true;
}

template <class T, int NC>
__global__ void __launch_bounds__(128) k_bc_transmissive(S3<T> Q, int64_t M, int64_t N, const StepCtl* ctl) {
  int64_t i, j;
  if (!ghost_cell(M, N, i, j)) return;
  if (ctl && !ctl->active) return;
  const int64_t si = mirror_idx(i, M), sj = mirror_idx(j, N);
#pragma unroll
  for (int k = 0; k < NC; ++k) Q.at(i, j, k) = Q.at(si, sj, k);
}

// The inflow state of the oblique-shock boundary, all eight driver channels.
template <class T>
struct Post8 {
  T v[8];
};

// unitest.py:207-227 apply_bc_refac, the oblique-shock / double-Mach boundary:
// rows 0..2 take the inflow state; top ghost columns copy column ny+2; right
// ghost rows copy row nx+2; bottom ghost columns take the inflow state for rows
// <= bound, a copy of column 3 for rows bound+1..bound+9 and a mirror with the
// normal momentum (and v) negated beyond.  The reference fills these with
// sequential numpy slices; right ghost row nx+3+k takes its first k
// bottom-ghost values from row nx+2's band and the rest from its own band,
// which the pointwise form below reproduces.
template <class T, int NC>
__global__ void __launch_bounds__(128) k_bc_dmr(S3<T> Q, int64_t nx, int64_t ny, int64_t bound, Post8<T> post,
                                                 const StepCtl* ctl) {
  int64_t i, j;
  if (!ghost_cell(nx + 6, ny + 6, i, j)) return;
  if (ctl && !ctl->active) return;
  T v[NC];
  if (i < 3) {
#pragma unroll
    for (int k = 0; k < NC; ++k) v[k] = post.v[k];
  } else if (j >= ny + 3) {
    const int64_t s = i < nx + 3 ? i : nx + 2;
#pragma unroll
    for (int k = 0; k < NC; ++k) v[k] = Q.at(s, ny + 2, k);
  } else if (j < 3) {
    const int64_t s = i < nx + 3 ? i : nx + 2;
    const int64_t band_row = (i >= nx + 3 && j < i - nx - 3) ? nx + 2 : i;
    if (band_row <= bound) {
#pragma unroll
      for (int k = 0; k < NC; ++k) v[k] = post.v[k];
    } else if (band_row <= bound + 9) {
#pragma unroll
      for (int k = 0; k < NC; ++k) v[k] = Q.at(s, 3, k);
    } else {
#pragma unroll
      for (int k = 0; k < NC; ++k) v[k] = Q.at(s, 5 - j, k);
      v[2] = -v[2];
      if constexpr (NC == 8) v[6] = -v[6];
    }
  } else {  // i >= nx + 3
#pragma unroll
    for (int k = 0; k < NC; ++k) v[k] = Q.at(nx + 2, j, k);
  }
#pragma unroll
  for (int k = 0; k < NC; ++k) Q.at(i, j, k) = v[k];
}

// ---------------------------------------------------------------------------
// CFL wave-speed maximum (Rie_prob_2d_rs.py:311-319): max over interior cells
// of sqrt(u^2+v^2) + sqrt(gamma*p/max(rho, 1e-14)), with u, v, p the primitive
// channels as con2primi writes them (utils.rs:22-29) and rho the raw density.
// AOS = true reads the primitives from channels 5, 6, 7 of a (M, N, C>=8)
// array instead (the first step of a run starting from the driver's array).
// ---------------------------------------------------------------------------
// np.maximum(rho, 1e-14) of the driver's CFL (Rie_prob_2d_rs.py:314): NaN in,
// NaN out (fmax would return the bound).
template <class T>
__device__ __forceinline__ T np_maximum(T x, T c) { return x != x ? x : fmax(x, c); }

// np.max propagates NaN (and inf dominates), so a non-finite wave speed makes
// the maximum non-finite and dt follows, as in the driver.  The speeds are
// non-negative or NaN (of either sign), so the maximum is one of unsigned
// integers: NaN's bits order above +inf's.
__device__ __forceinline__ unsigned long long max_bits(unsigned long long a, unsigned long long b) { return a > b ? a : b; }
__device__ __forceinline__ unsigned long long speed_bits(double x) { return (unsigned long long)__double_as_longlong(x); }

template <class T, bool AOS>
__global__ void __launch_bounds__(256) k_cfl_max(CView<T> q, int64_t nx, int64_t ny, T gamma, StepCtl* ctl) {
  if (!ctl->active || ctl->cmax_preset) return;
  unsigned long long best = 0;
  bool nonpos = false;  // FP64 positivity check of the recovered density and pressure
  const int64_t total = nx * ny;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e / ny + 3, j = e % ny + 3;
    if constexpr (!AOS && std::is_same<T, float>::value) {
      // FP32 state: the wave speed in FP32 (the state's own precision; the
      // maximum and dt stay FP64), the positivity of the recovered density and
      // pressure in FP64 without a divide: rho > 0 and E rho - |m|^2/2 > 0, for the
      // cells that an FP32 test does not clear by 2^-20 of E rho, four times its
      // own rounding (the FP64 pipe took 84 % of this kernel's time).
      const float r0 = q.at(i, j, 0), m1 = q.at(i, j, 1), m2 = q.at(i, j, 2), E = q.at(i, j, 3);
      const float Er = E * r0;
      if (!(r0 > 0.0f && Er < 1e37f && Er - 0.5f * (m1 * m1 + m2 * m2) > 0x1p-20f * Er && Er > 1e-30f)) {
        const double rd = r0, m1d = m1, m2d = m2;
        if (!(rd > 0.0) || !((double)E * rd - 0.5 * (m1d * m1d + m2d * m2d) > 0.0)) nonpos = true;
      }
      const float rho = fmaxf(r0, float(kEps));
      const float ir = __fdividef(1.0f, rho);
      const float uu = m1 * ir, vv = m2 * ir;
      const float pp = fmaxf(((float)gamma - 1.0f) * (E - 0.5f * rho * (uu * uu + vv * vv)), float(kEps));
      const float w = sqrtf(uu * uu + vv * vv) + sqrtf((float)gamma * pp * __fdividef(1.0f, np_maximum(r0, 1e-14f)));
      best = max_bits(best, speed_bits((double)w));
    } else {
      const f64 g((double)gamma), r0((double)q.at(i, j, 0));
      f64 uu, vv, pp;
      if constexpr (AOS) {
        uu = f64((double)q.at(i, j, 5));
        vv = f64((double)q.at(i, j, 6));
        pp = f64((double)q.at(i, j, 7));
      } else {
        const f64 rho = fmax(r0, f64(kEps));
        uu = f64((double)q.at(i, j, 1)) / rho;
        vv = f64((double)q.at(i, j, 2)) / rho;
        const f64 praw = (g - f64(1.0)) * (f64((double)q.at(i, j, 3)) - f64(0.5) * rho * (uu * uu + vv * vv));
        pp = fmax(praw, f64(kEps));
        if (!(r0 > f64(0.0)) || !(praw > f64(0.0))) nonpos = true;
      }
      const f64 speed = sqrt(uu * uu + vv * vv);
      const f64 c = sqrt(g * pp / np_maximum(r0, f64(1e-14)));
      best = max_bits(best, speed_bits((c + speed).v));
    }
  }
  nonpos = __any_sync(0xffffffffu, nonpos);
  if (nonpos && (threadIdx.x & 31) == 0) atomicOr(&ctl->status, 2);
  for (int off = 16; off > 0; off >>= 1) best = max_bits(best, __shfl_xor_sync(0xffffffffu, best, off));
  __shared__ unsigned long long sm[8];
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long b = sm[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) b = max_bits(b, sm[w]);
    atomicMax(&ctl->cmax_bits, b);
    if (b >= 0x7ff0000000000000ull) atomicOr(&ctl->status, 1);
  }
}

// FP64 sums of the four conserved planes over the interior (conservation
// diagnostics); one block-partial per block, added with atomicAdd.
template <class T>
__global__ void __launch_bounds__(256) k_totals(CView<T> q, int64_t nx, int64_t ny, double* out4) {
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  const int64_t total = nx * ny;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e / ny + 3, j = e % ny + 3;
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[k] += (double)q.at(i, j, k);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    for (int off = 16; off > 0; off >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], off);
    if ((threadIdx.x & 31) == 0) atomicAdd(out4 + k, acc[k]);
  }
}

// dt = CFL*dx / (cmax + 1e-16), clipped to the time left (Rie_prob_2d_rs.py:315-318).
__global__ void k_dt(StepCtl* ctl) {
  if (!ctl->active) return;
  ctl->cmax_preset = 0;
  const double cmax = __longlong_as_double((long long)ctl->cmax_bits) + 1e-16;
  double dt = ctl->cfl_dx / cmax;
  if (ctl->t_final >= 0.0) {
    const double remaining = ctl->t_final - ctl->t;
    if (remaining < dt) dt = remaining;
  }
  ctl->dt = dt;
}

// Start of a run of `add` steps: the loop condition of Rie_prob_2d_rs.py:335.
__global__ void k_run_begin(StepCtl* ctl, double t_final, long long add) {
  ctl->t_final = t_final;
  ctl->max_steps = ctl->steps + add;
  bool go = ctl->steps < ctl->max_steps;
  if (t_final >= 0.0) go = go && (ctl->t < t_final - 1e-12);
  ctl->active = go ? 1 : 0;
}

// End of a step: advance the clock, reset the reduction, decide whether the
// next step runs (Rie_prob_2d_rs.py:335, loop condition T < t_final - 1e-12).
__global__ void k_step_end(StepCtl* ctl) {
  if (!ctl->active) return;
  ctl->t += ctl->dt;
  ctl->steps += 1;
  ctl->cmax_bits = 0ull;
  bool more = ctl->steps < ctl->max_steps;
  if (ctl->t_final >= 0.0) more = more && (ctl->t < ctl->t_final - 1e-12);
  ctl->active = more ? 1 : 0;
}

// ---------------------------------------------------------------------------
// Small element-wise kernels of the drop-in API
// ---------------------------------------------------------------------------
template <class T, bool FAST, bool Y>
__global__ void k_flux(CView<T> q, int64_t rows, int64_t cols, T gamma, T* out) {
  int64_t row, col;
  if (!locate(rows, cols, row, col)) return;
  T s[4], f[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) s[k] = q.at(row, col, k);
  euler_flux<T, FAST, Y>(s, gamma, f);
#pragma unroll
  for (int k = 0; k < 4; ++k) out[(row * cols + col) * 4 + k] = f[k];
}

template <class T, bool FAST>
__global__ void k_con2primi(CView<T> q, int64_t rows, int64_t cols, T gamma, T* p, T* a, T* rho, T* u, T* v, T* h) {
  int64_t row, col;
  if (!locate(rows, cols, row, col)) return;
  const int64_t e = row * cols + col;
  con2prim<T, FAST>(q.at(row, col, 0), q.at(row, col, 1), q.at(row, col, 2), q.at(row, col, 3), gamma, p[e], a[e],
                    rho[e], u[e], v[e], h[e]);
}

// Solver planes -> the driver's (M, N, 8) array: conserved channels 0..3 and
// the primitive sync of Rie_prob_2d_rs.py:157-163 (rho_safe, u, v, p).
template <class T, bool FAST>
__global__ void k_export_aos8(Planes<T> Q, int64_t M, int64_t N, T gamma, double* out) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t i = (int64_t)blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= M || j >= N) return;
  const T q0 = Q.at(0, i, j), q1 = Q.at(1, i, j), q2 = Q.at(2, i, j), q3 = Q.at(3, i, j);
  T p, a, rho, u, v, h;
  con2prim<T, FAST>(q0, q1, q2, q3, gamma, p, a, rho, u, v, h);
  double* o = out + (i * N + j) * 8;
  o[0] = (double)q0; o[1] = (double)q1; o[2] = (double)q2; o[3] = (double)q3;
  o[4] = (double)rho; o[5] = (double)u; o[6] = (double)v; o[7] = (double)p;
}

// Caller's strided array (channels 0..3) -> solver planes.
template <class T>
__global__ void k_import_planes(CView<double> q, int64_t M, int64_t N, Planes<T> Q) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t i = (int64_t)blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= M || j >= N) return;
#pragma unroll
  for (int k = 0; k < 4; ++k) Q.at(k, i, j) = (T)q.at(i, j, k);
}

}  // inline namespace WENO_TU_NS
}  // namespace weno

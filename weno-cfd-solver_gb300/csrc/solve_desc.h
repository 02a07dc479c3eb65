// One solve of the batch: where its cells lie in the pools and (staged
// configuration) its faces in the workspace, and the arithmetic of both, which the
// kernels and the host share.  Element offsets and plane strides are 64-bit
// throughout: a solve of 15,500 x 15,500 cells with the sensor blend already has its
// ninth plane beyond 2^31 elements (100 GB in FP64, which the device holds).
#pragma once

#ifdef __CUDACC__
#define WENO_DESC_HD __host__ __device__ __forceinline__
#else
#define WENO_DESC_HD inline
#endif

namespace weno {

struct SolveDesc {
  long long off;  // element offset of plane 0 in each pool
  long long ps;   // plane stride (elements)
  int nx, ny;
  int ld;         // row pitch (elements): ny rounded up to a multiple of 16 bytes
  int bc;         // 0 transmissive (mirror), 1 oblique-shock / DMR segments
  int bound;      // DMR: last row of the inflow segment on the lower boundary
  double dx;      // cell size (dx = dy)
  double post[8]; // DMR inflow state: conserved channels 0..3, primitive channels 4..7
  // Staged tile configuration only: this solve's face workspace, element offsets
  // in the workspace pool (see k_staged_pass1).
  long long w_p1x, w_p1y, w_fx, w_fy;  // plane 0 of each array
  long long s_p1x, s_p1y, s_fx, s_fy;  // plane strides
  int l_p1x, l_p1y;                    // row pitches of P1x and of P1y / Fy (Fx uses ld)
};

// Element (row, col) of a plane with row pitch ld.
WENO_DESC_HD long long plane_elem(long long row, int ld, int col) { return row * ld + col; }
// Plane 0 of the solve's face arrays: P1x at face row fi and column c = J + 2, P1y at
// row r = I + 2 and face column fj, Fx at (fi, j), Fy at (i, fj).
WENO_DESC_HD long long p1x_elem(const SolveDesc& d, int fi, int c) { return d.w_p1x + plane_elem(fi, d.l_p1x, c); }
WENO_DESC_HD long long p1y_elem(const SolveDesc& d, int r, int fj) { return d.w_p1y + plane_elem(r, d.l_p1y, fj); }
WENO_DESC_HD long long fx_elem(const SolveDesc& d, int fi, int j) { return d.w_fx + plane_elem(fi, d.ld, j); }
WENO_DESC_HD long long fy_elem(const SolveDesc& d, int i, int fj) { return d.w_fy + plane_elem(i, d.l_p1y, fj); }

// Value k of the face at p[e]: its planes are `stride` elements apart.  The index
// type is the stride's: int for a tile in shared memory, long long for the workspace.
template <class T, class I>
WENO_DESC_HD T& plane_value(T* p, int k, I stride, I e) {
  return p[k * stride + e];
}

// Face workspace of one solve in the staged configuration (element counts; see
// k_staged_pass1), for rows padded to lq elements and nf flux planes: fills the
// layout fields of `d` (nx, ny, ld set) with offsets relative to the solve's block and
// returns the block's length.
inline long long staged_layout(SolveDesc& d, int lq, int nf) {
  auto up = [](long long x, long long q) { return (x + q - 1) / q * q; };
  const long long nx = d.nx, ny = d.ny;
  d.l_p1x = (int)up(ny + 4, lq);
  d.l_p1y = (int)up(ny + 1, lq);
  d.s_p1x = up((nx + 1) * d.l_p1x, 64);
  d.s_p1y = up((nx + 4) * d.l_p1y, 64);
  d.s_fx = up((nx + 1) * d.ld, 64);
  d.s_fy = up(nx * d.l_p1y, 64);
  d.w_p1x = 0;
  d.w_p1y = 8 * d.s_p1x;
  d.w_fx = d.w_p1y + 8 * d.s_p1y;
  d.w_fy = d.w_fx + nf * d.s_fx;
  return d.w_fy + nf * d.s_fy;
}

}  // namespace weno

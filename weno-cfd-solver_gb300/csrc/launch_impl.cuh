// Launcher definitions (see launch_api.h).  Included only by tu_exact.cu, tu_fast.cu
// and tu_df64.cu.
#pragma once

#include "kernels.cuh"
#include "launch_api.h"

namespace weno {

inline namespace WENO_TU_NS {
namespace detail {

inline dim3 grid2d(int64_t rows, int64_t cols, dim3 blk) {
  return dim3((unsigned)((cols + blk.x - 1) / blk.x), (unsigned)((rows + blk.y - 1) / blk.y), 1);
}

template <class T>
inline CView<T> cview(HostView v) {
  return CView<T>{static_cast<const T*>(v.p), v.s0, v.s1, v.s2};
}
template <class T>
inline Planes<T> planes(HostPlanes v) {
  return Planes<T>{static_cast<T*>(v.p), v.ps, v.ld};
}
template <class T>
inline S3<T> s3(HostView v) {
  return S3<T>{static_cast<T*>(const_cast<void*>(v.p)), v.s0, v.s1, v.s2};
}

const dim3 kBlk(32, 4, 1);

// Launch shape of a face or cell kernel over rows x cols threads.  FP64 and df64
// kernels are bound by a pipe that serves one warp at a time, so what counts is
// that no lane is idle and every SM has the same number of warps: the flattened
// index space, in blocks of one warp while there are fewer than 32 warps per SM
// (blocks of four would fill a part of the SMs, or leave a last wave).  FP32
// kernels are issue bound and keep the 2-D blocks (no division for the index)
// unless the grid fills the SMs and rounding its columns up to warps would idle
// more than 1 lane in 16 (100 x 100: flattened 4 % slower; 2000 x 70: 7 % faster).
struct Shape {
  dim3 grid, block;
};
template <class T>
inline Shape shape(int64_t rows, int64_t cols) {
  const int64_t padded = (cols + 31) / 32 * 32;
  const int64_t warps = (rows * cols + 31) / 32;
  if (is_f32<T> && (warps < 152 * 16 || (padded - cols) * 16 <= padded)) return Shape{grid2d(rows, cols, kBlk), kBlk};
  const unsigned block = !is_f32<T> && warps < 152 * 32 ? 32 : 128;
  return Shape{dim3((unsigned)((rows * cols + block - 1) / block), 1, 1), dim3(block, 1, 1)};
}

inline unsigned quad_blocks(int64_t rows, int64_t cols) {
  return rows > 0 && cols > 0 ? (unsigned)((rows * cols * 4 + 31) / 32) : 0u;
}

}  // namespace detail
}  // inline namespace WENO_TU_NS

template <class H, bool FAST>
cudaError_t Launch<H, FAST>::pass1(HostView u, int64_t rows, int64_t cols, double gamma, bool ydir, bool chr,
                                   HostPlanes PL, HostPlanes PR, double weps, cudaStream_t st) {
  using T = dev_t<H>;
  using namespace detail;
  if (rows <= 0 || cols <= 0) return cudaSuccess;
  const Shape g = shape<T>(rows, cols);
  auto U = cview<T>(u);
  auto L = planes<T>(PL), R = planes<T>(PR);
  if constexpr (!std::is_same<T, df64>::value) {
    if (!chr) {  // component-wise: one cell per thread, both of its face states
      const Shape gc = ydir ? shape<T>(rows, cols + 1) : shape<T>(rows + 1, cols);
      if (!ydir) k_pass1_cells<T, FAST, false><<<gc.grid, gc.block, 0, st>>>(U, rows, cols, L, R, (T)weps);
      else k_pass1_cells<T, FAST, true><<<gc.grid, gc.block, 0, st>>>(U, rows, cols, L, R, (T)weps);
    } else if (!ydir) {
      k_pass1<T, FAST, false, true><<<g.grid, g.block, 0, st>>>(U, rows, cols, (T)gamma, L, R, (T)weps);
    } else {
      k_pass1<T, FAST, true, true><<<g.grid, g.block, 0, st>>>(U, rows, cols, (T)gamma, L, R, (T)weps);
    }
  } else {
    if (!ydir && chr) k_pass1<T, FAST, false, true><<<g.grid, g.block, 0, st>>>(U, rows, cols, (T)gamma, L, R, (T)weps);
    else if (!ydir) k_pass1<T, FAST, false, false><<<g.grid, g.block, 0, st>>>(U, rows, cols, (T)gamma, L, R, (T)weps);
    else if (chr) k_pass1<T, FAST, true, true><<<g.grid, g.block, 0, st>>>(U, rows, cols, (T)gamma, L, R, (T)weps);
    else k_pass1<T, FAST, true, false><<<g.grid, g.block, 0, st>>>(U, rows, cols, (T)gamma, L, R, (T)weps);
    // the marked faces (reads one plane: 1 % of the pass)
    const T gm = (T)gamma, we = (T)weps;
    if (!ydir && chr) k_pass1_marked<false, true><<<g.grid, g.block, 0, st>>>(U, rows, cols, gm, L, R, we);
    else if (!ydir) k_pass1_marked<false, false><<<g.grid, g.block, 0, st>>>(U, rows, cols, gm, L, R, we);
    else if (chr) k_pass1_marked<true, true><<<g.grid, g.block, 0, st>>>(U, rows, cols, gm, L, R, we);
    else k_pass1_marked<true, false><<<g.grid, g.block, 0, st>>>(U, rows, cols, gm, L, R, we);
  }
  return cudaGetLastError();
}

template <class H, bool FAST>
cudaError_t Launch<H, FAST>::pass2(HostPlanes PL, HostPlanes PR, int64_t rows, int64_t cols, double gamma, bool ydir,
                                   int kind, void* a, void* b, void* c, void* d, int64_t ps, int64_t ld, double weps,
                                   cudaStream_t st) {
  using T = dev_t<H>;
  using namespace detail;
  if (rows <= 0 || cols <= 0) return cudaSuccess;
  const Shape g = shape<T>(rows, cols);
  auto L = planes<T>(PL), R = planes<T>(PR);
  Pass2Dst dst{a, b, c, d, ps, ld};
  const T gm = (T)gamma;
  if constexpr (FAST && !std::is_same<T, df64>::value) {
    // two faces per thread along the transverse direction (df64 keeps one:
    // its larger per-face register footprint outweighs the shared differences)
    const Shape g2 = ydir ? shape<T>((rows + 1) / 2, cols) : shape<T>(rows, (cols + 1) / 2);
#define WENO_P2T(Y, K) k_pass2_two<T, Y, K><<<g2.grid, g2.block, 0, st>>>(L, R, rows, cols, gm, dst, (T)weps)
    if (!ydir) {
      if (kind == 0) WENO_P2T(false, P2_STATES);
      else if (kind == 1) WENO_P2T(false, P2_HLLE);
      else WENO_P2T(false, P2_BLEND);
    } else {
      if (kind == 0) WENO_P2T(true, P2_STATES);
      else if (kind == 1) WENO_P2T(true, P2_HLLE);
      else WENO_P2T(true, P2_BLEND);
    }
#undef WENO_P2T
  } else {
#define WENO_P2(Y, K) k_pass2<T, FAST, Y, K><<<g.grid, g.block, 0, st>>>(L, R, rows, cols, gm, dst, (T)weps)
    if (!ydir) {
      if (kind == 0) WENO_P2(false, P2_STATES);
      else if (kind == 1) WENO_P2(false, P2_HLLE);
      else WENO_P2(false, P2_BLEND);
    } else {
      if (kind == 0) WENO_P2(true, P2_STATES);
      else if (kind == 1) WENO_P2(true, P2_HLLE);
      else WENO_P2(true, P2_BLEND);
    }
#undef WENO_P2
  }
  return cudaGetLastError();
}

template <class H, bool FAST>
cudaError_t Launch<H, FAST>::pass1_quads(HostView u, int64_t m, int64_t n, int dirs, double gamma, bool chr,
                                         const HostPlanes P[4], double weps, cudaStream_t st) {
  using T = dev_t<H>;
  using namespace detail;
  if constexpr (is_native_f64<T>) {
    const unsigned bx = (dirs & 1) ? quad_blocks(m - 5, n) : 0, by = (dirs & 2) ? quad_blocks(m, n - 5) : 0;
    if (bx + by == 0) return cudaSuccess;
    const auto U = cview<T>(u);
    const T gm = (T)gamma, we = (T)weps;
    const auto A = planes<T>(P[0]), B = planes<T>(P[1]), C = planes<T>(P[2]), D = planes<T>(P[3]);
    if (chr) k_pass1_quad<FAST, true><<<bx + by, 32, 0, st>>>(U, m, n, bx, gm, A, B, C, D, we);
    else k_pass1_quad<FAST, false><<<bx + by, 32, 0, st>>>(U, m, n, bx, gm, A, B, C, D, we);
    return cudaGetLastError();
  } else {
    return cudaErrorNotSupported;
  }
}

template <class H, bool FAST>
cudaError_t Launch<H, FAST>::pass2_quads(const HostPlanes P[4], int64_t m, int64_t n, int dirs, double gamma, int kind,
                                         const FaceDst& x, const FaceDst& y, double weps, cudaStream_t st) {
  using T = dev_t<H>;
  using namespace detail;
  if constexpr (is_native_f64<T>) {
    const unsigned bx = (dirs & 1) ? quad_blocks(m - 5, n - 6) : 0, by = (dirs & 2) ? quad_blocks(m - 6, n - 5) : 0;
    if (bx + by == 0) return cudaSuccess;
    const T gm = (T)gamma, we = (T)weps;
    const auto A = planes<T>(P[0]), B = planes<T>(P[1]), C = planes<T>(P[2]), D = planes<T>(P[3]);
    const Pass2Dst dx{x.a, x.b, x.c, x.d, x.ps, x.ld}, dy{y.a, y.b, y.c, y.d, y.ps, y.ld};
    if (kind == 0) k_pass2_quad<FAST, P2_STATES><<<bx + by, 32, 0, st>>>(A, B, C, D, m, n, bx, gm, dx, dy, we);
    else if (kind == 1) k_pass2_quad<FAST, P2_HLLE><<<bx + by, 32, 0, st>>>(A, B, C, D, m, n, bx, gm, dx, dy, we);
    else k_pass2_quad<FAST, P2_BLEND><<<bx + by, 32, 0, st>>>(A, B, C, D, m, n, bx, gm, dx, dy, we);
    return cudaGetLastError();
  } else {
    return cudaErrorNotSupported;
  }
}

template <class H, bool FAST>
cudaError_t Launch<H, FAST>::riemann(const void* ql, const void* fl, const void* qr, const void* fr, int64_t rows,
                                     int64_t cols, double gamma, bool ydir, int kind, void* out, void* a, void* b,
                                     void* c, int64_t ps, int64_t ld, cudaStream_t st) {
  using T = dev_t<H>;
  using namespace detail;
  if (rows <= 0 || cols <= 0) return cudaSuccess;
  const Shape g = shape<T>(rows, cols);
  const T *QL = static_cast<const T*>(ql), *FL = static_cast<const T*>(fl);
  const T *QR = static_cast<const T*>(qr), *FR = static_cast<const T*>(fr);
  Planes<T> A{static_cast<T*>(a), ps, ld}, B{static_cast<T*>(b), ps, ld}, C{static_cast<T*>(c), ps, ld};
  T* o = static_cast<T*>(out);
  const T gm = (T)gamma;
#define WENO_RS(Y, K) k_riemann<T, FAST, Y, K><<<g.grid, g.block, 0, st>>>(QL, FL, QR, FR, rows, cols, gm, o, A, B, C)
  if (!ydir) {
    if (kind == 0) WENO_RS(false, 0);
    else if (kind == 1) WENO_RS(false, 1);
    else WENO_RS(false, 2);
  } else {
    if (kind == 0) WENO_RS(true, 0);
    else if (kind == 1) WENO_RS(true, 1);
    else WENO_RS(true, 2);
  }
#undef WENO_RS
  return cudaGetLastError();
}

template <class H, bool FAST>
cudaError_t Launch<H, FAST>::blend(HostPlanes Fc, HostPlanes Fe, HostPlanes Pbar, int64_t rows, int64_t cols,
                                   double jp_lo, double jp_hi, void* out, cudaStream_t st) {
  using T = dev_t<H>;
  using namespace detail;
  if (rows <= 0 || cols <= 0) return cudaSuccess;
  if constexpr (!is_f32<T>) {
    const Shape g = shape<T>(rows, cols);
    auto C = planes<T>(Fc), E = planes<T>(Fe), P = planes<T>(Pbar);
    if (out) k_blend<T, FAST, true><<<g.grid, g.block, 0, st>>>(C, E, P, rows, cols, (T)jp_lo, (T)jp_hi, static_cast<T*>(out), C);
    else k_blend<T, FAST, false><<<g.grid, g.block, 0, st>>>(C, E, P, rows, cols, (T)jp_lo, (T)jp_hi, nullptr, C);
    return cudaGetLastError();
  } else {
    return cudaErrorNotSupported;  // residual_blend
  }
}

template <class H, bool FAST>
cudaError_t Launch<H, FAST>::residual(HostPlanes Fx, HostPlanes Fy, int64_t rows, int64_t cols, double dx, int stage,
                                      void* out, HostPlanes Qn, HostPlanes Qs, HostPlanes Qo, const StepCtl* ctl,
                                      cudaStream_t st) {
  using T = dev_t<H>;
  using namespace detail;
  if (rows <= 0 || cols <= 0) return cudaSuccess;
  const Shape g = shape<T>(rows, cols);
  auto X = planes<T>(Fx), Yp = planes<T>(Fy), N = planes<T>(Qn), S = planes<T>(Qs), O = planes<T>(Qo);
  T* o = static_cast<T*>(out);
  switch (stage) {
    case 0: k_residual<T, FAST, 0><<<g.grid, g.block, 0, st>>>(X, Yp, rows, cols, (T)dx, o, N, S, O, ctl); break;
    case 1: k_residual<T, FAST, 1><<<g.grid, g.block, 0, st>>>(X, Yp, rows, cols, (T)dx, o, N, S, O, ctl); break;
    case 2: k_residual<T, FAST, 2><<<g.grid, g.block, 0, st>>>(X, Yp, rows, cols, (T)dx, o, N, S, O, ctl); break;
    default: k_residual<T, FAST, 3><<<g.grid, g.block, 0, st>>>(X, Yp, rows, cols, (T)dx, o, N, S, O, ctl); break;
  }
  return cudaGetLastError();
}

template <class H, bool FAST>
cudaError_t Launch<H, FAST>::residual_blend(HostPlanes Fx, HostPlanes Fy, int64_t rows, int64_t cols, double dx,
                                            double jp_lo, double jp_hi, int stage, HostPlanes Qn, HostPlanes Qs,
                                            HostPlanes Qo, const StepCtl* ctl, cudaStream_t st) {
  using namespace detail;
  if (rows <= 0 || cols <= 0) return cudaSuccess;
  if constexpr (is_f32<H>) {
    const Shape g = shape<float>(rows, cols);
    const auto X = planes<float>(Fx), Yp = planes<float>(Fy), N = planes<float>(Qn), S = planes<float>(Qs),
               O = planes<float>(Qo);
    const float d = (float)dx, lo = (float)jp_lo, hi = (float)jp_hi;
    if (stage == 1) k_residual_blend<1><<<g.grid, g.block, 0, st>>>(X, Yp, rows, cols, d, lo, hi, N, S, O, ctl);
    else if (stage == 2) k_residual_blend<2><<<g.grid, g.block, 0, st>>>(X, Yp, rows, cols, d, lo, hi, N, S, O, ctl);
    else k_residual_blend<3><<<g.grid, g.block, 0, st>>>(X, Yp, rows, cols, d, lo, hi, N, S, O, ctl);
    return cudaGetLastError();
  } else {
    return cudaErrorNotSupported;
  }
}

template <class H, bool FAST>
cudaError_t Launch<H, FAST>::flux(HostView q, int64_t rows, int64_t cols, double gamma, bool ydir, void* out,
                                  cudaStream_t st) {
  using T = dev_t<H>;
  using namespace detail;
  if (rows <= 0 || cols <= 0) return cudaSuccess;
  const Shape g = shape<T>(rows, cols);
  if (ydir) k_flux<T, FAST, true><<<g.grid, g.block, 0, st>>>(cview<T>(q), rows, cols, (T)gamma, static_cast<T*>(out));
  else k_flux<T, FAST, false><<<g.grid, g.block, 0, st>>>(cview<T>(q), rows, cols, (T)gamma, static_cast<T*>(out));
  return cudaGetLastError();
}

template <class H, bool FAST>
cudaError_t Launch<H, FAST>::con2primi(HostView q, int64_t rows, int64_t cols, double gamma, void* p, void* a,
                                       void* rho, void* u, void* v, void* h, cudaStream_t st) {
  using T = dev_t<H>;
  using namespace detail;
  if (rows <= 0 || cols <= 0) return cudaSuccess;
  const Shape g = shape<T>(rows, cols);
  k_con2primi<T, FAST><<<g.grid, g.block, 0, st>>>(cview<T>(q), rows, cols, (T)gamma, static_cast<T*>(p),
                                           static_cast<T*>(a), static_cast<T*>(rho), static_cast<T*>(u),
                                           static_cast<T*>(v), static_cast<T*>(h));
  return cudaGetLastError();
}

template <class H, bool FAST>
cudaError_t Launch<H, FAST>::bc_transmissive(HostView q, int nc, int64_t M, int64_t N, const StepCtl* ctl,
                                             cudaStream_t st) {
  using T = dev_t<H>;
  using namespace detail;
  const unsigned g = (unsigned)((ghost_count(M, N) + 127) / 128);
  if (nc == 8) k_bc_transmissive<T, 8><<<g, 128, 0, st>>>(s3<T>(q), M, N, ctl);
  else k_bc_transmissive<T, 4><<<g, 128, 0, st>>>(s3<T>(q), M, N, ctl);
  return cudaGetLastError();
}

template <class H, bool FAST>
cudaError_t Launch<H, FAST>::bc_dmr(HostView q, int nc, int64_t nx, int64_t ny, int64_t bound, const double* post8,
                                    const StepCtl* ctl, cudaStream_t st) {
  using T = dev_t<H>;
  using namespace detail;
  const unsigned g = (unsigned)((ghost_count(nx + 6, ny + 6) + 127) / 128);
  Post8<T> post;
  for (int k = 0; k < 8; ++k) post.v[k] = T(post8[k]);
  if (nc == 8) k_bc_dmr<T, 8><<<g, 128, 0, st>>>(s3<T>(q), nx, ny, bound, post, ctl);
  else k_bc_dmr<T, 4><<<g, 128, 0, st>>>(s3<T>(q), nx, ny, bound, post, ctl);
  return cudaGetLastError();
}

template <class H, bool FAST>
cudaError_t Launch<H, FAST>::cfl_max(HostView q, bool aos, int64_t nx, int64_t ny, double gamma, StepCtl* ctl,
                                     int sm_count, cudaStream_t st) {
  using T = dev_t<H>;
  const int64_t total = nx * ny;
  int64_t blocks = (total + 255) / 256;
  const int64_t cap = (int64_t)sm_count * 8;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  if (aos) k_cfl_max<T, true><<<(unsigned)blocks, 256, 0, st>>>(detail::cview<T>(q), nx, ny, (T)gamma, ctl);
  else k_cfl_max<T, false><<<(unsigned)blocks, 256, 0, st>>>(detail::cview<T>(q), nx, ny, (T)gamma, ctl);
  return cudaGetLastError();
}

template <class H, bool FAST>
cudaError_t Launch<H, FAST>::export_aos8(HostPlanes Q, int64_t M, int64_t N, double gamma, double* out,
                                         cudaStream_t st) {
  using T = dev_t<H>;
  using namespace detail;
  const dim3 g = grid2d(M, N, kBlk);
  k_export_aos8<T, FAST><<<g, kBlk, 0, st>>>(planes<T>(Q), M, N, (T)gamma, out);
  return cudaGetLastError();
}

template <class H, bool FAST>
cudaError_t Launch<H, FAST>::totals(HostView q, int64_t nx, int64_t ny, double* out4, int sm_count, cudaStream_t st) {
  using T = dev_t<H>;
  int64_t blocks = (nx * ny + 255) / 256;
  if (blocks > (int64_t)sm_count * 4) blocks = (int64_t)sm_count * 4;
  if (blocks < 1) blocks = 1;
  cudaError_t e = cudaMemsetAsync(out4, 0, 4 * sizeof(double), st);
  if (e) return e;
  k_totals<T><<<(unsigned)blocks, 256, 0, st>>>(detail::cview<T>(q), nx, ny, out4);
  return cudaGetLastError();
}

template <class H, bool FAST>
cudaError_t Launch<H, FAST>::import_planes(HostView q, int64_t M, int64_t N, HostPlanes Q, cudaStream_t st) {
  using T = dev_t<H>;
  using namespace detail;
  const dim3 g = grid2d(M, N, kBlk);
  k_import_planes<T><<<g, kBlk, 0, st>>>(cview<double>(q), M, N, planes<T>(Q));
  return cudaGetLastError();
}

}  // namespace weno

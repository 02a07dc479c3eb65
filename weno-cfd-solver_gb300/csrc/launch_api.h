// Host-side launchers of the residual kernels, one set per (arithmetic type,
// arithmetic policy).  The definitions live in launch_impl.cuh and are compiled
// only in tu_exact.cu (--fmad=false: reference-identical IEEE doubles) and
// tu_fast.cu (--fmad=true: the FAST forms), so the policy of a kernel is fixed
// by the translation unit it was built in.  This header only declares them.
#pragma once

#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>

namespace weno {

// Strided read-only view of a caller array (elements, not bytes).
struct HostView {
  const void* p;
  int64_t s0, s1, s2;
};

// Plane set: component k, element (r, c) at p[k*ps + r*ld + c].
struct HostPlanes {
  void* p;
  int64_t ps, ld;
};

// Where pass 2 puts its faces (see Launch::pass2).
struct FaceDst {
  void *a, *b, *c, *d;
  int64_t ps, ld;
};

// FP64 grids of few faces take four lanes per face and one launch for both sweeps
// (Launch::pass1_quads, pass2_quads): there the one-thread form is a chain of
// dependent operations (64 x 64 residual: 4 x 50 us in its passes), and the quads'
// repeated averages, a third more of the FP64 pipe, cost less.  The line lies where the
// quads' one-warp blocks of eight faces no longer fill whole waves: an SM holds 16 of
// them at the registers of the exact characteristic pass 1 (126), 14 at those of the
// exact blend's pass 2 (138), and a sweep is one such wave, both sweeps are two.  FAST
// component-wise kernels are ahead up to 24.  Residual in us, quads against one thread
// per face, below and above the line:
//   exact, HLLE     142^2 198 : 226 (char), 152 : 181 (cons)   145^2 263 : 233, 150^2 192 : 189
//   exact, blend    130^2 234 : 240 (char), 177 : 195 (cons)   138^2 256 : 242, 208 : 197
//   FAST, char      142^2  96 : 110 (HLLE), 124 : 139 (blend)  150^2 111 : 106, 147 : 135
//   FAST, cons      172^2  84 :  91 (HLLE), 118 : 122 (blend)
// and one sweep's reconstruction: exact char 140^2 78 : 103, 155^2 133 : 109; FAST char
// 140^2 41 : 43, 155^2 53 : 45; FAST cons 172^2 34 : 37.
constexpr int kQuadBlocksMost = 24;
constexpr int quad_blocks_per_sm(bool fast, bool cons, bool blend) {
  return fast ? (cons ? kQuadBlocksMost : 16) : (blend ? 14 : 16);
}
inline bool within_quads(int64_t m, int64_t n, int blocks_per_sm) {
  const int64_t most = (int64_t)152 * 8 * blocks_per_sm;  // faces of a sweep
  return m > 5 && n > 5 && (m - 5) * n <= most && m * (n - 5) <= most;
}
inline bool quad_faces(int64_t m, int64_t n, bool fast, bool cons, bool blend) {
  return within_quads(m, n, quad_blocks_per_sm(fast, cons, blend));
}
// Grids whose workspace has room for both sweeps at once (reported without the mode
// and the reconstruction, so for the largest of the above).
inline bool quad_room(int64_t m, int64_t n) { return within_quads(m, n, kQuadBlocksMost); }

struct StepCtl;
namespace dfm {
struct df64;
}

template <class T, bool FAST>
struct Launch {
  // Pass 1 over `rows x cols` faces (x: rows = m-5, cols = n; y: rows = m, cols = n-5).
  static cudaError_t pass1(HostView u, int64_t rows, int64_t cols, double gamma, bool ydir, bool chr,
                           HostPlanes PL, HostPlanes PR, double weps, cudaStream_t st);
  // Pass 2 over the final face array.  kind 0: dense q_l, f_l, q_r, f_r into
  // a..d; kind 1: HLLE flux planes into a; kind 2: HLLC planes into a, HLLE
  // planes into b, mean pressure plane into c.  ps/ld describe a, b, c.
  static cudaError_t pass2(HostPlanes PL, HostPlanes PR, int64_t rows, int64_t cols, double gamma, bool ydir,
                           int kind, void* a, void* b, void* c, void* d, int64_t ps, int64_t ld, double weps,
                           cudaStream_t st);
  // Both passes of an (m, n) array with four lanes per face (double only): dirs 1 the
  // x sweep, 2 the y sweep, 3 both in one launch; P holds q_l, q_r of x, then of y.
  static cudaError_t pass1_quads(HostView u, int64_t m, int64_t n, int dirs, double gamma, bool chr,
                                 const HostPlanes P[4], double weps, cudaStream_t st);
  static cudaError_t pass2_quads(const HostPlanes P[4], int64_t m, int64_t n, int dirs, double gamma, int kind,
                                 const FaceDst& x, const FaceDst& y, double weps, cudaStream_t st);
  // Riemann solver on dense (rows, cols, 4) face arrays.  kind 0 HLLC / 1 HLLE
  // -> dense out; kind 2 -> planes Fc (a), Fe (b), pbar (c).
  static cudaError_t riemann(const void* ql, const void* fl, const void* qr, const void* fr, int64_t rows,
                             int64_t cols, double gamma, bool ydir, int kind, void* out, void* a, void* b, void* c,
                             int64_t ps, int64_t ld, cudaStream_t st);
  // Sensor blend; writes dense `out` if non-null, else in place into Fc.
  static cudaError_t blend(HostPlanes Fc, HostPlanes Fe, HostPlanes Pbar, int64_t rows, int64_t cols, double jp_lo,
                           double jp_hi, void* out, cudaStream_t st);
  // Flux difference over (rows, cols) = (m-6, n-6) cells.  stage 0: dense out;
  // stages 1..3: SSP-RK3 combination into Qo planes (interior offset 3).
  static cudaError_t residual(HostPlanes Fx, HostPlanes Fy, int64_t rows, int64_t cols, double dx, int stage,
                              void* out, HostPlanes Qn, HostPlanes Qs, HostPlanes Qo, const StepCtl* ctl,
                              cudaStream_t st);
  // The same with the sensor blend of the faces (planes as pass 2 kind 2 leaves them)
  // inside, stages 1..3, float only.
  static cudaError_t residual_blend(HostPlanes Fx, HostPlanes Fy, int64_t rows, int64_t cols, double dx, double jp_lo,
                                    double jp_hi, int stage, HostPlanes Qn, HostPlanes Qs, HostPlanes Qo,
                                    const StepCtl* ctl, cudaStream_t st);
  static cudaError_t flux(HostView q, int64_t rows, int64_t cols, double gamma, bool ydir, void* out, cudaStream_t st);
  static cudaError_t con2primi(HostView q, int64_t rows, int64_t cols, double gamma, void* p, void* a, void* rho,
                               void* u, void* v, void* h, cudaStream_t st);
  // Boundary fills on nc (4 or 8) channels of a strided array, in place.
  static cudaError_t bc_transmissive(HostView q, int nc, int64_t M, int64_t N, const StepCtl* ctl, cudaStream_t st);
  static cudaError_t bc_dmr(HostView q, int nc, int64_t nx, int64_t ny, int64_t bound, const double* post8,
                            const StepCtl* ctl, cudaStream_t st);
  // CFL reduction into ctl->cmax_bits; aos = read primitives from channels 5..7.
  static cudaError_t cfl_max(HostView q, bool aos, int64_t nx, int64_t ny, double gamma, StepCtl* ctl,
                             int sm_count, cudaStream_t st);
  static cudaError_t export_aos8(HostPlanes Q, int64_t M, int64_t N, double gamma, double* out, cudaStream_t st);
  static cudaError_t totals(HostView q, int64_t nx, int64_t ny, double* out4, int sm_count, cudaStream_t st);
  static cudaError_t import_planes(HostView q, int64_t M, int64_t N, HostPlanes Q, cudaStream_t st);
};

// Control-block kernels (precision independent).
cudaError_t launch_dt(StepCtl* ctl, cudaStream_t st);
cudaError_t launch_step_end(StepCtl* ctl, cudaStream_t st);
cudaError_t launch_run_begin(StepCtl* ctl, double t_final, long long add, cudaStream_t st);

extern template struct Launch<double, false>;
extern template struct Launch<double, true>;
extern template struct Launch<float, true>;
extern template struct Launch<dfm::df64, true>;

}  // namespace weno

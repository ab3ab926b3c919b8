// Implicit time integration on the device: BDF1 or Crank-Nicolson steps
// solved by Newton-Raphson, each correction by BiCGSTAB with a Jacobi
// (diagonal) preconditioner on the device CSR Jacobian -- the consumer of
// the reference's Jacobian in its implicit tests
// (tests_cpp/eigen_2d_euler_riemann_implicit/main.cc:31-44: Pressio's
// implicit stepper, create_newton_solver, iterative::Bicgstab).
//
// Step n -> n+1 with f the velocity (ode_constants.hpp):
//   BDF1  R(y) = y - y_n - dt f(y)                    J_R = I - dt Jf(y)
//   CN    R(y) = y - y_n - dt/2 (f(y) + f(y_n))       J_R = I - dt/2 Jf(y)
// Newton (nonlinear_least_squares.hpp:50-112): per iteration R and J_R at y,
// solve J_R d = R, stop before updating when |d|_2 < tol (Pressio's default
// criterion, the absolute l2 norm of the correction), else y <- y - d.
// BiCGSTAB follows the standard preconditioned algorithm (van der Vorst)
// that Eigen's BiCGSTAB implements, with reductions in a fixed order.
//
// A linear solve is one cooperative launch (k_bicgstab): an iteration's two
// matrix-vector products, its vector updates and its dot products are a few
// microseconds of work each, so as separate launches (17 per iteration, with
// a read of the residual by the host) an iteration took 105 us whatever its
// size.  Inside one kernel the five points of an iteration where every block
// needs every other's result are barriers over the resident blocks.  64^2
// Euler WENO3 (16,384 rows of 36): 19 us per iteration, about half of it the
// barriers and sums; two Crank-Nicolson steps (20 Newton, 489 BiCGSTAB
// iterations) 66.7 -> 12.5 ms.  The FP64 units set the rest: with the
// iteration's scalars divided on the FP64 pipe by every warp it took 24 us,
// with every thread summing and one warp per scheduler 34 us.
#include <cmath>
#include <algorithm>
#include <cstdint>
#include <memory>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "csr_rows.hpp"
#include "numerics.cuh"
#include "problem_impl.hpp"

namespace pda {
namespace impl {

constexpr int RB = 512;       // threads per block of the solver
constexpr int LPR = 4;        // lanes per matrix row: 9 to 95 entries a row
constexpr int MAX_BLOCKS = 2048;

// System of one Newton iteration: R, J_R = I + c Jf in place of Jf's values,
// and the reciprocals of J_R's diagonal.  LPR lanes per row.
__global__ void __launch_bounds__(256)
k_system(int scheme, long n, const int *__restrict__ rowptr, const int *__restrict__ colidx,
         const double *__restrict__ y, const double *__restrict__ yn, const double *__restrict__ f,
         const double *__restrict__ fn, double dt, double c, double *__restrict__ J, double *__restrict__ dinv,
         double *__restrict__ R) {
  const long r = ((long)blockIdx.x * blockDim.x + threadIdx.x) / LPR;
  const int lane = threadIdx.x % LPR;
  if (r >= n) return;
  if (lane == 0) {
    if (scheme == 0) R[r] = y[r] - yn[r] - dt * f[r];
    else R[r] = y[r] - yn[r] - (dt / 2.) * (f[r] + fn[r]);
  }
  row_batches<1, LPR>(rowptr[r], rowptr[r + 1], lane, [&](unsigned q) {
    double v = c * J[q];
    if (colidx[q] == r) {
      v += 1.;
      dinv[r] = div_rn(1., v);
    }
    J[q] = v;
  });
}

__global__ void k_minus(long n, const double *__restrict__ x, double *__restrict__ y) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] -= x[i];
}

// What the host reads after a solve.
struct SolveInfo {
  double rr, bb, dd;  // |r|^2, |b|^2, |x|^2
  int iters;
  int error;  // a barrier's wait ran out
};

struct SolveArgs {
  long n;
  const int *rowptr, *colidx;
  const double *A, *dinv, *b;
  double *x, *r, *p, *v, *s, *t, *y, *z;  // vectors written here
  double *part;                           // [4][MAX_BLOCKS] block sums
  unsigned *arrived;                      // barrier arrivals, zero at launch
  SolveInfo *info;                        // zero at launch
  double tol2;
  int maxIt;
};

// Barrier over the resident blocks of a cooperative launch.  Arrivals count
// up; each wait is bounded and a wait that runs out sets the error flag, on
// which every block leaves.
constexpr unsigned POLLS = 1u << 24;
struct GridBarrier {
  unsigned *arrived;
  int *error;
  unsigned target = 0;
  __device__ bool sync() {
    __shared__ int failed;
    __syncthreads();
    target += gridDim.x;
    if (threadIdx.x == 0) {
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrived) : "memory");
      int bad = 0;
      for (unsigned k = 0;; ++k) {
        unsigned now;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(arrived) : "memory");
        if ((int)(now - target) >= 0) break;
        if (k >= POLLS || ((k & 1023u) == 1023u && *(volatile int *)error != 0)) {
          atomicExch(error, 1);
          bad = 1;
          break;
        }
      }
      failed = bad;
    }
    __syncthreads();
    return failed == 0;
  }
};

// GB300 takes 64 cycles per FP64 warp instruction and scheduler, whatever its
// active lanes, so sums are laid out for few of them: only warps that hold
// values add, over no more lanes than hold them.
// Sum over the lanes that are a multiple of STRIDE (the others hold zeros).
template <int STRIDE>
__device__ __forceinline__ double warp_sum(double s) {
#pragma unroll
  for (int o = 16; o >= STRIDE; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}
// sums of v[0..N-1] over the block, to the block's places in part[0..N-1]; active: whether this warp holds any
template <int STRIDE, int N>
__device__ void block_sums(const double (&v)[N], bool active, double *part) {
  constexpr int W = RB / 32;
  __shared__ double red[N][W];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const double w = active ? warp_sum<STRIDE>(v[k]) : 0.;
    if (lane == 0) red[k][warp] = w;
  }
  __syncthreads();
  if (warp < N) {
    double w = lane < W ? red[warp][lane] : 0.;
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
    if (lane == 0) part[warp * MAX_BLOCKS + blockIdx.x] = w;
  }
}
// the blocks' sums added up, the same in every block: warp k sum k
template <int N>
__device__ void grid_sums(const double *part, double (&v)[N]) {
  __shared__ double tot[N];
  static_assert(N <= RB / 32, "one warp per sum");
  const int k = threadIdx.x / 32;
  if (k < N) {
    double w = 0.;
    for (unsigned i = threadIdx.x % 32; i < gridDim.x; i += 32) w += __ldcg(part + k * MAX_BLOCKS + i);
    w = warp_sum<1>(w);
    if (threadIdx.x % 32 == 0) tot[k] = w;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = tot[i];
  __syncthreads();
}
// row r of A times x, by LPR lanes (all lanes get the sum); a lane's loads go out in batches of UN.  Microseconds per
// BiCGSTAB iteration with UN = 3 / 5 / 9 / 13: rows of 9 entries (3000 1D cells) 20.1 / 20.6 / 22.0 / 22.8, of 36 (64^2;
// 200^2) 20.5 / 20.9 / 20.3 / 21.0 and 61.7 / 60.5 / 59.6 / 66.3, of 52 (256^2) 191 / 152 / 164 / 142, of 95 (32^3) 189 /
// 145 / 148 / 140.
__device__ __forceinline__ double row_times(const SolveArgs &a, long r, int lane, const double *x) {
  constexpr int UN = 9;
  double s = 0.;
  const int end = __ldg(a.rowptr + r + 1);
  row_batches<UN, LPR>(__ldg(a.rowptr + r), end, lane, [&](unsigned q) {
    int c[UN];
    double w[UN];
#pragma unroll
    for (int u = 0; u < UN; ++u) {
      const bool in = q + u * LPR < (unsigned)end;
      c[u] = in ? __ldg(a.colidx + q + u * LPR) : -1;
      w[u] = in ? __ldg(a.A + q + u * LPR) : 0.;
    }
    double g[UN];
#pragma unroll
    for (int u = 0; u < UN; ++u) g[u] = c[u] >= 0 ? x[c[u]] : 0.;
#pragma unroll
    for (int u = 0; u < UN; ++u)
      if (c[u] >= 0) s = fma(w[u], g[u], s);
  });
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, LPR);
  return s;
}

// Solve A x = b from x = 0.  Cooperative launch, RB threads per block; a
// block owns a run of consecutive rows.
__global__ void __launch_bounds__(RB, 1) k_bicgstab(SolveArgs a) {
  const long chunk = (a.n + gridDim.x - 1) / gridDim.x;
  const long lo = chunk * blockIdx.x < a.n ? chunk * blockIdx.x : a.n, hi = lo + chunk < a.n ? lo + chunk : a.n;
  const long own = lo + threadIdx.x;                      // vector entries own, own + RB, ... below hi
  const bool active = lo + threadIdx.x / 32 * 32 < hi;    // this warp holds vector entries
  const int lane = threadIdx.x % LPR;
  const long warpRow = lo + threadIdx.x / 32 * (32 / LPR);  // first row of this warp's lane groups
  const long group = lo + threadIdx.x / LPR;
  const bool rowsHere = warpRow < hi;
  GridBarrier bar{a.arrived, &a.info->error};
  int phase = 0;
  double *const parts[2] = {a.part, a.part + 2 * MAX_BLOCKS};  // one is read while the next is written
  double one[1] = {0.}, two[2];
  for (long i = own; i < hi; i += RB) {
    const double bi = a.b[i];
    a.r[i] = bi;
    a.x[i] = 0.;
    a.p[i] = 0.;
    a.v[i] = 0.;
    one[0] = fma(bi, bi, one[0]);
  }
  block_sums<1>(one, active, parts[phase]);
  if (!bar.sync()) return;
  grid_sums(parts[phase], one);
  phase ^= 1;
  const double bb = one[0];
  double rr = bb, rho = 1., alpha = 1., omega = 1., rhoNext = bb, dd = 0.;
  int it = 0;
  if (bb > 0.) {
    while (it < a.maxIt) {
      ++it;
      const double beta = div_rn(rhoNext, rho) * div_rn(alpha, omega);  // on the integer pipe
      rho = rhoNext;
      for (long i = own; i < hi; i += RB) {
        const double pi = fma(beta, fma(-omega, a.v[i], a.p[i]), a.r[i]);
        a.p[i] = pi;
        a.y[i] = pi * a.dinv[i];
      }
      if (!bar.sync()) return;
      one[0] = 0.;
      for (long w = warpRow, r = group; w < hi; w += RB / LPR, r += RB / LPR) {
        const double v = row_times(a, r < hi ? r : hi - 1, lane, a.y);
        if (r < hi && lane == 0) {
          a.v[r] = v;
          one[0] = fma(a.b[r], v, one[0]);
        }
      }
      block_sums<LPR>(one, rowsHere, parts[phase]);
      if (!bar.sync()) return;
      grid_sums(parts[phase], one);
      phase ^= 1;
      alpha = div_rn(rho, one[0]);
      for (long i = own; i < hi; i += RB) {
        const double si = fma(-alpha, a.v[i], a.r[i]);
        a.s[i] = si;
        a.z[i] = si * a.dinv[i];
      }
      if (!bar.sync()) return;
      two[0] = two[1] = 0.;
      for (long w = warpRow, r = group; w < hi; w += RB / LPR, r += RB / LPR) {
        const double t = row_times(a, r < hi ? r : hi - 1, lane, a.z);
        if (r < hi && lane == 0) {
          a.t[r] = t;
          two[0] = fma(t, t, two[0]);
          two[1] = fma(t, a.s[r], two[1]);
        }
      }
      block_sums<LPR>(two, rowsHere, parts[phase]);
      if (!bar.sync()) return;
      grid_sums(parts[phase], two);
      phase ^= 1;
      omega = two[0] > 0. ? div_rn(two[1], two[0]) : 0.;
      two[0] = two[1] = 0.;
      for (long i = own; i < hi; i += RB) {
        a.x[i] += fma(alpha, a.y[i], omega * a.z[i]);
        const double ri = fma(-omega, a.t[i], a.s[i]);
        a.r[i] = ri;
        two[0] = fma(ri, ri, two[0]);
        two[1] = fma(a.b[i], ri, two[1]);
      }
      block_sums<1>(two, active, parts[phase]);
      if (!bar.sync()) return;
      grid_sums(parts[phase], two);
      phase ^= 1;
      rr = two[0];
      rhoNext = two[1];
      if (!(rr >= 0.) || rr <= a.tol2 * bb) break;
    }
    // |x|^2 (each thread sums the entries that it wrote)
    one[0] = 0.;
    for (long i = own; i < hi; i += RB) one[0] = fma(a.x[i], a.x[i], one[0]);
    block_sums<1>(one, active, parts[phase]);
    if (!bar.sync()) return;
    grid_sums(parts[phase], one);
    dd = one[0];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.info->rr = rr;
    a.info->bb = bb;
    a.info->dd = dd;
    a.info->iters = it;
  }
}

// Device buffers of the solver.  A problem keeps up to KEPT_BYTES of them for its
// next call; larger ones are given back when the call ends, which costs the next
// call 1.2 to 1.8 ms of allocation (a call of 80 BiCGSTAB iterations: 256^2 WENO3,
// 100 MB, 10.8 ms kept and 12.0 allocated; 512^2 WENO5, 545 MB, 52.3 and 54.1).
constexpr size_t KEPT_BYTES = 256ul << 20;
struct Work {
  DevBuf<double> Un, Vn, V, J, dinv, R, d, r, p, v, s, t, y, z, part;
  DevBuf<unsigned> arrived;
  DevBuf<SolveInfo> info;
  int blocks = 0;
  size_t bytes() const {
    size_t n = J.n + part.n;
    for (auto *b : {&Un, &Vn, &V, &dinv, &R, &d, &r, &p, &v, &s, &t, &y, &z}) n += b->n;
    return n * sizeof(double);
  }
  void prepare(long n, long nnz) {
    for (auto *b : {&Un, &Vn, &V, &dinv, &R, &d, &r, &p, &v, &s, &t, &y, &z}) b->alloc((size_t)n);
    J.alloc((size_t)nnz);
    part.alloc(4 * MAX_BLOCKS);
    arrived.alloc(1);
    info.alloc(1);
    // every block resident: one per SM, whose registers 512 threads at 96 each leave no room for a second one, and no
    // more than the rows fill
    int dev = 0, sms = 0;
    PDA_CUDA(cudaGetDevice(&dev));
    PDA_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const long want = (n * LPR + RB - 1) / RB;
    blocks = (int)std::max<long>(std::min({want, (long)sms, (long)MAX_BLOCKS}), 1);
  }
};

unsigned g1(long n) { return (unsigned)((n + 255) / 256); }

// solve J_R d = R (x0 = 0); *dd = |d|^2, *relres the relative residual
int bicgstab(Work &w, long n, const int *rowptr, const int *colidx, double tol, int maxIt, cudaStream_t st,
             double *relres, double *dd) {
  PDA_CUDA(cudaMemsetAsync(w.arrived.p, 0, sizeof(unsigned), st));
  PDA_CUDA(cudaMemsetAsync(w.info.p, 0, sizeof(SolveInfo), st));
  SolveArgs a{n,      rowptr, colidx, w.J.p, w.dinv.p, w.R.p,     w.d.p,       w.r.p,    w.p.p,     w.v.p,
              w.s.p,  w.t.p,  w.y.p,  w.z.p, w.part.p, w.arrived.p, w.info.p, tol * tol, maxIt};
  void *args[] = {&a};
  PDA_CUDA(cudaLaunchCooperativeKernel((const void *)k_bicgstab, dim3((unsigned)w.blocks), dim3(RB), args, 0, st));
  SolveInfo h{};
  PDA_CUDA(cudaMemcpyAsync(&h, w.info.p, sizeof(h), cudaMemcpyDeviceToHost, st));
  PDA_CUDA(cudaStreamSynchronize(st));
  if (h.error) throw Error(PDA_ERR_INTERNAL, "BiCGSTAB: a wait between thread blocks ran out");
  *dd = h.dd;
  *relres = h.bb > 0. ? std::sqrt(h.rr / h.bb) : 0.;
  return h.iters;
}

}  // namespace impl
}  // namespace pda

using pda::Error;

extern "C" {

pda_status pda_advance_implicit(pda_problem *p, double *d_U, double t0, double dt, int64_t n_steps, int scheme,
                                double newton_tol, int newton_max_iters, double linear_tol, int linear_max_iters,
                                double *info) {
  PDA_API_BEGIN
  PDA_REQUIRE(p && d_U && n_steps >= 0 && (scheme == 0 || scheme == 1) && newton_max_iters >= 1 &&
                  linear_max_iters >= 1,
              PDA_ERR_INVALID_ARGUMENT, "invalid argument");
  pda_problem &P = *p;
  PDA_REQUIRE(P.dofsSample == P.dofsStencil, PDA_ERR_UNSUPPORTED, "implicit time integration needs a full mesh");
  const long n = (long)P.dofsStencil;
  int64_t rows = 0, cols = 0, nnz = 0;
  pda_status st = pda_jacobian_shape(p, &rows, &cols, &nnz);
  if (st != PDA_OK) throw Error(st, pda_last_error());
  if (!P.implicitWork) P.implicitWork = std::make_shared<pda::impl::Work>();
  pda::impl::Work &w = *std::static_pointer_cast<pda::impl::Work>(P.implicitWork);
  struct GiveBack {  // on every way out
    std::shared_ptr<void> &work;
    ~GiveBack() {
      if (std::static_pointer_cast<pda::impl::Work>(work)->bytes() > pda::impl::KEPT_BYTES) work.reset();
    }
  } giveBack{P.implicitWork};
  w.prepare(n, (long)nnz);
  cudaStream_t s = P.stream;
  pda::ensure_device_pattern(P);
  const int *rowptr = P.d_rowptr.p, *colidx = P.d_colidx.p;
  int totalNewton = 0, totalLinear = 0, maxNewton = 0;
  double worstRel = 0.;
  double t = t0;
  for (int64_t step = 0; step < n_steps; ++step) {
    PDA_CUDA(cudaMemcpyAsync(w.Un.p, d_U, (size_t)n * sizeof(double), cudaMemcpyDeviceToDevice, s));
    if (scheme == 1) {
      st = pda_velocity(p, w.Un.p, t, w.Vn.p);
      if (st != PDA_OK) throw Error(st, pda_last_error());
    }
    const double c = scheme == 0 ? -dt : -dt / 2.;
    int it = 0;
    for (; it < newton_max_iters; ++it) {
      st = pda_velocity_and_jacobian(p, d_U, t + dt, w.V.p, w.J.p);
      if (st != PDA_OK) throw Error(st, pda_last_error());
      pda::impl::k_system<<<pda::impl::g1(n * pda::impl::LPR), 256, 0, s>>>(
          scheme, n, rowptr, colidx, d_U, w.Un.p, w.V.p, w.Vn.p, dt, c, w.J.p, w.dinv.p, w.R.p);
      PDA_CUDA(cudaGetLastError());
      double rel = 0., dd = 0.;
      totalLinear += pda::impl::bicgstab(w, n, rowptr, colidx, linear_tol, linear_max_iters, s, &rel, &dd);
      worstRel = std::max(worstRel, rel);
      if (std::sqrt(dd) < newton_tol) break;  // stop before updating, as Pressio does
      pda::impl::k_minus<<<pda::impl::g1(n), 256, 0, s>>>(n, w.d.p, d_U);
    }
    totalNewton += it + 1;
    maxNewton = std::max(maxNewton, it + 1);
    t = t + dt;
  }
  PDA_CUDA(cudaStreamSynchronize(s));
  if (info) {
    info[0] = (double)totalNewton;
    info[1] = (double)maxNewton;
    info[2] = (double)totalLinear;
    info[3] = worstRel;
  }
  PDA_API_END
}

}  // extern "C"

// One Gauss-Newton iteration of hyper-reduced LSPG (BDF1 or BDF2) in one
// launch: sample-mesh velocity V, the product Jf D of the sample-mesh
// Jacobian with the trial space's latent Jacobian D formed face by face
// (never assembling Jf), the LSPG residual R = cf V + (y + cn y_n [+ cnm1
// y_n-1]) and JR = cf Jf D + D at the sample dofs, the block partial sums of
// JR^T JR, JR^T R and R^T R, and, in the last block to finish, their
// reduction, the k x k solve and the latent update (Pressio's
// LspgUnsteadyResidualJacobianPolicyHypRed,
// lspg_unsteady_rj_policy_hypred.hpp:180-264).
//
// Jf D row by row: Jf's row is the sum over the row's faces of
// +-h^-1 (JN dU/dq + JP dU/dq) with dU/dq the reconstruction gradients, so
//   (Jf D)_row = sum_faces +-h^-1 (JN (sum_s gN_s D_s) + JP (sum_s gP_s D_s)),
// one face and one latent column per thread.  Near-boundary rows use the
// first-order Jacobian with the ghost dependence folded into the row's own
// cell by the BC factors (the assembled Jacobian's rule), i.e. D of a ghost
// is the factor times D of the cell.  Same products as forming Jf and then
// Jf D (the assembled path), in another order: equal to rounding.
//
// Blocks [0, nbInner) take inner rows, the others near-boundary rows; each
// block takes RPB rows through the phases of k_rows_vj_inner_par /
// k_rows_vj_nearbd_par (GB300's narrow FP64 units make the per-thread
// instruction chain the cost, so the work of a row is spread over threads).
// An iteration is one wave of blocks and its time one block's chain, not a
// rate: at 628 shallow-water rows with 12 latents about 43,000 cycles, of which
// the loads, face values and fluxes take 17,000, the columns and the products
// 10,000, the groups' sums 5,000 and the solve 11,000.  A Gauss-Newton step
// with its decoder went 51.4 -> 48.6 us with the L D L^T solve and the batched
// sums, 44.8 with the rows' states and histories on warps of their own and the
// copies' table entries loaded ahead, 43.3 with the fluxes on warps that start
// when the values are there.
#pragma once

#include "kernels.cuh"

namespace pda {

constexpr int kLspgKMax = 32;

// Rows per block are chosen at launch (rpb <= RPB_MAX) so that the grid
// covers the SMs once where the row count allows (a second block on one SM
// doubles that SM's chain) and the dynamic shared memory fits.
template <int FAM> struct FusedPar {
  static constexpr int NF = 2 * Fam<FAM>::dim, NDPC = Fam<FAM>::ndpc, DIM = Fam<FAM>::dim;
  static constexpr int RPB_MAX = Fam<FAM>::dim == 3 ? 4 : 8;
  static constexpr int SIDE = pad_warp(RPB_MAX * NF * NDPC);
  static constexpr int PART = pad_warp(RPB_MAX * NF);
  // phase A's two sides, phase B's four parts, and two warps for the rows' states and histories: all side by side,
  // or phase B and these two on phase A's warps
  static constexpr int threads(bool beside) {
    return beside ? 2 * SIDE + 4 * PART + 64 : (2 * SIDE > 4 * PART + 64 ? 2 * SIDE : 4 * PART + 64);
  }
  static_assert(RPB_MAX * NF <= PART && RPB_MAX * NDPC <= 32, "a warp covers the block's faces and rows");
  static constexpr size_t kSmemLimit = 160 * 1024;  // dynamic shared memory per block
  // dynamic shared memory per row: staged D of the row's stencil cells, the
  // per-face J D columns and the row's JR rows
  static size_t smem_row(int S, int K) {
    return sizeof(double) * ((size_t)DIM * S * NDPC * K + (size_t)NF * NDPC * K + (size_t)NDPC * (K + 1));
  }
};

// Blocks are reduced in groups of kLspgGroup: the last block of a group to
// finish sums the group's partial sums in block order, the last group to
// finish sums the group sums in group order and solves.  Both levels run one
// thread per entry with independent loads, since a chain of dependent FP64
// adds costs ~70 cycles a step on GB300.

// sum of rows [r0, r1) of a [rows][ne] array, entry by entry, in row order;
// a group's loads all in flight
__device__ inline double lspg_sum_rows(const double *__restrict__ a, int ne, int e, int r0, int r1) {
  double s = 0.;
  for (int r = r0; r < r1; r += kLspgGroup) {
    double v[kLspgGroup];
#pragma unroll
    for (int k = 0; k < kLspgGroup; ++k) v[k] = r + k < r1 ? a[(long)(r + k) * ne + e] : 0.;
#pragma unroll
    for (int k = 0; k < kLspgGroup; ++k)
      if (r + k < r1) s += v[k];
  }
  return s;
}

// Index tables of the normal equations' triangles, filled while phase A waits
// for its loads: entry e of the upper triangle of order K (row major) as (ua,
// ub), and the lower-triangle pairs (pi, pl), pi >= pl, of the augmented order
// K + 1, by pl descending, so that the pairs with pl > j are the first
// (K - j)(K + 1 - j) / 2.
struct LspgTables {
  static constexpr int KA = kLspgKMax + 1, N = KA * (KA + 1) / 2;
  unsigned char ua[N], ub[N], pi[N], pl[N];
};
__device__ __forceinline__ void lspg_tables(LspgTables &t, int K, int from, int count) {
  const int Ka = K + 1;
  for (int q = from; q < Ka * (Ka + 1) / 2; q += count) {
    int l = Ka - 1, rem = q;
    while (rem >= Ka - l) {
      rem -= Ka - l;
      --l;
    }
    t.pi[q] = (unsigned char)(l + rem);
    t.pl[q] = (unsigned char)l;
    int a = 0;
    rem = q;
    while (a < K && rem >= K - a) {
      rem -= K - a;
      ++a;
    }
    t.ua[q] = (unsigned char)a;
    t.ub[q] = (unsigned char)(a + rem);
  }
}

// Elimination of pivot d = H_jj outside the integer pipe's window (a basis or a
// state in extreme units), where the products H_rj H_cj would leave the range of
// their quotient: H_rc -= (s H_rj H_cj) / m with d = m / s, s a power of two.
// Out of line: no ordinary pivot comes here.  Returns 1 / d.
static __device__ __noinline__ double lspg_pivot_scaled(double (*H)[LspgTables::KA + 1], int j, int np, double d,
                                                        const LspgTables &t) {
  const int ex = (int)(__double_as_longlong(d) >> 52), cut = min(max(ex, 1), 2045);
  const double s = __longlong_as_double((long long)(2046 - cut) << 52), m = d * s;
  for (int q = threadIdx.x; q < np; q += blockDim.x) {
    const int row = t.pi[q], col = t.pl[q];
    H[row][col] -= H[row][j] * s * H[col][j] / m;
  }
  return s / m;
}

// reduce the group sums in group order, factor, solve, update (the calling
// block): L D L^T elimination of the matrix [H g; g^T .] augmented by the
// right-hand side, whose last row becomes D L^-1 g in the trailing updates (no
// separate forward substitution), then a lane-parallel back substitution by
// warp 0.  The chain of pivots is what it costs: a reciprocal on the integer
// pipe (250 cycles) where a reciprocal square root on GB300's FP64 pipe takes
// about 1,000, and each trailing update one round of the whole block, since an
// FP64 instruction holds a scheduler for 64 cycles.
__device__ inline void lspg_solve_rt(int K, int nparts, const double *__restrict__ partial, double *__restrict__ x,
                                     double tol, int first, LspgFlags *f, const LspgTables &t) {
  constexpr int KA = LspgTables::KA;
  __shared__ double H[KA][KA + 1];
  __shared__ double rr;
  const int ntri = K * (K + 1) / 2, ne = ntri + K + 1, Ka = K + 1;
  const int lane = threadIdx.x & 31;
  for (int e = threadIdx.x; e < ne; e += blockDim.x) {
    const double s = lspg_sum_rows(partial, ne, e, 0, nparts);
    if (e < ntri) H[t.ub[e]][t.ua[e]] = s;
    else if (e < ntri + K) H[K][e - ntri] = s;  // the right-hand side as the augmented row
    else rr = s;
  }
  __syncthreads();
  bool ok = true;
  double rd = 0.;  // lane j: reciprocal of pivot j
  // this thread's pair of the trailing triangle, the same for every pivot (further ones in a loop)
  const int q0 = threadIdx.x;
  const int row0 = t.pi[q0 < LspgTables::N ? q0 : 0], col0 = t.pl[q0 < LspgTables::N ? q0 : 0];
#pragma unroll 1
  for (int j = 0; j < K; ++j) {
    const double d = H[j][j];
    const int np = (Ka - 1 - j) * (Ka - j) / 2;
    // positive and finite, tested on the bits (no FP64 instruction)
    const long long db = __double_as_longlong(d);
    if (!(db > 0 && ip::in_window(d))) {
      if (!(db > 0 && db < 0x7FF0000000000000LL)) {
        ok = false;
        break;
      }
      const double r = lspg_pivot_scaled(H, j, np, d, t);
      if (lane == j) rd = r;
      __syncthreads();
      continue;
    }
    // trailing lower triangle (the augmented row included): H_rc -= (H_rj H_cj) / d, the product beside the reciprocal
    double h = 0., p = 0.;
    if (q0 < np) {
      h = H[row0][col0];
      p = H[row0][j] * H[col0][j];
    }
    const double r = div_rn<true>(1., d);
    if (lane == j) rd = r;
    if (q0 < np) H[row0][col0] = fma(-p, r, h);
#pragma unroll 1
    for (int q = q0 + blockDim.x; q < np; q += blockDim.x) {
      const int row = t.pi[q], col = t.pl[q];
      H[row][col] = fma(-(H[row][j] * H[col][j]), r, H[row][col]);
    }
    __syncthreads();
  }
  if (threadIdx.x >= 32) return;
  double sv = lane < K ? H[K][lane] : 0.;  // D L^-1 g
  double corr = 0.;
  if (ok) {
#pragma unroll 1
    for (int i = K - 1; i >= 0; --i) {
      const double di = __shfl_sync(0xffffffffu, sv * rd, i);
      if (lane == i) sv = di;
      if (lane < i) sv = fma(-H[i][lane], di, sv);
    }
    if (lane < K) x[lane] -= sv;
    double c2 = lane < K ? sv * sv : 0.;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c2 += __shfl_xor_sync(0xffffffffu, c2, o);
    corr = c2;
  }
  if (lane == 0) {
    // the first iteration of a step starts the step's count and flag
    const double c = sqrt_rn(corr), res = sqrt_rn(rr);
    f->iters = first ? 1 : f->iters + 1;
    f->lastCorr = c;
    f->lastRes = res;
    if (!(res <= f->maxRes)) f->maxRes = res;
    f->converged = (!ok || c < tol) ? 1 : 0;
  }
}

// one face of a block's rows: the flux and face values in double, the
// Jacobian terms in JT (double, or float for the inexact Gauss-Newton step)
template <int FAM, int SCHEME, typename JT> struct FusedFace {
  static constexpr int NDPC = Fam<FAM>::ndpc, G = 2 * SchemeTraits<SCHEME>::h;
  double fl[NDPC];
  double uN[NDPC], uP[NDPC];
  JT JN[NDPC * NDPC], JP[NDPC * NDPC];
  JT gN[NDPC][G], gP[NDPC][G];
};

// 16-byte global -> shared copy that does not hold up the issuing warp
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// JT: the scalar type of the Jacobian terms (double: the exact Jacobian of
// the sample-mesh residual; float: an approximate one, on GB300's far wider
// FP32 units, for an inexact Gauss-Newton step on the same double residual)
// BESIDE: the fluxes and the rows' states on warps beside the face values', a
// shorter chain for one wave of blocks; without it half as many threads, and so
// twice as many resident blocks, for grids of several waves
template <int FAM, int SCHEME, typename JT, bool BESIDE>
__global__ void __launch_bounds__(FusedPar<FAM>::threads(BESIDE))
k_lspg_fused(RowTable ti, RowTable tn, int rpb, int nbInner, MeshArgs m, Phys p, LspgArgs a) {
  if (!a.first && a.f->converged) return;
  using F = Fam<FAM>;
  using FP = FusedPar<FAM>;
  using FF = FusedFace<FAM, SCHEME, JT>;
  constexpr bool kExact = sizeof(JT) == sizeof(double);
  constexpr int NDPC = F::ndpc, DIM = F::dim, H = SchemeTraits<SCHEME>::h, S = 2 * H + 1, G = 2 * H;
  constexpr int NF = FP::NF;
  __shared__ FF fd[FP::RPB_MAX][NF];
  __shared__ double sY[FP::RPB_MAX][NDPC];    // state at the row's cell
  __shared__ double sSrc[FP::RPB_MAX][NDPC];  // source-term velocity (shallow water: Coriolis)
  __shared__ double sSJ[FP::RPB_MAX][NDPC * NDPC];  // its Jacobian
  __shared__ double sHist[2][FP::RPB_MAX * NDPC];   // y_n, y_n-1 at the row's dofs
  __shared__ int sRow[FP::RPB_MAX];
  __shared__ LspgTables tabs;
  __shared__ typename F::Side sSide[FP::RPB_MAX][NF][2];  // the two face states' halves of the flux
  extern __shared__ double dyn[];
  constexpr int THREADS = FP::threads(BESIDE), kHandOver = 2 * FP::SIDE + 4 * FP::PART;
  const int tid = threadIdx.x, K = a.K, RD = rpb * NDPC, CB = NDPC * K;  // CB: D doubles per cell
  double *sD = dyn;                                  // [rpb][DIM][S][NDPC][K] staged D of stencil cells
  double *ctb = sD + (size_t)rpb * DIM * S * CB;     // [rpb][NF][NDPC][K]
  double *sJR = ctb + (size_t)rpb * NF * NDPC * K;   // [RD][K + 1]
  const bool inner = (int)blockIdx.x < nbInner;
  const RowTable &t = inner ? ti : tn;
  const int e0 = (inner ? (int)blockIdx.x : (int)blockIdx.x - nbInner) * rpb;
  // D of the stencil cells (inner rows: the scheme's stencil; near rows: the
  // first-order cells) staged by asynchronous copies that overlap phase A
  {
    const int npos = inner ? S : 3, chunks = CB / 2;
    const int total = rpb * DIM * npos * chunks;
    // (a round's table entries are loaded before its copies are issued: one wait for the table, not one per copy)
    constexpr int UN = 6;
    for (int w0 = tid; w0 < total; w0 += UN * THREADS) {
      int cell[UN], at[UN];
#pragma unroll
      for (int u = 0; u < UN; ++u) {
        const int w = w0 + u * THREADS;
        const int ch = w % chunks, pa = w / chunks, ps = pa % npos, ax = (pa / npos) % DIM, rl = pa / (npos * DIM);
        const int e = e0 + rl;
        at[u] = w < total && e < t.nrows ? ((rl * DIM + ax) * S + ps) * CB + 2 * ch : -1;
        if (at[u] >= 0)
          cell[u] = inner ? t.src[((size_t)e * DIM + ax) * S + ps] : t.src1[((size_t)e * DIM + ax) * 3 + ps];
      }
#pragma unroll
      for (int u = 0; u < UN; ++u) {
        const int ch = (w0 + u * THREADS) % chunks;
        if (at[u] >= 0) cp_async16(sD + at[u], a.D + (size_t)cell[u] * CB + 2 * ch);
      }
    }
  }
  // the rows' states and source terms (one warp), the history of their dofs and the tables (another)
  auto row_state_and_source = [&](int rl) {
    const int e = e0 + rl;
    if (rl >= rpb || e >= t.nrows) return;
    const int cell = t.cell[e];
    double y[NDPC];
#pragma unroll
    for (int d = 0; d < NDPC; ++d) y[d] = __ldg(a.y + (size_t)cell * NDPC + d);
#pragma unroll
    for (int d = 0; d < NDPC; ++d) {
      sY[rl][d] = y[d];
      sSrc[rl][d] = 0.;
    }
#pragma unroll
    for (int i = 0; i < NDPC * NDPC; ++i) sSJ[rl][i] = 0.;
    if constexpr (FAM == Swe2d) {
      // Coriolis source (swe_2d_prob_class.hpp:983-1012) and its Jacobian
      const double u0 = y[0], u1 = y[1], u2 = y[2];
      // (divisions on the integer pipe, the IEEE quotients)
      sSrc[rl][1] = -div_rn(p.coriolis * u2, u0);
      sSrc[rl][2] = div_rn(p.coriolis * u1, u0);
      sSJ[rl][1 * 3 + 0] = div_rn(p.coriolis * u2, (u0 * u0));
      sSJ[rl][1 * 3 + 2] = div_rn(-p.coriolis, u0);
      sSJ[rl][2 * 3 + 1] = div_rn(p.coriolis, u0);
      sSJ[rl][2 * 3 + 0] = div_rn(-p.coriolis * u1, (u0 * u0));
    }
  };
  // GB300 issues one FP64 warp instruction per ~64 cycles per sub-partition
  // whatever the number of active lanes, so the time is the longest per-warp
  // chain.  Phase A's warps hand the face values over before they go on to the
  // gradients; phase B's, beside them, form the two face states' halves of the
  // flux (parts 0, 1, then part 0 their combination) and JN, JP (parts 2, 3).
  const int nrow = min(rpb, t.nrows - e0);
  if (tid < 2 * FP::SIDE) {  // phase A: (side, row, face, dof): one side of the face value (+ gradient for inner rows)
    const int side = tid / FP::SIDE;
    const bool on = tid % FP::SIDE < nrow * NF * NDPC;  // (the other lanes repeat the first)
    const int slot = on ? tid % FP::SIDE : 0;
    const int rl = slot / (NF * NDPC), f = (slot / NDPC) % NF, d = slot % NDPC, ax = f >> 1, fs = f & 1;
    const size_t base = ((size_t)(e0 + rl) * DIM + ax) * S;
    double q[G];
    FF &o = fd[rl][f];
    auto hand_over = [&](double v) {
      if (on) (side == 0 ? o.uN : o.uP)[d] = v;
      if constexpr (BESIDE) bar_arrive<1>(kHandOver);
    };
    if (inner) {
#pragma unroll
      for (int s = 0; s < G; ++s) q[s] = __ldg(a.y + (size_t)t.src[base + fs + s] * NDPC + d);
      JT u, gg[G];
      if constexpr (kExact) {
        face_grad_side<SCHEME>(side, u, gg, q, hand_over);
      } else {
        // the value in double (it enters V and R); the gradient in float
        hand_over(face_value_side<SCHEME>(side, q));
        JT qf[G];
#pragma unroll
        for (int s = 0; s < G; ++s) qf[s] = (JT)q[s];
        face_grad_side<SCHEME>(side, u, gg, qf);
      }
      JT *gs = side == 0 ? o.gN[d] : o.gP[d];
#pragma unroll
      for (int s = 0; s < G; ++s)
        if (on) gs[s] = gg[s];
    } else {
#pragma unroll
      for (int s = 0; s < G; ++s) {
        double qe[NDPC];
        load_entry<NDPC>(qe, a.y, t.src[base + fs + s], t.flip[base + fs + s], m.reflect[ax], m, t.gsx, t.gsy,
                         base + fs + s);
        q[s] = qe[d];
      }
      hand_over(face_value_side<SCHEME>(side, q));
    }
  }
  if constexpr (!BESIDE) __syncthreads();
  const int tb = BESIDE ? tid - 2 * FP::SIDE : tid;  // this thread's place in phase B and the rows' warps
  if (tb < 0) {
    // (phase A's, beside them)
  } else if (tb < 4 * FP::PART) {  // phase B: (part, row, face)
    const int part = tb / FP::PART, slot = tb % FP::PART;
    const int rl = slot / NF, f = slot % NF, ax = f >> 1, fs = f & 1;
    const bool on = slot < nrow * NF;
    if constexpr (BESIDE) bar_wait<1>(kHandOver);
    if (part < 2) {
      // (one stream for all axes of the warp)
      if (on) F::flux_side_ax(sSide[rl][f][part], part == 0 ? fd[rl][f].uN : fd[rl][f].uP, p, ax);
      if (part == 1) bar_arrive<2>(2 * FP::PART);
      else bar_wait<2>(2 * FP::PART);
      if (part == 0 && on) {
        FF &o = fd[rl][f];
        const typename F::Side &L = sSide[rl][f][0], &R = sSide[rl][f][1];
        F::template flux_combine<0>(o.fl, o.uN, o.uP, L, R, p);  // the combination does not depend on the axis
      }
    } else if (on) {
      FF &o = fd[rl][f];
      double uN[NDPC], uP[NDPC];
#pragma unroll
      for (int d = 0; d < NDPC; ++d) {
        uN[d] = o.uN[d];
        uP[d] = o.uP[d];
      }
      if (!inner) {
        // first-order Jacobian at the face's two cells (ghosts through their recipes)
        const size_t b1 = ((size_t)(e0 + rl) * DIM + ax) * 3;
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          double qe[NDPC];
          load_entry<NDPC>(qe, a.y, t.src1[b1 + fs + s], t.flip1[b1 + fs + s], m.reflect[ax], m, t.gsx1, t.gsy1,
                           b1 + fs + s);
#pragma unroll
          for (int d = 0; d < NDPC; ++d) (s == 0 ? uN : uP)[d] = qe[d];
        }
      }
      JT J2[NDPC * NDPC], vN[NDPC], vP[NDPC];
#pragma unroll
      for (int d = 0; d < NDPC; ++d) {
        vN[d] = (JT)uN[d];
        vP[d] = (JT)uP[d];
      }
      // (one stream for all axes of the warp; the Jacobian that is not stored is not computed)
      if (part == 2) F::flux_jac_ax(o.JN, J2, vN, vP, p, ax);
      else F::flux_jac_ax(J2, o.JP, vN, vP, p, ax);
    }
  } else if (tb < 4 * FP::PART + 32) {
    row_state_and_source(tb - 4 * FP::PART);
  } else if (tb < 4 * FP::PART + 64) {
    const int rk = tb - 4 * FP::PART - 32;
    if (rk < nrow * NDPC) {
      const int r = t.rows[e0 + rk / NDPC];
      if (rk % NDPC == 0) sRow[rk / NDPC] = r;
      sHist[0][rk] = a.yn[(size_t)r * NDPC + rk % NDPC];
      sHist[1][rk] = a.ynm1[(size_t)r * NDPC + rk % NDPC];
    }
    lspg_tables(tabs, K, rk, 32);
  }
  cp_async_wait_all();
  __syncthreads();
  // phase C: (row, face, column c): the face's (JN dU_N + JP dU_P) D column
  for (int w = tid; w < rpb * NF * K; w += blockDim.x) {
    const int rl = w / (NF * K), f = (w / K) % NF, c = w % K, ax = f >> 1, fs = f & 1;
    const int e = e0 + rl;
    if (e >= t.nrows) continue;
    const FF &o = fd[rl][f];
    const double *Dax = sD + ((size_t)rl * DIM + ax) * S * CB;  // staged D of this axis' positions
    JT dN[NDPC], dP[NDPC];
    if (inner) {
#pragma unroll
      for (int d = 0; d < NDPC; ++d) {
        dN[d] = JT(0);
        dP[d] = JT(0);
      }
#pragma unroll
      for (int s = 0; s < G; ++s) {
        const double *Ds = Dax + (size_t)(fs + s) * CB;
#pragma unroll
        for (int d = 0; d < NDPC; ++d) {
          const JT dv = (JT)Ds[d * K + c];
          dN[d] = fma(o.gN[d][s], dv, dN[d]);
          dP[d] = fma(o.gP[d][s], dv, dP[d]);
        }
      }
    } else {
      const size_t b1 = ((size_t)e * DIM + ax) * 3;
      const double *fac = t.jfac + ((size_t)e * DIM + ax) * NDPC;
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int pos = fs + s;
        const bool ghost = t.jpos1[b1 + pos] < 0;
        const double *Ds = Dax + (size_t)(ghost ? 1 : pos) * CB;  // position 1 is the row's cell
#pragma unroll
        for (int d = 0; d < NDPC; ++d) {
          const double dv = Ds[d * K + c];
          (s == 0 ? dN : dP)[d] = (JT)(ghost ? fac[d] * dv : dv);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < NDPC; ++k) {
      JT acc = JT(0);
#pragma unroll
      for (int d = 0; d < NDPC; ++d) {
        acc = fma(o.JN[k * NDPC + d], dN[d], acc);
        acc = fma(o.JP[k * NDPC + d], dP[d], acc);
      }
      ctb[(((size_t)rl * NF + f) * NDPC + k) * K + c] = (double)acc;
    }
  }
  __syncthreads();
  // phase D: (row, k, column c <= K): JR = cf Jf D + D and, in column K, R
  for (int w = tid; w < RD * (K + 1); w += blockDim.x) {
    const int rk = w / (K + 1), c = w % (K + 1), rl = rk / NDPC, k = rk % NDPC;
    const int e = e0 + rl;
    double val = 0.;
    if (e < t.nrows) {
      const double *Dself = sD + ((size_t)rl * DIM * S + (inner ? H : 1)) * CB;  // axis 0, the row's cell
      if (c < K) {
        double jd = 0.;
#pragma unroll
        for (int ax = 0; ax < DIM; ++ax)
          jd = fma(m.hinv[ax],
                   ctb[(((size_t)rl * NF + 2 * ax) * NDPC + k) * K + c] -
                       ctb[(((size_t)rl * NF + 2 * ax + 1) * NDPC + k) * K + c],
                   jd);
        if constexpr (FAM == Swe2d) {
#pragma unroll
          for (int j = 0; j < NDPC; ++j) jd = fma(sSJ[rl][k * NDPC + j], Dself[j * K + c], jd);
        }
        val = fma(a.cf, jd, Dself[k * K + c]);
      } else {
        double vk = 0.;
#pragma unroll
        for (int ax = 0; ax < DIM; ++ax) vk += m.hinv[ax] * (fd[rl][2 * ax].fl[k] - fd[rl][2 * ax + 1].fl[k]);
        if constexpr (FAM == Swe2d) vk += sSrc[rl][k];
        const size_t q = (size_t)sRow[rl] * NDPC + k;
        a.V[q] = vk;
        const double ynp1 = sY[rl][k];
        double yn = sHist[0][rk], ynm1 = sHist[1][rk];
        if (a.first) {
          ynm1 = yn;
          yn = ynp1;
          a.ynm1[q] = ynm1;
          a.yn[q] = yn;
        }
        // Pressio's ops::update(helper, 0, y_n+1, 1, y_n, cn[, y_n-1, cnm1])
        const double helper = a.bdf2 ? 1. * ynp1 + a.cn * yn + a.cnm1 * ynm1 : 1. * ynp1 + a.cn * yn;
        val = a.cf * vk + 1. * helper;
      }
    }
    sJR[(size_t)rk * (K + 1) + c] = val;
  }
  __syncthreads();
  // phase E: block partial sums of the upper triangle of JR^T JR, of JR^T R, R^T R
  const int ntri = K * (K + 1) / 2, ne = ntri + K + 1;
  for (int q = tid; q < ne; q += blockDim.x) {
    // (the upper triangle, then the columns against R, then R against itself)
    const int ia = q < ntri ? tabs.ua[q] : (q < ntri + K ? q - ntri : K), ib = q < ntri ? tabs.ub[q] : K;
    double s = 0.;
    for (int i = 0; i < RD; ++i) s = fma(sJR[(size_t)i * (K + 1) + ia], sJR[(size_t)i * (K + 1) + ib], s);
    a.partial[(long)blockIdx.x * ne + q] = s;
  }
  // the last block of a group reduces the group; the last group solves (no
  // block waits for another).  ticket[0] counts groups, ticket[1 + g] blocks.
  __shared__ unsigned last;
  const int nb = (int)gridDim.x, ng = lspg_groups(nb), grp = (int)blockIdx.x / kLspgGroup;
  const int g0 = grp * kLspgGroup, g1 = min(nb, g0 + kLspgGroup);
  double *gsum = a.partial + (long)nb * ne;  // [groups][ne] after the block sums
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(a.ticket + 1 + grp, 1u) == (unsigned)(g1 - g0 - 1) ? 1u : 0u;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int q = tid; q < ne; q += blockDim.x) gsum[(long)grp * ne + q] = lspg_sum_rows(a.partial, ne, q, g0, g1);
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    a.ticket[1 + grp] = 0u;
    last = atomicAdd(a.ticket, 1u) == (unsigned)(ng - 1) ? 1u : 0u;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  lspg_solve_rt(K, ng, gsum, a.x, a.tol, a.first, a.f, tabs);
  if (tid == 0) *a.ticket = 0u;
}

}  // namespace pda

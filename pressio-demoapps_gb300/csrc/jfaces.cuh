// Velocity + exact Jacobian on the inner box of a natural-order full mesh,
// each face computed once, the CSR values assembled in the same kernel.
//
// The reference (and k_rows_vj_inner) evaluates, for every row, the WENO
// reconstruction with gradients and the Rusanov flux Jacobians of its left and
// right faces, so every face is computed twice, and accumulates
//     J[row k, col(c_s) j] += (JLNeg(k,j) * gLNeg(j,s)) * h^-1    (left face)
//     J[row k, col(c_s) j] += (JLPos(k,j) * gLPos(j,s)) * h^-1
//     J[row k, col(c_s) j] -= (JRNeg(k,j) * gRNeg(j,s)) * h^-1    (right face)
//     J[row k, col(c_s) j] -= (JRPos(k,j) * gRPos(j,s)) * h^-1
// (mixin_directional_flux_balance_jacobian.hpp:222-282), x then y then z.
// Every product term belongs to one face and is the same for the two cells
// that share it.  k_jtile takes one axis per launch: a block owns 32
// consecutive faces of one line of the box (31 cells; the face at a tile's
// end is computed by both neighbouring tiles), one warp per dof.  Warp k
// reconstructs dof k's two face states with their gradients, the warps then
// form the flux and its left and right Jacobian (in stages, or the first two
// whole), and warp k finally takes row k of the Jacobian: lane by lane the face's product terms (Neg and Pos, per
// stencil position s, one column dof j at a time), the right face's from the
// next lane, added in the reference's order (left Neg, left Pos, right Neg,
// right Pos) into the CSR values.  The
// centre block gathers every axis: the first axis's launch starts it from
// zero, later axes continue the partial sum stored in J (the same
// additions in the same order), and the last adds the shallow-water
// Coriolis terms.  Velocities follow the same pattern.  Results are
// bit-identical to the per-row formulation; DRAM traffic is the state reads,
// the CSR values written (the centre block re-read once per later axis) and
// the velocity.
// Used when no stencil repeats a cell (periodic axes of at least 2H+1 cells).
//
// What bounds it: issue and waits, FP64 no longer.  A 2D Euler WENO5 face took
// 2,850 FP64 instructions when one thread held it whole (its gradients and
// Jacobians in 128 registers, 4 warps per scheduler) and takes 1,280 here:
// terms whose factor is a known zero or one are left out (weno5_side_grad,
// weno3_side_grad, euler4_flux_jac2, EulerJac, the gradient's end components),
// exact powers of two join a sum, and the products run on the integer pipe,
// which the 32 warps per SM of the split by dof can hide.  512^2 WENO5 V + J
// 3.24 -> 1.87 ms (issue 49 %, FP64 pipe 60 %; a fifth of the stalls wait for
// instructions, a sixth at barriers), 41 x 37 x 43 WENO3 1.35 -> 0.95 ms by the
// split, 0.89 by the WENO3 gradients, 0.80 by the stages.  With the WENO5
// gradients' products on the FP64 pipe 2.20 ms; with 7 / 9 resident blocks of
// the 2D kernel 2.07 / 2.13 ms; with one copy of the gradients' common part for
// both sides 2.00 ms (its coefficients spill).
#pragma once

#include "kernels.cuh"

namespace pda {

template <int FAM, int SCHEME> struct JTileCfg {
  static constexpr int NDPC = Fam<FAM>::ndpc, DIM = Fam<FAM>::dim, H = SchemeTraits<SCHEME>::h, G = 2 * H;
  static constexpr int LANES = 32, TW = LANES - 1;  // faces and cells per tile
  static constexpr int THREADS = LANES * NDPC;
  // resident blocks per SM the register allocation must allow: about 32 warps
  static constexpr int MINBLOCKS = NDPC == 4 ? 8 : (NDPC == 5 ? 6 : 10);
};

// What the stages of a face's flux Jacobians hand to one another (EulerJac), a
// lane per face.  Elsewhere two warps form a whole Jacobian each: the small
// families have few terms in common, and 2D WENO5 needs the shared memory's
// share of L1 for its spilled registers (512^2 1905 us so, 1935 in stages;
// WENO3 1091 and 1025; 41 x 37 x 43 WENO3 885 and 799, WENO5 1553 and 1531).
template <int FAM, int SCHEME> struct EulerFace {
  static constexpr int NDPC = Fam<FAM>::ndpc, DIM = Fam<FAM>::dim;
  static constexpr bool staged = FAM == Euler3d || (FAM == Euler2d && SCHEME == Weno3);
  struct Kept {  // read by the rows' entries
    double v[2][DIM][32], V2[2][32], H[2][32];  // the two states' velocity, |v|^2, enthalpy
    double g[2][NDPC][32], smax[32];            // wave speed and its derivatives
  };
  struct Passing {
    double p[2][32], A2[2][32], inv[2][32];  // pressure, a^2 / (gamma - 1), 1 / (rho + r)
    double r[32], RT[32], v[DIM][32], H[32], V2es[32], a[32], ga[32], rel[DIM][32];  // Roe averages
  };
};
struct Nothing {};

template <int FAM, int SCHEME> struct JTileSmem {
  using C = JTileCfg<FAM, SCHEME>;
  using EF = EulerFace<FAM, SCHEME>;
  double u[2][C::NDPC][C::LANES];                 // face states, left- and right-biased
  double fl[C::NDPC][C::LANES];                   // face fluxes
  double g[2][C::NDPC][C::G - 1][C::LANES];       // their gradients: cells 0..G-2 (Neg), 1..G-1 (Pos)
  typename std::conditional<EF::staged, typename EF::Kept, Nothing>::type kept;
  union {
    double J[2][C::NDPC][C::NDPC][C::LANES];      // flux Jacobians / jac_scale
    typename EF::Passing pass;                    // (before them)
  };
};

// The 2D or 3D Euler face's Rusanov flux and twice its two Jacobians for a
// normal along a fixed axis, by the tile's warps in four stages with a barrier
// between: euler4/5_flux and euler4/5_flux_jac with the products by the
// normal's zeros and ones left out, what the three have in common formed once,
// quotients by one divisor together, and the factors of 1/2 (exact) joined to a
// sum or left to the caller, who scales by half as much; every other rounding
// is theirs.  Two warps that each went through a whole Jacobian formed both
// states and the Roe averages twice while the others waited.
template <int FAM, int SCHEME, int AXIS> struct EulerJac {
  static constexpr int DIM = Fam<FAM>::dim, N = DIM + 2, E = DIM + 1;
  using M = IpMul;
  using Smem = JTileSmem<FAM, SCHEME>;
  Smem &sm;
  const int tx;
  const double gamma, gm1;
  __device__ EulerJac(Smem &s, int lane, double gam) : sm(s), tx(lane), gamma(gam), gm1(gam - 1.) {}

  static __device__ __forceinline__ void quot_dim(double o[DIM], const double x[DIM], double y) {
    if constexpr (DIM == 2) {
      const Quot2 q = div2_rn(x[0], x[1], y);
      o[0] = q.q0, o[1] = q.q1;
    } else {
      const Quot3 q = div3_rn(x[0], x[1], x[2], y);
      o[0] = q.q0, o[1] = q.q1, o[2] = q.q2;
    }
  }
  static __device__ __forceinline__ double square(const double v[DIM]) {
    double V2 = M::mul(v[0], v[0]);
#pragma unroll
    for (int k = 1; k < DIM; ++k) V2 = V2 + M::mul(v[k], v[k]);
    return V2;
  }
  // warps 0, 1: the left and right state; 2: r = sqrt(rho_L rho_R) and RT = sqrt(rho_R / rho_L)
  __device__ __forceinline__ void states(int w) {
    constexpr double es = 1.e-30;
    if (w < 2) {
      const double r = sm.u[w][0][tx], qE = sm.u[w][E][tx];
      double m[DIM], v[DIM];
#pragma unroll
      for (int k = 0; k < DIM; ++k) m[k] = sm.u[w][1 + k][tx];
      quot_dim(v, m, r + es);
      const double V2 = square(v), p = M::mul(gm1, fma_p2(-0.5, M::mul(r, V2), qE));
      sm.kept.H[w][tx] = div_rn(qE + p, r);
      sm.kept.V2[w][tx] = V2;
      sm.pass.p[w][tx] = p;
#pragma unroll
      for (int k = 0; k < DIM; ++k) sm.kept.v[w][k][tx] = v[k];
    } else if (w == 2) {
      const double rL = sm.u[0][0][tx], rR = sm.u[1][0][tx];
      sm.pass.r[tx] = sqrt_rn(M::mul(rR, rL));
      sm.pass.RT[tx] = sqrt_rn(div_rn(rR, rL));
    }
  }
  // warps 0, 1: the Roe averages (0: sound speed and wave speed, 1: their direction); 2, 3: one state's quotients
  __device__ __forceinline__ void averages(int w) {
    constexpr double es = 1.e-30;
    if (w < 2) {
      const double RT = sm.pass.RT[tx], T1 = 1. + RT;
      double x[DIM], v[DIM];
#pragma unroll
      for (int k = 0; k < DIM; ++k) x[k] = sm.kept.v[0][k][tx] + M::mul(RT, sm.kept.v[1][k][tx]);
      quot_dim(v, x, T1);
      const double V2 = square(v);
      if (w == 0) {
        const double H = div_rn(sm.kept.H[0][tx] + M::mul(RT, sm.kept.H[1][tx]), T1);
        const double a = sqrt_rn(M::mul(gm1, fma_p2(-0.5, V2, H)));
        sm.kept.smax[tx] = sqrt_rn(V2) + a;
        sm.pass.ga[tx] = div_rn(0.5 * gm1, a);
        sm.pass.a[tx] = a;
        sm.pass.H[tx] = H;
#pragma unroll
        for (int k = 0; k < DIM; ++k) sm.pass.v[k][tx] = v[k];
      } else {
        const double V2es = V2 + es;
        double rel[DIM];
        quot_dim(rel, v, sqrt_rn(V2es));
        sm.pass.V2es[tx] = V2es;
#pragma unroll
        for (int k = 0; k < DIM; ++k) sm.pass.rel[k][tx] = rel[k];
      }
    } else if (w < 4) {
      const int X = w - 2;
      const double aX = sqrt_rn(M::mul(gm1, fma_p2(-0.5, sm.kept.V2[X][tx], sm.kept.H[X][tx])));
      sm.pass.A2[X][tx] = div_rn(M::mul(aX, aX), gm1);
      sm.pass.inv[X][tx] = div_rn(1., sm.u[X][0][tx] + sm.pass.r[tx]);
    }
  }
  // warps 0, 1: the wave speed's derivatives with respect to a state; 2: the flux
  __device__ __forceinline__ void speeds(int w) {
    if (w < 2) {
      double v[DIM], x[DIM], rel[DIM];
#pragma unroll
      for (int k = 0; k < DIM; ++k) {
        v[k] = sm.pass.v[k][tx];
        x[k] = sm.kept.v[w][k][tx];
        rel[k] = sm.pass.rel[k][tx];
      }
      double m = M::mul(x[0] + v[0], rel[0]), VV = M::mul(x[0], v[0]);
#pragma unroll
      for (int k = 1; k < DIM; ++k) {
        m = m + M::mul(x[k] + v[k], rel[k]);
        VV = VV + M::mul(x[k], v[k]);
      }
      const double inv = sm.pass.inv[w][tx], a = sm.pass.a[tx];
      const double t = fma_p2(0.5, M::mul(gamma - 2., sm.kept.V2[w][tx]),
                              fma_p2(0.5, (sm.pass.V2es[tx] + VV) + (sm.kept.H[w][tx] - sm.pass.H[tx]),
                                     -sm.pass.A2[w][tx]));
      sm.kept.g[w][0][tx] = M::mul(inv, fma_p2(-0.5, m, M::mul(sm.pass.ga[tx], t)));
      double n[DIM], q[DIM], qE;
#pragma unroll
      for (int k = 0; k < DIM; ++k) n[k] = M::mul(gm1, v[k] + M::mul(gm1, x[k]));
      const double nE = M::mul(M::mul(inv, gamma), gm1);
      if constexpr (DIM == 2) {
        const Quot3 o = div3_rn(n[0], n[1], nE, a);
        q[0] = o.q0, q[1] = o.q1, qE = o.q2;
      } else {
        const Quot4 o = div4_rn(n[0], n[1], n[2], nE, a);
        q[0] = o.q0, q[1] = o.q1, q[2] = o.q2, qE = o.q3;
      }
#pragma unroll
      for (int k = 0; k < DIM; ++k) sm.kept.g[w][1 + k][tx] = M::mul(inv, fma_p2(-0.5, q[k], rel[k]));
      sm.kept.g[w][E][tx] = 0.5 * qE;
    } else if (w == 2) {
      const double smax = sm.kept.smax[tx];
      const double mL = M::mul(sm.u[0][0][tx], sm.kept.v[0][AXIS][tx]);
      const double mR = M::mul(sm.u[1][0][tx], sm.kept.v[1][AXIS][tx]);
      auto put = [&](int i, double fL, double fR) {
        sm.fl[i][tx] = 0.5 * (fL + fR + M::mul(smax, sm.u[0][i][tx] - sm.u[1][i][tx]));
      };
      put(0, mL, mR);
#pragma unroll
      for (int k = 0; k < DIM; ++k) {
        double fL = M::mul(mL, sm.kept.v[0][k][tx]), fR = M::mul(mR, sm.kept.v[1][k][tx]);
        if (k == AXIS) {
          fL = fL + sm.pass.p[0][tx];
          fR = fR + sm.pass.p[1][tx];
        }
        put(1 + k, fL, fR);
      }
      put(E, M::mul(mL, sm.kept.H[0][tx]), M::mul(mR, sm.kept.H[1][tx]));
    }
  }
  // warp i: row i of the two Jacobians (the same thread reads them back)
  __device__ __forceinline__ void row(int i) {
    const double dq = sm.u[0][i][tx] - sm.u[1][i][tx], smax = sm.kept.smax[tx];
#pragma unroll 1
    for (int X = 0; X < 2; ++X) {
      const double diag = X == 0 ? smax : -smax;
      double v[DIM];
#pragma unroll
      for (int k = 0; k < DIM; ++k) v[k] = sm.kept.v[X][k][tx];
      const double un = v[AXIS];
      double *o = &sm.J[X][i][0][tx];
      double tt[N];
#pragma unroll
      for (int j = 0; j < N; ++j) tt[j] = M::mul(sm.kept.g[X][j][tx], dq);
      if (i == 0) {
#pragma unroll
        for (int j = 0; j < N; ++j) o[32 * j] = j == 0 ? diag + tt[j] : (j == 1 + AXIS ? 1. + tt[j] : tt[j]);
      } else if (i == E) {
        const double H = sm.kept.H[X][tx];
        o[0] = M::mul(fma_p2(0.5, M::mul(gm1, sm.kept.V2[X][tx]), -H), un) + tt[0];
#pragma unroll
        for (int l = 0; l < DIM; ++l) {
          const double wu = M::mul(M::mul(gm1, v[l]), un);
          o[32 * (1 + l)] = (l == AXIS ? H - wu : -wu) + tt[1 + l];
        }
        o[32 * E] = (diag + M::mul(gamma, un)) + tt[E];
      } else if (i == 1 + AXIS) {
        o[0] = fma_p2(0.5, M::mul(gm1, sm.kept.V2[X][tx]), -M::mul(un, un)) + tt[0];
#pragma unroll
        for (int l = 0; l < DIM; ++l) {
          const double w = M::mul(gm1, v[l]);
          o[32 * (1 + l)] = (l == AXIS ? diag + (un - w + un) : -w) + tt[1 + l];
        }
        o[32 * E] = gm1 + tt[E];
      } else {
        const double vk = sm.kept.v[X][i - 1][tx];
        o[0] = -M::mul(vk, un) + tt[0];
#pragma unroll
        for (int l = 0; l < DIM; ++l) {
          if (l == AXIS) o[32 * (1 + l)] = vk + tt[1 + l];
          else o[32 * (1 + l)] = l == i - 1 ? (diag + un) + tt[1 + l] : tt[1 + l];
        }
        o[32 * E] = tt[E];
      }
    }
  }
};

// grid: x = lines of the box along AXIS (first other axis fastest), y and z =
// face chunks of TW faces, y fastest
template <int FAM, int SCHEME, int AXIS>
__global__ void __launch_bounds__(JTileCfg<FAM, SCHEME>::THREADS, JTileCfg<FAM, SCHEME>::MINBLOCKS)
k_jtile(Box b, MeshArgs m, Phys p, const double *__restrict__ U, const int *__restrict__ rowptr,
        double *__restrict__ V, double *__restrict__ J) {
  using F = Fam<FAM>;
  using C = JTileCfg<FAM, SCHEME>;
  constexpr int NDPC = C::NDPC, DIM = C::DIM, H = C::H, G = C::G, TW = C::TW;
  constexpr bool FIRST = AXIS == 0, LAST = AXIS == DIM - 1;
  constexpr int A1 = AXIS == 0 ? 1 : 0, A2 = AXIS == 2 ? 1 : 2;
  __shared__ JTileSmem<FAM, SCHEME> sm;
  const int tx = threadIdx.x, k = threadIdx.y;  // face or cell of the tile; its dof (row of the Jacobian)
  const int nb1 = b.hi[A1] - b.lo[A1], nb2 = b.hi[A2] - b.lo[A2];
  const int line = blockIdx.x;
  const bool lineOk = line < nb1 * nb2;
  int c[3];
  c[A1] = b.lo[A1] + (lineOk ? line % nb1 : 0);
  c[A2] = b.lo[A2] + (lineOk ? line / nb1 : 0);
  const int f0 = b.lo[AXIS] + (int)(blockIdx.y + gridDim.y * blockIdx.z) * TW;
  const int f = f0 + tx;  // this thread's face, between cells f - 1 and f
  const bool faceOk = lineOk && f <= b.hi[AXIS];
  const bool cellOk = lineOk && tx < TW && f < b.hi[AXIS];  // cell f: faces tx (left), tx + 1 (right)
  const double hinv = m.hinv[AXIS];
  auto cell_at = [&](int axis, int pos) {  // cell of this line's position with one coordinate replaced
    int cc[3] = {c[0], c[1], c[2]};
    bool mir;
    cc[axis] = map_cell(pos, b.n[axis], b.mode[axis], mir);
    return cc[0] + b.n[0] * (cc[1] + b.n[1] * cc[2]);
  };

  // ---- the face states of dof k with their gradients
  if (faceOk) {
    double q[G];
#pragma unroll
    for (int s = 0; s < G; ++s) q[s] = __ldg(U + (long)cell_at(AXIS, f - H + s) * NDPC + k);
#pragma unroll 1
    for (int side = 0; side < 2; ++side) {
      double u, g[G - 1];
      if constexpr (SCHEME == Weno5) {
        double g6[G];
        face_grad_side<SCHEME, IpMul>(side, u, g6, q);
#pragma unroll
        for (int s = 0; s < G - 1; ++s) g[s] = side == 0 ? g6[s] : g6[s + 1];
      } else if (side == 0) {
        weno3_side_grad<false, IpMul>(u, g, q[0], q[1], q[2], NoHandOver{});
      } else {
        weno3_side_grad<true, IpMul>(u, g, q[1], q[2], q[3], NoHandOver{});
      }
      sm.u[side][k][tx] = u;
#pragma unroll
      for (int s = 0; s < G - 1; ++s) sm.g[side][k][s][tx] = g[s];
    }
  }
  __syncthreads();

  // ---- flux and flux Jacobians, left and right: in stages, or by the first two warps
  if constexpr (EulerFace<FAM, SCHEME>::staged) {
    EulerJac<FAM, SCHEME, AXIS> ej(sm, tx, p.gamma);
    if (faceOk) ej.states(k);
    __syncthreads();
    if (faceOk) ej.averages(k);
    __syncthreads();
    if (faceOk) ej.speeds(k);
  } else if (k < 2 && faceOk) {
    double uN[NDPC], uP[NDPC], fl[NDPC];
#pragma unroll
    for (int d = 0; d < NDPC; ++d) {
      uN[d] = sm.u[0][d][tx];
      uP[d] = sm.u[1][d][tx];
    }
    F::template flux_jac_tile<AXIS, IpMul>(k, fl, [&](int i, int j, double x) { sm.J[k][i][j][tx] = x; }, uN, uP, p);
    if (k == 0) {
#pragma unroll
      for (int d = 0; d < NDPC; ++d) sm.fl[d][tx] = fl[d];
    }
  }

  // ---- the cell: its row position and the ranks of the blocks along AXIS in the sorted CSR row
  c[AXIS] = f;
  long gid = 0;
  int rank[1 + 2 * H];
  double u0 = 0., u1 = 0., u2 = 0.;
  if (cellOk) {
    const int own = c[0] + b.n[0] * (c[1] + b.n[1] * c[2]);
    gid = own;
    int at[2 * H];
    rank[0] = 0;
#pragma unroll
    for (int e = 0; e < 2 * H; ++e) {
      at[e] = cell_at(AXIS, f + (e < H ? e - H : e - H + 1));
      rank[0] += at[e] < own ? 1 : 0;
      rank[1 + e] = own < at[e] ? 1 : 0;
    }
#pragma unroll
    for (int e = 0; e < 2 * H; ++e)
#pragma unroll
      for (int y = 0; y < 2 * H; ++y) rank[1 + e] += at[y] < at[e] ? 1 : 0;
#pragma unroll
    for (int a = 0; a < DIM; ++a)
      if (a != AXIS) {
#pragma unroll
        for (int y = 0; y < 2 * H; ++y) {
          const int o = cell_at(a, c[a] + (y < H ? y - H : y - H + 1));
          rank[0] += o < own ? 1 : 0;
#pragma unroll
          for (int e = 0; e < 2 * H; ++e) rank[1 + e] += o < at[e] ? 1 : 0;
        }
      }
    if constexpr (FAM == Swe2d && LAST) {
      u0 = __ldg(U + gid * 3);
      u1 = __ldg(U + gid * 3 + 1);
      u2 = __ldg(U + gid * 3 + 2);
    }
  }
  __syncthreads();
  if constexpr (EulerFace<FAM, SCHEME>::staged)
    if (faceOk) EulerJac<FAM, SCHEME, AXIS>(sm, tx, p.gamma).row(k);
  double *Jrow = J;
  if (cellOk) {
    // velocity: sum over the axes in order (the first from zero), sources last
    double v = hinv * (sm.fl[k][tx] - sm.fl[k][tx + 1]);
    if (!FIRST) v = V[gid * NDPC + k] + v;
    if constexpr (FAM == Swe2d && LAST) {
      if (k == 1) v -= div_rn(p.coriolis * u2, u0);
      if (k == 2) v += div_rn(p.coriolis * u1, u0);
    }
    V[gid * NDPC + k] = v;
    Jrow = J + rowptr[gid * NDPC + k];
  }

  // ---- CSR values of row k, one column dof at a time
  const double hs = hinv * F::jac_scale;
#pragma unroll 1
  for (int j = 0; j < NDPC; ++j) {
    // the face's terms (JNeg(k,j) gNeg(j,s)) h^-1, s = 0..G-2, and (JPos(k,j) gPos(j,s)) h^-1, s = 1..G-1;
    // tN[G-1] and tP[0], products of a zero gradient, stay out of the sums
    double tN[G], tP[G];
    {
      const double ln = sm.J[0][k][j][tx], lp = sm.J[1][k][j][tx];
      double gN[G - 1], gP[G - 1];
#pragma unroll
      for (int s = 0; s < G - 1; ++s) {
        gN[s] = sm.g[0][j][s][tx];
        gP[s] = sm.g[1][j][s][tx];
      }
      bool in = ip::in_window(ln, lp, hs);
#pragma unroll
      for (int s = 0; s < G - 1; ++s) in = in && ip::in_window(gN[s], gP[s]);
      if (in) {
#pragma unroll
        for (int s = 0; s < G - 1; ++s) {
          tN[s] = ip::mul_u(ip::mul_u(ln, gN[s]), hs);
          tP[s + 1] = ip::mul_u(ip::mul_u(lp, gP[s]), hs);
        }
      } else {
#pragma unroll
        for (int s = 0; s < G - 1; ++s) {
          tN[s] = ip::mul_call(ip::mul_call(ln, gN[s]), hs);
          tP[s + 1] = ip::mul_call(ip::mul_call(lp, gP[s]), hs);
        }
        // an infinite or NaN Jacobian entry makes the left-out products NaN; they enter every sum
        // beside the other side's term of the same cell
        if (not_finite(ln)) tP[G - 1] = ln - ln;
        if (not_finite(lp)) tN[0] = lp - lp;
      }
    }
    double rN[G], rP[G];  // the right face's
#pragma unroll
    for (int s = 0; s < G - 1; ++s) {
      rN[s] = __shfl_down_sync(0xffffffffu, tN[s], 1);
      rP[s + 1] = __shfl_down_sync(0xffffffffu, tP[s + 1], 1);
    }
    if (!cellOk) continue;
    {
      // centre block: left face slot H, right face slot H - 1
      double *dst = Jrow + rank[0] * NDPC + j;
      double acc = FIRST ? tN[H] : *dst + tN[H];
      acc += tP[H];
      acc -= rN[H - 1];
      acc -= rP[H - 1];
      if constexpr (FAM == Swe2d && LAST) {
        // swe_2d_prob_class.hpp:997-1012
        if (k == 1 && j == 0) acc += div_rn(p.coriolis * u2, (u0 * u0));
        if (k == 1 && j == 2) acc += div_rn(-p.coriolis, u0);
        if (k == 2 && j == 1) acc += div_rn(p.coriolis, u0);
        if (k == 2 && j == 0) acc += div_rn(-p.coriolis * u1, (u0 * u0));
      }
      *dst = acc;
    }
    // off-centre blocks along AXIS: offset d takes the left face's slot d + H and the right face's d + H - 1
#pragma unroll
    for (int e = 0; e < 2 * H; ++e) {
      const int d = e < H ? e - H : e - H + 1;
      const int sL = d + H, sR = d + H - 1;
      double acc;
      if (sL == 0) acc = tN[0];
      else if (sL < G - 1) acc = tN[sL] + tP[sL];
      else if (sL == G - 1) acc = tP[sL];
      else acc = -rP[G - 1];
      if (sL < G) {
        if (sR >= 0) acc -= rN[sR];
        if (sR >= 1) acc -= rP[sR];
      }
      Jrow[rank[1 + e] * NDPC + j] = acc;
    }
  }
}

}  // namespace pda

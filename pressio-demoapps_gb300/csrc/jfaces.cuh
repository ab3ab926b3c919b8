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
// reconstructs dof k's two face states with their gradients, the first two
// then form the flux and its left and right Jacobian, and warp k finally takes row k of
// the Jacobian: lane by lane the face's product terms (Neg and Pos, per
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
// What bounds it: FP64 instructions, 2,850 per 2D Euler WENO5 face when one
// thread held a whole face (its gradients and Jacobians in 128 registers, 4
// warps per scheduler).  Here a face takes 1,280: terms whose factor is a
// known zero or one are left out (weno5_side_grad, euler_flux_jac2, the
// gradient's end components), exact powers of two join a sum, and the
// products run on the integer pipe, which the 32 warps per SM of the split by
// dof can hide.  512^2 WENO5 V + J 3.24 -> 1.91 ms (FP64 pipe 61 % busy, issue
// 48 %; the rest waits at the barriers around the Jacobians' two warps), 41 x
// 37 x 43 WENO3 1.35 -> 0.95 ms.  With the gradients' products on the FP64
// pipe instead: 2.20 and 0.95 ms; with 7 / 9 resident blocks of the 2D kernel
// 2.07 / 2.13 ms.
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

template <int FAM, int SCHEME> struct JTileSmem {
  using C = JTileCfg<FAM, SCHEME>;
  double u[2][C::NDPC][C::LANES];                 // face states, left- and right-biased
  double fl[C::NDPC][C::LANES];                   // face fluxes
  double g[2][C::NDPC][C::G - 1][C::LANES];       // their gradients: cells 0..G-2 (Neg), 1..G-1 (Pos)
  double J[2][C::NDPC][C::NDPC][C::LANES];        // flux Jacobians / jac_scale
};

// grid: x = lines of the box along AXIS (first other axis fastest), y = face
// chunks of TW faces
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
  const int f0 = b.lo[AXIS] + (int)blockIdx.y * TW;
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
      double u, g[G];
      face_grad_side<SCHEME, IpMul>(side, u, g, q);
      sm.u[side][k][tx] = u;
#pragma unroll
      for (int s = 0; s < G - 1; ++s) sm.g[side][k][s][tx] = side == 0 ? g[s] : g[s + 1];
    }
  }
  __syncthreads();

  // ---- flux and flux Jacobians, left and right, by the first two warps
  if (k < 2 && faceOk) {
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

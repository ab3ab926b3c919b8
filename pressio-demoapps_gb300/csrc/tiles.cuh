// Tiled face kernels for WENO3 / WENO5 on natural-order full meshes.
//
// The FP64 pipe bounds this path on GB300, so the kernels minimise FP64
// operations while keeping every value bit-identical to the reference:
//  * products by powers of two are fused into the following sum (w5_* in
//    numerics.cuh: the product is exact, so one rounding equals two);
//  * each face is computed once (the reference computes it from both cells);
//  * the smoothness indicators of a cell triple (WENO5) or pair (WENO3) and
//    the alpha terms built from them enter up to three one-sided
//    reconstructions of neighbouring faces with identical expression trees
//    (impl/weno5.hpp:112-178, impl/weno3.hpp:82-131), so they are computed
//    once per cell into shared memory and reused;
//  * the reference's divisions and square roots, its products by small
//    integers, 1/2 and constants, and the products of two variables run on
//    the integer pipe (fp64_intpipe.cuh), bit for bit; the quarter of a
//    square is exact and joins the following sum;
//  * an FP64 instruction takes the FP64 pipe 64 issue slots, an integer
//    product about 30, so the two pipes share the products until both are
//    about equally loaded: 166 FP64 instructions per 2D Euler WENO5 face
//    (271 with all products of two variables on the FP64 pipe), FP64 pipe
//    74 % busy, ALU pipe 61 %, issue slots 64 %.  The operands of a group of
//    products are checked together, which leaves one basic block in which
//    they overlap.  1024^2: 0.40 ms per face pass (0.634 ms before; 0.58 with
//    the faster division alone, 0.425 with the weights' products moved but
//    checked one by one and the flux's on the FP64 pipe);
//  * the code stays small enough for the instruction cache: the per-dof
//    loops of the cell and face phases are not unrolled (face states kept in
//    registers by predicated moves) and every division and square root is
//    an out-of-line call.  Fully unrolled with inline divisions the kernel
//    is a straight line of about 10^4 instructions per thread, and
//    instruction-fetch stalls were its largest stall reason;
//  * boundary faces of the mirror-type boundary conditions (2D Neumann and
//    slip wall, whose ghost layers are exact mirror images,
//    euler_2d_ghost_filler_neumann.hpp:101-276,
//    swe_2d_ghost_filler_inviscid_wall.hpp:99-278) are computed in the same
//    pass by mirrored loads, so no per-row boundary kernel is needed.
//
// Block: LANES threads along the face axis x NR lines; a block produces TW
// faces of each of its NR lines (TW = LANES - 3 for WENO5, LANES - 2 for
// WENO3).  Small meshes take a warp per dof instead of a loop over the dofs,
// and two warps form the two states' halves of the flux (SPLIT): a block's
// chain is then a third as long, at the price of two barriers.  Loads along y/z are strided gathers of whole 32-40 byte cells, so
// no sector is fetched for nothing.
#pragma once

#include "kernels.cuh"

namespace pda {

// v[d] = x for a runtime d, with v kept in registers (predicated moves)
template <int N>
__device__ __forceinline__ void set_dof(double (&v)[N], int d, double x) {
#pragma unroll
  for (int k = 0; k < N; ++k)
    if (k == d) v[k] = x;
}

// K0 x0 and K1 x1 with one check
template <int K0, int K1>
__device__ __forceinline__ void mul_k_all(double x0, double x1, double &y0, double &y1) {
  if (ip::in_window(x0, x1)) {
    y0 = ip::mul_small_u<K0>(x0);
    y1 = ip::mul_small_u<K1>(x1);
  } else {
    y0 = ip::mul_call((double)K0, x0);
    y1 = ip::mul_call((double)K1, x1);
  }
}
// one weighted candidate on the FP64 pipe: (alpha s) (P / 6)
static __device__ __noinline__ double w5_term_call(double alpha, double s, double P) {
  if (ip::in_window(alpha, s) && (ip::hi_word(P) << 1 | ip::lo_word(P)) == 0) return P;  // alpha, s > 0
  return (alpha * s) * (P * (1. / 6.));
}

static __device__ __noinline__ double w3_term_call(double alpha, double s, double P) {
  if (ip::in_window(alpha, s) && (ip::hi_word(P) << 1 | ip::lo_word(P)) == 0) return P;
  return (alpha * s) * (P * 0.5);
}

template <int SCHEME, int LANES_ = 64> struct TileCfg;
template <int LANES_> struct TileCfg<Weno5, LANES_> {
  static constexpr int H = 3, LANES = LANES_, TW = LANES - 3, NCELL = TW + 5, NA = 5;
};
template <int LANES_> struct TileCfg<Weno3, LANES_> {
  static constexpr int H = 2, LANES = LANES_, TW = LANES - 2, NCELL = TW + 3, NA = 2;
};

// shared memory of one tile: the cells of NR lines and their alpha terms; with
// a warp per dof (SPLIT) also the face states and the two halves of the flux
template <int FAM, int LANES> struct FaceTileSplit {
  double u[2][Fam<FAM>::ndpc][LANES];
  typename Fam<FAM>::Side side[2][LANES];
};
struct FaceTileWhole {};
template <int FAM, int SCHEME, int NR, int LANES, bool SPLIT = false> struct FaceTileSmem {
  using C = TileCfg<SCHEME, LANES>;
  double sU[NR][Fam<FAM>::ndpc][C::NCELL + 1];
  double sA[NR][Fam<FAM>::ndpc][C::NA][LANES];
  typename std::conditional<SPLIT, FaceTileSplit<FAM, LANES>, FaceTileWhole>::type sp;
};

// One tile: lines lineGroup*NR .. +NR-1 of the box (the lines run along AXIS,
// numbered with the first other axis fastest), faces chunk*TW .. +TW-1 of
// each line.  Called by every thread of a LANES x NR block; SPLIT: of a LANES x
// NR x ndpc block, a thread's z its dof.
template <int FAM, int SCHEME, int AXIS, int NR, int LANES, bool SPLIT = false>
__device__ __forceinline__ void face_tile(FaceTileSmem<FAM, SCHEME, NR, LANES, SPLIT> &sm, const Box &b, const Phys &p,
                                          const double *__restrict__ U, double *__restrict__ Fout,
                                          long lineGroup, int chunk) {
  using F = Fam<FAM>;
  using C = TileCfg<SCHEME, LANES>;
  constexpr int NDPC = F::ndpc, TW = C::TW, NCELL = C::NCELL, H = C::H;
  constexpr int A1 = AXIS == 0 ? 1 : 0, A2 = AXIS == 2 ? 1 : 2;  // the two other axes
  auto &sU = sm.sU;
  auto &sA = sm.sA;

  const int tx = threadIdx.x, ty = threadIdx.y;
  const int dz = SPLIT ? (int)threadIdx.z : 0;  // this thread's first dof, and the step to its next
  constexpr int DZ = SPLIT ? NDPC : 1;
  const int nb1 = b.hi[A1] - b.lo[A1], nb2 = b.hi[A2] - b.lo[A2];
  const int nf = b.hi[AXIS] - b.lo[AXIS] + 1;
  const long line = lineGroup * NR + ty;
  const bool lineOk = line < (long)nb1 * nb2;
  const int c1 = lineOk ? b.lo[A1] + (int)(line % nb1) : b.lo[A1];
  const int c2 = lineOk ? b.lo[A2] + (int)(line / nb1) : b.lo[A2];
  const int f0 = b.lo[AXIS] + chunk * TW;  // first face of the tile
  long stride[3];
  stride[0] = 1;
  stride[1] = b.n[0];
  stride[2] = (long)b.n[0] * b.n[1];
  const long base = (long)c1 * stride[A1] + (long)c2 * stride[A2];

  // ---- phase A: cells f0-H .. f0+TW+H-2 of this line into shared memory
  for (int k = tx; k < NCELL; k += LANES) {
    bool mir;
    const int c = map_cell(f0 - H + k, b.n[AXIS], b.mode[AXIS], mir);
    const double *src = U + (base + (long)c * stride[AXIS]) * NDPC;
#pragma unroll
    for (int e = 0; e < NDPC; e += DZ) {
      const int d = e + dz;
      double v = __ldg(src + d);
      if (mir && d == b.reflect[AXIS]) v = -v;
      sU[ty][d][k] = v;
    }
  }
  __syncthreads();

  // ---- phase B: per-cell alpha terms
  constexpr double epsilon = 1e-6;
  if constexpr (SCHEME == Weno5) {
    // center c = f0 - 2 + tx uses cells c-1, c, c+1 = sU[tx .. tx+2]
    constexpr double oneOvten = 1. / 10., threeOvten = 3. / 10., sixOvten = 6. / 10.,
                     thirteenOvtwelve = 13. / 12.;
    if (tx + 2 < NCELL) {
#pragma unroll 1
      for (int d = dz; d < NDPC; d += DZ) {
        const double a = sU[ty][d][tx], m = sU[ty][d][tx + 1], c = sU[ty][d][tx + 2];
        double a3, c3;
        mul_k_all<3, 3>(a, c, a3, c3);
        const double X = w5_curv(a, m, c);
        const double YL = fma_p2(-4., m, a) + c3;  // w5_slopeL
        const double YC = a - c;
        const double YR = fma_p2(-4., m, a3) + c;  // w5_slopeR
        double D, sL, sC, sR;
        if (ip::in_window(X, YL, YC, YR)) {
          D = ip::mul_u(ip::mul_const_u(X, thirteenOvtwelve), X);
          sL = ip::square_u(YL);
          sC = ip::square_u(YC);
          sR = ip::square_u(YR);
        } else {
          D = ip::mul_call(ip::mul_call(thirteenOvtwelve, X), X);
          sL = ip::mul_call(YL, YL);
          sC = ip::mul_call(YC, YC);
          sR = ip::mul_call(YR, YR);
        }
        const double BL = fma_p2(0.25, sL, D);
        const double BC = fma_p2(0.25, sC, D);
        const double BR = fma_p2(0.25, sR, D);
        double eL, eC, eR;
        if (ip::in_window(BL, BC, BR)) {
          eL = ip::mul_const_u(BL, 2. * epsilon);
          eC = ip::mul_const_u(BC, 2. * epsilon);
          eR = ip::mul_const_u(BR, 2. * epsilon);
          sL = ip::square_u(BL);
          sC = ip::square_u(BC);
          sR = ip::square_u(BR);
        } else {
          eL = ip::mul_call(BL, 2. * epsilon);
          eC = ip::mul_call(BC, 2. * epsilon);
          eR = ip::mul_call(BR, 2. * epsilon);
          sL = ip::mul_call(BL, BL);
          sC = ip::mul_call(BC, BC);
          sR = ip::mul_call(BR, BR);
        }
        const double dL = epsilon * epsilon + eL + sL;
        const double dC = epsilon * epsilon + eC + sC;
        const double dR = epsilon * epsilon + eR + sR;
        const Quot2 aL = div2_rn(oneOvten, threeOvten, dL);
        const Quot2 aR = div2_rn(threeOvten, oneOvten, dR);
        sA[ty][d][0][tx] = aL.q0;                 // uNeg alpha0 of face c+1+1/2
        sA[ty][d][1][tx] = aL.q1;                 // uPos alpha0 of face c+1/2
        sA[ty][d][2][tx] = div_rn(sixOvten, dC);  // uNeg alpha1 of face c+1/2, uPos alpha1 of face c-1/2
        sA[ty][d][3][tx] = aR.q0;                 // uNeg alpha2 of face c-1/2
        sA[ty][d][4][tx] = aR.q1;                 // uPos alpha2 of face c-2+1/2
      }
    }
  } else {
    // pair k = (f0 - 2 + tx, f0 - 1 + tx) uses cells sU[tx], sU[tx+1]
    constexpr double two = 2., oneOvthree = 1. / 3., twoOvthree = 2. / 3.;
    if (tx + 1 < NCELL) {
#pragma unroll 1
      for (int d = dz; d < NDPC; d += DZ) {
        const double a = sU[ty][d][tx], c = sU[ty][d][tx + 1];
        const double X = a - c;
        double B, e, q;
        if (ip::in_window(X)) {
          B = ip::square_u(X);
        } else {
          B = ip::mul_call(X, X);
        }
        if (ip::in_window(B)) {
          e = ip::mul_const_u(B, two * epsilon);
          q = ip::square_u(B);
        } else {
          e = ip::mul_call(B, two * epsilon);
          q = ip::mul_call(B, B);
        }
        const double den = epsilon * epsilon + e + q;
        sA[ty][d][0][tx] = div_rn(oneOvthree, den);
        sA[ty][d][1][tx] = div_rn(twoOvthree, den);
      }
    }
  }
  __syncthreads();

  // ---- phase C: face f = f0 + tx between cells f-1 and f
  const int f = f0 + tx;
  const bool faceOk = lineOk && tx < TW && f <= b.hi[AXIS];
  if (!SPLIT && !faceOk) return;
  double uN[NDPC], uP[NDPC];
  auto put_states = [&](int d, double l, double r) {
    if constexpr (SPLIT) {
      sm.sp.u[0][d][tx] = l;
      sm.sp.u[1][d][tx] = r;
    } else {
      set_dof(uN, d, l);
      set_dof(uP, d, r);
    }
  };
  if (SPLIT && !faceOk) {
    // (no face; the block's barriers below are for all)
  } else if constexpr (SCHEME == Weno5) {
    constexpr double oneOvsix = 1. / 6.;
#pragma unroll 1
    for (int d = dz; d < NDPC; d += DZ) {
      // left cell i = f-1: cells i-2..i+3 = sU[tx .. tx+5]; centers i-1..i+2 = sA[.][tx .. tx+3]
      const double qim2 = sU[ty][d][tx], qim1 = sU[ty][d][tx + 1], qi = sU[ty][d][tx + 2];
      const double qip1 = sU[ty][d][tx + 3], qip2 = sU[ty][d][tx + 4], qip3 = sU[ty][d][tx + 5];
      double k7a, k11a, k5a, k5b, k11b, k7b;
      if (ip::in_window(qim1, qi, qip1, qip2)) {
        k7a = ip::mul_small_u<7>(qim1);
        k11a = ip::mul_small_u<11>(qi);
        k5a = ip::mul_small_u<5>(qi);
        k5b = ip::mul_small_u<5>(qip1);
        k11b = ip::mul_small_u<11>(qip1);
        k7b = ip::mul_small_u<7>(qip2);
      } else {
        k7a = ip::mul_call(7., qim1);
        k11a = ip::mul_call(11., qi);
        k5a = ip::mul_call(5., qi);
        k5b = ip::mul_call(5., qip1);
        k11b = ip::mul_call(11., qip1);
        k7b = ip::mul_call(7., qip2);
      }
      // 6 x the candidate polynomials: w5_pFarL, w5_pMidL, w5_pMidR, w5_pFarR
      const double P0 = fma_p2(2., qim2, -k7a) + k11a;
      const double P1 = fma_p2(2., qip1, -qim1 + k5a);
      const double P2 = fma_p2(2., qi, k5b) - qip2;
      const double P3 = fma_p2(2., qip3, k11b - k7b);
      const double n0 = sA[ty][d][0][tx], n1 = sA[ty][d][2][tx + 1], n2 = sA[ty][d][3][tx + 2];
      const double r0 = sA[ty][d][1][tx + 1], r1 = sA[ty][d][2][tx + 2], r2 = sA[ty][d][4][tx + 3];
      const double sn = div_rn(1., (n0 + n1 + n2)), sp = div_rn(1., (r0 + r1 + r2));
      double t[6];
      if (ip::in_window(P0, P1, P2, P3, n0, n1, n2, r0, r1, r2, sn, sp)) {
        const double p0 = ip::mul_const_u(P0, oneOvsix), p1 = ip::mul_const_u(P1, oneOvsix);
        const double p2 = ip::mul_const_u(P2, oneOvsix), p3 = ip::mul_const_u(P3, oneOvsix);
        t[0] = ip::mul_u(ip::mul_u(n0, sn), p0);
        t[1] = ip::mul_u(ip::mul_u(n1, sn), p1);
        t[2] = ip::mul_u(ip::mul_u(n2, sn), p2);
        t[3] = ip::mul_u(ip::mul_u(r0, sp), p1);
        t[4] = ip::mul_u(ip::mul_u(r1, sp), p2);
        t[5] = ip::mul_u(ip::mul_u(r2, sp), p3);
      } else {
        t[0] = w5_term_call(n0, sn, P0);
        t[1] = w5_term_call(n1, sn, P1);
        t[2] = w5_term_call(n2, sn, P2);
        t[3] = w5_term_call(r0, sp, P1);
        t[4] = w5_term_call(r1, sp, P2);
        t[5] = w5_term_call(r2, sp, P3);
      }
      put_states(d, t[0] + t[1] + t[2], t[3] + t[4] + t[5]);
    }
  } else {
    // p0 = (-q_{i-1} + 3 q_i) / 2, p1 = (q_i + q_{i+1}) / 2, p2 = (3 q_{i+1} - q_{i+2}) / 2
#pragma unroll 1
    for (int d = dz; d < NDPC; d += DZ) {
      // left cell i = f-1: cells i-1..i+2 = sU[tx .. tx+3]; pairs i-1, i, i+1 = sA[.][tx .. tx+2]
      const double qim1 = sU[ty][d][tx], qi = sU[ty][d][tx + 1], qip1 = sU[ty][d][tx + 2],
                   qip2 = sU[ty][d][tx + 3];
      double k3a, k3b;
      mul_k_all<3, 3>(qi, qip1, k3a, k3b);
      // 2 x the candidate polynomials
      const double P0 = -qim1 + k3a, P1 = qi + qip1, P2 = k3b - qip2;
      const double n0 = sA[ty][d][0][tx], n1 = sA[ty][d][1][tx + 1];
      const double r0 = n1, r1 = sA[ty][d][0][tx + 2];
      const double sn = div_rn(1., (n0 + n1)), sp = div_rn(1., (r0 + r1));
      double t[4];
      if (ip::in_window(P0, P1, P2, n0, n1, r1, sn, sp)) {
        t[0] = ip::mul_u(ip::mul_u(n0, sn), ip::half_u(P0));
        t[1] = ip::mul_u(ip::mul_u(n1, sn), ip::half_u(P1));
        t[2] = ip::mul_u(ip::mul_u(r0, sp), ip::half_u(P1));
        t[3] = ip::mul_u(ip::mul_u(r1, sp), ip::half_u(P2));
      } else {
        t[0] = w3_term_call(n0, sn, P0);
        t[1] = w3_term_call(n1, sn, P1);
        t[2] = w3_term_call(r0, sp, P1);
        t[3] = w3_term_call(r1, sp, P2);
      }
      put_states(d, t[0] + t[1], t[2] + t[3]);
    }
  }
  double fl[NDPC];
  if constexpr (SPLIT) {
    // the flux in two halves, then their combination
    __syncthreads();
    if (dz < 2 && faceOk) {
      double q[NDPC];
#pragma unroll
      for (int d = 0; d < NDPC; ++d) q[d] = sm.sp.u[dz][d][tx];
      F::template flux_side<AXIS>(sm.sp.side[dz][tx], q, p);
    }
    __syncthreads();
    if (dz != 0 || !faceOk) return;
#pragma unroll
    for (int d = 0; d < NDPC; ++d) {
      uN[d] = sm.sp.u[0][d][tx];
      uP[d] = sm.sp.u[1][d][tx];
    }
    F::template flux_combine<AXIS>(fl, uN, uP, sm.sp.side[0][tx], sm.sp.side[1][tx], p);
  } else {
    F::template flux<AXIS, false, true>(fl, uN, uP, p);
  }
  // output layout of k_struct_faces: face axis index fastest within its line
  // ordering [A2][A1][face] for AXIS=0, [k][face][i] for AXIS=1, [face][j][i] for AXIS=2
  const int fi = f - b.lo[AXIS];
  const int i1 = c1 - b.lo[A1], i2 = c2 - b.lo[A2];
  long o;
  if (AXIS == 0) o = fi + (long)nf * (i1 + (long)nb1 * i2);
  else if (AXIS == 1) o = i1 + (long)nb1 * (fi + (long)nf * i2);
  else o = i1 + (long)nb1 * (i2 + (long)nb2 * fi);
#pragma unroll
  for (int d = 0; d < NDPC; ++d) Fout[o * NDPC + d] = fl[d];
}

// Resident blocks per SM the register allocation must allow: 32 warps per SM,
// or fewer where the tile's shared memory admits fewer blocks (3D: 7), so the
// cap never forces spills that buy no occupancy.  2D Euler, 1024^2, whole
// velocity: 0.848 ms with 8 blocks of 128 threads (64 registers), 0.857 with
// 7 (72), 0.868 with 6 (80), 0.910 with 5.
template <int FAM, int SCHEME, int NR, int LANES, bool SPLIT = false>
struct FaceTileMinBlocks {
  static constexpr int kSmemPerSM = 228 * 1024, kReservedPerBlock = 1024;
  static constexpr int threads = LANES * NR * (SPLIT ? Fam<FAM>::ndpc : 1);
  static constexpr int bySmem =
      kSmemPerSM / ((int)sizeof(FaceTileSmem<FAM, SCHEME, NR, LANES, SPLIT>) + kReservedPerBlock);
  static constexpr int byWarps = 1024 / threads;
  static constexpr int value = bySmem < byWarps ? (bySmem > 0 ? bySmem : 1) : byWarps;
};

// grid: x = line groups of NR lines, y = face chunks of TW faces
template <int FAM, int SCHEME, int AXIS, int NR, int LANES, bool SPLIT = false>
__global__ void __launch_bounds__((FaceTileMinBlocks<FAM, SCHEME, NR, LANES, SPLIT>::threads),
                                  (FaceTileMinBlocks<FAM, SCHEME, NR, LANES, SPLIT>::value))
k_faces_tile(Box b, Phys p, const double *__restrict__ U, double *__restrict__ Fout) {
  __shared__ FaceTileSmem<FAM, SCHEME, NR, LANES, SPLIT> sm;
  face_tile<FAM, SCHEME, AXIS, NR, LANES, SPLIT>(sm, b, p, U, Fout, (long)blockIdx.x, (int)blockIdx.y);
}

}  // namespace pda

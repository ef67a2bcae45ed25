// trid_solve.cuh -- the symmetric tridiagonal solvers of the many-CTA eigensolver (syevt_cluster.cu,
// syevt_mid.cu) and of the Ritz step (vec_kernels.cu): the Sturm count with lagged rescaling and the
// inverse iteration of one eigenvector in two solves. The one-CTA eigensolvers keep the forms of
// syevt_common.cuh, whose order of operations fixed_order solves are held to.
#pragma once
#include "syevt_common.cuh"

namespace dmrg {
namespace {

// Number of eigenvalues of T(d,e) strictly below x: sign changes of the leading minors
// D_j = (d_j - x) D_{j-1} - e_{j-1}^2 D_{j-2}. The carried pair is (D_{j-1}, t_j) with
// t_j = -e_{j-1}^2 D_{j-2}: each step is one FMA for D_j and one product t_{j+1} from D_{j-1}, two
// independent operations, so only the FMA is on the dependent chain. Signs are counted on the high
// words (an isolated exact zero gives the same count with either sign). After every 8 steps the
// pair is rescaled by the power of two that brought its larger magnitude after the fourth of them
// into [1, 2): the factor is ready before the chain needs it. The pair goes 12 steps without a
// rescaling, each of which may multiply it by the norm of T, so T has to come with a norm near 1
// (unit_scale): at 1e-26 the pair would underflow and never recover. With blocks of 85, 70 and 40
// rows in one launch the lagged rescaling and the bit counts took 108 to 100 us.
__device__ int sturm_lagged(const double* __restrict__ d, const double* __restrict__ e2, int n,
                           double x) {
  double D = d[0] - x;
  double t = -e2[0];                      // t_1 = -e_0^2 D_{-1}, D_{-1} = 1
  int hp = __double2hiint(D);
  unsigned c = unsigned(hp) >> 31;
  int j = 1;
  for (; j + 8 <= n; j += 8) {
    double dx[8], ee[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      dx[q] = d[j + q] - x;
      ee[q] = e2[j + q];
    }
    double sc = 1.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const double Dn = fma(dx[q], D, t);
      t = -ee[q] * D;
      D = Dn;
      const int h = __double2hiint(Dn);
      c += unsigned(h ^ hp) >> 31;
      hp = h;
      if (q == 3) {
        const int fld = max(h & 0x7fffffff, __double2hiint(t) & 0x7fffffff) >> 20;
        if (fld != 0 && fld != 0x7ff) sc = __hiloint2double((1023 - min(fld - 1023, 1022)) << 20, 0);
      }
    }
    D *= sc;
    t *= sc;
  }
  for (; j < n; ++j) {
    const double Dn = fma(d[j] - x, D, t);
    t = -e2[j] * D;
    D = Dn;
    const int h = __double2hiint(Dn);
    c += unsigned(h ^ hp) >> 31;
    hp = h;
  }
  return int(c);
}

// LU factors of one solver thread in shared memory: element k at [k * stride] (threads
// interleaved, so that neighbouring threads touch neighbouring words). U has two superdiagonals;
// the second is e[k+1] where rows were swapped and zero elsewhere, so it is not stored.
struct LeanSlot {
  double *u0, *u1, *l;     // reciprocal pivots, first superdiagonal, multipliers
  int* piv;
  int stride;
};

// One thread: the vector of (T - lam I)^{-1} applied twice to the pseudo-random start vector of
// column col, normalised, into z (element r at z[r * zs]). With lam good to the last bits the
// first solve leaves other eigenvectors at ~1e-16 ||T|| / gap and the second squares that; a third
// only turns the vectors of equal eigenvalues towards each other (the worst residual of degenerate
// test blocks fell from 5e-13 to 3e-14 without it). The factorisation carries the first forward
// solve along and takes one reciprocal a step, for either pivot; the solves run in groups of 8
// steps whose loads are issued first; the normalisation is applied in the next pass. What bounds it
// is the chain of dependent steps: ~115 cycles for a factorisation step (the reciprocal), ~25 for a
// solve step.
__device__ void lean_inverse_iteration(const double* __restrict__ d, const double* __restrict__ e,
                                       int n, double lam, double* z, int zs, int col, double tn,
                                       LeanSlot f) {
  const int S = f.stride;
  const double pert = 2.2e-16 * tn;
  double dk = d[0] - lam, ek = n > 1 ? e[0] : 0.0;
  double zk = prand(0, col);
#pragma unroll 4
  for (int k = 0; k + 1 < n; ++k) {
    const double sub = e[k];                  // T(k+1, k)
    const double dn = d[k + 1] - lam;
    const double en = (k + 2 < n) ? e[k + 1] : 0.0;
    const bool sw = fabs(dk) < fabs(sub);     // swap rows k and k+1
    const double r = 1.0 / (sw ? sub : (dk == 0.0 ? pert : dk));
    const double lk = (sw ? dk : sub) * r;
    const double u1 = sw ? dn : ek;
    f.u0[k * S] = r;
    f.u1[k * S] = u1;
    f.l[k * S] = lk;
    f.piv[k * S] = sw;
    dk = fma(-lk, u1, sw ? ek : dn);
    ek = sw ? -lk * en : en;
    const double zr = prand(k + 1, col);
    const double zt = sw ? zr : zk;           // row k of P z
    z[k * zs] = zt;
    zk = fma(-lk, zt, sw ? zk : zr);
  }
  f.u0[(n - 1) * S] = 1.0 / ((dk == 0.0) ? pert : dk);
  f.u1[(n - 1) * S] = 0.0;
  f.piv[(n - 1) * S] = 0;
  z[(n - 1) * zs] = zk;
  double inv = 1.0;
  for (int it = 0; it < 2; ++it) {
    if (it > 0) {
      // solve P L y = inv z; z[k] is carried in a register. Loads of a group precede its stores,
      // and every store goes below the indices still to be loaded.
      zk = inv * z[0];
      int k = 0;
      for (; k + 8 < n; k += 8) {
        double zz[8], ll[8];
        int pp[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          zz[q] = inv * z[(k + 1 + q) * zs];
          ll[q] = f.l[(k + q) * S];
          pp[q] = f.piv[(k + q) * S];
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const double zt = pp[q] ? zz[q] : zk;
          z[(k + q) * zs] = zt;
          zk = fma(-ll[q], zt, pp[q] ? zk : zz[q]);
        }
      }
      for (; k + 1 < n; ++k) {
        const double zn = inv * z[(k + 1) * zs];
        const bool sw = f.piv[k * S];
        const double zt = sw ? zn : zk;
        z[k * zs] = zt;
        zk = fma(-f.l[k * S], zt, sw ? zk : zn);
      }
      z[(n - 1) * zs] = zk;
    }
    // solve U x = y (x[k+1], x[k+2] carried in registers)
    double x1 = 0.0, x2 = 0.0;
    int k = n - 1;
    for (; k >= 7; k -= 8) {
      double zz[8], a0[8], a1[8], a2[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        zz[q] = z[(k - q) * zs];
        a0[q] = f.u0[(k - q) * S];
        a1[q] = f.u1[(k - q) * S];
        a2[q] = f.piv[(k - q) * S] && k - q + 2 < n ? e[k - q + 1] : 0.0;
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const double xk = fma(-a2[q], x2, fma(-a1[q], x1, zz[q])) * a0[q];
        z[(k - q) * zs] = xk;
        x2 = x1;
        x1 = xk;
      }
    }
    for (; k >= 0; --k) {
      const double a2 = f.piv[k * S] && k + 2 < n ? e[k + 1] : 0.0;
      const double xk = fma(-a2, x2, fma(-f.u1[k * S], x1, z[k * zs])) * f.u0[k * S];
      z[k * zs] = xk;
      x2 = x1;
      x1 = xk;
    }
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int i = 0;
#pragma unroll 2
    for (; i + 4 <= n; i += 4) {
      s0 = fma(z[i * zs], z[i * zs], s0);
      s1 = fma(z[(i + 1) * zs], z[(i + 1) * zs], s1);
      s2 = fma(z[(i + 2) * zs], z[(i + 2) * zs], s2);
      s3 = fma(z[(i + 3) * zs], z[(i + 3) * zs], s3);
    }
    for (; i < n; ++i) s0 = fma(z[i * zs], z[i * zs], s0);
    const double nr = sqrt((s0 + s1) + (s2 + s3));
    if (nr == 0.0) {
      for (int r = 0; r < n; ++r) z[r * zs] = prand(r, col + 7 * (it + 1));
      inv = 1.0;
    } else {
      inv = 1.0 / nr;
    }
  }
#pragma unroll 8
  for (int r = 0; r < n; ++r) z[r * zs] *= inv;
}

}  // namespace
}  // namespace dmrg

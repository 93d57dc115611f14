// Coefficients of the strong-form step (step.cuh, step_visc.cuh) from the caller's star matrices, flux
// solvers and connectivity: per element U, star rows, anelastic coefficients and V rows (FacL), and the
// gather table.
#pragma once
#include "step_visc.cuh"

namespace edge_b200 {

// Nine lanes share a face, lane a its row a of the 9 x 9 solvers; what they exchange goes through this
// (a thread per face keeps its matrices in local memory: 6.2 ms for 72,864 elements, this one 1.34, each with
// its launch and the check read back).
struct FaceTeam {
  double S[9][9], N[9][9], U[9][3], V0[9][3], red[9];
};
constexpr int kTeams = 3;          // per warp
constexpr int kBuildWarps = 4;     // per block
// Share of the flux solvers (of a scaled row, of the own side's largest entry) that the three directions
// may leave out, and that the strong form then drops. Godunov solvers leave rounding: at most 3e-15 over
// layered, jittered and strongly contrasting media (30 in vp), free surfaces and outflow. FP64 takes
// thirty times that; in FP32 the solvers themselves are rounded to 6e-8.
template <typename T>
constexpr double rankTol() {
  return sizeof(T) == 8 ? 1e-13 : 1e-9;
}

__device__ __forceinline__ double teamMax(FaceTeam &t, int a, double v, int from, int to) {
  __syncwarp();
  t.red[a] = v;
  __syncwarp();
  double m = 0;
#pragma unroll
  for (int i = 0; i < 9; i++)
    if (i >= from && i < to) m = fmax(m, t.red[i]);
  return m;
}

// Row and column scales of a flux solver, one for the stresses and one for the velocities (as
// inputs and as outputs they differ by the moduli and impedances): M_ij / (r_i c_j) has entries of
// at most one. (A scale per row or column would blow up the rounding of those that vanish; the
// scales of a face without a neighbour are those of fsE[0], before a free surface's velocity
// columns cancel.)
struct Scales {
  double rS, rV, cS, cV;
  __device__ __forceinline__ double r(int i) const { return i < 6 ? rS : rV; }
  __device__ __forceinline__ double c(int j) const { return j < 6 ? cS : cV; }
};
__device__ __forceinline__ Scales scales(FaceTeam &t, int a, const double (&M)[9]) {
  double mS = 0, mV = 0;
#pragma unroll
  for (int j = 0; j < 9; j++) (j < 6 ? mS : mV) = fmax(j < 6 ? mS : mV, fabs(M[j]));
  Scales s;
  s.rS = teamMax(t, a, fmax(mS, mV), 0, 6);
  s.rV = teamMax(t, a, fmax(mS, mV), 6, 9);
  if (!(s.rS > 0)) s.rS = 1.0;
  if (!(s.rV > 0)) s.rV = 1.0;
  s.cS = teamMax(t, a, mS / s.r(a), 0, 9);
  s.cV = teamMax(t, a, mV / s.r(a), 0, 9);
  if (!(s.cS > 0)) s.cS = 1.0;
  if (!(s.cV > 0)) s.cV = 1.0;
  return s;
}

// Orthonormal basis Q (3 x 9, in every lane) of the rows of the scaled solver, this lane's row S, by
// Gram-Schmidt with pivoting, each direction orthogonalised twice; a direction without a row left is
// zero. Returns what this lane's row keeps outside Q (squared norm).
__device__ __forceinline__ double rowBasis(FaceTeam &t, int a, double (&S)[9], double (&Q)[3][9]) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double n2 = 0;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 9; j++) {
      n2 += S[j] * S[j];
      t.S[a][j] = S[j];
    }
    t.red[a] = n2;
    __syncwarp();
    int piv = 0;
    double best = 0;
#pragma unroll
    for (int i = 0; i < 9; i++)
      if (t.red[i] > best) {
        best = t.red[i];
        piv = i;
      }
    double v[9];
#pragma unroll
    for (int j = 0; j < 9; j++) v[j] = best > 0 ? t.S[piv][j] : 0.0;
#pragma unroll
    for (int pass = 0; pass < 2; pass++)
#pragma unroll
      for (int kk = 0; kk < k; kk++) {
        double d = 0;
#pragma unroll
        for (int j = 0; j < 9; j++) d += v[j] * Q[kk][j];
#pragma unroll
        for (int j = 0; j < 9; j++) v[j] -= d * Q[kk][j];
      }
    double l2 = 0;
#pragma unroll
    for (int j = 0; j < 9; j++) l2 += v[j] * v[j];
    // rows of unit scale: what rounding leaves of a dependent row is no direction
    const double inv = l2 > 1e-24 ? 1.0 / sqrt(l2) : 0.0;
    double d = 0;
#pragma unroll
    for (int j = 0; j < 9; j++) {
      Q[k][j] = v[j] * inv;
      d += S[j] * Q[k][j];
    }
#pragma unroll
    for (int j = 0; j < 9; j++) S[j] -= d * Q[k][j];
  }
  double res = 0;
#pragma unroll
  for (int j = 0; j < 9; j++) res += S[j] * S[j];
  return res;
}

// U = A^T R of the team's U (9 x 3): three orthonormal columns A and the triangle R; a column without
// anything left is zero
__device__ __forceinline__ void qrU(const FaceTeam &t, double (&A)[3][9], double (&Rm)[3][3]) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double v[9];
#pragma unroll
    for (int i = 0; i < 9; i++) v[i] = t.U[i][k];
#pragma unroll
    for (int kk = 0; kk < 3; kk++) Rm[kk][k] = 0;
#pragma unroll
    for (int pass = 0; pass < 2; pass++)
#pragma unroll
      for (int kk = 0; kk < k; kk++) {
        double d = 0;
#pragma unroll
        for (int i = 0; i < 9; i++) d += v[i] * A[kk][i];
        Rm[kk][k] += d;
#pragma unroll
        for (int i = 0; i < 9; i++) v[i] -= d * A[kk][i];
      }
    double l2 = 0;
#pragma unroll
    for (int i = 0; i < 9; i++) l2 += v[i] * v[i];
    const double len = sqrt(l2), inv = len > 1e-12 ? 1.0 / len : 0.0;
    Rm[k][k] = len > 1e-12 ? len : 0.0;
#pragma unroll
    for (int i = 0; i < 9; i++) A[k][i] = v[i] * inv;
  }
}
// R x = b
__device__ __forceinline__ void solveR(const double (&Rm)[3][3], const double (&b)[3], double (&x)[3]) {
#pragma unroll
  for (int k = 2; k >= 0; k--) {
    double v = b[k];
#pragma unroll
    for (int kk = k + 1; kk < 3; kk++) v -= Rm[k][kk] * x[kk];
    x[k] = Rm[k][k] > 0 ? v / Rm[k][k] : 0.0;
  }
}

// Per face: V1 of its reader (a function of the reader's fsE[1] alone, so that parts of a partition agree
// on it), U and V0; with face 0 the element's other coefficients. Counts lanes that find solvers not of
// rank 3 in this form in *bad. Values leave as whole 16-byte chunks.
template <typename T>
__global__ void __launch_bounds__(kBuildWarps * 32)
    kBuildStep(const double *fsE, const double *starE, const double *fsA, const double *starA, const double *srcA,
               int rm, const int32_t *elFaEl, const uint8_t *fId, const uint8_t *vId, const uint8_t *faType,
               int64_t nEl, int order, int E, T *fac, uint32_t *gath, int *bad) {
  __shared__ FaceTeam teams[kBuildWarps][kTeams + 1];
  constexpr double tol = rankTol<T>(), tol2 = tol * tol;
  const int l = threadIdx.x & 31, team = l / 9, a = l - 9 * team;  // (lanes 27 .. 31 repeat the last team's item)
  FaceTeam &t = teams[threadIdx.x >> 5][team];
  const int64_t items = nEl * 4, stride = int64_t(gridDim.x) * kBuildWarps * kTeams;
  for (int64_t i0 = (int64_t(blockIdx.x) * kBuildWarps + (threadIdx.x >> 5)) * kTeams; i0 < items; i0 += stride) {
    const int64_t i = min(i0 + min(team, kTeams - 1), items - 1);
    const bool mine = team < kTeams && i0 + team < items;
    const int64_t ef = i, e = ef >> 2;
    const int f = int(ef & 3), ty = faType[ef];
    // value k of the element's coefficients (16-byte chunks interleaved over E elements)
    constexpr int W = 16 / int(sizeof(T));
    const int rows = rm ? FacL<3>::rows : FacL<0>::rows, oStar = rm ? FacL<3>::star : FacL<0>::star;
    const int V = (rm ? FacL<3>::src + 12 * rm : FacL<0>::V) + f * 72;
    const int len = V - f * 72 + 288;
    T *const fe = fac + (e / E) * (int64_t(len) * E) + (e % E) * W;
    // four values from k on (a multiple of four)
    const auto put4 = [&](int k, double v0, double v1, double v2, double v3) {
      if (!mine) return;
      T *p = fe + k / W * (E * W);
      if constexpr (W == 4) {
        *reinterpret_cast<float4 *>(p) = make_float4(float(v0), float(v1), float(v2), float(v3));
      } else {
        *reinterpret_cast<double2 *>(p) = make_double2(v0, v1);
        *reinterpret_cast<double2 *>(p + E * W) = make_double2(v2, v3);
      }
    };
    const bool inner = ty == FT_INNER;
    const int64_t n = inner ? elFaEl[ef] : e;
    const int fo = inner ? fId[ef] : f;
    // V1: the neighbour reads this element's projection at its own face, through its fsE[1] there
    double v1[3] = {0, 0, 0}, M[9], N[9], S[9], Q[3][9];
    bool off;
    {
      const double *p = fsE + (nEl * 4 + n * 4 + fo) * 81 + a * 9;
#pragma unroll
      for (int j = 0; j < 9; j++) M[j] = __ldg(p + j);
      const Scales s1 = scales(t, a, M);
#pragma unroll
      for (int j = 0; j < 9; j++) S[j] = M[j] / (s1.r(a) * s1.c(j));
      off = !(rowBasis(t, a, S, Q) <= tol2) && inner;
#pragma unroll
      for (int j = 0; j < 9; j++)
        if (j == a && inner)
#pragma unroll
          for (int k = 0; k < 3; k++) v1[k] = s1.c(j) * Q[k][j];
    }
    // this lane's rows: M what U's basis comes from, N the own side
    const double *pm = fsE + (nEl * 4 + ef) * 81 + a * 9, *pn = fsE + ef * 81 + a * 9;
    double add[9];
#pragma unroll
    for (int j = 0; j < 9; j++) {
      M[j] = __ldg(pm + j);
      N[j] = __ldg(pn + j);
      add[j] = 0;
    }
    const Scales sc0 = scales(t, a, N), sc1 = scales(t, a, M);
    const Scales sc = inner ? sc1 : sc0;
    // the own side's largest entries per kind of column in the rows' scales: where the element is much
    // stiffer than its neighbour they exceed those of fsE[1], and so does their rounding
    double nS = 0, nV = 0;
#pragma unroll
    for (int j = 0; j < 9; j++) (j < 6 ? nS : nV) = fmax(j < 6 ? nS : nV, fabs(N[j]));
    const double topS = fmax(sc.cS, teamMax(t, a, nS / sc.r(a), 0, 9));
    const double topV = fmax(sc.cV, teamMax(t, a, nV / sc.r(a), 0, 9));
    const double nrm[3] = {f == 2 ? -1.0 : f == 3 ? 1.0 : 0.0, f == 1 ? -1.0 : f == 3 ? 1.0 : 0.0,
                           f == 0 ? -1.0 : f == 3 ? 1.0 : 0.0};
    {
      // N = fsE[0] + sum_d n_fd star_d (+ fsE[1] of a free surface, which reads this element)
      const double *st = starE + e * 72;
      double sd[3][3];
#pragma unroll
      for (int s = 0; s < 3; s++) {
        const int idx = kStarIdx[a][s], col = kStarCol[a][s];
        double v[3] = {0, 0, 0};
        if (idx >= 0)
#pragma unroll
          for (int d = 0; d < 3; d++) v[d] = __ldg(st + d * 24 + idx);
#pragma unroll
        for (int j = 0; j < 9; j++)
          if (j == col) add[j] += nrm[0] * v[0] + nrm[1] * v[1] + nrm[2] * v[2];
#pragma unroll
        for (int d = 0; d < 3; d++) sd[d][s] = kStarDir[0][d] * v[0] + kStarDir[1][d] * v[1] + kStarDir[2][d] * v[2];
      }
#pragma unroll
      for (int j = 0; j < 9; j++) {
        N[j] += add[j];
        if (ty == FT_FREE) N[j] += M[j];
        if (!inner) M[j] = N[j];
      }
      if (f == 0) {
        // the star rows along the derivative directions of the generated products
        put4(oStar + a * 12, sd[0][0], sd[0][1], sd[0][2], sd[1][0]);
        put4(oStar + a * 12 + 4, sd[1][1], sd[1][2], sd[2][0], sd[2][1]);
        put4(oStar + a * 12 + 8, sd[2][2], 0, 0, 0);
      }
    }
    if (mine && a == 0)
      gath[ef] = inner ? uint32_t((n * 4 + fo) * 4 + kFacePerm[order - 2][fo][f][vId[ef]]) : kNoNeighbour;
#pragma unroll
    for (int j = 0; j < 9; j++) S[j] = M[j] = M[j] / (sc.r(a) * sc.c(j));
    off = !(rowBasis(t, a, S, Q) <= tol2) || off;
    // U (scaled rows), then V0 from U V0^T = N: every lane holds U and solves for its own column
#pragma unroll
    for (int k = 0; k < 3; k++) {
      double u = 0;
#pragma unroll
      for (int j = 0; j < 9; j++) u += M[j] * Q[k][j];
      t.U[a][k] = u;
    }
    put4(f * 4 * rows + a * 4, sc.r(a) * t.U[a][0], sc.r(a) * t.U[a][1], sc.r(a) * t.U[a][2], 0);
#pragma unroll
    for (int j = 0; j < 9; j++) t.N[a][j] = N[j] / sc.r(a);
    __syncwarp();
    double A[3][9], Rm[3][3], b[3], x[3], nj[9];
    qrU(t, A, Rm);
#pragma unroll
    for (int i2 = 0; i2 < 9; i2++) nj[i2] = t.N[i2][a];
    double res = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      b[k] = 0;
#pragma unroll
      for (int i2 = 0; i2 < 9; i2++) b[k] += A[k][i2] * nj[i2];
    }
#pragma unroll
    for (int i2 = 0; i2 < 9; i2++) {
      const double d = nj[i2] - A[0][i2] * b[0] - A[1][i2] * b[1] - A[2][i2] * b[2];
      res += d * d;
    }
    solveR(Rm, b, x);
#pragma unroll
    for (int k = 0; k < 3; k++) t.V0[a][k] = x[k];
    put4(V + 8 * a, x[0], x[1], x[2], v1[0]);
    put4(V + 8 * a + 4, v1[1], v1[2], 0, 0);
    // residuals against the largest entry of the column's kind
    const double top = a < 6 ? topS : topV;
    off = off || !(res <= tol2 * top * top);
    __syncwarp();
    if (rm) {
      // anelastic rows (lanes 0 .. 5): UA over the same basis, and the same V0 has to give
      // fsA[0]' = fsA[0] + sum_d n_fd starA_d
      const int s = a < 6 ? a : 0;
      const double *f0 = fsA + ef * 54 + s * 9, *f1 = fsA + (nEl * 4 + ef) * 54 + s * 9, *sa = starA + e * 27;
      double na[9], ma[9], mS = 0, mV = 0, sda[6];
#pragma unroll
      for (int j = 0; j < 9; j++) {
        na[j] = __ldg(f0 + j);
        ma[j] = __ldg(f1 + j);
        const double v = fmax(fabs(na[j]), inner ? fabs(ma[j]) : 0.0);
        if (j < 6)
          mS = fmax(mS, v);
        else
          mV = fmax(mV, v);
      }
      const double aS = teamMax(t, a, mS, 0, 6) * (topS / sc.cS), aV = teamMax(t, a, mV, 0, 6) * (topV / sc.cV);
#pragma unroll
      for (int i2 = 0; i2 < 2; i2++) {
        const int idx = kStarAIdx[s][i2], col = 6 + kStarACol[s][i2];
        double v[3] = {0, 0, 0};
        if (idx >= 0)
#pragma unroll
          for (int d = 0; d < 3; d++) v[d] = __ldg(sa + d * 9 + idx);
#pragma unroll
        for (int j = 0; j < 9; j++)
          if (j == col) na[j] += nrm[0] * v[0] + nrm[1] * v[1] + nrm[2] * v[2];
#pragma unroll
        for (int d = 0; d < 3; d++)
          sda[2 * d + i2] = kStarDir[0][d] * v[0] + kStarDir[1][d] * v[1] + kStarDir[2][d] * v[2];
      }
#pragma unroll
      for (int j = 0; j < 9; j++) {
        if (ty == FT_FREE) na[j] += ma[j];
        if (!inner) ma[j] = na[j];
      }
      if (a < 6) {
        double u[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
          u[k] = 0;
#pragma unroll
          for (int j = 0; j < 9; j++) u[k] += ma[j] / sc.c(j) * Q[k][j];
        }
        put4(f * 4 * rows + (9 + s) * 4, u[0], u[1], u[2], 0);
#pragma unroll
        for (int j = 0; j < 9; j++) {
          const double lim = tol * (j < 6 ? aS : aV);
          double r1 = ma[j], r0 = na[j];
#pragma unroll
          for (int k = 0; k < 3; k++) {
            r1 -= u[k] * sc.c(j) * Q[k][j];
            r0 -= u[k] * t.V0[j][k];
          }
          off = off || !(fabs(r1) <= lim) || !(fabs(r0) <= lim);
        }
        if (f == 0) {
          put4(FacL<3>::starA + s * 8, sda[0], sda[1], sda[2], sda[3]);
          put4(FacL<3>::starA + s * 8 + 4, sda[4], sda[5], 0, 0);
          for (int k = 4 * s; k < 12 * rm; k += 24) {
            const double *p = srcA + e * 12 * rm + k;
            put4(FacL<3>::src + k, p[0], p[1], p[2], p[3]);
          }
        }
      }
    }
    if (off && mine) atomicAdd(bad, 1);
  }
}

}  // namespace edge_b200

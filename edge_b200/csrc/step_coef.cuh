// Coefficients of the strong-form step (step.cuh) from the caller's star matrices, flux solvers and
// connectivity: per element U, star rows and V rows (kFacLen values), and the gather table.
#pragma once
#include "step.cuh"

namespace edge_b200 {

// Orthonormal basis Q (3 x 9) of the rows of S (9 x 9) by Gram-Schmidt with pivoting, each direction
// orthogonalised twice; a direction without a row left is zero. Returns the largest squared norm
// that a row keeps outside Q. S is overwritten.
__device__ __forceinline__ double rowBasis(double (&S)[9][9], double (&Q)[3][9]) {
  for (int k = 0; k < 3; k++) {
    double best = 0, v[9];
#pragma unroll
    for (int j = 0; j < 9; j++) v[j] = 0;
#pragma unroll
    for (int i = 0; i < 9; i++) {
      double n2 = 0;
#pragma unroll
      for (int j = 0; j < 9; j++) n2 += S[i][j] * S[i][j];
      if (n2 > best) {
        best = n2;
#pragma unroll
        for (int j = 0; j < 9; j++) v[j] = S[i][j];
      }
    }
    for (int pass = 0; pass < 2; pass++)
#pragma unroll
      for (int kk = 0; kk < 3; kk++)
        if (kk < k) {
          double d = 0;
#pragma unroll
          for (int j = 0; j < 9; j++) d += v[j] * Q[kk][j];
#pragma unroll
          for (int j = 0; j < 9; j++) v[j] -= d * Q[kk][j];
        }
    double n2 = 0;
#pragma unroll
    for (int j = 0; j < 9; j++) n2 += v[j] * v[j];
    // rows of unit scale: what rounding leaves of a dependent row is no direction
    const double inv = n2 > 1e-24 ? 1.0 / sqrt(n2) : 0.0;
#pragma unroll
    for (int kk = 0; kk < 3; kk++)
      if (kk == k)
#pragma unroll
        for (int j = 0; j < 9; j++) Q[kk][j] = v[j] * inv;
#pragma unroll
    for (int i = 0; i < 9; i++) {
      double d = 0;
#pragma unroll
      for (int j = 0; j < 9; j++) d += S[i][j] * v[j];
      d *= inv * inv;
#pragma unroll
      for (int j = 0; j < 9; j++) S[i][j] -= d * v[j];
    }
  }
  double res = 0;
#pragma unroll
  for (int i = 0; i < 9; i++) {
    double n2 = 0;
#pragma unroll
    for (int j = 0; j < 9; j++) n2 += S[i][j] * S[i][j];
    res = n2 > res ? n2 : res;
  }
  return res;
}

// Row and column scales of a flux solver, one for the stresses and one for the velocities (as
// inputs and as outputs they differ by the moduli and impedances): S = M_ij / (r_i c_j) with entries
// of at most one. (A scale per row or column would blow up the rounding of those that vanish; the
// scales of a face without a neighbour are those of fsE[0], before a free surface's velocity
// columns cancel.)
struct Scales {
  double rS, rV, cS, cV;
  __device__ __forceinline__ double r(int i) const { return i < 6 ? rS : rV; }
  __device__ __forceinline__ double c(int j) const { return j < 6 ? cS : cV; }
};
__device__ __forceinline__ Scales scales(const double (&M)[9][9]) {
  Scales s{0, 0, 0, 0};
#pragma unroll
  for (int i = 0; i < 9; i++)
#pragma unroll
    for (int j = 0; j < 9; j++) {
      if (i < 6)
        s.rS = fmax(s.rS, fabs(M[i][j]));
      else
        s.rV = fmax(s.rV, fabs(M[i][j]));
    }
  if (!(s.rS > 0)) s.rS = 1.0;
  if (!(s.rV > 0)) s.rV = 1.0;
#pragma unroll
  for (int i = 0; i < 9; i++)
#pragma unroll
    for (int j = 0; j < 9; j++) {
      if (j < 6)
        s.cS = fmax(s.cS, fabs(M[i][j]) / s.r(i));
      else
        s.cV = fmax(s.cV, fabs(M[i][j]) / s.r(i));
    }
  if (!(s.cS > 0)) s.cS = 1.0;
  if (!(s.cV > 0)) s.cV = 1.0;
  return s;
}

__device__ __forceinline__ void load81(const double *p, double (&M)[9][9]) {
#pragma unroll
  for (int i = 0; i < 9; i++)
#pragma unroll
    for (int j = 0; j < 9; j++) M[i][j] = __ldg(p + i * 9 + j);
}

constexpr double kRankTol2 = 1e-18;  // squared share of a scaled row outside three directions

// One face per thread, part 0: V1 of the face's reader (a function of the reader's fsE[1] alone, so
// that parts of a partition agree on it); part 1: U and V0 of the face. Counts faces whose flux
// solvers are not of rank 3 in this form in *bad.
template <typename T>
__global__ void __launch_bounds__(64) kBuildStep(const double *fsE, const double *starE, const int32_t *elFaEl,
                                                 const uint8_t *fId, const uint8_t *vId, const uint8_t *faType,
                                                 int64_t nEl, int order, int E, T *fac, uint32_t *gath, int *bad) {
  const int64_t total = (nEl * 4 + 31) / 32 * 64;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += int64_t(gridDim.x) * blockDim.x) {
    // neighbouring threads take the same part
    const int part = int((i >> 5) & 1);
    const int64_t ef = (i >> 6) * 32 + (i & 31);
    if (ef >= nEl * 4) continue;
    const int64_t e = ef >> 2;
    const int f = int(ef & 3), ty = faType[ef];
    // value i of the element's coefficients (16-byte chunks interleaved over E elements)
    constexpr int W = 16 / int(sizeof(T));
    T *const fe = fac + (e / E) * (int64_t(kFacLen) * E) + (e % E) * W;
    const auto put = [&](int i, double v) { fe[i / W * (E * W) + i % W] = T(v); };
    const int V = kFacV + f * 72;
    double M[9][9], Q[3][9];
    if (part == 0) {
      // (the neighbour reads this element's projection at its own face: its fsE[1] there)
      gath[ef] = kNoNeighbour;
      if (ty != FT_INNER) {
#pragma unroll
        for (int j = 0; j < 9; j++) {
          for (int k = 3; k < 8; k++) put(V + 8 * j + k, 0);
        }
        continue;
      }
      const int64_t n = elFaEl[ef];
      const int fo = fId[ef];
      gath[ef] = uint32_t((n * 4 + fo) * 4 + kFacePerm[order - 2][fo][f][vId[ef]]);
      load81(fsE + ((nEl + n) * 4 + fo) * 81, M);
      const Scales sc = scales(M);
#pragma unroll
      for (int a = 0; a < 9; a++)
#pragma unroll
        for (int j = 0; j < 9; j++) M[a][j] /= sc.r(a) * sc.c(j);
      if (rowBasis(M, Q) > kRankTol2) atomicAdd(bad, 1);
#pragma unroll
      for (int j = 0; j < 9; j++) {
#pragma unroll
        for (int k = 0; k < 3; k++) put(V + 8 * j + 3 + k, sc.c(j) * Q[k][j]);
        put(V + 8 * j + 6, 0);
        put(V + 8 * j + 7, 0);
      }
      continue;
    }
    // own side: N = fsE[0] + sum_d n_fd star_d (+ fsE[1] of a free surface, which reads this element)
    double N[9][9];
    load81(fsE + ef * 81, N);
    Scales sc = scales(N);
    const double n0 = f == 2 ? -1.0 : f == 3 ? 1.0 : 0.0, n1 = f == 1 ? -1.0 : f == 3 ? 1.0 : 0.0,
                 n2 = f == 0 ? -1.0 : f == 3 ? 1.0 : 0.0;
    const double *st = starE + e * 72;
#pragma unroll
    for (int q = 0; q < 9; q++) {
      double sd[3][3];
#pragma unroll
      for (int s = 0; s < 3; s++) {
        const int idx = kStarIdx[q][s], col = kStarCol[q][s];
        double v[3] = {0, 0, 0};
        if (idx >= 0)
#pragma unroll
          for (int d = 0; d < 3; d++) v[d] = __ldg(st + d * 24 + idx);
        const double add = n0 * v[0] + n1 * v[1] + n2 * v[2];
#pragma unroll
        for (int j = 0; j < 9; j++)
          if (j == col) N[q][j] += add;
#pragma unroll
        for (int d = 0; d < 3; d++) sd[d][s] = kStarDir[0][d] * v[0] + kStarDir[1][d] * v[1] + kStarDir[2][d] * v[2];
      }
      if (f == 0) {
        // the star rows along the derivative directions of the generated products
        const int o = kFacStar + q * 12;
#pragma unroll
        for (int d = 0; d < 3; d++)
#pragma unroll
          for (int s = 0; s < 3; s++) put(o + 3 * d + s, sd[d][s]);
#pragma unroll
        for (int s = 9; s < 12; s++) put(o + s, 0);
      }
    }
    if (ty == FT_INNER) {
      load81(fsE + (nEl * 4 + ef) * 81, M);
      sc = scales(M);
    } else {
      if (ty == FT_FREE) {
        load81(fsE + (nEl * 4 + ef) * 81, M);
#pragma unroll
        for (int a = 0; a < 9; a++)
#pragma unroll
          for (int j = 0; j < 9; j++) N[a][j] += M[a][j];
      }
#pragma unroll
      for (int a = 0; a < 9; a++)
#pragma unroll
        for (int j = 0; j < 9; j++) M[a][j] = N[a][j];
    }
    double S[9][9];
#pragma unroll
    for (int a = 0; a < 9; a++)
#pragma unroll
      for (int j = 0; j < 9; j++) S[a][j] = M[a][j] = M[a][j] / (sc.r(a) * sc.c(j));
    bool off = rowBasis(S, Q) > kRankTol2;
    // scaled U = (M / r c) Q^T, its orthonormal columns A = U Rm^-1 (twice)
    double U[9][3], A[3][9], Rm[3][3];
#pragma unroll
    for (int a = 0; a < 9; a++)
#pragma unroll
      for (int k = 0; k < 3; k++) {
        double u = 0;
#pragma unroll
        for (int j = 0; j < 9; j++) u += M[a][j] * Q[k][j];
        U[a][k] = u;
      }
#pragma unroll
    for (int k = 0; k < 3; k++) {
      double v[9];
#pragma unroll
      for (int a = 0; a < 9; a++) v[a] = U[a][k];
#pragma unroll
      for (int kk = 0; kk < 3; kk++) Rm[kk][k] = 0;
#pragma unroll
      for (int pass = 0; pass < 2; pass++)
#pragma unroll
        for (int kk = 0; kk < k; kk++) {
          double d = 0;
#pragma unroll
          for (int a = 0; a < 9; a++) d += v[a] * A[kk][a];
          Rm[kk][k] += d;
#pragma unroll
          for (int a = 0; a < 9; a++) v[a] -= d * A[kk][a];
        }
      double n = 0;
#pragma unroll
      for (int a = 0; a < 9; a++) n += v[a] * v[a];
      const double len = sqrt(n);
      Rm[k][k] = len > 1e-12 ? len : 0.0;
#pragma unroll
      for (int a = 0; a < 9; a++) A[k][a] = len > 1e-12 ? v[a] / len : 0.0;
    }
    // V0: U V0^T = N, column by column (residuals against the largest entry of the column's kind)
#pragma unroll
    for (int a = 0; a < 9; a++)
#pragma unroll
      for (int j = 0; j < 9; j++) N[a][j] /= sc.r(a);
    const int U0 = kFacU + f * 36;
#pragma unroll
    for (int a = 0; a < 9; a++) {
#pragma unroll
      for (int k = 0; k < 3; k++) put(U0 + a * 4 + k, sc.r(a) * U[a][k]);
      put(U0 + a * 4 + 3, 0);
    }
#pragma unroll
    for (int j = 0; j < 9; j++) {
      double b[3];
      const double top = j < 6 ? sc.cS : sc.cV;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        b[k] = 0;
#pragma unroll
        for (int a = 0; a < 9; a++) b[k] += A[k][a] * N[a][j];
      }
      double res = 0;
#pragma unroll
      for (int a = 0; a < 9; a++) {
        const double d = N[a][j] - A[0][a] * b[0] - A[1][a] * b[1] - A[2][a] * b[2];
        res += d * d;
      }
      off = off || !(res <= kRankTol2 * top * top);
      double x[3];
#pragma unroll
      for (int k = 2; k >= 0; k--) {
        double t = b[k];
#pragma unroll
        for (int kk = k + 1; kk < 3; kk++) t -= Rm[k][kk] * x[kk];
        x[k] = Rm[k][k] > 0 ? t / Rm[k][k] : 0.0;
      }
#pragma unroll
      for (int k = 0; k < 3; k++) put(V + 8 * j + k, x[k]);
    }
    if (off) atomicAdd(bad, 1);
  }
}

}  // namespace edge_b200

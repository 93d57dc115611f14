// Strong-form GTS step with attenuation (see step.cuh for the form and the characteristics).
//
// The anelastic rows follow the same scheme: their flux solvers act through the same three incoming
// waves (U has six more rows, V0 and V1 are shared), so a face carries three rows for fifteen, and
// own and neighbour flux of all of them are lifted once. With sources the derivatives do not run
// out: the elastic update is Q* = Q + sum_{d<O} c_d der_{d+1}, c_d = dt^(d+1)/(d+1)!, so one level more
// than the time integral needs, which replaces the volume product. The anelastic derivatives are
// linear in the elastic ones, der_{d+1} = w (Psi_d + der_d) per mechanism (w its frequency, Psi the
// strain rate term, the same for all), and the update adds w (sum_d c_d Psi_d - TIA), TIA the time
// integral; unrolled, that is A* = kappa A + sum_d lambda_d Psi_d with scalars
//   kappa = 1 - w sum_d c_d w^d,  lambda_d = w (c_d - sum_{k>d} c_k w^(k-d)),
// so no time-integral tile of the RM * 6 anelastic rows is kept, only their sums lambda Psi in
// registers (B(O-1) modes per mechanism).
//
// A CTA has nine elastic and six anelastic warps (one CTA per SM). The source terms of the elastic
// stress rows are shared out evenly: anelastic warp s takes mechanism 0 of row s (s < 3) or its own
// row (s >= 3), velocity warp 6 + s the other mechanisms of row s.
// Measured (48,000 elements, order 4, 8 runs, 3 mechanisms, FP32): 1.03 ms a step, in weak form 1.58 + 0.74;
// FP64, 24,576 elements, one run: 0.38, was 0.76 + 0.42. Bound: shared-memory pipe 70%, barriers.
#pragma once
#include "step.cuh"

namespace edge_b200 {

template <typename T, int O, int R, int RM>
struct VGeo {
  using S = SGeo<T, O, R>;
  static constexpr int NT = 480, E = S::E, SB = S::SB, GF = S::GF;
  static constexpr size_t nX = S::nX, nXA = size_t(RM) * 6 * 32 * SB, nF = S::nF;
  static constexpr size_t nS = S::nWt > nX ? S::nWt : nX;  // incoming characteristics, then source rows
  static constexpr size_t smMax = 227 * 1024;
  static constexpr size_t offXA = nX * sizeof(T), offS = offXA + nXA * sizeof(T), end0 = offS + nS * sizeof(T);
  // face projections in tiles of their own (the anelastic update then runs beside them), else over
  // the anelastic rows
  static constexpr bool pSep = end0 + 4 * nF * sizeof(T) <= smMax;
  // whole rows of every mechanism fit up to order 5 in FP32 and order 4 in FP64
  static constexpr bool ok = end0 <= smMax && (pSep || 4 * nF <= nXA);
  static constexpr size_t offP = pSep ? end0 : offXA, end1 = pSep ? end0 + 4 * nF * sizeof(T) : end0;
  static constexpr bool dofTile = end1 + nX * sizeof(T) <= smMax;
  static constexpr size_t offD = end1, end2 = end1 + (dofTile ? nX * sizeof(T) : 0);
  using L = FacL<RM>;
  static constexpr size_t bytesU = size_t(E) * L::V * sizeof(T), bytesV = size_t(E) * (L::len - L::V) * sizeof(T);
  static constexpr bool smemU = E <= 4 && end2 + bytesU <= smMax;
  static constexpr bool smemV = smemU && end2 + bytesU + bytesV <= smMax;
  static constexpr size_t offU = end2, offV = offU + (smemU ? bytesU : 0), smem = offV + (smemV ? bytesV : 0);
  // kLiftVisc: incoming characteristics, elastic and anelastic rows
  static constexpr size_t offDL = S::nWt * sizeof(T), offAL = offDL + nX * sizeof(T);
  static constexpr size_t smemLift = offAL + nXA * sizeof(T);
  static constexpr int ctasLift = sizeof(T) == 4 && O <= 4 ? 2 : 1;
};

// the anelastic rows m * 6 + s of a group in and out (row order of the DOF array and the tile)
template <typename T, int O, int R, int RM, bool IN>
__device__ __forceinline__ void rowsA(T *XA, T *dofsA, int64_t e0, int nv, int s, int l) {
  constexpr int SB = SGeo<T, O, R>::SB;
#pragma unroll
  for (int m = 0; m < RM; m++) {
    if constexpr (IN)
      rowsIn<T, O, R, SB, RM * 6>(XA, dofsA, e0, nv, m * 6 + s, l);
    else
      rowsOut<T, O, R, SB, RM * 6>(XA, dofsA, e0, nv, m * 6 + s, l);
  }
}

// o += c * row
template <typename T, int B, int SB>
__device__ __forceinline__ void axpyRow(const T *X, int row, int l, T c, T *o) {
  T y[B];
  ldRow<T, B>(rowPtr<T, SB>(X, row, l), y);
#pragma unroll
  for (int n = 0; n < B; n++) o[n] = fmaT(c, y[n], o[n]);
}

// CTA barrier that elastic and anelastic warps reach in code of their own (the two recursions below
// hold the same number of them): bar.sync counts warps, whatever instruction they arrive from
__device__ __forceinline__ void barAll() { asm volatile("bar.sync 0;" ::: "memory"); }

// Level D: der_{D+1} from der_D in X and XA, elastic warps (acc: Q*, ti: the time integral; csrc of
// velocity warp q: the source rows q - 6 of mechanisms 1 ..). The warps' roles have recursions of
// their own, so that neither keeps the other's values in registers.
template <typename T, int O, int R, int RM, int D>
__device__ __forceinline__ void ckElastic(T *X, const T *XA, T *SRC, int q, int l, const int (&cols)[3],
                                          const T (&cs)[3][3], const T (&csrc)[RM][3], T dt, T sca, T *acc, T *ti) {
  if constexpr (D < O) {
    using G = SGeo<T, O, R>;
    constexpr int B = G::B, SB = G::SB;
    T d[B];
#pragma unroll
    for (int n = 0; n < B; n++) d[n] = T(0);
    if (q >= 6) {
#pragma unroll
      for (int m = 1; m < RM; m++)
#pragma unroll
        for (int i = 0; i < 3; i++) axpyRow<T, B, SB>(XA, m * 6 + i, l, csrc[m][i], d);
      stRow<T, B>(rowPtr<T, SB>(SRC, q, l), d);
#pragma unroll
      for (int n = 0; n < B; n++) d[n] = T(0);
    }
    Mix3<T, SB> z{rowPtr<T, SB>(X, cols[0], l), rowPtr<T, SB>(X, cols[1], l), rowPtr<T, SB>(X, cols[2], l), cs};
    CkMul<O, 1>::template run<T>(z, d);
    barAll();
    const T scb = sca * dt / T(D + 2);
    if (q < 6) addSrcRows<T, B, SB>(SRC, q, l, d);
    if constexpr (D + 1 < O) {
      stRow<T, B>(rowPtr<T, SB>(X, q, l), d);
#pragma unroll
      for (int n = 0; n < B; n++) ti[n] = fmaT(scb, d[n], D == 0 ? dt * acc[n] : ti[n]);
    }
#pragma unroll
    for (int n = 0; n < B; n++) acc[n] = fmaT(sca, d[n], acc[n]);
    if constexpr (D + 1 < O) barAll();
    ckElastic<T, O, R, RM, D + 1>(X, XA, SRC, q, l, cols, cs, csrc, dt, scb, acc, ti);
  }
}
// the same for anelastic warp s (sp: the sums lambda Psi; csrc: row s < 3 of mechanism 0, or the
// diagonal entries of row s >= 3)
template <typename T, int O, int R, int RM, int D>
__device__ __forceinline__ void ckAnelastic(const T *X, T *XA, T *SRC, int s, int l, const int (&cols)[2],
                                            const T (&ca)[3][2], const T (&csrc)[3], const double *omega,
                                            const T (&lam)[RM][O], T (*sp)[nModes(O - 1)]) {
  if constexpr (D < O) {
    using G = SGeo<T, O, R>;
    constexpr int B = G::B, NN = nModes(O - 1), SB = G::SB;
    T d[B];
#pragma unroll
    for (int n = 0; n < B; n++) d[n] = T(0);
#pragma unroll
    for (int i = 0; i < 3; i++)
      if (s < 3 || i < RM) axpyRow<T, B, SB>(XA, s < 3 ? i : i * 6 + s, l, csrc[i], d);
    stRow<T, B>(rowPtr<T, SB>(SRC, s, l), d);
#pragma unroll
    for (int n = 0; n < NN; n++) d[n] = T(0);
    Mix2<T, SB> z{rowPtr<T, SB>(X, cols[0], l), rowPtr<T, SB>(X, cols[1], l), ca};
    CkMul<O, 1>::template run<T>(z, d);
    barAll();
#pragma unroll
    for (int m = 0; m < RM; m++) {
#pragma unroll
      for (int n = 0; n < NN; n++) sp[m][n] = D == 0 ? lam[m][D] * d[n] : fmaT(lam[m][D], d[n], sp[m][n]);
      if constexpr (D + 1 < O) {
        const T om = T(omega[m]);
        T *p = rowPtr<T, SB>(XA, m * 6 + s, l);
        T v[B];
        ldRow<T, B>(p, v);
#pragma unroll
        for (int n = 0; n < B; n++) v[n] = om * (n < NN ? d[n < NN ? n : 0] + v[n] : v[n]);
        stRow<T, B>(p, v);
      }
    }
    if constexpr (D + 1 < O) barAll();
    ckAnelastic<T, O, R, RM, D + 1>(X, XA, SRC, s, l, cols, ca, csrc, omega, lam, sp);
  }
}
// face projections of a row whose time integral holds all modes
template <typename T, int O, int R>
__device__ __forceinline__ void projectTi(T *P, const T *ti, int q, int l) {
  constexpr size_t nF = SGeo<T, O, R>::nF;
  projectPair<T, O, R>(P + 2 * nF, P + 3 * nF, ti, ti, T(1), q, l);
  projectFace<T, O, R, 0>(P, ti, ti, T(1), q, l);
  projectFace<T, O, R, 1>(P + nF, ti, ti, T(1), q, l);
}

template <typename T, int O, int R, int RM>
__global__ void __launch_bounds__(480, 1) kStepVisc(const StepArgs<T> a) {
  using G = SGeo<T, O, R>;
  using V = VGeo<T, O, R, RM>;
  using L = FacL<RM>;
  constexpr int B = G::B, E = G::E, SB = G::SB, NN = nModes(O - 1);
  extern __shared__ __align__(16) unsigned char smem[];
  T *const X = reinterpret_cast<T *>(smem);
  T *const XA = reinterpret_cast<T *>(smem + V::offXA);
  T *const SR = reinterpret_cast<T *>(smem + V::offS);
  T *const P = reinterpret_cast<T *>(smem + V::offP);
  T *const D = reinterpret_cast<T *>(smem + V::offD);
  T *const bufU = reinterpret_cast<T *>(smem + V::offU);
  T *const bufV = reinterpret_cast<T *>(smem + V::offV);
  const int64_t nGroups = (a.elCount + E - 1) / E;
  const auto inGroup = [&](int64_t g) { return int(min(a.elCount - g * E, int64_t(E))); };
  const T dt0 = T(a.dt);
  // pending characteristics: warp q < 12 takes row q; gather entry and own part of the current group
  uint32_t gs = kNoNeighbour;
  T w[G::GF];
  {
    const int q = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int64_t g = blockIdx.x;
    if (q < 9) {
      if constexpr (V::dofTile) rowsIn<T, O, R, SB>(D, a.dofsE, a.elFirst + g * E, inGroup(g), q, l);
    } else {
      rowsA<T, O, R, RM, true>(XA, a.dofsA, a.elFirst + g * E, inGroup(g), q - 9, l);
    }
    if constexpr (V::smemU) issueFac<T, O, R, RM>(a, bufU, 0, L::V, g, nGroups);
    const bool pend = a.faceIn && q < 12 && l / R < inGroup(g);
    const int64_t e = pend ? a.elFirst + g * E + l / R : a.elFirst;
    if (pend) gs = __ldg(a.gath + e * 4 + q / 3);
    if (q < 12) rowNeighbour<T, O, R>(a.faceIn, SR, q, gs, l);
    rowOwn<T, O, R>(a, q < 12 ? q : 0, e, l % R, pend, w);
  }
  cpAsyncCommit();
  for (int64_t g = blockIdx.x; g < nGroups; g += gridDim.x) {
    int tid = threadIdx.x;
    asm volatile("" : "+r"(tid));  // (see kStep)
    const int q = tid >> 5, l = tid & 31;
    const int eo = l / R, r = l % R;
    const int nv = inGroup(g);
    const bool valid = eo < nv;
    const int64_t e0 = a.elFirst + g * E, e = valid ? e0 + eo : a.elFirst;
    const int64_t gn = g + gridDim.x;
    const bool validN = eo < inGroup(gn);
    const int64_t e0n = a.elFirst + gn * E, en = validN ? e0n + eo : a.elFirst;
    const T dt = a.grpDt ? T(a.grpDt[g]) : dt0;
    const T *const facE = facPtr<T, O, R, RM>(a.fac, e);
    const T *const cU = V::smemU ? bufU + eo * G::W : facE;
    const T *const cV = V::smemV ? bufV + eo * G::W : facE + L::V * E;
    const FacU<T, O, R, RM> su{cU, q};
    RegU<T> ru;
    if constexpr (!V::smemU) {
#pragma unroll
      for (int f = 0; f < 4; f++) su(f, ru.u[f]);
    }
    cpAsyncWait<0>();
    __syncwarp();
    if (a.faceIn && q < 12) {
      rowFinish<T, O, R>(SR, q, gs, l, w);
      gs = validN ? __ldg(a.gath + en * 4 + q / 3) : kNoNeighbour;
    }
    __syncthreads();
    if constexpr (V::smemV) issueFac<T, O, R, RM>(a, bufV, L::V, L::len, g, nGroups);
    cpAsyncCommit();
    const auto lift = [&](T *row) {
      if constexpr (V::smemU)
        liftApply<T, O, R>(SR, su, l, row);
      else
        liftApply<T, O, R>(SR, ru, l, row);
    };
    // what the group's second barrier leaves free for the next group
    const auto issueNext = [&]() {
      if constexpr (V::smemU) issueFac<T, O, R, RM>(a, bufU, 0, L::V, gn, nGroups);
      if constexpr (!V::smemV) prefetchFac<T, O, R, RM>(a, V::smemU ? L::V : 0, L::len, gn, nGroups);
      if constexpr (V::dofTile)
        if (q < 9) rowsIn<T, O, R, SB>(D, a.dofsE, e0n, inGroup(gn), q, l);
      cpAsyncCommit();
    };
    if (q < 9) {
      T acc[B];
      if constexpr (V::dofTile)
        ldRow<T, B>(rowPtr<T, SB>(D, q, l), acc);
      else
        ldRowG<T, B>(gRow<T, R, G::GB>(a.dofsE, e, 9, q, r), acc, valid);
      if (a.faceIn) lift(acc);
      stRow<T, B>(rowPtr<T, SB>(X, q, l), acc);
      int cols[3];
      T cs[3][3], csrc[RM][3], st[12];
      ldFac<12, T, O, R>(cU, L::star + q * 12, st);
#pragma unroll
      for (int i = 0; i < 3; i++) {
        cols[i] = kStarCol[q][i];
#pragma unroll
        for (int d = 0; d < 3; d++) cs[d][i] = st[3 * d + i];
      }
#pragma unroll
      for (int m = 1; m < RM; m++) {
        ldFac<12, T, O, R>(cU, L::src + m * 12, st);
#pragma unroll
        for (int i = 0; i < 3; i++) csrc[m][i] = q == 7 ? st[3 + i] : q == 8 ? st[6 + i] : st[i];
      }
      barAll();
      issueNext();
      T ti[B];
      ckElastic<T, O, R, RM, 0>(X, XA, SR, q, l, cols, cs, csrc, dt, dt, acc, ti);
      if (a.tDofs && valid) stRowG<T, B>(gRow<T, R, G::GB>(a.tDofs, e, 9, q, r), ti);
      // the updated rows out through this warp's rows of X
      T *p = rowPtr<T, SB>(X, q, l);
      stRow<T, B>(p, acc);
#pragma unroll
      for (int n = B; n < G::GB; n++) p[n] = T(0);
      __syncwarp();
      rowsOut<T, O, R, SB>(X, a.dofsE, e0, nv, q, l);
      projectTi<T, O, R>(P, ti, q, l);
      cpAsyncWait<1>();
      barAll();
    } else {
      const int s = q - 9;
      if (a.faceIn) {
        // the completed anelastic rows, also to device memory: the update at the group's end reads them
        T up[B];
#pragma unroll
        for (int n = 0; n < B; n++) up[n] = T(0);
        lift(up);
#pragma unroll
        for (int m = 0; m < RM; m++) {
          const T om = T(a.omega[m]);
          T *p = rowPtr<T, SB>(XA, m * 6 + s, l);
          T v[B];
          ldRow<T, B>(p, v);
#pragma unroll
          for (int n = 0; n < B; n++) v[n] = fmaT(om, up[n], v[n]);
          stRow<T, B>(p, v);
#pragma unroll
          for (int n = B; n < G::GB; n++) p[n] = T(0);
        }
        __syncwarp();
        rowsA<T, O, R, RM, false>(XA, a.dofsA, e0, nv, s, l);
      }
      int cols[2];
      T ca[3][2], csrc[3], st[12];
      ldFac<8, T, O, R>(cU, L::starA + s * 8, st);
#pragma unroll
      for (int i = 0; i < 2; i++) {
        cols[i] = 6 + kStarACol[s][i];
#pragma unroll
        for (int d = 0; d < 3; d++) ca[d][i] = st[2 * d + i];
      }
#pragma unroll
      for (int m = 0; m < RM; m++) {
        ldFac<12, T, O, R>(cU, L::src + m * 12, st);
        if (s >= 3) {
          csrc[m] = s == 3 ? st[9] : s == 4 ? st[10] : st[11];
        } else if (m == 0) {
#pragma unroll
          for (int i = 0; i < 3; i++) csrc[i] = s == 0 ? st[i] : s == 1 ? st[3 + i] : st[6 + i];
        }
      }
      // kappa and lambda of the update
      T kap[RM], lam[RM][O];
#pragma unroll
      for (int m = 0; m < RM; m++) {
        const T om = T(a.omega[m]);
        T c[O];
        c[0] = dt;
#pragma unroll
        for (int d = 1; d < O; d++) c[d] = c[d - 1] * dt / T(d + 1);
        T tail = T(0);  // sum_{k > d} c_k w^(k - d), from the last level down
#pragma unroll
        for (int d = O - 1; d >= 0; d--) {
          lam[m][d] = om * (c[d] - tail);
          tail = om * (c[d] + tail);
        }
        kap[m] = T(1) - tail;
      }
      barAll();
      issueNext();
      T sp[RM][NN];
      ckAnelastic<T, O, R, RM, 0>(X, XA, SR, s, l, cols, ca, csrc, a.omega, lam, sp);
      if constexpr (!V::pSep) {
        // the face tiles lie over the anelastic rows: the update waits for their readers
        cpAsyncWait<1>();
        barAll();
        if (s < 3 && a.faceIn) rowNeighbour<T, O, R>(a.faceIn, SR, q, gs, l);
        rowOwn<T, O, R>(a, s < 3 ? q : 0, en, r, validN && a.faceIn && s < 3, w);
        for (int t = q; t < 4 * G::CW; t += 15)
          charTask<T, O, R>(a, P + t / G::CW * G::nF, cV + t / G::CW * 72 * E, t / G::CW, t % G::CW, l, e, r, valid);
        barAll();
      }
      // A* = kappa A + sum lambda Psi: the rows once more (from L2), then the next group's rows
      rowsA<T, O, R, RM, true>(XA, a.dofsA, e0, nv, s, l);
      cpAsyncCommit();
      cpAsyncWait<0>();
      __syncwarp();
#pragma unroll
      for (int m = 0; m < RM; m++) {
        T *p = rowPtr<T, SB>(XA, m * 6 + s, l);
        T v[B];
        ldRow<T, B>(p, v);
#pragma unroll
        for (int n = 0; n < B; n++) v[n] = n < NN ? fmaT(kap[m], v[n], sp[m][n < NN ? n : 0]) : kap[m] * v[n];
        stRow<T, B>(p, v);
#pragma unroll
        for (int n = B; n < G::GB; n++) p[n] = T(0);
      }
      __syncwarp();
      rowsA<T, O, R, RM, false>(XA, a.dofsA, e0, nv, s, l);
      __syncwarp();
      rowsA<T, O, R, RM, true>(XA, a.dofsA, e0n, inGroup(gn), s, l);
      if constexpr (V::pSep) barAll();
    }
    // characteristics (and the next group's pending rows)
    if (V::pSep || q < 9) {
      if (a.faceIn && q < 12) rowNeighbour<T, O, R>(a.faceIn, SR, q, gs, l);
      rowOwn<T, O, R>(a, q < 12 ? q : 0, en, r, validN && a.faceIn && q < 12, w);
      for (int t = q; t < 4 * G::CW; t += 15)
        charTask<T, O, R>(a, P + t / G::CW * G::nF, cV + t / G::CW * 72 * E, t / G::CW, t % G::CW, l, e, r, valid);
      if constexpr (!V::pSep) barAll();
    }
    cpAsyncCommit();
  }
  cpAsyncWait<0>();
}

// the pending surface integrals on their own (kLift with the anelastic rows)
template <typename T, int O, int R, int RM>
__global__ void __launch_bounds__(480, VGeo<T, O, R, RM>::ctasLift) kLiftVisc(const StepArgs<T> a) {
  using G = SGeo<T, O, R>;
  using V = VGeo<T, O, R, RM>;
  constexpr int B = G::B, E = G::E, SB = G::SB;
  extern __shared__ __align__(16) unsigned char smem[];
  T *const wt = reinterpret_cast<T *>(smem);
  T *const D = reinterpret_cast<T *>(smem + V::offDL);
  T *const XA = reinterpret_cast<T *>(smem + V::offAL);
  const int q = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int eo = l / R, r = l % R;
  const int64_t nGroups = (a.elCount + E - 1) / E;
  for (int64_t g = blockIdx.x; g < nGroups; g += gridDim.x) {
    const int nv = int(min(a.elCount - g * E, int64_t(E)));
    const bool valid = eo < nv;
    const int64_t e0 = a.elFirst + g * E, e = valid ? e0 + eo : a.elFirst;
    if (q < 9)
      rowsIn<T, O, R, SB>(D, a.dofsE, e0, nv, q, l);
    else
      rowsA<T, O, R, RM, true>(XA, a.dofsA, e0, nv, q - 9, l);
    cpAsyncCommit();
    RegU<T> ru;
    const FacU<T, O, R, RM> su{facPtr<T, O, R, RM>(a.fac, e), q};
#pragma unroll
    for (int f = 0; f < 4; f++) su(f, ru.u[f]);
    if (q < 12) liftRow<T, O, R, false>(a, a.face, wt, q, l, e, r, valid);
    cpAsyncWait<0>();
    __syncthreads();
    T acc[B];
    if (q < 9) {
      ldRow<T, B>(rowPtr<T, SB>(D, q, l), acc);
    } else {
#pragma unroll
      for (int n = 0; n < B; n++) acc[n] = T(0);
    }
    liftApply<T, O, R>(wt, ru, l, acc);
    if (q < 9) {
      T *p = rowPtr<T, SB>(D, q, l);
      stRow<T, B>(p, acc);
#pragma unroll
      for (int n = B; n < G::GB; n++) p[n] = T(0);
      __syncwarp();
      rowsOut<T, O, R, SB>(D, a.dofsE, e0, nv, q, l);
    } else {
      const int s = q - 9;
#pragma unroll
      for (int m = 0; m < RM; m++) {
        const T om = T(a.omega[m]);
        T *p = rowPtr<T, SB>(XA, m * 6 + s, l);
        T v[B];
        ldRow<T, B>(p, v);
#pragma unroll
        for (int n = 0; n < B; n++) v[n] = fmaT(om, acc[n], v[n]);
        stRow<T, B>(p, v);
#pragma unroll
        for (int n = B; n < G::GB; n++) p[n] = T(0);
      }
      __syncwarp();
      rowsA<T, O, R, RM, false>(XA, a.dofsA, e0, nv, s, l);
    }
    __syncthreads();
  }
}

}  // namespace edge_b200

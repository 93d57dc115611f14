// GTS step of the elastic configurations in strong form, with both sides' fluxes as characteristics.
//
// Strong form. By parts, sum_d star_d K_d M^-1 = sum_d star_d (-K_d^T M^-1) + sum_f (sum_d n_fd
// star_d) fluxL_f fluxT_f (n_f: outward normal of the reference face), and the first sum applied to
// the time-integrated DOFs TI is the Taylor series itself: sum_k dt^(k+1)/(k+1)! der_(k+1). So the
// volume integral costs two accumulations per derivative (the updated DOFs Q* = sum_k dt^k/k! der_k
// beside TI) instead of a product with its own star mixes, TI is needed by its own warp only (and
// stays in registers), and the DOF rows are read once. The element's own flux solver becomes
// fsE[0]' = fsE[0] + sum_d n_fd star_d.
//
// Characteristics. fsE[0]' and fsE[1] of a face both act through the three waves that enter the
// element there (the Godunov state differs from the element's own trace by its own incoming
// waves): [fsE[0]' | fsE[1]] = U [V0^T | V1^T] with U 9x3 (a free surface: U V0^T = fsE[0]' + fsE[1],
// outflow: fsE[0]'). An element therefore writes, per face, three rows for itself (V0^T P, P the
// face projection of TI) and three for its neighbour (the neighbour's V1^T P), and the next launch
// (or kLift, which closes a call) adds the neighbour's rows turned into its face basis, mixes
// U w (three products per mode) and lifts once per face -- own and neighbour flux together. Faces 2
// and 3 share one product each way (FluxPairC).
//
// Against the weak form with nine pre-mixed rows per face (one 9x9-rank mix for each side, a lift
// for each side, volume product) this is 3,150 instead of 5,670 instructions per warp and element
// group at order 5, eight barriers instead of thirteen, and 90.5 KB of device memory traffic per element
// with 16 runs. Whole steps, order 5: 663,552 elements, 16 runs, FP32 29.4 -> 18.3 ms; one run, FP64
// 11.0 -> 3.98 ms. Bound: barriers and shared-memory latency at 18 warps per SM (issue 47%, DRAM 39%).
#pragma once
#include "kernels.cuh"

namespace edge_b200 {

// Coefficients of an element (kBuildStep), in the kernel's precision: U [4][9 or 15][4] (three values
// and a zero; with attenuation the anelastic stress rows follow the nine elastic ones), star rows
// [9][12] (derivative direction d, slot i at 3 d + i), with attenuation the anelastic star rows [6][8]
// (2 d + i) and source matrices [RM][12], then [4][9][8]: V0[i][0..2], the neighbour's V1[i][0..2] and
// two zeros. The 16-byte chunks of the E = 32 / R elements of a kernel group are interleaved
// ([element / E][chunk][E][W]), so that a warp's lanes load consecutive chunks (with one run per
// lane's element, a chunk at an element's stride would take a cache line per lane: 32 instead of 4
// wavefronts a load).
template <int RM>
struct FacL {
  static constexpr int rows = 9 + (RM ? 6 : 0);
  static constexpr int U = 0, star = 16 * rows, starA = star + 108, src = starA + (RM ? 48 : 0),
                       V = src + 12 * RM, len = V + 288;
};
constexpr uint32_t kNoNeighbour = 0xffffffffu;

template <typename T, int O, int R>
struct SGeo {
  static constexpr int B = nModes(O), F = nFaceModes(O), E = 32 / R, NT = 288;
  static constexpr int W = 16 / int(sizeof(T));  // values per 16-byte chunk
  static constexpr int GB = padGlobal<T>(B), GF = padGlobal<T>(F);
  static constexpr int CW = GF / W;              // chunks per face row
  static constexpr int NC = (F + 3) / 4;         // four-mode chunks per face row
  static constexpr int NK = nModes(O - 1);       // modes the derivatives change
  static constexpr int SB = padRow<T>(B), SP = padRow<T>(NK);
  // face rows [row][32 lanes][GF] with their chunks permuted (swz), so that eight lanes of a
  // 128-bit phase hit distinct banks without padding
  static constexpr int P2 = CW % 8 == 0 ? 8 : CW % 4 == 0 ? 4 : CW % 2 == 0 ? 2 : 1;
  __device__ __forceinline__ static int swz(int l) { return (l / (8 / P2)) & (P2 - 1); }
  static constexpr size_t nX = size_t(9) * 32 * SB;     // derivatives of even level, DOF rows out
  static constexpr size_t nF = size_t(9) * 32 * GF;     // one face's projections
  static constexpr size_t nWt = size_t(12) * 32 * GF;   // incoming characteristics of the four faces
  static constexpr size_t nOdd = size_t(9) * 32 * SP;   // derivatives of odd level
  static constexpr size_t nWP = nWt > nOdd ? nWt : nOdd;
  static constexpr size_t smSm = 228 * 1024, smCta = 227 * 1024;
  // CTAs per SM the registers and the shared memory are sized for. FP32: the rows of a lane (Q*, TI,
  // a derivative) take about 2 B + 30 registers: two CTAs up to order 5, one at order 6. FP64 rows
  // take twice that: two CTAs up to order 3.
  static constexpr int ctas = sizeof(T) == 4 ? (O <= 5 ? 2 : 1) : (O <= 3 ? 2 : 1);
  static constexpr size_t budget = smSm / ctas - 1024 < smCta ? smSm / ctas - 1024 : smCta;
  // face projections over X, four faces at a time where they fit beside the other tiles, else two
  static constexpr size_t nP4 = 4 * nF > nX ? 4 * nF : nX;
  static constexpr int NFR = (nP4 + nWP + nX) * sizeof(T) <= budget ? 4 : 2;
  static constexpr size_t nP = NFR == 4 ? nP4 : 2 * nF > nX ? 2 * nF : nX;
  // incoming characteristics and derivatives of odd level behind them, then the tile the next
  // group's DOF rows arrive in
  static constexpr size_t offW = nP * sizeof(T), offD = offW + nWP * sizeof(T);
  static constexpr bool dofTile = offD + nX * sizeof(T) <= budget;
  static constexpr size_t offC = offD + (dofTile ? nX * sizeof(T) : 0);
  // coefficients by cp.async a group ahead: U and the star rows, and the V rows, each where they
  // fit (with few runs per element they are read straight from global memory instead)
  static constexpr size_t bytesU = size_t(E) * FacL<0>::V * sizeof(T), bytesV = size_t(E) * (FacL<0>::len - FacL<0>::V) * sizeof(T);
  static constexpr bool smemU = E <= 4 && offC + bytesU <= budget;
  static constexpr bool smemV = smemU && offC + bytesU + bytesV <= budget;
  static constexpr size_t offV = offC + (smemU ? bytesU : 0);
  static constexpr size_t smem = offV + (smemV ? bytesV : 0);
  static_assert(smem <= smCta && offW % 16 == 0 && offD % 16 == 0 && offC % 16 == 0 && offV % 16 == 0,
                "shared-memory regions");
  // the face tiles reach rows that the last derivative is read from: a barrier between
  static constexpr bool lastReadsX = (O - 1) % 2 == 1;
  // rows of the characteristic sums in flight: all nine, but for order 5 in FP32 with V in shared
  // memory, where their loads would take the registers of what lives around them
  static constexpr int charUnroll = sizeof(T) == 4 && O == 5 && smemV ? 3 : 9;
  // kLift: incoming characteristics, DOF tile, U
  // (order 5 in FP32 on 48,000 / 82,944 tets, three against two CTAs: 0.63 against 0.70 ms with 16
  // runs, 0.138 against 0.111 ms with one, whose U values are held in registers)
  static constexpr int ctasLift = sizeof(T) == 4 ? (O <= 4 || (O == 5 && R >= 8) ? 3 : 2) : (O <= 4 ? 2 : 1);
  static constexpr size_t offDL = nWt * sizeof(T), offCL = offDL + nX * sizeof(T);
  static constexpr bool liftTile = offCL + (smemU ? bytesU : 0) <= smCta;
  static constexpr size_t smemLift = (liftTile ? offCL : offDL) + (smemU ? bytesU : 0);
};

// 16-byte chunk c of face row `row`, lane l
template <typename T, int O, int R>
__device__ __forceinline__ T *faceChunk(T *t, int row, int l, int c) {
  using G = SGeo<T, O, R>;
  return t + (row * 32 + l) * G::GF + (c ^ G::swz(l)) * G::W;
}
// four modes from four-mode chunk j of a face row (those past the row are not touched)
template <typename T, int O, int R>
__device__ __forceinline__ void ldFace4(const T *t, int row, int l, int j, T (&v)[4]) {
  using G = SGeo<T, O, R>;
  if constexpr (sizeof(T) == 4) {
    ld4<T>(faceChunk<T, O, R>(const_cast<T *>(t), row, l, j), v);
  } else {
    const double2 a = *reinterpret_cast<const double2 *>(faceChunk<T, O, R>(const_cast<T *>(t), row, l, 2 * j));
    v[0] = a.x;
    v[1] = a.y;
    v[2] = v[3] = 0;
    if (2 * j + 1 < G::CW) {
      const double2 b = *reinterpret_cast<const double2 *>(faceChunk<T, O, R>(const_cast<T *>(t), row, l, 2 * j + 1));
      v[2] = b.x;
      v[3] = b.y;
    }
  }
}
template <typename T>
__device__ __forceinline__ void stChunk(T *p, const T *v) {
  if constexpr (sizeof(T) == 4)
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else
    *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
}
template <typename T>
__device__ __forceinline__ void ldChunk(const T *p, T *v) {
  if constexpr (sizeof(T) == 4) {
    const float4 t = *reinterpret_cast<const float4 *>(p);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
  } else {
    const double2 t = *reinterpret_cast<const double2 *>(p);
    v[0] = t.x; v[1] = t.y;
  }
}
// four modes into four-mode chunk j of a face row
template <typename T, int O, int R>
__device__ __forceinline__ void stFace4(T *t, int row, int l, int j, const T *v) {
  using G = SGeo<T, O, R>;
#pragma unroll
  for (int h = 0; h < 4; h += G::W)
    if ((4 * j + h) / G::W < G::CW) stChunk<T>(faceChunk<T, O, R>(t, row, l, (4 * j + h) / G::W), v + h);
}

// characteristic rows in device memory: those written for the neighbours as
// [element][face][3][chunk][run][W], the elements' own as [element / E][face][3][chunk][E * R][W], so
// that the lanes of a warp move consecutive 16-byte chunks
template <typename T, int O, int R>
__device__ __forceinline__ int64_t charRow(int64_t slot, int k, int r) {
  using G = SGeo<T, O, R>;
  return ((slot * 3 + k) * (G::CW * R) + r) * G::W;
}

template <typename T, int O, int R>
__device__ __forceinline__ int64_t ownRow(int64_t e, int t, int r) {
  using G = SGeo<T, O, R>;
  return ((e / G::E * 12 + t) * (G::CW * 32) + (e % G::E) * R + r) * G::W;
}

// Row t = 3 f + k of the incoming characteristics is its own part plus the neighbour's, turned into
// this element's face basis. A lane's row has four sources of latency (the gather entry, the
// neighbour's row behind it, its own row, and the DOF rows), so kStep fetches them a group ahead:
// rowNeighbour starts the copy of the neighbours' rows into the tile (with few runs
// consecutive lanes the consecutive chunks of a neighbour's row; gs of the lane's own element), rowOwn loads the own row,
// and rowFinish turns and adds in place; liftRow does it at once.
template <typename T, int O, int R>
__device__ __forceinline__ void rowNeighbour(const T *in, T *wt, int t, uint32_t gs, int l) {
  using G = SGeo<T, O, R>;
  if constexpr (R >= 8) {  // a chunk of eight runs fills a line: every lane its own row
    if (gs == kNoNeighbour) return;
    const T *nb = in + charRow<T, O, R>(gs >> 2, t % 3, l % R);
#pragma unroll
    for (int c = 0; c < G::CW; c++) cpAsync16(faceChunk<T, O, R>(wt, t, l, c), nb + c * (R * G::W));
    return;
  }
#pragma unroll
  for (int it = 0; it < G::CW; it++) {
    const int k = it * 32 + l, eo = k / (G::CW * R), c = k - eo * (G::CW * R);
    const uint32_t s = __shfl_sync(0xffffffffu, gs, eo * R);
    if (s != kNoNeighbour)
      cpAsync16(faceChunk<T, O, R>(wt, t, eo * R + c % R, c / R), in + charRow<T, O, R>(s >> 2, t % 3, 0) + c * G::W);
  }
}
template <typename T, int O, int R>
__device__ __forceinline__ void rowOwn(const StepArgs<T> &a, int t, int64_t e, int r, bool valid, T *v) {
  using G = SGeo<T, O, R>;
  const T *own = a.wOwn + ownRow<T, O, R>(e, t, r);
#pragma unroll
  for (int c = 0; c < G::CW; c++) {
    if (valid) {
      ldChunk<T>(own + c * (32 * G::W), v + c * G::W);
    } else {
#pragma unroll
      for (int i = 0; i < G::W; i++) v[c * G::W + i] = T(0);
    }
  }
}
template <int O, typename T>
__device__ __forceinline__ void turnRow(uint32_t o, const T *x, T *v) {
  if (o == 0)
    OriMul<O, 0>::template run<T>(x, v);
  else if (o == 1)
    OriMul<O, 1>::template run<T>(x, v);
  else
    OriMul<O, 2>::template run<T>(x, v);
}
template <typename T, int O, int R>
__device__ __forceinline__ void rowFinish(T *wt, int t, uint32_t gs, int l, T *v) {
  using G = SGeo<T, O, R>;
  if (gs != kNoNeighbour) {
    T x[G::GF];
#pragma unroll
    for (int c = 0; c < G::CW; c++) ldChunk<T>(faceChunk<T, O, R>(wt, t, l, c), x + c * G::W);
    turnRow<O, T>(gs & 3u, x, v);
  }
#pragma unroll
  for (int c = 0; c < G::CW; c++) stChunk<T>(faceChunk<T, O, R>(wt, t, l, c), v + c * G::W);
}
template <typename T, int O, int R, bool LTS>
__device__ __forceinline__ void liftRow(const StepArgs<T> &a, const T *in, T *wt, int t, int l, int64_t e, int r,
                                        bool valid) {
  using G = SGeo<T, O, R>;
  T v[G::GF], x[G::GF];
  const uint32_t gs = valid ? __ldg(a.gath + e * 4 + t / 3) : kNoNeighbour;
  rowOwn<T, O, R>(a, t, e, r, valid, v);
  if (gs != kNoNeighbour) {
    int64_t slot = gs >> 2;
    if constexpr (LTS) {
      // what the neighbour wrote over this element's step: its two-step sum, or its half-step rows
      const int rel = a.ltsRel[e * 4 + t / 3];
      if (rel != LTS_EQ) {
        in = rel == LTS_GT ? a.faceSum : a.firstTs ? a.faceHalf1 : a.faceHalf2;
        slot = int64_t((rel == LTS_GT ? a.sumIdx : a.halfIdx)[gs >> 4]) * 4 + (gs >> 2 & 3);
      }
    }
    const T *nb = in + charRow<T, O, R>(slot, t % 3, r);
#pragma unroll
    for (int c = 0; c < G::CW; c++) ldChunk<T>(nb + c * (R * G::W), x + c * G::W);
    turnRow<O, T>(gs & 3u, x, v);
  }
#pragma unroll
  for (int c = 0; c < G::CW; c++) stChunk<T>(faceChunk<T, O, R>(wt, t, l, c), v + c * G::W);
}

// four modes of s = U w of face f (u: this row's three values)
template <typename T, int O, int R>
__device__ __forceinline__ void liftMix(const T *wt, int f, const T *u, int l, int j, T (&s)[4]) {
  T w0[4], w1[4], w2[4];
  ldFace4<T, O, R>(wt, 3 * f, l, j, w0);
  ldFace4<T, O, R>(wt, 3 * f + 1, l, j, w1);
  ldFace4<T, O, R>(wt, 3 * f + 2, l, j, w2);
  if constexpr (sizeof(T) == 4) {
    // packed pairs: half the issue slots, the same rounding
#pragma unroll
    for (int h = 0; h < 4; h += 2) {
      float2 p = __fmul2_rn(make_float2(u[0], u[0]), make_float2(w0[h], w0[h + 1]));
      p = __ffma2_rn(make_float2(u[1], u[1]), make_float2(w1[h], w1[h + 1]), p);
      p = __ffma2_rn(make_float2(u[2], u[2]), make_float2(w2[h], w2[h + 1]), p);
      s[h] = p.x;
      s[h + 1] = p.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; i++) s[i] = fmaT(u[2], w2[i], fmaT(u[1], w1[i], u[0] * w0[i]));
  }
}
template <typename T, int O, int R, int FA, int C = 0>
__device__ __forceinline__ void liftFace(const T *wt, const T *u, int l, T *acc) {
  if constexpr (C < SGeo<T, O, R>::NC) {
    T s[4];
    liftMix<T, O, R>(wt, FA, u, l, C, s);
    FluxTC<O, FA, C>::template run<T>(s, acc);
    liftFace<T, O, R, FA, C + 1>(wt, u, l, acc);
  }
}
template <typename T, int O, int R, int C = 0>
__device__ __forceinline__ void liftPair(const T *wt, const T *u2, const T *u3, int l, T *acc) {
  if constexpr (C < SGeo<T, O, R>::NC) {
    T s2[4], s3[4];
    liftMix<T, O, R>(wt, 2, u2, l, C, s2);
    liftMix<T, O, R>(wt, 3, u3, l, C, s3);
    FluxPairC<O, C>::template lift<T>(s2, s3, acc);
    liftPair<T, O, R, C + 1>(wt, u2, u3, l, acc);
  }
}
// coefficients of element e (its first chunk): in device memory, and n values at offset `off` of it
// or of the same layout in shared memory
template <typename T, int O, int R, int RM>
__device__ __forceinline__ const T *facPtr(const T *fac, int64_t e) {
  using G = SGeo<T, O, R>;
  return fac + (e / G::E) * (FacL<RM>::len * G::E) + (e % G::E) * G::W;
}
template <int N, typename T, int O, int R>
__device__ __forceinline__ void ldFac(const T *p, int off, T *v) {
  using G = SGeo<T, O, R>;
#pragma unroll
  for (int i = 0; i < N; i += G::W) ldChunk<T>(p + (off + i) * G::E, v + i);
}
// U of row q per face: read where it is used (shared memory; rare launches), or held in registers
// since the start of the group (device memory)
template <typename T, int O, int R, int RM>
struct FacU {
  const T *p;
  int q;
  __device__ __forceinline__ void operator()(int f, T (&u)[4]) const { ldFac<4, T, O, R>(p, FacL<RM>::U + f * (4 * FacL<RM>::rows) + q * 4, u); }
};
template <typename T>
struct RegU {
  T u[4][4];
  __device__ __forceinline__ void operator()(int f, T (&v)[4]) const {
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = u[f][i];
  }
};

// the flux of the four faces into a row (U(f, u): its values of U at face f)
template <typename T, int O, int R, typename Z>
__device__ __forceinline__ void liftApply(const T *wt, const Z &U, int l, T *acc) {
  T u[4], u3[4];
  U(0, u);
  liftFace<T, O, R, 0>(wt, u, l, acc);
  U(1, u);
  liftFace<T, O, R, 1>(wt, u, l, acc);
  U(2, u);
  U(3, u3);
  liftPair<T, O, R>(wt, u, u3, l, acc);
}

// cp.async of coefficients [from, to) of group g's elements into buf, in the same layout
template <typename T, int O, int R, int RM>
__device__ __forceinline__ void issueFac(const StepArgs<T> &a, T *buf, int from, int to, int64_t g, int64_t nGroups) {
  using G = SGeo<T, O, R>;
  if (g >= nGroups) return;
  const int n = (to - from) / G::W * G::E;
  for (int i = threadIdx.x; i < n; i += 32 * FacL<RM>::rows) {
    const int eo = i % G::E;
    if (g * G::E + eo >= a.elCount) continue;
    cpAsync16(buf + i * G::W, facPtr<T, O, R, RM>(a.fac, a.elFirst + g * G::E + eo) + (from + i / G::E * G::W) * G::E);
  }
}
// the same coefficients into L2 (a group ahead, where the kernel reads them from device memory)
template <typename T, int O, int R, int RM>
__device__ __forceinline__ void prefetchFac(const StepArgs<T> &a, int from, int to, int64_t g, int64_t nGroups) {
  using G = SGeo<T, O, R>;
  if (g >= nGroups) return;
  const char *p = reinterpret_cast<const char *>(a.fac + ((a.elFirst + g * G::E) / G::E * FacL<RM>::len + from) * G::E);
  const int bytes = (to - from) * G::E * int(sizeof(T));
  for (int i = threadIdx.x * 128; i < bytes; i += 32 * FacL<RM>::rows * 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + i));
}

// DOF rows of a group between device memory and the tile rows of warp q: with one run per element
// consecutive lanes move the consecutive chunks of an element's row (a row per lane would touch a
// cache line per lane), with more runs those of an element's runs. nv: elements of the group.
// row: of the nRows of the DOF array and its tile
template <typename T, int O, int R, int S, int NR = 9>
__device__ __forceinline__ void rowsIn(T *tile, const T *dofs, int64_t e0, int nv, int q, int l) {
  using G = SGeo<T, O, R>;
  if constexpr (R == 1) {
    constexpr int C = G::GB / G::W;
#pragma unroll
    for (int it = 0; it < C; it++) {
      const int k = it * 32 + l, eo = k / C, c = k - eo * C;
      if (eo < nv) cpAsync16(tile + (q * 32 + eo) * S + c * G::W, dofs + ((e0 + eo) * NR + q) * G::GB + c * G::W);
    }
  } else {
    if (l / R < nv) copyRows<T, R, G::GB, S, true>(tile, dofs, e0 + l / R, NR, q, l / R, l % R);
  }
}
template <typename T, int O, int R, int S, int NR = 9>
__device__ __forceinline__ void rowsOut(const T *tile, T *dofs, int64_t e0, int nv, int q, int l) {
  using G = SGeo<T, O, R>;
  if constexpr (R == 1) {
    constexpr int C = G::GB / G::W;
#pragma unroll
    for (int it = 0; it < C; it++) {
      const int k = it * 32 + l, eo = k / C, c = k - eo * C;
      T v[G::W];
      ldChunk<T>(tile + (q * 32 + eo) * S + c * G::W, v);
      if (eo < nv) stChunk<T>(dofs + ((e0 + eo) * NR + q) * G::GB + c * G::W, v);
    }
  } else {
    if (l / R < nv)
      storeRowsCoalesced<T, R, G::GB, S, true>(tile, dofs + ((e0 + l / R) * NR + q) * int64_t(R * G::GB), q, l / R, l % R);
  }
}

// face projections of this warp's row, four modes at a time (few values in registers beside Q* and
// TI), into their tiles
template <typename T, int O, int R, int C = 0>
__device__ __forceinline__ void projectPair(T *t2, T *t3, const T *ti, const T *acc, T dt, int q, int l) {
  if constexpr (C < SGeo<T, O, R>::NC) {
    T p2[4], p3[4];
    FluxPairC<O, C>::template project<T>(ti, acc, dt, p2, p3);
    stFace4<T, O, R>(t2, q, l, C, p2);
    stFace4<T, O, R>(t3, q, l, C, p3);
    projectPair<T, O, R, C + 1>(t2, t3, ti, acc, dt, q, l);
  }
}
template <typename T, int O, int R, int FA, int C = 0>
__device__ __forceinline__ void projectFace(T *t, const T *ti, const T *acc, T dt, int q, int l) {
  if constexpr (C < SGeo<T, O, R>::NC) {
    T p[4];
    FluxLC<O, FA, C>::template run<T>(ti, acc, dt, p);
    stFace4<T, O, R>(t, q, l, C, p);
    projectFace<T, O, R, FA, C + 1>(t, ti, acc, dt, q, l);
  }
}

// derivatives D .. O-1 (see CkStep): acc accumulates Q*, ti the time integral of the first NK modes
// (H: th that over the first half of the step, for LTS)
template <typename T, int O, int R, int D, bool H>
__device__ __forceinline__ void ckStrong(T *X, T *XP, int q, int l, const int (&cols)[3], const T (&cs)[3][3], T dt,
                                         T sca, T scaH, T *acc, T *ti, T *th) {
  if constexpr (D < O) {
    using G = SGeo<T, O, R>;
    constexpr int NN = nModes(O - D);
    constexpr bool IN_P = (D - 1) % 2 == 1, OUT_P = D % 2 == 1;
    constexpr int SI = IN_P ? G::SP : G::SB, SO = OUT_P ? G::SP : G::SB;
    const T *in = IN_P ? XP : X;
    T *out = OUT_P ? XP : X;
    T d[NN];
#pragma unroll
    for (int n = 0; n < NN; n++) d[n] = T(0);
    Mix3<T, SI> z{rowPtr<T, SI>(in, cols[0], l), rowPtr<T, SI>(in, cols[1], l), rowPtr<T, SI>(in, cols[2], l), cs};
    CkMul<O, D>::template run<T>(z, d);
    if constexpr (D + 1 < O) stRow<T, NN>(rowPtr<T, SO>(out, q, l), d);
    // sca = dt^D / D!
    const T scb = sca * dt / T(D + 1);
    // scaH = (dt / 2)^D / D!
    const T scbH = H ? scaH * (dt * T(0.5)) / T(D + 1) : T(0);
#pragma unroll
    for (int n = 0; n < NN; n++) {
      if constexpr (H) th[n] = fmaT(scbH, d[n], D == 1 ? (dt * T(0.5)) * acc[n] : th[n]);
      ti[n] = fmaT(scb, d[n], D == 1 ? dt * acc[n] : ti[n]);
      acc[n] = fmaT(sca, d[n], acc[n]);
    }
    if constexpr (D + 1 < O) __syncthreads();
    ckStrong<T, O, R, D + 1, H>(X, XP, q, l, cols, cs, dt, scb, scbH, acc, ti, th);
  }
}

// characteristics of one 16-byte chunk c of face f's modes (its projections in tile p): the element's
// own rows and its neighbour's, to device memory
// LTS: also added up over the two steps of a pair for a larger neighbour (faceSum)
template <typename T, int O, int R, int LTS = 0>
__device__ __forceinline__ void charTask(const StepArgs<T> &a, const T *p, const T *V, int f, int c, int l, int64_t e,
                                         int r, bool valid) {
  using G = SGeo<T, O, R>;
  T w[6][G::W];
#pragma unroll
  for (int k = 0; k < 6; k++)
#pragma unroll
    for (int i = 0; i < G::W; i++) w[k][i] = T(0);
#pragma unroll(G::charUnroll)
  for (int i = 0; i < 9; i++) {
    T x[G::W], v[8];
    ldChunk<T>(faceChunk<T, O, R>(const_cast<T *>(p), i, l, c), x);
#pragma unroll
    for (int k = 0; k < 8; k += G::W) ldChunk<T>(V + (i * 8 + k) * G::E, v + k);
#pragma unroll
    for (int k = 0; k < 6; k++) {
      if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int h = 0; h < 4; h += 2) {
          const float2 t = __ffma2_rn(make_float2(v[k], v[k]), make_float2(x[h], x[h + 1]), make_float2(w[k][h], w[k][h + 1]));
          w[k][h] = t.x;
          w[k][h + 1] = t.y;
        }
      } else {
#pragma unroll
        for (int u = 0; u < G::W; u++) w[k][u] = fmaT(v[k], x[u], w[k][u]);
      }
    }
  }
  if (!valid) return;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    stChunk<T>(a.wOwn + ownRow<T, O, R>(e, 3 * f + k, r) + c * (32 * G::W), w[k]);
    stChunk<T>(a.face + charRow<T, O, R>(e * 4 + f, k, r) + c * (R * G::W), w[3 + k]);
  }
  if constexpr (LTS > 0) {
    if (a.ltsFlags[e] & LTS_HAS_LARGER) {
      const int64_t slot = int64_t(a.sumIdx[e]) * 4 + f;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        T *p2 = a.faceSum + charRow<T, O, R>(slot, k, r) + c * (R * G::W);
        T x[G::W];
        ldChunk<T>(p2, x);
#pragma unroll
        for (int u = 0; u < G::W; u++) x[u] = a.firstTs ? w[3 + k][u] : x[u] + w[3 + k][u];
        stChunk<T>(p2, x);
      }
    }
  }
}

// The neighbour's rows of the half-step projections in tile p, for elements with a smaller neighbour:
// faceHalf1 over the first half of the step, faceHalf2 over the second (what this thread's charTask
// wrote for the whole step less the first half)
template <typename T, int O, int R>
__device__ __forceinline__ void halfTask(const StepArgs<T> &a, const T *p, const T *V, int f, int c, int l, int64_t e,
                                         int r, bool half) {
  using G = SGeo<T, O, R>;
  T w[3][G::W];
#pragma unroll
  for (int k = 0; k < 3; k++)
#pragma unroll
    for (int i = 0; i < G::W; i++) w[k][i] = T(0);
#pragma unroll 3
  for (int i = 0; i < 9; i++) {
    T x[G::W], v[8];
    ldChunk<T>(faceChunk<T, O, R>(const_cast<T *>(p), i, l, c), x);
#pragma unroll
    for (int k = 0; k < 8; k += G::W) ldChunk<T>(V + (i * 8 + k) * G::E, v + k);
#pragma unroll
    for (int k = 0; k < 3; k++)
#pragma unroll
      for (int u = 0; u < G::W; u++) w[k][u] = fmaT(v[3 + k], x[u], w[k][u]);
  }
  if (!half) return;
  const int64_t slot = int64_t(a.halfIdx[e]) * 4 + f;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const int64_t o = charRow<T, O, R>(slot, k, r) + c * (R * G::W);
    T x[G::W];
    ldChunk<T>(a.face + charRow<T, O, R>(e * 4 + f, k, r) + c * (R * G::W), x);
    stChunk<T>(a.faceHalf1 + o, w[k]);
#pragma unroll
    for (int u = 0; u < G::W; u++) x[u] -= w[k][u];
    stChunk<T>(a.faceHalf2 + o, x);
  }
}

// One GTS step of elements [elFirst, elFirst + elCount) up to their surface integrals: the pending
// characteristics of the previous step (faceIn and wOwn, none when faceIn is null) complete the DOF
// rows, the recursion updates them, and this step's characteristics leave in face and wOwn.
// Measured (48,000 elements, order 5, 16 runs, FP32): 1.22 ms; order 4, 8 runs: 0.35 ms.
// LTS 1, 2: the local step of a time group (rate-2 local time stepping; nothing is pending then): the
// neighbours' rows also summed over two steps, and with 2 the half-step rows
template <typename T, int O, int R, int LTS = 0>
__global__ void __launch_bounds__(SGeo<T, O, R>::NT, LTS == 2 ? 1 : SGeo<T, O, R>::ctas) kStep(const StepArgs<T> a) {
  using G = SGeo<T, O, R>;
  constexpr int B = G::B, E = G::E, SB = G::SB;
  extern __shared__ __align__(16) unsigned char smem[];
  T *const X = reinterpret_cast<T *>(smem);
  T *const XP = reinterpret_cast<T *>(smem + G::offW);  // incoming characteristics, then derivatives of odd level
  T *const D = reinterpret_cast<T *>(smem + G::offD);
  T *const bufU = reinterpret_cast<T *>(smem + G::offC);
  T *const bufV = reinterpret_cast<T *>(smem + G::offV);
  const int64_t nGroups = (a.elCount + E - 1) / E;
  // elements of group g
  const bool pending = LTS == 0 && a.faceIn;
  const auto inGroup = [&](int64_t g) { return int(min(a.elCount - g * E, int64_t(E))); };
  const T dt0 = T(a.dt);
  uint32_t gs0 = kNoNeighbour, gs1 = kNoNeighbour;
  T w0[G::GF], w1[G::GF];
  {
    const int q = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int eo = l / R, r = l % R;
    const int64_t g = blockIdx.x;
    if constexpr (G::dofTile) rowsIn<T, O, R, SB>(D, a.dofsE, a.elFirst + g * E, inGroup(g), q, l);
    if constexpr (G::smemU) issueFac<T, O, R, 0>(a, bufU, 0, FacL<0>::V, g, nGroups);
    // pending characteristics: warp q takes rows q and (q < 3) q + 9; gather entries and own parts of
    // the current group
    const int t1 = q < 3 ? q + 9 : q;
    const bool pend = pending && g * E + eo < a.elCount;
    const int64_t e = pend ? a.elFirst + g * E + eo : a.elFirst;
    if (pend) {
      gs0 = __ldg(a.gath + e * 4 + q / 3);
      gs1 = __ldg(a.gath + e * 4 + t1 / 3);
    }
    rowNeighbour<T, O, R>(a.faceIn, XP, q, gs0, l);
    rowOwn<T, O, R>(a, q, e, r, pend, w0);
    if (q < 3) rowNeighbour<T, O, R>(a.faceIn, XP, t1, gs1, l);
    rowOwn<T, O, R>(a, t1, e, r, pend && q < 3, w1);
  }
  cpAsyncCommit();
  for (int64_t g = blockIdx.x; g < nGroups; g += gridDim.x) {
    // a new name for the thread index in every group: offsets derived from it are computed where they
    // are used instead of being kept (and spilled) across the loop
    int tid = threadIdx.x;
    asm volatile("" : "+r"(tid));
    const int q = tid >> 5, l = tid & 31;
    const int eo = l / R, r = l % R;
    const int t1 = q < 3 ? q + 9 : q;
    const bool valid = g * E + eo < a.elCount;
    const int64_t e = valid ? a.elFirst + g * E + eo : a.elFirst;
    const int64_t gn = g + gridDim.x;
    const T dt = LTS == 0 && a.grpDt ? T(a.grpDt[g]) : dt0;
    const T *const facE = facPtr<T, O, R, 0>(a.fac, e);
    const T *const cU = G::smemU ? bufU + eo * G::W : facE;
    const T *const cV = G::smemV ? bufV + eo * G::W : facE + FacL<0>::V * E;
    // U and star rows: read where they are used from shared memory, from here on from device memory
    RegU<T> ru;
    T st[12];
    const FacU<T, O, R, 0> su{cU, q};
    if constexpr (!G::smemU) {
#pragma unroll
      for (int f = 0; f < 4; f++) su(f, ru.u[f]);
      ldFac<12, T, O, R>(cU, FacL<0>::star + q * 12, st);
    }
    // the next group's element of this lane
    const bool validN = gn < nGroups && gn * E + eo < a.elCount;
    const int64_t en = validN ? a.elFirst + gn * E + eo : a.elFirst;
    cpAsyncWait<0>();
    __syncwarp();
    if (pending) {
      rowFinish<T, O, R>(XP, q, gs0, l, w0);
      if (q < 3) rowFinish<T, O, R>(XP, t1, gs1, l, w1);
      gs0 = gs1 = kNoNeighbour;
      if (validN) {
        gs0 = __ldg(a.gath + en * 4 + q / 3);
        gs1 = __ldg(a.gath + en * 4 + t1 / 3);
      }
    }
    __syncthreads();
    // every warp is past the previous group's characteristics, the last readers of V and of X
    if constexpr (G::smemV) issueFac<T, O, R, 0>(a, bufV, FacL<0>::V, FacL<0>::len, g, nGroups);
    cpAsyncCommit();
    T acc[B];
    if constexpr (G::dofTile) {
      ldRow<T, B>(rowPtr<T, SB>(D, q, l), acc);
    } else {
      ldRowG<T, B>(gRow<T, R, G::GB>(a.dofsE, e, 9, q, r), acc, valid);
    }
    if (pending) {
      if constexpr (G::smemU)
        liftApply<T, O, R>(XP, su, l, acc);
      else
        liftApply<T, O, R>(XP, ru, l, acc);
    }
    stRow<T, B>(rowPtr<T, SB>(X, q, l), acc);
    if constexpr (G::smemU) ldFac<12, T, O, R>(cU, FacL<0>::star + q * 12, st);
    int cols[3];
    T cs[3][3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
      cols[i] = kStarCol[q][i];
#pragma unroll
      for (int d = 0; d < 3; d++) cs[d][i] = st[3 * d + i];
    }
    __syncthreads();
    // every thread read this group's U and star rows
    if constexpr (G::smemU) issueFac<T, O, R, 0>(a, bufU, 0, FacL<0>::V, gn, nGroups);
    if constexpr (!G::smemV) prefetchFac<T, O, R, 0>(a, G::smemU ? FacL<0>::V : 0, FacL<0>::len, gn, nGroups);
    cpAsyncCommit();
    T ti[G::NK], th[LTS == 2 ? G::NK : 1];
    ckStrong<T, O, R, 1, LTS == 2>(X, XP, q, l, cols, cs, dt, dt, dt * T(0.5), acc, ti, th);
    if (a.tDofs && valid) {
      T t[B];
#pragma unroll
      for (int n = 0; n < B; n++) t[n] = n < G::NK ? ti[n < G::NK ? n : 0] : dt * acc[n];
      stRowG<T, B>(gRow<T, R, G::GB>(a.tDofs, e, 9, q, r), t);
    }
    // the updated rows out through this warp's tile rows, then the next group's rows in
    if constexpr (G::dofTile) {
      T *p = rowPtr<T, SB>(D, q, l);
      stRow<T, B>(p, acc);
#pragma unroll
      for (int n = B; n < G::GB; n++) p[n] = T(0);
      __syncwarp();
      rowsOut<T, O, R, SB>(D, a.dofsE, a.elFirst + g * E, inGroup(g), q, l);
      __syncwarp();
      rowsIn<T, O, R, SB>(D, a.dofsE, a.elFirst + gn * E, inGroup(gn), q, l);
    } else if (valid) {
      stRowG<T, B>(gRow<T, R, G::GB>(a.dofsE, e, 9, q, r), acc);
    }
    cpAsyncCommit();
    // face projections, two or four faces at a time
    if constexpr (G::lastReadsX) __syncthreads();
    projectPair<T, O, R>(X, X + G::nF, ti, acc, dt, q, l);
    if constexpr (G::NFR == 4) {
      projectFace<T, O, R, 0>(X + 2 * G::nF, ti, acc, dt, q, l);
      projectFace<T, O, R, 1>(X + 3 * G::nF, ti, acc, dt, q, l);
    }
    // V (the copies since are the next group's U and DOF rows)
    cpAsyncWait<2>();
    __syncthreads();
    // (every warp is past the recursion: the tile of odd derivatives takes the next group's rows)
    if (pending) {
      rowNeighbour<T, O, R>(a.faceIn, XP, q, gs0, l);
      if (q < 3) rowNeighbour<T, O, R>(a.faceIn, XP, t1, gs1, l);
    }
    cpAsyncCommit();
    if constexpr (G::NFR == 2) {
      for (int t = q; t < 2 * G::CW; t += 9) {
        const int i = t / G::CW, c = t - i * G::CW;
        charTask<T, O, R, LTS>(a, X + i * G::nF, cV + (i + 2) * 72 * E, i + 2, c, l, e, r, valid);
      }
      __syncthreads();
      projectFace<T, O, R, 0>(X, ti, acc, dt, q, l);
      projectFace<T, O, R, 1>(X + G::nF, ti, acc, dt, q, l);
      __syncthreads();
    }
    // (both arrays are set on every path: they do not live through the group)
    rowOwn<T, O, R>(a, q, en, r, validN && pending, w0);
    rowOwn<T, O, R>(a, t1, en, r, validN && pending && q < 3, w1);
    for (int t = q; t < G::NFR * G::CW; t += 9) {
      const int i = t / G::CW, c = t - i * G::CW;
      const int f = G::NFR == 4 ? (i + 2) & 3 : i;
      charTask<T, O, R, LTS>(a, X + i * G::nF, cV + f * 72 * E, f, c, l, e, r, valid);
    }
    if constexpr (LTS == 2) {
      const bool half = valid && (a.ltsFlags[e] & LTS_HAS_SMALLER);
      if (__any_sync(0xffffffffu, half)) {  // (the same in every warp)
#pragma unroll
        for (int p = 0; p < 4; p += G::NFR) {
          __syncthreads();
          if (p == 0) projectPair<T, O, R>(X, X + G::nF, th, acc, dt * T(0.5), q, l);
          if (p + G::NFR == 4) {
            projectFace<T, O, R, 0>(X + (2 - p) * G::nF, th, acc, dt * T(0.5), q, l);
            projectFace<T, O, R, 1>(X + (3 - p) * G::nF, th, acc, dt * T(0.5), q, l);
          }
          __syncthreads();
          for (int t = q; t < G::NFR * G::CW; t += 9) {
            const int i = t / G::CW, c = t - i * G::CW;
            const int f = (i + p + 2) & 3;
            halfTask<T, O, R>(a, X + i * G::nF, cV + f * 72 * E, f, c, l, e, r, half);
          }
        }
      }
    }
  }
  cpAsyncWait<0>();
}

// The pending surface integrals on their own (the closing half of a step): face holds the
// characteristics written for the elements by their neighbours, wOwn their own. Measured: 8.5 ms at
// 663,552 elements, order 5, 16 runs, FP32 (4,963 GB/s of its bytes, 0.75 of the copy rate).
template <typename T, int O, int R, bool LTS = false>
__global__ void __launch_bounds__(SGeo<T, O, R>::NT, SGeo<T, O, R>::ctasLift) kLift(const StepArgs<T> a) {
  using G = SGeo<T, O, R>;
  constexpr int B = G::B, E = G::E, SB = G::SB;
  extern __shared__ __align__(16) unsigned char smem[];
  T *const wt = reinterpret_cast<T *>(smem);
  T *const D = reinterpret_cast<T *>(smem + G::offDL);
  T *const bufU = reinterpret_cast<T *>(smem + (G::liftTile ? G::offCL : G::offDL));
  const int q = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int eo = l / R, r = l % R;
  const int64_t nGroups = (a.elCount + E - 1) / E;
  for (int64_t g = blockIdx.x; g < nGroups; g += gridDim.x) {
    const bool valid = g * E + eo < a.elCount;
    const int64_t e = valid ? a.elFirst + g * E + eo : a.elFirst;
    const int nv = int(min(a.elCount - g * E, int64_t(E)));
    if constexpr (G::liftTile) rowsIn<T, O, R, SB>(D, a.dofsE, a.elFirst + g * E, nv, q, l);
    if constexpr (G::smemU) issueFac<T, O, R, 0>(a, bufU, 0, FacL<0>::V, g, nGroups);
    cpAsyncCommit();
    const FacU<T, O, R, 0> su{G::smemU ? bufU + eo * G::W : facPtr<T, O, R, 0>(a.fac, e), q};
    RegU<T> ru;
    if constexpr (!G::smemU) {
#pragma unroll
      for (int f = 0; f < 4; f++) su(f, ru.u[f]);
    }
    liftRow<T, O, R, LTS>(a, a.face, wt, q, l, e, r, valid);
    if (q < 3) liftRow<T, O, R, LTS>(a, a.face, wt, q + 9, l, e, r, valid);
    cpAsyncWait<0>();
    __syncthreads();
    T acc[B];
    if constexpr (G::liftTile)
      ldRow<T, B>(rowPtr<T, SB>(D, q, l), acc);
    else
      ldRowG<T, B>(gRow<T, R, G::GB>(a.dofsE, e, 9, q, r), acc, valid);
    if constexpr (G::smemU)
      liftApply<T, O, R>(wt, su, l, acc);
    else
      liftApply<T, O, R>(wt, ru, l, acc);
    if constexpr (G::liftTile) {
      T *p = rowPtr<T, SB>(D, q, l);
      stRow<T, B>(p, acc);
#pragma unroll
      for (int n = B; n < G::GB; n++) p[n] = T(0);
      __syncwarp();
      rowsOut<T, O, R, SB>(D, a.dofsE, a.elFirst + g * E, nv, q, l);
    } else if (valid) {
      stRowG<T, B>(gRow<T, R, G::GB>(a.dofsE, e, 9, q, r), acc);
    }
    // every warp read the characteristics and U before the next group's arrive
    __syncthreads();
  }
}

}  // namespace edge_b200

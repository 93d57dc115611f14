// Halo exchange: the face rows that parts of a partition send each other (edge_b200_pack_faces,
// edge_b200_unpack_faces).
//
// A block has room for nine rows of face modes. Weak form: the projections, [9][R][GF], in
// configurations with pre-mixing already through the reader's flux solver fsE[1]. Strong form: three
// characteristic rows, [3][chunk][R][W], and a mark behind them. Each part takes the form that its own
// flux solvers allow, so a block can arrive in the other one. fsE[1] of the face between the parts is of
// rank 3 then (the strong part checked it), fsE[1] = r U (Q c) with the scales r, c and the row basis Q that
// both parts compute from the same 81 values (step_coef.cuh), and the rows follow from each other:
//   characteristics w = Q c P        projections whose fsE[1] P is the same: P = Q^T w / c
//   pre-mixed rows  N = r U w        characteristics w = U^+ (N / r)
#pragma once
#include "step_coef.cuh"

namespace edge_b200 {

constexpr uint4 kHaloMark = {0x7fa5c3e1u, 0x51e0c4a7u, 0x7fe1a5c3u, 0x0c4a751eu};
constexpr uint32_t kNoReader = 0xffffffffu;

// the rows of face slots (element * 4 + face) to a packed buffer with stride16 x 16 bytes per slot, 16
// bytes per thread; slots outside the face buffer are skipped
static __global__ void kFacePack(const uint4 *face, uint4 *buf, const int32_t *slots, int n, int64_t stride16,
                                 int64_t nSlots, bool strong) {
  const int64_t blk16 = strong ? stride16 / 3 : stride16, total = (int64_t)n * blk16;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t k = i / blk16, w = i % blk16;
    const int64_t sl = slots[k];
    if (sl < 0 || sl >= nSlots) continue;
    buf[k * stride16 + w] = face[sl * blk16 + w];
    if (strong && w == 0) buf[k * stride16 + blk16] = kHaloMark;
  }
}

// the face (element * 4 + face) that reads each slot, kNoReader where none does (set before)
static __global__ void kFaceReaders(const int32_t *elFaEl, const uint8_t *fId, const uint8_t *faType, int64_t nFaces,
                                    uint32_t *reader) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < nFaces; i += int64_t(gridDim.x) * blockDim.x)
    if (faType[i] == FT_INNER) reader[int64_t(elFaEl[i]) * 4 + fId[i]] = uint32_t(i);
}

// The way back, a warp per slot: a block of this part's form is copied, one of the other form turned
// into it through the reading face's fsE[1] (reader null: such blocks are skipped).
template <typename T>
__global__ void __launch_bounds__(kBuildWarps * 32)
    kFaceUnpack(uint4 *face, const uint4 *buf, const int32_t *slots, int n, int64_t stride16, int64_t nSlots, int R,
                bool strong, bool premix, const double *fsE, const uint32_t *reader) {
  __shared__ FaceTeam teams[kBuildWarps][kTeams + 1];
  __shared__ double mats[kBuildWarps][3][9];
  const int l = threadIdx.x & 31, wi = threadIdx.x >> 5, a = l % 9;  // (every nine lanes do the same)
  FaceTeam &t = teams[wi][l / 9];
  const int64_t blk16 = strong ? stride16 / 3 : stride16, row16 = stride16 / 9;
  for (int64_t k = int64_t(blockIdx.x) * kBuildWarps + wi; k < n; k += int64_t(gridDim.x) * kBuildWarps) {
    const int64_t sl = slots[k];
    if (sl < 0 || sl >= nSlots) continue;
    const uint4 *src = buf + k * stride16;
    uint4 *dst = face + sl * blk16;
    const uint4 m = src[stride16 / 3];
    const bool isStrong = m.x == kHaloMark.x && m.y == kHaloMark.y && m.z == kHaloMark.z && m.w == kHaloMark.w;
    if (isStrong == strong) {
      // six chunks a lane in flight: a block's 192 chunks at order 5 with 16 runs at once
      for (int64_t w0 = l; w0 < blk16; w0 += 6 * 32) {
        uint4 v[6];
#pragma unroll
        for (int i = 0; i < 6; i++)
          if (w0 + i * 32 < blk16) v[i] = src[w0 + i * 32];
#pragma unroll
        for (int i = 0; i < 6; i++)
          if (w0 + i * 32 < blk16) dst[w0 + i * 32] = v[i];
      }
      continue;
    }
    const uint32_t rd = reader ? reader[sl] : kNoReader;
    if (rd == kNoReader) continue;
    // the 3 x 9 matrix of the turn, entry (k, i): out_k = sum_i, or the other way out_i = sum_k
    double M[9], S[9], Q[3][9], u[3], g[3];
    const double *p = fsE + (nSlots + int64_t(rd)) * 81 + a * 9;
#pragma unroll
    for (int j = 0; j < 9; j++) M[j] = __ldg(p + j);
    const Scales sc = scales(t, a, M);
#pragma unroll
    for (int j = 0; j < 9; j++) S[j] = M[j] = M[j] / (sc.r(a) * sc.c(j));
    rowBasis(t, a, S, Q);
#pragma unroll
    for (int j = 0; j < 3; j++) {
      u[j] = g[j] = 0;
#pragma unroll
      for (int i = 0; i < 9; i++) {
        u[j] += M[i] * Q[j][i];
        if (i == a) g[j] = strong ? sc.c(i) * Q[j][i] : Q[j][i] / sc.c(i);
      }
      t.U[a][j] = u[j];
    }
    __syncwarp();
    if (premix && strong) {
      double A[3][9], Rm[3][3], b[3];
      qrU(t, A, Rm);
#pragma unroll
      for (int j = 0; j < 3; j++)
#pragma unroll
        for (int i = 0; i < 9; i++)
          if (i == a) b[j] = A[j][i] / sc.r(i);
      solveR(Rm, b, g);
    } else if (premix) {
#pragma unroll
      for (int j = 0; j < 3; j++) g[j] = sc.r(a) * u[j];
    }
    if (l < 9)
#pragma unroll
      for (int j = 0; j < 3; j++) mats[wi][j][a] = g[j];
    __syncwarp();
    constexpr int W = 16 / int(sizeof(T));
    const int CW = int(row16) / R;  // chunks of a row
    union Chunk {
      uint4 q;
      T v[W];
    };
    for (int i = l; i < int(row16); i += 32) {
      const int iw = i, is = (i % CW) * R + i / CW;  // the chunk in a weak-form and in a characteristic row
      if (strong) {
        double o[3][W] = {};
        for (int q = 0; q < 9; q++) {
          Chunk c;
          c.q = src[q * row16 + iw];
#pragma unroll
          for (int j = 0; j < 3; j++)
#pragma unroll
            for (int v = 0; v < W; v++) o[j][v] += mats[wi][j][q] * double(c.v[v]);
        }
#pragma unroll
        for (int j = 0; j < 3; j++) {
          Chunk c;
#pragma unroll
          for (int v = 0; v < W; v++) c.v[v] = T(o[j][v]);
          dst[j * row16 + is] = c.q;
        }
      } else {
        Chunk w[3];
#pragma unroll
        for (int j = 0; j < 3; j++) w[j].q = src[j * row16 + is];
        for (int q = 0; q < 9; q++) {
          Chunk c;
#pragma unroll
          for (int v = 0; v < W; v++) {
            double o = 0;
#pragma unroll
            for (int j = 0; j < 3; j++) o += mats[wi][j][q] * double(w[j].v[v]);
            c.v[v] = T(o);
          }
          dst[q * row16 + iw] = c.q;
        }
      }
    }
    __syncwarp();  // mats and the team are free for the next slot
  }
}

}  // namespace edge_b200

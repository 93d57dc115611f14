// KernelSet implementation for one configuration; included by the inst_*.cu translation units.
#pragma once
#include "kernel_set.h"
#include "step_visc.cuh"

namespace edge_b200 {

template <typename T, int O, int R, int RM>
class KernelSetImpl final : public KernelSet {
  using G = Geo<T, O, R, RM>;
  int numSms_ = 0, occLocal_ = 1, occNeigh_ = 1, occRecv_ = 1, occLocalLts_ = 1, occLocalSum_ = 1,
      occStep_ = 1, occLift_ = 1, capLocal_ = 0, capNeigh_ = 0;

  // attenuation: the strong-form step where the anelastic rows fit its shared memory
  static constexpr bool viscStrong = [] {
    if constexpr (RM == 3)
      return VGeo<T, O, R, RM>::ok;
    else
      return false;
  }();

  static StepArgs<T> cast(const StepArgsRaw &a) {
    StepArgs<T> b;
    b.dofsE = static_cast<T *>(a.dofsE);
    b.dofsA = static_cast<T *>(a.dofsA);
    b.tDofs = static_cast<T *>(a.tDofs);
    b.face = static_cast<T *>(a.face);
    b.starE = a.starE;
    b.starA = a.starA;
    b.srcA = a.srcA;
    b.fsE = a.fsE;
    b.fsA = a.fsA;
    b.elFaEl = a.elFaEl;
    b.fId = a.fId;
    b.vId = a.vId;
    b.faType = a.faType;
    b.nEl = a.nEl;
    b.elFirst = a.elFirst;
    b.elCount = a.elCount;
    b.dt = a.dt;
    for (int i = 0; i < 3; i++) b.omega[i] = a.omega[i];
    b.faceSum = static_cast<T *>(a.faceSum);
    b.faceHalf1 = static_cast<T *>(a.faceHalf1);
    b.faceHalf2 = static_cast<T *>(a.faceHalf2);
    b.ltsFlags = a.ltsFlags;
    b.ltsRel = a.ltsRel;
    b.sumIdx = a.sumIdx;
    b.halfIdx = a.halfIdx;
    b.firstTs = a.firstTs;
    b.fsLR = static_cast<const T *>(a.fsLR);
    b.fac = static_cast<const T *>(a.fac);
    b.gath = a.gath;
    b.wOwn = static_cast<T *>(a.wOwn);
    b.faceIn = static_cast<const T *>(a.faceIn);
    b.grpDt = a.grpDt;
    return b;
  }
  static constexpr size_t smemLocal() { return G::smemLocalGts; }
  static constexpr size_t smemNeigh() { return G::smemNeigh; }
  static constexpr size_t smemRecv() { return G::smemLocal; }

 public:
  cudaError_t init(int device) override {
    cudaError_t e;
    if ((e = cudaDeviceGetAttribute(&numSms_, cudaDevAttrMultiProcessorCount, device))) return e;
    if ((e = cudaFuncSetAttribute(kLocal<T, O, R, RM, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smemLocal())))
      return e;
    if ((e = cudaFuncSetAttribute(kNeigh<T, O, R, RM, G::premix>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smemNeigh())))
      return e;
    if ((e = cudaFuncSetAttribute(kRecv<T, O, R, RM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smemRecv())))
      return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occLocal_, kLocal<T, O, R, RM, 0>, G::NT, smemLocal())))
      return e;
    if constexpr (G::fuseWeak) {
      if ((e = cudaFuncSetAttribute(kLocal<T, O, R, RM, 0, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)smemLocal())) ||
          (e = cudaFuncSetAttribute(kRecv<T, O, R, RM, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)smemRecv())))
        return e;
    }
    if constexpr (viscStrong) {
      using V = VGeo<T, O, R, RM>;
      if ((e = cudaFuncSetAttribute(kStepVisc<T, O, R, RM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)V::smem)))
        return e;
      if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occStep_, kStepVisc<T, O, R, RM>, V::NT, V::smem))) return e;
      if ((e = cudaFuncSetAttribute(kLiftVisc<T, O, R, RM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)V::smemLift)))
        return e;
      if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occLift_, kLiftVisc<T, O, R, RM>, V::NT, V::smemLift)))
        return e;
      occStep_ = occStep_ < 1 ? 1 : occStep_;
      occLift_ = occLift_ < 1 ? 1 : occLift_;
    }
    if constexpr (RM == 0) {
      using S = SGeo<T, O, R>;
      if ((e = cudaFuncSetAttribute(kStep<T, O, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::smem)))
        return e;
      if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occStep_, kStep<T, O, R>, S::NT, S::smem))) return e;
      if ((e = cudaFuncSetAttribute(kLift<T, O, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::smemLift)))
        return e;
      if constexpr (G::ltsOk) {
        if ((e = cudaFuncSetAttribute(kStep<T, O, R, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::smem)) ||
            (e = cudaFuncSetAttribute(kStep<T, O, R, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::smem)) ||
            (e = cudaFuncSetAttribute(kLift<T, O, R, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)S::smemLift)))
          return e;
      }
      if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occLift_, kLift<T, O, R>, S::NT, S::smemLift))) return e;
      occStep_ = occStep_ < 1 ? 1 : occStep_;
      occLift_ = occLift_ < 1 ? 1 : occLift_;
    }
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occNeigh_, kNeigh<T, O, R, RM, G::premix>, G::NT, smemNeigh())))
      return e;
    if constexpr (G::premixLts != G::premix) {
      if ((e = cudaFuncSetAttribute(kNeigh<T, O, R, RM, G::premixLts>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)smemNeigh())))
        return e;
    }
    if constexpr (G::ltsOk) {
      if ((e = cudaFuncSetAttribute(kLocal<T, O, R, RM, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)G::smemLocalLts)))
        return e;
      if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occLocalLts_, kLocal<T, O, R, RM, 2>, G::NT,
                                                             G::smemLocalLts)))
        return e;
      occLocalLts_ = occLocalLts_ < 1 ? 1 : occLocalLts_;
      if ((e = cudaFuncSetAttribute(kLocal<T, O, R, RM, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)G::smemLocalSums)))
        return e;
      if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occLocalSum_, kLocal<T, O, R, RM, 1>, G::NT,
                                                             G::smemLocalSums)))
        return e;
      occLocalSum_ = occLocalSum_ < 1 ? 1 : occLocalSum_;
    }
    occLocal_ = occLocal_ < 1 ? 1 : occLocal_;
    occNeigh_ = occNeigh_ < 1 ? 1 : occNeigh_;
    return cudaSuccess;
  }
  int elementsPerCta() const override { return G::E; }
  int ctasLocal(bool strong) const override {
    return capLocal_ > 0 ? capLocal_ : numSms_ * (strong ? occStep_ : occLocal_);
  }
  int ctasNeigh(bool strong) const override {
    return capNeigh_ > 0 ? capNeigh_ : numSms_ * (strong ? occLift_ : occNeigh_);
  }
  void setGridCaps(int local, int neigh) override {
    capLocal_ = local;
    capNeigh_ = neigh;
  }

  static int grid(int64_t nEl, int cap) {
    int64_t groups = (nEl + G::E - 1) / G::E;
    return (int)(groups < cap ? (groups < 1 ? 1 : groups) : cap);
  }

  cudaError_t local(const StepArgsRaw &a, cudaStream_t s) override {
    if (a.elCount < 1) return cudaSuccess;
    if constexpr (viscStrong) {
      using V = VGeo<T, O, R, RM>;
      if (a.fac) {
        kStepVisc<T, O, R, RM>
            <<<grid(a.elCount, ctasLocal(true)), V::NT, V::smem, s>>>(cast(a));
        return cudaGetLastError();
      }
    }
    if constexpr (RM == 0) {
      using S = SGeo<T, O, R>;
      if (a.fac) {
        kStep<T, O, R><<<grid(a.elCount, ctasLocal(true)), S::NT, S::smem, s>>>(cast(a));
        return cudaGetLastError();
      }
    }
    if constexpr (G::fuseWeak) {
      if (a.faceIn) {
        kLocal<T, O, R, RM, 0, true><<<grid(a.elCount, ctasLocal(false)), G::NT, smemLocal(), s>>>(cast(a));
        return cudaGetLastError();
      }
    }
    kLocal<T, O, R, RM, 0><<<grid(a.elCount, ctasLocal(false)), G::NT, smemLocal(), s>>>(cast(a));
    return cudaGetLastError();
  }
  bool strongSupported() const override { return RM == 0 || viscStrong; }
  bool strongLts() const override { return RM == 0 && G::ltsOk; }
  cudaError_t localLts(const StepArgsRaw &a, cudaStream_t s) override {
    if constexpr (G::ltsOk) {
      if (a.elCount < 1) return cudaSuccess;
      if constexpr (RM == 0) {
        using S = SGeo<T, O, R>;
        if (a.fac) {
          kStep<T, O, R, 2><<<grid(a.elCount, numSms_), S::NT, S::smem, s>>>(cast(a));
          return cudaGetLastError();
        }
      }
      kLocal<T, O, R, RM, 2><<<grid(a.elCount, numSms_ * occLocalLts_), G::NT, G::smemLocalLts, s>>>(cast(a));
      return cudaGetLastError();
    } else {
      return cudaErrorNotSupported;
    }
  }
  cudaError_t localLtsSums(const StepArgsRaw &a, cudaStream_t s) override {
    if constexpr (G::ltsOk) {
      if (a.elCount < 1) return cudaSuccess;
      if constexpr (RM == 0) {
        using S = SGeo<T, O, R>;
        if (a.fac) {
          kStep<T, O, R, 1><<<grid(a.elCount, numSms_ * occStep_), S::NT, S::smem, s>>>(cast(a));
          return cudaGetLastError();
        }
      }
      kLocal<T, O, R, RM, 1><<<grid(a.elCount, numSms_ * occLocalSum_), G::NT, G::smemLocalSums, s>>>(cast(a));
      return cudaGetLastError();
    } else {
      return cudaErrorNotSupported;
    }
  }
  bool ltsSupported() const override { return G::ltsOk; }
  bool premix() const override { return G::premix; }
  bool fuseWeak() const override { return G::fuseWeak; }
  int fsPairStride() const override { return G::FSP; }
  cudaError_t neigh(const StepArgsRaw &a, cudaStream_t s) override {
    if (a.elCount < 1) return cudaSuccess;
    if constexpr (viscStrong) {
      using V = VGeo<T, O, R, RM>;
      if (a.fac) {
        kLiftVisc<T, O, R, RM>
            <<<grid(a.elCount, ctasNeigh(true)), V::NT, V::smemLift, s>>>(cast(a));
        return cudaGetLastError();
      }
    }
    if constexpr (RM == 0) {
      using S = SGeo<T, O, R>;
      if (a.fac) {
        kLift<T, O, R><<<grid(a.elCount, ctasNeigh(true)), S::NT, S::smemLift, s>>>(cast(a));
        return cudaGetLastError();
      }
    }
    kNeigh<T, O, R, RM, G::premix><<<grid(a.elCount, ctasNeigh(false)), G::NT, smemNeigh(), s>>>(cast(a));
    return cudaGetLastError();
  }
  cudaError_t neighLts(const StepArgsRaw &a, cudaStream_t s) override {
    if (a.elCount < 1) return cudaSuccess;
    if constexpr (RM == 0 && G::ltsOk) {
      using S = SGeo<T, O, R>;
      if (a.fac) {
        kLift<T, O, R, true><<<grid(a.elCount, numSms_ * occLift_), S::NT, S::smemLift, s>>>(cast(a));
        return cudaGetLastError();
      }
    }
    kNeigh<T, O, R, RM, G::premixLts><<<grid(a.elCount, ctasNeigh(false)), G::NT, smemNeigh(), s>>>(cast(a));
    return cudaGetLastError();
  }
  cudaError_t recv(const StepArgsRaw &a, const RecvArgs &r, cudaStream_t s) override {
    const int g = (r.nGrp + G::E - 1) / G::E;
    if (g == 0) return cudaSuccess;
    if constexpr (G::fuseWeak) {
      if (a.faceIn && !a.fac) {
        kRecv<T, O, R, RM, true><<<g, G::NT, smemRecv(), s>>>(cast(a), r);
        return cudaGetLastError();
      }
    }
    kRecv<T, O, R, RM><<<g, G::NT, smemRecv(), s>>>(cast(a), r);
    return cudaGetLastError();
  }
  cudaError_t sources(void *dofsE, const SrcArgs &sa, cudaStream_t s) override {
    if (sa.nGrp == 0) return cudaSuccess;
    kSources<T, O, R><<<sa.nGrp, 128, 0, s>>>(static_cast<T *>(dofsE), sa);
    return cudaGetLastError();
  }
};

}  // namespace edge_b200

// registry of one translation unit: a function returning the matching configuration
#define EDGE_B200_CFG(T, O, R, RM, prec)                                    \
  if (precision == prec && order == O && runs == R && rms == RM)           \
    return new edge_b200::KernelSetImpl<T, O, R, RM>();

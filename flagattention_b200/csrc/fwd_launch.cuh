// Host launcher for one head dimension of the forward kernel; each fwd_d*.cu instantiates one D
// so the variants compile in parallel.
#pragma once
#include "fwd_kernel.cuh"
#include "fwd_solo.cuh"

namespace b200attn {

struct FwdLaunch {
  CUtensorMap tmQ, tmK, tmV, tmO;  // tmO only when args.o_tma
  FwdArgs args;
  dim3 grid;
  bool bf16, dropout;
  bool solo = false;     // D <= 64, plain mode, 16-bit output: one query tile per block (fwd_solo.cuh)
  bool split64 = false;  // D = 128, plain mode: the 64-key softmax pipeline (fwd_kernel's SPLIT64)
  cudaStream_t stream;
};

template <int D, bool BF16, bool DROPOUT, bool SPLIT64 = false, bool MERGE = false>
int launch_fwd_variant(const FwdLaunch& L) {
  auto kernel = fwd_kernel<D, BF16, DROPOUT, SPLIT64, MERGE>;
  constexpr int smem_max = FwdSmem<D>::TOTAL > FwdSmem<D>::DUAL_TOTAL ? FwdSmem<D>::TOTAL : FwdSmem<D>::DUAL_TOTAL;
  const int smem = L.args.dual_stream ? FwdSmem<D>::DUAL_TOTAL : FwdSmem<D>::TOTAL;
  static PerDeviceOnce attr_once;  // one per kernel variant
  const int rc = attr_once.run([&]() -> int {
    B200ATTN_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max));
    return B200ATTN_OK;
  });
  if (rc) return rc;
  return launch(CHAINED, kernel, L.grid, 384, smem, L.stream, L.tmQ, L.tmK, L.tmV, L.tmO, L.args);
}

template <int D, bool BF16, bool DROPOUT>
int launch_fwd_solo_variant(const FwdLaunch& L) {
  auto kernel = fwd_solo_kernel<D, BF16, DROPOUT>;
  static PerDeviceOnce attr_once;  // one per kernel variant
  const int rc = attr_once.run([&]() -> int {
    B200ATTN_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SoloSmem<D>::TOTAL));
    return B200ATTN_OK;
  });
  if (rc) return rc;
  return launch(CHAINED, kernel, L.grid, SoloSmem<D>::THREADS, SoloSmem<D>::TOTAL, L.stream, L.tmQ, L.tmK, L.tmV, L.tmO, L.args);
}

template <int D>
int launch_fwd_d(const FwdLaunch& L) {
  if (L.args.merge_o != nullptr) {  // (no dropout; D = 128 always with a band here)
    return L.bf16 ? launch_fwd_variant<D, true, false, D == 128, true>(L) : launch_fwd_variant<D, false, false, D == 128, true>(L);
  }
  if constexpr (D <= 64) {
    if (L.solo) {
      if (L.bf16) return L.dropout ? launch_fwd_solo_variant<D, true, true>(L) : launch_fwd_solo_variant<D, true, false>(L);
      return L.dropout ? launch_fwd_solo_variant<D, false, true>(L) : launch_fwd_solo_variant<D, false, false>(L);
    }
  }
  if constexpr (D == 128) {
    if (L.split64) {
      if (L.bf16) return L.dropout ? launch_fwd_variant<D, true, true, true>(L) : launch_fwd_variant<D, true, false, true>(L);
      return L.dropout ? launch_fwd_variant<D, false, true, true>(L) : launch_fwd_variant<D, false, false, true>(L);
    }
  }
  if (L.bf16) {
    return L.dropout ? launch_fwd_variant<D, true, true>(L) : launch_fwd_variant<D, true, false>(L);
  }
  return L.dropout ? launch_fwd_variant<D, false, true>(L) : launch_fwd_variant<D, false, false>(L);
}

int launch_fwd_d16(const FwdLaunch& L);
int launch_fwd_d32(const FwdLaunch& L);
int launch_fwd_d64(const FwdLaunch& L);
int launch_fwd_d128(const FwdLaunch& L);

}  // namespace b200attn

// pass_kernel.cuh -- the per-pass kernel template and its launcher, shared by
// kernels.cu (complex operators) and kernels_real.cu (real operators).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "kernels.h"
#include "pass.h"
#include "pass_device.cuh"
#include "per_context.h"

namespace dmg {

// One pass over the whole state or (HALF, pass.h) half of it: the block stages
// the pass's tables once, then grid-strides over the tiles.  Two instances: with
// the half range's tile numbering in it, a pass of a state that fits a few blocks
// took 2 to 3 % longer (5 to 9 qubits, launch and latency).
template <typename T, int K, int CLS, bool HALF>
__global__ void __launch_bounds__(kThreads) k_pass(T* __restrict__ re, T* __restrict__ im,
                                                   const PassDesc<K>* __restrict__ dp,
                                                   const HalfMap* __restrict__ half, const int* __restrict__ herm) {
  constexpr int D = 1 << K;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const PassHeader& h = dp->h;
  const HalfMap* hm = HALF && *herm ? half : nullptr;
  const uint64_t ntiles = hm ? hm->count : h.ntiles;
  const int tile = (1 << h.g) * D * D;
  T* sre = reinterpret_cast<T*>(smem_raw);
  T* sim = sre + tile;
  auto& tb = *reinterpret_cast<PassTables<T, K, CLS>*>(smem_raw + ((2 * (size_t)tile * sizeof(T) + 15) & ~(size_t)15));
  load_tables<T, K, CLS>(dp, tb);
  __syncthreads();
  pdl_wait();
  pdl_begin();
  // Full-size tiles of narrow passes (2^(K-1) entry pairs per thread): the
  // next tile's loads go out before the current tile is transformed.
  constexpr int P = K >= 1 ? 1 << (K - 1) : 1;
  if constexpr ((K >= 1 && K <= 2) || (std::is_same<T, float>::value && base_class(CLS) == CLS_DENSE)) {
    if (tile == 2 * kThreads * P) {
      uint64_t t = blockIdx.x;
      if (t >= ntiles) return;
      TileRegs<T, P> x;
      const int lf = free_offset(h);
      uint64_t base = tile_base(h, hm, t);
      load_regs<T, K, CLS, P>(re, im, h, tb, base, x);
      for (; t < ntiles; t += gridDim.x) {
        regs_to_smem<T, K, CLS, P>(h, tb, x, sre, sim);
        __syncthreads();
        const uint64_t tn = t + gridDim.x;
        const uint64_t base_n = tn < ntiles ? tile_base(h, hm, tn) : 0;
        if (tn < ntiles) load_regs<T, K, CLS, P>(re, im, h, tb, base_n, x);
        tile_body<T, K, CLS>(re, im, h, tb, base, sre, sim, lf);
        base = base_n;
      }
      return;
    }
  }
  for (uint64_t t = blockIdx.x; t < ntiles; t += gridDim.x) run_tile<T, K, CLS>(re, im, h, tb, tile_base(h, hm, t), sre, sim);
}

// ---------------------------------------------------------------- launchers
// Dynamic shared memory for the largest tile, and the largest shared-memory
// carveout so that the resident-block count the occupancy query reports is
// the one the launches get.
template <typename T, int K, int CLS, bool HALF>
inline cudaError_t configure_pass() {
  constexpr int D = 1 << K;
  cudaError_t e = cudaFuncSetAttribute(k_pass<T, K, CLS, HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)pass_smem_bytes<T, K, CLS>(kThreads * D));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_pass<T, K, CLS, HALF>, cudaFuncAttributePreferredSharedMemoryCarveout,
                             (int)cudaSharedmemCarveoutMaxShared);
  return e;
}

// Whether a class has a half-range instance: complex64 passes run whole, and so
// do the monomial ones of 2 qubits and more, but on the pipelined kernel.
template <typename T, int K, int CLS>
constexpr bool half_instance() {
  constexpr int C = base_class(CLS);
  if (std::is_same<T, float>::value || C == CLS_RLIN) return false;
  return K == 1 || C == CLS_DENSE || C == CLS_SPARSE || C == CLS_SUPER;
}

template <typename T, int K, int CLS, bool HALF = false>
inline cudaError_t launch_one(const LaunchArgs& a, cudaStream_t s) {
  if constexpr (!HALF) {
    if (a.half) {
      if constexpr (half_instance<T, K, CLS>()) return launch_one<T, K, CLS, true>(a, s);
      else return cudaErrorInvalidValue;
    }
  }
  const size_t smem = pass_smem_bytes<T, K, CLS>(a.tile_entries);
  static PerContext configured;  // per instance
  const cudaError_t e = configured.get([](int*) { return configure_pass<T, K, CLS, HALF>(); });
  if (e != cudaSuccess) return e;
  return launch_kernel(a.pdl, k_pass<T, K, CLS, HALF>, a.grid, kThreads, smem, s, static_cast<T*>(a.re),
                       static_cast<T*>(a.im), static_cast<const PassDesc<K>*>(a.desc), a.half, a.herm);
}

}  // namespace dmg

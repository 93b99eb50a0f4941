// kernels_mono.cu -- monomial passes of 2 to 4 qubits (MOVE, SIGNED, PHASE) on
// states of many tiles: out[a][b] = f[a][b] in[src a][srcb b].
//
// A PHASE pass is bound by GB300's FP64 pipe (four operations an entry: 8200
// cycles a 4-qubit tile on an SM, against 5700 for its bytes at HBM's rate), a
// MOVE or SIGNED pass by HBM, so loads, arithmetic and stores have to run at
// the same time.  One persistent block per SM (two for K = 2, 3) keeps several
// tiles in flight: 16-byte asynchronous copies bring a tile's touched runs into
// a ring of shared-memory stages, one barrier a tile; every thread then takes
// the same positions of each tile, so the shared-memory offsets of their
// sources, the factors and the global offsets are found once per pass and stay
// in registers, and the results go straight from registers to memory.  The
// tiled kernel (pass_kernel.cuh) loads, waits, transforms and stores, and looks
// the factors up for every entry; it stays for states of few tiles.  Measured,
// before and after: 15 qubits, 4-qubit PHASE (half range, FP64) 5.8 -> 4.5 ms with
// the mirrors, 3.9 the FP64 pipe alone; 14 qubits 1.41 -> 1.15 ms; 14-qubit SIGNED
// 1.19 -> 0.93 ms (7.5 TB/s); 13-qubit CX 201 -> 176 us; complex64 at 15 qubits
// 4.45 -> 2.82 ms (6.0 TB/s).
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.h"
#include "pass_device.cuh"
#include "per_context.h"
#include "tc.cuh"

namespace dmg {

namespace {

template <typename T, int K>
struct Mono {
  static constexpr int D = 1 << K, TILE = 256 << K;         // entries of a full tile
  static constexpr int V = 16 / (int)sizeof(T);             // entries of a 16-byte chunk
  static constexpr int NT = K <= 3 ? 256 : 512;             // threads
  static constexpr int P = TILE / V / NT;                   // chunks a thread takes
  static constexpr int STAGE = 2 * TILE * (int)sizeof(T);   // bytes, re then im
  static constexpr int ROOM = K <= 3 ? 98304 : 196608;      // two blocks per SM, or one
  static constexpr int ST = ROOM / STAGE < 6 ? ROOM / STAGE : 6;
  static_assert(P >= 1 && P * V * NT == TILE && ST >= 3, "tile split");
};

// Position of entry s of a stage: its 16-byte chunks XORed within the 128-byte
// row by the row's low bits (linear over GF(2), as tile_sw).
template <int V>
__device__ __forceinline__ int chunk_sw(int s) {
  const int q = s / V;
  return (q ^ ((q >> 3) & 7)) * V + (s & (V - 1));
}

template <int K>
__device__ __forceinline__ int deposit(int x, const int32_t* pos) {
  int r = 0;
#pragma unroll
  for (int i = 0; i < K; i++) r |= ((x >> i) & 1) << pos[i];
  return r;
}

template <typename T>
struct alignas(16) Chunk {
  T v[16 / sizeof(T)];
};

// c ? a : b, its sign flipped if neg.  Integer words: a select of doubles
// takes the FP64 pipe.
__device__ __forceinline__ double pick(bool c, double a, double b, bool neg) {
  const int h = c ? __double2hiint(a) : __double2hiint(b), l = c ? __double2loint(a) : __double2loint(b);
  return __hiloint2double(h ^ (neg ? (int)0x80000000 : 0), l);
}
__device__ __forceinline__ float pick(bool c, float a, float b, bool neg) {
  const float x = c ? a : b;
  return neg ? flip(x) : x;
}
__device__ __forceinline__ df64 pick(bool c, df64 a, df64 b, bool neg) {
  return df64(pick(c, a.hi, b.hi, neg), pick(c, a.lo, b.lo, neg));
}

template <typename T, int K, int CLS>
__global__ void __launch_bounds__(Mono<T, K>::NT, K <= 3 ? 2 : 1)
    k_mono(T* __restrict__ re, T* __restrict__ im, const PassDesc<K>* __restrict__ dp,
           const HalfMap* __restrict__ half, const int* __restrict__ herm) {
  using M = Mono<T, K>;
  constexpr int V = M::V, P = M::P, NT = M::NT, ST = M::ST;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t s_base[ST];
  const PassHeader& h = dp->h;
  const int tid = threadIdx.x, L = h.L;
  const HalfMap* hm = half && *herm ? half : nullptr;
  const uint64_t ntiles = hm ? hm->count : h.ntiles;

  // ---- this thread's positions of every tile
  uint64_t goff[P];
  int src[P][V];                 // shared-memory positions of the sources
  T fr[P][V], fi[P][V];          // factors (PHASE)
  uint32_t kinds = 0, ld = 0, st = 0;
#pragma unroll
  for (int c = 0; c < P; c++) {
    const int e = V * (tid + NT * c), run = e >> L;
    uint64_t off = (uint64_t)(e & ((1 << L) - 1));
    for (int j = 0; j < h.mhi; j++) off |= (uint64_t)((run >> j) & 1) << h.hipos[j];
    goff[c] = off;
    ld |= ((h.ldmask[run >> 5] >> (run & 31)) & 1u) << c;
    st |= ((h.stmask[run >> 5] >> (run & 31)) & 1u) << c;
#pragma unroll
    for (int u = 0; u < V; u++) {
      const int loc = e + u, a = pext_local<K>(loc, h.lket), b = pext_local<K>(loc, h.lbra);
      const int sa = dp->op.src[a], sb = dp->op.srcb[b];
      src[c][u] = chunk_sw<V>(loc ^ deposit<K>(a ^ sa, h.lket) ^ deposit<K>(b ^ sb, h.lbra));
      if (CLS != CLS_MOVE) kinds |= (uint32_t)dp->op.fk[a * M::D + b] << (3 * (c * V + u));
      if (CLS == CLS_PHASE) {
        fr[c][u] = coef<T>(dp->op.fre[a * M::D + b]);
        fi[c][u] = coef<T>(dp->op.fim[a * M::D + b]);
      }
    }
  }

  // A diagonal operator: a thread reads what it copied itself, and its warps
  // need not meet the others at all.
  bool diag = true;
#pragma unroll
  for (int a = 0; a < M::D; a++) diag = diag && dp->op.src[a] == a && dp->op.srcb[a] == a;

  auto load = [&](uint64_t t, int stage) {
    if (t < ntiles) {
      const uint64_t base = tile_base(h, hm, t);
      T* s = reinterpret_cast<T*>(smem + stage * M::STAGE);
#pragma unroll
      for (int c = 0; c < P; c++)
        if ((ld >> c) & 1) {
          const int q = chunk_sw<V>(V * (tid + NT * c));
          tc::cp_async16(s + q, re + base + goff[c]);
          tc::cp_async16(s + M::TILE + q, im + base + goff[c]);
        }
      if (tid == 0) s_base[stage] = base;
    }
    tc::cp_async_commit();
  };

  pdl_wait();
  pdl_begin();
  uint64_t t = blockIdx.x;
#pragma unroll
  for (int s = 0; s < ST - 1; s++) load(t + (uint64_t)s * gridDim.x, s);
  int stage = 0;
  for (; t < ntiles; t += gridDim.x) {
    tc::cp_async_wait<ST - 2>();
    if (!diag) __syncthreads();  // the stage is complete for all, and all are done with the one before it
    load(t + (uint64_t)(ST - 1) * gridDim.x, stage == 0 ? ST - 1 : stage - 1);
    const uint64_t base = diag ? tile_base(h, hm, t) : s_base[stage];
    const T* sre = reinterpret_cast<const T*>(smem + stage * M::STAGE);
    const T* sim = sre + M::TILE;
#pragma unroll
    for (int c = 0; c < P; c++) {
      if (!((st >> c) & 1)) continue;
      Chunk<T> wr, wi;
#pragma unroll
      for (int u = 0; u < V; u++) {
        const T vr = sre[src[c][u]], vi = sim[src[c][u]];
        const uint32_t fk = CLS == CLS_MOVE ? (uint32_t)FK_ONE : (kinds >> (3 * (c * V + u))) & 7u;
        if (CLS == CLS_PHASE && fk == FK_GEN) {
          wr.v[u] = madd(fr[c][u], vr, -fi[c][u] * vi);
          wi.v[u] = madd(fr[c][u], vi, fi[c][u] * vr);
        } else if (CLS == CLS_MOVE || (CLS == CLS_PHASE && fk == FK_ONE)) {
          wr.v[u] = vr;
          wi.v[u] = vi;
        } else {  // -x, i x = -vi + i vr, -i x = vi - i vr
          const bool swap = fk == FK_PI || fk == FK_NI;
          wr.v[u] = pick(swap, vi, vr, fk == FK_NEG || fk == FK_PI);
          wi.v[u] = pick(swap, vr, vi, fk == FK_NEG || fk == FK_NI);
        }
      }
      __stcg(reinterpret_cast<float4*>(re + base + goff[c]), *reinterpret_cast<const float4*>(&wr));
      __stcg(reinterpret_cast<float4*>(im + base + goff[c]), *reinterpret_cast<const float4*>(&wi));
    }
    stage = stage + 1 == ST ? 0 : stage + 1;
  }
  tc::cp_async_wait<0>();
}

template <typename T, int K, int CLS>
cudaError_t launch_mono_one(const LaunchArgs& a, cudaStream_t s) {
  using M = Mono<T, K>;
  constexpr int smem = M::ST * M::STAGE;
  static PerContext configured;  // per instance
  const cudaError_t e = configured.get([](int*) {
    cudaError_t c = cudaFuncSetAttribute(k_mono<T, K, CLS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (c == cudaSuccess)
      c = cudaFuncSetAttribute(k_mono<T, K, CLS>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               (int)cudaSharedmemCarveoutMaxShared);
    return c;
  });
  if (e != cudaSuccess) return e;
  return launch_kernel(a.pdl, k_mono<T, K, CLS>, a.grid, M::NT, smem, s, static_cast<T*>(a.re), static_cast<T*>(a.im),
                       static_cast<const PassDesc<K>*>(a.desc), a.half, a.herm);
}

template <typename T, int K>
cudaError_t launch_mono_k(const LaunchArgs& a, cudaStream_t s) {
  switch (a.cls) {
    case CLS_MOVE: return launch_mono_one<T, K, CLS_MOVE>(a, s);
    case CLS_SIGNED: return launch_mono_one<T, K, CLS_SIGNED>(a, s);
    case CLS_PHASE: return launch_mono_one<T, K, CLS_PHASE>(a, s);
    default: return cudaErrorInvalidValue;
  }
}

template <typename T>
cudaError_t launch_mono_t(const LaunchArgs& a, cudaStream_t s) {
  switch (a.K) {
    case 2: return launch_mono_k<T, 2>(a, s);
    case 3: return launch_mono_k<T, 3>(a, s);
    case 4: return launch_mono_k<T, 4>(a, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

// A tile for every block: at 10 qubits (1024 tiles) a CX takes 12.0 us, 12.4 on
// the tiled kernel; below, blocks would find their positions for no tile.
unsigned mono_grid(int K, int cls, int tile_entries, uint64_t ntiles, int sms) {
  if (K < 2 || K > 4 || tile_entries != 256 << K) return 0;
  if (cls != CLS_MOVE && cls != CLS_SIGNED && cls != CLS_PHASE) return 0;
  const uint64_t cap = (uint64_t)sms * (K <= 3 ? 2 : 1);
  return ntiles >= cap ? (unsigned)cap : 0;
}

cudaError_t launch_mono(const LaunchArgs& a, cudaStream_t s) {
  if (a.arith == AR_DF64) return launch_mono_t<df64>(a, s);
  return a.fp32 ? launch_mono_t<float>(a, s) : launch_mono_t<double>(a, s);
}

}  // namespace dmg

// kernels.cu -- the superoperator pass kernels of the GB300 density-matrix engine.
//
// One kernel template (pass_kernel.cuh) covers every FP32-pipe / FP64 pass:
// element type T (double, float, or double-float pairs), width K (1..4 qubits)
// and arithmetic class (pass.h); the real-operator instances live in
// kernels_real.cu and the tensor-core passes in tensor.cu.  A block owns one tile at a time
// (grid-stride over tiles): it loads the tile's touched runs with 16-byte
// vector loads into shared memory, transforms them, and stores them back.
// Monomial classes (MOVE/SIGNED/PHASE) fuse the permutation and the per-entry
// factor into the store, so they cost no FP64 arithmetic beyond one complex
// multiply (PHASE) and never more than one HBM read and write per entry.
// DENSE/SPARSE apply U to the ket bits of each column and V to the bra bits
// of each row; V = conj(U) makes the pass U (x) conj(U) on the 2K target bits,
// V = I makes it a ket-only pass (the reference's forward/backward stages).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "kernels.h"
#include "pass.h"
#include "pass_device.cuh"
#include "pass_kernel.cuh"

namespace dmg {

// 3- and 4-qubit SPARSE passes of complex64 states run as dense ones: on the
// FP32 pipe a dense row is 4 * 2^K multiply-adds fed by 16-byte broadcast
// coefficient loads, where the sparse row walk costs several dependent
// shared-memory loads per nonzero and runs slower at every density these
// fused blocks have; the runs that such a pass does not load count as zeros
// (kZeroUnloaded).  (FP64 and double-float keep the sparse walk: their
// multiply-adds, not the loads, bound them.)
template <typename T, int K>
constexpr bool sparse_as_dense() {
  return std::is_same<T, float>::value && K >= 3;
}

template <typename T, int K>
static cudaError_t launch_k(const LaunchArgs& a, cudaStream_t s) {
  switch (a.cls) {
    case CLS_MOVE: return launch_one<T, K, CLS_MOVE>(a, s);
    case CLS_SIGNED: return launch_one<T, K, CLS_SIGNED>(a, s);
    case CLS_PHASE: return launch_one<T, K, CLS_PHASE>(a, s);
    case CLS_DENSE:
      if (a.real && K <= 2) return launch_pass_real(a, s);
      return launch_one<T, K, CLS_DENSE>(a, s);
    case CLS_SPARSE:
      if (a.real && K <= 2) return launch_pass_real(a, s);
      if (sparse_as_dense<T, K>()) return launch_one<T, K, CLS_DENSE>(a, s);
      return launch_one<T, K, CLS_SPARSE>(a, s);
    case CLS_RLIN:
      if (K == 1) return launch_one<T, 1, CLS_RLIN>(a, s);
      return cudaErrorInvalidValue;
    case CLS_SUPER:
      if (K == 1) return launch_one<T, 1, CLS_SUPER>(a, s);
      if (K == 2) return launch_one<T, 2, CLS_SUPER>(a, s);
      return cudaErrorInvalidValue;
    default: return cudaErrorInvalidValue;
  }
}

template <typename T>
static cudaError_t launch_t(const LaunchArgs& a, cudaStream_t s) {
  switch (a.K) {
    case 1: return launch_k<T, 1>(a, s);
    case 2: return launch_k<T, 2>(a, s);
    case 3: return launch_k<T, 3>(a, s);
    case 4: return launch_k<T, 4>(a, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_pass(const LaunchArgs& a, cudaStream_t s) {
  if (a.tc) {
    if (a.arith == AR_FP64) return launch_pass_tc64(a, s);
    if (a.arith == AR_FP32) return launch_pass_tc32(a, s);
    return launch_pass_tc(a, s);
  }
  if (a.direct1) return launch_pass1(a, s);
  if (a.mono) return launch_mono(a, s);
  if (a.arith == AR_DF64) return launch_t<df64>(a, s);
  return a.fp32 ? launch_t<float>(a, s) : launch_t<double>(a, s);
}

template <typename T, int K, int CLS>
static cudaError_t occ_query(int* blocks) {
  constexpr int D = 1 << K;
  int nb = 0;
  const size_t smem = pass_smem_bytes<T, K, CLS>(kThreads * D);
  cudaError_t e = configure_pass<T, K, CLS, false>();
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_pass<T, K, CLS, false>, kThreads, smem);
  *blocks = nb > 0 ? nb : 1;
  return e;
}
// Asked once per instance and context: an upload asks for every pass, and the
// attribute calls and the query took 6 us each time.
template <typename T, int K, int CLS>
static int occ_one() {
  static PerContext occ;
  int nb = 1;
  return occ.get(occ_query<T, K, CLS>, &nb) == cudaSuccess ? nb : 1;
}

template <typename T, int K>
static int occ_k(int cls) {
  switch (cls) {
    case CLS_MOVE: return occ_one<T, K, CLS_MOVE>();
    case CLS_SIGNED: return occ_one<T, K, CLS_SIGNED>();
    case CLS_PHASE: return occ_one<T, K, CLS_PHASE>();
    case CLS_DENSE: return occ_one<T, K, CLS_DENSE>();
    case CLS_SPARSE: return sparse_as_dense<T, K>() ? occ_one<T, K, CLS_DENSE>() : occ_one<T, K, CLS_SPARSE>();
    case CLS_SUPER: return K <= 1 ? occ_one<T, 1, CLS_SUPER>() : occ_one<T, 2, CLS_SUPER>();
    default: return occ_one<T, 1, CLS_RLIN>();
  }
}

int pass_blocks_per_sm(int K, int cls, int arith) {
  if (arith == AR_FP32) {
    switch (K) { case 1: return occ_k<float, 1>(cls); case 2: return occ_k<float, 2>(cls); case 3: return occ_k<float, 3>(cls); default: return occ_k<float, 4>(cls); }
  }
  if (arith == AR_DF64) {
    switch (K) { case 1: return occ_k<df64, 1>(cls); case 2: return occ_k<df64, 2>(cls); case 3: return occ_k<df64, 3>(cls); default: return occ_k<df64, 4>(cls); }
  }
  switch (K) { case 1: return occ_k<double, 1>(cls); case 2: return occ_k<double, 2>(cls); case 3: return occ_k<double, 3>(cls); default: return occ_k<double, 4>(cls); }
}

// ---------------------------------------------------------------- df64 format
// In place, once per fused run: each FP64 entry becomes the double-float pair
// (hi, lo) = (round(x), round(x - hi)) in the same 8 bytes, and back.  GB300's FP64
// pipe, conversions included, bounds these (four and three operations a number),
// so floats are widened by integer work: three operations and one.  13 qubits, both
// ways with the run's last mirror: 1910 -> 1500 us.
__device__ __forceinline__ double widen(float f) {
  const uint32_t u = __float_as_uint(f), e = u & 0x7F800000u;
  if (e == 0 || e == 0x7F800000u) return (u << 1) == 0 ? __hiloint2double((int)u, 0) : (double)f;  // zeros; the rest is rare
  return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7FFFFFFFu) >> 3) + 0x38000000u)), (int)(u << 29));
}
__device__ __forceinline__ df64 narrow(double x) {
  const float hi = __double2float_rn(x);
  return df64(hi, __double2float_rn(x - widen(hi)));
}
__global__ void k_to_df64(double2* __restrict__ re, double2* __restrict__ im, uint64_t pairs) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < pairs; i += (uint64_t)gridDim.x * blockDim.x) {
    const double2 a = re[i], b = im[i];
    const df64 a0 = narrow(a.x), a1 = narrow(a.y), b0 = narrow(b.x), b1 = narrow(b.y);
    reinterpret_cast<float4*>(re)[i] = make_float4(a0.hi, a0.lo, a1.hi, a1.lo);
    reinterpret_cast<float4*>(im)[i] = make_float4(b0.hi, b0.lo, b1.hi, b1.lo);
  }
}
__global__ void k_from_df64(double2* __restrict__ re, double2* __restrict__ im, uint64_t pairs) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < pairs; i += (uint64_t)gridDim.x * blockDim.x) {
    const float4 a = reinterpret_cast<const float4*>(re)[i], b = reinterpret_cast<const float4*>(im)[i];
    re[i] = make_double2(widen(a.x) + widen(a.y), widen(a.z) + widen(a.w));
    im[i] = make_double2(widen(b.x) + widen(b.y), widen(b.z) + widen(b.w));
  }
}
cudaError_t launch_to_df64(void* re, void* im, uint64_t N, unsigned grid, cudaStream_t s) {
  k_to_df64<<<grid, 256, 0, s>>>((double2*)re, (double2*)im, N / 2);
  return cudaGetLastError();
}
cudaError_t launch_from_df64(void* re, void* im, uint64_t N, unsigned grid, cudaStream_t s) {
  k_from_df64<<<grid, 256, 0, s>>>((double2*)re, (double2*)im, N / 2);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- conj transpose
// In place A'[x*dim + y] = conj(A[y*dim + x]): the reference's adjoint stage
// between its forward and backward passes (block_transpose,
// src/dmsim_nvgpu_omp.cuh:825-855), done as swaps of tile pairs (I, J), I <= J,
// staged in shared memory so both the loads and the stores are coalesced.
template <typename T>
__global__ void __launch_bounds__(256) k_conj_transpose(T* __restrict__ re, T* __restrict__ im, int n) {
  constexpr int TS = 32;
  __shared__ T a_re[TS][TS + 1], a_im[TS][TS + 1], b_re[TS][TS + 1], b_im[TS][TS + 1];
  const uint64_t dim = 1ull << n;
  const int ts = dim < TS ? (int)dim : TS;
  const uint64_t nt = dim / ts;
  const int tx = threadIdx.x & 31, ty0 = threadIdx.x >> 5;  // 32 x 8 threads
  for (uint64_t p = blockIdx.x; p < nt * nt; p += gridDim.x) {
    const uint64_t I = p / nt, J = p % nt;
    if (I > J) continue;  // uniform over the block
    if (tx < ts)
      for (int ty = ty0; ty < ts; ty += 8) {
        const uint64_t ia = (I * ts + ty) * dim + J * ts + tx;  // tile (I,J)
        const uint64_t ib = (J * ts + ty) * dim + I * ts + tx;  // tile (J,I)
        a_re[ty][tx] = re[ia];
        a_im[ty][tx] = im[ia];
        b_re[ty][tx] = re[ib];
        b_im[ty][tx] = im[ib];
      }
    __syncthreads();
    if (tx < ts)
      for (int ty = ty0; ty < ts; ty += 8) {
        const uint64_t ia = (I * ts + ty) * dim + J * ts + tx;
        const uint64_t ib = (J * ts + ty) * dim + I * ts + tx;
        re[ia] = b_re[tx][ty];
        im[ia] = flip(b_im[tx][ty]);
        re[ib] = a_re[tx][ty];
        im[ib] = flip(a_im[tx][ty]);
      }
    __syncthreads();
  }
}

cudaError_t launch_conj_transpose(void* re, void* im, int n, bool fp32, unsigned grid, cudaStream_t s) {
  if (fp32) k_conj_transpose<float><<<grid, 256, 0, s>>>((float*)re, (float*)im, n);
  else k_conj_transpose<double><<<grid, 256, 0, s>>>((double*)re, (double*)im, n);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- half-range passes
// Between half-range passes over different qubit sets (pass.h) the entries
// that the last set left stale and the next one needs are the conjugates of
// their transposes: A[c*dim + r] = conj(A[r*dim + c]) where r & from > c & from
// and r & to <= c & to (to = 0: every stale one).  About half of the stale
// entries, a quarter of the state read and a quarter written.  The last mirror
// of a run (`last`) fills every stale entry and makes the pairs that were both
// computed exactly Hermitian too, so that the state passes the check below
// again.  32 x 32 entry blocks through shared memory, both sides coalesced;
// blocks that the sets' bits >= 5 rule out are skipped.  Entries are moved as
// bits, `neg` is their sign bits (two in a double-float entry).
__global__ void __launch_bounds__(256) k_mirror(uint64_t* __restrict__ re, uint64_t* __restrict__ im, int n,
                                                uint32_t from, uint32_t to, int last, uint64_t neg,
                                                const int* __restrict__ herm) {
  using U = uint64_t;
  constexpr int TS = 32;
  __shared__ U s_re[TS][TS + 1], s_im[TS][TS + 1];
  pdl_wait();
  pdl_begin();
  if (!*herm) return;
  const uint64_t dim = 1ull << n;
  const uint32_t nt = (uint32_t)(dim / TS);
  const uint32_t hf = from & ~(TS - 1u), ht = to & ~(TS - 1u);
  const uint32_t tx = threadIdx.x & 31, ty0 = threadIdx.x >> 5;
  for (uint64_t p = blockIdx.x; p < (uint64_t)nt * nt; p += gridDim.x) {
    const uint32_t R = (uint32_t)(p & (nt - 1)) * TS, C = (uint32_t)(p >> (n - 5)) * TS;
    if ((R & hf) < (C & hf) || (R & ht) > (C & ht)) continue;                 // nothing stale, nothing needed
    if ((from & (TS - 1u)) == 0 && (R & hf) == (C & hf) && !(last && R >= C)) continue;  // all ties
    for (uint32_t ty = ty0; ty < TS; ty += 8) {
      const uint64_t i = (uint64_t)(R + ty) * dim + C + tx;  // rho[C + tx][R + ty]
      s_re[ty][tx] = re[i];
      s_im[ty][tx] = im[i];
    }
    __syncthreads();
    for (uint32_t ty = ty0; ty < TS; ty += 8) {
      const uint32_t r = R + tx, c = C + ty;
      const uint32_t rf = r & from, cf = c & from;
      const bool stale = rf > cf && (r & to) <= (c & to);
      const uint64_t i = (uint64_t)c * dim + r;
      if (stale || (last && rf == cf && r > c)) {
        re[i] = s_re[tx][ty];
        im[i] = s_im[tx][ty] ^ neg;
      } else if (last && r == c) {
        im[i] = 0;
      }
    }
    __syncthreads();
  }
}

cudaError_t launch_mirror(void* re, void* im, int n, int arith, uint32_t from, uint32_t to, bool last,
                          const int* herm, int sms, bool pdl, cudaStream_t s) {
  if (n < 5 || arith == AR_FP32) return cudaErrorInvalidValue;
  // an odd grid: a block's tiles then run through all the residues that the sets' bits decide by
  const uint64_t nt = 1ull << (n - 5);
  const unsigned grid = (unsigned)std::min<uint64_t>(nt * nt, (uint64_t)sms * 8 - 1);
  return launch_kernel(pdl, k_mirror, grid, 256, 0, s, (uint64_t*)re, (uint64_t*)im, n, from, to, (int)last,
                       arith == AR_DF64 ? 0x8000000080000000ull : 0x8000000000000000ull, herm);
}

// rho may have been written from outside (dmsim_set_dm, the device pointers),
// so a run that would use half-range passes on it first compares every entry
// with its transpose, bit by value: one read of the state.  A NaN fails.  The
// blocks stop at the first difference that any of them finds, so that a large state
// without the symmetry (one equal to its transpose but for rounding among them)
// pays for one round of tiles: 13 qubits, 12 CX passes on an arbitrary state took
// 3.84 ms with the full read, 3.75 now.
__global__ void __launch_bounds__(256) k_check_hermitian(const double* __restrict__ re, const double* __restrict__ im,
                                                         int n, int* herm) {
  constexpr int TS = 32;
  __shared__ double s_re[TS][TS + 1], s_im[TS][TS + 1];
  const uint64_t dim = 1ull << n;
  const uint32_t nt = (uint32_t)(dim / TS);
  const uint32_t tx = threadIdx.x & 31, ty0 = threadIdx.x >> 5;
  bool ok = true;
  for (uint64_t p = blockIdx.x; p < (uint64_t)nt * nt; p += gridDim.x) {
    const uint32_t R = (uint32_t)(p & (nt - 1)) * TS, C = (uint32_t)(p >> (n - 5)) * TS;
    if (R > C) continue;
    const bool others = threadIdx.x != 0 || *(volatile const int*)herm != 0;
    for (uint32_t ty = ty0; ty < TS; ty += 8) {
      const uint64_t i = (uint64_t)(R + ty) * dim + C + tx;
      s_re[ty][tx] = re[i];
      s_im[ty][tx] = im[i];
    }
    __syncthreads();
    for (uint32_t ty = ty0; ty < TS; ty += 8) {
      const uint64_t i = (uint64_t)(C + ty) * dim + R + tx;
      ok = ok && re[i] == s_re[tx][ty] && im[i] == -s_im[tx][ty];
    }
    if (__syncthreads_or(!ok || !others)) break;
  }
  if (!ok) *herm = 0;  // every writer writes the same value
}

__global__ void k_set_flag(int* f, int v) { *f = v; }

cudaError_t launch_check_hermitian(const void* re, const void* im, int n, int* herm, int sms, cudaStream_t s) {
  if (n < 5) return cudaErrorInvalidValue;
  const uint64_t nt = 1ull << (n - 5);
  const unsigned grid = (unsigned)std::min<uint64_t>(nt * nt, (uint64_t)sms * 8 - 1);
  k_set_flag<<<1, 1, 0, s>>>(herm, 1);
  k_check_hermitian<<<grid, 256, 0, s>>>((const double*)re, (const double*)im, n, herm);
  return cudaGetLastError();
}

cudaError_t launch_set_flag(int* flag, int value, cudaStream_t s) {
  k_set_flag<<<1, 1, 0, s>>>(flag, value);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- renormalisation
// complex64 mode: every R passes, trace(rho) is summed in FP64 and rho is made
// Hermitian with unit trace, A <- (A + A^dagger) / (2 tr), each entry in the
// state's precision scaled by the FP64 trace (tile pairs as in
// k_conj_transpose).
template <typename T>
__global__ void __launch_bounds__(256) k_trace(const T* __restrict__ re, int n, double* __restrict__ out) {
  const uint64_t dim = 1ull << n;
  double acc = 0;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < dim; i += (uint64_t)gridDim.x * blockDim.x)
    acc += (double)re[i * dim + i];
  __shared__ double sh[256];
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if (threadIdx.x < st) sh[threadIdx.x] += sh[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicAdd(out, sh[0]);
}

template <typename T>
__global__ void __launch_bounds__(256) k_hermitise(T* __restrict__ re, T* __restrict__ im, int n,
                                                   const double* __restrict__ trace) {
  constexpr int TS = 32;
  __shared__ T a_re[TS][TS + 1], a_im[TS][TS + 1], b_re[TS][TS + 1], b_im[TS][TS + 1];
  const uint64_t dim = 1ull << n;
  const int ts = dim < TS ? (int)dim : TS;
  const uint64_t nt = dim / ts;
  const double inv = 1.0 / *trace;
  const int tx = threadIdx.x & 31, ty0 = threadIdx.x >> 5;
  for (uint64_t p = blockIdx.x; p < nt * nt; p += gridDim.x) {
    const uint64_t I = p / nt, J = p % nt;
    if (I > J) continue;
    if (tx < ts)
      for (int ty = ty0; ty < ts; ty += 8) {
        const uint64_t ia = (I * ts + ty) * dim + J * ts + tx, ib = (J * ts + ty) * dim + I * ts + tx;
        a_re[ty][tx] = re[ia];
        a_im[ty][tx] = im[ia];
        b_re[ty][tx] = re[ib];
        b_im[ty][tx] = im[ib];
      }
    __syncthreads();
    if (tx < ts)
      for (int ty = ty0; ty < ts; ty += 8) {
        const uint64_t ia = (I * ts + ty) * dim + J * ts + tx, ib = (J * ts + ty) * dim + I * ts + tx;
        // new A[x][y] = (A[x][y] + conj(A[y][x])) / 2 / tr, in the state's
        // precision with the FP64 trace's scale (FP64 arithmetic on FP32
        // entries would be bound by the f32 <-> f64 conversion rate)
        const T h = (T)(0.5 * inv);
        re[ia] = (a_re[ty][tx] + b_re[tx][ty]) * h;
        im[ia] = (a_im[ty][tx] - b_im[tx][ty]) * h;
        re[ib] = (b_re[ty][tx] + a_re[tx][ty]) * h;
        im[ib] = (b_im[ty][tx] - a_im[tx][ty]) * h;
      }
    __syncthreads();
  }
}

cudaError_t launch_renormalise(void* re, void* im, int n, bool fp32, double* d_trace, unsigned grid, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(d_trace, 0, sizeof(double), s);
  if (e != cudaSuccess) return e;
  const unsigned tg = (unsigned)std::min<uint64_t>((1ull << n) / 256 + 1, 1024);
  if (fp32) {
    k_trace<float><<<tg, 256, 0, s>>>((const float*)re, n, d_trace);
    k_hermitise<float><<<grid, 256, 0, s>>>((float*)re, (float*)im, n, d_trace);
  } else {
    k_trace<double><<<tg, 256, 0, s>>>((const double*)re, n, d_trace);
    k_hermitise<double><<<grid, 256, 0, s>>>((double*)re, (double*)im, n, d_trace);
  }
  return cudaGetLastError();
}

// ---------------------------------------------------------------- utilities
template <typename T>
__global__ void k_set_basis(T* re, T* im, uint64_t idx) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    re[idx] = (T)1;
    im[idx] = (T)0;
  }
}

template <typename T>
__global__ void k_get_diag(const T* __restrict__ re, uint64_t dim, double* __restrict__ out) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i < dim) out[i] = (double)re[i * dim + i];
}

cudaError_t launch_set_zero_state(void* re, void* im, uint64_t N, bool fp32, cudaStream_t s) {
  const size_t es = fp32 ? 4 : 8;
  cudaError_t e = cudaMemsetAsync(re, 0, N * es, s);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(im, 0, N * es, s);
  if (e != cudaSuccess) return e;
  if (fp32) k_set_basis<float><<<1, 32, 0, s>>>((float*)re, (float*)im, 0);
  else k_set_basis<double><<<1, 32, 0, s>>>((double*)re, (double*)im, 0);
  return cudaGetLastError();
}

cudaError_t launch_get_diag(const void* re, uint64_t dim, bool fp32, double* d_out, cudaStream_t s) {
  const unsigned blocks = (unsigned)((dim + 255) / 256);
  if (fp32) k_get_diag<float><<<blocks, 256, 0, s>>>((const float*)re, dim, d_out);
  else k_get_diag<double><<<blocks, 256, 0, s>>>((const double*)re, dim, d_out);
  return cudaGetLastError();
}

}  // namespace dmg

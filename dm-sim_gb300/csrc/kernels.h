// kernels.h -- host-side entry points of the pass kernels (kernels.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "pass.h"

namespace dmg {

// Arithmetic of a pass: the state's element type.
enum Arith : int { AR_FP64 = 0, AR_FP32 = 1, AR_DF64 = 2 };

// A pass may be launched while the one before it is still running (programmatic
// dependent launch): it finds its tables, then waits for the other's end before
// it touches the state (pdl_wait), and only then lets the next one start
// (pdl_begin): a chain of them stays in order, and one kernel at most waits on the
// SMs beside the running one.
template <typename... P, typename... A>
cudaError_t launch_kernel(bool pdl, void (*k)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(block);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = at;
  c.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&c, k, static_cast<P>(args)...);
}
#if defined(__CUDACC__)
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_begin() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

struct LaunchArgs {
  bool pdl;            // may start before the pass before it has ended
  void* re;            // device real parts (double, float, or double-float pairs)
  void* im;            // device imaginary parts
  const void* desc;    // device PassDesc<K>
  int K, cls;
  bool fp32;           // complex64 state
  int arith;           // Arith
  unsigned grid;       // blocks
  int tile_entries;    // G * 4^K
  bool hadamard;       // kPassHadamard pass (pass.h)
  bool real;           // DENSE/SPARSE pass whose U and V are real (pass.h kPassRealOperator)
  bool tc;             // tensor-core pass, K = 3, 4: desc is a TcDesc<K> (double-float or FP32 state) or,
                       // for an FP64 state, a TcDesc64<K>
  int* err;            // device flag set to 1 when a bounded wait of a tensor pass runs out
  bool direct1;        // 1-qubit pass run by the register kernel (kernels_k1.cu)
  bool mono;           // monomial pass on the pipelined kernel (kernels_mono.cu)
  int q0, n;           // its qubit and the state's qubit count
  const HalfMap* half; // device map of a half-range pass (pass.h), else null
  const int* herm;     // device flag: half-range passes run on the half range (the state is Hermitian)
};

// Launch one pass on stream s.
cudaError_t launch_pass(const LaunchArgs& a, cudaStream_t s);
// Resident blocks per SM of the kernel instance for (K, cls, arithmetic).
int pass_blocks_per_sm(int K, int cls, int arith);
// 1-qubit MOVE / SIGNED / PHASE / DENSE passes without shared memory (kernels_k1.cu).
bool direct1_class(int cls);
cudaError_t launch_pass1(const LaunchArgs& a, cudaStream_t s);
// Monomial passes of 2 to 4 qubits on states of many tiles (kernels_mono.cu): its
// grid, 0 for a pass that it does not take, and the launch.
unsigned mono_grid(int K, int cls, int tile_entries, uint64_t ntiles, int sms);
cudaError_t launch_mono(const LaunchArgs& a, cudaStream_t s);
// Several narrow passes in one sweep (kernels_multi.cu): desc is a MultiDesc.
cudaError_t launch_multi(const LaunchArgs& a, cudaStream_t s);
// Real-operator instances of the 1- and 2-qubit DENSE/SPARSE kernels (kernels_real.cu).
cudaError_t launch_pass_real(const LaunchArgs& a, cudaStream_t s);
// Tensor-core passes (tensor.cu): launch, and resident blocks per SM.
cudaError_t launch_pass_tc(const LaunchArgs& a, cudaStream_t s);
int tc_blocks_per_sm(int K, int arith);
// Tensor-core passes on a complex64 (FP32) state (tensor32.cu): two
// persistent 512-thread blocks per SM.
cudaError_t launch_pass_tc32(const LaunchArgs& a, cudaStream_t s);
// FP64-width tensor-core passes on an FP64 state (tensor64.cu): one
// persistent 1024-thread block per SM.
cudaError_t launch_pass_tc64(const LaunchArgs& a, cudaStream_t s);
// In place: FP64 entries <-> double-float pairs (the fused path's working format)
cudaError_t launch_to_df64(void* re, void* im, uint64_t N, unsigned grid, cudaStream_t s);
cudaError_t launch_from_df64(void* re, void* im, uint64_t N, unsigned grid, cudaStream_t s);
// In place A'[x*2^n + y] = conj(A[y*2^n + x]) (the reference's adjoint stage)
cudaError_t launch_conj_transpose(void* re, void* im, int n, bool fp32, unsigned grid, cudaStream_t s);
// Entries stale under `from` that `to` needs (0: every one) <- conj of their
// transposes, if *herm.  last: also make the ties exactly Hermitian.
cudaError_t launch_mirror(void* re, void* im, int n, int arith, uint32_t from, uint32_t to, bool last,
                          const int* herm, int sms, bool pdl, cudaStream_t s);
// *herm <- 1 if rho (FP64 entries) equals its conjugate transpose exactly, else 0
cudaError_t launch_check_hermitian(const void* re, const void* im, int n, int* herm, int sms, cudaStream_t s);
cudaError_t launch_set_flag(int* flag, int value, cudaStream_t s);
// rho <- (rho + rho^dagger) / (2 trace), trace summed in FP64 into d_trace
cudaError_t launch_renormalise(void* re, void* im, int n, bool fp32, double* d_trace, unsigned grid, cudaStream_t s);
// rho <- |0..0><0..0|
cudaError_t launch_set_zero_state(void* re, void* im, uint64_t N, bool fp32, cudaStream_t s);
// d_out[i] = Re rho[i][i] (FP64 whatever the state precision)
cudaError_t launch_get_diag(const void* re, uint64_t dim, bool fp32, double* d_out, cudaStream_t s);

}  // namespace dmg

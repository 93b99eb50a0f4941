// engine_internal.h -- per-pass bookkeeping shared inside the engine.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../../include/dmsim_gb300.h"
#include "plan.h"

namespace dmg {

struct PassInfo {
  int K, cls;
  bool transpose;       // the in-place conjugate transpose (reference-order plans)
  int conv;             // 1: FP64 -> double-float before a fused run, 2: back after it
  bool renorm;          // complex64: FP64 trace + Hermitian renormalisation
  size_t desc_off;      // byte offset of the descriptor in the device blob
  int tile_entries;
  unsigned grid;
  double bytes[2];      // algorithmic bytes moved (reads + writes): run on the whole state, and as planned
                        // (half range where `half`, with the mirror passes)
  int nbasic;
  bool tc;              // runs on the tensor cores (tensor.cu)
  bool hadamard;        // kPassHadamard pass (pass.h)
  bool real;            // real operator (kernels_real.cu for K <= 2)
  bool direct1;         // 1-qubit pass on the register kernel (kernels_k1.cu)
  bool mono;            // monomial pass on the pipelined kernel (kernels_mono.cu)
  int merged;           // > 1: launched with the merged - 1 passes after it, in one sweep (kernels_multi.cu)
  size_t multi_off, multi_half_off;  // its MultiDesc and HalfMap in the device blob
  unsigned multi_grid;
  double multi_saved[2];  // bytes that the sweep moves less than its passes one by one, whole and as planned
  int q0;               // first target qubit
  uint32_t half;        // half-range pass: its qubit set S (0: the whole state)
  uint32_t stale;       // the set under which the state is up to date before the pass: a mirror pass goes first
  size_t half_off;      // byte offset of its HalfMap in the device blob
  PassFeatures feat;
  cudaEvent_t ev0, ev1; // per-pass timing (record mode)
};

// Passes that apply no gates (K = 0) report these class codes.
constexpr int kRecConvert = 16, kRecTranspose = 17, kRecRenorm = 18;

struct PassRecord {
  PassFeatures feat;
  double ms;
  double bytes[2];      // as PassInfo
  unsigned grid;
};

// For the batched sweep (batch.cpp): upload a plan made elsewhere (no real-linear
// gates, no channels); enqueue |0..0><0..0| and every pass of
// s's uploaded plan on stream st (e.g. inside another stream's capture); a bounded
// wait that runs out sets the caller's device word *err_word.
int sim_upload_plan(dmsim_handle s, const std::vector<PassSpec>& specs, uint32_t n_basic);
cudaError_t sim_enqueue(dmsim_handle s, cudaStream_t st, int* err_word, std::string& err);
// algorithmic bytes of s's uploaded plan (reads + writes of every pass)
double sim_plan_bytes(dmsim_handle s);

}  // namespace dmg

// Host check of the launchers in a process with several CUDA contexts (a second
// device, the same device after a reset), against a fake runtime: every kernel
// of every pass launches in each context, the limits are set once per context,
// and an occupancy query that failed is asked again.
#include "fake_cudart.h"

#include "kernels.h"

using namespace dmg;

static int launch_all() {
  static int err_word;
  int bad = 0;
  auto go = [&](LaunchArgs a, const char* what) {
    a.grid = 1;
    a.err = &err_word;
    const cudaError_t e = launch_pass(a, nullptr);
    if (e != cudaSuccess) {
      std::printf("context %llu: %s K=%d cls=%d arith=%d refused\n", fake::ctx, what, a.K, a.cls, a.arith);
      bad++;
    }
  };
  for (int arith : {AR_FP64, AR_FP32, AR_DF64})
    for (int K = 1; K <= 4; K++) {
      LaunchArgs a = {};
      a.K = K;
      a.n = 12;
      a.arith = arith;
      a.fp32 = arith == AR_FP32;
      a.tile_entries = 256 << K;
      for (int cls : {CLS_MOVE, CLS_SIGNED, CLS_PHASE, CLS_DENSE, CLS_SPARSE}) {
        a.cls = cls;
        go(a, "tiled");
        if (K >= 2 && cls <= CLS_PHASE) {
          a.mono = true;
          go(a, "monomial");
          a.mono = false;
        }
        if (K >= 3 && cls >= CLS_DENSE) {
          a.tc = true;
          go(a, "tensor");
          a.tc = false;
        }
      }
    }
  return bad;
}

int main() {
  int bad = 0;
  for (unsigned long long ctx : {1ull, 2ull, 1ull, 3ull}) {
    fake::ctx = ctx;
    bad += launch_all();
    const int set = fake::attribute_calls;
    bad += launch_all();
    if (fake::attribute_calls != set) bad++, std::printf("limits set again in context %llu\n", ctx);
  }
  if (fake::launches == 0) bad++, std::printf("nothing launched\n");
  // a failed query falls back and is not kept
  fake::ctx = 4;
  fake::fail_query = true;
  pass_blocks_per_sm(4, CLS_DENSE, AR_FP64);
  tc_blocks_per_sm(4, AR_DF64);
  fake::fail_query = false;
  if (pass_blocks_per_sm(4, CLS_DENSE, AR_FP64) != 3) bad++, std::printf("a failed occupancy query was kept\n");
  const int q = fake::queries;
  tc_blocks_per_sm(4, AR_DF64);
  if (fake::queries == q) bad++, std::printf("a failed tensor occupancy query was kept\n");
  const int asked = fake::queries;
  pass_blocks_per_sm(4, CLS_DENSE, AR_FP64);
  if (fake::queries != asked) bad++, std::printf("occupancy asked twice in a context\n");
  if (bad == 0) std::printf("ok %d launches\n", fake::launches);
  return bad != 0;
}

// kernels_multi.cu -- consecutive narrow passes in one sweep of the state: 1-qubit
// gates and channels and CX gates that act on two qubits between them.
//
// Gate by gate, most passes are bound by memory or by their launch.  A thread
// takes the 16 entries rho[(a, b)] of the two ket and the two bra bits into
// registers, applies the passes to them one after the other -- each in its own
// arithmetic, operation by operation what the pass by itself does
// (kernels_k1.cu), so the results are the same bit for bit -- and writes them
// back.  Operators are staged in shared memory, in the state's arithmetic, once
// per block.  Which runs go together is estimated at upload (engine.cpp:
// merge_passes): FP64 dense operators and channels hardly ever do, as the FP64 pipe
// bounds them and three blocks of four warps an SM feed it worse than the 1-qubit
// kernel's.  Measured, passes one by one and merged: 13 qubits mixed gates gate by
// gate 166 -> 135 ms, 10 qubits 4.8 -> 4.0, 12 qubits double-float 9.8 -> 7.1 ms, 8
// qubits 2.12 -> 1.62 ms; the 7-qubit noisy ansatz 523 -> 452 us.
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "kernels.h"
#include "pass_device.cuh"

namespace dmg {

namespace {

template <typename T>
struct OpShared {
  T c[32];
  int kind, p, flags;
  int8_t fk[4];
};

// One op on the four entries (a, b) of qubit P: entry a + 2 b at base + a (1 << P) + b (4 << P).
template <typename T, int P, typename F>
__device__ __forceinline__ void each_group(T (&xr)[16], T (&xi)[16], F&& f) {
  constexpr int A = 1 << P, B = 4 << P, OA = 2 >> P, OB = 8 >> P;
#pragma unroll
  for (int o = 0; o < 4; o++) {
    const int s = (o & 1) * OA + (o >> 1) * OB;
    f(xr[s], xr[s + A], xr[s + B], xr[s + A + B], xi[s], xi[s + A], xi[s + B], xi[s + A + B]);
  }
}

template <typename T, bool RE>
__device__ __forceinline__ void dense4(const OpShared<T>& op, T& r0, T& r1, T& r2, T& r3, T& i0, T& i1, T& i2, T& i3) {
  const T xr[4] = {r0, r1, r2, r3}, xi[4] = {i0, i1, i2, i3};
  T yr[4], yi[4], zr[4], zi[4];
#pragma unroll
  for (int b = 0; b < 2; b++)
#pragma unroll
    for (int a = 0; a < 2; a++) {
      Acc<T> ar, ai;
#pragma unroll
      for (int c = 0; c < 2; c++) {
        ar.mad(op.c[a * 2 + c], xr[c + 2 * b]);
        ai.mad(op.c[a * 2 + c], xi[c + 2 * b]);
        if constexpr (!RE) {
          ar.mad(-op.c[4 + a * 2 + c], xi[c + 2 * b]);
          ai.mad(op.c[4 + a * 2 + c], xr[c + 2 * b]);
        }
      }
      yr[a + 2 * b] = ar.get();
      yi[a + 2 * b] = ai.get();
    }
#pragma unroll
  for (int a = 0; a < 2; a++)
#pragma unroll
    for (int b = 0; b < 2; b++) {
      Acc<T> ar, ai;
#pragma unroll
      for (int d = 0; d < 2; d++) {
        ar.mad(op.c[8 + b * 2 + d], yr[a + 2 * d]);
        ai.mad(op.c[8 + b * 2 + d], yi[a + 2 * d]);
        if constexpr (!RE) {
          ar.mad(-op.c[12 + b * 2 + d], yi[a + 2 * d]);
          ai.mad(op.c[12 + b * 2 + d], yr[a + 2 * d]);
        }
      }
      zr[a + 2 * b] = ar.get();
      zi[a + 2 * b] = ai.get();
    }
  r0 = zr[0], r1 = zr[1], r2 = zr[2], r3 = zr[3];
  i0 = zi[0], i1 = zi[1], i2 = zi[2], i3 = zi[3];
}

template <typename T>
__device__ __forceinline__ void swap2(T& a, T& b) {
  const T t = a;
  a = b;
  b = t;
}
// An entry times its factor.
template <typename T>
__device__ __forceinline__ void factor(const OpShared<T>& op, int k, T& r, T& i) {
  const int fk = op.fk[k];
  if (fk == FK_ONE) return;
  if (fk == FK_GEN) {
    const T fr = op.c[k], fi = op.c[4 + k], x = r, y = i;
    r = madd(fr, x, -fi * y);
    i = madd(fr, y, fi * x);
  } else if (fk == FK_NEG) {
    r = flip(r);
    i = flip(i);
  } else if (fk == FK_PI) {
    const T x = r;
    r = flip(i);
    i = x;
  } else {
    const T x = r;
    r = i;
    i = flip(x);
  }
}

template <typename T, int P>
__device__ __forceinline__ void apply1(const OpShared<T>& op, T (&xr)[16], T (&xi)[16]) {
  const int kind = op.kind, fl = op.flags;
  if (kind == MO_DENSE) {
    each_group<T, P>(xr, xi, [&](T& r0, T& r1, T& r2, T& r3, T& i0, T& i1, T& i2, T& i3) {
      dense4<T, false>(op, r0, r1, r2, r3, i0, i1, i2, i3);
    });
  } else if (kind == MO_REAL) {
    each_group<T, P>(xr, xi, [&](T& r0, T& r1, T& r2, T& r3, T& i0, T& i1, T& i2, T& i3) {
      dense4<T, true>(op, r0, r1, r2, r3, i0, i1, i2, i3);
    });
  } else if (kind == MO_HADAMARD) {
    if constexpr (std::is_same<T, double>::value) {  // FP64 only, as its passes by themselves
      each_group<T, P>(xr, xi, [&](T& r0, T& r1, T& r2, T& r3, T& i0, T& i1, T& i2, T& i3) {
        auto h = [](T& x0, T& x1, T& x2, T& x3) {
          const T s0 = x0 + x1, d0 = x0 - x1, s1 = x2 + x3, d1 = x2 - x3;
          x0 = half_of(s0 + s1);
          x1 = half_of(d0 + d1);
          x2 = half_of(s0 - s1);
          x3 = half_of(d0 - d1);
        };
        h(r0, r1, r2, r3);
        h(i0, i1, i2, i3);
        if (fl & 2) r1 = flip(r1), r2 = flip(r2), i1 = flip(i1), i2 = flip(i2);
        if (fl & 1) {
          swap2(r0, r3);
          swap2(r1, r2);
          swap2(i0, i3);
          swap2(i1, i2);
        }
      });
    }
  } else if (kind == MO_MONO) {
    each_group<T, P>(xr, xi, [&](T& r0, T& r1, T& r2, T& r3, T& i0, T& i1, T& i2, T& i3) {
      if (fl & 1) {
        swap2(r0, r3);
        swap2(r1, r2);
        swap2(i0, i3);
        swap2(i1, i2);
      }
      if (fl & 2) {  // factors, at [a * 2 + b] of entry a + 2 b
        factor(op, 0, r0, i0);
        factor(op, 2, r1, i1);
        factor(op, 1, r2, i2);
        factor(op, 3, r3, i3);
      }
    });
  } else {  // MO_CHANNEL: kernels_k1.cu's simple superoperators
    const int diag = fl & 3;
    const bool crossed = fl & 4;
    each_group<T, P>(xr, xi, [&](T& r0, T& r1, T& r2, T& r3, T& i0, T& i1, T& i2, T& i3) {
      auto ch = [&](T& x0, T& x1, T& x2, T& x3) {
        T y0, y1, y2, y3;
        if (diag == 3) {
          y0 = madd(op.c[1], x3, madd(op.c[0], x0, T(0)));
          y3 = madd(op.c[3], x3, madd(op.c[2], x0, T(0)));
        } else if (diag == 1) {
          y0 = madd(op.c[1], x3, madd(op.c[0], x0, T(0)));
          y3 = madd(op.c[3], x3, T(0));
        } else {
          y0 = madd(op.c[0], x0, T(0));
          y3 = madd(op.c[3], x3, T(0));
        }
        if (crossed) {
          y2 = madd(op.c[5], x1, madd(op.c[4], x2, T(0)));
          y1 = madd(op.c[7], x1, madd(op.c[6], x2, T(0)));
        } else {
          y2 = madd(op.c[4], x2, T(0));
          y1 = madd(op.c[7], x1, T(0));
        }
        x0 = y0, x1 = y1, x2 = y2, x3 = y3;
      };
      ch(r0, r1, r2, r3);
      ch(i0, i1, i2, i3);
    });
  }
}

// CX with control qubit C of the pair, on the ket and the bra bits.
template <typename T, int C>
__device__ __forceinline__ void apply_cx(T (&x)[16]) {
  constexpr int c = 1 << C, t = 2 >> C;
#pragma unroll
  for (int bra = 0; bra < 16; bra += 4) swap2(x[bra + c], x[bra + c + t]);
#pragma unroll
  for (int ket = 0; ket < 4; ket++) swap2(x[ket + 4 * c], x[ket + 4 * (c + t)]);
}

// A 2-qubit channel of real terms between the diagonal entries and of every other
// entry's own, first qubit F of the pair: index i's bits are at entry bits F, 1 - F.
template <typename T, int F>
__device__ __forceinline__ void apply_channel2(const OpShared<T>& op, T (&x)[16]) {
  constexpr int b0 = 1 << F, b1 = 2 >> F;
  auto at = [](int a, int b) { return ((a & 1) * b0 + (a >> 1) * b1) + 4 * ((b & 1) * b0 + (b >> 1) * b1); };
  T y[4];
#pragma unroll
  for (int o = 0; o < 4; o++) {
    T acc = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) acc = madd(op.c[o * 4 + j], x[at(j, j)], acc);
    y[o] = acc;
  }
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 4; b++) x[at(a, b)] = a == b ? y[a] : madd(op.c[16 + a * 4 + b], x[at(a, b)], T(0));
}

template <typename T, bool HALF>
__global__ void __launch_bounds__(kMultiThreads, 3) k_multi(T* __restrict__ re, T* __restrict__ im,
                                                            const MultiDesc* __restrict__ dp, int n,
                                                            const HalfMap* __restrict__ half,
                                                            const int* __restrict__ herm) {
  __shared__ OpShared<T> s_op[kMultiOps];
  const int nops = dp->nops;
  for (int i = threadIdx.x; i < nops * 32; i += blockDim.x) s_op[i >> 5].c[i & 31] = coef<T>(dp->op[i >> 5].c[i & 31]);
  for (int i = threadIdx.x; i < nops; i += blockDim.x) {
    s_op[i].kind = dp->op[i].kind;
    s_op[i].p = dp->op[i].p;
    s_op[i].flags = dp->op[i].flags;
    for (int k = 0; k < 4; k++) s_op[i].fk[k] = dp->op[i].fk[k];
  }
  __syncthreads();
  pdl_wait();
  pdl_begin();
  const HalfMap* hm = HALF && *herm ? half : nullptr;
  const uint64_t ngroups = hm ? hm->count : 1ull << (2 * n - 4);
  const int qa = dp->qa, qb = dp->qb;
  const uint64_t ma = 1ull << qa, mb = 1ull << qb;
  for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < ngroups; g += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t i;
    if (hm) {
      i = half_base(*hm, g, 0);
    } else {
      i = g;
      const int pos[4] = {qa, qb, qa + n, qb + n};  // ascending: qa < qb < n
#pragma unroll
      for (int j = 0; j < 4; j++) i = ((i >> pos[j]) << (pos[j] + 1)) | (i & ((1ull << pos[j]) - 1));
    }
    T xr[16], xi[16];
#pragma unroll
    for (int e = 0; e < 16; e++) {
      const uint64_t k = i + (e & 1 ? ma : 0) + (e & 2 ? mb : 0) + (((e & 4 ? ma : 0) + (e & 8 ? mb : 0)) << n);
      xr[e] = ld1<T>(re + k);
      xi[e] = ld1<T>(im + k);
    }
    for (int o = 0; o < nops; o++) {
      const OpShared<T>& op = s_op[o];
      if (op.kind == MO_CX) {
        if (op.p == 0) {
          apply_cx<T, 0>(xr);
          apply_cx<T, 0>(xi);
        } else {
          apply_cx<T, 1>(xr);
          apply_cx<T, 1>(xi);
        }
      } else if (op.kind == MO_CHANNEL2) {
        if (op.p == 0) {
          apply_channel2<T, 0>(op, xr);
          apply_channel2<T, 0>(op, xi);
        } else {
          apply_channel2<T, 1>(op, xr);
          apply_channel2<T, 1>(op, xi);
        }
      } else if (op.p == 0) {
        apply1<T, 0>(op, xr, xi);
      } else {
        apply1<T, 1>(op, xr, xi);
      }
    }
#pragma unroll
    for (int e = 0; e < 16; e++) {
      const uint64_t k = i + (e & 1 ? ma : 0) + (e & 2 ? mb : 0) + (((e & 4 ? ma : 0) + (e & 8 ? mb : 0)) << n);
      st1<T>(re + k, xr[e]);
      st1<T>(im + k, xi[e]);
    }
  }
}

template <typename T>
cudaError_t launch_multi_t(const LaunchArgs& a, cudaStream_t s) {
  auto* k = k_multi<T, false>;
  if constexpr (!std::is_same<T, float>::value) {
    if (a.half) k = k_multi<T, true>;
  } else if (a.half) {
    return cudaErrorInvalidValue;
  }
  return launch_kernel(a.pdl, k, a.grid, kMultiThreads, 0, s, static_cast<T*>(a.re), static_cast<T*>(a.im),
                       static_cast<const MultiDesc*>(a.desc), a.n, a.half, a.herm);
}

}  // namespace

cudaError_t launch_multi(const LaunchArgs& a, cudaStream_t s) {
  if (a.n < 2) return cudaErrorInvalidValue;
  if (a.arith == AR_DF64) return launch_multi_t<df64>(a, s);
  return a.fp32 ? launch_multi_t<float>(a, s) : launch_multi_t<double>(a, s);
}

}  // namespace dmg

// kernels_k1.cu -- 1-qubit passes without shared memory.  A 1-qubit pass
// touches each group of four entries rho[(a, b)] (a = ket bit q, b = bra bit
// q + n) on its own, so a thread takes whole groups straight from global
// memory -- consecutive threads take consecutive groups, so every load and
// store instruction of a warp is coalesced -- applies U on the ket bit and V
// on the bra bit in registers (the same operation order and accumulator as
// the tiled kernel), and writes back the entries the pass changes.  No tile
// staging, no barriers: these passes (most of the plain gate-by-gate path)
// are bound by HBM or by the arithmetic alone.
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "kernels.h"
#include "pass_device.cuh"

namespace dmg {

namespace {

// -x if n (32-bit integer work: a select of doubles takes the FP64 pipe)
__device__ __forceinline__ double xor_sign(double x, bool n) {
  return __hiloint2double(__double2hiint(x) ^ (n ? (int)0x80000000 : 0), __double2loint(x));
}

template <typename T, int CLS_, bool HALF>
__global__ void __launch_bounds__(256) k_pass1(T* __restrict__ re, T* __restrict__ im,
                                               const PassDesc<1>* __restrict__ dp, int q, int n,
                                               const HalfMap* __restrict__ half, const int* __restrict__ herm) {
  constexpr int CLS = base_class(CLS_);
  constexpr bool RE = real_class(CLS_);
  constexpr bool kMono = CLS == CLS_MOVE || CLS == CLS_SIGNED || CLS == CLS_PHASE;
  constexpr bool kSuper = CLS == CLS_SUPER;
  constexpr bool kHad = CLS_ == CLS_HADAMARD;
  const PassOp<1>& op = dp->op;
  // double-float: warps without a group (states below 5 qubits) leave the FP64 pipe's
  // conversions of the operator to the others: 3 qubits, dense 9.8 -> 7.9 us
  if (std::is_same<T, df64>::value && !kSuper && (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u) >= 1ull << (2 * n - 2)) return;
  // the operator, uniform over the grid (a few dozen bytes from L1)
  T ur[4], ui[4], vr[4], vi[4], fr[4], fi[4];
  int src[2], srcb[2], fk[4];
  bool need[4], chg[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    ur[i] = coef<T>(op.ure[i]);
    ui[i] = coef<T>(op.uim[i]);
    vr[i] = coef<T>(op.vre[i]);
    vi[i] = coef<T>(op.vim[i]);
    fr[i] = coef<T>(op.fre[i]);
    fi[i] = coef<T>(op.fim[i]);
    fk[i] = op.fk[i];
  }
  src[0] = op.src[0];
  src[1] = op.src[1];
  srcb[0] = op.srcb[0];
  srcb[1] = op.srcb[1];
  // a channel's superoperator, and its nonzero terms: bit 4 o + j for output
  // o = 2a + b and input j = 2c + e
  __shared__ T s_sr[kSuper ? 16 : 1], s_si[kSuper ? 16 : 1];
  __shared__ uint32_t s_nz, s_cplx;
  uint32_t nz = 0, cplx = 0;
  if constexpr (kSuper) {
    if (threadIdx.x < 32) {
      const int i = threadIdx.x & 15;
      const double mr = op.sre[i], mi = op.sim[i];
      s_sr[i] = coef<T>(mr);
      s_si[i] = coef<T>(mi);
      const uint32_t m = __ballot_sync(0xffffffffu, mr != 0.0 || mi != 0.0), mc = __ballot_sync(0xffffffffu, mi != 0.0);
      if (threadIdx.x == 0) {
        s_nz = m & 0xFFFFu;
        s_cplx = mc & 0xFFFFu;
      }
    }
    __syncthreads();
    nz = s_nz;
    cplx = s_cplx;
  }
  // simple: real, every output has its own term, outputs 0 and 3 the other's too
  // (diag: bit 0 for output 0, bit 1 for output 3; not the latter alone) and
  // outputs 1 and 2 each other's (crossed) or not, and nothing else
  constexpr uint32_t kOwn = 0x8421u, kCross = 0x0240u;
  const uint32_t diag = (nz >> 3 & 1) | (nz >> 11 & 2);
  const bool simple = kSuper && cplx == 0 && (nz & ~(kCross | 0x1008u)) == kOwn && diag != 2 &&
                      ((nz & kCross) == 0 || (nz & kCross) == kCross);
  const bool crossed = (nz & kCross) != 0;
  T sc[kSuper ? 8 : 1];
  if constexpr (kSuper) {
    constexpr int at[8] = {0, 3, 12, 15, 5, 6, 9, 10};
#pragma unroll
    for (int i = 0; i < 8; i++) sc[i] = s_sr[at[i]];
  }
  // entry e = a + 2b: which change, which are read (unrolled comparisons,
  // so that the small arrays stay in registers)
  int sidx[4];
#pragma unroll
  for (int e = 0; e < 4; e++) {
    const int a = e & 1, b = e >> 1;
    sidx[e] = src[a] + 2 * srcb[b];
    chg[e] = !kMono || sidx[e] != e || fk[a * 2 + b] != FK_ONE;
  }
#pragma unroll
  for (int e = 0; e < 4; e++) {
    bool nd = !kMono;
#pragma unroll
    for (int e2 = 0; e2 < 4; e2++) nd = nd || (chg[e2] && sidx[e2] == e);
    need[e] = nd;
  }

  const bool hswap = kHad && op.ure[0] * op.ure[1] < 0, hneg = kHad && op.ure[0] * op.ure[2] < 0;
  const HalfMap* hm = HALF && *herm ? half : nullptr;  // the half range of the groups, if any
  const uint64_t ngroups = hm ? hm->count : 1ull << (2 * n - 2);
  const uint64_t mq = 1ull << q, mb = 1ull << (q + n);
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  pdl_wait();
  pdl_begin();
  for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < ngroups; g += stride) {
    uint64_t i;
    if (hm) {
      i = half_base(*hm, g, 0);
    } else {
      i = ((g >> q) << (q + 1)) | (g & (mq - 1));
      i = ((i >> (q + n)) << (q + n + 1)) | (i & (mb - 1));
    }
    uint64_t idx[4];
    idx[0] = i;
    idx[1] = i + mq;
    idx[2] = i + mb;
    idx[3] = i + mq + mb;
    T xr[4], xi[4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
      xr[e] = need[e] ? ld1<T>(re + idx[e]) : T(0);
      xi[e] = need[e] ? ld1<T>(im + idx[e]) : T(0);
    }
    T outr[4], outi[4];
    if constexpr (kMono) {
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int a = e & 1, b = e >> 1, s = sidx[e], k = a * 2 + b;
        const T r = s == 0 ? xr[0] : s == 1 ? xr[1] : s == 2 ? xr[2] : xr[3];
        const T m = s == 0 ? xi[0] : s == 1 ? xi[1] : s == 2 ? xi[2] : xi[3];
        if (CLS == CLS_MOVE || fk[k] == FK_ONE) {
          outr[e] = r;
          outi[e] = m;
        } else if (CLS == CLS_PHASE && fk[k] == FK_GEN) {
          outr[e] = madd(fr[k], r, -fi[k] * m);
          outi[e] = madd(fr[k], m, fi[k] * r);
        } else if (fk[k] == FK_NEG) {
          outr[e] = flip(r);
          outi[e] = flip(m);
        } else if (fk[k] == FK_PI) {
          outr[e] = flip(m);
          outi[e] = r;
        } else {
          outr[e] = m;
          outi[e] = flip(r);
        }
      }
    } else if constexpr (kHad) {
      // sqrt(1/2) (1 1; 1 -1) on either side: sums and differences, a half of
      // them exactly -- four FP64 additions an entry instead of eight
      // multiply-adds, and no rounded sqrt(1/2).  Row a of U is rs_a (1, p_a)
      // sqrt(1/2), p_0 = -p_1: out[a][b] = rs_a rs_b z[p_a < 0][p_b < 0], by the
      // place it is stored at.  13 qubits, half range: 501 -> 300 us a pass (the
      // FP64 pipe alone 223, HBM 167); with the outputs chosen by value, selects
      // of doubles that run on the FP64 pipe, it took 567.
      T z[2][4];  // real, imaginary parts; index i + 2 j
#pragma unroll
      for (int c = 0; c < 2; c++) {
        const T* x = c ? xi : xr;
        const T s0 = x[0] + x[1], d0 = x[0] - x[1], s1 = x[2] + x[3], d1 = x[2] - x[3];
        z[c][0] = half_of(s0 + s1);
        z[c][1] = half_of(d0 + d1);
        z[c][2] = half_of(s0 - s1);
        z[c][3] = half_of(d0 - d1);
      }
#pragma unroll
      for (int e = 0; e < 4; e++) {
        outr[e] = z[0][e];
        outi[e] = z[1][e];
        if (e == 1 || e == 2) {
          outr[e] = xor_sign(outr[e], hneg);
          outi[e] = xor_sign(outi[e], hneg);
        }
      }
      if (hswap) {
        const uint64_t a = idx[0], b = idx[1];
        idx[0] = idx[3];
        idx[1] = idx[2];
        idx[2] = b;
        idx[3] = a;
      }
    } else if (kSuper && simple) {
      // real terms only between the two diagonal entries and between the two
      // others (every named channel): 8 to 16 multiply-adds a group, in the order
      // of the general loop, whose skipped terms cost selects on the FP64 pipe.
      // 11 qubits, depolarising, half range: 34.7 -> 22.5 us a pass.
      if (diag == 3) {
#pragma unroll
        for (int p = 0; p < 2; p++) {
          const T* x = p ? xi : xr;
          T* out = p ? outi : outr;
          out[0] = madd(sc[1], x[3], madd(sc[0], x[0], T(0)));
          out[3] = madd(sc[3], x[3], madd(sc[2], x[0], T(0)));
        }
      } else if (diag == 1) {
#pragma unroll
        for (int p = 0; p < 2; p++) {
          const T* x = p ? xi : xr;
          T* out = p ? outi : outr;
          out[0] = madd(sc[1], x[3], madd(sc[0], x[0], T(0)));
          out[3] = madd(sc[3], x[3], T(0));
        }
      } else {
#pragma unroll
        for (int p = 0; p < 2; p++) {
          const T* x = p ? xi : xr;
          T* out = p ? outi : outr;
          out[0] = madd(sc[0], x[0], T(0));
          out[3] = madd(sc[3], x[3], T(0));
        }
      }
      if (crossed) {
#pragma unroll
        for (int p = 0; p < 2; p++) {
          const T* x = p ? xi : xr;
          T* out = p ? outi : outr;
          out[2] = madd(sc[5], x[1], madd(sc[4], x[2], T(0)));
          out[1] = madd(sc[7], x[1], madd(sc[6], x[2], T(0)));
        }
      } else {
#pragma unroll
        for (int p = 0; p < 2; p++) {
          const T* x = p ? xi : xr;
          T* out = p ? outi : outr;
          out[2] = madd(sc[4], x[2], T(0));
          out[1] = madd(sc[7], x[1], T(0));
        }
      }
    } else if constexpr (kSuper) {
      // the terms in index order, the zero ones skipped (the same for every thread)
#pragma unroll
      for (int o = 0; o < 4; o++) {
        T ar = 0, ai = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
          if (!((nz >> (4 * o + j)) & 1)) continue;
          const int x = (j >> 1) + 2 * (j & 1);
          const T mr = s_sr[4 * o + j];
          ar = madd(mr, xr[x], ar);
          ai = madd(mr, xi[x], ai);
          if ((cplx >> (4 * o + j)) & 1) {
            const T mi = s_si[4 * o + j];
            ar = madd(-mi, xi[x], ar);
            ai = madd(mi, xr[x], ai);
          }
        }
        outr[(o >> 1) + 2 * (o & 1)] = ar;
        outi[(o >> 1) + 2 * (o & 1)] = ai;
      }
    } else {
      // ket step: y[a][b] = sum_c U[a][c] x[c][b]
      T yr[4], yi[4];
#pragma unroll
      for (int b = 0; b < 2; b++)
#pragma unroll
        for (int a = 0; a < 2; a++) {
          Acc<T> ar, ai;
#pragma unroll
          for (int c = 0; c < 2; c++) {
            ar.mad(ur[a * 2 + c], xr[c + 2 * b]);
            ai.mad(ur[a * 2 + c], xi[c + 2 * b]);
            if constexpr (!RE) {
              ar.mad(-ui[a * 2 + c], xi[c + 2 * b]);
              ai.mad(ui[a * 2 + c], xr[c + 2 * b]);
            }
          }
          yr[a + 2 * b] = ar.get();
          yi[a + 2 * b] = ai.get();
        }
      // bra step: out[a][b] = sum_d V[b][d] y[a][d]
#pragma unroll
      for (int a = 0; a < 2; a++)
#pragma unroll
        for (int b = 0; b < 2; b++) {
          Acc<T> ar, ai;
#pragma unroll
          for (int d = 0; d < 2; d++) {
            ar.mad(vr[b * 2 + d], yr[a + 2 * d]);
            ai.mad(vr[b * 2 + d], yi[a + 2 * d]);
            if constexpr (!RE) {
              ar.mad(-vi[b * 2 + d], yi[a + 2 * d]);
              ai.mad(vi[b * 2 + d], yr[a + 2 * d]);
            }
          }
          outr[a + 2 * b] = ar.get();
          outi[a + 2 * b] = ai.get();
        }
    }
#pragma unroll
    for (int e = 0; e < 4; e++)
      if (chg[e]) {
        st1<T>(re + idx[e], outr[e]);
        st1<T>(im + idx[e], outi[e]);
      }
  }
}

template <typename T, int CLS_>
cudaError_t launch1(const LaunchArgs& a, cudaStream_t s) {
  // two instances, as for the tiled kernel (pass_kernel.cuh)
  auto* k = k_pass1<T, CLS_, false>;
  if constexpr (!std::is_same<T, float>::value) {
    if (a.half) k = k_pass1<T, CLS_, true>;
  } else if (a.half) {
    return cudaErrorInvalidValue;
  }
  return launch_kernel(a.pdl, k, a.grid, 256, 0, s, static_cast<T*>(a.re), static_cast<T*>(a.im),
                       static_cast<const PassDesc<1>*>(a.desc), a.q0, a.n, a.half, a.herm);
}

template <typename T>
cudaError_t launch1_t(const LaunchArgs& a, cudaStream_t s) {
  switch (a.cls) {
    case CLS_MOVE: return launch1<T, CLS_MOVE>(a, s);
    case CLS_SIGNED: return launch1<T, CLS_SIGNED>(a, s);
    case CLS_PHASE: return launch1<T, CLS_PHASE>(a, s);
    case CLS_DENSE:
      if constexpr (std::is_same<T, double>::value)
        if (a.hadamard) return launch1<T, CLS_HADAMARD>(a, s);
      return a.real ? launch1<T, CLS_DENSE_REAL>(a, s) : launch1<T, CLS_DENSE>(a, s);
    case CLS_SUPER: return launch1<T, CLS_SUPER>(a, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

bool direct1_class(int cls) {
  return cls == CLS_MOVE || cls == CLS_SIGNED || cls == CLS_PHASE || cls == CLS_DENSE || cls == CLS_SUPER;
}

cudaError_t launch_pass1(const LaunchArgs& a, cudaStream_t s) {
  if (a.K != 1 || !direct1_class(a.cls)) return cudaErrorInvalidValue;
  if (a.arith == AR_DF64) return launch1_t<df64>(a, s);
  return a.fp32 ? launch1_t<float>(a, s) : launch1_t<double>(a, s);
}

}  // namespace dmg

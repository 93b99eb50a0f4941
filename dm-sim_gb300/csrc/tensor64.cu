// tensor64.cu -- dense K = 3, 4 qubit passes on the tensor cores for an FP64
// state, at FP64 width: the products on the tensor cores, the rest on the
// integer pipe and a few conversions on GB300's FP64 pipe (1/60 of the FP32
// rate).
//
// A pass is two products per tile, as in the double-float tensor pass: the
// ket step multiplies every tile column x (2^K complex entries as R = 2^(K+1)
// reals) by the real embedding W = [[Ur, -Ui], [Ui, Ur]], the bra step the
// result's columns by V.  Here every operand value is an integer times a
// power of two, split into 7 balanced base-256 digits (|digit| <= 128, exact
// in FP16):
//   * a state column (ket step): the FP64 bits are aligned to the column's
//     largest exponent, |v| <= 2^55 (55 significant bits for the column's
//     largest value);
//   * an operator row (host, TcDesc64): w = t 2^ew with |t| <= 2^55;
//   * a bra-step column: the ket step's exact integer outputs, aligned to the
//     bra column's own magnitude (54-55 significant bits for its largest).
// Digit pairs of orders i + j = 0..7 are summed by tcgen05.mma into one FP32
// accumulator per order; every partial sum is an integer below 7 R 2^14 <=
// 2^22, so the sums are exact.  Two conversions that the digits and the sums
// would need are left to the tensor cores: a digit plus 128 is a byte of the
// aligned value, and a byte is an FP16 number times 2^-24 as it is; and the
// sums start at 0.75 minus the 128s' share, so that an accumulator's FP32 bits
// are an integer.  The orders are combined in 64-bit integer arithmetic (orders
// 6 and 7 floored at 2^-43 of order 0) and the bra step's result is rounded
// once to FP64 from the 64-bit integer.  Each value is held with 55 significant
// bits relative to its column's largest (block floating point per column of
// 2^K entries), an operator's entry relative to its row's largest.  The error of
// an output, per step, X its column's largest value, w its row: at most one unit
// (2^-54 X) a value (the conversions err by half of one, the shifts by one), half
// a unit (2^-55 max|w|) an entry, and the orders that are left out and floored:
// 2^-54 X (|w|_1 + (1.04 D + 1) max|w|), D = 2^K.
//
// Threads: 1024 (32 warps, 64 registers each), one block per SM, as two
// independent groups of 16 warps that take alternate tiles of the block, each
// with its own tile buffer, digit operand, tensor-memory accumulator set,
// mbarriers and named barrier: while one group waits at a barrier or on its
// products, the other issues, with eight warps per scheduler to hide the
// integer work's latency.  Every thread holds a quarter of a column: in the
// digit steps thread (warp w, lane l) of a group owns tile column 8 (w & 15)
// + (l & 7) and quarter l >> 3 of it (half l >> 4, values (l >> 3) & 1 of
// that half; the four quarters of a column in one warp); in the accumulator
// steps column m = 32 (w & 3) + l -- the TMEM lane quadrant its warp may read
// -- and quarter ((w & 15) >> 2).  The group's first warp issues its MMAs.
// Per tile:
//   1. wait for the tile (copied one tile ahead), column maxima, ket digits
//      -> A;  2. the ket MMAs;  3. ket accumulators -> exact int64 outputs in
//      place of the tile;  4. bra magnitude keys, bra digits -> A;  5. the bra
//      MMAs, and the group's next tile loaded into the freed buffer;  6. bra
//      accumulators -> FP64 -> global stores.
// Three group barriers per tile (after steps 1, 3 and 4); the first two also
// OR the threads' timeout flags.  Every wait is bounded; on expiry the group
// leaves its loop at the next such barrier, waits (bounded) for its own copies
// and MMAs in flight, sets the error flag, and the block releases its TMEM;
// the host reports DMSIM_ERR_TIMEOUT.
//
// What bounds it: the ALU, the FP64 pipe's conversions and shared memory are
// each near half busy; a group's steps follow one another, and tensor memory
// and the digit operands leave room for two groups.  A 4-qubit pass over half
// of a 14-qubit state (2.2 GB read, 2.2 written) takes 1.93 ms, of which a
// group spends about a fifth on each of: ket digits, MMAs, outputs.  It took
// 2.6 ms with the digits converted to BF16 one by one and the sums taken apart
// by an FP32 addition each (156 against 224 instructions a value, now fewer).
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.h"
#include "pass_device.cuh"
#include "per_context.h"
#include "tc.cuh"

namespace dmg {

namespace {

constexpr int kT64Threads = 1024;
constexpr int kT64GroupThreads = 512;
constexpr uint32_t kT64WaitPolls = 1u << 24;

template <int K>
struct T64 {
  static constexpr int D = 1 << K, R = 2 * D, G = 128 / D, TILE = 128 * D;
  // entries from a loaded tile's real array to its imaginary array: 16-entry
  // pieces 18 entries apart, and an offset of 8 pieces' banks between the two
  static constexpr int ASTR = TILE / 16 * 18 + 8;
  static constexpr uint32_t SBO = 16 * R;                  // bytes between 8-row groups of an R-wide operand
  static constexpr uint32_t A_BYTES = 128 * R * 2;         // one digit slice of the 128 columns
  static constexpr uint32_t B_BYTES = R * R * 2;           // one digit slice of W or V
  static constexpr uint32_t SET_COLS = kTc64Orders * R;    // accumulators of one group
  static constexpr uint32_t TMEM_COLS = 2 * SET_COLS;      // 512 (K = 4), 256 (K = 3)
  static constexpr uint32_t BUF_BYTES = 2 * ASTR * 8;      // one group's tile buffer
  static constexpr uint32_t BI_BYTES = kTc64Orders * R * 16;  // one side's starting sums: 8 FP16 for each row of B
  static constexpr uint32_t AI_BYTES = 2 * 128 * 16;          // their A operand: 8 columns (1 1 1 0 ...), 8 of zeros
  static_assert(TMEM_COLS <= 512, "two accumulator sets must fit in tensor memory");
  static_assert(ASTR % 2 == 0 && BUF_BYTES % 16 == 0, "16-byte copies need aligned destinations");
};

// Layout of a loaded tile in shared memory: local entry e at piece_off(e),
// 16-entry pieces (128 bytes) 18 entries apart, so that
// the pieces' banks rotate by two 8-byte words per piece.  Each thread of the
// ket step reads one column of the operator's targets (entries whose indices
// differ in the target bits); with the pieces rotated, the columns a warp
// reads at once fall into different banks even when the targets are the low
// bits.  piece_off is additive over disjoint bit fields.
__device__ __forceinline__ int piece_off(int e) { return e + 2 * (e >> 4); }

template <int K>
struct T64Group {
  static constexpr int D = 1 << K;
  uint64_t full;          // the group's tile loads
  uint64_t mma;           // the group's ket and bra commits, alternating
  uint64_t nbase;         // global index of the group's next tile
  int brkey[128];         // per bra column: magnitude key of the ket outputs
  alignas(16) uint16_t colE[128 / D][D];  // exponent field of ket column (b, f)'s grid, at [f][b]
};

template <int K>
struct T64Tables {
  static constexpr int D = 1 << K;
  uint64_t hiofl[16], hiofh[16];  // offset of run r of a tile: hiofl[r & 15] + hiofh[r >> 4]
  uint64_t offk[D], offb[D];      // offset of output (a, b), free bits aside: offk[a] + offb[b]
  uint16_t stored[D];             // bit a of [b]: the run of output (a, b) is stored; all: every run of the tile is
  int allstored;
  T64Group<K> grp[2];
  int pk[D], pb[D];  // piece_off of the ket / bra index bits
  int ew0[D], ews1[D];  // row exponents of W; of V, by 2^20
  int ewmin1;           // the least of V's
  int hipos[8];
  // the half range of the tiles (HalfMap), if `half`
  int half, mlog, ngap, s, inv;
  uint64_t count;
  uint32_t koff[1 << kHalfMaxS];
  uint8_t gpos[20], gwidth[20];
  uint32_t slot;
};

template <int K>
constexpr size_t t64_smem_bytes() {
  using S = T64<K>;
  return 2 * (size_t)kTc64Slices * S::A_BYTES + 2 * (size_t)kTc64Slices * S::B_BYTES + 2 * (size_t)S::BUF_BYTES +
         2 * (size_t)S::BI_BYTES + S::AI_BYTES + sizeof(T64Tables<K>);
}

// Named barrier of group g (ids 1, 2), and the same with an OR of p over the group.
__device__ __forceinline__ void group_bar(int g) { tc::named_bar<kT64GroupThreads>(1 + g); }
__device__ __forceinline__ bool group_bar_or(int g, bool p) { return tc::named_bar_or<kT64GroupThreads>(1 + g, p); }

__device__ __forceinline__ uint64_t shr_u64(uint64_t x, uint32_t s) {  // s >= 64 gives 0
  uint64_t r;
  asm("shr.b64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));
  return r;
}
__device__ __forceinline__ int64_t shr_s64(int64_t x, uint32_t s) {  // s >= 64 gives the sign
  int64_t r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));
  return r;
}
__device__ __forceinline__ int64_t shl_s64(int64_t x, uint32_t s) {
  int64_t r;
  asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));
  return r;
}

// v + 0x80 in each of the bytes 0..6: the bytes (the top one with bit 56) are
// the digits of v plus 128.
constexpr uint64_t kDigitBias = 0x0080808080808080ull;

// An FP64 value (bits lo, hi) on its column's grid: v = x 2^(1077 - Ec) as
// an integer, |v| <= 2^55; ecm is the column's largest exponent field (hi &
// 0x7FF00000, at least 64 << 20).  kConvert: 1077 - Ec added to the exponent
// field and one conversion on the FP64 pipe, rounded to nearest (zeros and
// subnormals become numbers below 2^-9, hence 0); grids of 2^1077 and above,
// where the exponent field could wrap, shift the significand instead.  Without
// kConvert all do, on the ALU, towards zero.  Three values in four convert: a
// 4-qubit pass at 14 qubits took 2100 us, with all 2170, half 2240, none 2430.
template <bool kConvert>
__device__ __forceinline__ int64_t align_fp64(uint32_t lo, uint32_t hi, uint32_t ecm) {
  if (kConvert && ecm < (1077u << 20)) {
    const uint32_t h = hi + (1077u << 20) - ecm;
    return __double2ll_rn(__longlong_as_double((long long)(((uint64_t)h << 32) | lo)));
  }
  const uint32_t d = (ecm - (hi & 0x7FF00000u)) >> 20;
  const uint64_t mant = ((uint64_t)((hi & 0x000FFFFFu) | 0x00100000u) << 32) | lo;
  const int64_t v = (int64_t)shr_u64(mant << 2, d);
  return (int32_t)hi < 0 ? -v : v;
}

// Store the 7 digit slices of NV consecutive K indices (k0 ..) of operand row
// `row`, u = value + kDigitBias: a byte b is the FP16 number b 2^-24 as it is
// (subnormal; the top digit has 9 bits), so a pair of digits is a byte permute
// or a mask, and nothing is converted.  The 128 that each digit is too large by
// is taken off by the accumulators' starting values (issue_step).  One 16-byte
// (NV = 8) or 8-byte (NV = 4) store per slice.
template <int NV>
__device__ __forceinline__ void store_digits(unsigned char* sA, uint32_t a_bytes, uint32_t off,
                                             const uint64_t (&u)[NV]) {
  uint32_t w[NV / 2] = {};
  auto put = [&](int j) {
    if constexpr (NV == 8)
      *reinterpret_cast<uint4*>(sA + j * a_bytes + off) = make_uint4(w[0], w[1], w[2], w[3]);
    else
      *reinterpret_cast<uint2*>(sA + j * a_bytes + off) = make_uint2(w[0], w[1]);
  };
#pragma unroll
  for (int p = 0; p < NV / 2; p++) w[p] = __byte_perm((uint32_t)(u[2 * p] >> 32), (uint32_t)(u[2 * p + 1] >> 32), 0x7632);
  put(0);
#pragma unroll
  for (int j = 1; j < kTc64Slices; j += 2) {
    // bytes 7 - j and 6 - j of each value: digits j and j + 1
    uint32_t h[NV / 2];
#pragma unroll
    for (int p = 0; p < NV / 2; p++) {
      const uint64_t a = u[2 * p], b = u[2 * p + 1];
      h[p] = j == 1 ? __byte_perm((uint32_t)(a >> 32), (uint32_t)(b >> 32), 0x5410)
                    : __byte_perm((uint32_t)a, (uint32_t)b, j == 3 ? 0x7632 : 0x5410);
      w[p] = __byte_perm(h[p], 0, 0x4341);
    }
    put(j);
#pragma unroll
    for (int p = 0; p < NV / 2; p++) w[p] = h[p] & 0x00FF00FFu;
    put(j + 1);
  }
}

// Y = sum_o S_o 2^(43-8o), orders 6 and 7 each floored, from the accumulators'
// bits kAcc0 + S_o (0.75 + S_o 2^-24 in FP32, |S_o| < 2^22).  Two orders make
// one 32-bit word (b << 8) + b' = p + kAccPair with |p| < 2^30; the constants
// come off at the end.  |Y| < 2^63.
constexpr uint32_t kAcc0 = 0x3F400000u;
constexpr uint32_t kAccPair = 0x7F400000u;  // 257 kAcc0 mod 2^32
constexpr uint64_t kAccSum = ((uint64_t)kAcc0 << 43) + ((uint64_t)kAccPair << 27) + ((uint64_t)kAccPair << 11) +
                             (kAccPair >> 5) + (kAcc0 >> 13);
__device__ __forceinline__ int64_t combine_orders(uint32_t b0, uint32_t b1, uint32_t b2, uint32_t b3, uint32_t b4,
                                                  uint32_t b5, uint32_t b6, uint32_t b7) {
  const uint32_t r12 = b1 * 256u + b2, r34 = b3 * 256u + b4, r56 = b5 * 256u + b6;
  uint64_t acc = (uint64_t)r34 * 2048u + ((r56 >> 5) + (b7 >> 13));
  acc += (uint64_t)r12 * 134217728u;
  acc += (uint64_t)(b0 * 2048u) << 32;
  return (int64_t)(acc - kAccSum);
}

__device__ __forceinline__ int64_t combine_sums(const float (&s)[kTc64Orders][4], int c) {
  auto b = [&](int o) { return __float_as_uint(s[o][c]); };
  return combine_orders(b(0), b(1), b(2), b(3), b(4), b(5), b(6), b(7));
}

// The FP64 bits of Y 2^P: one conversion on the FP64 pipe (correctly
// rounded), then P added to the exponent field.  0 for Y = 0 and below the
// normal range.
__device__ __forceinline__ uint64_t to_fp64(int64_t Y, int P) {
  const uint64_t b = (uint64_t)__double_as_longlong(__ll2double_rn((long long)Y));
  const int E = (int)((b >> 52) & 0x7FF) + P;
  return (Y != 0 && E > 0) ? b + ((uint64_t)(int64_t)P << 52) : 0ull;
}
// The same for P >= -1022, as P 2^20: no integer falls below the normal range.
__device__ __forceinline__ uint64_t to_fp64_near(int64_t Y, uint32_t P20) {
  const uint64_t b = (uint64_t)__double_as_longlong(__ll2double_rn((long long)Y));
  const uint32_t h = (uint32_t)(b >> 32);
  return ((uint64_t)(h ? h + P20 : 0u) << 32) | (uint32_t)b;
}

// Position of the highest bit that differs from the sign, -1 if there is none.
__device__ __forceinline__ int leading_bit(int32_t x) {
  int r;
  asm("bfind.s32 %0, %1;" : "=r"(r) : "r"(x));
  return r;
}

// The group's first warp issues every product of a step, by its elected lane: digit slices A_0..A_6 of the
// 128 columns against the operator's slices, slice pairs of orders 0..7, the
// pairs of order o into the accumulator at TMEM column o*R of the set.  The
// operator's slices are consecutive R-row blocks of one K-major operand, so
// A_i against slices j0..j0+nb-1 is one MMA of N = nb*R.  The first product
// (128 columns of ones against three FP16 numbers a row, TcDesc64::start) sets
// every accumulator to 0.75 - 128 2^-24 sum w: the digits' excess of 128 taken
// off, and a sum whose FP32 bits are an integer (kAcc0 + S).  The warp stays
// together and one lane issues: with the addresses worked out in one lane's
// branch an MMA took 140 cycles, more than it runs, and a pass 2.10 ms for 1.93.
template <int K>
__device__ __forceinline__ void issue_step(const unsigned char* sA, const unsigned char* sBside,
                                           const unsigned char* sAI, const unsigned char* sBI, uint32_t dset,
                                           uint32_t elected) {
  using S = T64<K>;
  constexpr int R = S::R;
  const uint32_t a0 = tc::smem_u32(sA), b0 = tc::smem_u32(sBside);
  // K columns 8..15: A's zeros, 128 rows (2 KB) on; B's are whatever finite
  // numbers follow the row group (the next rows' or side's, or A's ones)
  tc::mma_f16kind_if(elected, dset, tc::smem_desc(tc::smem_u32(sAI), 2048, 128),
                     tc::smem_desc(tc::smem_u32(sBI), 128, 128), tc::idesc_f16_f32(128, kTc64Orders * R), 0u);
#pragma unroll
  for (int i = 0; i < kTc64Slices; i++) {
    const int nb = i == 0 ? kTc64Slices : kTc64Orders - i;  // (i, 0..6 or 7-i)
#pragma unroll
    for (int kk = 0; kk < R / 16; kk++)
      tc::mma_f16kind_if(elected, dset + i * R, tc::smem_desc(a0 + i * S::A_BYTES + kk * 256, tc::kLbo, S::SBO),
                         tc::smem_desc(b0 + kk * 256, tc::kLbo, S::SBO), tc::idesc_f16_f32(128, nb * R), 1u);
  }
}

}  // namespace

template <int K>
__global__ void __launch_bounds__(kT64Threads, 1)
    k_pass_tc64(uint64_t* __restrict__ re, uint64_t* __restrict__ im, const TcDesc64<K>* __restrict__ dp,
                int* __restrict__ err, const HalfMap* __restrict__ hmap, const int* __restrict__ herm, int n) {
  using S = T64<K>;
  constexpr int D = S::D, R = S::R, G = S::G, TILE = S::TILE, ASTR = S::ASTR;
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* sB = smem + 2 * kTc64Slices * S::A_BYTES;                          // W digits, then V digits
  uint64_t* bufs = reinterpret_cast<uint64_t*>(sB + 2 * kTc64Slices * S::B_BYTES);  // [group][re, im][ASTR]
  unsigned char* sBI = reinterpret_cast<unsigned char*>(bufs + 4 * ASTR);  // starting sums of W's, then of V's rows
  unsigned char* sAI = sBI + 2 * S::BI_BYTES;
  T64Tables<K>& tb = *reinterpret_cast<T64Tables<K>*>(sAI + S::AI_BYTES);
  const PassHeader& h = dp->h;
  const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
  const int g = w >> 4, gtid = tid & (kT64GroupThreads - 1), wg = w & 15;
  constexpr int NV = D / 2;  // values a thread holds: a quarter of a column's 2D reals
  // digit steps: column mc = 8 wg + (l & 7), quarter qc = l >> 3 -- half hc =
  // qc >> 1 (real or imaginary parts), values cc NV .. cc NV + NV - 1 of it,
  // cc = qc & 1 (the four quarters of a column in one warp)
  const int mc = 8 * wg + (l & 7), qc = l >> 3, hc = qc >> 1, cc = qc & 1;
  const int rc = mc / G, fc = mc & (G - 1);
  // accumulator steps: column m = 32 (w & 3) + l -- the TMEM lane quadrant
  // its warp may read -- quarter q = (wg >> 2) & 3: half q >> 1, values
  // chunk NV .. of it, chunk = q & 1
  const int m = 32 * (w & 3) + l, q = (wg >> 2) & 3, half = q >> 1, chunk = q & 1;
  const int r = m / G, f = m & (G - 1);
  unsigned char* sA = smem + g * kTc64Slices * S::A_BYTES;  // the group's digit operand (ket, then bra)
  uint64_t* buf = bufs + (size_t)g * 2 * ASTR;             // the group's tile, then its ket outputs
  T64Group<K>& gp = tb.grp[g];

  // ---- per-pass tables, the operator's digits, tensor memory, barriers
  {
    constexpr int per_slice = S::B_BYTES / 16;
    for (int i = tid; i < 2 * kTc64Slices * per_slice; i += blockDim.x) {
      const int side = i / (kTc64Slices * per_slice), rest = i % (kTc64Slices * per_slice);
      reinterpret_cast<uint4*>(sB)[i] = reinterpret_cast<const uint4*>(&dp->sl[side][0][0])[rest];
    }
    for (int i = tid; i < (int)(2 * S::BI_BYTES / 16); i += blockDim.x)
      reinterpret_cast<uint4*>(sBI)[i] = reinterpret_cast<const uint4*>(&dp->start[0][0])[i];
    if (tid < 256)  // FP16 1 1 1 0 0 0 0 0 in 128 rows, then the zeros
      reinterpret_cast<uint4*>(sAI)[tid] = tid < 128 ? make_uint4(0x3C003C00u, 0x00003C00u, 0, 0) : make_uint4(0, 0, 0, 0);
  }
  const int mhi = h.mhi, L = h.L;
  if (tid < 32) {
    uint64_t off = 0;
    for (int j = 0; j < 4; j++)
      if ((tid & 16 ? j + 4 : j) < mhi) off |= (uint64_t)((tid >> j) & 1) << h.hipos[tid & 16 ? j + 4 : j];
    (tid & 16 ? tb.hiofh : tb.hiofl)[tid & 15] = off;
  }
  if (tid < D) {
    int lk = 0, lb = 0;
    for (int i = 0; i < K; i++) {
      lk |= ((tid >> i) & 1) << h.lket[i];
      lb |= ((tid >> i) & 1) << h.lbra[i];
    }
    tb.pk[tid] = piece_off(lk);
    tb.pb[tid] = piece_off(lb);
    tb.ew0[tid] = dp->ew[0][tid];
    tb.ews1[tid] = dp->ew[1][tid] * (1 << 20);
  }
  if (tid < D) {
    uint32_t st = 0;
    for (int a = 0; a < D; a++) {
      int e = 0;
      for (int i = 0; i < K; i++) e |= (((a >> i) & 1) << h.lket[i]) | (((tid >> i) & 1) << h.lbra[i]);
      st |= ((h.stmask[(e >> L) >> 5] >> ((e >> L) & 31)) & 1u) << a;
    }
    tb.stored[tid] = (uint16_t)st;
  }
  if (tid < 2 * D) {
    const int i = tid & (D - 1), side = tid / D;  // side 0: ket index i, 1: bra index i
    int e = 0;
    for (int k = 0; k < K; k++) e |= ((i >> k) & 1) << (side ? h.lbra[k] : h.lket[k]);
    const int run = e >> L;
    uint64_t off = 0;
    for (int j = 0; j < mhi; j++) off |= (uint64_t)((run >> j) & 1) << h.hipos[j];
    off += (uint64_t)(e & ((1 << L) - 1));
    (side ? tb.offb : tb.offk)[i] = off;
  }
  if (tid == 0) {
    int all = 1;
    for (int run = 0; run < (1 << mhi); run++) all &= (int)((h.stmask[run >> 5] >> (run & 31)) & 1);
    tb.allstored = all;
    int e = dp->ew[1][0];
    for (int i = 1; i < D; i++) e = min(e, dp->ew[1][i]);
    tb.ewmin1 = e;
    const HalfMap* hm = hmap && *herm ? hmap : nullptr;
    tb.half = hm != nullptr;
    tb.count = hm ? hm->count : h.ntiles;
    if (hm) {
      tb.mlog = hm->mlog;
      tb.ngap = hm->ngap;
      tb.s = hm->s;
      tb.inv = (int)hm->inv;
    }
  }
  if (hmap && tid >= 32 && tid < 64) tb.koff[tid - 32] = (uint32_t)hmap->koff[tid - 32];
  if (hmap && tid >= 64 && tid < 84) {
    tb.gpos[tid - 64] = hmap->pos[tid - 64];
    tb.gwidth[tid - 64] = hmap->width[tid - 64];
  }
  if (tid < 8) tb.hipos[tid] = h.hipos[tid];
  if (w == 0) {
    tc::tmem_alloc(&tb.slot, S::TMEM_COLS);
    tc::tmem_relinquish();
  }
  if (tid == 0) {
    for (int gi = 0; gi < 2; gi++) {
      tc::mbar_init(&tb.grp[gi].full, kT64GroupThreads);
      tc::mbar_init(&tb.grp[gi].mma, 1);
    }
    tc::mbar_fence_init();
  }
  tc::fence_proxy_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tb.slot + (uint32_t)g * S::SET_COLS;  // the group's accumulator set
  const uint32_t tlane = (uint32_t)(32 * (w & 3)) << 16;

  auto free_off = [&](int ff) {  // local offset of free group ff
    int o = 0;
    for (int j = 0; j < h.g; j++) o |= ((ff >> j) & 1) << h.freepos[j];
    return o;
  };
  const int lf = free_off(f);  // accumulator steps: free offset of column (., f) in the state
  // digit steps: column (b = rc, fc)'s values a = cc NV + i of half hc at
  // buf[basec + the strides tb.pk[1, 2, 4] of i's bits]
  const int basec = hc * ASTR + tb.pb[rc] + piece_off(free_off(fc)) + tb.pk[cc * NV];
  const uint64_t ntiles = tb.count, gstep = 2 * (uint64_t)gridDim.x;
  const int runlen = 1 << L;
  // The ket step's exact integer outputs Y(a, b) of column (b, ff) replace
  // the tile in its buffer, at [hh][a][b ^ (a & 1)][ff]: the ket step writes,
  // for one a, 32 consecutive words per warp, and the bra step reads, for one
  // b, columns a of both parities -- both free of bank conflicts.
  auto yoff = [&](int hh, int a, int b, int ff) { return hh * ASTR + (a * D + (b ^ (a & 1))) * G + ff; };
  auto tile_base_s = [&](uint64_t t) {  // tile_base / half_base from the staged positions
    if (tb.half) {
      uint32_t I, J;
      half_pair((uint32_t)(t >> tb.mlog), tb.s, (uint32_t)tb.inv, I, J);
      uint64_t x = (t & ((1ull << tb.mlog) - 1)) << L;
      for (int i = 0; i < tb.ngap; i++) {
        const int p = tb.gpos[i];
        x = ((x >> p) << (p + tb.gwidth[i])) | (x & ((1ull << p) - 1));
      }
      return x | tb.koff[I] | ((uint64_t)tb.koff[J] << n);
    }
    uint64_t base = t << L;
    for (int j = 0; j < mhi; j++) {
      const int p = tb.hipos[j];
      base = ((base >> p) << (p + 1)) | (base & ((1ull << p) - 1));
    }
    return base;
  };

  // Loads of a tile into the group's buffer, by every thread of the group
  // after a group barrier that frees it: 16-byte asynchronous copies, a
  // thread's the same entries of the real and the imaginary array, each
  // thread's arriving on the group's barrier when they have landed.  (1-D bulk
  // copies of 128 bytes took a warp about 90 cycles each to issue: 2900 cycles
  // a tile on half the warps, of 20000.)
  auto copy_tile = [&](uint64_t base) {
#pragma unroll
    for (int k = 0; k < TILE / 2 / kT64GroupThreads; k++) {
      const int e0 = 2 * (gtid + k * kT64GroupThreads), run = e0 >> L;
      const uint64_t src = base + tb.hiofl[run & 15] + tb.hiofh[run >> 4] + (uint64_t)(e0 & (runlen - 1));
      uint64_t* dst = buf + piece_off(e0);
      tc::cp_async16(dst, re + src);
      tc::cp_async16(dst + ASTR, im + src);
    }
    tc::cp_async_arrive(&gp.full);
  };

  // outstanding asynchronous work of this thread's view; a phase that did not
  // complete stays pending (the teardown waits for it again)
  uint32_t phf = 0, phm = 0;
  int pendf = 0, pendm = 0;
  bool bad = false;  // one of this thread's waits expired
  auto wait = [&](uint64_t* bar, uint32_t& ph, int& pend) {
    if (!tc::mbar_wait_bounded(bar, ph, kT64WaitPolls)) {
      bad = true;
      return false;
    }
    ph ^= 1u;
    pend = 0;
    return true;
  };

  // ---- prologue: the group's first tile in flight
  pdl_wait();
  pdl_begin();
  uint64_t t = blockIdx.x + (uint64_t)g * gridDim.x;
  uint64_t tbase = t < ntiles ? tile_base_s(t) : 0;
  if (t < ntiles) {
    copy_tile(tbase);
    pendf = 1;
  }

  for (; t < ntiles; t += gstep) {
    // ---- 1: the tile's values of column (b = rc, fc), quarter qc, its grid
    // (the largest exponent of the column's four quarters, two shuffles
    // away), its ket digits
    wait(&gp.full, phf, pendf);
    {
      uint64_t u[NV];
      uint32_t emx = 0;
      const int p1 = tb.pk[1], p2 = tb.pk[2], p4 = tb.pk[4];
#pragma unroll
      for (int i = 0; i < NV; i++) {
        u[i] = buf[basec + (i & 1 ? p1 : 0) + (i & 2 ? p2 : 0) + (i & 4 ? p4 : 0)];
        emx = max(emx, (uint32_t)(u[i] >> 32) & 0x7FF00000u);
      }
      emx = max(emx, __shfl_xor_sync(0xffffffffu, emx, 8));
      emx = max(emx, __shfl_xor_sync(0xffffffffu, emx, 16));
      const uint32_t ecm = max(emx, 64u << 20);
      if (qc == 0) gp.colE[fc][rc] = (uint16_t)(ecm >> 20);
#pragma unroll
      for (int i = 0; i < NV; i++) {
        const uint32_t lo = (uint32_t)u[i], hi = (uint32_t)(u[i] >> 32);
        u[i] = (uint64_t)((i & 3) != 3 ? align_fp64<true>(lo, hi, ecm) : align_fp64<false>(lo, hi, ecm)) + kDigitBias;
      }
      store_digits<NV>(sA, S::A_BYTES, tc_kmajor_offset(mc, hc * D + cc * NV, S::SBO), u);
    }
    tc::fence_proxy_async_smem();
    tc::fence_before_sync();
    if (group_bar_or(g, bad)) break;
    tc::fence_after_sync();

    // ---- 2: ket products
    if (wg == 0) {
      const uint32_t elected = tc::elect_one();
      issue_step<K>(sA, sB, sAI, sBI, tmem, elected);
      if (elected) tc::mma_commit(&gp.mma);
    }
    pendm = 1;
    const uint64_t tn = t + gstep;
    // one thread finds the group's next tile while the products run (every
    // thread reads it in step 5, two barriers on)
    if (gtid == kT64GroupThreads - 1 && tn < ntiles) gp.nbase = tile_base_s(tn);

    // ---- 3: ket outputs of column (b = r, f) -> exact integers, in place of
    // the tile
    if (wait(&gp.mma, phm, pendm)) {
      tc::fence_after_sync();
#pragma unroll
      for (int c4 = 0; c4 < NV; c4 += 4) {
        float sv[kTc64Orders][4];
        const uint32_t ta = tmem + tlane + half * D + chunk * NV + c4;
#pragma unroll
        for (int o = 0; o < kTc64Orders; o++) tc::tmem_ld4(ta + o * R, sv[o]);
        tc::tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 4; c++) buf[yoff(half, chunk * NV + c4 + c, r, f)] = (uint64_t)combine_sums(sv, c);
      }
    }
    tc::fence_before_sync();
    if (group_bar_or(g, bad)) break;
    tc::fence_after_sync();

    // ---- 4: bra digits of column (a = rc, fc), quarter qc.  The column's key
    // is the largest of the grid Ec(b) plus the leading bit of Y_b's high word
    // (|Y_b| <= 2^(33 + bit)), over the four quarters, two shuffles away; Y_b
    // shifts right by key - 22 - Ec(b), so |v| <= 2^55.  Left shifts are for
    // columns that cancelled to below 2^-8 of what their inputs could give: rare.
    {
      uint64_t u[NV];
      int sh[NV], key = 0, least = 0;
      uint32_t ee[NV / 2];
      if constexpr (NV == 8) {
        const uint4 e = *reinterpret_cast<const uint4*>(&gp.colE[fc][cc * NV]);
        ee[0] = e.x, ee[1] = e.y, ee[2] = e.z, ee[3] = e.w;
      } else {
        const uint2 e = *reinterpret_cast<const uint2*>(&gp.colE[fc][cc * NV]);
        ee[0] = e.x, ee[1] = e.y;
      }
#pragma unroll
      for (int i = 0; i < NV; i++) {
        u[i] = buf[yoff(hc, rc, cc * NV + i, fc)];
        sh[i] = (int)(i & 1 ? ee[i / 2] >> 16 : ee[i / 2] & 0xFFFFu);
        key = max(key, sh[i] + leading_bit((int32_t)(u[i] >> 32)));
      }
      key = max(key, __shfl_xor_sync(0xffffffffu, key, 8));
      key = max(key, __shfl_xor_sync(0xffffffffu, key, 16));
      if (qc == 0) gp.brkey[mc] = key;
#pragma unroll
      for (int i = 0; i < NV; i++) {
        sh[i] = key - 22 - sh[i];
        least = min(least, sh[i]);
      }
      if (least >= 0) {
#pragma unroll
        for (int i = 0; i < NV; i++) u[i] = (uint64_t)shr_s64((int64_t)u[i], (uint32_t)sh[i]) + kDigitBias;
      } else {
#pragma unroll
        for (int i = 0; i < NV; i++)
          u[i] = (uint64_t)(sh[i] >= 0 ? shr_s64((int64_t)u[i], (uint32_t)sh[i])
                                       : shl_s64((int64_t)u[i], (uint32_t)(-sh[i]))) + kDigitBias;
      }
      store_digits<NV>(sA, S::A_BYTES, tc_kmajor_offset(mc, hc * D + cc * NV, S::SBO), u);
    }
    tc::fence_proxy_async_smem();
    tc::fence_before_sync();
    group_bar(g);
    tc::fence_after_sync();

    // ---- 5: bra products; the group's next tile into the freed buffer
    if (wg == 0) {
      const uint32_t elected = tc::elect_one();
      issue_step<K>(sA, sB + kTc64Slices * S::B_BYTES, sAI, sBI + S::BI_BYTES, tmem, elected);
      if (elected) tc::mma_commit(&gp.mma);
    }
    pendm = 1;
    const uint64_t nbase = gp.nbase;
    if (tn < ntiles) {
      copy_tile(nbase);
      pendf = 1;
    }

    // ---- 6: bra outputs of column (a = r, f) -> FP64 -> the tile's stored runs
    if (wait(&gp.mma, phm, pendm)) {
      tc::fence_after_sync();
      const int pa = gp.brkey[m] + tb.ew0[r] - 993;
      const bool near = pa + tb.ewmin1 >= -1022;
      const uint32_t pa20 = (uint32_t)pa << 20;
      const uint64_t s1 = tb.offb[1], s2 = tb.offb[2];
#pragma unroll
      for (int c4 = 0; c4 < NV; c4 += 4) {
        float sv[kTc64Orders][4];
        const uint32_t ta = tmem + tlane + half * D + chunk * NV + c4;
#pragma unroll
        for (int o = 0; o < kTc64Orders; o++) tc::tmem_ld4(ta + o * R, sv[o]);
        tc::tmem_wait_ld();
        uint64_t* col = (half ? im : re) + tbase + lf + tb.offk[r] + tb.offb[chunk * NV + c4];
        if (tb.allstored && near) {  // the common case
#pragma unroll
          for (int c = 0; c < 4; c++)
            col[(c & 1 ? s1 : 0) + (c & 2 ? s2 : 0)] =
                to_fp64_near(combine_sums(sv, c), pa20 + (uint32_t)tb.ews1[chunk * NV + c4 + c]);
        } else {
#pragma unroll
          for (int c = 0; c < 4; c++) {
            const int b = chunk * NV + c4 + c;
            if (!((tb.stored[b] >> r) & 1)) continue;  // a run the pass does not change
            col[(c & 1 ? s1 : 0) + (c & 2 ? s2 : 0)] = to_fp64(combine_sums(sv, c), pa + tb.ews1[b] / (1 << 20));
          }
        }
      }
    }
    tc::fence_before_sync();  // the next tile's first group barrier orders these reads before its MMAs
    tbase = nbase;
  }

  // ---- teardown: nothing of this group may still be in flight when the
  // block's tensor memory and shared memory are released (bounded, after an
  // expiry)
  if (group_bar_or(g, bad)) {
    if (pendm) tc::mbar_wait_bounded(&gp.mma, phm, kT64WaitPolls << 2);
    if (pendf) tc::mbar_wait_bounded(&gp.full, phf, kT64WaitPolls << 2);
    if (gtid == 0) atomicExch(err, 1);
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (w == 0) tc::tmem_dealloc(tb.slot, S::TMEM_COLS);
}

template <int K>
static cudaError_t configure_tc64() {
  constexpr size_t smem = t64_smem_bytes<K>();
  static_assert(smem <= 227 * 1024, "one block's shared memory");
  cudaError_t e = cudaFuncSetAttribute(k_pass_tc64<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_pass_tc64<K>, cudaFuncAttributePreferredSharedMemoryCarveout,
                             (int)cudaSharedmemCarveoutMaxShared);
  return e;
}

template <int K>
static cudaError_t launch_tc64_k(const LaunchArgs& a, cudaStream_t s) {
  static PerContext configured;
  const cudaError_t e = configured.get([](int*) { return configure_tc64<K>(); });
  if (e != cudaSuccess) return e;
  return launch_kernel(a.pdl, k_pass_tc64<K>, a.grid, kT64Threads, t64_smem_bytes<K>(), s, static_cast<uint64_t*>(a.re),
                       static_cast<uint64_t*>(a.im), static_cast<const TcDesc64<K>*>(a.desc), a.err, a.half, a.herm,
                       a.n);
}

cudaError_t launch_pass_tc64(const LaunchArgs& a, cudaStream_t s) {
  if (!a.err || (a.K != 3 && a.K != 4) || a.arith != AR_FP64) return cudaErrorInvalidValue;
  return a.K == 3 ? launch_tc64_k<3>(a, s) : launch_tc64_k<4>(a, s);
}

}  // namespace dmg

// pass.h -- one superoperator pass over the vectorised density matrix.
//
// The state is the 4^n-entry array A with A[c*2^n + r] = rho[r][c]: the layout
// of DM-Sim's dm_real_res/dm_imag_res after sim() (src/dmsim_nvgpu_omp.cuh:
// 456-459), held as separate real and imaginary arrays.  Ket qubit q is bit q
// of the index and bra qubit q is bit q+n.  A pass applies a K-qubit operator
// U (K <= 4) as U (x) conj(U) on bits {q_i} and {q_i + n} in place.
//
// Tiling.  A tile is the closed set of G * 4^K entries (G = 256/2^K groups)
// that the operator mixes, chosen so that it is made of 2^mhi contiguous runs
// of 2^L entries: the low L index bits (which hold the low target bits plus
// log2(G) free bits) are contiguous in memory and the mhi target bits at or
// above L select the run.  Loads and stores of a run are coalesced 16-byte
// vector accesses whatever qubits the pass targets.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define DMG_HD __host__ __device__
#else
#define DMG_HD
#endif

namespace dmg {

constexpr int kThreads = 256;  // threads per block of every pass kernel
constexpr int kMaxK = 4;       // widest fused operator
constexpr int kMaxD = 16;      // 2^kMaxK

// Arithmetic class of a pass; selects the kernel instance.
enum PassClass : int32_t {
  CLS_MOVE = 0,    // monomial superoperator, every factor exactly 1 (X, CX, SWAP, Toffoli blocks)
  CLS_SIGNED = 1,  // monomial, factors in {1,-1,+i,-i}: sign and re/im swaps only (Y, Z, S, CZ)
  CLS_PHASE = 2,   // monomial with general complex factors (T, U1, controlled phases)
  CLS_DENSE = 3,   // general U, applied ket side then bra side (dense rows)
  CLS_SPARSE = 4,  // general U with sparse rows (per-row column lists)
  CLS_RLIN = 5,    // real-linear 1-qubit map (DM-Sim's SRN gate), K = 1
  CLS_SUPER = 6,   // general superoperator (a noise channel), K <= 2: 4^K x 4^K on the (ket, bra) sub-index
  CLS_COUNT = 7
};

// Kernel instances for DENSE / SPARSE passes whose U and V are real (the
// imaginary parts vanish, e.g. H, RY and their products with permutations):
// two real multiply-adds per complex term instead of four.  The host classes
// stay CLS_DENSE / CLS_SPARSE; PassHeader::flags marks such passes.
constexpr int kClsRealOffset = 16;
constexpr int CLS_DENSE_REAL = kClsRealOffset + CLS_DENSE;
constexpr int CLS_SPARSE_REAL = kClsRealOffset + CLS_SPARSE;
DMG_HD constexpr int base_class(int c) { return c % kClsRealOffset; }
DMG_HD constexpr bool real_class(int c) { return c >= kClsRealOffset; }
constexpr int32_t kPassRealOperator = 1;  // PassHeader::flags bit
constexpr int32_t kPassHadamard = 2;      // flags bit: 1 qubit, V = conj(U), every entry of U is +-sqrt(1/2)
// Instance of the 1-qubit register kernel for kPassHadamard passes on an FP64 state.
constexpr int CLS_HADAMARD = 2 * kClsRealOffset + 3;

// Factor kinds of a monomial superoperator entry f[a][b].
enum FactorKind : int8_t { FK_ONE = 0, FK_NEG = 1, FK_PI = 2, FK_NI = 3, FK_GEN = 4 };

struct PassHeader {
  int32_t K, cls;
  int32_t L;         // low run bits
  int32_t mhi;       // number of target bits >= L
  int32_t g;         // log2 of groups per tile
  int32_t flags;     // kPassRealOperator: U and V are real; kPassHadamard
  uint64_t ntiles;   // tiles in the state
  int32_t hipos[8];  // global positions of the high target bits, ascending
  int32_t lket[4];   // local bit position of ket target i (qubit q_i)
  int32_t lbra[4];   // local bit position of bra target i (bit q_i + n)
  int32_t freepos[8];// local positions of the g free low bits, ascending
  uint32_t ldmask[8];   // bit h set: run h is read (it holds a source of a stored entry)
  uint32_t stmask[8];   // bit h set: run h is written (it holds an entry the pass changes)
};

// Operator payload for width K (D = 2^K).  A pass applies U to the ket
// sub-index and V to the bra sub-index; a superoperator pass has V = conj(U),
// a ket-only pass (the reference's forward/backward stages) has V = I.
template <int K>
struct PassOp {
  static constexpr int D = 1 << K;
  double ure[D * D], uim[D * D];   // U row-major (DENSE/SPARSE)
  double vre[D * D], vim[D * D];   // V row-major (DENSE/SPARSE)
  double fre[D * D], fim[D * D];   // f[a*D+b] = U[a][src a] * V[b][srcb b] (PHASE)
  double rlin[16];                 // RLIN: ket 4x4 real map on (r0,i0,r1,i1)
  double rlinb[16];                // RLIN: bra 4x4 real map
  int8_t nnz[D], nnzb[D];          // SPARSE: nonzeros per row of U and of V
  int8_t nnzmax, nnzbmax;          // SPARSE: largest row count of U and of V
  // SUPER: S[(a*D+b)*D*D + (c*D+e)] maps entry (c, e) to entry (a, b)
  double sre[K <= 2 ? D * D * D * D : 1], sim[K <= 2 ? D * D * D * D : 1];
  int8_t col[D * D], colb[D * D];  // SPARSE: column lists per row
  int8_t src[D], srcb[D];          // monomial: source index of row a of U / row b of V
  int8_t fk[D * D];                // monomial: factor kind of f[a][b]
};

template <int K>
struct PassDesc {
  PassHeader h;
  PassOp<K> op;
};

// ---- several narrow passes in one sweep (kernels_multi.cu)
constexpr int kMultiOps = 16, kMultiThreads = 128;
enum MultiKind : int32_t { MO_DENSE = 0, MO_REAL = 1, MO_HADAMARD = 2, MO_MONO = 3, MO_CHANNEL = 4, MO_CX = 5, MO_CHANNEL2 = 6 };
struct MultiOp {
  // DENSE, REAL: U, V (re, im each); MONO: f re, im at [a * 2 + b]; CHANNEL: its eight terms;
  // CHANNEL2: the terms between the diagonal entries at [to * 4 + from], then the others' own at 16 + [a * 4 + b]
  double c[32];
  int32_t kind;
  int32_t p;      // 0: on qubit qa (CX: its control; CHANNEL2: its first qubit), 1: on qubit qb
  int32_t flags;  // HADAMARD: 1 outputs swapped, 2 the mixed ones negated; MONO: 1 X, 2 factors; CHANNEL: as its kernel
  int8_t fk[4];   // MONO: FactorKind at [a * 2 + b]
};
struct MultiDesc {
  int32_t nops, qa, qb;  // qa < qb
  MultiOp op[kMultiOps];
};

// ---- half-range passes
// rho is Hermitian through a whole run (U rho U^dagger and every channel keep
// it so), so a pass may leave one entry of every pair rho[r][c], rho[c][r]
// stale.  S is a set of qubits that the pass does not target: all the entries
// of a tile have the same ket bits and the same bra bits on S, so the tile as
// a whole has r & S <= c & S or it has not, and only the tiles that have are
// enumerated -- (1 + 2^-|S|) / 2 of them.  Consecutive passes share one S as
// long as none targets a qubit of it; between two different sets, and at the
// end of the run, a mirror pass copies the conjugate transpose into the stale
// entries that the next set needs.  FP64 and double-float runs only.
// Measured, whole against half with the mirrors: 14 qubits, 200 mixed gates
// fused, 460 -> 266 ms; 13 qubits gate by gate 264 -> 145 ms; 10 qubits fused
// (state in L2) 0.63 -> 0.52 ms.
//
// Tiles (or, for the register kernel, groups of four entries) are numbered
// k = pair << mlog | m: `pair` counts the ordered pairs I <= J of S values,
// m the remaining bits.  The global index of the first entry is m << L with
// zero gaps inserted at the S bits and at the high target bits, plus koff[I]
// and boff[J].
constexpr int kHalfMaxS = 5;  // 33/64 of the tiles
struct HalfMap {
  uint32_t mask;             // S
  int32_t s;                 // |S|, 1..kHalfMaxS
  int32_t mlog;
  int32_t ngap;
  uint64_t count;            // tiles (groups) of the half range
  uint32_t inv;              // ceil(2^16 / (2^s + 1)): the pair's row without a division
  uint8_t pos[20], width[20];// gaps, ascending: `width` zero bits at `pos`
  uint64_t koff[1 << kHalfMaxS], boff[1 << kHalfMaxS];
};

// The p-th pair I <= J < B = 2^s: rows I and B-1-I of the triangle together
// hold B + 1 pairs.
DMG_HD inline void half_pair(uint32_t p, int s, uint32_t inv, uint32_t& I, uint32_t& J) {
  const uint32_t B = 1u << s;
  const uint32_t i = (p * inv) >> 16;
  const uint32_t j = p - i * (B + 1);
  const bool lower = j < B - i;
  I = lower ? i : B - 1 - i;
  J = lower ? i + j : j - 1;
}
// Global index of the first entry of tile k of the half range.
DMG_HD inline uint64_t half_base(const HalfMap& hm, uint64_t k, int L) {
  uint32_t I, J;
  half_pair((uint32_t)(k >> hm.mlog), hm.s, hm.inv, I, J);
  uint64_t x = (k & ((1ull << hm.mlog) - 1)) << L;
  for (int g = 0; g < hm.ngap; g++) {
    const int p = hm.pos[g];
    x = ((x >> p) << (p + hm.width[g])) | (x & ((1ull << p) - 1));
  }
  return x | hm.koff[I] | hm.boff[J];
}

// ---- tensor-core passes (K = 3, 4; double-float or complex64 state)
// The ket step multiplies each tile column x (2^K complex entries, as 2R
// reals [re; im]) by the real embedding W = [[Ur, -Ui], [Ui, Ur]] (R x R,
// R = 2^(K+1)); the bra step does the same with V.  Both factors are split
// into BF16 "slices" of 8 bits each on a per-row (W) or per-column (x)
// power-of-two grid, so every slice product is an exact multiple of one unit
// per order i + j and the FP32 tensor-core sums of each order are exact; the
// orders are added in double-float.  The W/V slices are computed on the host.
constexpr int kTcSlices = 6;

// Byte offset of element (row, k) of a K-major, unswizzled BF16 tensor-core
// operand: 8-row x 16-byte core matrices (128 contiguous bytes), 128 bytes
// apart along k, `sbo` bytes apart between 8-row groups.
DMG_HD constexpr uint32_t tc_kmajor_offset(uint32_t row, uint32_t k, uint32_t sbo) {
  return (row >> 3) * sbo + (k >> 3) * 128u + (row & 7) * 16u + (k & 7) * 2u;
}

// ---- FP64-width tensor-core passes (K = 3, 4; FP64 state)
// Every operand value is an integer on a power-of-two grid, split into 7
// balanced base-256 digits (|digit| <= 128, exact in FP16): 55 significant
// bits for the largest value of each column of the state, 56 for each row
// of the operator.  Slice pairs of orders i + j = 0..7 accumulate exactly in
// FP32 (every partial sum is an integer below 2^22), the orders are combined
// in 64-bit integer arithmetic and rounded once to FP64.  The state's digits
// are stored as digit + 128 times 2^-24 (a byte is that FP16 subnormal as it
// is); the sums start 128 times the operator's digits lower.
constexpr int kTc64Slices = 7;
constexpr int kTc64Orders = 8;

template <int K>
struct TcDesc64 {
  static constexpr int D = 1 << K, R = 2 * D;
  PassHeader h;  // tile geometry, g = 7 - K (128 columns per step)
  // Row exponents: row n of W (0) or V (1) equals 2^ew[side][n mod D] times
  // sum_j digit_j 256^(6-j); rows n and n + D (the real and imaginary parts
  // of output n) hold the same magnitudes and share the exponent.
  int32_t ew[2][D];
  // digits j = 0..6 of W (0) and V (1): FP16 bits, K-major core-matrix layout
  alignas(16) uint16_t sl[2][kTc64Slices][R * R];
  // the order sums' starting values 0.75 - 128 2^-24 C, C = sum over the slice
  // pairs of order o and over k of w_j[n][k]: row o R + n is the FP16 numbers
  // 0.75, -c1 2^-9, -c0 2^-17 and five zeros, C = 256 c1 + c0, |c0| <= 128
  alignas(16) uint16_t start[2][kTc64Orders * R * 8];
};

template <int K>
struct TcDesc {
  static constexpr int D = 1 << K, R = 2 * D;
  PassHeader h;  // tile geometry, g = 7 - K (128 columns per step)
  // slices of W (0) and V (1): row n of W = sum_j sl[0][j][n][.], slice j on
  // the grid 2^(e_n - 7 - 8j) with |W[n][.]| < 2^e_n (BF16 bits at true
  // scale, K-major core-matrix layout).  For a complex64 state, slices 0..2
  // hold each entry's own BF16 x 3 split (hi, mid, lo) instead.
  alignas(16) uint16_t sl[2][kTcSlices][R * R];
};

}  // namespace dmg

// Integer and float64 GEMMs as triangular digit products on the tcgen05
// tensor cores.
//
// An operand element is a fixed-point number X written in s balanced digits
// of 8 bits, X = sum_p sigma_p 256^(...), sigma_p in [-128, 128], each exact
// in float16.  Digit products with the same p + q = d share a weight, so
// with D_d = sum over p + q = d of sum_k sigma^A_p sigma^B_q
//   integers  (p counts from the lowest digit):  A B = sum_d D_d 256^d
//             modulo 256^s: exactly the diagonals d < s are kept, and the
//             result is numc's wrapped sum (numc wraps in the storage width
//             on every path, src/intrinsics/gemm_avx2.h:1480-1990);
//   float64   (p counts from the highest digit; Ozaki, Ogita, Oishi, Rump,
//             Numer. Algorithms 59, 2012): the diagonals d < s carry the
//             result down to 2^-8s of the row and column maxima.
// Both keep the same s (s + 1) / 2 products: 3, 10 and 36 for 16-, 32- and
// 64-bit integers, 36 for float64 with 8 digits.
//
// What bounds it: a kernel that multiplies one digit pair at a time fetches
// every digit plane up to s times (8.2 TB/s of operands from L2 and 36 % of
// the tensor peak for float64 at 4096^3).  Here one pipeline stage holds all
// s digit planes of a 16-deep K step of both operands, and all their
// products are issued from that one copy.  The accumulators of the s
// diagonals lie side by side in TMEM (BN columns each), so the digits q of B,
// stacked as rows of one shared-memory tile, form one wide MMA per digit p of
// A: columns [p + q] accumulate A_p B_q for a whole range of q at once (N up
// to 256), and operand traffic per multiply-add falls by 2.25 for s = 8.
// float64 4096^3, s = 8: 7.00 -> 2.82 ms for the GEMM (1750 TFLOP/s of slice
// products, 0.91 of the measured bf16 peak); what is left is the MMAs of 64
// columns (48 cycles each instead of 32: shared-memory reads of A) and the
// read-back below.
//
// FP32 accumulation in TMEM is exact while K_chunk * (p + q + 1) * 2^14 <=
// 2^24, so after 1024 / s of K the diagonals are read back as integers and
// folded into wide integers held in registers.  Where the diagonals fill TMEM
// (8 of 64 columns, 4 of 128) they are released in two groups at different
// times, each read back while the other is multiplied.
//
// The operand layout is written by the digit passes as the shared-memory
// image of a stage: blocks of 128 rows (A) or BN rows (B^T), per block and
// 16-deep K step the s digit planes one after another, 32-byte rows in the
// 32-byte-swizzle order that the MMA reads.  A stage is then one or two
// contiguous bulk copies, without tensor maps, and ragged last blocks store
// only the rows that they have.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <type_traits>

#include "kernels.h"
#include "phase_timing.h"
#include "status.h"
#include "tc_common.cuh"

namespace numc_k {
namespace {

constexpr int kBM = 128;       // rows of a tile (one CTA, M = 128 MMAs)
constexpr int kKS = 16;        // K depth of a K step (one MMA)
constexpr int kRowBytes = kKS * 2;
constexpr int kEpiWarps = 16;  // 4 per TMEM lane quarter
constexpr int kMmaHigh = 2 + kEpiWarps;   // the second issuing warp
constexpr int kThreads = 32 * (kMmaHigh + 1);
constexpr int kRingBytes = 196608;
constexpr uint32_t kMagicBits = 0x4B400000u;   // 1.5 x 2^23 as a float

inline int64_t round_up(int64_t x, int64_t a) { return (x + a - 1) / a * a; }

// ---- digit layout -----------------------------------------------------------
// Element offset of the 8-element chunk c (0 or 1) of row r, K step kb, digit
// p, in an operand of R rows cut into blocks of BR rows, s digits, Ks K steps.
__device__ __forceinline__ int64_t digit_offset(int64_t r, int kb, int p, int c, int64_t R,
                                                int BR, int s, int64_t Ks) {
  const int64_t b = r / BR;
  const int rb = (int)(R - b * BR < BR ? R - b * BR : BR);   // rows of this block
  const int rl = (int)(r - b * BR);
  return b * BR * s * Ks * kKS + ((int64_t)kb * s + p) * rb * kKS + rl * kKS +
         (c ^ ((rl >> 2) & 1)) * 8;
}

// Digits of two elements as a float16 pair, from byte `i` (0..3) of two words
// whose bytes hold digit + 128: 0x6400 | byte is 1024 + byte in float16.
__device__ __forceinline__ uint32_t half2_minus_1152(uint32_t v) {
  const uint32_t bias = 0x64806480u;   // 1152 = 1024 + 128
  const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&v),
                            *reinterpret_cast<const __half2 *>(&bias));
  return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ uint32_t digit_pair(uint32_t w0, uint32_t w1, int i) {
  const uint32_t v = __byte_perm(w0, w1, i | i << 4 | (4 + i) << 8 | (4 + i) << 12);
  return half2_minus_1152((v & 0x00ff00ffu) | 0x64006400u);
}

// One operand of the digit pass: R rows of src[r * rs_row + k * rs_k], cut
// into blocks of BR rows.
struct DigitOperand {
  const void *src;
  int64_t rs_row, rs_k, R;
  uint16_t *dst;
  int BR;
  const unsigned long long *maxbits = nullptr;   // float64: largest |x| of each row (bits)
  int headroom = 0;                               // float64: added to every row's exponent
};

// 8 elements along k from k0 (zero past K), 16-byte loads where the row is
// contiguous and aligned.
template <typename T>
__device__ __forceinline__ void load8(const T *row, int64_t rs_k, int64_t k0, int64_t K,
                                      T (&x)[8]) {
  const T *p = row + k0 * rs_k;
  if (rs_k == 1 && k0 + 8 <= K && ((uintptr_t)p & 15) == 0) {
    constexpr int V = 16 / sizeof(T);
#pragma unroll
    for (int i = 0; i < 8 / V; i++) {
      const uint4 v = *reinterpret_cast<const uint4 *>(p + i * V);
      *reinterpret_cast<uint4 *>(&x[i * V]) = v;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; i++) x[i] = k0 + i < K ? p[i * rs_k] : T(0);
  }
}

// The digit pass: a warp takes 8 rows x 32 k (rows of 4 eight-element
// chunks), a block 64 rows x 32 k.  Contiguous rows are read as whole 128- or
// 256-byte lines, row-contiguous operands (B, read as B^T) as 8-element
// segments that fill sectors; per digit a warp writes two runs of 256 bytes.
// Every block clears its share of C for a K-split GEMM that adds into it.
template <typename T, int S>
__global__ void __launch_bounds__(256)
int_digits(DigitOperand a, DigitOperand b, int64_t K, int64_t Ks, unsigned kgroups,
           unsigned groups_a, T *zero, int64_t rso, int64_t cso, int64_t M, int64_t N) {
  tc::griddep_launch_dependents();   // the GEMM may launch and set up meanwhile
  if (zero) {
    const int64_t n = M * N, step = (int64_t)gridDim.x * 256;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += step)
      zero[i / N * rso + i % N * cso] = 0;
  }
  unsigned rg = blockIdx.x / kgroups;
  const unsigned kg = blockIdx.x % kgroups;
  const bool second = rg >= groups_a;
  const DigitOperand &o = second ? b : a;
  if (second) rg -= groups_a;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t r = (int64_t)rg * 64 + warp * 8 + (lane >> 2);
  const int64_t k0 = (int64_t)kg * 32 + (lane & 3) * 8;
  const int kb = (int)(k0 / kKS), c = (int)(k0 / 8) & 1;
  if (r >= o.R || kb >= Ks) return;
  T x[8];
  load8((const T *)o.src + r * o.rs_row, o.rs_k, k0, K, x);
  // digit + 128 per byte: adding 0x80 to every byte position makes the
  // bytes of the (wrapped) sum the balanced digits
  const T c80 = (T)0x8080808080808080ull;
#pragma unroll
  for (int i = 0; i < 8; i++) x[i] = (T)(x[i] + c80);
#pragma unroll
  for (int p = 0; p < S; p++) {
    uint32_t h[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint64_t u0 = x[2 * j], u1 = x[2 * j + 1];
      h[j] = digit_pair((uint32_t)(u0 >> (p & 4) * 8), (uint32_t)(u1 >> (p & 4) * 8), p & 3);
    }
    *reinterpret_cast<uint4 *>(o.dst + digit_offset(r, kb, p, c, o.R, o.BR, S, Ks)) =
        make_uint4(h[0], h[1], h[2], h[3]);
  }
}

// ---- float64 ----------------------------------------------------------------

// Bit tests on float64 values: GB300's FP64 pipe is slow, so compares on
// doubles are done on their IEEE bit patterns in the integer pipes.
__device__ __forceinline__ bool finite_bits(unsigned long long a) {
  return a < 0x7FF0000000000000ull;
}
// frexp exponent of a non-negative finite double given as bits (0 for 0):
// x = m 2^e with m in [0.5, 1).
__device__ __forceinline__ int frexp_exp_bits(unsigned long long a) {
  if (a == 0) return 0;
  const int field = (int)(a >> 52);
  if (field) return field - 1022;
  return (64 - __clzll((long long)a)) - 1074;   // subnormal: a * 2^-1074
}

// Largest of the warp's values, in every lane.
__device__ __forceinline__ unsigned long long warp_max(unsigned long long m) {
  const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(m >> 32));
  const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(m >> 32) == hi ? (unsigned)m : 0u);
  return (unsigned long long)hi << 32 | lo;
}

// One operand of the maxima pass: out[row] = max over k of |src[row * rs_row +
// k * rs_k]| as IEEE bits (atomicMax on the bit pattern orders non-negative
// doubles), flags[row / flag_rows] = gen for non-finite values.
struct MaxOperand {
  const unsigned long long *src;
  int64_t rs_row, rs_k, R;
  unsigned long long *out, *flags;
  int flag_rows;
};

// A block takes 32 rows x 128 k of one operand (row groups from `groups_a` on: the
// second's), read along whichever axis is contiguous, with the maxima in
// registers.  Before, a shared-memory atomic per element in a launch per operand:
// maxima and digits together (8 digits) took 235 us at 4096^3, now 195; 32 now
// 14.5 at 512^3, 61 now 42 at 1000 x 3000 x 700.  The digit pass is bound by HBM:
// 0.8 GB at 4096^3.
__global__ void __launch_bounds__(256)
absmax_rows(MaxOperand a, MaxOperand b, int64_t K, unsigned kgroups, unsigned groups_a,
            unsigned long long gen) {
  tc::griddep_launch_dependents();   // the digit pass may launch meanwhile
  __shared__ unsigned long long rmax[8][32];
  unsigned rg = blockIdx.x / kgroups;
  const bool second = rg >= groups_a;
  const MaxOperand &o = second ? b : a;
  if (second) rg -= groups_a;
  const int64_t r0 = (int64_t)rg * 32, k0 = (int64_t)(blockIdx.x % kgroups) * 128;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool kfast = o.rs_k == 1 || o.rs_row != 1;
  // row and k of this thread's value (i, j): 4 rows a warp with the lanes along
  // k, or the lanes along the rows
  unsigned long long v[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int64_t r = r0 + (kfast ? warp * 4 + i : lane);
      const int64_t k = k0 + (kfast ? lane + 32 * j : warp * 16 + 4 * i + j);
      v[i][j] = r < o.R && k < K ? o.src[r * o.rs_row + k * o.rs_k] & 0x7FFFFFFFFFFFFFFFull : 0;
    }
  bool bad = false;
  unsigned long long m[4] = {};
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      if (!finite_bits(v[i][j])) bad = true;
      else m[i] = max(m[i], v[i][j]);
    }
  if (kfast) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const unsigned long long w = warp_max(m[i]);
      if (lane == 0) rmax[0][warp * 4 + i] = w;
    }
  } else {
    rmax[warp][lane] = max(max(m[0], m[1]), max(m[2], m[3]));
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) o.flags[r0 / o.flag_rows] = gen;
  if (warp == 0) {
    unsigned long long w = rmax[0][lane];
    if (!kfast)
#pragma unroll
      for (int i = 1; i < 8; i++) w = max(w, rmax[i][lane]);
    if (r0 + lane < o.R && w) atomicMax(&o.out[r0 + lane], w);
  }
}

// X = round(x 2^(8s - 1 - e)) for |x| < 2^e, |X| <= 2^(8s - 1) (below 2^63 for
// s = 8): the significand shifted in integers, non-finite x as 0 (its tile is
// recomputed).
__device__ __forceinline__ int64_t fixed_point(uint64_t bits, int e, int s) {
  const uint64_t a = bits & 0x7FFFFFFFFFFFFFFFull;
  if (a == 0 || !finite_bits(a)) return 0;
  const int field = (int)(a >> 52);
  uint64_t m = a & 0xFFFFFFFFFFFFFull;
  int ea = field - 1023;
  if (field) m |= 1ull << 52;
  else ea = -1022;                           // subnormal: no implicit bit
  const int sh = ea - 52 - e + 8 * s - 1;    // X = m * 2^sh
  if (sh >= 0) m <<= sh;
  else if (sh < -54) m = 0;
  else m = (m + (1ull << (-sh - 1))) >> -sh;
  return bits >> 63 ? -(int64_t)m : (int64_t)m;
}

// Digits of float64 operands, highest first: with y = X + 0x80 in each of the
// s bytes, byte s - 1 - p of y is digit p + 128, and the top one may be 256
// (X = 2^(8s - 1); for s = 8 the sum wraps there, to a top byte of 0).
__global__ void __launch_bounds__(256)
f64_digits(DigitOperand a, DigitOperand b, int64_t K, int64_t Ks, unsigned kgroups,
           unsigned groups_a, int s) {
  tc::griddep_launch_dependents();   // the GEMM may launch and set up meanwhile
  unsigned rg = blockIdx.x / kgroups;
  const unsigned kg = blockIdx.x % kgroups;
  const bool second = rg >= groups_a;
  const DigitOperand &o = second ? b : a;
  if (second) rg -= groups_a;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t r = (int64_t)rg * 64 + warp * 8 + (lane >> 2);
  const int64_t k0 = (int64_t)kg * 32 + (lane & 3) * 8;
  const int kb = (int)(k0 / kKS), c = (int)(k0 / 8) & 1;
  const bool live = r < o.R && kb < Ks;
  uint64_t y[8];
  if (live) load8((const uint64_t *)o.src + r * o.rs_row, o.rs_k, k0, K, y);
  tc::griddep_wait();   // the maxima are there
  if (!live) return;
  const int e = frexp_exp_bits(o.maxbits[r]) + o.headroom;
  const uint64_t c80 = 0x8080808080808080ull >> (64 - 8 * s);
  uint32_t top[8];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int64_t X = fixed_point(y[i], e, s);
    y[i] = (uint64_t)X + c80;
    const uint32_t t = (uint32_t)(y[i] >> (8 * s - 8));
    top[i] = (X > 0 && t == 0) ? 256u : t;
  }
  const int64_t rb = o.R - r / o.BR * o.BR < o.BR ? o.R - r / o.BR * o.BR : o.BR;
  uint16_t *dst = o.dst + digit_offset(r, kb, 0, c, o.R, o.BR, s, Ks);
  uint32_t h[4];
#pragma unroll
  for (int j = 0; j < 4; j++)
    h[j] = half2_minus_1152((top[2 * j] | top[2 * j + 1] << 16) + 0x64006400u);
  *reinterpret_cast<uint4 *>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
#pragma unroll
  for (int i = 6; i >= 0; i--) {   // byte i of y is digit p = s - 1 - i
    if (i > s - 2) continue;
#pragma unroll
    for (int j = 0; j < 4; j++)
      h[j] = digit_pair((uint32_t)(y[2 * j] >> (i & 4) * 8), (uint32_t)(y[2 * j + 1] >> (i & 4) * 8),
                        i & 3);
    dst += rb * kKS;
    *reinterpret_cast<uint4 *>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
  }
}

// ---- the GEMM ----------------------------------------------------------------

struct DigitGemm {
  const uint16_t *pa, *pb;       // digit planes of A and B^T
  int64_t rso, cso;
  int M, N, Ks;                  // Ks: 16-deep K steps
  int tiles_m, tiles_n, ksplit;  // work units: tiles x K splits
  unsigned *status;
  WaitCfg wc;
  // integers: bias added to every row (numc_linear), or null
  const void *bias;
  int64_t bias_stride;
  // float64: maxima, non-finite flags and the original operands
  const unsigned long long *amax, *bmax, *flags_a, *flags_b;
  unsigned long long gen;
  const double *A, *B;
  int64_t rsa, csa, rsb, csb, K;
  int headroom;
};

// Shared-memory descriptor of a K-major tile of 32-byte rows in the 32-byte
// swizzle (mode 6): 8-row atoms of 256 bytes (stride byte offset); the leading
// byte offset is unused.  Low word: start address and leading offset; the high
// word is the same for every tile.
__device__ __forceinline__ uint32_t sdesc_lo(uint32_t saddr) {
  return ((saddr >> 4) & 0x3FFF) | 1u << 16;
}
constexpr uint32_t kSdescHi = (256u >> 4) | 1u << 14 | 6u << 29;
__device__ __forceinline__ uint64_t sdesc(uint32_t lo) {
  return (uint64_t)kSdescHi << 32 | lo;
}

// The S digit planes of n K steps of a block with `rows` of ROWS rows: one copy
// where the block is full, else a copy per plane (the image holds only its rows),
// each issued by a lane of its own: one lane took 75 cycles a copy, more than the
// plane's MMAs.
template <int S, int ROWS>
__device__ __forceinline__ void load_planes(uint32_t dst, const uint16_t *src, int rows, int n,
                                            uint32_t bar, int lane) {
  if (rows == ROWS) {
    if (lane == 0) tc::bulk_load(dst, src, n * S * ROWS * kRowBytes, bar);
  } else if (lane < n * S) {
    tc::bulk_load(dst + lane * ROWS * kRowBytes, src + (int64_t)lane * rows * kKS, rows * kRowBytes,
              bar);
  }
}

__device__ __forceinline__ bool wait_all(uint64_t *bar, uint32_t parity, const DigitGemm &P,
                                         unsigned code = kStatusTimeoutMma) {
  return tc::mbar_wait_warp(tc::smem_u32(bar), parity, P.status, code, P.wc.limit_ns);
}

// (hi, frac) += t, a signed 64-bit number in units of the fraction.
__device__ __forceinline__ void add_frac(unsigned long long &hi, uint32_t &frac,
                                         unsigned long long t) {
  uint32_t h0 = (uint32_t)hi, h1 = (uint32_t)(hi >> 32);
  const uint32_t t0 = (uint32_t)t, t1 = (uint32_t)(t >> 32), sign = (uint32_t)((int)t1 >> 31);
  asm("add.cc.u32 %0, %0, %3;\n addc.cc.u32 %1, %1, %4;\n addc.u32 %2, %2, %5;"
      : "+r"(frac), "+r"(h0), "+r"(h1)
      : "r"(t0), "r"(t1), "r"(sign));
  hi = (unsigned long long)h1 << 32 | h0;
}

// (hi + frac 2^-32) 2^e as a double, rounded once (twice only where the result
// is subnormal).
__device__ __forceinline__ double wide_to_double(long long hi, uint32_t frac, int e) {
  // as many bits of the fraction as fit below hi in 63 bits, the rest as a
  // sticky bit (below the rounding position: hi has 30 bits or more then)
  const unsigned long long mag = hi < 0 ? ~(unsigned long long)hi : (unsigned long long)hi;
  const int room = min(32, __clzll((long long)mag) - 1);
  const uint32_t kept = room == 0 ? 0 : frac >> (32 - room);
  const bool sticky = room < 32 && (frac << room) != 0;
  return ldexp(__ll2double_rn((hi << room) | (long long)kept | (long long)sticky), e - room);
}

// S digits; TMEM holds NS >= S diagonals of BN columns.  T: output type.
template <int S, int BN, typename T>
struct DigitCfg {
  static constexpr bool F64 = std::is_same<T, double>::value;
  static constexpr int NS = S > 4 ? 8 : S > 2 ? 4 : 2;
  // K steps of a pipeline stage: fewer digits make a step cheaper, and a stage
  // has to outlast the issuing warps' wait and commit
  static constexpr int KST = S > 4 ? 1 : S > 2 ? 2 : 4;
  // the longest exact accumulation chain, 1024 / S of K, in K steps
  static constexpr int CHUNK = 1024 / S / kKS / KST * KST;
  // a stage: KST K steps of A's digit planes, then of B's
  static constexpr int A_STEP = S * kBM * kRowBytes, B_STEP = S * BN * kRowBytes;
  static constexpr int A_BYTES = KST * A_STEP, B_BYTES = KST * B_STEP;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = kRingBytes / STAGE_BYTES < 8 ? kRingBytes / STAGE_BYTES : 8;
  static constexpr int NBUF = 512 / (NS * BN);          // TMEM buffers of NS diagonals
  // Diagonals [0, LOW) form the low release group, [LOW, S) the high one.  With
  // one buffer: near equal products in both, so that each group's read-back
  // hides under the other's MMAs.  With two or more, one group: a whole chunk
  // is read back under the next one's MMAs.
  static constexpr int LOW = NBUF > 1 ? S : S == 8 ? 5 : S == 7 ? 4 : S == 4 ? 2 : 3;
  static constexpr int CW = BN / 4;                     // columns of an epilogue thread
  static constexpr int SMEM = 1024 + STAGES * STAGE_BYTES + kEpiWarps * 2048 + 512;
  static_assert(SMEM <= 232448, "shared memory");
};

// Rows of 64 bytes of a warp's 32 x (64 / sizeof(T)) block through shared
// memory, so that a store instruction covers whole row segments.
template <typename T, int CW>
__device__ __forceinline__ void store_block(const T (&v)[CW], uint8_t *stage, T *C, int64_t rso,
                                            int64_t cso, int row0, int col0, int M, int N,
                                            int lane, bool vec, bool add) {
  constexpr int E = 64 / sizeof(T) < CW ? 64 / sizeof(T) : CW;   // columns per pass
  constexpr int V = 16 / sizeof(T);                               // elements per 16 bytes
  constexpr int NC = E / V;                                       // 16-byte chunks per row
#pragma unroll
  for (int c0 = 0; c0 < CW; c0 += E) {
#pragma unroll
    for (int q = 0; q < NC; q++) {
      T tmp[V];
#pragma unroll
      for (int j = 0; j < V; j++) tmp[j] = v[c0 + q * V + j];
      *reinterpret_cast<uint4 *>(stage + lane * 64 + ((q ^ (lane >> 1)) & 3) * 16) =
          *reinterpret_cast<const uint4 *>(tmp);
    }
    __syncwarp();
    if (vec) {
#pragma unroll
      for (int it = 0; it < NC; it++) {
        const int r = it * (32 / NC) + lane / NC, q = lane % NC;
        const uint4 w = *reinterpret_cast<const uint4 *>(stage + r * 64 + ((q ^ (r >> 1)) & 3) * 16);
        if (row0 + r < M && col0 + c0 + (q + 1) * V <= N)
          *reinterpret_cast<uint4 *>(C + (int64_t)(row0 + r) * rso + col0 + c0 + q * V) = w;
        else if (row0 + r < M) {
          T tmp[V];
          *reinterpret_cast<uint4 *>(tmp) = w;
#pragma unroll
          for (int j = 0; j < V; j++)
            if (col0 + c0 + q * V + j < N)
              C[(int64_t)(row0 + r) * rso + col0 + c0 + q * V + j] = tmp[j];
        }
      }
    } else {
#pragma unroll 4
      for (int i = lane; i < 32 * E; i += 32) {
        const int r = i / E, c = i % E, q = c / V;
        const T x = *reinterpret_cast<const T *>(stage + r * 64 + ((q ^ (r >> 1)) & 3) * 16 +
                                                 (c % V) * sizeof(T));
        if (row0 + r < M && col0 + c0 + c < N) {
          T *dst = C + (int64_t)(row0 + r) * rso + (int64_t)(col0 + c0 + c) * cso;
          if constexpr (std::is_same<T, unsigned>::value ||
                        std::is_same<T, unsigned long long>::value) {
            if (add) {
              atomicAdd(dst, x);
              continue;
            }
          }
          *dst = x;
        }
      }
    }
    __syncwarp();
  }
}

// Work unit u: origin of its output tile and its range of K steps.
template <int BN>
__device__ __forceinline__ void unit(const DigitGemm &P, int u, int &m0, int &n0, int &k0,
                                     int &k1) {
  constexpr int GM = 16;   // 2048 rows of tiles: their B columns stay in L2
  const int ks = u % P.ksplit, t = u / P.ksplit;
  const int group = t / (GM * P.tiles_n);
  const int first_m = group * GM;
  const int gm = min(P.tiles_m - first_m, GM);
  const int local = t - group * GM * P.tiles_n;
  m0 = (first_m + local % gm) * kBM;
  n0 = (local / gm) * BN;
  k0 = (int)((int64_t)P.Ks * ks / P.ksplit);
  k1 = (int)((int64_t)P.Ks * (ks + 1) / P.ksplit);
}

// End of the chunk of GROUP that begins at K step kc.  The high group's chunks
// are offset by half a chunk (its first is short), so that the two groups are
// read back at different times, each under the other's MMAs: with common
// chunk ends both stood still for the whole read-back (3054 against 2993 us at
// 4096^3, S = 8).
template <typename Cfg, int GROUP>
__device__ __forceinline__ int chunk_end(int kc, int k0, int k1) {
  constexpr int FIRST = (Cfg::CHUNK / Cfg::KST + 1) / 2 * Cfg::KST;
  return min(k1, GROUP == 1 && kc == k0 ? kc + FIRST : kc + Cfg::CHUNK);
}

// Issue every MMA of the low (0) or high (1) group of diagonals, [0, h0) or
// [h0, S).  One MMA covers A_p times B's digits q..: its columns are the
// diagonals p + q, p + q + 1, ... of the group.
template <int S, int BN, typename T, int GROUP>
__device__ __forceinline__ void issue_group(const DigitGemm &P, uint8_t *smem, uint32_t tmem,
                                            uint64_t *full, uint64_t *empty, uint64_t *tfull,
                                            uint64_t *tempty) {
  using Cfg = DigitCfg<S, BN, T>;
  constexpr int NS = Cfg::NS, ST = Cfg::STAGES, NBUF = Cfg::NBUF;
  constexpr uint32_t A_PLANE = kBM * kRowBytes / 16, B_PLANE = BN * kRowBytes / 16;
  const bool lead = tc::elect_one();
  const int units = P.tiles_m * P.tiles_n * P.ksplit;
  int g = 0, chunk = 0;   // stages and chunks across units
  for (int u = blockIdx.x; u < units; u += gridDim.x) {
    int m0, n0, k0, k1;
    unit<BN>(P, u, m0, n0, k0, k1);
    for (int kc = k0, ke; kc < k1; kc = ke, chunk++) {
      ke = chunk_end<Cfg, GROUP>(kc, k0, k1);
      const int buf = chunk % NBUF;
      const uint32_t d0 = tmem + buf * NS * BN;
      if (chunk >= NBUF && !wait_all(&tempty[2 * buf + GROUP], ((chunk / NBUF) & 1) ^ 1, P)) return;
      for (int ks = kc; ks < ke; ks += Cfg::KST, g++) {
        const int st = g % ST;
        if (!wait_all(&full[st], (g / ST) & 1, P)) return;
        tc::tc_fence_after();
        uint32_t sa = sdesc_lo(tc::smem_u32(smem + st * Cfg::STAGE_BYTES));
        uint32_t sb = sa + Cfg::A_BYTES / 16;
        constexpr int D0 = GROUP == 0 ? 0 : Cfg::LOW, D1 = GROUP == 0 ? Cfg::LOW : S;
        constexpr int W = 256 / BN;   // diagonals of one MMA
#pragma unroll
        for (int i = 0; i < Cfg::KST; i++, sa += Cfg::A_STEP / 16, sb += Cfg::B_STEP / 16) {
          if (ks + i >= ke) break;
#pragma unroll
          for (int p = 0; p < D1; p++) {
            // diagonals max(D0, p) .. D1 - 1: digits d - p of B
#pragma unroll
            for (int d = p > D0 ? p : D0; d < D1; d += W) {
              const int n = D1 - d < W ? D1 - d : W;
              tc::mma_f16_lead(d0 + d * BN, sdesc(sa + p * A_PLANE), sdesc(sb + (d - p) * B_PLANE),
                      tc::idesc_f16_f32(kBM, n * BN), p > 0 ? 1u : ks + i > kc, lead);
            }
          }
        }
        tc::mma_commit_lead(tc::smem_u32(&empty[st]), lead);
      }
      tc::mma_commit_lead(tc::smem_u32(&tfull[2 * buf + GROUP]), lead);
    }
  }
}

template <int S, int BN, typename T>
__global__ void __launch_bounds__(kThreads, 1)
digit_gemm(const DigitGemm P, T *__restrict__ C) {
  using Cfg = DigitCfg<S, BN, T>;
  constexpr int NS = Cfg::NS, CHUNK = Cfg::CHUNK;
  constexpr int ST = Cfg::STAGES, NBUF = Cfg::NBUF, LOW = Cfg::LOW, CW = Cfg::CW;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t *epi = smem + ST * Cfg::STAGE_BYTES;
  uint64_t *bars = (uint64_t *)(epi + kEpiWarps * 2048);
  uint64_t *full = bars, *empty = full + ST;
  uint64_t *tfull = empty + ST, *tempty = tfull + 2 * NBUF;   // [buffer][half]
  uint64_t *drain = tempty + 2 * NBUF;
  uint32_t *tmem_slot = (uint32_t *)(drain + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int units = P.tiles_m * P.tiles_n * P.ksplit;
  if (threadIdx.x == 0) {
    for (int i = 0; i < ST; i++) {
      tc::mbar_init(tc::smem_u32(&full[i]), 1);
      tc::mbar_init(tc::smem_u32(&empty[i]), S > LOW ? 2 : 1);   // issuing warps
    }
    for (int b = 0; b < 2 * NBUF; b++) {
      tc::mbar_init(tc::smem_u32(&tfull[b]), 1);
      tc::mbar_init(tc::smem_u32(&tempty[b]), kEpiWarps);
    }
    tc::mbar_init(tc::smem_u32(drain), S > LOW ? 2 : 1);
    tc::fence_barrier_init();
  }
  if (warp == 1) tc::tmem_alloc(tc::smem_u32(tmem_slot), 512);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  tc::griddep_wait();   // the digit pass has completed

  if (warp == 0) {
    int g = 0;   // stage counter across units
    bool live = true;
    for (int u = blockIdx.x; u < units && live; u += gridDim.x) {
      int m0, n0, k0, k1;
      unit<BN>(P, u, m0, n0, k0, k1);
      const int ra = min(kBM, P.M - m0), rb = min(BN, P.N - n0);
      const uint16_t *srca = P.pa + (int64_t)m0 * S * P.Ks * kKS;
      const uint16_t *srcb = P.pb + (int64_t)n0 * S * P.Ks * kKS;
      for (int kb = k0; kb < k1; kb += Cfg::KST, g++) {
        const int st = g % ST;
        if (g >= ST) {
          live = wait_all(&empty[st], ((g / ST) & 1) ^ 1, P, kStatusTimeoutProducer);
          if (!live) break;
        }
        if (P.wc.starve) continue;   // give-up test: no load, no barrier completes
        const int n = min(Cfg::KST, k1 - kb);
        const uint32_t fbar = tc::smem_u32(&full[st]);
        const uint32_t sa = tc::smem_u32(smem + st * Cfg::STAGE_BYTES);
        if (lane == 0) tc::mbar_arrive_expect_tx(fbar, (uint32_t)(n * S * (ra + rb) * kRowBytes));
        __syncwarp();
        load_planes<S, kBM>(sa, srca + (int64_t)kb * S * ra * kKS, ra, n, fbar, lane);
        load_planes<S, BN>(sa + Cfg::A_BYTES, srcb + (int64_t)kb * S * rb * kKS, rb, n, fbar,
                           lane ^ 16);
      }
    }
    __syncwarp();
  } else if (warp == 1 || warp == kMmaHigh) {
    // Two issuing warps: one multiplies the low group of diagonals, one the
    // high group, each in its own TMEM columns.  While one waits for its group
    // to be read back the other runs ahead, up to the depth of the ring, and
    // the per-step waits of the two overlap (float64 4096^3, S = 8: 3.23 ms with
    // one warp issuing both groups, 3.10 with two; S = 5: 2.04 and 1.86).
    // A whole warp runs the loop, so that descriptors and addresses stay in
    // uniform registers, and one elected lane issues (3.79 against 3.60 ms with the loop under
    // one lane: the moves into uniform registers bounded the issue rate).
    if (warp == 1) issue_group<S, BN, T, 0>(P, smem, tmem, full, empty, tfull, tempty);
    else if (S > LOW) issue_group<S, BN, T, 1>(P, smem, tmem, full, empty, tfull, tempty);
    // Every MMA issued above completes before TMEM is released, also when
    // the loop gave up (a commit with none outstanding arrives at once).
    if (warp == 1 || S > LOW) {
      tc::mma_commit_lead(tc::smem_u32(drain), tc::elect_one());
      wait_all(drain, 0, P, kStatusTimeoutDrain);
    }
  } else {
    const int quad = warp & 3, quarter = (warp - 2) >> 2;
    const int cbase = quarter * CW;
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    uint8_t *stage = epi + (warp - 2) * 2048;
    // Weight of diagonal d (without a fraction).
    auto weight = [](int d) { return 1ull << (8 * (Cfg::F64 ? 3 - (d & 3) : d)); };
    int chunk0 = 0, chunk1 = 0;   // chunks of the two groups, across units
    bool ok = true;
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
      int m0, n0, k0, k1;
      unit<BN>(P, u, m0, n0, k0, k1);
      // Integers: the sum modulo 2^bits.  float64: sum_d D_d 256^(3-d) as a
      // 64-bit integer, with a 32-bit fraction below it for the diagonals past 3
      // (|sum| <= K 2^14 (2^24 + 2 2^16 + ...) < 2^63 for K <= 2^24).
      using Acc = typename std::conditional<sizeof(T) == 8, unsigned long long, unsigned>::type;
      constexpr bool FRAC = Cfg::F64 && S > 4;
      Acc acc[CW];
      [[maybe_unused]] uint32_t frac[FRAC ? CW : 1];
#pragma unroll
      for (int j = 0; j < CW; j++) acc[j] = 0;
      if constexpr (FRAC) {
#pragma unroll
        for (int j = 0; j < CW; j++) frac[j] = 0;
      }
      // Read one group's diagonals back at the end of its chunk and fold them in.
      auto drain_group = [&](auto group, int chunk) {
        constexpr int GROUP = decltype(group)::value;
        const int buf = chunk % NBUF;
        bool done = tc::mbar_wait_bounded(tc::smem_u32(&tfull[2 * buf + GROUP]),
                                          (chunk / NBUF) & 1, P.status, kStatusTimeoutEpilogue,
                                          P.wc.limit_ns);
        if (!__all_sync(0xffffffffu, done)) return false;   // tcgen05.ld is warp-collective
        tc::tc_fence_after();
        // 8 columns of one diagonal at a time, the highest diagonal first, the
        // next ones' load in flight while one is folded in
        constexpr int D0 = GROUP == 0 ? 0 : LOW, D1 = GROUP == 0 ? LOW : S;
        constexpr int ND = D1 > D0 ? D1 - D0 : 1;   // (an empty group is never read)
        constexpr int NB = ND * (CW / 8);
        auto column = [&](int i) {
          return tmem + lane_off + (buf * NS + D1 - 1 - i % ND) * BN + cbase + i / ND * 8;
        };
        uint32_t r[2][8];
        [[maybe_unused]] unsigned long long t[8];
        tc::tmem_ld_32x32b_x8(column(0), r[0]);
#pragma unroll
        for (int i = 0; i < NB; i++) {
          const int d = D1 - 1 - i % ND, c0 = i / ND * 8;
          uint32_t(&v)[8] = r[i & 1];
          tc::tmem_ld_wait();
          if (i + 1 < NB) tc::tmem_ld_32x32b_x8(column(i + 1), r[(i + 1) & 1]);
          // Each sum f is an integer, |f| <= 2^24: adding 1.5 x 2^23 leaves
          // f + kMagicBits in the bits where |f| <= 2^22, at the FP32 rate
          // (conversions run at an eighth of it and held up the next
          // chunk: 3.17 against 3.10 ms at 4096^3, S = 8).  Larger sums
          // (digits nearly all alike) are read again and converted.
          uint32_t over = 0;
#pragma unroll
          for (int j = 0; j < 8; j++) {
            v[j] = __float_as_uint(__uint_as_float(v[j]) + 12582912.0f);
            over |= v[j] ^ 0x4B000000u;
          }
          if ((d + 1) * CHUNK * kKS > 256 && __any_sync(0xffffffffu, over >> 23)) {
            tc::tmem_ld_32x32b_x8(column(i), v);
            tc::tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 8; j++)
              v[j] = kMagicBits + (uint32_t)__float2int_rn(__uint_as_float(v[j]));
          }
          if (i == NB - 1) {   // the group is read back
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(tc::smem_u32(&tempty[2 * buf + GROUP]));
          }
          if constexpr (FRAC) {
            // a group's diagonals of the fraction (4..) or above it (0..3) in
            // one 64-bit sum, the conversions' bias taken out at its start
            const bool low = d >= 4;
            const bool first = i % ND == 0 || d == 3;
            const unsigned long long w = 1ull << (8 * ((low ? 7 : 3) - d));
            unsigned long long bias = 0;
            for (int q = D0; q < D1; q++)
              if ((q >= 4) == low) bias += (unsigned long long)kMagicBits << (8 * ((low ? 7 : 3) - q));
#pragma unroll
            for (int j = 0; j < 8; j++) t[j] = v[j] * w + (first ? 0 - bias : t[j]);
            if (d == D0 || d == 4) {
#pragma unroll
              for (int j = 0; j < 8; j++) {
                if (low) add_frac(acc[c0 + j], frac[c0 + j], t[j]);
                else acc[c0 + j] += t[j];
              }
            }
          } else {
#pragma unroll
            for (int j = 0; j < 8; j++) {
              if constexpr (sizeof(T) == 8) {
                if (Cfg::F64 || d < 4) acc[c0 + j] += v[j] * weight(d);
                else acc[c0 + j] += (unsigned long long)(v[j] << (8 * (d & 3))) << 32;
              } else {
                acc[c0 + j] += v[j] << (8 * d);
              }
            }
          }
        }
        return true;
      };
      // in the order in which the groups reach their chunk ends
      unsigned chunks0 = 0, chunks1 = 0;
      for (int p0 = k0, p1 = S > LOW ? k0 : k1; ok && (p0 < k1 || p1 < k1);) {
        const int e0 = chunk_end<Cfg, 0>(p0, k0, k1), e1 = chunk_end<Cfg, 1>(p1, k0, k1);
        if (p1 >= k1 || (p0 < k1 && e0 <= e1)) {
          ok = drain_group(std::integral_constant<int, 0>(), chunk0 + chunks0);
          chunks0++;
          p0 = e0;
        } else {
          ok = drain_group(std::integral_constant<int, 1>(), chunk1 + chunks1);
          chunks1++;
          p1 = e1;
        }
      }
      if (!ok) break;
      chunk0 += chunks0;
      chunk1 += chunks1;
      if constexpr (!FRAC) {   // take the bias of the conversions out
        unsigned long long w = 0;
#pragma unroll
        for (int d = 0; d < S; d++) w += weight(d) * (d < LOW ? chunks0 : chunks1);
#pragma unroll
        for (int j = 0; j < CW; j++) acc[j] -= (Acc)(w * kMagicBits);
      }
      const int row0 = m0 + quad * 32, col0 = n0 + cbase;
      if constexpr (Cfg::F64) {
        const int row = row0 + lane;
        bool nonfinite = P.flags_a[m0 / kBM] == P.gen;
#pragma unroll 1
        for (int c = n0 / 64; c < (n0 + BN) / 64 && c * 64 < P.N; c++)
          nonfinite |= P.flags_b[c] == P.gen;
        double out[CW];
        if (nonfinite) {
          // numc's arithmetic: one FMA chain per output in k order.
#pragma unroll 1
          for (int j = 0; j < CW; j++) {
            double f = 0.0;
            if (row < P.M && col0 + j < P.N)
#pragma unroll 1
              for (int64_t k = 0; k < P.K; k++)
                f = __fma_rn(P.A[(int64_t)row * P.rsa + k * P.csa],
                             P.B[k * P.rsb + (int64_t)(col0 + j) * P.csb], f);
            if (row < P.M && col0 + j < P.N)
              C[(int64_t)row * P.rso + (int64_t)(col0 + j) * P.cso] = f;
          }
        } else {
          const int base = (row < P.M ? frexp_exp_bits(P.amax[row]) : 0) + P.headroom - 38;
#pragma unroll
          for (int j = 0; j < CW; j++) {
            const int e = base + (col0 + j < P.N ? frexp_exp_bits(P.bmax[col0 + j]) : 0);
            if constexpr (FRAC) out[j] = wide_to_double((long long)acc[j], frac[j], e);
            else out[j] = ldexp(__ll2double_rn((long long)acc[j]), e);
          }
          const bool vec = P.cso == 1 && P.rso % 2 == 0 && ((uintptr_t)C & 15) == 0;
          store_block<T, CW>(out, stage, C, P.rso, P.cso, row0, col0, P.M, P.N, lane, vec, false);
        }
      } else {
        T out[CW];
#pragma unroll
        for (int j = 0; j < CW; j++) out[j] = (T)acc[j];
        if (P.bias && k0 == 0) {
#pragma unroll
          for (int j = 0; j < CW; j++)
            if (col0 + j < P.N) out[j] = (T)(out[j] + ((const T *)P.bias)[(col0 + j) * P.bias_stride]);
        }
        const bool add = P.ksplit > 1;
        const bool vec = !add && P.cso == 1 && P.rso % (16 / (int)sizeof(T)) == 0 &&
                         ((uintptr_t)C & 15) == 0;
        store_block<T, CW>(out, stage, C, P.rso, P.cso, row0, col0, P.M, P.N, lane, vec, add);
      }
      __syncwarp();   // reconverge before the next unit's tcgen05.ld
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, 512);
  }
}

// ---- launch ------------------------------------------------------------------

template <int S, int BN, typename T>
cudaError_t launch_digit_gemm(DigitGemm P, T *C, cudaStream_t s) {
  using Cfg = DigitCfg<S, BN, T>;
  auto kern = digit_gemm<S, BN, T>;
  static LaunchCache lc;
  cudaError_t e;
  if ((e = smem_attr_once(lc, (const void *)kern, Cfg::SMEM))) return e;
  P.tiles_m = (P.M + kBM - 1) / kBM;
  P.tiles_n = (P.N + BN - 1) / BN;
  P.wc = wait_cfg();
  const int64_t units = (int64_t)P.tiles_m * P.tiles_n * P.ksplit;
  if (units >= 1ll << 31) return cudaErrorInvalidConfiguration;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  cfg.gridDim = dim3((unsigned)std::min<int64_t>(units, sm_count()));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = Cfg::SMEM;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if ((e = cudaLaunchKernelEx(&cfg, kern, P, C))) return e;
  count_launch();
  return cudaGetLastError();
}

struct OzLayout {
  int64_t Kp;
  size_t amax, bmax, flags_a, flags_b, a, b, total;
};

OzLayout oz_layout(int64_t M, int64_t K, int64_t N, int s) {
  OzLayout L;
  L.Kp = round_up(K > 0 ? K : 1, 64);
  L.amax = 0;
  L.bmax = (size_t)round_up(M * 8, 256);
  L.flags_a = L.bmax + (size_t)round_up(N * 8, 256);
  L.flags_b = L.flags_a + (size_t)round_up(((M + kBM - 1) / kBM) * 8, 256);
  L.a = L.flags_b + (size_t)round_up(((N + 63) / 64) * 8, 256);
  L.b = L.a + (size_t)round_up((int64_t)s * M * L.Kp * 2, 256);
  L.total = L.b + (size_t)round_up((int64_t)s * N * L.Kp * 2, 256);
  return L;
}

std::atomic<unsigned long long> g_oz_gen{0x0a2a000000000000ull};

// Blocks of the digit pass, 64 rows x 32 k each (0: more than a grid holds).
struct DigitGrid {
  unsigned kgroups, groups_a, blocks;
};
DigitGrid digit_grid(int64_t M, int64_t K, int64_t N) {
  const int64_t kg = (K + 31) / 32, ga = (M + 63) / 64, gb = (N + 63) / 64;
  const int64_t n = kg * (ga + gb);
  return DigitGrid{(unsigned)kg, (unsigned)ga, n < (1ll << 31) ? (unsigned)n : 0u};
}

}  // namespace

size_t ozaki_workspace(int64_t M, int64_t K, int64_t N, int slices) {
  return oz_layout(M, K, N, slices).total;
}

cudaError_t launch_ozaki(const Gemm &g, int slices, void *ws_v, size_t ws_bytes, cudaStream_t s) {
  if (g.M == 0 || g.N == 0) return cudaSuccess;
  if (g.K == 0) return launch_simt(NUMC_DTYPE_FLOAT64, g, 0, s);   // C = 0
  if (slices < 1 || slices > 8) return cudaErrorInvalidValue;
  if (g.M >= (1ll << 31) || g.N >= (1ll << 31) || g.K >= (1ll << 31))
    return cudaErrorInvalidValue;
  const OzLayout L = oz_layout(g.M, g.K, g.N, slices);
  if (ws_bytes < L.total || ((uintptr_t)ws_v & 255)) return cudaErrorInvalidValue;
  char *ws = (char *)ws_v;
  unsigned *status = status_word();
  if (!status) return cudaErrorMemoryAllocation;
  PhaseMark mark(s);
  const unsigned long long gen = ++g_oz_gen;
  auto *amax = (unsigned long long *)(ws + L.amax), *bmax = (unsigned long long *)(ws + L.bmax);
  auto *fa = (unsigned long long *)(ws + L.flags_a), *fb = (unsigned long long *)(ws + L.flags_b);
  cudaError_t e = cudaMemsetAsync(ws, 0, L.flags_a, s);   // maxima start at +0
  if (e) return e;
  const int64_t kg = (g.K + 127) / 128, ga = (g.M + 31) / 32, gb = (g.N + 31) / 32;
  const DigitGrid dg = digit_grid(g.M, g.K, g.N);
  if (ga > 65535 || gb > 65535 || kg * (ga + gb) >= 1ll << 31 || !dg.blocks)
    return cudaErrorInvalidConfiguration;
  absmax_rows<<<(unsigned)(kg * (ga + gb)), 256, 0, s>>>(
      MaxOperand{(const unsigned long long *)g.a, g.rsa, g.csa, g.M, amax, fa, kBM},
      MaxOperand{(const unsigned long long *)g.b, g.csb, g.rsb, g.N, bmax, fb, 64}, g.K, (unsigned)kg,
      (unsigned)ga, gen);
  // The leading diagonals' sum stays below K 2^38.1: past K = 2^24 A's digits
  // leave one more bit of headroom per doubling.
  int headroom = 0;
  while (g.K > (1ll << (24 + headroom))) headroom++;
  // 8 diagonals of 64 columns fill TMEM, or 4 of 128
  const int BN = slices > 4 ? 64 : 128;
  DigitGemm P = {};
  P.pa = (const uint16_t *)(ws + L.a);
  P.pb = (const uint16_t *)(ws + L.b);
  P.Ks = (int)((g.K + kKS - 1) / kKS);
  const DigitOperand oa{g.a, g.rsa, g.csa, g.M, (uint16_t *)(ws + L.a), kBM, amax, headroom};
  const DigitOperand ob{g.b, g.csb, g.rsb, g.N, (uint16_t *)(ws + L.b), BN, bmax, 0};
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr;   // launched while the maxima pass ends
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  cfg.gridDim = dim3(dg.blocks);
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if ((e = cudaLaunchKernelEx(&cfg, f64_digits, oa, ob, g.K, (int64_t)P.Ks, dg.kgroups, dg.groups_a,
                              slices)))
    return e;
  count_launch(2);
  mark.split_done();
  P.rso = g.rso; P.cso = g.cso;
  P.M = (int)g.M; P.N = (int)g.N;
  P.ksplit = 1;
  P.status = status;
  P.amax = amax; P.bmax = bmax; P.flags_a = fa; P.flags_b = fb; P.gen = gen;
  P.A = (const double *)g.a; P.B = (const double *)g.b;
  P.rsa = g.rsa; P.csa = g.csa; P.rsb = g.rsb; P.csb = g.csb; P.K = g.K;
  P.headroom = headroom;
  double *C = (double *)g.c;
  switch (slices) {
  case 1: e = launch_digit_gemm<1, 128, double>(P, C, s); break;
  case 2: e = launch_digit_gemm<2, 128, double>(P, C, s); break;
  case 3: e = launch_digit_gemm<3, 128, double>(P, C, s); break;
  case 4: e = launch_digit_gemm<4, 128, double>(P, C, s); break;
  case 5: e = launch_digit_gemm<5, 64, double>(P, C, s); break;
  case 6: e = launch_digit_gemm<6, 64, double>(P, C, s); break;
  case 7: e = launch_digit_gemm<7, 64, double>(P, C, s); break;
  default: e = launch_digit_gemm<8, 64, double>(P, C, s); break;
  }
  mark.gemm_done();
  return e;
}

// ---- 16-, 32- and 64-bit integers -------------------------------------------

namespace {

// How an integer problem runs: columns per tile and K splits (0 columns: not
// here), and the estimated times in us here and on the CUDA cores.
struct IntPlan {
  int BN = 0, ksplit = 1;
  double us = 0, simt_us = 0;
  int64_t Ks = 0;
  size_t b = 0, total = 0;
};

IntPlan int_plan(int bytes, int64_t M, int64_t K, int64_t N) {
  IntPlan p;
  if (M <= 0 || N <= 0 || K <= 0 || M >= (1ll << 30) || N >= (1ll << 30) || K >= (1ll << 30))
    return p;
  if (!digit_grid(M, K, N).blocks) return p;
  p.Ks = (K + kKS - 1) / kKS;
  const int s = bytes, sms = sm_count() > 0 ? sm_count() : 152;
  double best = 1e30;
  for (int BN = 64; BN <= 128; BN += 64) {
    if (bytes == 8 && BN == 128) continue;    // 8 diagonals of 128 columns exceed TMEM
    const int64_t tiles = ((M + kBM - 1) / kBM) * ((N + BN - 1) / BN);
    // Measured cycles of a K step (4096^3), of a unit's start and end, and of
    // adding a tile into C.
    const double step = bytes == 8 ? 1200 : bytes == 4 ? (BN == 64 ? 424 : 788)
                                                       : (BN == 64 ? 187 : 275);
    for (int ks = 1; ks <= 32 && ks <= std::max<int64_t>(1, p.Ks / 4); ks++) {
      if (ks > 1 && bytes == 2) break;        // no 16-bit atomics
      const int64_t rounds = (tiles * ks + sms - 1) / sms;
      const double t =
          rounds * ((p.Ks + ks - 1) / ks * step + 3000 + (ks > 1 ? 0.7 * kBM * BN : 0));
      if (t < best) {
        best = t;
        p.BN = BN;
        p.ksplit = ks;
      }
    }
  }
  // The line to the CUDA cores, from both sides' times (digits / CUDA cores, us,
  // back to back in a graph, GB300):
  //            64^3      256^3      512^3      1024^3    2048x128x256  64x5000x64
  //   int16  6.6/3.2   8.1/7.0    9.4/19.6   14/92       7.3/11.6      52/96
  //   int32  8.1/3.2  10.5/7.0   11.1/19.3   23/96       9.1/11.6      11/95
  //   int64 12.5/5.0  13.6/13.8  16.8/45.8   60/335     15.5/25.0      19/225
  // Here: two launches and the passes' bytes besides the units' cycles; there
  // the longer of the K loop of one thread and of all multiply-adds (a low
  // estimate: near the line the CUDA cores keep the problem).
  const double elems = (double)(M + N) * K, out = (double)M * N;
  p.us = 5.5 + best / 1900 + elems * 3 * bytes / 4e6 + out * bytes * (p.ksplit > 1 ? 2 : 1) / 3e6;
  p.simt_us = 2.5 + std::max(K * (bytes == 8 ? 0.042 : 0.0185),
                             2 * out * K / (bytes == 8 ? 6.4e6 : 18e6));
  p.b = (size_t)round_up((int64_t)s * M * p.Ks * kKS * 2, 256);
  p.total = p.b + (size_t)round_up((int64_t)s * N * p.Ks * kKS * 2, 256);
  return p;
}

int int_bytes(NumcDType dt) {
  switch (dt) {
  case NUMC_DTYPE_INT16: case NUMC_DTYPE_UINT16: return 2;
  case NUMC_DTYPE_INT32: case NUMC_DTYPE_UINT32: return 4;
  case NUMC_DTYPE_INT64: case NUMC_DTYPE_UINT64: return 8;
  default: return 0;
  }
}

template <typename T>
cudaError_t run_int(const Gemm &g, const IntPlan &ip, char *ws, unsigned *status,
                    cudaStream_t s) {
  constexpr int S = sizeof(T);
  const DigitGrid dg = digit_grid(g.M, g.K, g.N);
  const DigitOperand oa{g.a, g.rsa, g.csa, g.M, (uint16_t *)ws, kBM};
  const DigitOperand ob{g.b, g.csb, g.rsb, g.N, (uint16_t *)(ws + ip.b), ip.BN};
  PhaseMark mark(s);
  int_digits<T, S><<<dg.blocks, 256, 0, s>>>(oa, ob, g.K, ip.Ks, dg.kgroups, dg.groups_a,
                                             ip.ksplit > 1 ? (T *)g.c : nullptr, g.rso, g.cso,
                                             g.M, g.N);
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e) return e;
  mark.split_done();
  DigitGemm P = {};
  P.pa = oa.dst;
  P.pb = ob.dst;
  P.rso = g.rso; P.cso = g.cso;
  P.M = (int)g.M; P.N = (int)g.N; P.Ks = (int)ip.Ks;
  P.ksplit = ip.ksplit;
  P.status = status;
  P.bias = g.bias;
  P.bias_stride = g.bias_stride;
  if constexpr (S == 8) e = launch_digit_gemm<8, 64, T>(P, (T *)g.c, s);
  else e = ip.BN == 64 ? launch_digit_gemm<S, 64, T>(P, (T *)g.c, s)
                       : launch_digit_gemm<S, 128, T>(P, (T *)g.c, s);
  mark.gemm_done();
  return e;
}

}  // namespace

size_t int_digits_workspace(NumcDType dt, int64_t M, int64_t K, int64_t N) {
  const int bytes = int_bytes(dt);
  if (!bytes) return 0;
  const IntPlan p = int_plan(bytes, M, K, N);
  return p.BN && p.us < p.simt_us ? p.total : 0;
}

cudaError_t launch_int_digits(NumcDType dt, const Gemm &g, void *ws, size_t ws_bytes,
                              unsigned *status, cudaStream_t s) {
  const int bytes = int_bytes(dt);
  const IntPlan p = int_plan(bytes, g.M, g.K, g.N);
  if (!bytes || !p.BN || ws_bytes < p.total || ((uintptr_t)ws & 255)) return cudaErrorInvalidValue;
  if (!status) return cudaErrorMemoryAllocation;
  if (bytes == 8) return run_int<unsigned long long>(g, p, (char *)ws, status, s);
  if (bytes == 4) return run_int<unsigned>(g, p, (char *)ws, status, s);
  return run_int<unsigned short>(g, p, (char *)ws, status, s);
}

}  // namespace numc_k

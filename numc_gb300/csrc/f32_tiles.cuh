#pragma once

// One output tile of a float32 GEMM on the CUDA cores, for one problem
// (gemm_f32.cu) and for many (gemm_grouped.cu): a block computes it in numc's
// arithmetic from operands copied asynchronously into shared memory; element
// offsets are 32-bit (fits).

#include "kernels.h"
#include "simt_common.cuh"

namespace numc_k {
namespace f32 {

using u64 = unsigned long long;

__device__ __forceinline__ void fma2(u64 &d, u64 a, u64 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

__device__ __forceinline__ u64 twice(float a) {
  u64 d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(a));
  return d;
}

// A block's BM x BN outputs from shared memory to C, a warp along a row: rows from
// `r0` and columns from `c0` of the tile, inside the matrix.  Bounds, bias and
// column addresses once per column of lanes (with each element's own, shallow
// products were bound by it: 4000 x 16 x 4001 50 -> 25 us, 1000 x 30 x 1000 8.0 ->
// 5.4, 8192 x 64 x 8192 291 -> 216; 2000 x 1999 x 1501 247 -> 244).
template <int BM, int BN, int THREADS>
__device__ __forceinline__ void store_tile(const Gemm &g, const float *tile, int64_t m0, int64_t n0,
                                           int r0, int c0) {
  const int r1 = (int)min((int64_t)BM, g.M - m0), c1 = (int)min((int64_t)BN, g.N - n0);
  float *out = (float *)g.c + m0 * g.rso + n0 * g.cso;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
#pragma unroll
  for (int cc = 0; cc < BN; cc += 32) {
    const int c = cc + lane;
    if (c < c0 || c >= c1) continue;
    const float bias = g.bias ? ((const float *)g.bias)[(n0 + c) * g.bias_stride] : 0.0f;
    float *dst = out + c * g.cso + (r0 + warp) * g.rso;
    const float *src = tile + c + (r0 + warp) * BN;
#pragma unroll 4
    for (int r = r0 + warp; r < r1; r += THREADS / 32) {
      *dst = g.bias ? simt::add_elem<float>(*src, bias) : *src;
      dst += THREADS / 32 * g.rso;
      src += THREADS / 32 * BN;
    }
  }
}

// TY x TX threads of TM x TN outputs.
template <int TY, int TX, int TM, int TN>
struct F32Cfg {
  static constexpr int BK = 16, BM = TY * TM, BN = TX * TN;
  // pitches that spread the stores of 16 k a row or column over the banks
  static constexpr int APITCH = BM + 4, BPITCH = BN + 4;
  static constexpr int STAGES = 3, STAGE = BK * (APITCH + BPITCH);   // floats
  static constexpr int SMEM = (STAGES * STAGE + BM * BN) * 4;   // the ring, edge sums
};

// 4 bytes from global to shared memory; `bytes` = 0 writes zero instead.
__device__ __forceinline__ void copy4(uint32_t dst, const float *src, int bytes = 4) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes));
}

__device__ __forceinline__ void store4(uint32_t dst, float x) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(dst), "f"(x));
}

// The copies of one tile's slabs by a block's threads.  The last tiles move inside
// the matrix, so that no load needs a check of rows or columns: they compute some
// outputs of their neighbours again and leave them unstored.  A matrix narrower
// than a tile repeats its last row or column.
template <int TY, int TX, int TM, int TN>
struct F32Loads {
  using Cfg = F32Cfg<TY, TX, TM, TN>;
  static constexpr int THREADS = TY * TX, BK = Cfg::BK, BM = Cfg::BM, BN = Cfg::BN;
  static constexpr int LA = BM * BK / THREADS, LB = BK * BN / THREADS;
  static_assert(BM % (THREADS / BK) == 0 && BN % (THREADS / BK) == 0, "load mapping");
  const float *pa, *pb;
  int64_t step_a, step_b;
  int oa[LA], ob[LB];   // element offsets (fits())
  bool a_k, b_n;

  // Element q of a thread's share of a slab: along k first where k is the
  // contiguous axis (A) or along columns (B).
  __device__ __forceinline__ int a_row(int q) const {
    return a_k ? threadIdx.x / BK + q * (THREADS / BK) : (threadIdx.x + THREADS * q) % BM;
  }
  __device__ __forceinline__ int a_kk(int q) const {
    return a_k ? threadIdx.x % BK : (threadIdx.x + THREADS * q) / BM;
  }
  __device__ __forceinline__ int b_col(int q) const {
    return b_n ? (threadIdx.x + THREADS * q) % BN : threadIdx.x / BK + q * (THREADS / BK);
  }
  __device__ __forceinline__ int b_kk(int q) const {
    return b_n ? (threadIdx.x + THREADS * q) / BN : threadIdx.x % BK;
  }
  // (m0, n0): the tile's first output
  __device__ __forceinline__ void start(const float *a, const float *b, int64_t rsa, int64_t csa,
                                        int64_t rsb, int64_t csb, int64_t M, int64_t N, int64_t m0,
                                        int64_t n0) {
    a_k = csa == 1, b_n = csb == 1 || rsb != 1;
    pa = a + m0 * rsa, pb = b + n0 * csb;
    step_a = BK * csa, step_b = BK * rsb;
    const int mr = (int)min((int64_t)BM, M - m0) - 1, nr = (int)min((int64_t)BN, N - n0) - 1;
#pragma unroll
    for (int q = 0; q < LA; q++) oa[q] = min(a_row(q), mr) * (int)rsa + a_kk(q) * (int)csa;
#pragma unroll
    for (int q = 0; q < LB; q++) ob[q] = b_kk(q) * (int)rsb + min(b_col(q), nr) * (int)csb;
  }
  // The next slab into the stage at shared address `sa`; `left` k steps, this
  // slab included.
  __device__ __forceinline__ void slab(uint32_t sa, int64_t left) {
    const uint32_t sb = sa + BK * Cfg::APITCH * 4;
    if (left >= BK) {
#pragma unroll
      for (int q = 0; q < LA; q++) copy4(sa + (a_kk(q) * Cfg::APITCH + a_row(q)) * 4, pa + oa[q]);
#pragma unroll
      for (int q = 0; q < LB; q++) copy4(sb + (b_kk(q) * Cfg::BPITCH + b_col(q)) * 4, pb + ob[q]);
    } else {   // past K: zeros, from an address inside the matrix
#pragma unroll
      for (int q = 0; q < LA; q++)
        copy4(sa + (a_kk(q) * Cfg::APITCH + a_row(q)) * 4, a_kk(q) < left ? pa + oa[q] : pa,
              a_kk(q) < left ? 4 : 0);
#pragma unroll
      for (int q = 0; q < LB; q++)
        copy4(sb + (b_kk(q) * Cfg::BPITCH + b_col(q)) * 4, b_kk(q) < left ? pb + ob[q] : pb,
              b_kk(q) < left ? 4 : 0);
    }
    pa += step_a;
    pb += step_b;
  }
  // -0 for the zeros that this thread's own copies, complete, wrote past K in B's part
  // of the stage at `sa`: fma(+0, -0, x) is x, -0 included.
  __device__ __forceinline__ void past_k(uint32_t sa, int left) const {
    const uint32_t sb = sa + BK * Cfg::APITCH * 4;
#pragma unroll
    for (int q = 0; q < LB; q++)
      if (b_kk(q) >= left) store4(sb + (b_kk(q) * Cfg::BPITCH + b_col(q)) * 4, -0.0f);
  }
};

// A thread's outputs of one tile.
template <int TY, int TX, int TM, int TN>
struct F32Acc {
  using Cfg = F32Cfg<TY, TX, TM, TN>;
  static constexpr int THREADS = TY * TX, BK = Cfg::BK, BN = Cfg::BN;
  u64 acc[TM][TN / 2];
  // numc's remainder tiles (rows from er, columns from ec, where K spans several
  // blocks of 256) sum each K block from zero: at a block's end their chains
  // are added to sums in shared memory and start again.
  uint32_t edge_i, edge_j;   // this thread's rows and columns among them

  // rows 4 c + i of thread ty, columns in pairs: conflict-free 16-byte reads
  static __device__ __forceinline__ int row_of(int i) {
    return i / 4 * (4 * TY) + (int)threadIdx.x / TX * 4 + i % 4;
  }
  static __device__ __forceinline__ int col_of(int j) {
    const int tx = threadIdx.x % TX;
    return j < TN / 4 * 4 ? j / 4 * (4 * TX) + tx * 4 + j % 4 : TN / 4 * (4 * TX) + tx * 2 + j % 4;
  }
  __device__ __forceinline__ bool is_edge(int i, int j) const { return (edge_i >> i | edge_j >> j) & 1; }
  __device__ __forceinline__ float output(int i, int j) const {
    return __uint_as_float((uint32_t)(acc[i][j / 2] >> (32 * (j & 1))));
  }

  __device__ __forceinline__ void start(int64_t M, int64_t N, int64_t K, int isa, int64_t m0,
                                        int64_t n0) {
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < TN / 2; j++) acc[i][j] = 0;   // (+0, +0)
    edge_i = edge_j = 0;
    if (!simt::float_edges_needed<float>(K)) return;
    const int64_t er = simt::edge_row<float>(M, isa), ec = simt::edge_col<float>(N, isa);
#pragma unroll
    for (int i = 0; i < TM; i++) edge_i |= m0 + row_of(i) >= er ? 1u << i : 0;
#pragma unroll
    for (int j = 0; j < TN; j++) edge_j |= n0 + col_of(j) >= ec ? 1u << j : 0;
  }

  __device__ __forceinline__ void slab(const float *As) {
    const float *Bs = As + BK * Cfg::APITCH;
    // operands of the next k are read while this k's FMAs run
    float4 a[2][TM / 4];
    u64 b[2][TN / 2];
    auto fetch = [&](int k) {
#pragma unroll
      for (int i = 0; i < TM; i += 4)
        a[k & 1][i / 4] = *reinterpret_cast<const float4 *>(As + k * Cfg::APITCH + row_of(i));
#pragma unroll
      for (int j = 0; j < TN / 4; j++) {
        const ulonglong2 v =
            *reinterpret_cast<const ulonglong2 *>(Bs + k * Cfg::BPITCH + col_of(4 * j));
        b[k & 1][2 * j] = v.x;
        b[k & 1][2 * j + 1] = v.y;
      }
      if constexpr (TN % 4 != 0)
        b[k & 1][TN / 2 - 1] = *reinterpret_cast<const u64 *>(Bs + k * Cfg::BPITCH + col_of(TN - 2));
    };
    fetch(0);
#pragma unroll
    for (int k = 0; k < BK; k++) {
      if (k + 1 < BK) fetch(k + 1);
#pragma unroll
      for (int i = 0; i < TM; i++) {
        const float4 v = a[k & 1][i / 4];
        const u64 aa = twice(i % 4 == 0 ? v.x : i % 4 == 1 ? v.y : i % 4 == 2 ? v.z : v.w);
#pragma unroll
        for (int j = 0; j < TN / 2; j++) fma2(acc[i][j], aa, b[k & 1][j]);
      }
    }
  }

  // The first n k steps of a slab, n below its depth.
  __device__ __forceinline__ void part_slab(const float *As, int n) {
    const float *a0 = As + row_of(0), *b0 = As + BK * Cfg::APITCH;
#pragma unroll 1
    for (int k = 0; k < n; k++, a0 += Cfg::APITCH, b0 += Cfg::BPITCH) {
      u64 b[TN / 2];
#pragma unroll
      for (int j = 0; j < TN; j += 2) b[j / 2] = *reinterpret_cast<const u64 *>(b0 + col_of(j));
#pragma unroll
      for (int i = 0; i < TM; i++) {
        const u64 aa = twice(a0[row_of(i) - row_of(0)]);
#pragma unroll
        for (int j = 0; j < TN / 2; j++) fma2(acc[i][j], aa, b[j]);
      }
    }
  }

  // The end of slab t of `slabs`: remainder outputs at the end of a K block but the
  // last, which to_shared adds.
  // bsum: the tile's edge sums, THREADS apart, this thread's first.
  __device__ __forceinline__ void end_slab(int64_t t, int64_t slabs, float *bsum) {
    if (!(edge_i | edge_j) || (t + 1) * BK % simt::kNumcKC != 0 || t + 1 == slabs) return;
    const bool first = t < simt::kNumcKC / BK;
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < TN; j++)
        if (is_edge(i, j)) {
          float *b = bsum + (i * TN + j) * THREADS;
          *b = first ? output(i, j) : simt::add_rn<float>(*b, output(i, j));
          acc[i][j / 2] &= j & 1 ? 0xffffffffull : 0xffffffff00000000ull;
        }
  }

  // The outputs to shared memory, where the block's threads store them row by
  // row: a thread's own 4 columns went out as quarters of 32-byte sectors
  // (2000 x 1999 x 1501 269 -> 247 us, 1000^3 66 -> 61).  `tile` may be the edge
  // sums' or the ring's space.
  __device__ __forceinline__ void to_shared(float *tile, const float *bsum) {
    if (edge_i | edge_j) {
#pragma unroll
      for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++)
          if (is_edge(i, j)) {
            const u64 v = __float_as_uint(simt::add_rn<float>(bsum[(i * TN + j) * THREADS], output(i, j)));
            acc[i][j / 2] = j & 1 ? (acc[i][j / 2] & 0xffffffffull) | v << 32
                                  : (acc[i][j / 2] & 0xffffffff00000000ull) | v;
          }
    }
    __syncthreads();   // everyone is done with the last slab and the edge sums
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < TN; j += 2)
        *reinterpret_cast<u64 *>(tile + row_of(i) * BN + col_of(j)) = acc[i][j / 2];
    __syncthreads();
  }
};

// ---- small problems ------------------------------------------------------------
//
// With few tiles the K loop's latency decides: a thread holds 2 x 2 or 4 x 4
// outputs, A lies in shared memory row by row so that one 16-byte read brings a
// row's next four k, and slabs are 32 deep, copied 16 bytes at a time where
// the operand's strides and alignment allow it.  SMALL is numc's unpacked path
// (its narrow tiles' scalar columns round product and sum separately); else the
// packed path, remainder outputs summed per 256-deep K block in registers.
//
// Of a last slab only the steps below K may count: one past it, fma(0, 0, x), makes
// +0 of a chain that ended in -0, as numc's does where every product underflows
// from below.  Those steps run in a loop of their own (20 x 3 x 20 3.5 -> 2.8 us,
// 150 x 127 x 150 3.6 -> 3.9, 500 grouped problems of 16 to 256 135 -> 118), except with
// 4 x 4 outputs and 16-byte copies of both operands, where that loop spoils the
// order of the main one (512^3 13.8 -> 14.9): there B's rows past K are kPastK, and
// fma(+0, -0, x) is x.
// Measured, us before (2 x 2 outputs of 32 x 32 tiles, element copies) and after:
//   96^3 4.3 / 3.2, 128^3 4.5 / 3.0, 256 x 784 x 128 17.7 / 9.8, 64 x 1000 x 64 22 / 11.5,
//   512^3 18.7 / 14.0, 200 x 3000 x 200 67 / 36.5, 700^3 51 / 29.
template <int TY, int TX, int TM, int TN>
struct F32SmallCfg {
  // 2 x 2: 64 deep (256 x 784 x 128: 9.7 us, 14.4 with 32, 10.0 with 128); 4 x 4:
  // 32 (64: the same on aligned operands, 33 against 24 us on 255 x 783 x 127)
  static constexpr int BK = TM == 2 ? 64 : 32, BM = TY * TM, BN = TX * TN;
  static constexpr int APITCH = BK + 4, BPITCH = BN + 4;
  static constexpr int STAGES = TM == 2 ? 3 : 4, STAGE = BM * APITCH + BK * BPITCH;   // floats
  static constexpr int SMEM = STAGES * STAGE * 4;
};

// 16 bytes from global to shared memory, zeros past `bytes`.
__device__ __forceinline__ void copy16(uint32_t dst, const float *src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes));
}

static __device__ const float4 kPastK = {-0.0f, -0.0f, -0.0f, -0.0f};

template <int TY, int TX, int TM, int TN, bool SMALL, bool VA, bool VB>
__device__ __forceinline__ void f32_small_tile(const Gemm &g, int64_t m0, int64_t n0, float *smem) {
  using Cfg = F32SmallCfg<TY, TX, TM, TN>;
  constexpr int THREADS = TY * TX, BK = Cfg::BK, BM = Cfg::BM, BN = Cfg::BN;
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const float *A = (const float *)g.a, *B = (const float *)g.b;
  const int mr = (int)min((int64_t)BM, g.M - m0) - 1, nr = (int)min((int64_t)BN, g.N - n0) - 1;
  const bool a_k = g.csa == 1, b_n = g.csb == 1 || g.rsb != 1;
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  constexpr bool PAD = TM == 4 && VA && VB;   // kPastK past K, no loop for a part of a slab
  // Rows and columns past the matrix repeat the last one (in 16-byte copies:
  // columns past it are zeros); k past K is zeros (but PAD), from an address inside.
  // Strides fit 32 bits (the launcher checks).
  const float *pa = A + m0 * g.rsa, *pb = B + n0 * g.csb;
  const int rsa = (int)g.rsa, csa = (int)g.csa, rsb = (int)g.rsb, csb = (int)g.csb;
  auto load = [&](int stage, int left) {   // k steps left, this slab included
    const uint32_t sa = sbase + stage * Cfg::STAGE * 4, sb = sa + BM * Cfg::APITCH * 4;
    const bool full = left >= BK;
    if constexpr (VA) {
#pragma unroll
      for (int q = 0; q < BM * BK / 4 / THREADS; q++) {
        const int e = tid + q * THREADS, r = e / (BK / 4), k = e % (BK / 4) * 4;
        const int n = full ? 4 : max(0, min(4, left - k));
        copy16(sa + (r * Cfg::APITCH + k) * 4, pa + min(r, mr) * rsa + (n ? k : 0), 4 * n);
      }
    } else {
#pragma unroll
      for (int q = 0; q < BM * BK / THREADS; q++) {
        const int e = tid + q * THREADS, r = a_k ? e / BK : e % BM, k = a_k ? e % BK : e / BM;
        const bool in = full || k < left;
        copy4(sa + (r * Cfg::APITCH + k) * 4, pa + min(r, mr) * rsa + (in ? k : 0) * csa, in ? 4 : 0);
      }
    }
    if constexpr (VB) {
#pragma unroll
      for (int q = 0; q < BK * BN / 4 / THREADS; q++) {
        const int e = tid + q * THREADS, k = e / (BN / 4), c = e % (BN / 4) * 4;
        const int n = full || k < left ? max(0, min(4, nr + 1 - c)) : 0;
        const bool past = PAD && !full && k >= left;
        copy16(sb + (k * Cfg::BPITCH + c) * 4, past ? &kPastK.x : n ? pb + k * rsb + c : pb,
               past ? 16 : 4 * n);
      }
    } else {
#pragma unroll
      for (int q = 0; q < BK * BN / THREADS; q++) {
        const int e = tid + q * THREADS, k = b_n ? e / BN : e % BK, c = b_n ? e % BN : e / BK;
        const bool in = full || k < left;
        copy4(sb + (k * Cfg::BPITCH + c) * 4, pb + (in ? k : 0) * rsb + min(c, nr) * csb, in ? 4 : 0);
      }
    }
    pa += BK * g.csa;
    pb += BK * g.rsb;
  };
  auto row_of = [&](int i) { return i * TY + ty; };   // A's rows: distinct banks across ty
  auto col_of = [&](int j) { return tx * TN + j; };

  float acc[TM][TN], bsum[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int j = 0; j < TN; j++) acc[i][j] = bsum[i][j] = 0.0f;
  uint32_t edge = 0, unfused = 0;   // remainder outputs; scalar columns
  if constexpr (SMALL) {
#pragma unroll
    for (int j = 0; j < TN; j++)
      if (simt::small_col_unfused<float>(n0 + col_of(j), g.N, g.isa)) unfused |= 1u << j;
  } else if (simt::float_edges_needed<float>(g.K)) {
    const int64_t er = simt::edge_row<float>(g.M, g.isa), ec = simt::edge_col<float>(g.N, g.isa);
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < TN; j++)
        if (m0 + row_of(i) >= er || n0 + col_of(j) >= ec) edge |= 1u << (i * TN + j);
  }

  auto step = [&](float a, float b, float x, int j) {
    return SMALL && (unfused >> j & 1) ? simt::madd_unfused(a, b, x) : __fmaf_rn(a, b, x);
  };
  auto end_block = [&](int t) {   // remainder outputs at the end of their K block, in slab t
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < TN; j++)
        if (edge >> (i * TN + j) & 1) {
          bsum[i][j] = t < simt::kNumcKC / BK ? acc[i][j] : simt::add_rn<float>(bsum[i][j], acc[i][j]);
          acc[i][j] = 0.0f;
        }
  };
  const int slabs = (int)((g.K + BK - 1) / BK);
#pragma unroll
  for (int t = 0; t < Cfg::STAGES - 1; t++) {
    if (t < slabs) load(t, (int)g.K - t * BK);
    asm volatile("cp.async.commit_group;");
  }
  const int whole = PAD ? slabs : (int)g.K / BK;
  for (int t = 0; t < whole; t++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(Cfg::STAGES - 2) : "memory");
    __syncthreads();   // slab t has arrived, and everyone is done with slab t - 1
    const int tn = t + Cfg::STAGES - 1;
    if (tn < slabs) load(tn % Cfg::STAGES, (int)g.K - tn * BK);
    asm volatile("cp.async.commit_group;");
    const float *As = smem + t % Cfg::STAGES * Cfg::STAGE, *Bs = As + BM * Cfg::APITCH;
    // Operands of the next four k are read while this four's FMAs run (2 x 2 outputs
    // and element copies: the compiler's own order is the faster one, 12.2
    // against 16.0 us for 255 x 783 x 127; 2 x 2 and 16-byte copies: 9.6 against 13.1
    // for 256 x 784 x 128).
    constexpr int P = TM * TN > 4 || (VA && VB) ? 2 : 1;
    float av[P][TM][4], bv[P][4][TN];
    auto fetch = [&](int k4) {
      float(&a)[TM][4] = av[k4 / 4 % P];
      float(&b)[4][TN] = bv[k4 / 4 % P];
#pragma unroll
      for (int i = 0; i < TM; i++)
        *reinterpret_cast<float4 *>(a[i]) =
            *reinterpret_cast<const float4 *>(As + row_of(i) * Cfg::APITCH + k4);
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const float *src = Bs + (k4 + k) * Cfg::BPITCH + col_of(0);
        if constexpr (TN == 4) *reinterpret_cast<float4 *>(b[k]) = *reinterpret_cast<const float4 *>(src);
        else *reinterpret_cast<float2 *>(b[k]) = *reinterpret_cast<const float2 *>(src);
      }
    };
    if (P == 2) fetch(0);
    // (the unpacked path's problems are a few slabs: fetching the code of a whole
    // one's steps took longer than running it, 96^3 5.2 -> 4.2 us, the same 500
    // grouped problems 118 -> 107)
#pragma unroll (SMALL ? 4 : BK / 4)
    for (int k4 = 0; k4 < BK; k4 += 4) {
      if (P == 1) fetch(k4);
      else if (k4 + 4 < BK) fetch(k4 + 4);
      const float(&a)[TM][4] = av[k4 / 4 % P];
      const float(&b)[4][TN] = bv[k4 / 4 % P];
#pragma unroll
      for (int k = 0; k < 4; k++)
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
          for (int j = 0; j < TN; j++) acc[i][j] = step(a[i][k], b[k][j], acc[i][j], j);
    }
    if (!SMALL && edge && ((t + 1) * BK % simt::kNumcKC == 0 || t + 1 == slabs)) end_block(t);
  }
  if (whole < slabs) {
    // the last slab's steps below K, four at a time (unrolled: 25 x 829 x 274 14.2 ->
    // 14.0 us; the unpacked path: see above)
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const float *a0 = smem + whole % Cfg::STAGES * Cfg::STAGE + row_of(0) * Cfg::APITCH;
    const float *b0 = smem + whole % Cfg::STAGES * Cfg::STAGE + BM * Cfg::APITCH + col_of(0);
    const int n = (int)g.K - whole * BK;
    int k = 0;
#pragma unroll (SMALL ? 1 : 4)
    for (; k + 4 <= n; k += 4) {
      float a[TM][4], b[4][TN];
#pragma unroll
      for (int i = 0; i < TM; i++)
        *reinterpret_cast<float4 *>(a[i]) =
            *reinterpret_cast<const float4 *>(a0 + i * TY * Cfg::APITCH + k);
#pragma unroll
      for (int q = 0; q < 4; q++)
#pragma unroll
        for (int j = 0; j < TN; j += 2)
          *reinterpret_cast<float2 *>(b[q] + j) =
              *reinterpret_cast<const float2 *>(b0 + (k + q) * Cfg::BPITCH + j);
#pragma unroll
      for (int q = 0; q < 4; q++)
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
          for (int j = 0; j < TN; j++) acc[i][j] = step(a[i][q], b[q][j], acc[i][j], j);
    }
#pragma unroll 1
    for (; k < n; k++) {
      float a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; i++) a[i] = a0[i * TY * Cfg::APITCH + k];
#pragma unroll
      for (int j = 0; j < TN; j++) b[j] = b0[k * Cfg::BPITCH + j];
#pragma unroll
      for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = step(a[i], b[j], acc[i][j], j);
    }
    if (!SMALL && edge) end_block(whole);
  }
#pragma unroll
  for (int i = 0; i < TM; i++) {
    const int64_t row = m0 + row_of(i);
    if (row >= g.M) continue;
    float *c = (float *)g.c + row * g.rso;
#pragma unroll
    for (int j = 0; j < TN; j++) {
      const int64_t col = n0 + col_of(j);
      if (col >= g.N) continue;
      float v = edge >> (i * TN + j) & 1 ? bsum[i][j] : acc[i][j];
      if (g.bias) v = simt::add_elem<float>(v, ((const float *)g.bias)[col * g.bias_stride]);
      c[col * g.cso] = v;
    }
  }
}

// The tiles' slab offsets and K are 32-bit.
inline bool fits(int64_t rsa, int64_t csa, int64_t rsb, int64_t csb, int64_t K) {
  return 128 * rsa + 64 * csa < 1ll << 31 && 64 * rsb + 96 * csb < 1ll << 31 &&
         K < (1ll << 31) - 64;
}

// 16-byte copies along k (A) and along columns (B).
__host__ __device__ inline bool vec_a(const void *a, int64_t rsa, int64_t csa) {
  return csa == 1 && rsa % 4 == 0 && ((uintptr_t)a & 15) == 0;
}
__host__ __device__ inline bool vec_b(const void *b, int64_t rsb, int64_t csb) {
  return csb == 1 && rsb % 4 == 0 && ((uintptr_t)b & 15) == 0;
}

}  // namespace f32
}  // namespace numc_k

// float32 GEMM on the CUDA cores with packed FMAs: numc's arithmetic, one
// fused multiply-add chain per output in k order (src/intrinsics/
// gemm_avx2.h:852-950), remainder tiles summed per K block.
//
// What bounds it: an SM's FP32 pipes take 128 FMAs a cycle, its shared memory
// returns 128 bytes a cycle (broadcasts included), and a scheduler issues one
// instruction a cycle.  With 8 x 8 outputs a thread a k costs a warp 16 cycles of
// shared reads for 16 cycles of FMAs, and scalar FFMAs fill every issue slot
// (46 TFLOP/s at 8192^3: 65 % of the FMA pipes).  Here a thread holds up to 8 x 12
// outputs, so that reads take 20 of 24 cycles, and fma.rn.f32x2 does two FMAs an
// instruction (each rounded as the scalar one is), which leaves issue slots for
// the reads, the moves that double A's values into pairs and the copies.
// Operands arrive by 4-byte cp.async in a three-stage ring (any strides and
// alignment; 16-byte copies need both).  Measured, us before and after:
//   1000^3 84 / 66, 2000 x 1999 x 1501 591 / 269, 300 x 2500 x 1700 168 / 111,
//   2048^3 511 / 394, 8192^3 23834 / 20098 (55 TFLOP/s).
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>

#include "kernels.h"
#include "simt_common.cuh"

namespace numc_k {
namespace {

using u64 = unsigned long long;

__device__ __forceinline__ void fma2(u64 &d, u64 a, u64 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

__device__ __forceinline__ u64 twice(float a) {
  u64 d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(a));
  return d;
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

template <int TY, int TX, int TM, int TN, int CTAS>
__global__ void __launch_bounds__(TY * TX, CTAS)
f32_gemm(const Gemm g, unsigned tiles_n) {
  using Cfg = F32Cfg<TY, TX, TM, TN>;
  constexpr int THREADS = TY * TX, BK = Cfg::BK, BM = Cfg::BM, BN = Cfg::BN;
  static_assert(BM % (THREADS / BK) == 0 && BN % (THREADS / BK) == 0, "load mapping");
  constexpr int LA = BM * BK / THREADS, LB = BK * BN / THREADS;
  // The last tiles move inside the matrix, so that no load needs a check of
  // rows or columns: they compute some outputs of their neighbours again and
  // leave them unstored.  A matrix narrower than a tile repeats its last row or
  // column.
  const int64_t mt = (int64_t)(blockIdx.x / tiles_n) * BM, nt = (int64_t)(blockIdx.x % tiles_n) * BN;
  const int64_t m0 = max((int64_t)0, min(mt, g.M - BM)), n0 = max((int64_t)0, min(nt, g.N - BN));
  extern __shared__ __align__(16) float smem[];

  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  // Element q of a thread's share of a slab: along k first where k is the
  // contiguous axis (A) or along columns (B).
  const bool a_k = g.csa == 1, b_n = g.csb == 1 || g.rsb != 1;
  auto a_row = [&](int q) { return a_k ? tid / BK + q * (THREADS / BK) : (tid + THREADS * q) % BM; };
  auto a_kk = [&](int q) { return a_k ? tid % BK : (tid + THREADS * q) / BM; };
  auto b_col = [&](int q) { return b_n ? (tid + THREADS * q) % BN : tid / BK + q * (THREADS / BK); };
  auto b_kk = [&](int q) { return b_n ? (tid + THREADS * q) / BN : tid % BK; };
  const float *pa = (const float *)g.a + m0 * g.rsa, *pb = (const float *)g.b + n0 * g.csb;
  const int mr = (int)min((int64_t)BM, g.M - m0) - 1, nr = (int)min((int64_t)BN, g.N - n0) - 1;
  int oa[LA], ob[LB];   // element offsets (the launcher checks that they fit)
#pragma unroll
  for (int q = 0; q < LA; q++) oa[q] = min(a_row(q), mr) * (int)g.rsa + a_kk(q) * (int)g.csa;
#pragma unroll
  for (int q = 0; q < LB; q++) ob[q] = b_kk(q) * (int)g.rsb + min(b_col(q), nr) * (int)g.csb;
  const int64_t step_a = BK * g.csa, step_b = BK * g.rsb;
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  auto load = [&](int stage, int64_t left) {   // k steps left, this slab included
    const uint32_t sa = sbase + stage * Cfg::STAGE * 4, sb = sa + BK * Cfg::APITCH * 4;
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
  };
  // rows 4 c + i of thread ty, columns in pairs: conflict-free 16-byte reads
  auto row_of = [&](int i) { return i / 4 * (4 * TY) + ty * 4 + i % 4; };
  auto col_of = [&](int j) {
    return j < TN / 4 * 4 ? j / 4 * (4 * TX) + tx * 4 + j % 4 : TN / 4 * (4 * TX) + tx * 2 + j % 4;
  };

  u64 acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int j = 0; j < TN / 2; j++) acc[i][j] = 0;   // (+0, +0)

  // numc's remainder tiles (rows from er, columns from ec, where K spans several
  // blocks of 256) sum each K block from zero: at a block's end their chains
  // are added to sums in shared memory and start again.
  const bool multi = simt::float_edges_needed<float>(g.K);
  const int64_t er = multi ? simt::edge_row<float>(g.M, g.isa) : g.M;
  const int64_t ec = multi ? simt::edge_col<float>(g.N, g.isa) : g.N;
  uint32_t edge_i = 0, edge_j = 0;   // this thread's rows and columns among them
#pragma unroll
  for (int i = 0; i < TM; i++) edge_i |= m0 + row_of(i) >= er ? 1u << i : 0;
#pragma unroll
  for (int j = 0; j < TN; j++) edge_j |= n0 + col_of(j) >= ec ? 1u << j : 0;
  float *bsum = smem + Cfg::STAGES * Cfg::STAGE + tid;
  auto is_edge = [&](int i, int j) { return (edge_i >> i | edge_j >> j) & 1; };
  auto output = [&](int i, int j) { return __uint_as_float((uint32_t)(acc[i][j / 2] >> (32 * (j & 1)))); };
  auto fold_edges = [&](bool first) {
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < TN; j++)
        if (is_edge(i, j)) {
          float *b = bsum + (i * TN + j) * THREADS;
          *b = first ? output(i, j) : simt::add_rn<float>(*b, output(i, j));
          acc[i][j / 2] &= j & 1 ? 0xffffffffull : 0xffffffff00000000ull;
        }
  };

  const int64_t slabs = (g.K + BK - 1) / BK;
#pragma unroll
  for (int t = 0; t < Cfg::STAGES - 1; t++) {
    if (t < slabs) load(t, g.K - t * BK);
    asm volatile("cp.async.commit_group;");
  }
  int stage = 0;
  for (int64_t t = 0; t < slabs; t++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(Cfg::STAGES - 2) : "memory");
    __syncthreads();   // slab t has arrived, and everyone is done with slab t - 1
    const int64_t tn = t + Cfg::STAGES - 1;
    const int into = stage == 0 ? Cfg::STAGES - 1 : stage - 1;
    if (tn < slabs) load(into, g.K - tn * BK);
    asm volatile("cp.async.commit_group;");
    const float *As = smem + stage * Cfg::STAGE, *Bs = As + BK * Cfg::APITCH;
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
    if (++stage == Cfg::STAGES) stage = 0;
    if ((edge_i | edge_j) && ((t + 1) * BK % simt::kNumcKC == 0 || t + 1 == slabs))
      fold_edges(t < simt::kNumcKC / BK);
  }

#pragma unroll
  for (int i = 0; i < TM; i++) {
    const int64_t row = m0 + row_of(i);
    if (row < mt || row >= g.M) continue;
    float *c = (float *)g.c + row * g.rso;
#pragma unroll
    for (int j = 0; j < TN; j++) {
      const int64_t col = n0 + col_of(j);
      if (col < nt || col >= g.N) continue;
      float v = is_edge(i, j) ? bsum[(i * TN + j) * THREADS] : output(i, j);
      if (g.bias) v = simt::add_elem<float>(v, ((const float *)g.bias)[col * g.bias_stride]);
      c[col * g.cso] = v;
    }
  }
}

template <int TY, int TX, int TM, int TN, int CTAS>
cudaError_t launch_tiles(const Gemm &g, cudaStream_t s) {
  using Cfg = F32Cfg<TY, TX, TM, TN>;
  constexpr int BM = Cfg::BM, BN = Cfg::BN, THREADS = TY * TX;
  auto kern = f32_gemm<TY, TX, TM, TN, CTAS>;
  const int64_t tm = (g.M + BM - 1) / BM, tn = (g.N + BN - 1) / BN;
  if (tm * tn >= 1ll << 31) return cudaErrorInvalidConfiguration;
  static LaunchCache lc;
  cudaError_t e = smem_attr_once(lc, (const void *)kern, Cfg::SMEM);
  if (e) return e;
  kern<<<(unsigned)(tm * tn), THREADS, Cfg::SMEM, s>>>(g, (unsigned)tn);
  count_launch();
  return cudaGetLastError();
}

// ---- small problems ------------------------------------------------------------
//
// With few tiles the K loop's latency decides: a thread holds 2 x 2 or 4 x 4
// outputs, A lies in shared memory row by row so that one 16-byte read brings a
// row's next four k, and slabs are 32 deep, copied 16 bytes at a time where
// the operand's strides and alignment allow it.  SMALL is numc's unpacked path
// (its narrow tiles' scalar columns round product and sum separately); else the
// packed path, remainder outputs summed per 256-deep K block in registers.
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

template <int TY, int TX, int TM, int TN, bool SMALL, bool VA, bool VB>
__global__ void __launch_bounds__(TY * TX)
f32_small_gemm(const Gemm g, unsigned tiles_n) {
  using Cfg = F32SmallCfg<TY, TX, TM, TN>;
  constexpr int THREADS = TY * TX, BK = Cfg::BK, BM = Cfg::BM, BN = Cfg::BN;
  const int64_t m0 = (int64_t)(blockIdx.x / tiles_n) * BM, n0 = (int64_t)(blockIdx.x % tiles_n) * BN;
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const float *A = (const float *)g.a, *B = (const float *)g.b;
  const int mr = (int)min((int64_t)BM, g.M - m0) - 1, nr = (int)min((int64_t)BN, g.N - n0) - 1;
  const bool a_k = g.csa == 1, b_n = g.csb == 1 || g.rsb != 1;
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  // Rows and columns past the matrix repeat the last one (in 16-byte copies:
  // columns past it are zeros); k past K is zeros, from an address inside.
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
        copy16(sb + (k * Cfg::BPITCH + c) * 4, n ? pb + k * rsb + c : pb, 4 * n);
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

  const int slabs = (int)((g.K + BK - 1) / BK);
#pragma unroll
  for (int t = 0; t < Cfg::STAGES - 1; t++) {
    if (t < slabs) load(t, (int)g.K - t * BK);
    asm volatile("cp.async.commit_group;");
  }
  for (int t = 0; t < slabs; t++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(Cfg::STAGES - 2) : "memory");
    __syncthreads();   // slab t has arrived, and everyone is done with slab t - 1
    const int tn = t + Cfg::STAGES - 1;
    if (tn < slabs) load(tn % Cfg::STAGES, (int)g.K - tn * BK);
    asm volatile("cp.async.commit_group;");
    const float *As = smem + t % Cfg::STAGES * Cfg::STAGE, *Bs = As + BM * Cfg::APITCH;
    // 4 x 4 outputs: operands of the next four k are read while this four's
    // FMAs run (2 x 2: the compiler's own order is the faster one)
    constexpr int P = TM * TN > 4 ? 2 : 1;
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
#pragma unroll
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
          for (int j = 0; j < TN; j++) {
            if constexpr (SMALL)
              acc[i][j] = unfused >> j & 1 ? simt::madd_unfused(a[i][k], b[k][j], acc[i][j])
                                           : __fmaf_rn(a[i][k], b[k][j], acc[i][j]);
            else acc[i][j] = __fmaf_rn(a[i][k], b[k][j], acc[i][j]);
          }
    }
    if (!SMALL && edge && ((t + 1) * BK % simt::kNumcKC == 0 || t + 1 == slabs)) {
#pragma unroll
      for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++)
          if (edge >> (i * TN + j) & 1) {
            bsum[i][j] = t < simt::kNumcKC / BK ? acc[i][j] : simt::add_rn<float>(bsum[i][j], acc[i][j]);
            acc[i][j] = 0.0f;
          }
    }
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

// 16-byte copies along k (A) and along columns (B).
bool vec_a(const Gemm &g) { return g.csa == 1 && g.rsa % 4 == 0 && ((uintptr_t)g.a & 15) == 0; }
bool vec_b(const Gemm &g) { return g.csb == 1 && g.rsb % 4 == 0 && ((uintptr_t)g.b & 15) == 0; }

template <int TY, int TX, int TM, int TN, bool SMALL>
cudaError_t launch_small(const Gemm &g, cudaStream_t s) {
  using Cfg = F32SmallCfg<TY, TX, TM, TN>;
  const int64_t tm = (g.M + Cfg::BM - 1) / Cfg::BM, tn = (g.N + Cfg::BN - 1) / Cfg::BN;
  if (tm * tn >= 1ll << 31) return cudaErrorInvalidConfiguration;
  const bool va = vec_a(g), vb = vec_b(g);
  auto kern = va ? (vb ? f32_small_gemm<TY, TX, TM, TN, SMALL, true, true>
                       : f32_small_gemm<TY, TX, TM, TN, SMALL, true, false>)
                 : (vb ? f32_small_gemm<TY, TX, TM, TN, SMALL, false, true>
                       : f32_small_gemm<TY, TX, TM, TN, SMALL, false, false>);
  static LaunchCache lc[4];
  cudaError_t e = smem_attr_once(lc[2 * va + vb], (const void *)kern, Cfg::SMEM);
  if (e) return e;
  kern<<<(unsigned)(tm * tn), TY * TX, Cfg::SMEM, s>>>(g, (unsigned)tn);
  count_launch();
  return cudaGetLastError();
}

}  // namespace

namespace {
// The kernels' slab offsets and K are 32-bit.
bool f32_fits(const Gemm &g) {
  return 128 * g.rsa + 64 * g.csa < 1ll << 31 && 64 * g.rsb + 96 * g.csb < 1ll << 31 &&
         g.K < (1ll << 31) - 64;
}
}  // namespace

bool launch_f32_unpacked(const Gemm &g, cudaStream_t s, cudaError_t *e) {
  if (!f32_fits(g)) return false;
  *e = launch_small<8, 8, 2, 2, true>(g, s);
  return true;
}

bool launch_f32_packed(const Gemm &g, cudaStream_t s, cudaError_t *e) {
  if (!f32_fits(g)) return false;
  // Tiles, and measured cycles per k of one CTA alone on an SM and of each of
  // several (GB300, 64 x 1000 x 64 to 8192^3), for operands that the small
  // kernel can copy 16 bytes at a time and for others: the K loop of an SM's
  // CTAs decides, so the tile whose count rounds best wins.
  static constexpr struct { int bm, bn; double one[2], each[2]; } kTiles[] = {
      {128, 96, {166, 166}, {140, 140}}, {128, 80, {143, 143}, {124, 124}},
      {128, 64, {129, 129}, {105, 105}}, {64, 64, {118, 118}, {62, 62}},
      {32, 64, {75, 75}, {38, 38}},      {32, 32, {47, 47}, {22, 22}},
      {32, 32, {38, 46}, {18, 23}},      {16, 16, {17, 23}, {8, 9}}};
  const int odd = !(vec_a(g) && vec_b(g));
  const int64_t sms = sm_count();
  int best = 0;
  double t_best = 1e300;
  for (int i = 0; i < 8; i++) {
    const auto &k = kTiles[i];
    const int64_t tiles = ((g.M + k.bm - 1) / k.bm) * ((g.N + k.bn - 1) / k.bn);
    const double t = std::max(k.one[odd], k.each[odd] * (double)((tiles + sms - 1) / sms));
    if (t < t_best) {
      best = i;
      t_best = t;
    }
  }
  switch (best) {
  case 0: *e = launch_tiles<16, 8, 8, 12, 2>(g, s); break;
  case 1: *e = launch_tiles<16, 8, 8, 10, 2>(g, s); break;
  case 2: *e = launch_tiles<16, 8, 8, 8, 3>(g, s); break;
  case 3: *e = launch_tiles<8, 8, 8, 8, 4>(g, s); break;
  case 4: *e = launch_tiles<8, 8, 4, 8, 6>(g, s); break;
  case 5: *e = launch_tiles<8, 8, 4, 4, 8>(g, s); break;
  case 6: *e = launch_small<8, 8, 4, 4, false>(g, s); break;
  default: *e = launch_small<8, 8, 2, 2, false>(g, s); break;
  }
  return true;
}

}  // namespace numc_k

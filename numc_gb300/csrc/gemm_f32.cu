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

}  // namespace

bool launch_f32_packed(const Gemm &g, cudaStream_t s, cudaError_t *e) {
  // Tiles, and measured cycles per k of one CTA alone on an SM and of each of
  // several (GB300; 1000^3, 300 x 2500 x 1700, 2000 x 1999 x 1501, 2048^3 and
  // 8192^3): the K loop of an SM's CTAs decides, so the tile whose count
  // rounds best wins.  The last entry is the 32 x 32 tile of the kernel with
  // 2 x 2 outputs a thread, the faster one where no SM gets two tiles.
  static constexpr struct { int bm, bn; double one, each; } kTiles[] = {
      {128, 96, 166, 140}, {128, 80, 143, 124}, {128, 64, 129, 105}, {64, 64, 118, 62},
      {32, 64, 75, 38},    {32, 32, 47, 22},    {32, 32, 36, 30}};
  int best = -1;
  double t_best = 0;
  const int64_t sms = sm_count();
  for (int i = 0; i < 7; i++) {
    const int64_t tiles = ((g.M + kTiles[i].bm - 1) / kTiles[i].bm) *
                          ((g.N + kTiles[i].bn - 1) / kTiles[i].bn);
    const double t = std::max(kTiles[i].one, kTiles[i].each * (double)((tiles + sms - 1) / sms));
    if (best < 0 || t < t_best) {
      best = i;
      t_best = t;
    }
  }
  // slab offsets are 32-bit
  const int64_t far = std::max({128 * g.rsa + 16 * g.csa, 16 * g.rsb + 96 * g.csb});
  if (best == 6 || far >= 1ll << 31) return false;
  switch (best) {
  case 0: *e = launch_tiles<16, 8, 8, 12, 2>(g, s); break;
  case 1: *e = launch_tiles<16, 8, 8, 10, 2>(g, s); break;
  case 2: *e = launch_tiles<16, 8, 8, 8, 3>(g, s); break;
  case 3: *e = launch_tiles<8, 8, 8, 8, 4>(g, s); break;
  case 4: *e = launch_tiles<8, 8, 4, 8, 6>(g, s); break;
  default: *e = launch_tiles<8, 8, 4, 4, 8>(g, s); break;
  }
  return true;
}

}  // namespace numc_k

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
//   1000^3 84 / 61, 2000 x 1999 x 1501 591 / 244, 300 x 2500 x 1700 168 / 109,
//   2048^3 511 / 363, 8192^3 23834 / 20247 (54 TFLOP/s).
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>

#include "f32_tiles.cuh"
#include "kernels.h"

namespace numc_k {
namespace {

using namespace f32;

template <int TY, int TX, int TM, int TN, int CTAS>
__global__ void __launch_bounds__(TY * TX, CTAS) f32_gemm(const Gemm g, unsigned tiles_n) {
  using Cfg = F32Cfg<TY, TX, TM, TN>;
  constexpr int BK = Cfg::BK, BM = Cfg::BM, BN = Cfg::BN;
  extern __shared__ __align__(16) float smem[];
  const int64_t mt = (int64_t)(blockIdx.x / tiles_n) * BM, nt = (int64_t)(blockIdx.x % tiles_n) * BN;
  const int64_t m0 = max((int64_t)0, min(mt, g.M - BM)), n0 = max((int64_t)0, min(nt, g.N - BN));
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  F32Loads<TY, TX, TM, TN> ld;
  F32Acc<TY, TX, TM, TN> acc;
  ld.start((const float *)g.a, (const float *)g.b, g.rsa, g.csa, g.rsb, g.csb, g.M, g.N, m0, n0);
  acc.start(g.M, g.N, g.K, g.isa, m0, n0);
  float *bsum = smem + Cfg::STAGES * Cfg::STAGE + threadIdx.x;

  const int64_t slabs = (g.K + BK - 1) / BK;
#pragma unroll
  for (int t = 0; t < Cfg::STAGES - 1; t++) {
    if (t < slabs) ld.slab(sbase + t * Cfg::STAGE * 4, g.K - t * BK);
    asm volatile("cp.async.commit_group;");
  }
  int stage = 0;
  // Of a last slab only the steps below K may count (see F32SmallCfg): they run in a
  // loop of their own (2000 x 17 x 2000 13.2 -> 12.0 us), whose code has to be fetched
  // for it (2000 x 1999 x 1501, operands not in L2, 246.0 -> 248.9).  The 128 x 80 tile's deep
  // products take B's steps past K as -0 instead (245.5; the other tiles' main
  // loops get slower for it: 1000 x 999 x 1000 60.6 -> 64.0).
  const int64_t whole = g.K / BK, last = TN == 10 && whole >= 16 ? slabs : whole;
  for (int64_t t = 0; t < last; t++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(Cfg::STAGES - 2) : "memory");
    if (TN == 10 && t == whole) ld.past_k(sbase + stage * Cfg::STAGE * 4, (int)(g.K % BK));
    __syncthreads();   // slab t has arrived, and everyone is done with slab t - 1
    const int64_t tn = t + Cfg::STAGES - 1;
    const int into = stage == 0 ? Cfg::STAGES - 1 : stage - 1;
    if (tn < slabs) ld.slab(sbase + into * Cfg::STAGE * 4, g.K - tn * BK);
    asm volatile("cp.async.commit_group;");
    acc.slab(smem + stage * Cfg::STAGE);
    if (++stage == Cfg::STAGES) stage = 0;
    acc.end_slab(t, slabs, bsum);
  }
  if (last < slabs) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    acc.part_slab(smem + stage * Cfg::STAGE, (int)(g.K % BK));
  }
  acc.to_shared(smem, bsum);
  store_tile<BM, BN, TY * TX>(g, smem, m0, n0, (int)(mt - m0), (int)(nt - n0));
}

template <int TY, int TX, int TM, int TN, bool SMALL, bool VA, bool VB>
__global__ void __launch_bounds__(TY * TX) f32_small_gemm(const Gemm g, unsigned tiles_n) {
  using Cfg = F32SmallCfg<TY, TX, TM, TN>;
  extern __shared__ __align__(16) float smem[];
  f32_small_tile<TY, TX, TM, TN, SMALL, VA, VB>(g, (int64_t)(blockIdx.x / tiles_n) * Cfg::BM,
                                                (int64_t)(blockIdx.x % tiles_n) * Cfg::BN, smem);
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

template <int TY, int TX, int TM, int TN, bool SMALL>
cudaError_t launch_small(const Gemm &g, cudaStream_t s) {
  using Cfg = F32SmallCfg<TY, TX, TM, TN>;
  const int64_t tm = (g.M + Cfg::BM - 1) / Cfg::BM, tn = (g.N + Cfg::BN - 1) / Cfg::BN;
  if (tm * tn >= 1ll << 31) return cudaErrorInvalidConfiguration;
  const bool va = vec_a(g.a, g.rsa, g.csa), vb = vec_b(g.b, g.rsb, g.csb);
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

bool f32_fits(const Gemm &g) { return fits(g.rsa, g.csa, g.rsb, g.csb, g.K); }

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
  // CTAs decides, so the tile whose count rounds best wins (500 x 1000 x 450, two
  // 32 x 32 tiles an SM: 43 us with the small kernel, 33 with the packed one).
  static constexpr struct { int bm, bn; double one[2], each[2]; } kTiles[] = {
      {128, 96, {166, 166}, {140, 140}}, {128, 80, {143, 143}, {124, 124}},
      {128, 64, {129, 129}, {105, 105}}, {64, 64, {118, 118}, {62, 62}},
      {32, 64, {75, 75}, {38, 38}},      {32, 32, {47, 47}, {22, 22}},
      {32, 32, {38, 64}, {18, 42}},      {16, 16, {17, 23}, {8, 9}}};
  const int odd = !(vec_a(g.a, g.rsa, g.csa) && vec_b(g.b, g.rsb, g.csb));
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

// numc_array_rand on the GPU: numc's four-lane xoshiro256** uniform fill
// (numc's src/random/kernel.h:18-400 and src/random/random.c:28-180),
// bit-identical to numc for every dtype and both of numc's fill paths.
//
// numc's generator state is per host thread (kernel.h:40-41): four
// xoshiro256** streams ("lanes").  A fill of n elements of `size` bytes:
//  * n * size <= 1 MiB: element 4j + l is lane l's j-th output (j < n/4),
//    the n % 4 tail continues lane 0; the lanes end n/4 steps further on
//    and lane 0 n % 4 more;
//  * otherwise numc splits it over T = min(n * size / 512 KiB, its OpenMP
//    maximum) threads with chunks of ceil(n / T) elements: element
//    start + 4j + l of the chunk at `start` is X(start + l + j) and its
//    tail element start + 4J + r is X(start + J + r), X(m) being lane 0's
//    output m steps on (J = chunk length / 4); every lane ends n steps on.
// Both index maps need the state m steps ahead for arbitrary m.  A
// xoshiro256** step is linear over GF(2)^256, so m steps are the matrix T^m.
// Two table forms are built once on the host and kept on each device: the rows
// of T^(2^k), k < 64, and for a few k the products of T^(2^k) with the 16 values
// of each of a state's 64 nibbles.
//
// A block of 256 threads owns 256 runs of 2^logr consecutive steps (64 runs of
// each of the four lanes in the small fill).  It jumps its start state there
// with the row tables (thread r computes bit r of each product, ballots
// assemble the words), then doubles its set of start states: stage k makes
// states [2^k, 2^(k+1)) from [0, 2^k) with T^(2^(logr + k)), each product 64
// nibble lookups shared by the eight warps.  The lookups of a warp are in one
// nibble's 16 values, a bank each.  Then every thread steps its run.  In the
// large fill the four outputs of step j are X(m..m+3) of one stream, so a
// thread generates each value once and slides a window of four.  Outputs go
// through shared memory so that a warp writes whole 128-byte rows.  The host
// advances its copy of the state with its own nibble tables.
//
// What bounds it: small fills, the latency of the jumps (46 us for any fill up
// to 1 MiB and 33 us of every larger one when each warp ran its 31 spreading
// products one after another through bit parities; 11 to 15 us now).  Large
// fills, the generator itself: 64 Mi values take 43 us as int8 and 57 as float32
// (4.7 TB/s; 82 before), its 64-bit logic in the half-rate integer pipe, on
// two blocks a multiprocessor.
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>
#include <unistd.h>

#include "kernels.h"

namespace numc_k {
namespace {

__host__ __device__ __forceinline__ uint64_t rotl64(uint64_t x, int k) {
  return (x << k) | (x >> (64 - k));
}
// xoshiro256**: output of state s, then the state update (kernel.h:177-189)
__host__ __device__ __forceinline__ uint64_t xo_output(const uint64_t s[4]) {
  return rotl64(s[1] * 5, 7) * 9;
}
__host__ __device__ __forceinline__ void xo_advance(uint64_t s[4]) {
  const uint64_t t = s[1] << 17;
  s[2] ^= s[0];
  s[3] ^= s[1];
  s[1] ^= s[2];
  s[0] ^= s[3];
  s[2] ^= t;
  s[3] = rotl64(s[3], 45);
}

// ---- T^(2^k) as 256 x 256 bit matrices ------------------------------------
// Vector bit 64 w + i is bit i of state word w.  col[k][b] = T^(2^k) e_b;
// bit b of row[k][r] = bit r of col[k][b].
constexpr int kPowers = 64;
constexpr size_t kRowWords64 = (size_t)kPowers * 256 * 4;   // the row tables
// device nibble tables: T^(2^k) for k = kNibLo .. kNibHi
constexpr int kNibLo = 5, kNibHi = 15;
constexpr int kNibWords = 64 * 8 * 16;                      // 32-bit words of one

struct Tables {
  uint64_t nib[kPowers][64][16][4];   // [k][nibble][value]: T^(2^k) (value << 4 nibble)
  uint64_t row[kPowers][256][4];
};
Tables *g_tables = nullptr;
std::once_flag g_tables_once;

void apply_nib_host(const uint64_t (*nib)[16][4], uint64_t v[4]) {
  uint64_t r[4] = {0, 0, 0, 0};
  for (int i = 0; i < 64; i++) {
    const uint64_t *e = nib[i][(v[i >> 4] >> (4 * (i & 15))) & 15];
    for (int w = 0; w < 4; w++) r[w] ^= e[w];
  }
  memcpy(v, r, sizeof r);
}

void build_tables() {
  Tables *t = new Tables;
  for (int k = 0; k < kPowers; k++) {
    memset(t->row[k], 0, sizeof t->row[k]);
    for (int b = 0; b < 256; b++) {   // column b: T^(2^k) e_b = T^(2^(k-1)) (T^(2^(k-1)) e_b)
      uint64_t v[4] = {0, 0, 0, 0};
      v[b >> 6] = 1ull << (b & 63);
      if (k == 0) {
        xo_advance(v);
      } else {
        apply_nib_host(t->nib[k - 1], v);
        apply_nib_host(t->nib[k - 1], v);
      }
      for (int w = 0; w < 4; w++)
        for (uint64_t x = v[w]; x; x &= x - 1)
          t->row[k][64 * w + __builtin_ctzll(x)][b >> 6] |= 1ull << (b & 63);
      uint64_t (*e)[4] = t->nib[k][b >> 2];
      const int bit = 1 << (b & 3);
      if (bit == 1) memset(e[0], 0, sizeof e[0]);
      for (int x = 0; x < bit; x++)
        for (int w = 0; w < 4; w++) e[bit + x][w] = e[x][w] ^ v[w];
    }
  }
  g_tables = t;
}

const Tables &tables() {
  std::call_once(g_tables_once, build_tables);
  return *g_tables;
}

// v = T^m v
void jump_host(uint64_t v[4], uint64_t m) {
  const Tables &t = tables();
  for (int k = 0; k < kPowers; k++)
    if ((m >> k) & 1) apply_nib_host(t.nib[k], v);
}

// Device copies of the tables (rows 512 KiB, nibbles 352 KiB as [nibble][word]
// [value] so that a word's 16 values lie in 16 banks), one per device, made on
// the first fill on that device and kept until exit.
std::mutex g_dev_mu;
uint64_t *g_dev_tables[64] = {nullptr};

cudaError_t device_tables(uint64_t **out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_dev_mu);
  if (!g_dev_tables[dev]) {
    const Tables &t = tables();
    std::vector<uint32_t> nib((size_t)(kNibHi - kNibLo + 1) * kNibWords);
    for (int k = kNibLo; k <= kNibHi; k++)
      for (int i = 0; i < 64; i++)
        for (int x = 0; x < 16; x++)
          for (int w = 0; w < 8; w++)
            nib[(size_t)(k - kNibLo) * kNibWords + (i * 8 + w) * 16 + x] =
                (uint32_t)(t.nib[k][i][x][w >> 1] >> (32 * (w & 1)));
    uint64_t *p = nullptr;
    const size_t rows = kRowWords64 * sizeof(uint64_t), nibs = nib.size() * sizeof(uint32_t);
    if ((e = dev_malloc((void **)&p, rows + nibs)) != cudaSuccess) return e;
    if ((e = cudaMemcpy(p, t.row, rows, cudaMemcpyHostToDevice)) != cudaSuccess ||
        (e = cudaMemcpy((char *)p + rows, nib.data(), nibs, cudaMemcpyHostToDevice)) !=
            cudaSuccess) {
      cudaFree(p);
      return e;
    }
    g_dev_tables[dev] = p;
  }
  *out = g_dev_tables[dev];
  return cudaSuccess;
}

// ---- numc's per-thread state -----------------------------------------------

// [word][lane], numc's layout
thread_local uint64_t t_state[4][4];
thread_local bool t_seeded = false;

uint64_t splitmix64(uint64_t *x) {
  uint64_t z = (*x += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

// 2^128 steps by xoshiro256's published jump polynomial (kernel.h:60-96).
void jump128(uint64_t s[4]) {
  static const uint64_t kJump[4] = {0x180ec6d33cfd0abaull, 0xd5a61266f0c9392cull,
                                    0xa9582618e03fc9aaull, 0x39abdc4529b1661cull};
  uint64_t acc[4] = {0, 0, 0, 0};
  for (int i = 0; i < 4; i++)
    for (int b = 0; b < 64; b++) {
      if ((kJump[i] >> b) & 1)
        for (int w = 0; w < 4; w++) acc[w] ^= s[w];
      xo_advance(s);
    }
  memcpy(s, acc, sizeof acc);
}

// prng_seed (kernel.h:100-121): lane 0 from splitmix64, lanes 1-3 jumped.
void seed_state(uint64_t seed) {
  uint64_t base[4];
  for (int w = 0; w < 4; w++) base[w] = splitmix64(&seed);
  for (int w = 0; w < 4; w++) t_state[w][0] = base[w];
  for (int l = 1; l < 4; l++) {
    jump128(base);
    for (int w = 0; w < 4; w++) t_state[w][l] = base[w];
  }
  t_seeded = true;
}

void ensure_seeded() {
  if (!t_seeded) seed_state(0xdeadbeefcafe1234ull);   // numc's default (kernel.h:123-126)
}

// numc's OpenMP maximum thread count (omp_get_max_threads()): 0 = not set,
// taken from OMP_NUM_THREADS or the online CPU count on first use.
std::atomic<int> g_threads{0};

int default_threads() {
  if (const char *e = getenv("OMP_NUM_THREADS")) {
    const int v = atoi(e);   // first entry of a nesting list
    if (v > 0) return v;
  }
  const long c = sysconf(_SC_NPROCESSORS_ONLN);
  return c > 0 ? (int)c : 1;
}

// ---- the fill kernel -------------------------------------------------------

constexpr int kThreads = 256, kWarps = kThreads / 32;

struct RandArgs {
  uint64_t base[4][4];     // [stream][word]: the four lanes (small fill), lane 0 (large)
  int64_t n;               // elements
  int64_t chunk;           // elements per numc thread (large fill)
  int64_t blocks_per_seg;  // blocks per numc thread's chunk (or the whole fill)
  int logr;                // log2 steps of a run
  void *out;
};

// Raw 64-bit output to the stored bits: integers keep the low bits;
// float32 (raw >> 41 | 0x3F800000) - 1, float64 (raw >> 11 | 0x3FF0...) - 1
// (random.c:28-39, kernel.h:200-212), both exact.
template <typename U, int KIND>
__device__ __forceinline__ U convert(uint64_t raw) {
  if constexpr (KIND == 1) {
    const float v = __fsub_rn(__uint_as_float((uint32_t)(raw >> 41) | 0x3F800000u), 1.0f);
    return (U)__float_as_uint(v);
  } else if constexpr (KIND == 2) {
    const double v =
        __dsub_rn(__longlong_as_double((long long)((raw >> 11) | 0x3FF0000000000000ull)), 1.0);
    return (U)__double_as_longlong(v);
  } else {
    return (U)raw;
  }
}

// Staging row of one lane: 4 outputs a step packed into sizeof(U) words.
template <typename U>
__device__ __forceinline__ void stage_step(uint32_t *wp, const U (&o)[4]) {
  if constexpr (sizeof(U) == 1) {
    wp[0] = (uint32_t)o[0] | ((uint32_t)o[1] << 8) | ((uint32_t)o[2] << 16) | ((uint32_t)o[3] << 24);
  } else if constexpr (sizeof(U) == 2) {
    *reinterpret_cast<uint2 *>(wp) =
        make_uint2((uint32_t)o[0] | ((uint32_t)o[1] << 16), (uint32_t)o[2] | ((uint32_t)o[3] << 16));
  } else if constexpr (sizeof(U) == 4) {
    *reinterpret_cast<uint4 *>(wp) = make_uint4(o[0], o[1], o[2], o[3]);
  } else {
    reinterpret_cast<uint4 *>(wp)[0] = make_uint4((uint32_t)o[0], (uint32_t)((uint64_t)o[0] >> 32),
                                                  (uint32_t)o[1], (uint32_t)((uint64_t)o[1] >> 32));
    reinterpret_cast<uint4 *>(wp)[1] = make_uint4((uint32_t)o[2], (uint32_t)((uint64_t)o[2] >> 32),
                                                  (uint32_t)o[3], (uint32_t)((uint64_t)o[3] >> 32));
  }
}

// Shared memory: two nibble tables (later the output stage), the states.
constexpr int kSmemBytes = 2 * kNibWords * 4 + 8 * kThreads * 4;

// NV = 4: the four lanes of a small fill, thread = run x 4 + lane; NV = 1: lane
// 0 of a large fill, thread = run.
template <typename U, int KIND, int NV>
__global__ void __launch_bounds__(kThreads)
rand_fill_kernel(const __grid_constant__ RandArgs a, const uint64_t *__restrict__ rows) {
  constexpr int kRuns = kThreads / NV;                       // of a block
  constexpr int kLogRuns = NV == 1 ? 8 : 6;
  extern __shared__ __align__(16) uint32_t smem[];
  uint32_t *tab = smem;                                      // [2][64][8][16]
  uint32_t(*st)[kThreads] = reinterpret_cast<uint32_t(*)[kThreads]>(smem + 2 * kNibWords);
  __shared__ uint32_t jump[2][NV][8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t seg = blockIdx.x / a.blocks_per_seg, lb = blockIdx.x % a.blocks_per_seg;
  const int64_t start = NV == 1 ? seg * a.chunk : 0;
  const int64_t len = NV == 1 ? min(a.chunk, a.n - start) : a.n;
  if (len <= 0) return;
  const int64_t J = len / 4, R = (int64_t)1 << a.logr;
  const int tail = (int)(len % 4);
  const int64_t jb = lb * kRuns * R;                         // the block's first step
  if (lb > 0 && jb >= J) return;   // block 0 of a chunk always runs (it may own only the tail)

  const uint32_t *nibs = reinterpret_cast<const uint32_t *>(rows + kRowWords64);
  auto fetch = [&](int k) {   // nibble table of T^(2^(logr + k))
    const uint32_t *src = nibs + (size_t)(a.logr + k - kNibLo) * kNibWords;
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(tab + (k & 1) * kNibWords);
    for (int i = tid * 4; i < kNibWords; i += kThreads * 4)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * 4), "l"(src + i));
    asm volatile("cp.async.commit_group;");
  };
  fetch(0);
  fetch(1);

  // T^(start + jb) of each stream: thread r owns row r; four powers' rows are
  // in flight at a time
  if (tid < NV * 8) jump[0][tid / 8][tid & 7] = (uint32_t)(a.base[tid / 8][(tid & 7) >> 1] >> (32 * (tid & 1)));
#pragma unroll
  for (int w = 0; w < 8; w++) st[w][tid] = 0;
  __syncthreads();
  uint64_t m = (uint64_t)(start + jb);
  int cur = 0;
  while (m) {
    ulonglong2 r[4][2];
    int cnt = 0;
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (m) {
        const int k = __ffsll((long long)m) - 1;
        m &= m - 1;
        const ulonglong2 *p = reinterpret_cast<const ulonglong2 *>(rows + ((size_t)k * 256 + tid) * 4);
        r[i][0] = p[0];
        r[i][1] = p[1];
        cnt++;
      }
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (i < cnt) {
#pragma unroll
        for (int q = 0; q < NV; q++) {
          const uint32_t *x = jump[cur][q];
          const uint32_t t = ((uint32_t)r[i][0].x & x[0]) ^ ((uint32_t)(r[i][0].x >> 32) & x[1]) ^
                             ((uint32_t)r[i][0].y & x[2]) ^ ((uint32_t)(r[i][0].y >> 32) & x[3]) ^
                             ((uint32_t)r[i][1].x & x[4]) ^ ((uint32_t)(r[i][1].x >> 32) & x[5]) ^
                             ((uint32_t)r[i][1].y & x[6]) ^ ((uint32_t)(r[i][1].y >> 32) & x[7]);
          const uint32_t word = __ballot_sync(0xffffffffu, __popc(t) & 1);
          if (lane == 0) jump[cur ^ 1][q][warp] = word;
        }
        cur ^= 1;
        __syncthreads();
      }
  }
  if (tid < NV * 8) st[tid & 7][tid / 8] = jump[cur][tid / 8][tid & 7];

  // Doubling: warp g looks up word g's eight nibbles of every state.
  for (int k = 0; k < kLogRuns; k++) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const uint32_t *t = tab + (k & 1) * kNibWords + warp * 8 * 8 * 16;
    const int count = NV << k;
    for (int i = lane; i < count; i += 32) {
      const uint32_t x = st[warp][i];
      uint32_t y[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
      for (int j = 0; j < 8; j++)
#pragma unroll
        for (int w = 0; w < 8; w++) y[w] ^= t[(j * 8 + w) * 16 + ((x >> (4 * j)) & 15)];
#pragma unroll
      for (int w = 0; w < 8; w++) atomicXor(&st[w][count + i], y[w]);
    }
    __syncthreads();   // everyone is done with this table
    if (k + 2 < kLogRuns) fetch(k + 2);
    else asm volatile("cp.async.commit_group;");
  }
  uint64_t s[4];
#pragma unroll
  for (int w = 0; w < 4; w++) s[w] = (uint64_t)st[2 * w][tid] | (uint64_t)st[2 * w + 1][tid] << 32;

  // Runs.  A warp stages 4 KiB at a time, 32 rows of 128 bytes: a row of each of
  // 32 runs (NV = 1, 16-byte skew a row) or four rows of each of 8 runs (16-byte
  // skew a run).
  constexpr int kStage = NV == 1 ? 32 / (int)sizeof(U) : 128 / (int)sizeof(U);   // steps
  constexpr int kRowElems = 128 / (int)sizeof(U);
  const int64_t jw = jb + (int64_t)warp * (kRuns / kWarps) * R;   // the warp's first step
  const int64_t j0 = jb + (int64_t)(tid / NV) * R, j1 = min(j0 + R, J);
  const int mysteps = (int)max((int64_t)0, j1 - j0);
  U *out = (U *)a.out + start;
  const bool vec16 = ((uintptr_t)out & 15) == 0;
  const bool full = jw + (kRuns / kWarps) * R <= J;
  uint32_t *stage = smem + warp * 32 * 36;
  auto row_ptr = [&](int q) { return stage + (NV == 1 ? q * 36 : (q >> 2) * 132 + (q & 3) * 32); };
  // first element of row q in pass c
  auto row_elem = [&](int q, int c) {
    return NV == 1 ? 4 * (jw + q * R) + (int64_t)c * kRowElems
                   : 4 * (jw + (q >> 2) * R) + (int64_t)(4 * c + (q & 3)) * kRowElems;
  };
  U win[3];
  if (NV == 1) {
#pragma unroll
    for (int l = 0; l < 3; l++) {
      win[l] = convert<U, KIND>(xo_output(s));
      xo_advance(s);
    }
  }
  for (int c = 0; c < R / kStage; c++) {
    const int nv = min(kStage, mysteps - c * kStage);
#pragma unroll(NV == 1 ? kStage : 8)
    for (int i = 0; i < kStage; i++) {
      if (i < nv) {
        const U o = convert<U, KIND>(xo_output(s));
        xo_advance(s);
        if (NV == 1) {
          const U v[4] = {win[0], win[1], win[2], o};
          stage_step<U>(row_ptr(lane) + i * (int)sizeof(U), v);
          win[0] = win[1];
          win[1] = win[2];
          win[2] = o;
        } else {
          reinterpret_cast<U *>(row_ptr(lane & ~3))[4 * i + (lane & 3)] = o;
        }
      }
    }
    __syncwarp();
    if (vec16 && full) {
      // every row complete: 8 lanes a row (16 bytes each), 4 rows a pass
#pragma unroll
      for (int p = 0; p < 8; p++) {
        const int q = 4 * p + (lane >> 3);
        *reinterpret_cast<uint4 *>(reinterpret_cast<char *>(out + row_elem(q, c)) + 16 * (lane & 7)) =
            *reinterpret_cast<const uint4 *>(row_ptr(q) + 4 * (lane & 7));
      }
    } else if (vec16) {
#pragma unroll 2
      for (int p = 0; p < 8; p++) {
        const int q = 4 * p + (lane >> 3), at = kRowElems / 8 * (lane & 7);
        const int64_t e0 = row_elem(q, c) + at, ne = min((int64_t)kRowElems / 8, 4 * J - e0);
        const uint32_t *src = row_ptr(q) + 4 * (lane & 7);
        if (ne == kRowElems / 8) {
          *reinterpret_cast<uint4 *>(out + e0) = *reinterpret_cast<const uint4 *>(src);
        } else {
          for (int e = 0; e < ne; e++) out[e0 + e] = reinterpret_cast<const U *>(src)[e];
        }
      }
    } else {
      for (int q = 0; q < 32; q++) {
        const int64_t e0 = row_elem(q, c), ne = min((int64_t)kRowElems, 4 * J - e0);
        const U *src = reinterpret_cast<const U *>(row_ptr(q));
        for (int e = lane; e < ne; e += 32) out[e0 + e] = src[e];
      }
    }
    __syncwarp();
  }
  // The chunk's tail continues stream 0 from step J (in the large fill the
  // window then holds X(start + J .. start + J + 2)).
  if (tail && (NV == 1 || (tid & 3) == 0) &&
      ((J == 0 && lb == 0 && tid == 0) || (j0 < J && j1 == J))) {
    for (int r = 0; r < tail; r++) {
      if (NV == 1) {
        out[4 * J + r] = win[r];
      } else {
        out[4 * J + r] = convert<U, KIND>(xo_output(s));
        xo_advance(s);
      }
    }
  }
}

template <typename U, int KIND>
cudaError_t launch_fill(const RandArgs &a, bool large, unsigned blocks, const uint64_t *rows,
                        cudaStream_t s) {
  static LaunchCache lc[2];
  auto kern = large ? rand_fill_kernel<U, KIND, 1> : rand_fill_kernel<U, KIND, 4>;
  cudaError_t e = smem_attr_once(lc[large], (const void *)kern, kSmemBytes);
  if (e) return e;
  kern<<<blocks, kThreads, kSmemBytes, s>>>(a, rows);
  count_launch();
  return cudaGetLastError();
}

}  // namespace

void rand_seed(uint64_t seed) { seed_state(seed); }

int rand_threads() {
  int t = g_threads.load();
  if (t <= 0) {
    t = default_threads();
    int expect = 0;
    g_threads.compare_exchange_strong(expect, t);
    t = g_threads.load();
  }
  return t;
}

void rand_set_threads(int threads) { g_threads.store(threads > 0 ? threads : 0); }

cudaError_t rand_fill(NumcDType dt, void *out, size_t n, cudaStream_t s) {
  ensure_seeded();
  if (n == 0) return cudaSuccess;
  uint64_t *tabs = nullptr;
  cudaError_t e = device_tables(&tabs);
  if (e != cudaSuccess) return e;
  const size_t size = numc_dtype_size(dt);
  const size_t bytes = n * size;
  RandArgs a;
  memset(&a, 0, sizeof a);
  a.n = (int64_t)n;
  a.out = out;
  bool large;
  int64_t per_seg_steps, nseg;
  if (bytes <= (1u << 20)) {        // NUMC_OMP_BYTE_THRESHOLD
    large = false;
    for (int q = 0; q < 4; q++)
      for (int w = 0; w < 4; w++) a.base[q][w] = t_state[w][q];
    nseg = 1;
    per_seg_steps = (int64_t)n / 4;
    // a run fills whole 128-byte rows of its four lanes' outputs
    a.logr = size == 1 ? 7 : size == 2 ? 6 : 5;
  } else {
    int64_t T = (int64_t)(bytes / (1u << 19));   // NUMC_OMP_BYTES_PER_THREAD
    T = std::min<int64_t>(T, rand_threads());
    if (T < 1) T = 1;
    large = true;
    for (int w = 0; w < 4; w++) a.base[0][w] = t_state[w][0];
    a.chunk = ((int64_t)n + T - 1) / T;
    nseg = T;
    per_seg_steps = a.chunk / 4;
    // The longest runs that still give half of the multiprocessors a block (a
    // block's start costs it as much as some 100 steps).  64 Mi float32, runs
    // of 256, 128, 64: 57, 66, 78 us; 16 Mi, 128, 64, 32: 23, 27, 38 us.
    a.logr = kNibHi - 7;
    while (a.logr > 5 && (((int64_t)n / 4) >> (a.logr + 8)) * 2 < sm_count()) a.logr--;
  }
  const int64_t steps_per_block = (int64_t)(large ? kThreads : kThreads / 4) << a.logr;
  a.blocks_per_seg = std::max<int64_t>(1, (per_seg_steps + steps_per_block - 1) / steps_per_block);
  const int64_t blocks = nseg * a.blocks_per_seg;
  if (blocks > 0x7FFFFFFFll) return cudaErrorInvalidConfiguration;
  switch (dt) {
  case NUMC_DTYPE_INT8: case NUMC_DTYPE_UINT8: e = launch_fill<uint8_t, 0>(a, large, (unsigned)blocks, tabs, s); break;
  case NUMC_DTYPE_INT16: case NUMC_DTYPE_UINT16: e = launch_fill<uint16_t, 0>(a, large, (unsigned)blocks, tabs, s); break;
  case NUMC_DTYPE_INT32: case NUMC_DTYPE_UINT32: e = launch_fill<uint32_t, 0>(a, large, (unsigned)blocks, tabs, s); break;
  case NUMC_DTYPE_INT64: case NUMC_DTYPE_UINT64: e = launch_fill<uint64_t, 0>(a, large, (unsigned)blocks, tabs, s); break;
  case NUMC_DTYPE_FLOAT32: e = launch_fill<uint32_t, 1>(a, large, (unsigned)blocks, tabs, s); break;
  case NUMC_DTYPE_FLOAT64: e = launch_fill<uint64_t, 2>(a, large, (unsigned)blocks, tabs, s); break;
  default: return cudaErrorInvalidValue;
  }
  if (e != cudaSuccess) return e;
  // numc's state after the fill: the small path moves every lane n/4 steps
  // and lane 0 n%4 more; the large path moves every lane n steps.
  for (int l = 0; l < 4; l++) {
    uint64_t v[4];
    for (int w = 0; w < 4; w++) v[w] = t_state[w][l];
    if (large) {
      jump_host(v, n);
    } else {
      jump_host(v, n / 4);
      if (l == 0)
        for (size_t r = 0; r < n % 4; r++) xo_advance(v);
    }
    for (int w = 0; w < 4; w++) t_state[w][l] = v[w];
  }
  return cudaSuccess;
}

}  // namespace numc_k

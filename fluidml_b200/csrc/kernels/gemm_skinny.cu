// Skinny GEMM: C[M, N] = A[M, K] * B[K, N] for M <= 32 (the pooler, batch-1 classifier heads,
// VGG's fully connected layers at batch 1).  With so few rows the product is a stream over the
// weights: HBM-bound on B (K*N*4 bytes read once), CUDA-core FMAs in fp32, no tensor cores.
//
//   K-major B (b_sk == 1, e.g. Gemm with transB: weights stored [N, K]):
//       one warp per output column walks its K slice with 16-byte loads (lane-contiguous in
//       k), keeps M partial sums per lane and reduces them with shuffles;
//   N-major B (b_sn == 1, e.g. MatMul with weights stored [K, N]) and any other strides:
//       one thread per output column (lane-contiguous in n) and k phase, A values broadcast from
//       shared memory (gemm_skinny_rows_kernel).
//
// K is split over gridDim.y so that the grid covers the machine.  Each split writes its
// partial [M, tile] block to scratch memory; the split that arrives last on the tile's
// counter adds the partials in split order (results do not depend on arrival order), applies
// the epilogue and resets the counter.  The scratch (counters first, then partials) is global
// memory beyond the inputs and outputs, owned by the library per (device, stream).
#include "gemm_common.cuh"
#include <cmath>
#include <map>
#include <mutex>
#include <utility>

namespace fml {
namespace {

constexpr int kMaxM = 32;
constexpr int kColsPerCta = 32;  // output columns per CTA
constexpr int kThreads = 256;
constexpr size_t kCounterBytes = 64 << 10;  // 16384 tile counters

struct SkinnyArgs {
  GemmProblem p;
  GemmEpilogue e;
  int splits, tiles_n;
  int64_t k_per_split;
  unsigned *counters;  // one per (batch, n tile)
  float *partials;     // [batch * tiles_n][splits][M][kColsPerCta]
};

// Arrival of one split's partial sums at a tile; true in the CTA that is to finish the tile.
__device__ __forceinline__ bool last_split(const SkinnyArgs &a, int64_t tile_id, int *flag) {
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) *flag = atomicAdd(a.counters + tile_id, 1u) == (unsigned)a.splits - 1u;
  __syncthreads();
  if (!*flag) return false;
  __threadfence();
  return true;
}

// K-major B.  ROWS 4 and 8: 16-byte-aligned operands, rows in groups of that many (4: at most four rows in
// all, classifier heads and poolers at batch 1 to 4).  These hold only their own path's registers (the
// general path's 32 accumulators per lane made a shared kernel 176 registers = one CTA per SM = 12 %
// occupancy, and a 411 MB weight matrix streamed at 48 % of DRAM's cycles), so two or three CTAs share
// an SM.  ROWS 0: anything else.
template <int ROWS>
__global__ void __launch_bounds__(kThreads, ROWS == 4 ? 3 : ROWS == 8 ? 2 : 1) gemm_skinny_kernel(SkinnyArgs a) {
  constexpr bool FEW = ROWS != 0;
  constexpr int R = FEW ? ROWS : 1;
  pdl_launch_dependents();
  // B is what this kernel streams; while the preceding kernel drains, start it towards L2
  l2_prefetch_span(a.p.b, ((a.p.K - 1) * a.p.b_sk + (a.p.N - 1) * a.p.b_sn + 1) * (int64_t)sizeof(float), 4 << 20);
  pdl_wait();
  __shared__ float red[kMaxM][kColsPerCta];
  __shared__ int last_flag;
  const int M = (int)a.p.M;
  const int tile = blockIdx.x, split = blockIdx.y, z = blockIdx.z;
  const int64_t z0 = z % a.p.nb0, z1 = z / a.p.nb0;
  const float *A = a.p.a + z0 * a.p.a_b0 + z1 * a.p.a_b1;
  const float *B = a.p.b + z0 * a.p.b_b0 + z1 * a.p.b_b1;
  const int64_t n0 = (int64_t)tile * kColsPerCta;
  const int64_t k0 = (int64_t)split * a.k_per_split, k1 = min(a.p.K, k0 + a.k_per_split);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

  {
    // warp w owns columns n0 + w, n0 + w + 8, ... ; lanes stride over k in float4 steps
    const bool vec = a.p.a_sk == 1 && (a.p.a_sm & 3) == 0 && (a.p.b_sn & 3) == 0 && (k0 & 3) == 0 &&
                     ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15) == 0;
    // The warp takes its four columns at once, so that eight weight loads are in flight per lane, the
    // row chunks are loaded once for all four columns, and the shuffle reductions are amortised.  Same
    // per-lane summation order as the general loop below.  (Row groups after the first find the
    // columns in L1 or L2: 5 x 1280 x 1000 took 44 us with a column and 32 predicated rows at a time.)
    for (int g = 0; FEW && g < (ROWS == 4 ? 1 : M); g += R) {  // the launcher checks `vec` before it picks these instantiations
      const int rows = ROWS == 4 ? M : min(R, M - g);
      const float *Ag = A + (int64_t)g * a.p.a_sm;
      const int64_t kv = k0 + ((k1 - k0) & ~(int64_t)3);
      float acc4[4][R];
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int m = 0; m < R; ++m) acc4[j][m] = 0.0f;
      // columns past the edge of a ragged tile read the last column again (their sums are dropped below)
      const float *bcol[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) bcol[j] = B + min(n0 + warp * 4 + j, a.p.N - 1) * a.p.b_sn;
      auto dot4 = [](float4 x, float4 y, float t) { return fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, t)))); };
      auto weights4 = [](const float *x) { return R == 4 ? __ldcs(reinterpret_cast<const float4 *>(x)) : *reinterpret_cast<const float4 *>(x); };
      int64_t k = k0 + lane * 4;
      for (; k + 128 < kv; k += 256) {
        float4 bw[4][2];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          bw[j][0] = weights4(bcol[j] + k);
          bw[j][1] = weights4(bcol[j] + k + 128);
        }
#pragma unroll
        for (int m = 0; m < R; ++m)
          if (m < rows) {
            const float4 a0 = *reinterpret_cast<const float4 *>(Ag + m * a.p.a_sm + k);
            const float4 a1 = *reinterpret_cast<const float4 *>(Ag + m * a.p.a_sm + k + 128);
#pragma unroll
            for (int j = 0; j < 4; ++j) acc4[j][m] = dot4(a1, bw[j][1], dot4(a0, bw[j][0], acc4[j][m]));
          }
      }
      for (; k < kv; k += 128) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 bv = weights4(bcol[j] + k);
#pragma unroll
          for (int m = 0; m < R; ++m)
            if (m < rows) acc4[j][m] = dot4(*reinterpret_cast<const float4 *>(Ag + m * a.p.a_sm + k), bv, acc4[j][m]);
        }
      }
      for (int64_t kt = kv + lane; kt < k1; kt += 32)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float bv = bcol[j][kt];
#pragma unroll
          for (int m = 0; m < R; ++m)
            if (m < rows) acc4[j][m] = fmaf(Ag[m * a.p.a_sm + kt], bv, acc4[j][m]);
        }
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int m = 0; m < R; ++m)
          if (m < rows) {
            float v = acc4[j][m];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) red[g + m][warp * 4 + j] = v;
          }
    }
    for (int c = FEW ? kColsPerCta : warp; c < kColsPerCta; c += kThreads / 32) {
      const int64_t n = n0 + c;
      float acc[kMaxM];
#pragma unroll
      for (int m = 0; m < kMaxM; ++m) acc[m] = 0.0f;
      if (n < a.p.N) {
        const float *brow = B + n * a.p.b_sn;
        if (vec) {
          const int64_t kv = k0 + ((k1 - k0) & ~(int64_t)3);
          int64_t k = k0 + lane * 4;
          // four independent 16-byte weight loads per lane and step: the kernel lives on memory-
          // level parallelism (weights are read once: streaming loads that do not pollute L1)
          for (; k + 384 < kv; k += 512) {
            const float4 b0 = __ldcs(reinterpret_cast<const float4 *>(brow + k));
            const float4 b1 = __ldcs(reinterpret_cast<const float4 *>(brow + k + 128));
            const float4 b2 = __ldcs(reinterpret_cast<const float4 *>(brow + k + 256));
            const float4 b3 = __ldcs(reinterpret_cast<const float4 *>(brow + k + 384));
#pragma unroll
            for (int m = 0; m < kMaxM; ++m)
              if (m < M) {
                const float *ap = A + m * a.p.a_sm + k;
                const float4 a0 = *reinterpret_cast<const float4 *>(ap), a1 = *reinterpret_cast<const float4 *>(ap + 128);
                const float4 a2 = *reinterpret_cast<const float4 *>(ap + 256), a3 = *reinterpret_cast<const float4 *>(ap + 384);
                float t = acc[m];
                t = fmaf(a0.x, b0.x, fmaf(a0.y, b0.y, fmaf(a0.z, b0.z, fmaf(a0.w, b0.w, t))));
                t = fmaf(a1.x, b1.x, fmaf(a1.y, b1.y, fmaf(a1.z, b1.z, fmaf(a1.w, b1.w, t))));
                t = fmaf(a2.x, b2.x, fmaf(a2.y, b2.y, fmaf(a2.z, b2.z, fmaf(a2.w, b2.w, t))));
                acc[m] = fmaf(a3.x, b3.x, fmaf(a3.y, b3.y, fmaf(a3.z, b3.z, fmaf(a3.w, b3.w, t))));
              }
          }
          for (; k < kv; k += 128) {
            const float4 bv = __ldcs(reinterpret_cast<const float4 *>(brow + k));
#pragma unroll
            for (int m = 0; m < kMaxM; ++m)
              if (m < M) {
                const float4 av = *reinterpret_cast<const float4 *>(A + m * a.p.a_sm + k);
                acc[m] = fmaf(av.x, bv.x, fmaf(av.y, bv.y, fmaf(av.z, bv.z, fmaf(av.w, bv.w, acc[m]))));
              }
          }
          for (int64_t k = kv + lane; k < k1; k += 32) {
            const float bv = brow[k];
#pragma unroll
            for (int m = 0; m < kMaxM; ++m)
              if (m < M) acc[m] = fmaf(A[m * a.p.a_sm + k], bv, acc[m]);
          }
        } else {
          for (int64_t k = k0 + lane; k < k1; k += 32) {
            const float bv = brow[k * a.p.b_sk];
#pragma unroll
            for (int m = 0; m < kMaxM; ++m)
              if (m < M) acc[m] = fmaf(A[m * a.p.a_sm + k * a.p.a_sk], bv, acc[m]);
          }
        }
      }
#pragma unroll
      for (int m = 0; m < kMaxM; ++m)
        if (m < M) {
          float v = acc[m];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
          if (lane == 0) red[m][c] = v;
        }
    }
  }
  __syncthreads();

  // red[m][c] = this split's partial sums.  Single split: finish directly.
  float *C = a.p.c + z0 * a.p.c_b0 + z1 * a.p.c_b1;
  const float *bias = a.p.bias ? a.p.bias + z0 * a.p.bias_b0 + z1 * a.p.bias_b1 : nullptr;
  const float *res = a.p.res ? a.p.res + z0 * a.p.res_b0 + z1 * a.p.res_b1 : nullptr;
  const int64_t tile_id = (int64_t)z * a.tiles_n + tile;
  if (a.splits > 1) {
    float *part = a.partials + ((tile_id * a.splits + split) * M) * kColsPerCta;
    for (int i = threadIdx.x; i < M * kColsPerCta; i += kThreads) part[i] = red[i / kColsPerCta][i % kColsPerCta];
    if (!last_split(a, tile_id, &last_flag)) return;
  }
  for (int i = threadIdx.x; i < M * kColsPerCta; i += kThreads) {
    const int m = i / kColsPerCta, c = i % kColsPerCta;
    const int64_t n = n0 + c;
    if (n >= a.p.N) continue;
    float acc;
    if (a.splits > 1) {
      acc = 0.0f;
      const float *base = a.partials + (tile_id * a.splits * M) * kColsPerCta + i;
      for (int sp = 0; sp < a.splits; ++sp) acc += __ldcg(base + (int64_t)sp * M * kColsPerCta);
    } else {
      acc = red[m][c];
    }
    const float bv = bias ? bias[m * a.p.bias_sm + n * a.p.bias_sn] : 0.0f;
    const float rv = res ? res[m * a.p.res_sm + n * a.p.res_sn] : 0.0f;
    C[m * a.p.c_sm + n * a.p.c_sn] = gemm_epilogue(a.e, acc, bv, rv);
  }
  if (a.splits > 1 && threadIdx.x == 0) a.counters[tile_id] = 0u;  // ready for the next launch
}

// N-major B: thread (c, kq) takes column n0 + c and every 8th k of the slice, for MR rows (M rounded up), in
// chunks of 128 k.  What bounds the small ones (16 rows, K and N of a few hundred) is the chain of latencies
// after the preceding kernel, so constant weights of the first chunk are in registers before the wait for
// it, each later chunk's are loaded under the products of the one before, bias and residual are fetched
// ahead, A is stored [k][row] (one 16-byte broadcast per four products), and the eight k phases are added
// up behind one barrier.
// Measured in a graph of such launches, before -> now: 16 x 128 x 384 10.9 -> 3.6 us, 31 x 768 x 3072
// 27.0 -> 19.1 us, 8 x 4096 x 1024 33.9 -> 11.7 us, 1 x 25088 x 4096 506 -> 113 us.
template <int MR>
__global__ void __launch_bounds__(kThreads, MR == 32 ? 1 : 2) gemm_skinny_rows_kernel(SkinnyArgs a) {
  constexpr int kChunk = 128, kPhases = kThreads / 32, kLoads = kChunk / kPhases, kPitch = MR + 4;
  constexpr int kItems = (MR * kColsPerCta + kThreads - 1) / kThreads;  // outputs per thread
  __shared__ __align__(16) float sh[kPhases * MR * kColsPerCta];         // A chunk, later the phases' sums
  __shared__ int last_flag;
  pdl_launch_dependents();
  const int M = (int)a.p.M;
  const int tile = blockIdx.x, split = blockIdx.y, z = blockIdx.z;
  const int64_t z0 = z % a.p.nb0, z1 = z / a.p.nb0;
  const float *A = a.p.a + z0 * a.p.a_b0 + z1 * a.p.a_b1;
  const int64_t n0 = (int64_t)tile * kColsPerCta;
  const int64_t k0 = (int64_t)split * a.k_per_split, k1 = min(a.p.K, k0 + a.k_per_split);
  const int c = threadIdx.x & 31, kq = threadIdx.x >> 5;
  const bool col = n0 + c < a.p.N;
  const float *B = a.p.b + z0 * a.p.b_b0 + z1 * a.p.b_b1 + (n0 + c) * a.p.b_sn;
  float w[kLoads];
  auto load = [&](int64_t kc) {
#pragma unroll
    for (int i = 0; i < kLoads; ++i) {
      const int64_t k = kc + kq + i * kPhases;
      w[i] = col && k < k1 ? __ldcs(B + k * a.p.b_sk) : 0.0f;
    }
  };
  if (a.p.b_constant) load(k0);
  l2_prefetch_span(a.p.b, ((a.p.K - 1) * a.p.b_sk + (a.p.N - 1) * a.p.b_sn + 1) * (int64_t)sizeof(float), 4 << 20);
  pdl_wait();
  if (!a.p.b_constant) load(k0);
  const float *bias = a.p.bias ? a.p.bias + z0 * a.p.bias_b0 + z1 * a.p.bias_b1 : nullptr;
  const float *res = a.p.res ? a.p.res + z0 * a.p.res_b0 + z1 * a.p.res_b1 : nullptr;
  float bv[kItems], rv[kItems];
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    const int m = kq + j * kPhases;  // (output items: row m, column c)
    const bool in = col && m < M;
    bv[j] = bias && in ? bias[m * a.p.bias_sm + (n0 + c) * a.p.bias_sn] : 0.0f;
    rv[j] = res && in ? res[m * a.p.res_sm + (n0 + c) * a.p.res_sn] : 0.0f;
  }
  float acc[MR];
#pragma unroll
  for (int m = 0; m < MR; ++m) acc[m] = 0.0f;
  for (int64_t kc = k0; kc < k1; kc += kChunk) {
    float x[MR * kChunk / kThreads];
    const int kk = threadIdx.x & (kChunk - 1), m_first = threadIdx.x / kChunk;
#pragma unroll
    for (int i = 0; i < MR * kChunk / kThreads; ++i) {
      const int m = m_first + i * (kThreads / kChunk);
      x[i] = m < M && kc + kk < k1 ? A[m * a.p.a_sm + (kc + kk) * a.p.a_sk] : 0.0f;
    }
    if (kc > k0) __syncthreads();  // the chunk before has been read
#pragma unroll
    for (int i = 0; i < MR * kChunk / kThreads; ++i) sh[kk * kPitch + m_first + i * (kThreads / kChunk)] = x[i];
    __syncthreads();
    float u[kLoads];
#pragma unroll
    for (int i = 0; i < kLoads; ++i) u[i] = w[i];
    if (kc + kChunk < k1) load(kc + kChunk);
#pragma unroll
    for (int i = 0; i < kLoads; ++i)
#pragma unroll
      for (int m = 0; m < MR; m += 4) {
        const float4 v = *reinterpret_cast<const float4 *>(sh + (kq + i * kPhases) * kPitch + m);
        acc[m] = fmaf(v.x, u[i], acc[m]);
        acc[m + 1] = fmaf(v.y, u[i], acc[m + 1]);
        acc[m + 2] = fmaf(v.z, u[i], acc[m + 2]);
        acc[m + 3] = fmaf(v.w, u[i], acc[m + 3]);
      }
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < MR; ++m) sh[(kq * MR + m) * kColsPerCta + c] = acc[m];
  __syncthreads();
  float v[kItems];
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    const int m = kq + j * kPhases;
    v[j] = 0.0f;
    if (m < MR)
#pragma unroll
      for (int ph = 0; ph < kPhases; ++ph) v[j] += sh[(ph * MR + m) * kColsPerCta + c];
  }
  const int64_t tile_id = (int64_t)z * a.tiles_n + tile;
  if (a.splits > 1) {
    float *part = a.partials + (tile_id * a.splits * M) * kColsPerCta;
#pragma unroll
    for (int j = 0; j < kItems; ++j)
      if (kq + j * kPhases < M) part[((int64_t)split * M + kq + j * kPhases) * kColsPerCta + c] = v[j];
    if (!last_split(a, tile_id, &last_flag)) return;
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      const int m = kq + j * kPhases;
      v[j] = 0.0f;
      if (m < M)
#pragma unroll 8
        for (int sp = 0; sp < a.splits; ++sp) v[j] += __ldcg(part + ((int64_t)sp * M + m) * kColsPerCta + c);
    }
  }
  float *C = a.p.c + z0 * a.p.c_b0 + z1 * a.p.c_b1;
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    const int m = kq + j * kPhases;
    if (col && m < M) C[m * a.p.c_sm + (n0 + c) * a.p.c_sn] = gemm_epilogue(a.e, v[j], bv[j], rv[j]);
  }
  if (a.splits > 1 && threadIdx.x == 0) a.counters[tile_id] = 0u;  // ready for the next launch
}

// K-major B, without a second CTA on any output: a CTA has four columns, its eight warps share out the rows (`groups` of R)
// and, 8 / groups of them, alternate chunks of 128 k values, DEPTH chunks in flight (sixteen 16-byte weight loads per lane
// with few rows); the sums meet in shared memory.  A classifier head is then one memory round trip and one block barrier, where the slices
// above meet through scratch memory: fence, counter and a second pass over the partial sums, 3 to 4 us of a small launch,
// and 32 columns x 8 slices a CTA were too few bytes in flight (1 x 4096 x 1000: 1.1 TB/s).  Weights that no earlier
// launch writes are asked for before the dependency wait.
// Captured graphs, us, slices -> this: 1 x 4096 x 1000 12.3 (weights from HBM 14.8) -> 3.2 (4.3), 1 x 1280 x 1000 6.8 -> 2.7,
// 1 x 25088 x 4096 66 -> 65, 3 x 768 x 768 6.8 -> 2.6, 8 x 4096 x 4096 39 -> 29.  Every CTA reads all rows again and has
// fixed phases of its own, so wide and flat products lose (1 x 256 x 50304 12 -> 77): columns_pay.
constexpr int kCtaCols = 4;

template <int V> __device__ __forceinline__ void warp_reduce_scatter(float (&v)[V], int lane) {
  // V sums over the warp in V - 1 exchanges and what is left of five: lane l ends with sums l * V / 32 .. (V >= 32), or
  // l * V / 32 alone (V < 32: lanes share)
  int n = V;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    if (n > 1) {
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int i = 0; i < V / 2; ++i)
        if (i < n / 2) {
          const float keep = up ? v[i + n / 2] : v[i], send = up ? v[i] : v[i + n / 2];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      n >>= 1;
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
}

template <int R, int DEPTH>
__global__ void __launch_bounds__(kThreads, 2) gemm_skinny_columns_kernel(const GemmProblem p, const GemmEpilogue e, const int groups) {
  constexpr int COLS = kCtaCols, V = R * COLS;
  pdl_launch_dependents();
  __shared__ float red[kThreads / 32][V];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, per = (kThreads / 32) / groups;  // warps of a row group
  const int z = blockIdx.z, row0 = warp / per * R, M = min(R, (int)p.M - row0);                // this warp's rows
  const int64_t z0 = z % p.nb0, z1 = z / p.nb0, n0 = (int64_t)blockIdx.x * COLS;
  const float *const A = p.a + z0 * p.a_b0 + z1 * p.a_b1 + row0 * p.a_sm;
  const float *const B = p.b + z0 * p.b_b0 + z1 * p.b_b1;
  const int step = per * 32, quads = (int)(p.K >> 2);  // (K is a multiple of 4)
  const float4 *bcol[COLS];           // columns past the edge read the last one again
#pragma unroll
  for (int j = 0; j < COLS; ++j) bcol[j] = reinterpret_cast<const float4 *>(B + min(n0 + j, p.N - 1) * p.b_sn);
  float4 w[DEPTH][COLS];
  auto load = [&](int q0) {
#pragma unroll
    for (int u = 0; u < DEPTH; ++u) {
      const int q = q0 + u * step;
#pragma unroll
      for (int j = 0; j < COLS; ++j) w[u][j] = q < quads ? __ldcs(bcol[j] + q) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  int q0 = warp % per * 32 + lane;
  if (p.b_constant) load(q0);
  pdl_wait();
  if (!p.b_constant) load(q0);
  // what the last phase adds, asked for now: output i = row * COLS + column
  const int fj = threadIdx.x % COLS, fm = threadIdx.x / COLS;
  const bool last = fm < (int)p.M && n0 + fj < p.N;
  float bias = 0.0f, res = 0.0f;
  if (last && p.bias) bias = p.bias[z0 * p.bias_b0 + z1 * p.bias_b1 + fm * p.bias_sm + (n0 + fj) * p.bias_sn];
  if (last && p.res) res = p.res[z0 * p.res_b0 + z1 * p.res_b1 + fm * p.res_sm + (n0 + fj) * p.res_sn];
  float acc[V];
#pragma unroll
  for (int i = 0; i < V; ++i) acc[i] = 0.0f;
  for (; q0 < quads; q0 += DEPTH * step) {
#pragma unroll
    for (int u = 0; u < DEPTH; ++u) {
      const int q = q0 + u * step;
      if (q >= quads) break;
#pragma unroll
      for (int m = 0; m < R; ++m)
        if (m < M) {
          const float4 x = reinterpret_cast<const float4 *>(A + m * p.a_sm)[q];
#pragma unroll
          for (int j = 0; j < COLS; ++j) {
            float &t = acc[m * COLS + j];
            t = fmaf(x.x, w[u][j].x, fmaf(x.y, w[u][j].y, fmaf(x.z, w[u][j].z, fmaf(x.w, w[u][j].w, t))));
          }
        }
    }
    if (q0 + DEPTH * step < quads) load(q0 + DEPTH * step);
  }
  warp_reduce_scatter<V>(acc, lane);
  if (V >= 32) {
#pragma unroll
    for (int i = 0; i < (V + 31) / 32; ++i) red[warp][lane * (V / 32) + i] = acc[i];
  } else if (lane % (32 / (V < 32 ? V : 32)) == 0) {
    red[warp][lane * V / 32] = acc[0];
  }
  __syncthreads();
  if (!last) return;
  const int group = fm / R;
  float v = 0.0f;
  for (int k = 0; k < per; ++k) v += red[group * per + k][threadIdx.x - group * V];
  p.c[z0 * p.c_b0 + z1 * p.c_b1 + fm * p.c_sm + (n0 + fj) * p.c_sn] = gemm_epilogue(e, v, bias, res);
}

// Rows and columns of B on 16-byte boundaries, k in one sweep of a few batches.
bool columns_possible(const GemmProblem &p) {
  if (p.b_sk != 1 || p.b_sn == 1 || p.a_sk != 1 || p.K % 4 || p.K > (1 << 20)) return false;
  if (p.a_sm % 4 || p.b_sn % 4 || !aligned16(p.a) || !aligned16(p.b) || p.a_b0 % 4 || p.a_b1 % 4 || p.b_b0 % 4 || p.b_b1 % 4) return false;
  return p.N < (1ll << 31);
}

struct SkinnyPlan {
  int splits, tiles_n;
  int64_t k_per_split;
  size_t counter_bytes, scratch_bytes;  // scratch = counters (256-byte aligned) + partials
};

SkinnyPlan plan_skinny(const GemmProblem &p) {
  SkinnyPlan pl;
  pl.tiles_n = (int)((p.N + kColsPerCta - 1) / kColsPerCta);
  const int64_t tiles = (int64_t)pl.tiles_n * p.nb0 * p.nb1;
  // enough CTAs for ~8 per SM, each split at least 256 k values long
  int64_t s = (kSms * 8 + tiles - 1) / tiles;
  // (with at most four rows the kernel is a chain of load latencies, not arithmetic: slices of
  // 128 k values already pay there; more rows keep slices of at least 256)
  s = std::min<int64_t>(s, std::max<int64_t>(1, p.K / (p.M <= 4 ? 128 : 256)));
  s = std::max<int64_t>(1, std::min<int64_t>(s, 64));
  int64_t per = (p.K + s - 1) / s;
  per = (per + 127) / 128 * 128;  // keeps every slice start 16-byte aligned and chunked
  pl.k_per_split = per;
  pl.splits = (int)((p.K + per - 1) / per);
  // The counters live in a region of fixed size at the start of the scratch, so that partial
  // sums of one launch never land where a later launch of another shape keeps its counters
  // (they must read zero at launch).  Products with more tiles than counters run unsplit.
  if ((size_t)tiles * 4 > kCounterBytes) { pl.splits = 1; pl.k_per_split = p.K; }
  pl.counter_bytes = pl.splits > 1 ? kCounterBytes : 0;
  pl.scratch_bytes = pl.splits > 1 ? pl.counter_bytes + (size_t)tiles * pl.splits * p.M * kColsPerCta * 4 : 0;
  return pl;
}

// Times of the three kernels in microseconds: fixed phases, then waves of CTAs at the SMs' rate, not below the weights'
// bytes.  Fitted to captured graphs of 51 K-major shapes (K 256 to 8192, N 768 to 50304) and 61 N-major ones below 16 M
// multiply-adds (K 128 to 4096, N 128 to 4096), 1 to 31 rows each, warm.  Taking the kernel with the smaller time costs 2 %
// over taking the faster one (K-major: columns always 15 %, at worst 1 x 256 x 50304 77 us for 12; slices always 22 %) and
// 0.3 % (columns or N-major rows; columns always 11 %, at worst 31 x 4096 x 128 2.7 times).
double columns_us(double m, double n, double k, double batch) {
  const double per_k = m <= 4 ? 0.3 + 0.058 * m : m <= 8 ? 0.31 + 0.186 * m : 0.78 + 0.205 * (m <= 16 ? m : 32);  // (a group of sixteen rows, or two)
  const double waves = std::max(1.0, n / kCtaCols * batch / (2.0 * kSms));
  return std::max(0.76 + waves * (1.76 + per_k * k / 1024), n * k * batch * 4 / 6.4e6);
}
double slices_us(const GemmProblem &p, const SkinnyPlan &pl) {
  const double waves = (double)pl.tiles_n * pl.splits * (double)(p.nb0 * p.nb1) / ((p.M <= 4 ? 3.0 : 2.0) * kSms);
  const double work = 2.85 + 2.2 * (double)p.M * (double)pl.k_per_split / 1024;
  return 1.04 + (pl.splits > 1 ? 2.79 : 0.0) +
         std::max((waves < 4 ? std::ceil(waves) : waves + 0.5) * work, 1.2 * (double)p.N * (double)p.K * (double)(p.nb0 * p.nb1) * 4 / 6.4e6);
}
double rows_us(const GemmProblem &p, const SkinnyPlan &pl) {
  const double per_k = p.M <= 4 ? 9.2 : p.M <= 8 ? 7.4 : p.M <= 16 ? 12.6 : 23.3, per_sm = p.M <= 16 ? 2.0 : 1.0;
  const double waves = std::max(1.0, (double)pl.tiles_n * pl.splits * (double)(p.nb0 * p.nb1) / (per_sm * kSms));
  return (pl.splits > 1 ? 2.82 : 0.0) + waves * (2.2 + per_k * (double)pl.k_per_split / 1024);
}
bool columns_pay(const GemmProblem &p, const SkinnyPlan &pl) {
  return columns_possible(p) && columns_us((double)p.M, (double)p.N, (double)p.K, (double)(p.nb0 * p.nb1)) <= slices_us(p, pl);
}

int launch_skinny(const GemmProblem &p, const GemmEpilogue &e, const SkinnyPlan &pl, void *scratch, cudaStream_t s) {
  SkinnyArgs a;
  a.p = p; a.e = e;
  a.splits = pl.splits; a.k_per_split = pl.k_per_split; a.tiles_n = pl.tiles_n;
  a.counters = reinterpret_cast<unsigned *>(scratch);
  a.partials = reinterpret_cast<float *>(reinterpret_cast<uint8_t *>(scratch) + pl.counter_bytes);
  const dim3 grid((unsigned)pl.tiles_n, (unsigned)pl.splits, (unsigned)(p.nb0 * p.nb1));
  if (p.b_sk == 1 && p.b_sn != 1) {
    // (k slices start at multiples of 128, so every slice keeps the 16-byte alignment of its row)
    const bool vec = p.a_sk == 1 && (p.a_sm & 3) == 0 && (p.b_sn & 3) == 0 && aligned16(p.a) && aligned16(p.b) &&
                     (p.a_b0 & 3) == 0 && (p.a_b1 & 3) == 0 && (p.b_b0 & 3) == 0 && (p.b_b1 & 3) == 0;
    if (vec && p.M <= 4) FML_LAUNCH((gemm_skinny_kernel<4>), grid, kThreads, 0, s, a);
    else if (vec) FML_LAUNCH((gemm_skinny_kernel<8>), grid, kThreads, 0, s, a);
    else FML_LAUNCH((gemm_skinny_kernel<0>), grid, kThreads, 0, s, a);
  } else if (p.M <= 4) {
    FML_LAUNCH((gemm_skinny_rows_kernel<4>), grid, kThreads, 0, s, a);
  } else if (p.M <= 8) {
    FML_LAUNCH((gemm_skinny_rows_kernel<8>), grid, kThreads, 0, s, a);
  } else if (p.M <= 16) {
    FML_LAUNCH((gemm_skinny_rows_kernel<16>), grid, kThreads, 0, s, a);
  } else {
    FML_LAUNCH((gemm_skinny_rows_kernel<32>), grid, kThreads, 0, s, a);
  }
  return FML_OK;
}

// Library-owned scratch, one buffer per (device, stream), grown on demand and cleared when it
// is (re)allocated.  Launches on one stream are ordered, so they can share it.
struct Scratch { void *ptr = nullptr; size_t bytes = 0; };
std::map<std::pair<int, cudaStream_t>, Scratch> g_scratch;
std::mutex g_scratch_mu;

int scratch_for(size_t bytes, cudaStream_t s, void **out) {
  int dev = 0;
  FML_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  Scratch &sc = g_scratch[{dev, s}];
  if (sc.bytes < bytes) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(s, &cap);
    FML_REQUIRE(cap == cudaStreamCaptureStatusNone, FML_CUDA_ERROR,
                "fml_gemm: the skinny-GEMM scratch must grow (%zu bytes) but the stream is being captured; "
                "run the call once outside the capture first", bytes);
    FML_CUDA(cudaStreamSynchronize(s));
    if (sc.ptr) FML_CUDA(cudaFree(sc.ptr));
    sc.ptr = nullptr;
    sc.bytes = 0;
    const size_t want = std::max<size_t>(bytes, 1 << 20);
    FML_CUDA(cudaMalloc(&sc.ptr, want));
    FML_CUDA(cudaMemset(sc.ptr, 0, want));
    sc.bytes = want;
  }
  *out = sc.ptr;
  return FML_OK;
}

}  // namespace

bool skinny_eligible(const GemmProblem &p) {
  return p.M >= 1 && p.M <= kMaxM && p.K >= 1 && p.N >= 1 && p.nb0 * p.nb1 <= 65535 &&
         (p.N + kColsPerCta - 1) / kColsPerCta <= 0x7fffffff;
}

static int launch_columns(const GemmProblem &p, const GemmEpilogue &e, cudaStream_t s) {
  const unsigned z = (unsigned)(p.nb0 * p.nb1);
  // row groups: as many as leave every warp a chunk of k, and enough that a warp has at most sixteen rows
  int groups = p.M > 16 ? 2 : 1;
  while (groups < 8 && p.M > groups && p.K * groups <= 4 * 128) groups *= 2;
  const int64_t rows = (p.M + groups - 1) / groups;
  auto columns = [&](auto kernel) -> int {
    FML_LAUNCH(kernel, dim3((unsigned)((p.N + kCtaCols - 1) / kCtaCols), 1, z), kThreads, 0, s, p, e, groups);
    return FML_OK;
  };
  if (rows == 1) return columns(gemm_skinny_columns_kernel<1, 4>);
  if (rows == 2) return columns(gemm_skinny_columns_kernel<2, 4>);
  if (rows <= 4) return columns(gemm_skinny_columns_kernel<4, 4>);
  if (rows <= 8) return columns(gemm_skinny_columns_kernel<8, 4>);
  return columns(gemm_skinny_columns_kernel<16, 2>);
}

int launch_gemm_skinny(const GemmProblem &p, const GemmEpilogue &e, cudaStream_t s) {
  const SkinnyPlan pl = plan_skinny(p);
  if (columns_pay(p, pl)) return launch_columns(p, e, s);
  void *scratch = nullptr;
  if (pl.scratch_bytes) {
    int st = scratch_for(pl.scratch_bytes, s, &scratch);
    if (st != FML_OK && columns_possible(p)) return launch_columns(p, e, s);  // (needs none: a stream that is being captured)
    if (st != FML_OK) return st;
  }
  return launch_skinny(p, e, pl, scratch, s);
}

size_t gemm_skinny_scratch_bytes(const GemmProblem &p) { return plan_skinny(p).scratch_bytes; }

bool gemm_skinny_by_columns(const GemmProblem &p) { return skinny_eligible(p) && columns_pay(p, plan_skinny(p)); }


// ---- the same product for callers that cannot let the library allocate ---------------------
//
// Some hosts may not have device memory allocated on their behalf while they call in: a
// serving loop that has handed all of HBM to its own pool, code that runs inside a section
// where cudaMalloc's implicit device synchronisation is not acceptable, or an embedding that
// audits every allocation.  fml_gemm's skinny path grows a cudaMalloc'ed scratch buffer on
// demand; the entry point below keeps its split-K counters and partial sums in an array that
// is part of the loaded module instead, so it never calls an allocating routine -- at the
// price of a fixed capacity.
constexpr size_t kStaticScratchBytes = 1 << 20;  // 64 KiB of tile counters + 960 KiB of partial sums
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

namespace {
constexpr int kMaxDevices = 64;
void *g_static_scratch_addr[kMaxDevices] = {nullptr};  // per device: where the array lives
std::mutex g_static_mu;
}  // namespace

}  // namespace fml

using namespace fml;

// Declared in fluidml_cuda.h.  The first call on each device does the set-up: it asks the
// runtime where this device's copy of the array is (a host-side symbol is not a device
// address) and clears the counter region, which has to read zero when a launch starts
// (every launch leaves it zero again).  That first call enqueues a memset and waits for it,
// so make it before any stream capture.  All calls on one device share the one array: two
// calls whose kernels can overlap (different streams, no ordering between them) race on it.
extern "C" int fml_gemm_skinny_noalloc(const fml_tensor *a, const fml_tensor *b, const fml_tensor *c,
                                       const fml_tensor *bias, const fml_tensor *residual,
                                       const fml_gemm_params *gp, void *stream) {
  FML_REQUIRE(gp, FML_BAD_ARG, "fml_gemm_skinny_noalloc: null params");
  FML_REQUIRE(gp->precision == FML_GEMM_AUTO || gp->precision == FML_GEMM_FP32, FML_UNSUPPORTED,
              "fml_gemm_skinny_noalloc: computes in fp32 FMA only");
  GemmProblem p;
  int st = analyse_gemm(a, b, c, bias, residual, p);
  if (st != FML_OK) return st;
  if (p.M == 0 || p.N == 0 || p.nb0 * p.nb1 == 0) return FML_OK;
  FML_REQUIRE(skinny_eligible(p), FML_UNSUPPORTED,
              "fml_gemm_skinny_noalloc: needs 1 <= M <= %d rows and K >= 1 (M = %lld, K = %lld)", kMaxM,
              (long long)p.M, (long long)p.K);
  const SkinnyPlan pl = plan_skinny(p);
  FML_REQUIRE(pl.scratch_bytes <= kStaticScratchBytes, FML_OUT_OF_MEMORY,
              "fml_gemm_skinny_noalloc: this product needs %zu bytes of split-K scratch, the built-in "
              "buffer holds %zu; use fml_gemm", pl.scratch_bytes, kStaticScratchBytes);
  GemmEpilogue e;
  e.divisor = gp->divisor == 0.0f ? 1.0f : gp->divisor;
  e.alpha = gp->alpha; e.beta = gp->beta; e.act = gp->act;
  e.c0 = gp->act_param[0]; e.c1 = gp->act_param[1]; e.c2 = gp->act_param[2];
  e.has_bias = bias != nullptr; e.has_res = residual != nullptr;
  cudaStream_t s = as_stream(stream);
  int dev = 0;
  FML_CUDA(cudaGetDevice(&dev));
  FML_REQUIRE(dev >= 0 && dev < kMaxDevices, FML_BAD_ARG, "fml_gemm_skinny_noalloc: device ordinal %d out of range", dev);
  void *scratch = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (!g_static_scratch_addr[dev]) {
      // The set-up below enqueues a memset and waits for it; inside a capture that would end up
      // in the caller's graph and the wait would invalidate the capture.  Refuse instead.
      cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
      FML_CUDA(cudaStreamIsCapturing(s, &cap));
      FML_REQUIRE(cap == cudaStreamCaptureStatusNone, FML_CUDA_ERROR,
                  "fml_gemm_skinny_noalloc: the first call on a device sets up the scratch array and must be made "
                  "outside stream capture");
      void *addr = nullptr;
      FML_CUDA(cudaGetSymbolAddress(&addr, g_static_scratch));
      FML_REQUIRE(addr != nullptr, FML_CUDA_ERROR, "fml_gemm_skinny_noalloc: no device address for the scratch array");
      FML_CUDA(cudaMemsetAsync(addr, 0, kCounterBytes, s));
      FML_CUDA(cudaStreamSynchronize(s));  // set-up is complete when this call returns
      g_static_scratch_addr[dev] = addr;
    }
    scratch = g_static_scratch_addr[dev];
  }
  if (columns_pay(p, pl)) return launch_columns(p, e, s);  // as fml_gemm (the capacity is checked all the same)
  return launch_skinny(p, e, pl, scratch, s);
}

// Declared in fluidml_cuda.h: measured below 16 M multiply-adds only.
extern "C" int fml_gemm_prefers_k_major(int64_t rows, int64_t n, int64_t k) {
  if (rows < 1 || rows >= kMaxM || n < 1 || k < 4 || k % 4 || rows * n * k > (16ll << 20)) return 0;
  GemmProblem p;
  memset(&p, 0, sizeof(p));
  p.M = rows; p.N = n; p.K = k; p.nb0 = p.nb1 = 1;
  return columns_us((double)rows, (double)n, (double)k, 1.0) <= rows_us(p, plan_skinny(p)) ? 1 : 0;
}

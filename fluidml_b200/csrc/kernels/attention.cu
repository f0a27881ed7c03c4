// Fused attention core: out = softmax(Q K^T / divisor + mask) V for one block of query rows
// of one head per CTA, all in fp32 FMA.
//
// At batch-1 sequence lengths the three launches this replaces (scores GEMM, masked softmax,
// context GEMM) are each a few microseconds of launch, ramp and drain around well under a
// microsecond of arithmetic (12 heads x 128 x 128 x 64 x 2 products = 50 MFLOP), and the
// score matrix makes a round trip through L2 between them.  Here K and V of the head are
// staged once in shared memory (they fit: S_k * (D + D_v) floats), the 16 x S_k block of
// scores never leaves the SM, and the fp32 FMAs give the oracle's precision without the
// 3xTF32 split.  Operands are arbitrary strided views, so the head split / merge transposes
// of the graph stay views.
#include "common.cuh"

namespace fml {
namespace {

constexpr int kRows = 16;      // query rows per CTA
constexpr int kThreads = 256;  // 16 threads per query row
constexpr size_t kSmemLimit = 200 * 1024;

struct AttnArgs {
  int64_t Sq, Sk, D, Dv, nb0, nb1;
  // element strides: batch outer, batch inner, row, col
  int64_t q_s[4], k_s[4], v_s[4], o_s[4], m_s[4];  // k: [.., D, Sk] -> k_s[2] = stride of d, k_s[3] = stride of j
  const float *q, *k, *v, *mask;
  float *out;
  float divisor;
};

__device__ __forceinline__ void cp_async16(float *dst_smem, const float *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst_smem)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// dst[row * pitch + col] = src[row * s_row + col * s_col] for a rows x cols tile.  Rows that
// are contiguous and 16-byte aligned stream in with asynchronous 16-byte copies (no register
// staging, all of them in flight at once); other layouts go through registers, four loads
// at a time.  The caller commits / waits on the async group.
__device__ __forceinline__ void load_tile(float *dst, int pitch, const float *src, int rows, int cols,
                                          int64_t s_row, int64_t s_col) {
  const bool vec = s_col == 1 && (cols & 3) == 0 && (s_row & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0;
  if (vec) {
    const int c4 = cols >> 2;
    for (int i = threadIdx.x; i < rows * c4; i += kThreads) {
      const int r = i / c4, c = (i - r * c4) << 2;
      cp_async16(dst + r * pitch + c, src + r * s_row + c);
    }
    return;
  }
  const bool by_rows = s_row == 1;  // rows are the contiguous direction: walk them fastest
  const int total = rows * cols;
  for (int i0 = threadIdx.x; i0 < total; i0 += 4 * kThreads) {
    float v[4];
    int at[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * kThreads;
      int r = 0, c = 0;
      if (i < total) {
        if (by_rows) { c = i / rows; r = i - c * rows; }
        else { r = i / cols; c = i - r * cols; }
      }
      at[u] = i < total ? r * pitch + c : -1;
      v[u] = i < total ? src[r * s_row + c * s_col] : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (at[u] >= 0) dst[at[u]] = v[u];
  }
}

// Shared-memory bandwidth (128 bytes per clock per SM, whatever the broadcast pattern of a
// 16-byte read) is what bounds the two products, so both use register tiles that do many
// FMAs per byte read:
//   scores   each half of the CTA takes half of the head dimension; a thread holds a 4 x 4
//            tile (rows rq + 4x, columns cq + 32u): per 4 values of d, 4 Q and 4 K 16-byte
//            reads feed 64 FMAs; the second half adds its partial scores to the first's.
//   context  warp w takes an eighth of the keys; a thread holds 4 rows x 8 output columns:
//            per key, 4 P values and two 16-byte V reads feed 32 FMAs; the eight partial
//            tiles are added in warp order through shared memory.
__global__ void __launch_bounds__(kThreads) attention_kernel(AttnArgs a) {
  const ExactDivisor div(a.divisor);  // 1 / sqrt(head size) is usually a power of two: a multiply, same bits
  pdl_prologue();
  extern __shared__ __align__(16) float smem[];
  const int D = (int)a.D, Dv = (int)a.Dv, Sk = (int)a.Sk;
  const int pk = D + 4;     // K / Q pitch: 16-byte aligned rows, conflict-free 16-byte reads
  const int pp = Sk | 1;    // score pitch, odd: rows rq, rq + 1, .. fall in different banks
  float *Qs = smem;                    // [kRows][pk]
  float *Ks = Qs + kRows * pk;         // [Sk][pk]
  float *Vs = Ks + (size_t)Sk * pk;    // [Sk][Dv]
  float *Red = Vs + (size_t)Sk * Dv;   // [8][kRows][Dv] partial context tiles
  float *Ps = Red + 8 * kRows * Dv;    // [kRows][pp]
  float *Ms = Ps + kRows * pp;         // [kRows or 1][Sk] mask values of this block
  const int64_t z0 = blockIdx.y % a.nb0, z1 = blockIdx.y / a.nb0;
  const int64_t row0 = (int64_t)blockIdx.x * kRows;
  const int rows = (int)min((int64_t)kRows, a.Sq - row0);
  const float *q = a.q + z1 * a.q_s[0] + z0 * a.q_s[1] + row0 * a.q_s[2];
  const float *k = a.k + z1 * a.k_s[0] + z0 * a.k_s[1];
  const float *v = a.v + z1 * a.v_s[0] + z0 * a.v_s[1];
  float *o = a.out + z1 * a.o_s[0] + z0 * a.o_s[1] + row0 * a.o_s[2];
  const float *m = a.mask ? a.mask + z1 * a.m_s[0] + z0 * a.m_s[1] + row0 * a.m_s[2] : nullptr;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (rows < kRows)  // the tail block: unused query rows must not feed NaNs into the tiles
    for (int i = threadIdx.x; i < (kRows - rows) * pk; i += kThreads) Qs[rows * pk + i] = 0.0f;
  load_tile(Qs, pk, q, rows, D, a.q_s[2], a.q_s[3]);
  load_tile(Ks, pk, k, Sk, D, a.k_s[3], a.k_s[2]);  // Ks[j][d] = K^T[d][j]
  const int mrows = m ? (a.m_s[2] == 0 ? 1 : rows) : 0;  // a mask that broadcasts over query rows is staged once
  if (mrows) load_tile(Ms, Sk, m, mrows, Sk, a.m_s[2], a.m_s[3]);
  cp_async_commit();
  load_tile(Vs, Dv, v, Sk, Dv, a.v_s[2], a.v_s[3]);  // V keeps streaming under the score phase
  cp_async_commit();
  cp_async_wait<1>();
  __syncthreads();

  // ---- scores: Ps[r][j] = q_r . k_j
  {
    const int half = warp >> 2, rq = warp & 3, cq = lane;
    const int n4 = D >> 2, d_lo = half ? n4 >> 1 : 0, d_hi = half ? n4 : n4 >> 1;
    for (int jb = 0; jb < Sk; jb += 128) {
      float acc[4][4];
      const float4 *k4[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[x][u] = 0.0f;
        k4[u] = reinterpret_cast<const float4 *>(Ks + (size_t)min(jb + cq + 32 * u, Sk - 1) * pk);
      }
      const float4 *q4 = reinterpret_cast<const float4 *>(Qs + rq * pk);
      const int qstep = pk;  // rows rq, rq + 4, rq + 8, rq + 12 are 4 * pk floats = pk float4 apart
#pragma unroll 2
      for (int d = d_lo; d < d_hi; ++d) {
        float4 qv[4], kv[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) qv[x] = q4[x * qstep + d];
#pragma unroll
        for (int u = 0; u < 4; ++u) kv[u] = k4[u][d];
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            acc[x][u] = fmaf(qv[x].x, kv[u].x, acc[x][u]);
            acc[x][u] = fmaf(qv[x].y, kv[u].y, acc[x][u]);
            acc[x][u] = fmaf(qv[x].z, kv[u].z, acc[x][u]);
            acc[x][u] = fmaf(qv[x].w, kv[u].w, acc[x][u]);
          }
      }
      // the first half stores, the second half adds: a fixed order
      for (int turn = 0; turn < 2; ++turn) {
        if (turn == half) {
#pragma unroll
          for (int x = 0; x < 4; ++x)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int j = jb + cq + 32 * u;
              if (j < Sk) {
                float *dst = Ps + (rq + 4 * x) * pp + j;
                *dst = turn ? *dst + acc[x][u] : acc[x][u];
              }
            }
        }
        __syncthreads();
      }
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  // ---- softmax(s / divisor + mask) over each row; a row's 16 threads are half a warp
  {
    const int r = threadIdx.x >> 4, cg = threadIdx.x & 15;
    const bool live = r < rows;
    float *p = Ps + r * pp;
    const float *mr = Ms + (mrows > 1 ? r * Sk : 0);
    float mx = -3.402823466e+38f;
    if (live)
      for (int j = cg; j < Sk; j += 16) {
        float sc = p[j];
        if (a.divisor != 1.0f) sc = div(sc);
        if (m) sc += mr[j];
        p[j] = sc;
        mx = fmaxf(mx, sc);
      }
#pragma unroll
    for (int o2 = 8; o2 > 0; o2 >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o2));
    float sum = 0.0f;
    if (live)
      for (int j = cg; j < Sk; j += 16) {
        const float e = expf(p[j] - mx);
        p[j] = e;
        sum += e;
      }
#pragma unroll
    for (int o2 = 8; o2 > 0; o2 >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o2);
    for (int j = cg; j < Sk; j += 16) p[j] = live ? p[j] / sum : 0.0f;
  }
  __syncthreads();
  // ---- context: out[r][dv] = sum_j P[r][j] V[j][dv]
  {
    const int rg = lane >> 3, cgp = lane & 7;
    const int per = (Sk + 7) >> 3, j_lo = min(Sk, warp * per), j_hi = min(Sk, j_lo + per);
    const float *p0 = Ps + rg * pp;
    for (int dv0 = 0; dv0 < Dv; dv0 += 64) {
      const int ca = dv0 + cgp * 4, cb = ca + 32;
      const bool has_a = ca < Dv, has_b = cb < Dv;
      float4 acc[4][2];
#pragma unroll
      for (int x = 0; x < 4; ++x) acc[x][0] = acc[x][1] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
      for (int j = j_lo; j < j_hi; ++j) {
        const float *vr = Vs + (size_t)j * Dv;
        const float4 va = has_a ? *reinterpret_cast<const float4 *>(vr + ca) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 vb = has_b ? *reinterpret_cast<const float4 *>(vr + cb) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const float pj = p0[4 * x * pp + j];
          acc[x][0].x = fmaf(pj, va.x, acc[x][0].x); acc[x][0].y = fmaf(pj, va.y, acc[x][0].y);
          acc[x][0].z = fmaf(pj, va.z, acc[x][0].z); acc[x][0].w = fmaf(pj, va.w, acc[x][0].w);
          acc[x][1].x = fmaf(pj, vb.x, acc[x][1].x); acc[x][1].y = fmaf(pj, vb.y, acc[x][1].y);
          acc[x][1].z = fmaf(pj, vb.z, acc[x][1].z); acc[x][1].w = fmaf(pj, vb.w, acc[x][1].w);
        }
      }
      if (dv0) __syncthreads();  // the previous pass's partial tiles have been consumed
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        float *dst = Red + ((size_t)warp * kRows + rg + 4 * x) * Dv;
        if (has_a) *reinterpret_cast<float4 *>(dst + ca) = acc[x][0];
        if (has_b) *reinterpret_cast<float4 *>(dst + cb) = acc[x][1];
      }
      __syncthreads();
      // add the eight partial tiles in warp order and store 16 rows x up to 64 columns
      const int w4 = min(64, Dv - dv0) >> 2;
      for (int i = threadIdx.x; i < kRows * w4; i += kThreads) {
        const int r = i / w4, c = dv0 + ((i - r * w4) << 2);
        if (r >= rows) continue;
        float4 t = *reinterpret_cast<const float4 *>(Red + (size_t)r * Dv + c);
#pragma unroll
        for (int w = 1; w < 8; ++w) {
          const float4 u = *reinterpret_cast<const float4 *>(Red + ((size_t)w * kRows + r) * Dv + c);
          t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
        }
        float *dst = o + r * a.o_s[2] + c * a.o_s[3];
        const bool ovec = a.o_s[3] == 1 && (a.o_s[2] & 3) == 0 && (reinterpret_cast<uintptr_t>(o) & 15) == 0;
        if (ovec) *reinterpret_cast<float4 *>(dst) = t;
        else { dst[0] = t.x; dst[a.o_s[3]] = t.y; dst[2 * a.o_s[3]] = t.z; dst[3 * a.o_s[3]] = t.w; }
      }
    }
  }
}

// Keys and values that do not fit in shared memory at once (long sequences) stream through it in
// chunks of 128 keys with the running-maximum ("online") softmax: per chunk the scores, their
// maximum m' = max(m, chunk max), the weights e = exp(s - m'), and the context accumulator and
// the normaliser l rescaled by exp(m - m') before the chunk's contribution is added; the output
// is accumulator / l.  The arithmetic is that of softmax followed by the product, in another
// order (within a few ulp per element).  Tiles, thread mappings and the warp-ordered reduction
// are those of attention_kernel.
constexpr int kChunk = 128;

__global__ void __launch_bounds__(kThreads) attention_flash_kernel(AttnArgs a) {
  const ExactDivisor div(a.divisor);  // 1 / sqrt(head size) is usually a power of two: a multiply, same bits
  pdl_prologue();
  extern __shared__ __align__(16) float smem[];
  const int D = (int)a.D, Dv = (int)a.Dv, Sk = (int)a.Sk;
  const int pk = D + 4, pp = kChunk | 1;
  float *Qs = smem;                        // [kRows][pk]
  float *Ks = Qs + kRows * pk;             // [kChunk][pk]
  float *Vs = Ks + (size_t)kChunk * pk;    // [kChunk][Dv]
  float *Red = Vs + (size_t)kChunk * Dv;   // [8][kRows][Dv]
  float *Ps = Red + 8 * kRows * Dv;        // [kRows][pp]
  float *Ms = Ps + kRows * pp;             // [kRows or 1][kChunk]
  float *row_m = Ms + kRows * kChunk;      // [kRows] running maximum
  float *row_l = row_m + kRows;            // [kRows] running normaliser
  float *row_scale = row_l + kRows;        // [kRows] exp(old maximum - new maximum) of the current chunk
  const int64_t z0 = blockIdx.y % a.nb0, z1 = blockIdx.y / a.nb0;
  const int64_t row0 = (int64_t)blockIdx.x * kRows;
  const int rows = (int)min((int64_t)kRows, a.Sq - row0);
  const float *q = a.q + z1 * a.q_s[0] + z0 * a.q_s[1] + row0 * a.q_s[2];
  const float *k = a.k + z1 * a.k_s[0] + z0 * a.k_s[1];
  const float *v = a.v + z1 * a.v_s[0] + z0 * a.v_s[1];
  float *o = a.out + z1 * a.o_s[0] + z0 * a.o_s[1] + row0 * a.o_s[2];
  const float *m = a.mask ? a.mask + z1 * a.m_s[0] + z0 * a.m_s[1] + row0 * a.m_s[2] : nullptr;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int mrows = m ? (a.m_s[2] == 0 ? 1 : rows) : 0;

  if (rows < kRows)
    for (int i = threadIdx.x; i < (kRows - rows) * pk; i += kThreads) Qs[rows * pk + i] = 0.0f;
  if (threadIdx.x < kRows) { row_m[threadIdx.x] = -3.402823466e+38f; row_l[threadIdx.x] = 0.0f; }
  load_tile(Qs, pk, q, rows, D, a.q_s[2], a.q_s[3]);
  // context accumulators of the threads that combine the partial tiles: 16 rows x Dv / 4 quads over
  // 256 threads = at most two per thread (Dv <= 128)
  float4 acc_out0 = make_float4(0.f, 0.f, 0.f, 0.f), acc_out1 = acc_out0;

  for (int j0 = 0; j0 < Sk; j0 += kChunk) {
    const int kc = min(kChunk, Sk - j0);
    __syncthreads();  // the previous chunk's K, V, P and partial tiles are no longer read
    load_tile(Ks, pk, k + (int64_t)j0 * a.k_s[3], kc, D, a.k_s[3], a.k_s[2]);
    if (mrows) load_tile(Ms, kChunk, m + (int64_t)j0 * a.m_s[3], mrows, kc, a.m_s[2], a.m_s[3]);
    cp_async_commit();
    load_tile(Vs, Dv, v + (int64_t)j0 * a.v_s[2], kc, Dv, a.v_s[2], a.v_s[3]);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    // ---- scores of the chunk
    {
      const int half = warp >> 2, rq = warp & 3, cq = lane;
      const int n4 = D >> 2, d_lo = half ? n4 >> 1 : 0, d_hi = half ? n4 : n4 >> 1;
      float acc[4][4];
      const float4 *k4[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[x][u] = 0.0f;
        k4[u] = reinterpret_cast<const float4 *>(Ks + (size_t)min(cq + 32 * u, kc - 1) * pk);
      }
      const float4 *q4 = reinterpret_cast<const float4 *>(Qs + rq * pk);
#pragma unroll 2
      for (int d = d_lo; d < d_hi; ++d) {
        float4 qv[4], kv[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) qv[x] = q4[x * pk + d];
#pragma unroll
        for (int u = 0; u < 4; ++u) kv[u] = k4[u][d];
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            acc[x][u] = fmaf(qv[x].x, kv[u].x, acc[x][u]);
            acc[x][u] = fmaf(qv[x].y, kv[u].y, acc[x][u]);
            acc[x][u] = fmaf(qv[x].z, kv[u].z, acc[x][u]);
            acc[x][u] = fmaf(qv[x].w, kv[u].w, acc[x][u]);
          }
      }
      for (int turn = 0; turn < 2; ++turn) {
        if (turn == half) {
#pragma unroll
          for (int x = 0; x < 4; ++x)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int j = cq + 32 * u;
              if (j < kc) {
                float *dst = Ps + (rq + 4 * x) * pp + j;
                *dst = turn ? *dst + acc[x][u] : acc[x][u];
              }
            }
        }
        __syncthreads();
      }
    }
    cp_async_wait<0>();
    __syncthreads();
    // ---- running softmax of the chunk
    {
      const int r = threadIdx.x >> 4, cg = threadIdx.x & 15;
      const bool live = r < rows;
      float *p = Ps + r * pp;
      const float *mr = Ms + (mrows > 1 ? r * kChunk : 0);
      const float m_old = row_m[r], l_old = row_l[r];
      float mx = m_old;
      if (live)
        for (int j = cg; j < kc; j += 16) {
          float sc = p[j];
          if (a.divisor != 1.0f) sc = div(sc);
          if (m) sc += mr[j];
          p[j] = sc;
          mx = fmaxf(mx, sc);
        }
#pragma unroll
      for (int o2 = 8; o2 > 0; o2 >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o2));
      float sum = 0.0f;
      for (int j = cg; j < kc; j += 16) {
        const float e = live ? expf(p[j] - mx) : 0.0f;
        p[j] = e;
        sum += e;
      }
#pragma unroll
      for (int o2 = 8; o2 > 0; o2 >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o2);
      __syncwarp();
      if (cg == 0) {
        const float sc = expf(m_old - mx);  // 0 for the first chunk (m_old is the float lowest)
        row_scale[r] = sc;
        row_m[r] = mx;
        row_l[r] = l_old * sc + sum;
      }
    }
    __syncthreads();
    // ---- context contribution of the chunk, added to the rescaled accumulators
    {
      const int rg = lane >> 3, cgp = lane & 7;
      const int per = (kc + 7) >> 3, j_lo = min(kc, warp * per), j_hi = min(kc, j_lo + per);
      const float *p0 = Ps + rg * pp;
      int pass = 0;
      for (int dv0 = 0; dv0 < Dv; dv0 += 64, ++pass) {
        const int ca = dv0 + cgp * 4, cb = ca + 32;
        const bool has_a = ca < Dv, has_b = cb < Dv;
        float4 acc[4][2];
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[x][0] = acc[x][1] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
        for (int j = j_lo; j < j_hi; ++j) {
          const float *vr = Vs + (size_t)j * Dv;
          const float4 va = has_a ? *reinterpret_cast<const float4 *>(vr + ca) : make_float4(0.f, 0.f, 0.f, 0.f);
          const float4 vb = has_b ? *reinterpret_cast<const float4 *>(vr + cb) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            const float pj = p0[4 * x * pp + j];
            acc[x][0].x = fmaf(pj, va.x, acc[x][0].x); acc[x][0].y = fmaf(pj, va.y, acc[x][0].y);
            acc[x][0].z = fmaf(pj, va.z, acc[x][0].z); acc[x][0].w = fmaf(pj, va.w, acc[x][0].w);
            acc[x][1].x = fmaf(pj, vb.x, acc[x][1].x); acc[x][1].y = fmaf(pj, vb.y, acc[x][1].y);
            acc[x][1].z = fmaf(pj, vb.z, acc[x][1].z); acc[x][1].w = fmaf(pj, vb.w, acc[x][1].w);
          }
        }
        if (dv0) __syncthreads();
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          float *dst = Red + ((size_t)warp * kRows + rg + 4 * x) * Dv;
          if (has_a) *reinterpret_cast<float4 *>(dst + ca) = acc[x][0];
          if (has_b) *reinterpret_cast<float4 *>(dst + cb) = acc[x][1];
        }
        __syncthreads();
        const int w4 = min(64, Dv - dv0) >> 2;
        const int i = threadIdx.x;  // 16 rows x at most 16 quads: one (row, quad) per thread and pass
        if (i < kRows * w4) {
          const int r = i / w4, c = dv0 + ((i - r * w4) << 2);
          float4 t = *reinterpret_cast<const float4 *>(Red + (size_t)r * Dv + c);
#pragma unroll
          for (int w = 1; w < 8; ++w) {
            const float4 u = *reinterpret_cast<const float4 *>(Red + ((size_t)w * kRows + r) * Dv + c);
            t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
          }
          const float sc = row_scale[r];
          float4 &ao = pass == 0 ? acc_out0 : acc_out1;
          ao.x = ao.x * sc + t.x; ao.y = ao.y * sc + t.y; ao.z = ao.z * sc + t.z; ao.w = ao.w * sc + t.w;
        }
      }
    }
  }
  // ---- out = accumulator / normaliser
  int pass = 0;
  for (int dv0 = 0; dv0 < Dv; dv0 += 64, ++pass) {
    const int w4 = min(64, Dv - dv0) >> 2;
    const int i = threadIdx.x;
    if (i < kRows * w4) {
      const int r = i / w4, c = dv0 + ((i - r * w4) << 2);
      if (r < rows) {
        const float l = row_l[r];
        const float4 ao = pass == 0 ? acc_out0 : acc_out1;
        const float4 t = make_float4(ao.x / l, ao.y / l, ao.z / l, ao.w / l);
        float *dst = o + r * a.o_s[2] + c * a.o_s[3];
        const bool ovec = a.o_s[3] == 1 && (a.o_s[2] & 3) == 0 && (reinterpret_cast<uintptr_t>(o) & 15) == 0;
        if (ovec) *reinterpret_cast<float4 *>(dst) = t;
        else { dst[0] = t.x; dst[a.o_s[3]] = t.y; dst[2 * a.o_s[3]] = t.z; dst[3 * a.o_s[3]] = t.w; }
      }
    }
  }
}

// Head sizes 32 and 64 whose rows are 16-byte-aligned runs (every model of the benchmark): the same
// computation as attention_kernel, arranged so that a call of a few microseconds is not spent on its own
// bookkeeping.  What bounds it is latency: one L2 round trip for Q and K, the shared-memory reads of the two
// products (about 1,300 + 400 clocks per 16 x 128 x 64 block) and one drain; attention_kernel took 10.4 us for 12
// heads of 128 x 128 of which 3.1 went into issuing the copies (a division per 16 bytes), 2.5 into the scores
// (partial sums added through shared memory in turns), 1.8 into the softmax and 2.0 into the context.  Here
//   - a thread's copies are a pointer and a step, worked out before the dependency wait;
//   - products are fma.rn.f32x2: the scores' pairs run along the head dimension (their two sums are added at
//     the end), the context's along the output columns;
//   - the halves of the head dimension leave their scores side by side and the softmax, four keys per read,
//     adds them; weights stay unnormalised and the finished row is divided once;
//   - keys beyond 128 come in chunks under a running maximum, the next chunk's K on its way during the softmax and
//     the context, its V during the next scores;
//   - 87 KB of shared memory for head size 64 (the partial contexts lie over K) and at most 128 registers: two
//     CTAs per SM overlap each other's phases where there are many (8 x 6 heads of 128: 384 CTAs).
// Captured graphs of one call after another, attention_kernel / attention_flash_kernel -> this one, us: 12 heads of
// 128 x 128 8.4 -> 7.3 (inside a BERT-base pass 10.3 -> 8.4), 36 of 77 9.8 -> 7.0, 48 of 128 22.6 -> 12.6, 16 of 77
// causal 10.5 -> 5.9, 12 of 256 30.2 -> 14.2, 8 of 300 38.7 -> 17.7, 64 of 128 x 32 16.7 -> 10.4, 2 of 16 5.3 -> 3.6.
// Left of a 7 us launch: 1.4 us to the first scores, 2.0 scores, 1.2 softmax, 1.1 context, 0.6 sum and store.
constexpr int kRowsKeys = 128;              // keys per chunk
constexpr int kRowsPP = kRowsKeys + 4;      // score pitch: 16-byte reads of four rows in different banks

__device__ __forceinline__ void fma2(unsigned long long &acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void cp_async16_or_zero(unsigned dst, const float *src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}

template <int D> constexpr size_t attn_rows_smem() {
  return (size_t)(kRows * (D + 4) + kRowsKeys * (D + 4) + kRowsKeys * D + 2 * kRows * kRowsPP + kRows) * sizeof(float);
}

// Scores of one chunk: rows rq, rq + 4, .. of Q against keys lane, lane + 32, .. over d4 in [d_lo, d_lo + N4).
template <int NU, int N4>
__device__ __forceinline__ void rows_scores(const float *q, const float *k, int pk, float *dst) {
  unsigned long long acc[4][NU];
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int u = 0; u < NU; ++u) acc[x][u] = 0ull;
#pragma unroll 2
  for (int d = 0; d < N4; ++d) {
    ulonglong2 qv[4], kv[NU];
#pragma unroll
    for (int x = 0; x < 4; ++x) qv[x] = *reinterpret_cast<const ulonglong2 *>(q + 4 * x * pk + 4 * d);
#pragma unroll
    for (int u = 0; u < NU; ++u) kv[u] = *reinterpret_cast<const ulonglong2 *>(k + 32 * u * pk + 4 * d);
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        fma2(acc[x][u], qv[x].x, kv[u].x);
        fma2(acc[x][u], qv[x].y, kv[u].y);
      }
  }
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int u = 0; u < NU; ++u) {
      const float2 t = unpack2(acc[x][u]);
      dst[4 * x * kRowsPP + 32 * u] = t.x + t.y;
    }
}

template <int D>
__global__ void __launch_bounds__(kThreads, 2) attention_rows_kernel(AttnArgs a, int causal) {
  constexpr int pk = D + 4, NV = D / 32, kPerRow = D / 4, kStep = kThreads / kPerRow;
  extern __shared__ __align__(16) float smem[];
  float *const Qs = smem;                      // [kRows][pk]
  float *const Ks = Qs + kRows * pk;           // [128][pk]; at the end the eight partial contexts [8][kRows][D]
  float *const Vs = Ks + kRowsKeys * pk;       // [128][D]
  float *const Ps = Vs + kRowsKeys * D;        // [2][kRows][kRowsPP]: scores of either half of d, then weights in the first
  float *const row_scale = Ps + 2 * kRows * kRowsPP;
  const ExactDivisor div(a.divisor);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int z0 = (int)(blockIdx.y % (unsigned)a.nb0), z1 = (int)(blockIdx.y / (unsigned)a.nb0);
  const int row0 = blockIdx.x * kRows, rows = min(kRows, (int)a.Sq - row0);
  const int Sk = causal ? min((int)a.Sk, row0 + kRows) : (int)a.Sk;  // no row of this block sees more
  // copies: this thread's 16-byte column and first row
  const int cr = threadIdx.x / kPerRow, cc = (threadIdx.x % kPerRow) * 4;
  const float *const q = a.q + z1 * a.q_s[0] + z0 * a.q_s[1] + (int64_t)row0 * a.q_s[2] + cc;
  const float *const k = a.k + z1 * a.k_s[0] + z0 * a.k_s[1] + cc;
  const float *const v = a.v + z1 * a.v_s[0] + z0 * a.v_s[1] + cc;
  const unsigned qd = (unsigned)__cvta_generic_to_shared(Qs + cr * pk + cc);
  const unsigned kd = (unsigned)__cvta_generic_to_shared(Ks + cr * pk + cc);
  const unsigned vd = (unsigned)__cvta_generic_to_shared(Vs + cr * D + cc);
  // softmax: sixteen threads per row, four adjacent keys at a time
  const int sr = threadIdx.x >> 4, sc4 = (threadIdx.x & 15) * 4;
  const bool live = sr < rows;
  const float *const mr = a.mask ? a.mask + z1 * a.m_s[0] + z0 * a.m_s[1] + (int64_t)(row0 + (live ? sr : 0)) * a.m_s[2] : nullptr;
  const bool m_vec = a.m_s[3] == 1 && (reinterpret_cast<uintptr_t>(mr) & 15) == 0;
  float *const o = a.out + z1 * a.o_s[0] + z0 * a.o_s[1] + (int64_t)(row0 + sr) * a.o_s[2];
  const bool o_vec = a.o_s[3] == 1 && (reinterpret_cast<uintptr_t>(o) & 15) == 0;

  auto load_k = [&](int j0) {  // rows up to the next multiple of 32; those that do not exist are zero
    const int kc = min(kRowsKeys, Sk - j0), kz = (kc + 31) & ~31;
    const float *src = k + (int64_t)j0 * a.k_s[3];
#pragma unroll 4
    for (int r = cr; r < kz; r += kStep) cp_async16_or_zero(kd + (unsigned)((r - cr) * pk * 4), src + (r < kc ? r : 0) * a.k_s[3], r < kc);
    cp_async_commit();
  };
  auto load_v = [&](int j0) {
    const int kc = min(kRowsKeys, Sk - j0), kz = (kc + 31) & ~31;
    const float *src = v + (int64_t)j0 * a.v_s[2];
#pragma unroll 4
    for (int r = cr; r < kz; r += kStep) cp_async16_or_zero(vd + (unsigned)((r - cr) * D * 4), src + (r < kc ? r : 0) * a.v_s[2], r < kc);
    cp_async_commit();
  };
  pdl_prologue();
#pragma unroll
  for (int r = cr; r < kRows; r += kStep) cp_async16_or_zero(qd + (unsigned)((r - cr) * pk * 4), q + (r < rows ? r : 0) * a.q_s[2], r < rows);
  load_k(0);
  load_v(0);

  float m_run = -3.402823466e+38f, l_run = 0.0f;  // of row sr, the same in its sixteen threads
  unsigned long long acc[4][NV][2];               // context: rows rg + 4x, columns cg * 4 + 32 v, over this warp's keys
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int n = 0; n < NV; ++n) acc[x][n][0] = acc[x][n][1] = 0ull;
  const int rg = lane >> 3, cg = (lane & 7) * 4;

  for (int j0 = 0; j0 < Sk; j0 += kRowsKeys) {
    const int kc = min(kRowsKeys, Sk - j0), nu = (kc + 31) >> 5;
    const bool more = j0 + kRowsKeys < Sk;
    float4 mv[2];  // this thread's mask values, on their way during the scores
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int j = sc4 + 64 * i;
      mv[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (!mr || j >= kc) continue;
      const float *src = mr + (int64_t)(j0 + j) * a.m_s[3];
      if (m_vec && j + 3 < kc) mv[i] = *reinterpret_cast<const float4 *>(src);
      else {
        mv[i].x = src[0];
        if (j + 1 < kc) mv[i].y = src[a.m_s[3]];
        if (j + 2 < kc) mv[i].z = src[2 * a.m_s[3]];
        if (j + 3 < kc) mv[i].w = src[3 * a.m_s[3]];
      }
    }
    cp_async_wait<1>();  // K (and Q); V may still be on its way
    __syncthreads();
    {
      const int half = warp >> 2, rq = warp & 3;
      const float *q_at = Qs + rq * pk + half * (D / 2), *k_at = Ks + lane * pk + half * (D / 2);
      float *dst = Ps + (half * kRows + rq) * kRowsPP + lane;
      if (nu == 4) rows_scores<4, D / 8>(q_at, k_at, pk, dst);
      else if (nu == 3) rows_scores<3, D / 8>(q_at, k_at, pk, dst);
      else if (nu == 2) rows_scores<2, D / 8>(q_at, k_at, pk, dst);
      else rows_scores<1, D / 8>(q_at, k_at, pk, dst);
    }
    __syncthreads();
    if (more) load_k(j0 + kRowsKeys);
    {
      float4 s[2];
      float mx = m_run;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int j = sc4 + 64 * i;
        if (j >= 32 * nu) continue;
        const float *p = Ps + sr * kRowsPP + j;
        const float4 p0 = *reinterpret_cast<const float4 *>(p), p1 = *reinterpret_cast<const float4 *>(p + kRows * kRowsPP);
        s[i] = make_float4(p0.x + p1.x, p0.y + p1.y, p0.z + p1.z, p0.w + p1.w);
        if (a.divisor != 1.0f) s[i] = make_float4(div(s[i].x), div(s[i].y), div(s[i].z), div(s[i].w));
        s[i].x += mv[i].x; s[i].y += mv[i].y; s[i].z += mv[i].z; s[i].w += mv[i].w;
        if (j < kc) mx = fmaxf(mx, s[i].x);
        if (j + 1 < kc) mx = fmaxf(mx, s[i].y);
        if (j + 2 < kc) mx = fmaxf(mx, s[i].z);
        if (j + 3 < kc) mx = fmaxf(mx, s[i].w);
      }
#pragma unroll
      for (int d = 8; d > 0; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
      float sum = 0.0f;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int j = sc4 + 64 * i;
        if (j >= 32 * nu) continue;
        float4 e = make_float4(0.f, 0.f, 0.f, 0.f);  // keys that do not exist weigh nothing
        if (j < kc) e.x = expf(s[i].x - mx);
        if (j + 1 < kc) e.y = expf(s[i].y - mx);
        if (j + 2 < kc) e.z = expf(s[i].z - mx);
        if (j + 3 < kc) e.w = expf(s[i].w - mx);
        *reinterpret_cast<float4 *>(Ps + sr * kRowsPP + j) = e;
        sum += (e.x + e.y) + (e.z + e.w);
      }
#pragma unroll
      for (int d = 8; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
      const float scale = j0 ? expf(m_run - mx) : 0.0f;
      m_run = mx;
      l_run = l_run * scale + sum;
      if (j0 && (threadIdx.x & 15) == 0) row_scale[sr] = scale;
    }
    if (more) cp_async_wait<1>();  // V; the next K may still be on its way
    else cp_async_wait<0>();
    __syncthreads();
    {
      if (j0) {
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const float t = row_scale[rg + 4 * x];
          const unsigned long long t2 = pack2(t, t);
#pragma unroll
          for (int n = 0; n < NV; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h) asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(acc[x][n][h]) : "l"(t2));
        }
      }
      const float *p = Ps + rg * kRowsPP + warp * 4 * nu, *vr = Vs + warp * 4 * nu * D + cg;  // 4 nu keys per warp
      for (int g = 0; g < nu; ++g, p += 4, vr += 4 * D) {
        float4 pv[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) pv[x] = *reinterpret_cast<const float4 *>(p + 4 * x * kRowsPP);
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          ulonglong2 vv[NV];
#pragma unroll
          for (int n = 0; n < NV; ++n) vv[n] = *reinterpret_cast<const ulonglong2 *>(vr + jj * D + 32 * n);
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            const float w = jj == 0 ? pv[x].x : jj == 1 ? pv[x].y : jj == 2 ? pv[x].z : pv[x].w;
            const unsigned long long w2 = pack2(w, w);
#pragma unroll
            for (int n = 0; n < NV; ++n) { fma2(acc[x][n][0], w2, vv[n].x); fma2(acc[x][n][1], w2, vv[n].y); }
          }
        }
      }
    }
    if (more) {
      __syncthreads();  // V, weights and scales of this chunk are no longer read
      load_v(j0 + kRowsKeys);
    }
  }
  // the warps' partial contexts, added in warp order (K was read before the last barrier but one)
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int n = 0; n < NV; ++n)
      *reinterpret_cast<ulonglong2 *>(Ks + (warp * kRows + rg + 4 * x) * D + cg + 32 * n) = make_ulonglong2(acc[x][n][0], acc[x][n][1]);
  __syncthreads();
  if (!live) return;
#pragma unroll
  for (int c = sc4; c < D; c += 64) {
    float4 t = *reinterpret_cast<const float4 *>(Ks + sr * D + c);
#pragma unroll
    for (int w = 1; w < 8; ++w) {
      const float4 u = *reinterpret_cast<const float4 *>(Ks + (w * kRows + sr) * D + c);
      t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
    }
    t = make_float4(t.x / l_run, t.y / l_run, t.z / l_run, t.w / l_run);
    float *dst = o + c * a.o_s[3];
    if (o_vec) *reinterpret_cast<float4 *>(dst) = t;
    else { dst[0] = t.x; dst[a.o_s[3]] = t.y; dst[2 * a.o_s[3]] = t.z; dst[3 * a.o_s[3]] = t.w; }
  }
}

// What attention_rows_kernel takes: head size 32 or 64 on both sides, rows of Q, K and V contiguous and on 16-byte
// boundaries (its copies are 16 bytes wide), offsets within a tile in 32 bits.
bool attn_rows_eligible(const AttnArgs &a) {
  if (a.D != a.Dv || (a.D != 32 && a.D != 64)) return false;
  if (a.q_s[3] != 1 || a.k_s[2] != 1 || a.v_s[3] != 1) return false;
  if (!aligned16(a.q) || !aligned16(a.k) || !aligned16(a.v)) return false;
  for (int i = 0; i < 2; ++i)
    if (a.q_s[i] % 4 || a.k_s[i] % 4 || a.v_s[i] % 4) return false;
  if (a.q_s[2] % 4 || a.k_s[3] % 4 || a.v_s[2] % 4) return false;
  return a.Sq < (1ll << 30) && a.Sk < (1ll << 30);
}

size_t attn_flash_smem_bytes(int64_t D, int64_t Dv) {
  return (size_t)(kRows * (D + 4) + kChunk * (D + 4) + kChunk * Dv + 8 * kRows * Dv + kRows * (kChunk | 1) +
                  kRows * kChunk + 3 * kRows) * sizeof(float);
}

size_t attn_smem_bytes(int64_t Sk, int64_t D, int64_t Dv) {
  return (size_t)(kRows * (D + 4) + Sk * (D + 4) + Sk * Dv + 8 * kRows * Dv + kRows * (Sk | 1) + kRows * Sk) * sizeof(float);
}

// Pads the tensor's dims to [b1, b0, rows, cols] (leading 1s) and returns its strides.
bool as4(const fml_tensor *t, int64_t shape[4], int64_t stride[4]) {
  if (t->rank < 2 || t->rank > 4) return false;
  const int pad = 4 - t->rank;
  for (int i = 0; i < 4; ++i) {
    shape[i] = i < pad ? 1 : t->shape[i - pad];
    stride[i] = i < pad ? 0 : t->stride[i - pad];
  }
  return true;
}

}  // namespace
}  // namespace fml

using namespace fml;

namespace fml {  // attention_tc.cu
bool attention_tc_shape_ok(int64_t s_q, int64_t s_k, int64_t d, int64_t d_v);
bool attention_tc_eligible(int64_t nb1, int64_t nb0, int64_t Sq, int64_t Sk, int64_t D, int64_t Dv, const int64_t *q_s,
                           const int64_t *k_s, const int64_t *v_s, const void *q, const void *k, const void *v);
int launch_attention_tc(int64_t nb1, int64_t nb0, int64_t Sq, int64_t Sk, int64_t D, int64_t Dv, const float *q,
                        const int64_t *q_s, const float *k, const int64_t *k_s, const float *v, const int64_t *v_s,
                        const float *mask, const int64_t *m_s, float divisor, float *out, const int64_t *o_s,
                        cudaStream_t s);
// attention_pair.cu
bool attention_pair_shape_ok(int64_t d, int64_t d_v);
int launch_attention_pair(int64_t nb1, int64_t nb0, int64_t Sq, int64_t Sk, const float *q, const int64_t *q_s, const float *k,
                          const int64_t *k_s, const float *v, const int64_t *v_s, const float *mask, const int64_t *m_s, bool causal,
                          float divisor, float *out, const int64_t *o_s, cudaStream_t s);
}  // namespace fml

// 1 when the tensor-core kernel (attention_tc.cu) takes blocks of these head sizes: such blocks are
// worth fusing whatever their size, the CUDA-core kernel only while the block is small.
extern "C" int fml_attention_on_tensor_cores(int64_t s_q, int64_t s_k, int64_t d, int64_t d_v) {
  return attention_tc_shape_ok(s_q, s_k, d, d_v) ? 1 : 0;
}

extern "C" int fml_attention_supported(int64_t s_q, int64_t s_k, int64_t d, int64_t d_v) {
  // any number of keys: those that do not fit in shared memory at once stream through it
  return s_q >= 1 && s_k >= 1 && d >= 4 && d_v >= 4 && d <= 128 && d_v <= 128 && (d & 3) == 0 && (d_v & 3) == 0 &&
                 (attn_smem_bytes(s_k, d, d_v) <= kSmemLimit || attn_flash_smem_bytes(d, d_v) <= kSmemLimit)
             ? 1 : 0;
}

// Blocks of any size are worth fusing when the half-precision-pair kernel takes their head size.
extern "C" int fml_attention_any_size(int64_t d, int64_t d_v) { return attention_pair_shape_ok(d, d_v) ? 1 : 0; }

static int attention_impl(const fml_tensor *q, const fml_tensor *kt, const fml_tensor *v, const fml_tensor *mask, bool causal,
                          float divisor, const fml_tensor *out, void *stream) {
  FML_REQUIRE(q && kt && v && out, FML_BAD_ARG, "fml_attention: null tensor");
  FML_REQUIRE(q->dtype == FML_F32 && kt->dtype == FML_F32 && v->dtype == FML_F32 && out->dtype == FML_F32 &&
                  (!mask || mask->dtype == FML_F32), FML_UNSUPPORTED, "fml_attention: fp32 only");
  FML_REQUIRE(divisor != 0.0f, FML_BAD_ARG, "fml_attention: divisor is zero");
  AttnArgs a;
  int64_t qs[4], ks[4], vs[4], os[4], ms[4] = {1, 1, 1, 1};
  FML_REQUIRE(as4(q, qs, a.q_s) && as4(kt, ks, a.k_s) && as4(v, vs, a.v_s) && as4(out, os, a.o_s) &&
                  (!mask || as4(mask, ms, a.m_s)), FML_UNSUPPORTED, "fml_attention: ranks 2 to 4 only");
  a.nb1 = qs[0]; a.nb0 = qs[1]; a.Sq = qs[2]; a.D = qs[3]; a.Sk = ks[3]; a.Dv = vs[3];
  FML_REQUIRE(ks[2] == a.D && vs[2] == a.Sk && os[2] == a.Sq && os[3] == a.Dv, FML_BAD_ARG,
              "fml_attention: shapes do not chain (Q [..,%lld,%lld], K^T [..,%lld,%lld], V [..,%lld,%lld])",
              (long long)a.Sq, (long long)a.D, (long long)ks[2], (long long)ks[3], (long long)vs[2], (long long)vs[3]);
  for (int i = 0; i < 2; ++i)
    FML_REQUIRE(ks[i] == qs[i] && vs[i] == qs[i] && os[i] == qs[i], FML_BAD_ARG,
                "fml_attention: batch dims of Q, K^T, V and the output must agree");
  if (mask) {
    const int64_t want[4] = {a.nb1, a.nb0, a.Sq, a.Sk};
    for (int i = 0; i < 4; ++i) {
      FML_REQUIRE(ms[i] == want[i] || ms[i] == 1, FML_BAD_ARG, "fml_attention: mask does not broadcast to the scores");
      if (ms[i] == 1) a.m_s[i] = 0;
    }
  }
  if (a.Sq == 0 || a.Dv == 0 || a.nb0 * a.nb1 == 0) return FML_OK;
  FML_REQUIRE(fml_attention_supported(a.Sq, a.Sk, a.D, a.Dv), FML_UNSUPPORTED,
              "fml_attention: needs head sizes that are multiples of 4 up to 128 and K, V of one head within "
              "%zu bytes of shared memory (S_k = %lld, D = %lld, D_v = %lld)", kSmemLimit, (long long)a.Sk,
              (long long)a.D, (long long)a.Dv);
  FML_REQUIRE(a.nb0 * a.nb1 <= 65535, FML_UNSUPPORTED, "fml_attention: more than 65535 heads x batches");
  a.q = (const float *)q->data; a.k = (const float *)kt->data; a.v = (const float *)v->data;
  a.mask = mask ? (const float *)mask->data : nullptr;
  a.out = (float *)out->data;
  a.divisor = divisor;
  if (attention_tc_eligible(a.nb1, a.nb0, a.Sq, a.Sk, a.D, a.Dv, a.q_s, a.k_s, a.v_s, a.q, a.k, a.v)) {
    if (attention_pair_shape_ok(a.D, a.Dv))
      return launch_attention_pair(a.nb1, a.nb0, a.Sq, a.Sk, a.q, a.q_s, a.k, a.k_s, a.v, a.v_s, a.mask, a.m_s, causal, divisor, a.out,
                                   a.o_s, as_stream(stream));
    return launch_attention_tc(a.nb1, a.nb0, a.Sq, a.Sk, a.D, a.Dv, a.q, a.q_s, a.k, a.k_s, a.v, a.v_s, a.mask, a.m_s,
                               divisor, a.out, a.o_s, as_stream(stream));
  }
  const bool whole = attn_smem_bytes(a.Sk, a.D, a.Dv) <= attn_flash_smem_bytes(a.D, a.Dv) ||
                     attn_flash_smem_bytes(a.D, a.Dv) > kSmemLimit;  // K and V of a head fit at once
  const size_t smem = whole ? attn_smem_bytes(a.Sk, a.D, a.Dv) : attn_flash_smem_bytes(a.D, a.Dv);
  static bool attr_set[64] = {false};
  int dev = 0;
  FML_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    FML_CUDA(cudaFuncSetAttribute(attention_rows_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)attn_rows_smem<32>()));
    FML_CUDA(cudaFuncSetAttribute(attention_rows_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)attn_rows_smem<64>()));
    FML_CUDA(cudaFuncSetAttribute(attention_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit));
    FML_CUDA(cudaFuncSetAttribute(attention_flash_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit));
    attr_set[dev] = true;
  }
  const dim3 grid((unsigned)((a.Sq + kRows - 1) / kRows), (unsigned)(a.nb0 * a.nb1));
  if (attn_rows_eligible(a)) {
    if (a.D == 64) FML_LAUNCH((attention_rows_kernel<64>), grid, kThreads, attn_rows_smem<64>(), as_stream(stream), a, causal ? 1 : 0);
    else FML_LAUNCH((attention_rows_kernel<32>), grid, kThreads, attn_rows_smem<32>(), as_stream(stream), a, causal ? 1 : 0);
  } else if (whole) FML_LAUNCH((attention_kernel), grid, kThreads, smem, as_stream(stream), a);
  else FML_LAUNCH((attention_flash_kernel), grid, kThreads, smem, as_stream(stream), a);
  return FML_OK;
}

extern "C" int fml_attention(const fml_tensor *q, const fml_tensor *kt, const fml_tensor *v,
                             const fml_tensor *mask, float divisor, const fml_tensor *out, void *stream) {
  return attention_impl(q, kt, v, mask, false, divisor, out, stream);
}

extern "C" int fml_attention_causal(const fml_tensor *q, const fml_tensor *kt, const fml_tensor *v, const fml_tensor *mask,
                                    float divisor, const fml_tensor *out, void *stream) {
  FML_REQUIRE(mask, FML_BAD_ARG, "fml_attention_causal: no mask");
  return attention_impl(q, kt, v, mask, true, divisor, out, stream);
}

// Whether fml_attention would run these operands on the tensor cores (tests and planners).
extern "C" int fml_attention_uses_tensor_cores(const fml_tensor *q, const fml_tensor *kt, const fml_tensor *v, int *uses) {
  FML_REQUIRE(q && kt && v && uses, FML_BAD_ARG, "fml_attention_uses_tensor_cores: null argument");
  AttnArgs a;
  int64_t qs[4], ks[4], vs[4];
  *uses = 0;
  if (q->dtype != FML_F32 || kt->dtype != FML_F32 || v->dtype != FML_F32) return FML_OK;
  if (!as4(q, qs, a.q_s) || !as4(kt, ks, a.k_s) || !as4(v, vs, a.v_s)) return FML_OK;
  *uses = attention_tc_eligible(qs[0], qs[1], qs[2], ks[3], qs[3], vs[3], a.q_s, a.k_s, a.v_s, q->data, kt->data, v->data) ? 1 : 0;
  return FML_OK;
}

// Epilogue of the tcgen05 GEMM kernels: sums the split-K partial tiles of a cluster, applies scaling,
// bias, activation and residual, and stores C.  Shared by gemm_tc.cu and gemm_pair.cu.
#pragma once
#include "gemm_common.cuh"
#include "tc_common.cuh"
#include <type_traits>

namespace fml {

// The activation is a template parameter of the kernel and bias / residual / scaling are
// cheap uniform predicates inside one short loop: every CTA runs each phase of this kernel
// once, so the cost of a phase is largely the instruction fetch of its (cold) code, and a
// compact, straight-line epilogue matters more than a branch-free one.
// erf by Abramowitz & Stegun 7.1.26: erf(x) = 1 - P(t) exp(-x^2) with t = 1 / (1 + 0.3275911 x), x >= 0, the formula itself
// within 1.5e-7.  Both pieces come from y = sqrt(log2 e) x, which is what is passed: exp(-x^2) = 2^(-y^2), for PTX's ex2.approx (2^-22
// of the result; it flushes what is below 2^-126, where x is beyond 9 and erf is 1), and t = 1 / (1 + (0.3275911 / sqrt(log2 e)) y)
// for its rcp.approx (1 ulp; the argument is at least 1).  In fp32 arithmetic the absolute error is about 6e-7, most of it
// the cancellation in 1 - P exp(-x^2) near 0 (tests/test_erf_formula_cpu.py restates it on the host and
// tests/test_gelu_epilogue_gpu.py holds the kernels to it), i.e. a GELU value off by at most 5e-7 |v| -- far below the
// product it is applied to.
// The exact erff is ~45 dependent instructions per element; with one epilogue warp per scheduler that was 35 us of a
// 134 us FFN launch at 2048 rows (4096 columns each).
constexpr float kSqrtLog2e = 1.2011224087864498f;
__device__ __forceinline__ float erf_fast(float x_scaled) {
  const float y = fabsf(x_scaled);
  float t;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(fmaf(0.27273748f, y, 1.0f)));
  float p = fmaf(1.061405429f, t, -1.453152027f);
  p = fmaf(p, t, 1.421413741f);
  p = fmaf(p, t, -0.284496736f);
  p = fmaf(p, t, 0.254829592f);
  return copysignf(fmaf(-p * t, ex2_approx(-y * y), 1.0f), x_scaled);
}

template <int ACT>
__device__ __forceinline__ float act_op(const GemmEpilogue &e, float v) {
  if (ACT == FML_ACT_GELU_ERF) return v * (erf_fast(v * (kSqrtLog2e * __frcp_rn(e.c0))) + e.c1) * e.c2;  // (the factor is loop-invariant)
  if (ACT == FML_ACT_RELU) return fmaxf(v, 0.0f);
  if (ACT == FML_ACT_TANH) return tanhf(v);
  if (ACT == FML_ACT_SIGMOID) return 1.0f / (1.0f + expf(-v));
  if (ACT == FML_ACT_SILU) return v / (1.0f + expf(-v));
  return v;
}

// Rows [split * 128 / S, (split + 1) * 128 / S) of the output tile: every rank of the cluster holds
// its fp32 partial tile in `staging` (row pitch in floats), the sum runs over the ranks in rank order
// (independent of timing), and consecutive threads take consecutive columns, so that the loads of bias
// and residual and the stores of C are full lines.  `et` in [0, NT) numbers the calling threads.
// COL_SCALE: column n of the accumulator is first multiplied by col_scale[n] (a power of two).
//
// Epilogue thread -> (column quad, row within a pass), worked out on the host: a kernel that runs each
// phase once feels an integer division (~100 dependent clocks).
struct EpilogueShape {
  int rows_pass;        // rows covered by one pass of the threads
  uint32_t quad_magic;  // et / (tile_n / 4) == (et * quad_magic) >> 16 for et < 256
};
inline EpilogueShape epilogue_shape(int tile_n, int threads) {
  const int quads = tile_n / 4;
  return {threads / quads, (uint32_t)((65536 + quads - 1) / quads)};
}

// preload() may run while the product is still being computed (after the dependency wait): it issues
// the loads that do not depend on it -- bias, column scales, the first row's residual -- whose L2 round
// trip is then off the critical path of a launch that does each phase once.  Only those values stay in
// registers; finish() works the geometry out again (kept live across the accumulator reads it spilled).
// PROJ: the columns are several projections side by side: those below x.rot_cols are heads whose first x.rot features
// get the rotary embedding (pair_rotates), those from x.act_from on the activation.
template <int ACT, int NT, bool COL_SCALE, bool PROJ = false> struct TileEpilogue {
  float4 bvec, cs, rvec;

  // Where this thread works.
  struct Where {
    const float *bias, *res;
    float *C;
    int64_t n_base, m_base;
    int rows_pass, r0, r1, r_end, r, c;
    bool vec, bias_per_col;
    __device__ __forceinline__ Where(const GemmProblem &p, const EpilogueShape &shape, int BN, int tile_m, int tile_n, int split, int S, int z0, int z1, int et) {
      const bool pow2_ranks = (S & (S - 1)) == 0;
      const int rows_per = pow2_ranks ? kBM >> (31 - __clz(S)) : (kBM + S - 1) / S;
      r0 = split * rows_per;
      r1 = min(kBM, r0 + rows_per);
      bias = p.bias ? p.bias + (int64_t)z0 * p.bias_b0 + (int64_t)z1 * p.bias_b1 : nullptr;
      res = p.res ? p.res + (int64_t)z0 * p.res_b0 + (int64_t)z1 * p.res_b1 : nullptr;
      C = p.c + (int64_t)z0 * p.c_b0 + (int64_t)z1 * p.c_b1;
      n_base = (int64_t)tile_n * BN;
      m_base = (int64_t)tile_m * kBM;
      r_end = (int)min((int64_t)r1, p.M - m_base);  // rows that exist
      // 16-byte path: unit column stride everywhere, every row start and the tile origin on a
      // 16-byte boundary, no ragged column edge inside this tile
      auto al4 = [](int64_t v) { return (v & 3) == 0; };
      vec = pow2_ranks && p.c_sn == 1 && al4(p.c_sm) && al4(n_base) && n_base + BN <= p.N && ((reinterpret_cast<uintptr_t>(C) & 15) == 0);
      if (bias) vec = vec && (p.bias_sn == 1 || p.bias_sn == 0) && al4(p.bias_sm) && ((reinterpret_cast<uintptr_t>(bias) & 15) == 0);
      if (res) vec = vec && p.res_sn == 1 && al4(p.res_sm) && ((reinterpret_cast<uintptr_t>(res) & 15) == 0);
      bias_per_col = bias && p.bias_sm == 0 && p.bias_sn == 1;  // the usual [N] bias: loaded once
      // Thread -> (column quad, row within a pass); rows advance by a constant, so every pointer of the
      // loop is stepped with one add per iteration.
      const int quads = BN >> 2, rsub = (int)(((uint32_t)et * shape.quad_magic) >> 16);
      rows_pass = shape.rows_pass;
      c = (et - rsub * quads) * 4;
      r = vec && rsub < rows_pass ? r0 + rsub : kBM;  // threads beyond the last full row of quads stay out
    }
  };

  __device__ __forceinline__ void preload(const GemmProblem &p, const EpilogueShape &shape, int BN, int tile_m, int tile_n, int split, int S, int z0, int z1,
                                          int et, const float *col_scale) {
    bvec = rvec = make_float4(0.f, 0.f, 0.f, 0.f);
    cs = make_float4(1.f, 1.f, 1.f, 1.f);
    const Where w(p, shape, BN, tile_m, tile_n, split, S, z0, z1, et);
    if (w.r >= w.r_end) return;
    if (w.bias_per_col) bvec = *reinterpret_cast<const float4 *>(w.bias + w.n_base + w.c);
    if (COL_SCALE) cs = *reinterpret_cast<const float4 *>(col_scale + w.n_base + w.c);
    if (w.res) rvec = *reinterpret_cast<const float4 *>(w.res + (w.m_base + w.r) * p.res_sm + w.n_base + w.c);
  }

  __device__ __forceinline__ void finish(const GemmProblem &p, const GemmEpilogue &e, const EpilogueShape &shape, float *staging, int pitch, int BN, int tile_m,
                                         int tile_n, int split, int S, int z0, int z1, int et, const float *col_scale, const GemmExtras &x = {}) {
    asm volatile("" : "+r"(tile_m), "+r"(tile_n), "+r"(et));  // recompute: nothing of preload()'s geometry is kept
    const Where w(p, shape, BN, tile_m, tile_n, split, S, z0, z1, et);
    const float *bias = w.bias, *res = w.res;
    float *C = w.C;
    const int64_t n_base = w.n_base, m_base = w.m_base;
    const int r0 = w.r0, r1 = w.r1, r_end = w.r_end, c = w.c;
    const bool bias_per_col = w.bias_per_col;
    const bool scale = e.divisor != 1.0f || e.alpha != 1.0f || (bias && e.beta != 1.0f);
    const float sc_div = e.divisor, sc_alpha = e.alpha, sc_beta = e.beta;
    const uint32_t staging_addr = smem_u32(staging);
    // (an activation that begins inside a group of four columns goes column by column: to decide it here, for every
    // group, cost 77 x 1024 x 7168 in slices 0.8 of 15 us)
    if (w.vec && !(PROJ && (x.act_from & 3))) {
      const int rows_pass = w.rows_pass;
      int r = w.r;
      const int64_t n = n_base + c;
      const float *sp = staging + (size_t)r * pitch + c;
      const int sp_step = rows_pass * pitch;
      float *cp = C + (m_base + r) * p.c_sm + n;
      const int64_t c_step = (int64_t)rows_pass * p.c_sm;
      const float *rp = res ? res + (m_base + r) * p.res_sm + n : nullptr;
      const int64_t r_step = (int64_t)rows_pass * p.res_sm;
      const float *bp = bias ? bias + (m_base + r) * p.bias_sm + (p.bias_sn ? n : 0) : nullptr;
      const int64_t b_step = (int64_t)rows_pass * p.bias_sm;
      const bool act_here = !PROJ || n >= x.act_from;
      // The rotary embedding pairs feature d with d +- rot / 2: the thread rot / 8 quads away in the same row, which is
      // in this warp because rot / 4 quads are an aligned power of two.
      const int feature = PROJ && x.rot && n < x.rot_cols ? (int)n % x.rot_head : 1 << 30;
      const bool rotate = PROJ && feature < x.rot;
      const int span = PROJ ? x.rot >> 2 : 1;
      const unsigned peers = PROJ && rotate ? (span == 32 ? 0xffffffffu : ((1u << span) - 1u) << ((et & 31) & ~(span - 1))) : 0u;
      auto one = [&](float4 acc, float4 bq, float4 rq, int row) {
        if (COL_SCALE) { acc.x *= cs.x; acc.y *= cs.y; acc.z *= cs.z; acc.w *= cs.w; }
        float v[4] = {acc.x, acc.y, acc.z, acc.w};
        const float bv[4] = {bq.x, bq.y, bq.z, bq.w}, rv[4] = {rq.x, rq.y, rq.z, rq.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float y = v[j];
          if (scale) {
            if (sc_div != 1.0f) y = y / sc_div;
            y = bias ? sc_alpha * y + sc_beta * bv[j] : sc_alpha * y;
          } else {
            y += bv[j];
          }
          v[j] = PROJ ? y : act_op<ACT>(e, y) + rv[j];
        }
        if (PROJ) {
          if (rotate) {  // two rounded products and a rounded sum, as rotary_kernel
            const int at = (int)((unsigned)(m_base + row) % (unsigned)x.rot_len) * x.rot + feature;
            const float4 cq = __ldg(reinterpret_cast<const float4 *>(x.rot_cos + at)), sq = __ldg(reinterpret_cast<const float4 *>(x.rot_sin + at));
            const float co[4] = {cq.x, cq.y, cq.z, cq.w}, si[4] = {sq.x, sq.y, sq.z, sq.w};
            const float sgn = feature < (x.rot >> 1) ? -1.0f : 1.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float other = __shfl_xor_sync(peers, v[j], span >> 1);
              v[j] = __fadd_rn(__fmul_rn(v[j], co[j]), __fmul_rn(sgn * other, si[j]));
            }
          }
          if (act_here) {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = act_op<ACT>(e, v[j]);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] += rv[j];
        }
        return make_float4(v[0], v[1], v[2], v[3]);
      };
      if (S == 1 && (!bias || bias_per_col)) {
        // Four rows at a time: their shared-memory and residual loads are all in flight before the first
        // store (the compiler keeps a load behind an earlier store, so row by row every load's latency
        // would be exposed: 32 rows per thread at tile 256).
        while (r + 3 * rows_pass < r_end) {
          float4 acc[4], rq[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            acc[u] = *reinterpret_cast<const float4 *>(sp + u * sp_step);
            rq[u] = res ? *reinterpret_cast<const float4 *>(rp + u * r_step) : make_float4(0.f, 0.f, 0.f, 0.f);
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) *reinterpret_cast<float4 *>(cp + u * c_step) = one(acc[u], bvec, rq[u], r + u * rows_pass);
          r += 4 * rows_pass; sp += 4 * sp_step; cp += 4 * c_step; rp += 4 * r_step;
        }
        if (res && r < r_end) rvec = *reinterpret_cast<const float4 *>(rp);
      }
      auto column_bias = [&]() {  // when it varies by row
        if (p.bias_sn == 1) return *reinterpret_cast<const float4 *>(bp);
        const float t = *bp;
        return make_float4(t, t, t, t);
      };
      if (S == 1) {
        for (; r < r_end; r += rows_pass) {
          const float4 acc = *reinterpret_cast<const float4 *>(sp), rq = rvec;
          if (bias && !bias_per_col) bvec = column_bias();
          rp += r_step;
          if (res && r + rows_pass < r_end) rvec = *reinterpret_cast<const float4 *>(rp);  // the next row's, under this row's arithmetic
          *reinterpret_cast<float4 *>(cp) = one(acc, bvec, rq, r);
          sp += sp_step; cp += c_step; bp += b_step;
        }
      } else {
        // Partial sums of the ranks through distributed shared memory, eight 16-byte loads in flight:
        // 8 / S rows of S ranks.
        const uint32_t own = staging_addr + (uint32_t)(r * pitch + c) * 4u;
        auto rows = [&](auto ranks) {
          constexpr int kRanks = decltype(ranks)::value, kRows = 8 / kRanks;
          uint32_t at[kRanks];
#pragma unroll
          for (int k = 0; k < kRanks; ++k) at[k] = cluster_smem_addr(own, (uint32_t)k);
          while (r < r_end) {
            float4 t[kRows][kRanks], rq[kRows];
            rq[0] = rvec;
#pragma unroll
            for (int u = 0; u < kRows; ++u) {
              const bool live = r + u * rows_pass < r_end;
              if (u > 0) rq[u] = res && live ? *reinterpret_cast<const float4 *>(rp + u * r_step) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
              for (int k = 0; k < kRanks; ++k)
                if (live)
                  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                               : "=f"(t[u][k].x), "=f"(t[u][k].y), "=f"(t[u][k].z), "=f"(t[u][k].w)
                               : "r"(at[k] + (uint32_t)(u * sp_step) * 4u) : "memory");
            }
#pragma unroll
            for (int u = 0; u < kRows; ++u) {
              if (r + u * rows_pass >= r_end) break;
              float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
              for (int k = 0; k < kRanks; ++k) { acc.x += t[u][k].x; acc.y += t[u][k].y; acc.z += t[u][k].z; acc.w += t[u][k].w; }
              if (bias && !bias_per_col) bvec = column_bias();
              *reinterpret_cast<float4 *>(cp) = one(acc, bvec, rq[u], r + u * rows_pass);
              cp += c_step; bp += b_step;
            }
            r += kRows * rows_pass;
            rp += kRows * r_step;
            if (res && r < r_end) rvec = *reinterpret_cast<const float4 *>(rp);
#pragma unroll
            for (int k = 0; k < kRanks; ++k) at[k] += (uint32_t)(kRows * sp_step) * 4u;
          }
        };
        if (S == 2) rows(std::integral_constant<int, 2>());
        else if (S == 4) rows(std::integral_constant<int, 4>());
        else rows(std::integral_constant<int, 8>());
      }
    } else {
      // ragged column edge or non-unit strides: one element at a time, indices recomputed
      const int quads = BN >> 2, count = (r1 - r0) * quads;
      for (int i = et; i < count; i += NT) {
        const int rr = i / quads, row = r0 + rr, col = (i - rr * quads) * 4;
        const int64_t m = m_base + row;
        if (m >= p.M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int64_t n = n_base + col + j;
          if (n >= p.N) continue;
          float acc = 0.0f;
          const uint32_t off = staging_addr + (uint32_t)(row * pitch + col + j) * 4u;
          if (S == 1) acc = staging[(size_t)row * pitch + col + j];
          else
            for (int rank = 0; rank < S; ++rank) acc += ld_cluster_f32(cluster_smem_addr(off, (uint32_t)rank));
          if (COL_SCALE) acc *= col_scale[n];
          const float bv = bias ? bias[m * p.bias_sm + n * p.bias_sn] : 0.0f;
          const float rv = res ? res[m * p.res_sm + n * p.res_sn] : 0.0f;
          float y = acc;
          if (scale) {
            if (sc_div != 1.0f) y = y / sc_div;
            y = bias ? sc_alpha * y + sc_beta * bv : sc_alpha * y;
          } else {
            y += bv;
          }
          C[m * p.c_sm + n * p.c_sn] = (PROJ && n < x.act_from ? y : act_op<ACT>(e, y)) + rv;
        }
      }
    }
  }
};

}  // namespace fml

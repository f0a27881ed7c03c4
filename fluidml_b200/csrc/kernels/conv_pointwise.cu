// Pointwise convolutions with little arithmetic on the CUDA cores: y[n, oc, p] = act(sum_ic w[oc, ic] (x[n, ic, p] s[n, ic])
// + b[oc]) + r[n, oc, p], in fp32 FMA.
//
// What bounds it: latency.  A layer of EfficientNet at one image has 3 to 20 million multiply-adds -- a microsecond of one
// SM in five's FMA units -- and the tensor-core kernel spends 8 to 11 us on it (patch, split into pairs, tensor memory,
// staged epilogue, split-K over a cluster).  Here a CTA owns 32 output channels x PX pixels; both operands are read as
// they lie (x [IC][pixels], w [IC][OC]: a row of each per input channel), every row of its k range is on its way at once
// by asynchronous copies, constant weights' before the preceding kernel has finished, and a lane multiplies 8 channels x 4
// pixels in f32x2 pairs (3 shared-memory reads of 16 bytes for 16 instructions).  The eight warps take different pixels,
// or share the pixels and take WK slices of k, added in slice order through shared memory; a cluster of S CTAs splits k
// further where the tiles alone leave most SMs idle (7 x 7 maps), its partial tiles added in rank order.
//
// Captured graphs, this kernel / the packed-weight one with tuned tiles, us: one image 96 -> 24 channels at 56 x 56 with
// gate 3.9 / 6.6, 144 -> 40 at 28 x 28 4.5 / 7.2, 80 -> 480 at 14 x 14 4.3 / 6.7, 1152 -> 320 at 7 x 7 7.2 / 10.5, the
// nineteen shapes of EfficientNet-B0 102 / 145 (and 1e-7 of the largest value off fp64 against 4e-7); five of 192 x 192
// 184 / 179, the better of the two per layer 160; sixteen 472 / 266.  So the two are timed against each other where
// Compile tunes; without tuning this kernel runs what its model puts below 6 us, and maps the packed kernel does not take
// (4 x 4: 5.9 us, 400 on the general path).
#include "gemm_common.cuh"
#include "tc_common.cuh"
#include <algorithm>

namespace fml {
namespace {

constexpr int kPwThreads = 256;
constexpr int kPwOC = 32;

struct PwArgs {
  const float *x, *w, *bias, *scale, *res;
  float *y;
  int OC, IC, HW, tiles_px, k_per_cta, k_chunk;
  int64_t x_sn, x_sc, y_sn, y_sc, w_sc, scale_sn, scale_sc, bias_stride;
  int act, w_constant;
};

__device__ __forceinline__ void cp16_or_zero(unsigned dst, const float *src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp4_or_zero(unsigned dst, const float *src, bool live) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(live ? 4 : 0) : "memory");
}
__device__ __forceinline__ void pw_fma2(unsigned long long &acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float pw_act(int act, float v) {
  switch (act) {
  case FML_ACT_RELU: return fmaxf(v, 0.0f);
  case FML_ACT_TANH: return tanhf(v);
  case FML_ACT_SIGMOID: return 1.0f / (1.0f + expf(-v));
  case FML_ACT_SILU: return v / (1.0f + expf(-v));
  default: return v;
  }
}

// WK: slices of k among the warps (the other 8 / WK take 32 pixels each).  VEC: rows of x and y on 16-byte boundaries.
template <int WK, bool VEC>
__global__ void __launch_bounds__(kPwThreads, 2) conv_pointwise_kernel(const PwArgs a) {
  constexpr int PX = 32 * (8 / WK);
  extern __shared__ __align__(16) float smem[];
  const int S = gridDim.z, rank = blockIdx.z;  // (one cluster along z)
  const int kc = a.k_chunk;
  float *const Wb = smem;                         // [2][kc][32]
  float *const Xb = Wb + 2 * kc * kPwOC;          // [2][kc][PX]
  float *const Gs = Xb + 2 * kc * PX;             // [k_per_cta] scales, if any
  float *const Red = smem;                        // [WK][8 / WK][32][32] at the end
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int img = blockIdx.x / a.tiles_px, p0 = (blockIdx.x - img * a.tiles_px) * PX, oc0 = blockIdx.y * kPwOC;
  const int k0 = rank * a.k_per_cta, k1 = min(a.IC, k0 + a.k_per_cta), nk = max(0, k1 - k0);
  const int px = min(PX, a.HW - p0);
  const float *const xp = a.x + (int64_t)img * a.x_sn + (int64_t)k0 * a.x_sc + p0;
  const float *const wp = a.w + (int64_t)k0 * a.w_sc + oc0;

  auto load_w = [&](int c, int buf) {  // 8 copies of 16 bytes per row
    const int rows = min(kc, nk - c * kc), col = (t & 7) * 4;
    const bool live = oc0 + col < a.OC;
    unsigned dst = (unsigned)__cvta_generic_to_shared(Wb + buf * kc * kPwOC + (t >> 3) * kPwOC + col);
    const float *src = wp + (int64_t)(c * kc + (t >> 3)) * a.w_sc + (live ? col : 0);
    for (int r = t >> 3; r < rows; r += kPwThreads / 8, dst += (kPwThreads / 8) * kPwOC * 4, src += (int64_t)(kPwThreads / 8) * a.w_sc) cp16_or_zero(dst, src, live);
  };
  auto load_x = [&](int c, int buf) {
    const int rows = min(kc, nk - c * kc);
    if (VEC) {
      constexpr int per = PX / 4, step = kPwThreads / per;
      const int col = (t % per) * 4;
      const bool live = col < px;  // (HW is a multiple of 4)
      unsigned dst = (unsigned)__cvta_generic_to_shared(Xb + buf * kc * PX + (t / per) * PX + col);
      const float *src = xp + (int64_t)(c * kc + t / per) * a.x_sc + (live ? col : 0);
      for (int r = t / per; r < rows; r += step, dst += step * PX * 4, src += (int64_t)step * a.x_sc) cp16_or_zero(dst, src, live);
    } else {
      constexpr int step = kPwThreads / PX > 0 ? kPwThreads / PX : 1;
      const int col = t % PX;
      const bool live = col < px;
      unsigned dst = (unsigned)__cvta_generic_to_shared(Xb + buf * kc * PX + (t / PX) * PX + col);
      const float *src = xp + (int64_t)(c * kc + t / PX) * a.x_sc + (live ? col : 0);
      for (int r = t / PX; r < rows; r += step, dst += step * PX * 4, src += (int64_t)step * a.x_sc) cp4_or_zero(dst, src, live);
    }
  };
  auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };

  const int chunks = (nk + kc - 1) / kc;
  pdl_launch_dependents();
  if (chunks > 0 && a.w_constant) load_w(0, 0);
  pdl_wait();
  if (chunks > 0 && !a.w_constant) load_w(0, 0);
  if (chunks > 0) load_x(0, 0);
  commit();
  if (a.scale)
    for (int k = t; k < nk; k += kPwThreads) Gs[k] = a.scale[(int64_t)img * a.scale_sn + (int64_t)(k0 + k) * a.scale_sc];

  const int wk = warp % WK, wpx = warp / WK, og = (lane >> 3) * 8, pg = (lane & 7) * 4;
  unsigned long long acc[4][4];  // [pixel][channel pair]
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
  for (int c = 0; c < chunks; ++c) {
    const int buf = c & 1, rows = min(kc, nk - c * kc);
    if (c + 1 < chunks) { load_w(c + 1, buf ^ 1); load_x(c + 1, buf ^ 1); commit(); asm volatile("cp.async.wait_group 1;" ::: "memory"); }
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const float *W = Wb + buf * kc * kPwOC + og, *X = Xb + buf * kc * PX + wpx * 32 + pg, *G = Gs + c * kc;
#pragma unroll 2
    for (int k = wk; k < rows; k += WK) {
      const ulonglong2 w0 = *reinterpret_cast<const ulonglong2 *>(W + k * kPwOC), w1 = *reinterpret_cast<const ulonglong2 *>(W + k * kPwOC + 4);
      float4 xv = *reinterpret_cast<const float4 *>(X + k * PX);
      if (a.scale) {
        const float g = G[k];
        xv = make_float4(__fmul_rn(xv.x, g), __fmul_rn(xv.y, g), __fmul_rn(xv.z, g), __fmul_rn(xv.w, g));
      }
      const float xs[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        unsigned long long x2;
        asm("mov.b64 %0, {%1, %1};" : "=l"(x2) : "f"(xs[i]));
        pw_fma2(acc[i][0], x2, w0.x); pw_fma2(acc[i][1], x2, w0.y);
        pw_fma2(acc[i][2], x2, w1.x); pw_fma2(acc[i][3], x2, w1.y);
      }
    }
    __syncthreads();  // this buffer is loaded again after the next chunk, and Red lies over both
  }
  // channel og + j, pixels pg .. pg + 3 of this lane
  auto row_of = [&](int j) {
    float4 v;
    float lo[4], hi[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) asm("mov.b64 {%0, %1}, %2;" : "=f"(lo[i]), "=f"(hi[i]) : "l"(acc[i][j >> 1]));
    v = (j & 1) ? make_float4(hi[0], hi[1], hi[2], hi[3]) : make_float4(lo[0], lo[1], lo[2], lo[3]);
    return v;
  };
  auto finish = [&](float4 v, int oc, int p) {  // p: pixel within the tile
    oc += oc0;
    if (oc >= a.OC || p >= px) return;
    const float b = a.bias ? a.bias[(int64_t)oc * a.bias_stride] : 0.0f;
    const int64_t at = (int64_t)img * a.y_sn + (int64_t)oc * a.y_sc + p0 + p;
    float o[4] = {pw_act(a.act, v.x + b), pw_act(a.act, v.y + b), pw_act(a.act, v.z + b), pw_act(a.act, v.w + b)};
    if (VEC) {
      if (a.res) {
        const float4 r = *reinterpret_cast<const float4 *>(a.res + at);
        o[0] += r.x; o[1] += r.y; o[2] += r.z; o[3] += r.w;
      }
      *reinterpret_cast<float4 *>(a.y + at) = make_float4(o[0], o[1], o[2], o[3]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (p + i < px) a.y[at + i] = a.res ? o[i] + a.res[at + i] : o[i];
    }
  };
  if (WK == 1 && S == 1) {
#pragma unroll
    for (int j = 0; j < 8; ++j) finish(row_of(j), og + j, wpx * 32 + pg);
    return;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) *reinterpret_cast<float4 *>(Red + ((wk * (8 / WK) + wpx) * 32 + og + j) * 32 + pg) = row_of(j);
  __syncthreads();
  // 8 x PX groups of four pixels; thread t takes group t, t + 256, ..
  float4 sum[8 / WK];
#pragma unroll
  for (int u = 0; u < 8 / WK; ++u) {
    const float *r = Red + (t + u * kPwThreads) * 4;
    sum[u] = *reinterpret_cast<const float4 *>(r);
#pragma unroll
    for (int k = 1; k < WK; ++k) {
      const float4 v = *reinterpret_cast<const float4 *>(r + k * (8 / WK) * 1024);
      sum[u].x += v.x; sum[u].y += v.y; sum[u].z += v.z; sum[u].w += v.w;
    }
  }
  if (S > 1) {
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 8 / WK; ++u) *reinterpret_cast<float4 *>(Red + (t + u * kPwThreads) * 4) = sum[u];
    cluster_sync_all();
    // groups are shared out among the ranks: rank takes those whose index modulo S is its own
    const int groups = 8 * PX;
    for (int i = t * S + rank; i < groups; i += kPwThreads * S) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int r = 0; r < S; ++r) {
        float4 q;
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(q.x), "=f"(q.y), "=f"(q.z), "=f"(q.w)
                     : "r"(cluster_smem_addr(smem_u32(Red + i * 4), (uint32_t)r)) : "memory");
        v.x += q.x; v.y += q.y; v.z += q.z; v.w += q.w;
      }
      const int rest = i & 255;  // [pixel group of 32][channel][four pixels]
      finish(v, rest >> 3, (i >> 8) * 32 + (rest & 7) * 4);
    }
    cluster_sync_relaxed();  // remote reads of this CTA's memory are over
    return;
  }
#pragma unroll
  for (int u = 0; u < 8 / WK; ++u) {
    const int i = t + u * kPwThreads, rest = i & 255;
    finish(sum[u], rest >> 3, (i >> 8) * 32 + (rest & 7) * 4);
  }
}

struct PwPlan { int wk, split, k_per_cta, k_chunk; size_t smem; };

// Time model in microseconds: fixed phases, then waves of CTAs (two to an SM) at its FMA rate.
bool plan_pointwise(int64_t n, int64_t hw, int64_t oc, int64_t ic, bool scaled, int want_wk, int want_split, PwPlan *best, double *us) {
  double best_us = 1e30;
  for (int wk : {1, 2, 4, 8})
    for (int split : {1, 2, 4, 8}) {
      if (want_wk && (wk != want_wk || split != want_split)) continue;
      if (split > 1 && (wk != 8 || ic < 32 * split)) continue;
      const int px = 32 * (8 / wk);
      const int64_t k = (ic + split - 1) / split;
      const int64_t ctas = n * ((hw + px - 1) / px) * ((oc + kPwOC - 1) / kPwOC) * split;
      if (ctas > (1ll << 30)) continue;
      const int chunk = (int)std::min<int64_t>(k, std::max(16, 40 * 1024 / ((kPwOC + px) * 4) / 8 * 8));
      const size_t smem = std::max(2 * (size_t)chunk * (kPwOC + px) * 4 + (scaled ? (size_t)k * 4 : 0), (size_t)8 * 4096);
      if (smem > 110 * 1024) continue;
      const double per = (double)kPwOC * px * (double)k / 128.0 / 1900.0 * 1.25;  // one CTA alone on an SM
      const double waves = (double)ctas / kSms;
      const double t = 2.2 + (wk > 1 ? 0.3 : 0.0) + (split > 1 ? 1.0 : 0.0) + 0.25 * (double)((k + chunk - 1) / chunk) + per * std::max(1.0, waves);
      if (t < best_us) { best_us = t; *best = {wk, split, (int)k, chunk, smem}; }
    }
  *us = best_us;
  return best_us < 1e30;
}

}  // namespace

// Whether the layer is one this kernel takes at all.
static bool pointwise_shape_ok(const fml_tensor *x, const fml_tensor *w, const fml_tensor *y, const fml_conv_params *p) {
  if (x->rank != 4 || w->rank != 4 || y->rank != 4 || x->dtype != FML_F32 || w->dtype != FML_F32 || y->dtype != FML_F32) return false;
  if (p->group > 1 || w->shape[2] != 1 || w->shape[3] != 1 || p->pads_begin[0] || p->pads_begin[1]) return false;
  if (p->strides[0] != 1 || p->strides[1] != 1 || p->act < FML_ACT_NONE || p->act > FML_ACT_SILU || p->act == FML_ACT_GELU_ERF) return false;
  if (p->precision != FML_GEMM_AUTO && p->precision != FML_GEMM_FP32) return false;
  const int64_t OC = w->shape[0], IC = w->shape[1], HW = x->shape[2] * x->shape[3];
  if (x->shape[1] != IC || y->shape[1] != OC || y->shape[0] != x->shape[0] || y->shape[2] != x->shape[2] || y->shape[3] != x->shape[3]) return false;
  if (w->stride[0] != 1 || OC % 4 || w->stride[1] % 4 || !aligned16(w->data) || HW < 2 || IC < 1) return false;
  auto planes = [](const fml_tensor *t) { return t->stride[3] == 1 && t->stride[2] == t->shape[3] && t->stride[1] > 0 && t->stride[0] >= 0; };
  return planes(x) && planes(y) && HW < (1ll << 30) && OC < (1ll << 20) && IC < (1ll << 20);
}

bool pointwise_fma_plan(const fml_tensor *x, const fml_tensor *w, const fml_tensor *y, const fml_conv_params *p, bool scaled, double *us) {
  PwPlan plan;
  return pointwise_shape_ok(x, w, y, p) && plan_pointwise(x->shape[0], x->shape[2] * x->shape[3], w->shape[0], w->shape[1], scaled, 0, 0, &plan, us);
}

int launch_pointwise_fma(const fml_tensor *x, const fml_tensor *w, const fml_tensor *bias, const fml_tensor *y, const fml_conv_params *p, cudaStream_t s,
                         const float *x_scale, int64_t x_scale_sn, int64_t x_scale_sc, const float *residual) {
  PwPlan plan;
  double us;
  const int64_t HW = x->shape[2] * x->shape[3];
  auto planned = [&](int wk, int split) { return plan_pointwise(x->shape[0], HW, w->shape[0], w->shape[1], x_scale != nullptr, wk, split, &plan, &us); };
  FML_REQUIRE(pointwise_shape_ok(x, w, y, p) && ((p->tile_n && planned(p->tile_n, p->split_k)) || planned(0, 0)),  // an impossible split: the model's
              FML_UNSUPPORTED, "fml_conv: not a pointwise layer of the FMA kernel");
  PwArgs a;
  a.x = (const float *)x->data; a.w = (const float *)w->data; a.y = (float *)y->data;
  a.bias = bias ? (const float *)bias->data : nullptr;
  a.bias_stride = 0;
  if (bias)
    for (int i = 0; i < bias->rank; ++i) if (bias->shape[i] != 1) a.bias_stride = bias->stride[i];
  a.scale = x_scale; a.scale_sn = x_scale_sn; a.scale_sc = x_scale_sc;
  a.res = residual;
  a.OC = (int)w->shape[0]; a.IC = (int)w->shape[1]; a.HW = (int)HW;
  a.x_sn = x->stride[0]; a.x_sc = x->stride[1]; a.y_sn = y->stride[0]; a.y_sc = y->stride[1]; a.w_sc = w->stride[1];
  a.act = p->act;
  a.w_constant = p->w_constant;
  a.k_per_cta = plan.k_per_cta; a.k_chunk = plan.k_chunk;
  const int px = 32 * (8 / plan.wk);
  a.tiles_px = (int)((HW + px - 1) / px);
  const int64_t tiles = (int64_t)a.tiles_px * x->shape[0], oc_tiles = (a.OC + kPwOC - 1) / kPwOC;
  FML_REQUIRE(tiles < (1ll << 31) && oc_tiles <= 65535, FML_UNSUPPORTED, "fml_conv: too many tiles");
  auto vec4 = [](int64_t v) { return v % 4 == 0; };
  const bool vec = HW % 4 == 0 && vec4(a.x_sn) && vec4(a.x_sc) && vec4(a.y_sn) && vec4(a.y_sc) && aligned16(a.x) && aligned16(a.y) && (!a.res || aligned16(a.res));
  using KernelFn = void (*)(const PwArgs);
  static const KernelFn kernels[4][2] = {{conv_pointwise_kernel<1, false>, conv_pointwise_kernel<1, true>}, {conv_pointwise_kernel<2, false>, conv_pointwise_kernel<2, true>},
                                         {conv_pointwise_kernel<4, false>, conv_pointwise_kernel<4, true>}, {conv_pointwise_kernel<8, false>, conv_pointwise_kernel<8, true>}};
  const KernelFn kernel = kernels[plan.wk == 1 ? 0 : plan.wk == 2 ? 1 : plan.wk == 4 ? 2 : 3][vec ? 1 : 0];
  static bool attr_set[64] = {false};
  int dev = 0;
  FML_CUDA(cudaGetDevice(&dev));
  if (!attr_set[dev & 63]) {
    for (const auto &row : kernels)
      for (KernelFn k : row) FML_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024));
    attr_set[dev & 63] = true;
  }
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)tiles, (unsigned)oc_tiles, (unsigned)plan.split);
  cfg.blockDim = dim3(kPwThreads);
  cfg.dynamicSmemBytes = plan.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = (unsigned)plan.split;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  FML_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
  return FML_OK;
}

}  // namespace fml

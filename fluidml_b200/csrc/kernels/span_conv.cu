// Span-based dynamic convolution of ConvBERT in one launch:
//
//   out[b, s, h, :] = sum_j softmax_j(logits[b, s, h, :])[j] * x[b, s + j - pad, h, :]        j = 0 .. K - 1, zero outside
//
// which the exported graph writes as Softmax over K taps, Pad of x along the sequence, K slices of either and a chain of
// Mul / Add: four launches that write and read the padded copy and the weights and read x K times from L2 (25 us a layer
// at 8 x 128 x 384).  Here a CTA takes kSpanRows positions: their softmaxes first (one thread each, in shared memory),
// then every thread runs down the positions with the K rows of its four features in registers, so x is read once.  The
// products and partial sums are rounded one by one in tap order, as the chain rounds them.  What bounds it: two
// dependent L2 round trips (logits, x -- both asked for at the start) and the launch.  8 x 128 x 6 heads of 64, nine taps,
// inside a ConvBERT pass: 4.6 us where Softmax 5.5, Pad 3.5 and the sum of products 12.4 were.
#include "common.cuh"
#include <algorithm>

namespace fml {
namespace {

constexpr int kSpanRows = 8;
constexpr int kSpanThreads = 128;

struct SpanArgs {
  const float *x, *logits;
  float *out;
  int S, heads, D, pad, quads;  // quads: groups of V features of a head
  int64_t x_s[4], l_s[4], o_s[4];
};

template <int K, int V>
__global__ void __launch_bounds__(kSpanThreads) span_conv_kernel(SpanArgs a) {
  extern __shared__ float w[];  // [kSpanRows][heads][K]
  pdl_prologue();
  const int b = blockIdx.y, s0 = blockIdx.x * kSpanRows, rows = min(kSpanRows, a.S - s0);
  const int units = a.heads * a.quads;
  constexpr int R = kSpanRows + K - 1;
  float xv[R][V];
  // rows s0 - pad .. of this thread's first features, on their way during the softmaxes
  auto load = [&](int u) {
    const int h = u / a.quads, d = (u - h * a.quads) * V;
    const float *p = a.x + b * a.x_s[0] + (int64_t)(s0 - a.pad) * a.x_s[1] + h * a.x_s[2] + d * a.x_s[3];
#pragma unroll
    for (int r = 0; r < R; ++r, p += a.x_s[1]) {
      const int s = s0 - a.pad + r;
#pragma unroll
      for (int v = 0; v < V; ++v) xv[r][v] = 0.0f;
      if (s < 0 || s >= a.S) continue;
      if (V == 4) {
        const float4 t = *reinterpret_cast<const float4 *>(p);
        xv[r][0] = t.x; xv[r][1] = t.y; xv[r][2] = t.z; xv[r][V - 1] = t.w;
      } else {
        xv[r][0] = *p;
      }
    }
  };
  int u = blockIdx.z * kSpanThreads + threadIdx.x;
  if (u < units) load(u);
  for (int i = threadIdx.x; i < rows * a.heads; i += kSpanThreads) {
    const int r = i / a.heads, h = i - r * a.heads;
    const float *l = a.logits + b * a.l_s[0] + (int64_t)(s0 + r) * a.l_s[1] + h * a.l_s[2];
    float t[K], m = -3.402823466e+38f, sum = 0.0f;
#pragma unroll
    for (int j = 0; j < K; ++j) { t[j] = l[j * a.l_s[3]]; m = fmaxf(m, t[j]); }
#pragma unroll
    for (int j = 0; j < K; ++j) { t[j] = expf(t[j] - m); sum += t[j]; }
#pragma unroll
    for (int j = 0; j < K; ++j) w[i * K + j] = t[j] / sum;
  }
  __syncthreads();
  const int step = gridDim.z * kSpanThreads;
  for (; u < units;) {
    const int h = u / a.quads, d = (u - h * a.quads) * V;
    float *o = a.out + b * a.o_s[0] + (int64_t)s0 * a.o_s[1] + h * a.o_s[2] + d * a.o_s[3];
#pragma unroll
    for (int r = 0; r < kSpanRows; ++r, o += a.o_s[1]) {
      if (r >= rows) break;
      const float *wr = w + (r * a.heads + h) * K;
      float acc[V];
#pragma unroll
      for (int v = 0; v < V; ++v) acc[v] = __fmul_rn(xv[r][v], wr[0]);
#pragma unroll
      for (int j = 1; j < K; ++j)
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] = __fadd_rn(acc[v], __fmul_rn(xv[r + j][v], wr[j]));
      if (V == 4) *reinterpret_cast<float4 *>(o) = make_float4(acc[0], acc[1], acc[2], acc[V - 1]);
      else *o = acc[0];
    }
    u += step;
    if (u < units) load(u);
  }
}

}  // namespace
}  // namespace fml

using namespace fml;

extern "C" int fml_span_convolution_supported(int64_t taps) { return taps == 3 || taps == 5 || taps == 7 || taps == 9; }

extern "C" int fml_span_convolution(const fml_tensor *x, const fml_tensor *logits, int64_t pad, const fml_tensor *out, void *stream) {
  FML_REQUIRE(valid_tensor(x) && valid_tensor(logits) && valid_tensor(out), FML_BAD_ARG, "fml_span_convolution: bad tensor");
  FML_REQUIRE(x->dtype == FML_F32 && logits->dtype == FML_F32 && out->dtype == FML_F32 && x->rank == 4 && logits->rank == 4 && out->rank == 4,
              FML_UNSUPPORTED, "fml_span_convolution: fp32 [batch, length, heads, features] only");
  SpanArgs a;
  for (int i = 0; i < 4; ++i) {
    FML_REQUIRE(out->shape[i] == x->shape[i] && (i == 3 || logits->shape[i] == x->shape[i]), FML_BAD_ARG, "fml_span_convolution: shapes");
    a.x_s[i] = x->stride[i]; a.l_s[i] = logits->stride[i]; a.o_s[i] = out->stride[i];
  }
  const int64_t B = x->shape[0], S = x->shape[1], heads = x->shape[2], D = x->shape[3], K = logits->shape[3];
  FML_REQUIRE(fml_span_convolution_supported(K) && pad >= 0 && pad < K, FML_UNSUPPORTED, "fml_span_convolution: 3, 5, 7 or 9 taps");
  if (B * S * heads * D == 0) return FML_OK;
  FML_REQUIRE(B <= 65535 && S < (1ll << 30) && heads <= 512 && D < (1 << 20), FML_UNSUPPORTED, "fml_span_convolution: sizes");
  a.x = (const float *)x->data; a.logits = (const float *)logits->data; a.out = (float *)out->data;
  a.S = (int)S; a.heads = (int)heads; a.D = (int)D; a.pad = (int)pad;
  auto al4 = [](const int64_t *s) { return s[0] % 4 == 0 && s[1] % 4 == 0 && s[2] % 4 == 0 && s[3] == 1; };
  const bool vec = D % 4 == 0 && al4(a.x_s) && al4(a.o_s) && aligned16(a.x) && aligned16(a.out);
  a.quads = (int)(vec ? D / 4 : D);
  const int64_t units = heads * a.quads;
  const dim3 grid((unsigned)((S + kSpanRows - 1) / kSpanRows), (unsigned)B, (unsigned)std::min<int64_t>(64, (units + kSpanThreads - 1) / kSpanThreads));
  const size_t smem = (size_t)kSpanRows * heads * K * sizeof(float);
  FML_REQUIRE(smem <= 48 * 1024, FML_UNSUPPORTED, "fml_span_convolution: heads x taps");
  using KernelFn = void (*)(SpanArgs);
  static const KernelFn kernels[4][2] = {{span_conv_kernel<3, 1>, span_conv_kernel<3, 4>}, {span_conv_kernel<5, 1>, span_conv_kernel<5, 4>},
                                         {span_conv_kernel<7, 1>, span_conv_kernel<7, 4>}, {span_conv_kernel<9, 1>, span_conv_kernel<9, 4>}};
  FML_LAUNCH(kernels[(K - 3) / 2][vec ? 1 : 0], grid, kSpanThreads, smem, as_stream(stream), a);
  return FML_OK;
}

// GEMM front end: shape analysis, the fp32 FMA kernel for operands the tensor-core path
// cannot take (arbitrary strides, tiny or unaligned shapes), and the C-ABI entry points.
#include "gemm_common.cuh"
#include <map>
#include <mutex>
#include <string>
#include <vector>

namespace fml {

int analyse_gemm(const fml_tensor *a, const fml_tensor *b, const fml_tensor *c,
                 const fml_tensor *bias, const fml_tensor *res, GemmProblem &p) {
  FML_REQUIRE(valid_tensor(a) && valid_tensor(b) && valid_tensor(c), FML_BAD_ARG, "fml_gemm: bad tensor");
  FML_REQUIRE(a->dtype == FML_F32 && b->dtype == FML_F32 && c->dtype == FML_F32, FML_UNSUPPORTED,
              "fml_gemm: fp32 only");
  FML_REQUIRE(a->rank >= 2 && b->rank >= 2 && c->rank >= 2 && a->rank <= c->rank && b->rank <= c->rank,
              FML_BAD_ARG, "fml_gemm: operand ranks");
  const int r = c->rank;
  p.prefetch = nullptr;
  p.prefetch_bytes = 0;
  p.b_constant = 0;
  p.M = c->shape[r - 2];
  p.N = c->shape[r - 1];
  p.K = a->shape[a->rank - 1];
  FML_REQUIRE(a->shape[a->rank - 2] == p.M && b->shape[b->rank - 2] == p.K && b->shape[b->rank - 1] == p.N,
              FML_BAD_ARG, "fml_gemm: inner dimensions do not match");
  p.a = (const float *)a->data; p.b = (const float *)b->data; p.c = (float *)c->data;
  p.bias = bias ? (const float *)bias->data : nullptr;
  p.res = res ? (const float *)res->data : nullptr;
  p.a_sm = a->stride[a->rank - 2]; p.a_sk = a->stride[a->rank - 1];
  p.b_sk = b->stride[b->rank - 2]; p.b_sn = b->stride[b->rank - 1];
  p.c_sm = c->stride[r - 2]; p.c_sn = c->stride[r - 1];
  int64_t bias_s[kMaxDims] = {0}, res_s[kMaxDims] = {0};
  if (bias) {
    FML_REQUIRE(valid_tensor(bias) && bias->dtype == FML_F32 && broadcast_strides(bias, c, bias_s),
                FML_BAD_ARG, "fml_gemm: bias does not broadcast to the output");
  }
  if (res) {
    FML_REQUIRE(valid_tensor(res) && res->dtype == FML_F32 && broadcast_strides(res, c, res_s),
                FML_BAD_ARG, "fml_gemm: residual does not broadcast to the output");
  }
  p.bias_sm = bias_s[r - 2]; p.bias_sn = bias_s[r - 1];
  p.res_sm = res_s[r - 2]; p.res_sn = res_s[r - 1];

  // batch dims, outermost first; operand 0..4 = c, a, b, bias, res
  Iter<5> it;
  it.rank = r - 2;
  for (int i = 0; i < r - 2; ++i) {
    it.shape[i] = c->shape[i];
    it.stride[0][i] = c->stride[i];
    const int ia = i - (r - a->rank), ib = i - (r - b->rank);
    if (ia >= 0) FML_REQUIRE(a->shape[ia] == c->shape[i] || a->shape[ia] == 1, FML_BAD_ARG, "fml_gemm: batch dims of A");
    if (ib >= 0) FML_REQUIRE(b->shape[ib] == c->shape[i] || b->shape[ib] == 1, FML_BAD_ARG, "fml_gemm: batch dims of B");
    it.stride[1][i] = (ia >= 0 && a->shape[ia] != 1) ? a->stride[ia] : 0;
    it.stride[2][i] = (ib >= 0 && b->shape[ib] != 1) ? b->stride[ib] : 0;
    it.stride[3][i] = bias_s[i];
    it.stride[4][i] = res_s[i];
  }
  if (it.rank == 0) { it.rank = 1; it.shape[0] = 1; for (int o = 0; o < 5; ++o) it.stride[o][0] = 0; }
  collapse(it);
  // fold the innermost batch dim into M when B does not vary over it and rows continue
  while (it.rank >= 1 && it.shape[it.rank - 1] > 1) {
    const int l = it.rank - 1;
    const bool ok = it.stride[2][l] == 0 && it.stride[0][l] == p.M * p.c_sm &&
                    it.stride[1][l] == p.M * p.a_sm &&
                    (!bias || it.stride[3][l] == p.M * p.bias_sm) &&
                    (!res || it.stride[4][l] == p.M * p.res_sm);
    if (!ok) break;
    p.M *= it.shape[l];
    if (it.rank == 1) { it.shape[0] = 1; for (int o = 0; o < 5; ++o) it.stride[o][0] = 0; }
    else --it.rank;
  }
  FML_REQUIRE(it.rank <= 2, FML_UNSUPPORTED, "fml_gemm: more than two independent batch dims");
  const int l = it.rank - 1;
  p.nb0 = it.shape[l];
  p.c_b0 = it.stride[0][l]; p.a_b0 = it.stride[1][l]; p.b_b0 = it.stride[2][l];
  p.bias_b0 = it.stride[3][l]; p.res_b0 = it.stride[4][l];
  if (it.rank == 2) {
    p.nb1 = it.shape[0];
    p.c_b1 = it.stride[0][0]; p.a_b1 = it.stride[1][0]; p.b_b1 = it.stride[2][0];
    p.bias_b1 = it.stride[3][0]; p.res_b1 = it.stride[4][0];
  } else {
    p.nb1 = 1;
    p.c_b1 = p.a_b1 = p.b_b1 = p.bias_b1 = p.res_b1 = 0;
  }
  return FML_OK;
}

namespace {

// 64x64 output tile, 16-deep k slab, 256 threads with a 4x4 micro-tile each.  Operands are
// read with their element strides, so any layout works; the k-fast / m-fast thread mapping
// of the loads follows whichever stride is 1.
constexpr int SB = 64, SK = 16;

__global__ void __launch_bounds__(256) gemm_simt_kernel(GemmProblem p, GemmEpilogue e) {
  pdl_prologue();
  __shared__ float As[SK][SB + 4];
  __shared__ float Bs[SK][SB + 4];
  const int64_t z = blockIdx.z, z0 = z % p.nb0, z1 = z / p.nb0;
  const float *A = p.a + z0 * p.a_b0 + z1 * p.a_b1;
  const float *B = p.b + z0 * p.b_b0 + z1 * p.b_b1;
  const int64_t m0 = (int64_t)blockIdx.y * SB, n0 = (int64_t)blockIdx.x * SB;
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  float acc[4][4] = {};
  const bool a_kfast = p.a_sk == 1, b_nfast = p.b_sn == 1;
  for (int64_t k0 = 0; k0 < p.K; k0 += SK) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e_ = t + i * 256;
      int mm, kk;
      if (a_kfast) { kk = e_ & 15; mm = e_ >> 4; } else { mm = e_ & 63; kk = e_ >> 6; }
      const int64_t gm = m0 + mm, gk = k0 + kk;
      As[kk][mm] = (gm < p.M && gk < p.K) ? A[gm * p.a_sm + gk * p.a_sk] : 0.0f;
      int nn, kb;
      if (b_nfast) { nn = e_ & 63; kb = e_ >> 6; } else { kb = e_ & 15; nn = e_ >> 4; }
      const int64_t gn = n0 + nn, gkb = k0 + kb;
      Bs[kb][nn] = (gn < p.N && gkb < p.K) ? B[gkb * p.b_sk + gn * p.b_sn] : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < SK; ++kk) {
      float av[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { av[i] = As[kk][ty * 4 + i]; bv[i] = Bs[kk][tx * 4 + i]; }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    __syncthreads();
  }
  float *C = p.c + z0 * p.c_b0 + z1 * p.c_b1;
  const float *bias = p.bias ? p.bias + z0 * p.bias_b0 + z1 * p.bias_b1 : nullptr;
  const float *res = p.res ? p.res + z0 * p.res_b0 + z1 * p.res_b1 : nullptr;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t m = m0 + ty * 4 + i, n = n0 + tx * 4 + j;
      if (m < p.M && n < p.N) {
        const float bv = bias ? bias[m * p.bias_sm + n * p.bias_sn] : 0.0f;
        const float rv = res ? res[m * p.res_sm + n * p.res_sn] : 0.0f;
        C[m * p.c_sm + n * p.c_sn] = gemm_epilogue(e, acc[i][j], bv, rv);
      }
    }
}

}  // namespace

int launch_gemm_simt(const GemmProblem &p, const GemmEpilogue &e, cudaStream_t s) {
  const int64_t batch = p.nb0 * p.nb1;
  FML_REQUIRE(batch <= 65535 && (p.M + SB - 1) / SB <= 65535, FML_UNSUPPORTED,
              "fml_gemm: batch or M too large for the fp32 kernel grid");
  dim3 grid((unsigned)((p.N + SB - 1) / SB), (unsigned)((p.M + SB - 1) / SB), (unsigned)batch);
  FML_LAUNCH((gemm_simt_kernel), grid, 256, 0, s, p, e);
  FML_CUDA(cudaGetLastError());
  return FML_OK;
}

static GemmEpilogue make_epilogue(const fml_gemm_params &gp, bool has_bias, bool has_res) {
  GemmEpilogue e;
  e.divisor = gp.divisor == 0.0f ? 1.0f : gp.divisor;
  e.alpha = gp.alpha; e.beta = gp.beta; e.act = gp.act;
  e.c0 = gp.act_param[0]; e.c1 = gp.act_param[1]; e.c2 = gp.act_param[2];
  e.has_bias = has_bias; e.has_res = has_res;
  return e;
}

}  // namespace fml

using namespace fml;

extern "C" void fml_gemm_default_params(fml_gemm_params *p) {
  if (!p) return;
  memset(p, 0, sizeof(*p));
  p->precision = FML_GEMM_AUTO;
  p->act = FML_ACT_NONE;
  p->divisor = 1.0f;
  p->alpha = 1.0f;
  p->beta = 1.0f;
  p->act_param[0] = 1.4142135381698608f;  // sqrt(2) in fp32
  p->act_param[1] = 1.0f;
  p->act_param[2] = 0.5f;
}

namespace {
enum class Path { kSimt, kTc, kPair };
struct Choice {
  Path path;
  TcPlan tc;
  PairPlan pair;
  GemmExtras x;
  bool parts = false;  // joined by the caller (a2, act_from) but not one launch here: fml_gemm runs the parts
};

// Dims [from, to) of dim `dim` of t.
fml_tensor part_of(const fml_tensor *t, int dim, int64_t from, int64_t to) {
  fml_tensor v = *t;
  v.shape[dim] = to - from;
  v.data = (char *)t->data + from * t->stride[dim] * 4;
  return v;
}
}  // namespace

static int resolve(const fml_tensor *a, const fml_tensor *b, const fml_tensor *c,
                   const fml_tensor *bias, const fml_tensor *res, const fml_gemm_params *gp,
                   GemmProblem &p, Choice &ch) {
  FML_REQUIRE(gp, FML_BAD_ARG, "fml_gemm: null params");
  GemmExtras &x = ch.x;
  x = GemmExtras();
  ch.parts = false;
  bool joined = true;  // A2's rows are walked as A's are
  fml_tensor whole;
  if (gp->a2.data) {
    const fml_tensor *a2 = &gp->a2;
    FML_REQUIRE(valid_tensor(a) && valid_tensor(a2) && valid_tensor(b) && a2->dtype == FML_F32 && a->rank >= 2 && b->rank == 2 && a2->rank == a->rank,
                FML_BAD_ARG, "fml_gemm: A2 needs A's rank and a B of rank 2");
    for (int i = 0; i + 1 < a->rank; ++i) FML_REQUIRE(a2->shape[i] == a->shape[i], FML_BAD_ARG, "fml_gemm: A2's shape");
    const int64_t k1 = a->shape[a->rank - 1], k2 = a2->shape[a->rank - 1];
    FML_REQUIRE(k1 > 0 && k2 > 0 && b->shape[0] == k1 + k2, FML_BAD_ARG, "fml_gemm: the columns of A and A2 are not the rows of B");
    FML_REQUIRE(gp->act == FML_ACT_NONE && gp->alpha == 1.0f && gp->beta == 1.0f && (gp->divisor == 1.0f || gp->divisor == 0.0f) && !gp->act_from && !gp->rot,
                FML_UNSUPPORTED, "fml_gemm: A2 with an activation, a scale or a rotation");
    const fml_tensor b2 = part_of(b, 0, k1, k1 + k2);
    GemmProblem p2;
    const int st = analyse_gemm(a2, &b2, c, bias, res, p2);
    if (st != FML_OK) return st;
    x.a2 = p2.a; x.a2_sm = p2.a_sm; x.a2_b0 = p2.a_b0; x.a2_b1 = p2.a_b1; x.k1 = k1; x.summed = gp->summed != 0;
    whole = *a;
    whole.shape[a->rank - 1] = k1 + k2;
    a = &whole;
    joined = p2.a_sk == 1;
    const int st1 = analyse_gemm(a, b, c, bias, res, p);
    if (st1 != FML_OK) return st1;
    joined = joined && p2.M == p.M && p2.nb0 == p.nb0 && p2.nb1 == p.nb1;
  } else {
    const int st = analyse_gemm(a, b, c, bias, res, p);
    if (st != FML_OK) return st;
  }
  if (gp->act_from) {
    FML_REQUIRE(gp->act_from > 0 && gp->act_from < p.N, FML_BAD_ARG, "fml_gemm: act_from is not a column");
    x.act_from = gp->act_from;
  }
  if (gp->rot) {
    FML_REQUIRE(gp->rot > 0 && gp->rot % 2 == 0 && gp->rot <= gp->rot_head && gp->rot_cols > 0 && gp->rot_cols <= p.N &&
                    gp->rot_cols % gp->rot_head == 0 && gp->rot_len > 0 && p.M % gp->rot_len == 0 && gp->rot_cos && gp->rot_sin && !res,
                FML_BAD_ARG, "fml_gemm: rotary embedding");
    FML_REQUIRE(gp->act_from ? gp->rot_cols <= gp->act_from : gp->act == FML_ACT_NONE, FML_UNSUPPORTED, "fml_gemm: an activation on rotated columns");
    x.rot = gp->rot; x.rot_head = gp->rot_head; x.rot_cols = gp->rot_cols; x.rot_len = gp->rot_len;
    x.rot_cos = gp->rot_cos; x.rot_sin = gp->rot_sin;
  }
  ch.path = Path::kSimt;
  if (joined && plan_gemm_pair(p, x, *gp, ch.pair)) ch.path = Path::kPair;
  else if (x.a2 || x.act_from) { ch.parts = true; return FML_OK; }
  else if (gp->precision != FML_GEMM_FP32 && plan_gemm_tc(p, *gp, ch.tc)) ch.path = Path::kTc;
  FML_REQUIRE(ch.path != Path::kSimt || gp->precision == FML_GEMM_AUTO || gp->precision == FML_GEMM_FP32,
              FML_MISALIGNED,
              "fml_gemm: a tensor-core precision was requested but the operands cannot be fed to "
              "TMA (need a unit-stride k or n dim, 16-byte aligned bases and row strides)");
  return FML_OK;
}

extern "C" int fml_gemm_plan(const fml_tensor *a, const fml_tensor *b, const fml_tensor *c,
                             const fml_gemm_params *gp, fml_gemm_plan_info *info) {
  FML_REQUIRE(info, FML_BAD_ARG, "fml_gemm_plan: null argument");
  GemmProblem p;
  Choice ch;
  int st = resolve(a, b, c, nullptr, nullptr, gp, p, ch);
  if (st != FML_OK) return st;
  memset(info, 0, sizeof(*info));
  if (ch.parts) return FML_OK;
  info->uses_tensor_cores = ch.path != Path::kSimt ? 1 : 0;
  if (ch.path == Path::kPair) {
    info->tile_n = ch.pair.tile_n; info->split_k = ch.pair.split_k; info->stages = ch.pair.stages_b;
    info->three_pass = 1; info->uses_packed = 1; info->stages_a = ch.pair.stages_a;
    info->shared_memory_bytes = ch.pair.smem_bytes;
  } else if (ch.path == Path::kTc) {
    const TcPlan &plan = ch.tc;
    info->tile_n = plan.tile_n; info->split_k = plan.split_k; info->stages = plan.stages;
    info->b_mn_major = plan.b_mn_major; info->three_pass = plan.three_pass;
    info->shared_memory_bytes = plan.smem_bytes;
  }
  return FML_OK;
}

extern "C" int fml_gemm_uses_tensor_cores(const fml_tensor *a, const fml_tensor *b,
                                          const fml_tensor *c, const fml_gemm_params *gp, int *uses) {
  FML_REQUIRE(uses, FML_BAD_ARG, "fml_gemm_uses_tensor_cores: null argument");
  GemmProblem p;
  Choice ch;
  int st = resolve(a, b, c, nullptr, nullptr, gp, p, ch);
  if (st != FML_OK) return st;
  *uses = ch.path != Path::kSimt ? 1 : 0;
  return FML_OK;
}

extern "C" int fml_gemm_uses_columns(const fml_tensor *a, const fml_tensor *b, const fml_tensor *c, const fml_gemm_params *gp, int *uses) {
  FML_REQUIRE(uses, FML_BAD_ARG, "fml_gemm_uses_columns: null argument");
  GemmProblem p;
  Choice ch;
  const int st = resolve(a, b, c, nullptr, nullptr, gp, p, ch);
  if (st != FML_OK) return st;
  *uses = !ch.parts && ch.path == Path::kSimt && p.M > 0 && p.N > 0 && gemm_skinny_by_columns(p) ? 1 : 0;
  return FML_OK;
}

extern "C" int fml_gemm(const fml_tensor *a, const fml_tensor *b, const fml_tensor *c,
                        const fml_tensor *bias, const fml_tensor *residual,
                        const fml_gemm_params *gp, void *stream) {
  GemmProblem p;
  Choice ch;
  int st = resolve(a, b, c, bias, residual, gp, p, ch);
  if (st != FML_OK) return st;
  if (p.M == 0 || p.N == 0 || p.nb0 * p.nb1 == 0) return FML_OK;
  if (ch.parts) {  // the parts one after the other, each with the tiles the library chooses for it
    fml_gemm_params q = *gp;
    q.tile_n = q.split_k = q.ctas_per_sm = 0;
    q.b_packed = nullptr;
    q.act_from = 0;
    memset(&q.a2, 0, sizeof(q.a2));
    const int rb = b->rank, rc = c->rank;
    if (gp->a2.data) {  // A's part with bias and residual, then A2's on top of it
      const int64_t k1 = a->shape[a->rank - 1];
      const fml_tensor b1 = part_of(b, 0, 0, k1), b2 = part_of(b, 0, k1, b->shape[0]);
      st = fml_gemm(a, &b1, c, bias, residual, &q, stream);
      return st != FML_OK ? st : fml_gemm(&gp->a2, &b2, c, nullptr, c, &q, stream);
    }
    for (int part = 0; part < 2; ++part) {  // the columns without the activation, then those with it
      const int64_t from = part ? gp->act_from : 0, to = part ? p.N : gp->act_from;
      const fml_tensor bp = part_of(b, rb - 1, from, to), cp = part_of(c, rc - 1, from, to);
      auto columns = [&](const fml_tensor *t, fml_tensor *v) -> const fml_tensor * {
        if (!t || t->rank == 0 || t->shape[t->rank - 1] == 1) return t;
        *v = part_of(t, t->rank - 1, from, to);
        return v;
      };
      fml_tensor bias_part, res_part;
      q.act = part ? gp->act : FML_ACT_NONE;
      if (part) q.rot = 0;
      st = fml_gemm(a, &bp, &cp, columns(bias, &bias_part), columns(residual, &res_part), &q, stream);
      if (st != FML_OK) return st;
    }
    return FML_OK;
  }
  GemmEpilogue e = make_epilogue(*gp, bias != nullptr, residual != nullptr);
  p.b_constant = gp->b_constant ? 1 : 0;
  if (gp->l2_prefetch && gp->l2_prefetch_bytes) {
    FML_REQUIRE((reinterpret_cast<uintptr_t>(gp->l2_prefetch) & 15) == 0, FML_MISALIGNED,
                "fml_gemm: the L2 prefetch hint must be 16-byte aligned");
    p.prefetch = static_cast<const char *>(gp->l2_prefetch);
    p.prefetch_bytes = gp->l2_prefetch_bytes;
  }
  if (ch.path == Path::kPair) return launch_gemm_pair(p, e, ch.x, ch.pair, gp->b_packed, as_stream(stream));
  st = ch.path == Path::kTc ? launch_gemm_tc(p, e, ch.tc, as_stream(stream))
       : skinny_eligible(p) ? launch_gemm_skinny(p, e, as_stream(stream)) : launch_gemm_simt(p, e, as_stream(stream));
  return st == FML_OK && ch.x.rot ? launch_rotary_in_place(p, ch.x, as_stream(stream)) : st;
}

// What a remembered choice of tiles belongs to: the device, the problem and its epilogue.
static std::string tuning_key(int device, const GemmProblem &p, const Choice &ch, const fml_gemm_params &gp, bool bias, bool residual) {
  const bool pair = ch.path == Path::kPair;
  char key[256];
  snprintf(key, sizeof(key), "%d|%lld,%lld,%lld,%lld,%lld|%d%d%d|%d,%d,%d,%d|%lld,%lld|%d,%d,%lld,%d", device, (long long)p.M, (long long)p.N, (long long)p.K,
           (long long)p.nb0, (long long)p.nb1, pair, pair ? 0 : ch.tc.b_mn_major, pair ? 1 : ch.tc.three_pass, gp.act, bias, residual,
           gp.divisor != 1.0f, (long long)p.c_sm, (long long)p.c_sn, ch.x.act_from, ch.x.rot ? ch.x.rot_cols : 0, (long long)ch.x.k1, ch.x.summed);
  return key;
}

extern "C" int fml_gemm_tuning_key(const fml_tensor *a, const fml_tensor *b, const fml_tensor *c, const fml_tensor *bias,
                                   const fml_tensor *residual, const fml_gemm_params *gp, int device, char *key, size_t bytes) {
  FML_REQUIRE(gp && key && bytes, FML_BAD_ARG, "fml_gemm_tuning_key: null argument");
  GemmProblem p;
  Choice ch;
  const int st = resolve(a, b, c, bias, residual, gp, p, ch);
  if (st != FML_OK) return st;
  snprintf(key, bytes, "%s", ch.parts || ch.path == Path::kSimt ? "" : tuning_key(device, p, ch, *gp, bias != nullptr, residual != nullptr).c_str());
  return FML_OK;
}

// One-off on-device tuning of (tile_n, split_k) for one GEMM, cached per device and problem signature.
// The reference tunes its MatMul / Gemm kernels the same way -- by running the candidates
// (there: six loop orders on the CPU, src/structure/kernel/generator/matmul.cpp:100-123) and
// keeping the fastest per layout triple.
extern "C" int fml_gemm_autotune(const fml_tensor *a, const fml_tensor *b, const fml_tensor *c,
                                 const fml_tensor *bias, const fml_tensor *residual,
                                 const fml_gemm_params *gp, void *stream, fml_gemm_params *tuned) {
  FML_REQUIRE(gp && tuned, FML_BAD_ARG, "fml_gemm_autotune: null argument");
  *tuned = *gp;
  GemmProblem p;
  Choice ch;
  int st = resolve(a, b, c, bias, residual, gp, p, ch);
  if (st != FML_OK) return st;
  if (ch.parts || ch.path == Path::kSimt || gp->tile_n != 0 || gp->split_k != 0) return FML_OK;  // nothing to choose
  const bool pair = ch.path == Path::kPair;
  int device = 0;
  FML_CUDA(cudaGetDevice(&device));
  const std::string key = tuning_key(device, p, ch, *gp, bias != nullptr, residual != nullptr);
  struct Tiles { int tile_n, split_k, ctas_per_sm; };
  static std::map<std::string, Tiles> cache;
  static std::mutex mu;
  auto take = [&](const Tiles &t) {
    tuned->tile_n = t.tile_n;
    tuned->split_k = t.split_k;
    tuned->ctas_per_sm = t.ctas_per_sm;
  };
  {
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(key);
    if (it != cache.end()) { take(it->second); return FML_OK; }
  }
  // Candidates run as a captured graph of back-to-back launches, as the products of a model do: timed
  // one by one from the host, launches of a few microseconds are paced by the host and the choice is noise.
  FML_CUDA(cudaStreamSynchronize(as_stream(stream)));
  cudaStream_t s;
  cudaEvent_t e0, e1;
  FML_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  FML_CUDA(cudaEventCreate(&e0));
  FML_CUDA(cudaEventCreate(&e1));
  const GemmEpilogue epi = make_epilogue(*gp, bias != nullptr, residual != nullptr);
  const int tn_opts[] = {32, 48, 64, 96, 128, 192, 256};
  const int sk_opts[] = {1, 2, 4, 8};
  float best = 1e30f;
  Tiles best_tiles = pair ? Tiles{ch.pair.tile_n, ch.pair.split_k, ch.pair.ctas_per_sm} : Tiles{ch.tc.tile_n, ch.tc.split_k, 0};
  std::vector<Tiles> seen;
  const bool exact = pair && pair_exact(p, ch.x, ch.pair.split_k, ch.pair.two_accs);  // (the plan without tuning is, if any is)
  for (int tn : tn_opts)
    for (int sk : sk_opts)
      for (int ctas = 1; ctas <= (pair ? 2 : 1); ++ctas) {
        fml_gemm_params q = *gp;
        q.tile_n = tn;
        q.split_k = sk;
        q.ctas_per_sm = ctas;
        Choice cand;
        if (pair ? !plan_gemm_pair(p, ch.x, q, cand.pair) : !plan_gemm_tc(p, q, cand.tc)) continue;
        if (pair && exact && !pair_exact(p, ch.x, cand.pair.split_k, cand.pair.two_accs)) continue;
        const Tiles id = pair ? Tiles{cand.pair.tile_n, cand.pair.split_k, cand.pair.ctas_per_sm}
                              : Tiles{cand.tc.tile_n, cand.tc.split_k, 0};
        bool dup = false;
        for (const auto &x : seen)
          dup = dup || (x.tile_n == id.tile_n && x.split_k == id.split_k && x.ctas_per_sm == id.ctas_per_sm);
        if (dup) continue;
        seen.push_back(id);
        auto launch = [&] {
          return pair ? launch_gemm_pair(p, epi, ch.x, cand.pair, gp->b_packed, s) : launch_gemm_tc(p, epi, cand.tc, s);
        };
        float one = 0.0f;
        bool ok = launch() == FML_OK;  // warm-up; skip what cannot launch
        cudaEventRecord(e0, s);
        ok = ok && launch() == FML_OK;
        cudaEventRecord(e1, s);
        if (cudaEventSynchronize(e1) != cudaSuccess || !ok) { cudaGetLastError(); continue; }
        cudaEventElapsedTime(&one, e0, e1);
        // Large products: one launch is well above what the host adds to it, so what is far behind goes no
        // further and two launches replace eight (a batch of 16 x 384 tokens of BERT-base spent 1.4 s of its
        // Compile on 32 launches of every candidate).
        if (one > 0.05f && one > 1.5f * best) continue;
        const int reps = one > 0.2f ? 2 : 8;
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        ok = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
        for (int r = 0; r < reps && ok; ++r) ok = launch() == FML_OK;
        ok = cudaStreamEndCapture(s, &graph) == cudaSuccess && ok && cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess;
        if (graph) cudaGraphDestroy(graph);
        float ms = 1e30f;
        for (int r = 0; r < 4 && ok; ++r) {  // the first replay warms up
          cudaEventRecord(e0, s);
          ok = cudaGraphLaunch(exec, s) == cudaSuccess;
          cudaEventRecord(e1, s);
          ok = cudaEventSynchronize(e1) == cudaSuccess && ok;
          float t = 0;
          cudaEventElapsedTime(&t, e0, e1);
          if (r && t / reps < ms) ms = t / reps;
        }
        if (exec) cudaGraphExecDestroy(exec);
        if (!ok) { cudaGetLastError(); continue; }
        if (ms < best) { best = ms; best_tiles = id; }
      }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaStreamDestroy(s);
  take(best_tiles);
  std::lock_guard<std::mutex> lock(mu);
  cache[key] = best_tiles;
  return FML_OK;
}

// Packed weights of the half-precision-pair kernel (gemm_pair.cu).
extern "C" size_t fml_gemm_packed_bytes(int64_t k, int64_t n) { return k > 0 && n > 0 ? pair_packed_bytes(k, n) : 0; }

extern "C" int fml_gemm_pack(const fml_tensor *b, void *packed, size_t bytes, void *stream) {
  FML_REQUIRE(valid_tensor(b) && b->dtype == FML_F32 && b->rank == 2 && packed, FML_BAD_ARG, "fml_gemm_pack: bad argument");
  const int64_t K = b->shape[0], N = b->shape[1];
  FML_REQUIRE(K > 0 && N > 0 && bytes >= pair_packed_bytes(K, N), FML_BAD_ARG, "fml_gemm_pack: the destination is too small");
  FML_REQUIRE(aligned16(packed), FML_MISALIGNED, "fml_gemm_pack: the destination must be 16-byte aligned");
  return pair_pack((const float *)b->data, K, N, b->stride[0], b->stride[1], packed, as_stream(stream));
}

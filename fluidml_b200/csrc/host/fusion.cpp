#include "fusion.h"
#include <cstdlib>
#include "fluidml_cuda.h"
#include <algorithm>
#include <cmath>
#include <unordered_map>
#include <unordered_set>

namespace fluidml {
namespace worker {
namespace {

using flow::Kind;
using flow::NodePtr;
using flow::RegionPtr;

struct Rewriter {
  flow::Flow &f;
  std::unordered_map<const flow::Region *, std::vector<NodePtr>> consumers;
  std::unordered_map<const flow::Region *, NodePtr> producer;
  std::unordered_set<const flow::Node *> dead;
  std::unordered_map<RegionPtr, RegionPtr> table_rows;  // the rows of a rotary table (FuseRotaryIntoGemm)

  explicit Rewriter(flow::Flow &flow) : f(flow) { Index(); }

  void Index() {
    consumers.clear();
    producer.clear();
    for (const auto &n : f.nodes) {
      if (dead.count(n.get())) continue;
      producer[n->output.get()] = n;
      for (const auto &r : n->inputs) consumers[r.get()].push_back(n);
    }
  }
  // The only consumer of `r`, provided `r` is an inner tensor nobody else reads.
  NodePtr Sole(const RegionPtr &r) {
    if (r->kind != flow::Region::kInner) return nullptr;
    auto it = consumers.find(r.get());
    if (it == consumers.end() || it->second.size() != 1) return nullptr;
    return it->second[0];
  }
  NodePtr SoleOfKind(const RegionPtr &r, Kind k) {
    NodePtr n = Sole(r);
    return n && n->kind == k ? n : nullptr;
  }
  void Kill(const NodePtr &n) { dead.insert(n.get()); }
  void Commit() {
    f.nodes.erase(std::remove_if(f.nodes.begin(), f.nodes.end(),
                                 [&](const NodePtr &n) { return dead.count(n.get()) != 0; }),
                  f.nodes.end());
    dead.clear();
    Index();
  }
};

bool IsConst(const RegionPtr &r) { return r->kind == flow::Region::kConstant; }

// The operand of a two-input node that is not `x`.
RegionPtr Other(const NodePtr &n, const RegionPtr &x) { return n->inputs[0] == x ? n->inputs[1] : n->inputs[0]; }

bool IsGemmLike(const NodePtr &n) {
  return n->kind == Kind::MatMul || n->kind == Kind::FusedGemm || n->kind == Kind::GemmConstantBias;
}

// MatMul / Gemm -> FusedGemm, keeping operands and attributes.
void PromoteToFusedGemm(const NodePtr &n) {
  if (n->kind == Kind::FusedGemm) return;
  if (n->kind == Kind::MatMul) {
    if (IsConst(n->inputs[1])) {
      n->consts = {n->inputs[1]};
      n->inputs = {n->inputs[0]};
      n->b_is_const = true;
    }
  } else {  // GemmConstantBias: consts = {B, C}
    n->b_is_const = true;
    n->has_bias = true;
  }
  n->kind = Kind::FusedGemm;
}

// ---- gather_add_fusion.cpp: Gather(table, ids) + constT + constT -> one embedding kernel
bool FuseEmbedding(Rewriter &rw, const NodePtr &g) {
  if (g->kind != Kind::GatherConstantDataTensor || g->consts[0]->meta.GetType() != Type::kFloat32) return false;
  NodePtr a0 = rw.SoleOfKind(g->output, Kind::AddCommon);
  if (!a0 || !IsConst(Other(a0, g->output))) return false;
  NodePtr a1 = rw.SoleOfKind(a0->output, Kind::AddCommon);
  if (!a1 || !IsConst(Other(a1, a0->output))) return false;
  g->kind = Kind::GatherConstantDataTensorAddTensorLhsAddTensorLhs;
  g->consts = {g->consts[0], Other(a0, g->output), Other(a1, a0->output)};
  g->output = a1->output;
  rw.Kill(a0);
  rw.Kill(a1);
  return true;
}

// ---- unsqueeze_sub_mul_fusion.cpp: Unsqueeze(+Unsqueeze) -> c - x -> * m
bool FuseMask(Rewriter &rw, const NodePtr &u) {
  if (u->kind != Kind::Unsqueeze || u->inputs[0]->meta.GetType() != Type::kFloat32) return false;
  std::vector<NodePtr> chain = {u};
  NodePtr cur = u;
  while (NodePtr nx = rw.SoleOfKind(cur->output, Kind::Unsqueeze)) { chain.push_back(nx); cur = nx; }
  NodePtr sub = rw.SoleOfKind(cur->output, Kind::SubConstantLhs);
  if (!sub) return false;
  NodePtr mul = rw.SoleOfKind(sub->output, Kind::MulConstant);
  if (!mul) return false;
  u->kind = Kind::UnsqueezeSubLhsScalarMulRhsScalar;
  u->value = sub->value;
  u->value2 = mul->value;
  u->output = mul->output;
  for (size_t i = 1; i < chain.size(); ++i) rw.Kill(chain[i]);
  rw.Kill(sub);
  rw.Kill(mul);
  return true;
}

// ---- MatMul/Gemm + constant bias -> epilogue
bool FuseBias(Rewriter &rw, const NodePtr &mm) {
  if (mm->kind != Kind::MatMul && !(mm->kind == Kind::FusedGemm && !mm->has_bias && !mm->has_mask && mm->act == 0 && !mm->has_residual)) return false;
  NodePtr add = rw.SoleOfKind(mm->output, Kind::AddCommon);
  if (!add) return false;
  RegionPtr bias = Other(add, mm->output);
  if (!IsConst(bias) || bias->meta.GetType() != Type::kFloat32) return false;
  if (add->output->meta != mm->output->meta) return false;  // the bias must not widen the result
  PromoteToFusedGemm(mm);
  mm->consts.push_back(bias);
  mm->has_bias = true;
  mm->output = add->output;
  rw.Kill(add);
  return true;
}

// ---- add_div_erf_add_mul_fusion.cpp: t -> t/c0 -> erf -> +c1 -> t*(.) -> *c2
// `t` is produced by `src`; returns the final Mul node and the constants.
bool MatchGelu(Rewriter &rw, const RegionPtr &t, NodePtr &div, NodePtr &erf, NodePtr &add, NodePtr &mul0, NodePtr &mul1) {
  if (t->kind != flow::Region::kInner) return false;
  auto it = rw.consumers.find(t.get());
  if (it == rw.consumers.end() || it->second.size() != 2) return false;
  div = mul0 = nullptr;
  for (const auto &c : it->second) {
    if (c->kind == Kind::DivConstantRhs) div = c;
    else if (c->kind == Kind::MulCommon) mul0 = c;
  }
  if (!div || !mul0) return false;
  erf = rw.SoleOfKind(div->output, Kind::Erf);
  if (!erf) return false;
  add = rw.SoleOfKind(erf->output, Kind::AddConstant);
  if (!add) return false;
  if (rw.Sole(add->output) != mul0 || Other(mul0, t) != add->output) return false;
  mul1 = rw.SoleOfKind(mul0->output, Kind::MulConstant);
  return mul1 != nullptr;
}

bool FuseGeluIntoGemm(Rewriter &rw, const NodePtr &mm) {
  if (!IsGemmLike(mm) || mm->act != 0 || mm->has_residual) return false;
  NodePtr div, erf, add, mul0, mul1;
  if (!MatchGelu(rw, mm->output, div, erf, add, mul0, mul1)) return false;
  PromoteToFusedGemm(mm);
  mm->act = FML_ACT_GELU_ERF;
  mm->act_param[0] = (float)div->value;
  mm->act_param[1] = (float)add->value;
  mm->act_param[2] = (float)mul1->value;
  mm->output = mul1->output;
  for (const auto &k : {div, erf, add, mul0, mul1}) rw.Kill(k);
  return true;
}

// Add(x, const bias) followed by the GELU chain, when no GEMM produced x: the reference's
// AddDivErfAddMulMul kernel.
bool FuseBiasGelu(Rewriter &rw, const NodePtr &a) {
  if (a->kind != Kind::AddCommon) return false;
  RegionPtr bias, x;
  if (IsConst(a->inputs[0]) && !IsConst(a->inputs[1])) { bias = a->inputs[0]; x = a->inputs[1]; }
  else if (IsConst(a->inputs[1]) && !IsConst(a->inputs[0])) { bias = a->inputs[1]; x = a->inputs[0]; }
  else return false;
  if (a->output->meta != x->meta) return false;
  NodePtr div, erf, add, mul0, mul1;
  if (!MatchGelu(rw, a->output, div, erf, add, mul0, mul1)) return false;
  a->kind = Kind::AddDivErfAddMulMul;
  a->inputs = {x};
  a->consts = {bias};
  a->act_param[0] = (float)div->value;
  a->act_param[1] = (float)add->value;
  a->act_param[2] = (float)mul1->value;
  a->output = mul1->output;
  for (const auto &k : {div, erf, add, mul0, mul1}) rw.Kill(k);
  return true;
}

// ---- GEMM -> Tanh / Relu / Sigmoid
bool FuseActivation(Rewriter &rw, const NodePtr &mm) {
  const bool conv = mm->kind == Kind::ConvWithPadding || mm->kind == Kind::ConvWithoutPadding;
  if (!(IsGemmLike(mm) || conv) || mm->act != 0 || mm->has_residual) return false;
  NodePtr act = rw.Sole(mm->output);
  if (!act) return false;
  int code = act->kind == Kind::Tanh ? FML_ACT_TANH : act->kind == Kind::Relu ? FML_ACT_RELU
             : act->kind == Kind::Sigmoid ? FML_ACT_SIGMOID : 0;
  if (!code) return false;
  if (!conv) PromoteToFusedGemm(mm);
  mm->act = code;
  mm->output = act->output;
  rw.Kill(act);
  return true;
}

// ---- GEMM + residual Add -> epilogue
bool FuseResidual(Rewriter &rw, const NodePtr &mm) {
  if (!IsGemmLike(mm) || mm->has_residual) return false;
  NodePtr add = rw.SoleOfKind(mm->output, Kind::AddCommon);
  if (!add) return false;
  RegionPtr res = Other(add, mm->output);
  if (IsConst(res) || res->meta != mm->output->meta || add->output->meta != mm->output->meta) return false;
  // the residual must not itself depend on this GEMM: it would, only if the GEMM's output had
  // another consumer, which Sole() excluded
  PromoteToFusedGemm(mm);
  mm->inputs.push_back(res);
  mm->has_residual = true;
  mm->output = add->output;
  rw.Kill(add);
  return true;
}

// ---- (G + R) + x -> G + (R + x) when G is a GEMM that has taken the GEMM R as its residual: x becomes R's.
// A parallel-residual block (attention and feed-forward both added to their input) then has no Add of its own:
// 23 launches of 6.4 us in a pass of a 24-layer GPT-NeoX at 4 x 512.  One rounding per sum, as before.
bool FuseSecondResidual(Rewriter &rw, const NodePtr &mm) {
  if (mm->kind != Kind::FusedGemm || !mm->has_residual) return false;
  NodePtr add = rw.SoleOfKind(mm->output, Kind::AddCommon);
  if (!add) return false;
  RegionPtr x = Other(add, mm->output);
  if (IsConst(x) || x->meta != mm->output->meta || add->output->meta != mm->output->meta) return false;
  const RegionPtr r = mm->inputs.back();
  auto it = rw.producer.find(r.get());
  if (it == rw.producer.end() || rw.Sole(r) != mm || r->meta != mm->output->meta) return false;
  const NodePtr g = it->second;
  if (rw.dead.count(g.get()) || !IsGemmLike(g) || g->has_residual) return false;
  // x does not depend on R: R's only reader is G, and G's only reader is the Add
  PromoteToFusedGemm(g);
  g->inputs.push_back(x);
  g->has_residual = true;
  mm->output = add->output;
  rw.Kill(add);
  return true;
}

// ---- Add(x, r) -> LayerNorm, when the Add did not fold into a GEMM
bool FuseAddLayerNorm(Rewriter &rw, const NodePtr &add) {
  if (add->kind != Kind::AddCommon || IsConst(add->inputs[0]) || IsConst(add->inputs[1])) return false;
  if (add->inputs[0]->meta != add->output->meta || add->inputs[1]->meta != add->output->meta) return false;
  NodePtr ln = rw.SoleOfKind(add->output, Kind::LayerNormalizationConstantScaleBias);
  if (!ln) return false;
  ln->kind = Kind::FusedLayerNorm;
  ln->inputs = {add->inputs[0], add->inputs[1]};
  ln->has_residual = true;
  rw.Kill(add);
  return true;
}

// A condition [1, .., S, S] over scores [.., S, S] that holds up to and including the diagonal and nowhere
// else.  It has to span both of the scores' own last dims: one true value broadcast over them is a
// "lower-triangular" 1 x 1 matrix, but hides nothing.
bool LowerTriangular(const flow::Region &cond, const Meta &scores) {
  const auto &shape = cond.meta.GetShape(), &over = scores.GetShape();
  const size_t rank = shape.size();
  if (rank < 2 || over.size() < rank || shape[rank - 1] != shape[rank - 2]) return false;
  if (shape[rank - 1] != over[over.size() - 1] || shape[rank - 2] != over[over.size() - 2]) return false;
  for (size_t i = 0; i + 2 < rank; ++i)
    if (shape[i] != 1) return false;
  const int64_t n = shape[rank - 1];
  for (int64_t r = 0; r < n; ++r)
    for (int64_t c = 0; c < n; ++c)
      if ((cond.constant->AsInt(r * n + c) != 0) != (c <= r)) return false;
  return true;
}

// ---- x / c -> + mask -> Softmax  (attention scores); the mask may also be a constant-condition
// Where that replaces masked scores by a scalar (a causal mask): Where(cond, s, y) feeds the
// softmax the same values as s + m with m = cond ? 0 : y whenever y is so negative that
// s + y rounds to y (the usual float lowest), so it becomes a baked additive mask.
bool FuseScaledMaskedSoftmax(Rewriter &rw, const NodePtr &div) {
  if (div->kind != Kind::DivConstantRhs) return false;
  NodePtr nx = rw.Sole(div->output);
  if (!nx) return false;
  NodePtr add = nullptr, where = nullptr, sm = nullptr;
  if (nx->kind == Kind::AddCommon) {
    add = nx;
    if (add->output->meta != div->output->meta) return false;
    sm = rw.SoleOfKind(add->output, Kind::Softmax);
  } else if (nx->kind == Kind::WhereConstantCondConstantScalarY) {
    where = nx;
    // s + y == y needs |y| >= 2^25 |s|: accept the float lowest and anything within 2^-40 of it
    if (where->output->meta != div->output->meta || !(where->value <= -3.0e26) ||
        where->consts.empty() || !where->consts[0]->constant)
      return false;
    sm = rw.SoleOfKind(where->output, Kind::Softmax);
  } else if (nx->kind == Kind::Softmax) {
    sm = nx;
  }
  if (!sm || sm->axis != (int64_t)sm->output->meta.GetRank() - 1) return false;
  RegionPtr mask = nullptr;
  if (where) {
    const RegionPtr &cond = where->consts[0];
    const int64_t n = (int64_t)cond->meta.GetElementsNum();
    std::vector<uint8_t> bytes((size_t)n * 4);
    float *m = reinterpret_cast<float *>(bytes.data());
    const float y = (float)where->value;
    for (int64_t i = 0; i < n; ++i) m[i] = cond->constant->AsInt(i) ? 0.0f : y;
    mask = rw.f.NewRegion(flow::Region::kConstant, where->name + "_additive_mask", Meta(Type::kFloat32, cond->meta.GetShape()));
    mask->constant = std::make_shared<Tensor>(mask->meta, std::move(bytes));
  }
  sm->kind = Kind::FusedSoftmax;
  sm->divisor = (float)div->value;
  sm->inputs = {div->inputs[0]};
  if (add) {
    sm->inputs.push_back(Other(add, div->output));
    sm->has_mask = true;
    rw.Kill(add);
  } else if (where) {
    sm->inputs.push_back(mask);
    sm->has_mask = true;
    sm->causal = LowerTriangular(*where->consts[0], where->output->meta) && where->value <= -1.0e30;
    rw.Kill(where);
  }
  rw.Kill(div);
  return true;
}

// ---- MatMul(Q, K^T) -> [scaled, masked] Softmax -> MatMul(P, V): one attention kernel when
// K and V of a head fit in shared memory
bool FuseAttention(Rewriter &rw, const NodePtr &qk) {
  if (qk->kind != Kind::MatMul || qk->inputs.size() != 2 || IsConst(qk->inputs[0]) || IsConst(qk->inputs[1])) return false;
  NodePtr sm = rw.Sole(qk->output);
  if (!sm || (sm->kind != Kind::Softmax && sm->kind != Kind::FusedSoftmax) || sm->inputs[0] != qk->output) return false;
  const size_t rank = sm->output->meta.GetRank();
  if (rank < 2 || rank > 4 || sm->axis != (int64_t)rank - 1) return false;
  NodePtr pv = rw.SoleOfKind(sm->output, Kind::MatMul);
  if (!pv || pv->inputs.size() != 2 || pv->inputs[0] != sm->output || IsConst(pv->inputs[1])) return false;
  const RegionPtr &q = qk->inputs[0], &kt = qk->inputs[1], &v = pv->inputs[1];
  const auto &qs = q->meta.GetShape(), &ks = kt->meta.GetShape(), &vs = v->meta.GetShape();
  if (qs.size() != rank || ks.size() != rank || vs.size() != rank) return false;
  if (q->meta.GetType() != Type::kFloat32 || kt->meta.GetType() != Type::kFloat32 || v->meta.GetType() != Type::kFloat32) return false;
  for (size_t i = 0; i + 2 < rank; ++i)
    if (qs[i] != ks[i] || qs[i] != vs[i]) return false;  // no batch broadcasting between the operands
  if (!fml_attention_supported(qs[rank - 2], ks[rank - 1], qs[rank - 1], vs[rank - 1])) return false;
  // The CUDA-core fused kernel computes in fp32 FMA (about 10 TFLOP/s): it wins while the three
  // launches it replaces are latency-bound; larger blocks are fused only when the tensor-core
  // attention kernel takes their head sizes (otherwise the score products are faster as GEMMs).
  double flops = 4.0 * (double)qs[rank - 2] * (double)ks[rank - 1] * (double)qs[rank - 1];
  double heads = 1.0;
  for (size_t i = 0; i + 2 < rank; ++i) heads *= (double)qs[i];
  flops *= heads;
  {
    // FLUIDML_ATTENTION_FUSION_MFLOP moves the limit (for measurements); blocks the tensor-core
    // kernel takes are fused up to `tc_limit`: beyond a few key blocks its serial phases lose to
    // the two batched tensor-core GEMMs around a softmax.  Head size 64 has a pipelined kernel and is
    // fused whatever its size.
    static const double limit = [] { const char *e = getenv("FLUIDML_ATTENTION_FUSION_MFLOP"); return e ? atof(e) * 1e6 : 256e6; }();
    static const double tc_limit = [] { const char *e = getenv("FLUIDML_ATTENTION_TC_FUSION_MFLOP"); return e ? atof(e) * 1e6 : 256e6; }();
    const bool tc = fml_attention_on_tensor_cores(qs[rank - 2], ks[rank - 1], qs[rank - 1], vs[rank - 1]) != 0;
    const bool any = tc && heads <= 65535.0 && fml_attention_any_size(qs[rank - 1], vs[rank - 1]) != 0;
    if (!any && flops > (tc ? std::max(limit, tc_limit) : limit)) return false;
  }
  qk->kind = Kind::FusedAttention;
  qk->inputs = {q, kt, v};
  qk->divisor = sm->kind == Kind::FusedSoftmax ? sm->divisor : 1.0f;
  qk->has_mask = sm->kind == Kind::FusedSoftmax && sm->has_mask;
  if (qk->has_mask) qk->inputs.push_back(sm->inputs[1]);
  qk->causal = qk->has_mask && sm->causal;
  qk->output = pv->output;
  rw.Kill(sm);
  rw.Kill(pv);
  return true;
}

// ---- Sigmoid(x) * x
bool FuseSilu(Rewriter &rw, const NodePtr &sg) {
  if (sg->kind != Kind::Sigmoid) return false;
  NodePtr mul = rw.SoleOfKind(sg->output, Kind::MulCommon);
  if (!mul || Other(mul, sg->output) != sg->inputs[0]) return false;
  sg->kind = Kind::Silu;
  sg->output = mul->output;
  rw.Kill(mul);
  return true;
}

// ---- Mul -> Add: one pass over the data instead of two (the span convolution of ConvBERT is a
// chain of nine such pairs, rotary embeddings two).  Same two roundings as the separate kernels.
bool FuseMulAdd(Rewriter &rw, const NodePtr &mul) {
  if (mul->kind != Kind::MulCommon || mul->inputs.size() != 2) return false;
  NodePtr add = rw.SoleOfKind(mul->output, Kind::AddCommon);
  if (!add || add->inputs.size() != 2 || add->inputs[0] == add->inputs[1]) return false;
  const RegionPtr other = Other(add, mul->output);
  for (const RegionPtr &r : {mul->inputs[0], mul->inputs[1], other, add->output})
    if (r->meta.GetType() != Type::kFloat32) return false;
  // the addend must not depend on this product (it cannot: the product has one consumer)
  mul->kind = Kind::FusedMulAdd;
  mul->inputs = {mul->inputs[0], mul->inputs[1], other};
  mul->output = add->output;
  rw.Kill(add);
  return true;
}

// ---- ReduceMean over H, W -> 1 x 1 Conv (+act) -> 1 x 1 Conv (+act): the gate of a squeeze-and-
// excite block.  Three launches that move a few kilobytes each become one (FLUIDML_FUSE_SE=0
// keeps them apart, for comparisons).
bool FuseSqueezeExcite(Rewriter &rw, const NodePtr &rm) {
  static const bool enabled = [] { const char *e = getenv("FLUIDML_FUSE_SE"); return !(e && e[0] == '0'); }();
  if (!enabled || rm->kind != Kind::ReduceMean) return false;
  const RegionPtr &x = rm->inputs[0];
  if (x->meta.GetRank() != 4 || x->meta.GetType() != Type::kFloat32) return false;
  std::vector<int64_t> axes = rm->axes;
  std::sort(axes.begin(), axes.end());
  if (axes != std::vector<int64_t>{2, 3}) return false;
  auto gate_conv = [](const NodePtr &cv, int64_t in_channels) {
    if (!cv || cv->group != 1 || cv->consts.empty() || cv->inputs.size() != 1) return false;
    const auto &ws = cv->consts[0]->meta.GetShape();
    if (ws.size() != 4 || ws[1] != in_channels || ws[2] != 1 || ws[3] != 1) return false;
    if (cv->consts[0]->meta.GetType() != Type::kFloat32 || !utils::IsDefaultLayout(cv->consts[0]->layout)) return false;
    if (cv->has_bias && (cv->consts.size() < 2 || cv->consts[1]->meta.GetElementsNum() != ws[0])) return false;
    for (int64_t s : cv->strides) if (s != 1) return false;
    for (int64_t d : cv->dilations) if (d != 1) return false;
    return cv->act == FML_ACT_NONE || cv->act == FML_ACT_RELU || cv->act == FML_ACT_TANH || cv->act == FML_ACT_SIGMOID ||
           cv->act == FML_ACT_SILU;
  };
  const int64_t C = x->meta.GetShape()[1];
  NodePtr c1 = rw.SoleOfKind(rm->output, Kind::ConvWithoutPadding);
  if (!gate_conv(c1, C)) return false;
  const int64_t Cr = c1->consts[0]->meta.GetShape()[0];
  NodePtr c2 = rw.SoleOfKind(c1->output, Kind::ConvWithoutPadding);
  if (!gate_conv(c2, Cr) || c2->consts[0]->meta.GetShape()[0] != C) return false;
  if (C > 4096 || Cr > 512 || x->meta.GetShape()[0] > 65535) return false;  // limits of fml_squeeze_excite_gate
  rm->kind = Kind::SqueezeExciteGate;
  rm->consts.clear();
  rm->consts.push_back(c1->consts[0]);
  if (c1->has_bias) rm->consts.push_back(c1->consts[1]);
  rm->consts.push_back(c2->consts[0]);
  if (c2->has_bias) rm->consts.push_back(c2->consts[1]);
  rm->has_bias = c1->has_bias;
  rm->has_bias2 = c2->has_bias;
  rm->act = c1->act;
  rm->act2 = c2->act;
  rm->output = c2->output;
  rw.Kill(c1);
  rw.Kill(c2);
  return true;
}

// ---- Mul(x [N, C, H, W], gate [N, C, 1, 1]) -> group-1 Conv: the gate multiplies x while the
// convolution gathers its operand (same fp32 rounding of the product), so the gated tensor -- the
// widest of a squeeze-and-excite block -- is neither written nor read back.
bool FuseGateIntoConv(Rewriter &rw, const NodePtr &mul) {
  if (mul->kind != Kind::MulCommon || mul->inputs.size() != 2) return false;
  NodePtr cv = rw.Sole(mul->output);
  if (!cv || (cv->kind != Kind::ConvWithPadding && cv->kind != Kind::ConvWithoutPadding)) return false;
  if (cv->group != 1 || cv->has_in_scale || cv->inputs.size() != 1 || cv->inputs[0] != mul->output) return false;
  const auto &os = mul->output->meta.GetShape();
  if (os.size() != 4 || mul->output->meta.GetType() != Type::kFloat32 || os[1] > 4096) return false;
  auto is_gate = [&](const RegionPtr &r) {
    const auto &gs = r->meta.GetShape();
    return r->meta.GetType() == Type::kFloat32 && gs.size() == 4 && (gs[0] == os[0] || gs[0] == 1) &&
           (gs[1] == os[1] || gs[1] == 1) && gs[2] == 1 && gs[3] == 1;
  };
  RegionPtr x, gate;
  if (mul->inputs[0]->meta.GetShape() == os && is_gate(mul->inputs[1])) { x = mul->inputs[0]; gate = mul->inputs[1]; }
  else if (mul->inputs[1]->meta.GetShape() == os && is_gate(mul->inputs[0])) { x = mul->inputs[1]; gate = mul->inputs[0]; }
  else return false;
  if (os[2] * os[3] == 1) return false;  // a gate times a gate: nothing to save
  cv->inputs = {x, gate};
  cv->has_in_scale = true;
  rw.Kill(mul);
  return true;
}

// ---- Conv + x -> the convolution's epilogue (the residual of an inverted bottleneck).  Group 1 and 2-D: what the
// packed-weight kernel may take; where another kernel runs, the sum is a launch of its own as before.
bool FuseResidualIntoConv(Rewriter &rw, const NodePtr &cv) {
  if ((cv->kind != Kind::ConvWithPadding && cv->kind != Kind::ConvWithoutPadding) || cv->group != 1 || cv->act != 0 || cv->has_residual) return false;
  NodePtr add = rw.SoleOfKind(cv->output, Kind::AddCommon);
  if (!add) return false;
  RegionPtr x = Other(add, cv->output);
  if (IsConst(x) || x == cv->output || x->meta != cv->output->meta || add->output->meta != cv->output->meta) return false;
  const auto &os = x->meta.GetShape();
  if (os.size() != 4 || os[2] * os[3] < 32 || x->meta.GetType() != Type::kFloat32) return false;
  cv->inputs.push_back(x);
  cv->has_residual = true;
  cv->output = add->output;
  rw.Kill(add);
  return true;
}

// ---- MulCommon -> FusedMulAdd -> FusedMulAdd ...: a sum of products (ConvBERT's span convolution
// adds nine windows times nine softmax columns) becomes one pass.  Matched at the last node of the
// chain and walked back to the plain product it starts from; every intermediate sum must have the
// next link as its only reader.  Same rounding order as the chain.
bool FuseMulAddChain(Rewriter &rw, const NodePtr &last) {
  if (last->kind != Kind::FusedMulAdd || last->inputs.size() != 3) return false;
  {  // `last` must end the chain: its result is not the addend of another link
    NodePtr next = rw.Sole(last->output);
    if (next && next->kind == Kind::FusedMulAdd && next->inputs.size() == 3 && next->inputs[2] == last->output) return false;
  }
  std::vector<NodePtr> links = {last};  // from the end backwards
  NodePtr head;                         // the MulCommon the chain starts from
  for (;;) {
    const RegionPtr &addend = links.back()->inputs[2];
    auto it = rw.producer.find(addend.get());
    if (it == rw.producer.end() || rw.Sole(addend) != links.back()) return false;
    const NodePtr &prod = it->second;
    if (prod->kind == Kind::FusedMulAdd && prod->inputs.size() == 3) { links.push_back(prod); continue; }
    if (prod->kind == Kind::MulCommon && prod->inputs.size() == 2) { head = prod; break; }
    return false;
  }
  const size_t pairs = links.size() + 1;
  if (pairs < 3 || pairs > 12) return false;  // fml_sum_of_products takes up to 12
  std::vector<RegionPtr> ops = {head->inputs[0], head->inputs[1]};
  for (size_t i = links.size(); i-- > 0;) { ops.push_back(links[i]->inputs[0]); ops.push_back(links[i]->inputs[1]); }
  for (const RegionPtr &r : ops)
    if (r->meta.GetType() != Type::kFloat32) return false;
  if (last->output->meta.GetType() != Type::kFloat32) return false;
  last->kind = Kind::FusedMulAddChain;
  last->inputs = ops;
  rw.Kill(head);
  for (size_t i = 1; i < links.size(); ++i) rw.Kill(links[i]);
  return true;
}

// ---- FusedMulAddChain over windows of a Pad along the sequence and the taps of a Softmax: x [b, s, h, d], padded with zeros
// along s, its windows starting at 0, 1, .., each times one tap of softmax(logits [b, s, h, taps]).  Four launches in one.
bool FuseSpanConvolution(Rewriter &rw, const NodePtr &chain) {
  if (chain->kind != Kind::FusedMulAddChain || chain->span || chain->inputs.size() % 2) return false;
  const int64_t taps = (int64_t)chain->inputs.size() / 2;
  if (!fml_span_convolution_supported(taps)) return false;
  const auto &os = chain->output->meta.GetShape();
  if (os.size() != 4 || chain->output->meta.GetType() != Type::kFloat32) return false;
  auto slice_of = [&](const RegionPtr &r) -> NodePtr {
    auto it = rw.producer.find(r.get());
    return it != rw.producer.end() && it->second->kind == Kind::Slice && it->second->inputs.size() == 1 && it->second->starts.size() == 4 && rw.Sole(r) == chain
               ? it->second : nullptr;
  };
  RegionPtr padded, weights;
  std::vector<NodePtr> slices;
  for (int64_t j = 0; j < taps; ++j) {
    NodePtr win = slice_of(chain->inputs[2 * j]), tap = slice_of(chain->inputs[2 * j + 1]);
    if (!win || !tap) return false;
    if (win->output->meta.GetShape() != os) std::swap(win, tap);  // a product may be written either way round
    const auto &ws = win->output->meta.GetShape(), &ts = tap->output->meta.GetShape();
    if (ws != os || ts.size() != 4 || ts[0] != os[0] || ts[1] != os[1] || ts[2] != os[2] || ts[3] != 1) return false;
    const int64_t at = win->starts[1];
    // (the chain's first sum, a product plus a product, has no order)
    if (at != j && !(j < 2 && at == 1 - j)) return false;
    if (j == 1 && at == slices[0]->starts[1]) return false;
    if (win->starts != std::vector<int64_t>{0, at, 0, 0} || tap->starts != std::vector<int64_t>{0, 0, 0, at}) return false;
    if (j == 0) { padded = win->inputs[0]; weights = tap->inputs[0]; }
    if (win->inputs[0] != padded || tap->inputs[0] != weights) return false;
    slices.push_back(win);
    slices.push_back(tap);
  }
  auto made_by = [&](const RegionPtr &r, Kind k) -> NodePtr {  // read by the slices only
    auto it = rw.producer.find(r.get());
    auto readers = rw.consumers.find(r.get());
    return it != rw.producer.end() && it->second->kind == k && r->kind == flow::Region::kInner && readers != rw.consumers.end() &&
                   (int64_t)readers->second.size() == taps ? it->second : nullptr;
  };
  const NodePtr pad = made_by(padded, Kind::Pad), sm = made_by(weights, Kind::Softmax);
  if (!pad || !sm || pad->inputs.size() != 1 || sm->inputs.size() != 1 || (sm->axis != 3 && sm->axis != -1)) return false;
  const RegionPtr &x = pad->inputs[0], &logits = sm->inputs[0];
  if (x->meta.GetShape() != os || x->meta.GetType() != Type::kFloat32 || logits->meta.GetType() != Type::kFloat32 || IsConst(x) || IsConst(logits)) return false;
  if (logits->meta.GetShape() != std::vector<int64_t>{os[0], os[1], os[2], taps} || pad->pads.size() != 8) return false;
  for (size_t i = 0; i < 8; ++i)
    if (i % 4 != 1 && pad->pads[i] != 0) return false;
  if (pad->pads[1] < 0 || pad->pads[5] < 0 || pad->pads[1] + pad->pads[5] != taps - 1) return false;
  if (os[0] > 65535 || os[2] * taps > 1024 || os[2] > 512) return false;  // limits of fml_span_convolution
  chain->inputs = {x, logits};
  chain->span = taps;
  chain->pads = {pad->pads[1]};
  for (const NodePtr &n : slices) rw.Kill(n);
  rw.Kill(pad);
  rw.Kill(sm);
  return true;
}

// ---- Rotary position embedding as exported (GPT-NeoX):
//   xr = x[..., :rot]; xp = x[..., rot:]
//   out = Concat(xr * cos + Concat(-xr[..., rot/2:], xr[..., :rot/2]) * sin, xp)
// Matched at the final Concat (after FuseMulAdd has made `xr * cos + (...)` one node); ten nodes per
// projection (five of them launches) become one.
bool FuseRotary(Rewriter &rw, const NodePtr &cat) {
  if (cat->kind != Kind::Concat2 || cat->inputs.size() != 2) return false;
  const RegionPtr &y = cat->output;
  const size_t rank = y->meta.GetRank();
  if (rank < 1 || y->meta.GetType() != Type::kFloat32) return false;
  const int64_t last = (int64_t)rank - 1;
  if (cat->axis != last && cat->axis != -1) return false;
  auto producer_of = [&](const RegionPtr &r) -> NodePtr {
    auto it = rw.producer.find(r.get());
    return it == rw.producer.end() ? nullptr : it->second;
  };
  // a Slice along the last axis only: returns its start there, -1 otherwise
  auto last_axis_slice = [&](const NodePtr &n) -> int64_t {
    if (!n || n->kind != Kind::Slice || n->inputs.size() != 1 || n->starts.size() != rank) return -1;
    const auto &is = n->inputs[0]->meta.GetShape(), &os = n->output->meta.GetShape();
    if (is.size() != rank || os.size() != rank) return -1;
    for (size_t i = 0; i + 1 < rank; ++i)
      if (n->starts[i] != 0 || is[i] != os[i]) return -1;
    return n->starts[rank - 1];
  };
  NodePtr fma = producer_of(cat->inputs[0]), pass = producer_of(cat->inputs[1]);
  if (!fma || fma->kind != Kind::FusedMulAdd || fma->inputs.size() != 3 || rw.Sole(fma->output) != cat) return false;
  NodePtr xr = producer_of(fma->inputs[0]);
  RegionPtr cosv = fma->inputs[1];
  if (last_axis_slice(xr) != 0) {  // the product may be written cos * xr
    xr = producer_of(fma->inputs[1]);
    cosv = fma->inputs[0];
    if (last_axis_slice(xr) != 0) return false;
  }
  const RegionPtr &src = xr->inputs[0];
  const int64_t rot = xr->output->meta.GetShape()[rank - 1], D = src->meta.GetShape()[rank - 1];
  if (rot < 2 || (rot & 1) || last_axis_slice(pass) != rot || pass->inputs[0] != src ||
      pass->output->meta.GetShape()[rank - 1] != D - rot || rw.Sole(pass->output) != cat)
    return false;
  NodePtr mul = producer_of(fma->inputs[2]);
  if (!mul || mul->kind != Kind::MulCommon || mul->inputs.size() != 2 || rw.Sole(mul->output) != fma) return false;
  NodePtr half_cat = producer_of(mul->inputs[0]);
  RegionPtr sinv = mul->inputs[1];
  if (!half_cat || half_cat->kind != Kind::Concat2) { half_cat = producer_of(mul->inputs[1]); sinv = mul->inputs[0]; }
  if (!half_cat || half_cat->kind != Kind::Concat2 || half_cat->inputs.size() != 2 || rw.Sole(half_cat->output) != mul ||
      (half_cat->axis != last && half_cat->axis != -1))
    return false;
  NodePtr neg = producer_of(half_cat->inputs[0]), lo = producer_of(half_cat->inputs[1]);
  if (!neg || neg->kind != Kind::Neg || rw.Sole(neg->output) != half_cat) return false;
  NodePtr hi = producer_of(neg->inputs[0]);
  if (last_axis_slice(hi) != rot / 2 || last_axis_slice(lo) != 0 || hi->inputs[0] != xr->output || lo->inputs[0] != xr->output ||
      hi->output->meta.GetShape()[rank - 1] != rot / 2 || lo->output->meta.GetShape()[rank - 1] != rot / 2 ||
      rw.Sole(hi->output) != neg || rw.Sole(lo->output) != half_cat)
    return false;
  // xr is read by the two half slices and the product, by nobody else
  {
    auto it = rw.consumers.find(xr->output.get());
    if (it == rw.consumers.end() || it->second.size() != 3 || xr->output->kind != flow::Region::kInner) return false;
  }
  for (const RegionPtr &t : {cosv, sinv}) {
    const auto &ts = t->meta.GetShape();
    if (t->meta.GetType() != Type::kFloat32 || ts.empty() || ts.size() > rank || ts.back() != rot) return false;
  }
  if (src->meta.GetType() != Type::kFloat32) return false;
  cat->kind = Kind::Rotary;
  cat->inputs = {src, cosv, sinv};
  cat->value = (double)rot;
  for (const NodePtr &n : {fma, pass, xr, mul, half_cat, neg, hi, lo}) rw.Kill(n);
  return true;
}

// A constant of our own making.
RegionPtr MakeConstant(flow::Flow &f, const std::string &name, std::vector<int64_t> shape, std::vector<uint8_t> bytes) {
  const RegionPtr r = f.NewRegion(flow::Region::kConstant, name, Meta(Type::kFloat32, shape));
  r->constant = std::make_shared<Tensor>(r->meta, std::move(bytes));
  return r;
}
// One that is put together from others when it is uploaded.
RegionPtr MakeConstant(flow::Flow &f, const std::string &name, std::vector<int64_t> shape, std::vector<Tensor::Block> blocks) {
  const RegionPtr r = f.NewRegion(flow::Region::kConstant, name, Meta(Type::kFloat32, shape));
  r->constant = std::make_shared<Tensor>(r->meta, std::move(blocks));
  return r;
}

bool HoldsFloats(const RegionPtr &r, size_t rank, size_t count) {
  return r->kind == flow::Region::kConstant && r->meta.GetType() == Type::kFloat32 && r->meta.GetRank() == rank && r->constant &&
         r->constant->ByteSize() == count * 4 && utils::IsDefaultLayout(r->layout);
}

// A product with a captured weight [K, N] and bias [N] (or none) in logical row-major order, nothing but an
// activation on top of it: what the passes below may join.  `rows` of it at least 32: fewer stay separate, on the
// weight-streaming kernel.
bool IsPlainProduct(const NodePtr &n) {
  if (n->kind != Kind::FusedGemm || !n->b_is_const || n->trans_a || n->trans_b || n->has_mask || n->two_a || n->divisor != 1.0f ||
      n->alpha != 1.0f || n->beta != 1.0f)
    return false;
  const RegionPtr &w = n->consts[0];
  if (w->meta.GetRank() != 2) return false;
  const int64_t K = w->meta.GetShape()[0], N = w->meta.GetShape()[1];
  return HoldsFloats(w, 2, (size_t)K * (size_t)N) && (!n->has_bias || (n->consts.size() >= 2 && HoldsFloats(n->consts[1], 1, (size_t)N)));
}
bool IsJoinable(const NodePtr &n) {
  if (!IsPlainProduct(n)) return false;
  const int64_t K = n->consts[0]->meta.GetShape()[0], N = n->consts[0]->meta.GetShape()[1];
  return K % 4 == 0 && K >= 16 && N % 4 == 0 && N >= 16 && (int64_t)n->output->meta.GetElementsNum() / N >= 32;
}

// ---- product -> Reshape [b, s, heads, size] -> Transpose (0, 2, 1, 3) -> Rotary: the rotation in the product's epilogue.
// The Rotary node stays, with one input and no launch.
bool FuseRotaryIntoGemm(Rewriter &rw, const NodePtr &rot) {
  if (rot->kind != Kind::Rotary || rot->inputs.size() != 3) return false;
  auto made_by = [&](const RegionPtr &r, Kind k) -> NodePtr {
    auto it = rw.producer.find(r.get());
    return it != rw.producer.end() && it->second->kind == k && rw.Sole(r) ? it->second : nullptr;
  };
  const NodePtr tr = made_by(rot->inputs[0], Kind::Transpose);
  if (!tr || tr->perm != std::vector<int64_t>{0, 2, 1, 3}) return false;
  const NodePtr rs = made_by(tr->inputs[0], Kind::Reshape);
  if (!rs) return false;
  const NodePtr mm = made_by(rs->inputs[0], Kind::FusedGemm);
  if (!mm || !IsJoinable(mm) || mm->act != 0 || mm->has_residual || mm->rot) return false;
  const auto &flat = mm->output->meta.GetShape(), &split = rs->output->meta.GetShape();
  if (flat.size() != 3 || split.size() != 4 || split[0] != flat[0] || split[1] != flat[1] || split[2] * split[3] != flat[2]) return false;
  const int64_t width = (int64_t)rot->value, length = flat[1];
  for (size_t i = 1; i < 3; ++i) {
    const RegionPtr &t = rot->inputs[i];
    const auto &ts = t->meta.GetShape();
    if (ts.size() < 2 || ts[ts.size() - 1] != width || ts[ts.size() - 2] != length || !HoldsFloats(t, ts.size(), (size_t)(width * length))) return false;
  }
  RegionPtr tables[2];
  for (size_t i = 0; i < 2; ++i) {  // rows of this node's own: the layout search may permute what other nodes read
    const RegionPtr &t = rot->inputs[1 + i];
    RegionPtr &rows = rw.table_rows[t];
    if (!rows) rows = MakeConstant(rw.f, t->name + "_rows", {length, width}, t->constant->Bytes());
    tables[i] = rows;
  }
  mm->consts.push_back(tables[0]);
  mm->consts.push_back(tables[1]);
  mm->rot = width;
  mm->rot_head = split[3];
  mm->rot_cols = flat[2];
  mm->rot_len = length;
  rot->inputs = {rot->inputs[0]};  // what the product has rotated: a view
  return true;
}

// Gains that LayerNorms of one tensor may share: powers of two near the geometric mean of theirs, feature by feature.  What is
// left of a norm's own, the factor of its products' weights, must not lie more than 12 times below its root mean square
// anywhere: else false.
//
// Why not 1: a row enters the products with one scale, and what lies far below the row's largest keeps an absolute error
// only.  Trained norms hold down the features that grow by orders of magnitude; without their gains such a feature sets the
// scale of all others.  Relative error (2-norm, operands split as the kernel splits them, exact sums, 64 x 1024 x 64) of
// separate norms / a shared one without gains / with these, two features of the row 10^4 times the others: 7e-8 / 1.8e-6 /
// 8e-8 with both gains 2^-10 there; 10^6 times, both 2^-17: 8e-8 / 1.8e-4 / 8e-8.  Where one norm holds down what the other
// lets through, half of the difference (in bits) stays: 10^6 times, 2^-4 against 1 (a factor 4): 6e-8 / 6e-7 / 1.5e-7; 2^-8
// (16): 6e-8 / 9e-6 / 6e-7.
bool SharedGains(const std::vector<NodePtr> &norms, int64_t K, std::vector<float> *shared, std::vector<std::vector<uint8_t>> *own) {
  auto gain = [&](const NodePtr &n, int64_t k) { return reinterpret_cast<const float *>(n->consts[0]->constant->Bytes().data())[k]; };
  shared->resize((size_t)K);
  for (int64_t k = 0; k < K; ++k) {
    double bits = 0.0;
    for (const NodePtr &n : norms) {
      const float g = std::fabs(gain(n, k));
      if (!(g >= 0x1p-60f && g <= 0x1p60f)) return false;
      bits += std::log2((double)g);
    }
    (*shared)[k] = std::ldexp(1.0f, (int)std::lround(bits / (double)norms.size()));
  }
  own->clear();
  for (const NodePtr &n : norms) {
    std::vector<uint8_t> left((size_t)K * 4);
    float *l = reinterpret_cast<float *>(left.data());
    double least = 1e300, squares = 0.0;
    for (int64_t k = 0; k < K; ++k) {
      l[k] = gain(n, k) / (*shared)[k];  // (exact)
      least = std::min(least, (double)std::fabs(l[k]));
      squares += (double)l[k] * (double)l[k];
    }
    if (least * 12.0 < std::sqrt(squares / (double)K)) return false;
    own->push_back(std::move(left));
  }
  return true;
}

// ---- LayerNorms of one tensor that feed products only (the two halves of a parallel-residual block): scale and
// shift move into the products, (x^ g + b) W + c = (x^ s) (g / s W) + (b W + c), worked out in 64 bits, and one LayerNorm with
// the gains s and no shift serves all.  Its readers are then siblings and merge.
bool FoldSharedLayerNorms(Rewriter &rw) {
  for (const NodePtr &first : rw.f.nodes) {
    if (first->kind != Kind::LayerNormalizationConstantScaleBias || first->inputs.size() != 1) continue;
    const RegionPtr x = first->inputs[0];
    const auto &shape = x->meta.GetShape();
    const int64_t last = (int64_t)shape.size() - 1;
    std::vector<NodePtr> norms;
    for (const NodePtr &n : rw.consumers[x.get()]) {
      if (n->kind != Kind::LayerNormalizationConstantScaleBias || n->inputs.size() != 1 || n->axis != first->axis || n->epsilon != first->epsilon) continue;
      if (n->axis != last && n->axis != -1) continue;
      bool ok = n->output->kind == flow::Region::kInner && n->consts.size() == 2 && HoldsFloats(n->consts[0], 1, (size_t)shape[last]) &&
                HoldsFloats(n->consts[1], 1, (size_t)shape[last]);
      const auto &readers = rw.consumers[n->output.get()];
      ok = ok && !readers.empty();
      for (const NodePtr &r : readers) {
        size_t uses = 0;
        for (const RegionPtr &in : r->inputs) uses += in == n->output;
        ok = ok && IsJoinable(r) && uses == 1 && r->inputs[0] == n->output && r->consts[0]->meta.GetShape()[0] == shape[last];
      }
      if (ok) norms.push_back(n);
    }
    if (norms.size() < 2) continue;
    const int64_t K = shape[last];
    std::vector<float> shared;
    std::vector<std::vector<uint8_t>> own;
    if (!SharedGains(norms, K, &shared, &own)) continue;
    for (size_t i = 0; i < norms.size(); ++i) {
      const NodePtr &n = norms[i];
      const auto factors = std::make_shared<Tensor>(n->consts[0]->meta, std::move(own[i]));
      const float *b = reinterpret_cast<const float *>(n->consts[1]->constant->Bytes().data());
      for (const NodePtr &r : rw.consumers[n->output.get()]) {
        const int64_t N = r->consts[0]->meta.GetShape()[1];
        const float *w = reinterpret_cast<const float *>(r->consts[0]->constant->Bytes().data());
        const float *c = r->has_bias ? reinterpret_cast<const float *>(r->consts[1]->constant->Bytes().data()) : nullptr;
        std::vector<uint8_t> cb((size_t)N * 4);
        std::vector<double> shift((size_t)N);
        for (int64_t j = 0; j < N; ++j) shift[j] = c ? (double)c[j] : 0.0;
        float *co = reinterpret_cast<float *>(cb.data());
        for (int64_t k = 0; k < K; ++k)
          for (int64_t j = 0; j < N; ++j) shift[j] += (double)b[k] * (double)w[k * N + j];
        for (int64_t j = 0; j < N; ++j) co[j] = (float)shift[j];
        r->consts[0] = MakeConstant(rw.f, r->name + "_normed.w", {K, N}, {{r->consts[0]->constant, 0, 0, factors}});
        const RegionPtr nc = MakeConstant(rw.f, r->name + "_normed.b", {N}, std::move(cb));
        if (r->has_bias) r->consts[1] = nc;
        else r->consts.insert(r->consts.begin() + 1, nc);
        r->has_bias = true;
        r->inputs[0] = norms[0]->output;
      }
      if (n != norms[0]) rw.Kill(n);
    }
    std::vector<uint8_t> gains((size_t)K * 4), zeros((size_t)K * 4);
    memcpy(gains.data(), shared.data(), gains.size());
    norms[0]->consts = {MakeConstant(rw.f, norms[0]->name + "_shared.g", {K}, std::move(gains)),
                        MakeConstant(rw.f, norms[0]->name + "_shared.b", {K}, std::move(zeros))};
    rw.Commit();
    return true;
  }
  return false;
}

// [W1; W2] and the sum of the biases: what a product over two left-hand sides reads.
void JoinWeights(flow::Flow &f, const NodePtr &into, const NodePtr &top, const NodePtr &bottom) {
  const int64_t N = top->consts[0]->meta.GetShape()[1], K1 = top->consts[0]->meta.GetShape()[0], K = K1 + bottom->consts[0]->meta.GetShape()[0];
  std::vector<Tensor::Block> w = {{top->consts[0]->constant, 0, 0, nullptr}, {bottom->consts[0]->constant, K1, 0, nullptr}};
  std::vector<uint8_t> bias;
  for (const NodePtr &n : {top, bottom}) {
    if (!n->has_bias) continue;
    const std::vector<uint8_t> &b = n->consts[1]->constant->Bytes();
    if (bias.empty()) { bias = b; continue; }
    for (int64_t j = 0; j < N; ++j) reinterpret_cast<float *>(bias.data())[j] += reinterpret_cast<const float *>(b.data())[j];
  }
  const std::string base = into->name + "_joined";
  into->consts = {MakeConstant(f, base + ".w", {K, N}, std::move(w))};
  into->has_bias = !bias.empty();
  if (into->has_bias) into->consts.push_back(MakeConstant(f, base + ".b", {N}, std::move(bias)));
}

// Whether [A1 | A2] [W1; W2] is as exact as A1 W1 + A2 W2.  In the joined product a row of both A has one power-of-two
// scale and a column of both W another; elements far below either keep an absolute error only.  That is enough where they
// meet weights like the others': what it costs, it costs a part of the sum that is small.  A small A2 against a large
// column of W2 (or A1, W1) is not: with halves that contribute alike, the joined product's relative error (2-norm, operands
// split as the kernel splits them, exact sums) against the separate ones' is 7.7e-8 / 7.7e-8 at weights 4 times apart,
// 8.9e-8 / 7.6e-8 at 16, 2.0e-7 at 64, 1.2e-5 at 4096, 3e-3 at 2^20.  An element's absolute error goes into a column by the
// column's root mean square, so these have to be within a factor of 4, column by column; blocks of which that does not
// hold stay two launches.  (The columns' scales do no harm: what is below them keeps 2^-39 of the largest.)
bool AlikeByColumns(const RegionPtr &a, const RegionPtr &b) {
  const int64_t N = a->meta.GetShape()[1];
  std::vector<double> mean[2];
  for (int i = 0; i < 2; ++i) {
    const RegionPtr &w = i ? b : a;
    const int64_t K = w->meta.GetShape()[0];
    mean[i].assign((size_t)N, 0.0);
    std::vector<float> v((size_t)N);
    for (int64_t k = 0; k < K; ++k) {
      w->constant->WriteRow(k, v.data());
      for (int64_t j = 0; j < N; ++j) mean[i][j] += (double)v[j] * (double)v[j];
    }
    for (int64_t j = 0; j < N; ++j) mean[i][j] /= (double)K;
  }
  for (int64_t j = 0; j < N; ++j)  // (squares)
    if (!(mean[0][j] <= 16.0 * mean[1][j] && mean[1][j] <= 16.0 * mean[0][j])) return false;
  return true;
}

// ---- A1 W1 + (A2 W2 + x) -> [A1 | A2] [W1; W2] + x: one launch, one reduction and one pass over the result for both
// halves of a parallel-residual block, where their weights are of one magnitude and the rows few enough (fml_gemm_joins_sums).
bool JoinSummedProducts(Rewriter &rw, const NodePtr &mm) {
  if (!IsJoinable(mm) || mm->act != 0 || mm->rot || !mm->has_residual || mm->inputs.size() != 2) return false;
  const RegionPtr r = mm->inputs[1];
  auto it = rw.producer.find(r.get());
  if (it == rw.producer.end() || rw.Sole(r) != mm) return false;
  const NodePtr g = it->second;
  if (!IsJoinable(g) || g->act != 0 || g->rot || g->inputs.size() != (g->has_residual ? 2u : 1u) || g->output->meta != mm->output->meta) return false;
  if (g->inputs[0]->meta.GetRank() != mm->inputs[0]->meta.GetRank() || g->act_from || mm->act_from) return false;
  const bool swap = mm->consts[0]->meta.GetShape()[0] % 32 != 0;  // k blocks must not straddle the seam
  const NodePtr &top = swap ? g : mm, &bottom = swap ? mm : g;
  if (top->consts[0]->meta.GetShape()[0] % 32 != 0) return false;
  const int64_t N = top->consts[0]->meta.GetShape()[1];
  if (!fml_gemm_joins_sums((int64_t)mm->output->meta.GetElementsNum() / N, N) || !AlikeByColumns(top->consts[0], bottom->consts[0])) return false;
  std::vector<RegionPtr> inputs = {top->inputs[0], bottom->inputs[0]};
  if (g->has_residual) inputs.push_back(g->inputs[1]);
  JoinWeights(rw.f, mm, top, bottom);
  mm->inputs = inputs;
  mm->has_residual = g->has_residual;
  mm->two_a = mm->summed = true;
  rw.Kill(g);
  return true;
}

// ---- Concat(A1, A2) along the features -> product: the product reads both where they are.
bool JoinConcatenatedProduct(Rewriter &rw, const NodePtr &cat) {
  if (cat->kind != Kind::Concat2 || cat->inputs.size() != 2 || IsConst(cat->inputs[0]) || IsConst(cat->inputs[1])) return false;
  const int64_t rank = (int64_t)cat->output->meta.GetRank();
  if (rank < 2 || (cat->axis != rank - 1 && cat->axis != -1)) return false;
  const NodePtr mm = rw.SoleOfKind(cat->output, Kind::FusedGemm);
  if (!mm || !IsJoinable(mm) || mm->act != 0 || mm->rot || mm->act_from || mm->inputs[0] != cat->output) return false;
  const int64_t k1 = cat->inputs[0]->meta.GetShape()[rank - 1], k2 = cat->inputs[1]->meta.GetShape()[rank - 1];
  if (k1 % 32 != 0 || k2 % 4 != 0) return false;
  mm->inputs[0] = cat->inputs[0];
  mm->inputs.insert(mm->inputs.begin() + 1, cat->inputs[1]);
  mm->two_a = true;
  rw.Kill(cat);
  return true;
}

// ---- 1-D pointwise convolution -> Transpose (0, 2, 1): the product [B, L, C] x [C, OC] it is, read and written with the
// channels innermost, where what stands in front is a depthwise convolution over a transposed view, whose result the layout
// search can leave in that order too (ConvBERT: nothing changes between the orders any more, and the product with the
// queries behind it reads rows).  Only layers that the packed convolution takes: the arithmetic stays half-precision pairs.
bool PointwiseAsProduct(Rewriter &rw, const NodePtr &cv) {
  if (cv->kind != Kind::ConvWithoutPadding || cv->inputs.size() != 1 || cv->group != 1 || cv->act != 0 || cv->has_in_scale || cv->has_residual) return false;
  const auto &xs = cv->inputs[0]->meta.GetShape();
  if (xs.size() != 3 || IsConst(cv->inputs[0]) || cv->strides != std::vector<int64_t>{1} || cv->dilations != std::vector<int64_t>{1}) return false;
  auto made_by = [&](const RegionPtr &r) -> NodePtr {
    auto it = rw.producer.find(r.get());
    return it == rw.producer.end() ? nullptr : it->second;
  };
  const NodePtr dw = made_by(cv->inputs[0]);
  if (!dw || rw.Sole(dw->output) != cv || (dw->kind != Kind::ConvWithPadding && dw->kind != Kind::ConvWithoutPadding) || dw->group != xs[1] || dw->group < 2) return false;
  const NodePtr before = made_by(dw->inputs[0]);
  if (!before || before->kind != Kind::Transpose || before->perm != std::vector<int64_t>{0, 2, 1}) return false;
  const NodePtr tr = rw.SoleOfKind(cv->output, Kind::Transpose);
  if (!tr || tr->perm != std::vector<int64_t>{0, 2, 1}) return false;
  const int64_t B = xs[0], IC = xs[1], L = xs[2];
  const auto &ws = cv->consts.at(0)->meta.GetShape();
  if (ws.size() != 3 || ws[1] != IC || ws[2] != 1) return false;
  const int64_t OC = ws[0];
  if (L % 4 != 0 || L < 32 || IC % 4 != 0 || IC < 32 || OC % 4 != 0 || OC < 64) return false;
  if (!HoldsFloats(cv->consts[0], 3, (size_t)(OC * IC)) || (cv->has_bias && !HoldsFloats(cv->consts.at(1), 1, (size_t)OC))) return false;
  std::vector<uint8_t> bytes((size_t)(OC * IC) * 4);
  const float *w = reinterpret_cast<const float *>(cv->consts[0]->constant->Bytes().data());
  float *wt = reinterpret_cast<float *>(bytes.data());
  for (int64_t o = 0; o < OC; ++o)
    for (int64_t c = 0; c < IC; ++c) wt[c * OC + o] = w[o * IC + c];
  std::vector<RegionPtr> consts = {MakeConstant(rw.f, cv->name + "_columns", {IC, OC}, std::move(bytes))};
  if (cv->has_bias) consts.push_back(cv->consts[1]);
  const RegionPtr rows = rw.f.NewRegion(flow::Region::kInner, cv->name + "_rows", Meta(Type::kFloat32, {B, L, IC}));
  tr->kind = Kind::FusedGemm;
  tr->inputs = {rows};
  tr->consts = std::move(consts);
  tr->b_is_const = true;
  tr->has_bias = cv->has_bias;
  cv->kind = Kind::Transpose;
  cv->perm = {0, 2, 1};
  cv->consts.clear();
  cv->has_bias = false;
  cv->output = rows;
  return true;
}

// ---- Conv -> SiLU: the activation rides in the convolution's epilogue
bool FuseSiluIntoConv(Rewriter &rw, const NodePtr &cv) {
  if ((cv->kind != Kind::ConvWithPadding && cv->kind != Kind::ConvWithoutPadding) || cv->act != 0) return false;
  NodePtr silu = rw.SoleOfKind(cv->output, Kind::Silu);
  if (!silu) return false;
  cv->act = FML_ACT_SILU;
  cv->output = silu->output;
  rw.Kill(silu);
  return true;
}

// ---- GEMMs that read the same activations with constant weights (the Q, K, V projections):
// one GEMM over the concatenated weights, the original outputs become column slices of its
// result (views, no copy).  Fewer launches and one pass over the shared A operand.  With `join` (the packed-weight
// kernel will run them) rotated projections and those with a GELU come along, the former in front, the latter last.
bool MergeSiblingGemms(flow::Flow &f, bool join) {
  auto eligible = [&](const NodePtr &n) {
    if (!IsPlainProduct(n) || n->has_residual || n->inputs.size() != 1 || n->output->kind != flow::Region::kInner || n->act_from) return false;
    if (n->act == 0 && !n->rot) return true;
    if (n->rot && n->rot_cols != n->consts[0]->meta.GetShape()[1]) return false;  // already merged
    return join && IsJoinable(n) && !(n->act && n->rot) && (n->act == 0 || n->act == FML_ACT_GELU_ERF);
  };
  auto place = [](const NodePtr &n) { return n->rot ? 0 : n->act ? 2 : 1; };
  auto together = [&](const NodePtr &a, const NodePtr &b) {  // same tables, same constants of the activation
    if (a->rot && b->rot)
      return a->rot == b->rot && a->rot_head == b->rot_head && a->rot_len == b->rot_len && a->consts[a->consts.size() - 2] == b->consts[b->consts.size() - 2] &&
             a->consts.back() == b->consts.back();
    if (a->act && b->act) return a->act == b->act && std::equal(a->act_param, a->act_param + 3, b->act_param);
    return (place(a) == 1 && place(b) == 1) || (IsJoinable(a) && IsJoinable(b));
  };
  for (size_t i = 0; i < f.nodes.size(); ++i) {
    const NodePtr &first = f.nodes[i];
    if (!eligible(first)) continue;
    std::vector<NodePtr> group = {first};
    for (size_t j = i + 1; j < f.nodes.size(); ++j) {
      const NodePtr &n = f.nodes[j];
      if (!eligible(n) || n->inputs[0] != first->inputs[0] || n->has_bias != first->has_bias) continue;
      if (n->consts[0]->meta.GetShape()[0] != first->consts[0]->meta.GetShape()[0]) continue;
      const auto &sa = n->output->meta.GetShape(), &sb = first->output->meta.GetShape();
      if (sa.size() != sb.size() || !std::equal(sa.begin(), sa.end() - 1, sb.begin())) continue;
      bool ok = true;
      for (const NodePtr &g : group) ok = ok && together(g, n);
      if (ok) group.push_back(n);
    }
    if (group.size() < 2) continue;
    std::stable_sort(group.begin(), group.end(), [&](const NodePtr &a, const NodePtr &b) { return place(a) < place(b); });
    const int64_t K = first->consts[0]->meta.GetShape()[0];
    int64_t total = 0;
    for (const auto &n : group) total += n->consts[0]->meta.GetShape()[1];
    // concatenated weights [K, total] and bias [total]
    std::vector<Tensor::Block> weights;
    std::vector<uint8_t> bbytes(first->has_bias ? (size_t)total * 4 : 0);
    int64_t col = 0;
    for (const auto &n : group) {
      const int64_t N = n->consts[0]->meta.GetShape()[1];
      weights.push_back({n->consts[0]->constant, 0, col, nullptr});
      if (n->has_bias) memcpy(bbytes.data() + (size_t)col * 4, n->consts[1]->constant->Bytes().data(), (size_t)N * 4);
      col += N;
    }
    const std::string base = first->name + "_merged";
    RegionPtr wcat = MakeConstant(f, base + ".w", {K, total}, std::move(weights));
    RegionPtr bcat = first->has_bias ? MakeConstant(f, base + ".b", {total}, std::move(bbytes)) : nullptr;
    std::vector<int64_t> mshape = first->output->meta.GetShape();
    mshape.back() = total;
    const RegionPtr merged = f.NewRegion(flow::Region::kInner, base, Meta(Type::kFloat32, mshape));
    // slices that hand the original outputs back
    std::vector<NodePtr> slices;
    col = 0;
    for (const auto &n : group) {
      auto sl = std::make_shared<flow::Node>();
      sl->kind = Kind::Slice;
      sl->name = n->name + "_slice";
      sl->inputs = {merged};
      sl->output = n->output;
      sl->starts.assign(mshape.size(), 0);
      sl->starts.back() = col;
      col += n->consts[0]->meta.GetShape()[1];
      slices.push_back(sl);
    }
    // what rides in the epilogue: the rotation of the columns in front, the activation of those at the end
    std::vector<RegionPtr> tables;
    int64_t rot_cols = 0, act_from = total;
    NodePtr with_rot, with_act;
    for (const auto &n : group) {
      const int64_t N = n->consts[0]->meta.GetShape()[1];
      if (n->rot) { with_rot = n; rot_cols += N; }
      if (n->act) { with_act = n; act_from -= N; }
    }
    if (with_rot) tables = {with_rot->consts[with_rot->consts.size() - 2], with_rot->consts.back()};
    const int64_t rot = with_rot ? with_rot->rot : 0, rot_head = with_rot ? with_rot->rot_head : 0, rot_len = with_rot ? with_rot->rot_len : 1;
    if (with_act) {
      first->act = with_act->act;
      std::copy(with_act->act_param, with_act->act_param + 3, first->act_param);
      first->act_from = act_from;  // 0: all of them
    }
    first->rot = rot; first->rot_head = rot_head; first->rot_cols = rot_cols; first->rot_len = rot_len;
    first->consts.clear();
    first->consts.push_back(wcat);
    if (bcat) first->consts.push_back(bcat);
    first->consts.insert(first->consts.end(), tables.begin(), tables.end());
    first->output = merged;
    std::unordered_set<const flow::Node *> gone;
    for (const auto &n : group)
      if (n != first) gone.insert(n.get());
    std::vector<NodePtr> next;
    for (const auto &n : f.nodes) {
      if (gone.count(n.get())) continue;
      next.push_back(n);
      if (n == first) next.insert(next.end(), slices.begin(), slices.end());
    }
    f.nodes = std::move(next);
    return true;
  }
  return false;
}

}  // namespace

size_t FusionPasses::Run(flow::Flow &flow, bool join, bool relayout) {
  const size_t before = flow.nodes.size();
  Rewriter rw(flow);
  using Pass = bool (*)(Rewriter &, const NodePtr &);
  // order matters: bias before GELU / activation before residual, residual before Add+LN
  const Pass passes[] = {FuseEmbedding, FuseMask, FuseBias, FuseGeluIntoGemm, FuseBiasGelu, FuseActivation,
                         FuseResidual, FuseSecondResidual, FuseAddLayerNorm, FuseScaledMaskedSoftmax, FuseAttention, FuseSilu, FuseSiluIntoConv, FuseSqueezeExcite, FuseGateIntoConv, FuseResidualIntoConv, FuseMulAdd, FuseRotary, FuseMulAddChain, FuseSpanConvolution};
  auto until_done = [&](Pass pass) {
    bool again = true;
    while (again) {
      again = false;
      for (size_t i = 0; i < flow.nodes.size(); ++i) {
        const NodePtr n = flow.nodes[i];
        if (pass(rw, n)) { rw.Commit(); again = true; break; }
      }
    }
  };
  for (Pass pass : passes) until_done(pass);
  if (join) {
    until_done(FuseRotaryIntoGemm);
    while (FoldSharedLayerNorms(rw)) {}
    if (relayout) until_done(PointwiseAsProduct);
  }
  while (MergeSiblingGemms(flow, join)) {}
  if (join) {
    rw.Index();
    until_done(JoinSummedProducts);
    until_done(JoinConcatenatedProduct);
  }
  // drop tensors nothing refers to any more
  std::unordered_set<const flow::Region *> live;
  for (const auto &n : flow.nodes) {
    live.insert(n->output.get());
    for (const auto &r : n->inputs) live.insert(r.get());
    for (const auto &r : n->consts) live.insert(r.get());
  }
  std::vector<RegionPtr> kept;
  for (const auto &r : flow.regions) {
    if (live.count(r.get()) || r->kind == flow::Region::kInput || r->kind == flow::Region::kOutput) kept.push_back(r);
    else flow.by_name.erase(r->name);
  }
  flow.regions = std::move(kept);
  return before - flow.nodes.size();
}

}  // namespace worker
}  // namespace fluidml

// Attention core on pairs of half-precision numbers (gemm_pair.cu): out = softmax(Q K^T / divisor + mask) V
// for head size 64, one CTA per (head, 128 query rows), keys in blocks of 64 with a running softmax.  The
// scores never leave the SM.
//
// What bounds it: the exponentials and operand splits (about 14 instructions per score and 6 per element
// of K and V), not the MMAs (768 clocks per 128 x 64 block against some 1300 issue slots per scheduler), so
// the work is laid out to keep the schedulers busy: separate warps split K and V for the block ahead while
// the softmax warps work on this one, and two CTAs share an SM.  Measured, 192 heads of 384 x 384: 51 us a launch,
// where two batched 3xTF32 GEMMs around a softmax took 163; 64 causal heads of 512: 25 us against 87.
//
//   warp 0      loads (tensor maps, 128-byte swizzle): Q once, K and V of a block into one of two raw stages
//   warp 1      MMAs: S = Q K^T with Q from tensor memory, O += P V with P from tensor memory; order
//               S(0), S(1), PV(0), S(2), PV(1) ..., so that the scores of the next block are computed while
//               the softmax of this one runs
//   warps 2-5   softmax, thread = query row = TMEM lane: scores -> P = exp(s - m), split and written over them
//   warps 6-9   split K and V: unswizzled core matrices [8 k values][row][16 bytes] in shared memory, K as
//               (key, 8 of d), V transposed as (d, 8 keys), so that both are K-major B operands
//
// Scales (powers of two).  Q per row, K and V per block, all from exact finite maxima (largest in [2^14, 2^15):
// 22 bits down to 2^-17 of it, below that an absolute error of 2^-39 of it); Q's and K's are divided out with the attention scale.  P is exp(s - m) times 2^x, x = (scale of O) - (scale of
// this block's V): O is one accumulator.  O is rescaled, by a round trip through registers, only when a
// block's maximum exceeds the reference m of a row by more than 4 in log2 or V's scale moves by more than 3:
// the largest P of a row is then within 2^-3 .. 2^7, and what its pair leaves out is below 2^-22 of it.
#include "gemm_common.cuh"
#include "pair_common.cuh"
#include <algorithm>
#include <cfloat>

namespace fml {
namespace {

constexpr int kThreads = 320, kKeys = 64, kD = 64;
constexpr int kRawStage = 2 * kKeys * kD * 4;    // K and V of a block, fp32: 32 KiB (= Q of the tile)
constexpr int kSplit = kKeys * kD * 4;           // hi and lo of K or V: 16 KiB
constexpr int kHalfSplit = kSplit / 2;           // offset of lo
constexpr uint32_t kColS = 0, kColO = 128, kColQ = 192;  // tensor memory: two score buffers (P over S), O, Q
enum { kNoMask = 0, kKeyMask = 1, kFullMask = 2, kCausal = 3 };

struct AttnPairArgs {
  int Sq, Sk, nb0;
  int q_h, q_b, k_h, k_b, v_h, v_b;  // whether the operand varies over heads / batches
  const float *mask;
  int64_t m_s[4], o_s[4];
  float *out;
  float inv_divisor;
  int *status;
};

template <int MASK>
__global__ void __launch_bounds__(kThreads, 2)
attention_pair_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                      const __grid_constant__ CUtensorMap map_v, const AttnPairArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  // [ raw stage 0 | raw stage 1 | split K | split V | mask | barriers ]
  const uint32_t raw0 = smem_u32(smem), split_k = raw0 + 2 * kRawStage, split_v = split_k + kSplit;
  uint8_t *const split_k_ptr = smem + 2 * kRawStage, *const split_v_ptr = split_k_ptr + kSplit;
  float *const mask_s = reinterpret_cast<float *>(split_v_ptr + kSplit);            // [2][64]
  int *const exp_s = reinterpret_cast<int *>(mask_s + 2 * kKeys);                   // [2][2]: scale exponents of K, V
  unsigned *const max_s = reinterpret_cast<unsigned *>(exp_s + 4);                  // [3][2]: their largest magnitudes
  uint64_t *const bars = reinterpret_cast<uint64_t *>(max_s + 8);
  const uint32_t bar0 = smem_u32(bars);
  const uint32_t bar_raw_full = bar0, bar_raw_empty = bar0 + 16, bar_s = bar0 + 32, bar_q_full = bar0 + 48, bar_q_ready = bar0 + 56,
                 bar_k_ready = bar0 + 64, bar_k_free = bar0 + 72, bar_v_ready = bar0 + 80, bar_p_ready = bar0 + 88, bar_pv = bar0 + 104, bar_final = bar0 + 112;
  uint32_t *const tmem_slot = reinterpret_cast<uint32_t *>(bars + 15);
  volatile int *const abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const bool leader = elect_one();
  const int q0 = blockIdx.x * kBM, h = blockIdx.y % a.nb0, b = blockIdx.y / a.nb0;
  int n_blocks = (a.Sk + kKeys - 1) / kKeys;
  if (MASK == kCausal) n_blocks = min(n_blocks, (q0 + kBM + kKeys - 1) / kKeys);  // keys beyond the tile's last row

  if (threadIdx.x == 0) {
    tma_prefetch_map(&map_q);
    tma_prefetch_map(&map_k);
    tma_prefetch_map(&map_v);
    for (int s = 0; s < 2; ++s) { mbar_init(bar_raw_full + 8u * s, 1); mbar_init(bar_raw_empty + 8u * s, 4); mbar_init(bar_s + 8u * s, 1); mbar_init(bar_p_ready + 8u * s, 4); }
    mbar_init(bar_q_full, 1);
    mbar_init(bar_q_ready, 4);
    mbar_init(bar_k_ready, 4);
    mbar_init(bar_k_free, 1);
    mbar_init(bar_v_ready, 4);
    mbar_init(bar_pv, 1);
    mbar_init(bar_final, 1);
    *abort_flag = 0;
    for (int i = 0; i < 6; ++i) max_s[i] = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(smem_u32(tmem_slot), 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // Only now may the next kernel start (tensor memory: see gemm_tc.cu).
  pdl_launch_dependents();
  pdl_wait();

  bool ok = true;
  if (warp == 0) {
    // ------------------------------------------------------------ loads: Q lands in raw stage 1, block j in stage j & 1
    if (g_drop_loads != 1) {
      if (leader) {
        mbar_expect_tx(bar_q_full, kRawStage);
        for (int i = 0; i < 2; ++i)
          tma_load_4d(raw0 + kRawStage + (uint32_t)i * (kBM * 128), &map_q, bar_q_full, 32 * i, q0, a.q_h ? h : 0, a.q_b ? b : 0);
      }
      int issued = 0;
      for (int j = 0; j < n_blocks && ok; ++j) {
        const uint32_t s = (uint32_t)j & 1u, ph = (uint32_t)(j >> 1) & 1u;
        if (j == 1) ok = mbar_wait_warp(bar_q_ready, 0u, abort_flag);  // Q has left its stage
        if (ok) ok = mbar_wait_warp(bar_raw_empty + 8u * s, ph ^ 1u, abort_flag);
        if (!ok) break;
        if (leader) {
          const uint32_t dst = raw0 + s * kRawStage, bar = bar_raw_full + 8u * s;
          mbar_expect_tx(bar, kRawStage);
          for (int i = 0; i < 2; ++i) {
            tma_load_4d(dst + (uint32_t)i * (kKeys * 128), &map_k, bar, 32 * i, j * kKeys, a.k_h ? h : 0, a.k_b ? b : 0);
            tma_load_4d(dst + (uint32_t)(2 + i) * (kKeys * 128), &map_v, bar, 32 * i, j * kKeys, a.v_h ? h : 0, a.v_b ? b : 0);
          }
        }
        ++issued;
      }
      if (!ok) {  // bounded drain of the loads in flight
        volatile int never = 0;
        mbar_wait_warp(bar_q_full, 0u, &never);
        for (int j = max(0, issued - 2); j < issued; ++j)
          mbar_wait_warp(bar_raw_full + 8u * ((uint32_t)j & 1u), (uint32_t)(j >> 1) & 1u, &never);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    const uint32_t idesc = instr_desc_f16(64);
    const uint64_t desc_k = smem_desc(split_k, kKeys * 16u, 128u, 0u), desc_v = smem_desc(split_v, kD * 16u, 128u, 0u);
    ok = mbar_wait_warp(bar_q_ready, 0u, abort_flag);
    for (int j = 0; j <= n_blocks && ok; ++j) {
      if (j < n_blocks) {  // scores of block j
        ok = mbar_wait_warp(bar_k_ready, (uint32_t)j & 1u, abort_flag);
        if (!ok) break;
        tc_fence_after();
        if (leader) {
          const uint32_t d = tmem_base + kColS + ((uint32_t)j & 1u) * 64u;
#pragma unroll
          for (int k = 0; k < kD / 16; ++k) {
            const uint32_t q_hi = tmem_base + kColQ + 8u * k, q_lo = q_hi + 32u;
            const uint64_t kh = desc_k + (uint64_t)(2 * k * (kKeys * 16) >> 4), kl = kh + (uint64_t)(kHalfSplit >> 4);
            umma_f16_ts(d, q_lo, kh, idesc, k ? 1u : 0u);
            umma_f16_ts(d, q_hi, kl, idesc, 1u);
            umma_f16_ts(d, q_hi, kh, idesc, 1u);
          }
          umma_commit(bar_s + 8u * ((uint32_t)j & 1u));
          umma_commit(bar_k_free);
        }
        __syncwarp();
      }
      if (j > 0) {  // context of block j - 1
        const uint32_t ph = (uint32_t)(j - 1) & 1u;
        ok = mbar_wait_warp(bar_v_ready, ph, abort_flag) && mbar_wait_warp(bar_p_ready + 8u * ph, (uint32_t)((j - 1) >> 1) & 1u, abort_flag);
        if (!ok) break;
        tc_fence_after();
        if (leader) {
          const uint32_t p = tmem_base + kColS + ph * 64u, d = tmem_base + kColO;
#pragma unroll
          for (int k = 0; k < kKeys / 16; ++k) {
            const uint32_t p_hi = p + 8u * k, p_lo = p_hi + 32u;
            const uint64_t vh = desc_v + (uint64_t)(2 * k * (kD * 16) >> 4), vl = vh + (uint64_t)(kHalfSplit >> 4);
            umma_f16_ts(d, p_lo, vh, idesc, (j == 1 && k == 0) ? 0u : 1u);
            umma_f16_ts(d, p_hi, vl, idesc, 1u);
            umma_f16_ts(d, p_hi, vh, idesc, 1u);
          }
          umma_commit(bar_pv);
        }
        __syncwarp();
      }
    }
    if (!ok) *abort_flag = 1;
    if (leader) umma_drain(bar_final);
    __syncwarp();
  } else if (warp < 6) {
    // ------------------------------------------------------------ softmax: thread = query row
    const int q = warp & 3, row = q * 32 + lane;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
    const int grow = q0 + row, row_in = min(grow, a.Sq - 1);
    int e_q = 0;
    ok = mbar_wait_warp(bar_q_full, 0u, abort_flag);
    if (ok) {
      float4 x[16];
      float m = 0.0f;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float4 *src = reinterpret_cast<const float4 *>(smem + kRawStage + i * (kBM * 128) + row * 128);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float4 y = src[c ^ (row & 7)];
          x[8 * i + c] = y;
          m = fmaxf(m, fmaxf(fmaxf(fabsf(y.x), fabsf(y.y)), fmaxf(fabsf(y.z), fabsf(y.w))));
        }
      }
      e_q = scale_exponent(m, 14);
      const float s = pow2(e_q);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          split_pair(x[8 * i + c].x, x[8 * i + c].y, s, hi[2 * c], lo[2 * c]);
          split_pair(x[8 * i + c].z, x[8 * i + c].w, s, hi[2 * c + 1], lo[2 * c + 1]);
        }
        tmem_st16(lane_addr + kColQ + 16u * i, hi);
        tmem_st16(lane_addr + kColQ + 32u + 16u * i, lo);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_q_ready);
    }
    constexpr float kLog2e = 1.4426950408889634f;
    float m_ref = 0.0f, l = 0.0f;
    int ev_ref = 0, ev_min = 0;
    for (int j = 0; j < n_blocks && ok; ++j) {
      const uint32_t buf = (uint32_t)j & 1u;
      ok = mbar_wait_warp(bar_s + 8u * buf, (uint32_t)(j >> 1) & 1u, abort_flag);
      if (!ok) break;
      tc_fence_after();
      const int ev = exp_s[2 * buf + 1];
      const float f = a.inv_divisor * pow2(max(-126, min(126, -(e_q + exp_s[2 * buf]))));
      const int key0 = j * kKeys;
      float v[64];
      tmem_ld32(lane_addr + kColS + buf * 64u, v);
      tmem_ld32(lane_addr + kColS + buf * 64u + 32u, v + 32);
      float m_blk = -FLT_MAX;  // (finite, for blocks without a visible key)
      if (MASK == kKeyMask) {
        const float *mk = mask_s + buf * kKeys;  // keys beyond the last one hold -infinity
#pragma unroll
        for (int i = 0; i < 64; ++i) v[i] = fmaf(v[i], f, mk[i]);
      } else if (MASK == kFullMask) {
        const float *mp = a.mask + (int64_t)b * a.m_s[0] + (int64_t)h * a.m_s[1] + row_in * a.m_s[2] + (int64_t)key0 * a.m_s[3];
#pragma unroll
        for (int i = 0; i < 64; ++i) v[i] = key0 + i < a.Sk ? fmaf(v[i], f, mp[i * a.m_s[3]]) : -INFINITY;
      } else {
        const int last = MASK == kCausal ? min(grow, a.Sk - 1) - key0 : a.Sk - 1 - key0;  // last visible key of the block
        if (__all_sync(0xffffffffu, last >= 63)) {
#pragma unroll
          for (int i = 0; i < 64; ++i) v[i] *= f;
        } else {
#pragma unroll
          for (int i = 0; i < 64; ++i) v[i] = i <= last ? v[i] * f : -INFINITY;
        }
      }
#pragma unroll
      for (int i = 0; i < 64; i += 4) m_blk = fmaxf(m_blk, fmaxf(fmaxf(v[i], v[i + 1]), fmaxf(v[i + 2], v[i + 3])));
      if (j == 0) {
        m_ref = m_blk;
        ev_ref = ev_min = ev;
      } else if (__any_sync(0xffffffffu, m_blk > m_ref + 4.0f / kLog2e) || abs(ev_ref - ev) > 3) {
        // rare: a new maximum out of reach, or a block of V far from those before it
        ok = mbar_wait_warp(bar_pv, (uint32_t)(j - 1) & 1u, abort_flag);
        if (!ok) break;
        tc_fence_after();
        const float m_new = fmaxf(m_ref, m_blk), fac_l = exp2f((m_ref - m_new) * kLog2e);
        ev_min = min(ev_min, ev);
        const int ev_new = min(ev, ev_min + 60);  // (keeps O finite; V so small beside an earlier block adds nothing)
        const float fac = fac_l * pow2(max(-126, ev_new - ev_ref));
        l *= fac_l;
        m_ref = m_new;
        ev_ref = ev_new;
#pragma unroll
        for (int c = 0; c < 64; c += 16) {
          uint32_t o[16];
          tmem_ld16(lane_addr + kColO + (uint32_t)c, o);
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * fac);
          tmem_st16(lane_addr + kColO + (uint32_t)c, o);
        }
        tmem_wait_st();
      }
      const int xi = max(ev_ref - ev, -60);
      const float x = (float)xi;
      float sum = 0.0f;
      uint32_t hi[32], lo[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        // exp(s - m) 2^x; the difference is formed first: the rounding of m log2(e) would show in every score
        const float p0 = ex2_approx(fmaf(v[2 * i] - m_ref, kLog2e, x)), p1 = ex2_approx(fmaf(v[2 * i + 1] - m_ref, kLog2e, x));
        sum += p0 + p1;
        split_pair(p0, p1, 1.0f, hi[i], lo[i]);
      }
      l += sum * pow2(-xi);
      tmem_st32(lane_addr + kColS + buf * 64u, hi);
      tmem_st32(lane_addr + kColS + buf * 64u + 32u, lo);
      tmem_wait_st();
      tc_fence_before();
      // PV's phase must not be two behind at the wait after the loop: the last scores only say that PV(n - 3) is over
      if (j > 0 && j == n_blocks - 1) ok = mbar_wait_warp(bar_pv, (uint32_t)(j - 1) & 1u, abort_flag);
      __syncwarp();
      if (ok && lane == 0) mbar_arrive(bar_p_ready + 8u * buf);  // (two barriers: the softmax may be a block ahead of PV)
    }
    // ---- out = O / l
    if (ok) ok = mbar_wait_warp(bar_pv, (uint32_t)(n_blocks - 1) & 1u, abort_flag);
    if (ok) {
      tc_fence_after();
      const float inv = pow2(-ev_ref) / l;
      float *dst = a.out + (int64_t)b * a.o_s[0] + (int64_t)h * a.o_s[1] + (int64_t)row_in * a.o_s[2];
      const bool vec = a.o_s[3] == 1 && (a.o_s[2] & 3) == 0 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
#pragma unroll
      for (int c = 0; c < 64; c += 32) {
        float o[32];
        __syncwarp();
        tmem_ld32(lane_addr + kColO + (uint32_t)c, o);
        if (grow >= a.Sq) {
        } else if (vec) {
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            *reinterpret_cast<float4 *>(dst + c + i) = make_float4(o[i] * inv, o[i + 1] * inv, o[i + 2] * inv, o[i + 3] * inv);
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) dst[(int64_t)(c + i) * a.o_s[3]] = o[i] * inv;
        }
      }
    }
  } else {
    // ------------------------------------------------------------ split of K and V
    const int t = threadIdx.x - 192, r = t & 63, half = t >> 6;
    for (int j = 0; j < n_blocks; ++j) {
      const uint32_t s = (uint32_t)j & 1u, slot = (uint32_t)j % 3u;
      float4 xk[8];
      float xv[32];
      if (ok) ok = mbar_wait_warp(bar_raw_full + 8u * s, (uint32_t)(j >> 1) & 1u, abort_flag);
      if (ok) {
        // K: key r, d in [32 half, 32 half + 32); V: d = r, keys in [32 half, 32 half + 32)
        const uint8_t *raw = smem + s * kRawStage;
        const float4 *src = reinterpret_cast<const float4 *>(raw + half * (kKeys * 128) + r * 128);
        float mk = 0.0f, mv = 0.0f;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          xk[c] = src[c ^ (r & 7)];
          mk = fmaxf(mk, fmaxf(fmaxf(fabsf(xk[c].x), fabsf(xk[c].y)), fmaxf(fabsf(xk[c].z), fabsf(xk[c].w))));
        }
        const uint8_t *rv = raw + (2 + (r >> 5)) * (kKeys * 128) + (r & 3) * 4;
        const int cv = (r & 31) >> 2;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int key = half * 32 + i;
          xv[i] = *reinterpret_cast<const float *>(rv + key * 128 + ((cv ^ (key & 7)) << 4));
          mv = fmaxf(mv, fabsf(xv[i]));
        }
        // (an infinity is in no maximum: it would flush the block's other keys and columns to zero)
        const unsigned wk = __reduce_max_sync(0xffffffffu, mk <= FLT_MAX ? __float_as_uint(mk) : 0u);
        const unsigned wv = __reduce_max_sync(0xffffffffu, mv <= FLT_MAX ? __float_as_uint(mv) : 0u);
        if (lane == 0) { atomicMax(max_s + 2 * slot, wk); atomicMax(max_s + 2 * slot + 1, wv); }
        if (MASK == kKeyMask && t < kKeys) {
          const int key = j * kKeys + t;
          // finite even where the mask is the lowest float: a row whose keys are all masked stays uniform
          mask_s[s * kKeys + t] = key < a.Sk ? a.mask[(int64_t)b * a.m_s[0] + (int64_t)h * a.m_s[1] + (int64_t)key * a.m_s[3]] : -INFINITY;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_raw_empty + 8u * s);
      } else {
        *abort_flag = 1;
      }
      named_barrier_sync(1, 128);  // reached by all four warps in every round, failed or not, so nobody is left waiting
      if (!ok) continue;
      const int ek = scale_exponent(__uint_as_float(max_s[2 * slot]), 14), ev = scale_exponent(__uint_as_float(max_s[2 * slot + 1]), 14);
      if (t == 0) {
        exp_s[2 * s] = ek;
        exp_s[2 * s + 1] = ev;
        const uint32_t next = slot == 0 ? 2u : slot - 1u;  // slot of block j + 2: free since this barrier
        max_s[2 * next] = max_s[2 * next + 1] = 0u;
      }
      if (j > 0) ok = mbar_wait_warp(bar_k_free, (uint32_t)(j - 1) & 1u, abort_flag);
      if (!ok) continue;
      const float sk = pow2(ek), sv = pow2(ev);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t hi[4], lo[4];
        split_pair(xk[2 * c].x, xk[2 * c].y, sk, hi[0], lo[0]);
        split_pair(xk[2 * c].z, xk[2 * c].w, sk, hi[1], lo[1]);
        split_pair(xk[2 * c + 1].x, xk[2 * c + 1].y, sk, hi[2], lo[2]);
        split_pair(xk[2 * c + 1].z, xk[2 * c + 1].w, sk, hi[3], lo[3]);
        uint8_t *o = split_k_ptr + (half * 4 + c) * (kKeys * 16) + r * 16;
        *reinterpret_cast<uint4 *>(o) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4 *>(o + kHalfSplit) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      }
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_k_ready);
      if (j > 0) ok = mbar_wait_warp(bar_pv, (uint32_t)(j - 1) & 1u, abort_flag);
      if (!ok) continue;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) split_pair(xv[8 * c + 2 * i], xv[8 * c + 2 * i + 1], sv, hi[i], lo[i]);
        uint8_t *o = split_v_ptr + (half * 4 + c) * (kD * 16) + r * 16;
        *reinterpret_cast<uint4 *>(o) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4 *>(o + kHalfSplit) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      }
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_v_ready);
    }
  }
  if (!ok) {
    if (leader) atomicOr(a.status, kStatusTimeout);
    *abort_flag = 1;
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

// 4-D map over [batch][head][row][d]; boxes of 32 floats x `box_rows` rows, 128-byte swizzle.
int attention_map(CUtensorMap *map, const float *base, int64_t rows, int64_t row_stride, int64_t nh, int64_t h_stride, int64_t nb,
                  int64_t b_stride, int box_rows) {
  return make_gemm_map(map, base, kD, rows, row_stride, nh, h_stride, nb, b_stride, 32, box_rows, CU_TENSOR_MAP_SWIZZLE_128B);
}

}  // namespace

// What attention_tc_eligible accepts (operands with unit-stride d and 16-byte aligned rows, blocks that
// belong on tensor cores) with head size 64.
bool attention_pair_shape_ok(int64_t d, int64_t d_v) { return d == kD && d_v == kD; }

int launch_attention_pair(int64_t nb1, int64_t nb0, int64_t Sq, int64_t Sk, const float *q, const int64_t *q_s, const float *k,
                          const int64_t *k_s, const float *v, const int64_t *v_s, const float *mask, const int64_t *m_s, bool causal,
                          float divisor, float *out, const int64_t *o_s, cudaStream_t s) {
  AttnPairArgs a;
  a.Sq = (int)Sq; a.Sk = (int)Sk; a.nb0 = (int)nb0;
  for (int i = 0; i < 4; ++i) { a.m_s[i] = mask ? m_s[i] : 0; a.o_s[i] = o_s[i]; }
  a.mask = mask; a.out = out; a.inv_divisor = 1.0f / divisor;
  a.q_h = q_s[1] != 0; a.q_b = q_s[0] != 0; a.k_h = k_s[1] != 0; a.k_b = k_s[0] != 0; a.v_h = v_s[1] != 0; a.v_b = v_s[0] != 0;
  a.status = device_status_word();
  FML_REQUIRE(a.status, FML_CUDA_ERROR, "fml_attention: no device status word");
  CUtensorMap mq, mk, mv;
  int st = attention_map(&mq, q, Sq, q_s[2], nb0, q_s[1], nb1, q_s[0], kBM);
  if (st == FML_OK) st = attention_map(&mk, k, Sk, k_s[3], nb0, k_s[1], nb1, k_s[0], kKeys);
  if (st == FML_OK) st = attention_map(&mv, v, Sk, v_s[2], nb0, v_s[1], nb1, v_s[0], kKeys);
  if (st != FML_OK) return st;
  const size_t smem = 2 * kRawStage + 2 * kSplit + 2 * kKeys * 4 + 4 * 4 + 8 * 4 + 15 * 8 + 16;
  using KernelFn = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const AttnPairArgs);
  static const KernelFn kernels[4] = {attention_pair_kernel<kNoMask>, attention_pair_kernel<kKeyMask>, attention_pair_kernel<kFullMask>,
                                      attention_pair_kernel<kCausal>};
  static bool attr_set[64] = {false};
  int dev = 0;
  FML_CUDA(cudaGetDevice(&dev));
  if (!attr_set[dev & 63]) {
    for (KernelFn f : kernels) FML_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_set[dev & 63] = true;
  }
  const int kind = causal ? kCausal : !mask ? kNoMask : m_s[2] == 0 ? kKeyMask : kFullMask;
  const dim3 grid((unsigned)((Sq + kBM - 1) / kBM), (unsigned)(nb0 * nb1));
  FML_CUDA(launch_kernel(kernels[kind], grid, dim3(kThreads), smem, s, mq, mk, mv, a));
  return FML_OK;
}

}  // namespace fml

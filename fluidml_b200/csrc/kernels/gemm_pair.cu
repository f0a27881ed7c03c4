// tcgen05 GEMM for constant right-hand sides (weights) on pairs of half-precision numbers: every fp32
// operand x is scaled by a power of two and split into hi = fp16(x), lo = fp16(x - hi), 22 significant
// bits together, and lo*hi + hi*lo + hi*hi are accumulated in fp32 (kind::f16).  The same products as
// the 3xTF32 kernel (gemm_tc.cu), whose truncated hi / lo carry 21 to 22 bits, but a kind::f16
// instruction consumes 16 k values where kind::tf32 consumes 8 and both take N / 2 clocks: half the
// tensor time.
//
// Range.  fp16 has 5 exponent bits, so both sides are scaled by powers of two (exact):
//   B  per column, at packing time (fml_gemm_pack): the column's largest magnitude lands in
//      [2^14, 2^15); elements 2^-17 below it still have all 22 bits, and below that an absolute error of
//      2^-39 of it.
//   A  per row and k slice, on the fly: the first k block (32 values) of the row puts its largest
//      magnitude into [2^3, 2^4).  Elements far below it keep an absolute error of 2^-28 of that
//      magnitude, below fp32's own rounding of the sum; 2^12 of headroom is left for larger values
//      further along, and a CTA with a long k range looks at 64 values spread over it as well: what comes
//      out of a convolution and a ReLU has stretches of zeros and of small values (VGG-16's first dense layer
//      took 351 us instead of 64 when two of 32 rows needed a second attempt).  A row whose first block is all zero takes 2^8, right for magnitudes from 2^-12 to
//      2^7.  A row that outgrows its scale overflows to infinity, which the finished accumulator shows
//      in every column, and one whose magnitudes stay below the default scale's reach is noticed by
//      their maximum: the CTA then finds the exact row maxima and does its tile a second time with
//      them (in captured graphs 128 x 768 x 3072: 10.7 us usually, 13.5 when one row is, 29.9 when all are).
//      Infinities and NaNs of the input come out as NaN, as in the 3xTF32 kernel.
// The powers of two are divided out again when the accumulator leaves tensor memory (rows) and in the
// epilogue (columns).
//
// B is stored packed: per k block of 32, per 8 columns, the 512-byte K-major atom (64-byte swizzle) of hi
// and the one of lo side by side.  A tile's share of a k block is then one contiguous run, fetched by one
// untiled bulk copy, and nothing of B is converted on chip.  (Bytes streamed: 4 per weight, as fp32.)
// Blocks of 32 rather than 64 k values: at tile 256 shared memory holds 128 KiB of B, and four blocks in
// flight cover the ~1 us of an L2 round trip where two did not (each block is ~0.4 us of MMAs).
//
// Roles, 320 threads: warp 0 loads (A boxes of 32 floats x 128 rows by tensor map, B runs; the two rings
// are filled independently, whichever has room), warp 1 issues the MMAs, warps 2-9 convert: two sets of
// four warps (a warp may write the 32 TMEM lanes of its index modulo 4) that take alternate blocks;
// thread = row.  A's fp32 stage is free as soon as it is converted, the
// tensor-memory stage and B's stage when the MMAs are done.  Epilogue, split-K over a cluster and
// bounded waits as in gemm_tc.cu.
#include "gemm_epilogue.cuh"
#include "pair_common.cuh"
#include <algorithm>
#include <cstdlib>

namespace fml {
namespace {

constexpr int kPairA = kBM * kPK * 4;        // bytes of A per block: a box of 128 rows x 128 bytes
constexpr int kDefaultExponent = 8;          // scale 2^8 of a row whose first k block is all zero
constexpr int kSampleBlocks = 48;            // from this many k blocks on, a row's scale is chosen with samples of all of them
constexpr int kPairThreads = 320;
constexpr int kConvThreads = 256;

struct PairArgs {
  GemmProblem p;
  GemmEpilogue e;
  GemmExtras x;
  EpilogueShape shape;
  const char *packed;       // B atoms
  const float *col_scale;   // 2^-s of each column
  int n_pad;                // columns in the packed image (multiple of 16)
  int tile_n, split_k, stages_a, stages_b, two_accs;
  int tiles_m, tiles_n, kb_total, kb_per_split;
  int *status;
};

// Stores a box of 32 rows x 32 floats (128-byte swizzle) from shared memory; what lies outside the tensor is left out.
__device__ __forceinline__ void tma_store_4d(const CUtensorMap *map, uint32_t src, int x, int y, int z, int w) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// A finished tile without split-K, residual or scaling leaves the accumulator for global memory without passing through
// other threads: a thread has a row, so column scale, bias, rotation (its partner features are in the same registers) and
// activation are applied 16 columns at a time as they come out of tensor memory, a warp's 32 x 32 box goes to shared
// memory (128-byte swizzle; the rings are free) and one lane hands it to a bulk store, which also clips ragged edges.
// TileEpilogue's second pass -- read the staged tile, finish it, store it -- took 3.6 us of a 128 x 192 tile (reads alone
// 1.4, stores alone 2.2, arithmetic alone 2.0, one after the other with two warps per scheduler), 6.8 with GELU.  Captured graphs, tuned, before and after:
// 1024 x 768 x 3072 17.5 -> 15.5 us, with GELU 21.3 -> 16.9; 6144 x 768 x 2304 62 -> 56; 6144 x 768 x 3072 with GELU
// 94 -> 82; 2048 x 1024 x 7168 with rotation and GELU 105 -> 90.
template <int ACT, bool PROJ>
__device__ __forceinline__ void store_tile_bulk(const PairArgs &a, const CUtensorMap *map_c, uint8_t *smem, uint32_t lane_addr, float row_inv,
                                                const float *col_mul, const float *col_add, int tile_m, int tile_n, int set, int q, int lane, int z0,
                                                int z1) {
  const int BN = a.tile_n, row0 = tile_m * kBM + q * 32;
  const bool rows = row0 < a.p.M;
  // this row's table entries; the tile's heads begin at multiples of rot_head >= 16 columns
  float co[16], si[16];
  const bool rotates = PROJ && a.x.rot && tile_n * BN < a.x.rot_cols;
  if (rotates) {
    const int at = (int)((unsigned)(row0 + lane) % (unsigned)a.x.rot_len) * 16;
#pragma unroll
    for (int j = 0; j < 16; j += 4) {
      const float4 c = __ldg(reinterpret_cast<const float4 *>(a.x.rot_cos + at + j)), s = __ldg(reinterpret_cast<const float4 *>(a.x.rot_sin + at + j));
      co[j] = c.x; co[j + 1] = c.y; co[j + 2] = c.z; co[j + 3] = c.w;
      si[j] = s.x; si[j + 1] = s.y; si[j + 2] = s.z; si[j + 3] = s.w;
    }
  }
  for (int c0 = set * 32; c0 < BN; c0 += 64) {
    uint8_t *box = smem + (size_t)((c0 >> 5) * 4 + q) * 4096 + lane * 128;
#pragma unroll 1
    for (int h = 0; h < 32; h += 16) {
      uint32_t r[16];
      float v[16];
      tmem_ld16(lane_addr + (uint32_t)(c0 + h), r);
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        const float4 m = *reinterpret_cast<const float4 *>(col_mul + c0 + h + j), b = *reinterpret_cast<const float4 *>(col_add + c0 + h + j);
        // powers of two: one rounding, the bias's sum
        v[j] = fmaf(__uint_as_float(r[j]) * row_inv, m.x, b.x); v[j + 1] = fmaf(__uint_as_float(r[j + 1]) * row_inv, m.y, b.y);
        v[j + 2] = fmaf(__uint_as_float(r[j + 2]) * row_inv, m.z, b.z); v[j + 3] = fmaf(__uint_as_float(r[j + 3]) * row_inv, m.w, b.w);
      }
      const int n = tile_n * BN + c0 + h;
      if (PROJ && rotates && n < a.x.rot_cols && n % a.x.rot_head == 0) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float lo = v[j], hi = v[j + 8];
          v[j] = __fadd_rn(__fmul_rn(lo, co[j]), __fmul_rn(-hi, si[j]));
          v[j + 8] = __fadd_rn(__fmul_rn(hi, co[j + 8]), __fmul_rn(lo, si[j + 8]));
        }
      }
      if (!PROJ || n >= a.x.act_from) {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = act_op<ACT>(a.e, v[j]);
      } else if (ACT != FML_ACT_NONE && n + 16 > a.x.act_from) {  // the activation begins within these columns
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = n + j >= a.x.act_from ? act_op<ACT>(a.e, v[j]) : v[j];
      }
#pragma unroll
      for (int j = 0; j < 16; j += 4)
        *reinterpret_cast<float4 *>(box + ((((h + j) >> 2) ^ (lane & 7)) << 4)) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
    }
    fence_async_smem();
    __syncwarp();
    if (lane == 0 && rows && tile_n * BN + c0 < a.p.N) {
      tma_store_4d(map_c, smem_u32(smem) + (uint32_t)((c0 >> 5) * 4 + q) * 4096u, tile_n * BN + c0, row0, a.p.c_b0 ? z0 : 0, a.p.c_b1 ? z1 : 0);
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
  }
  if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // shared memory stays until it has been read
}

// MODE: what else a launch does.  kProj: several projections of the same rows side by side (the queries, keys and
// values of an attention block and the first product of a feed-forward layer), with the rotary embedding on the
// first columns and the activation on the last (TileEpilogue).  kTwoA: A's columns come from two tensors, [A | A2] * B:
// the sum of two products (both halves of a parallel-residual block) or a concatenation's product, one launch
// and one reduction for both; k blocks do not straddle the seam (k1 is a multiple of 32).  A sum has a second accumulator where
// tensor memory has room (two_accs): lo * hi + hi * lo there, 2^-11 of the other's size, whose cuts then come once per
// sixteen k values instead of three times (pair_exact).
enum { kPlain = 0, kProj = 1, kTwoA = 2 };

// BULK: store_tile_bulk ends the launch.  (Both endings in one kernel cost its main loop 3 % -- registers.)
template <int ACT, int MODE, bool BULK>
__global__ void __launch_bounds__(kPairThreads, 2)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_a2,
                 const __grid_constant__ CUtensorMap map_c, const PairArgs a) {
  // (no static shared memory in this kernel: the dynamic part starts on a 1024-byte boundary)
  extern __shared__ __align__(1024) uint8_t smem[];
  const int BN = a.tile_n;
  const int pitch = BN + 4;
  const uint32_t b_bytes = (uint32_t)BN * kPairB;
  const size_t ring_bytes = (size_t)a.stages_a * kPairA + (size_t)a.stages_b * b_bytes;
  const size_t staging_bytes = ((size_t)kBM * pitch * 4 + 1023) / 1024 * 1024;
  const size_t data_bytes = ring_bytes > staging_bytes ? ring_bytes : staging_bytes;
  const uint32_t ring_a = smem_u32(smem), ring_b = ring_a + (uint32_t)a.stages_a * kPairA;
  float *staging = reinterpret_cast<float *>(smem);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + data_bytes);
  const uint32_t bar_full_a = smem_u32(bars), bar_empty_a = bar_full_a + 8u * a.stages_a;
  const uint32_t bar_full_b = bar_empty_a + 8u * a.stages_a, bar_conv = bar_full_b + 8u * a.stages_b;
  const uint32_t bar_empty_b = bar_conv + 8u * a.stages_b, bar_accum = bar_empty_b + 8u * a.stages_b;
  const uint32_t bar_decide = bar_accum + 8u, bar_final = bar_decide + 8u;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * a.stages_a + 3 * a.stages_b + 3);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  volatile int *redo_flag = reinterpret_cast<volatile int *>(tmem_slot + 2);
  unsigned *row_seen = reinterpret_cast<unsigned *>(tmem_slot + 4);          // [128], rows on the default scale: largest scaled magnitude
  signed char *row_exp = reinterpret_cast<signed char *>(row_seen + kBM);  // [128], scale exponent; -128: the default one

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const bool leader = elect_one();
  const int tile = blockIdx.x, tile_m = tile % a.tiles_m, tile_n = tile / a.tiles_m;
  const int split = blockIdx.y;
  const int z = blockIdx.z, z0 = z % (int)a.p.nb0, z1 = z / (int)a.p.nb0;
  const int kb0 = min(a.kb_total, split * a.kb_per_split);
  const int kb1 = min(a.kb_total, kb0 + a.kb_per_split);
  const int nkb = kb1 - kb0;
  const uint32_t acc_cols = ((uint32_t)BN + 31u) & ~31u, small = MODE == kTwoA && a.two_accs ? acc_cols : 0u;  // second accumulator
  const uint32_t a_col0 = acc_cols + small;
  uint32_t tmem_cols = 32;
  while (tmem_cols < a_col0 + 32u * (uint32_t)a.stages_b) tmem_cols <<= 1;
  // the packed run of this tile in k block kb; the last tile of a ragged N stops at the image's edge
  // (the columns it leaves unwritten in shared memory are never stored)
  const int n_cols = min(BN, a.n_pad - tile_n * BN);
  const uint32_t b_run = (uint32_t)n_cols * kPairB;
  const char *b_src = a.packed + ((size_t)kb0 * a.n_pad + (size_t)tile_n * BN) * kPairB;
  const size_t b_step = (size_t)a.n_pad * kPairB;
  // Weights that one row of tiles reads cross L2 once per pass: evict-first (gemm_tc.cu).
  const bool b_stream = a.tiles_m == 1;
  const uint64_t b_policy = b_stream ? l2_policy_evict_first() : 0ull;
  auto load_b = [&](int it, int s) {
    const uint32_t dst = ring_b + (uint32_t)s * b_bytes, bar = bar_full_b + 8u * s;
    mbar_expect_tx(bar, b_run);
    if (b_stream) bulk_load_hint(dst, b_src + (size_t)it * b_step, b_run, bar, b_policy);
    else bulk_load(dst, b_src + (size_t)it * b_step, b_run, bar);
  };

  if (threadIdx.x == 0) tma_prefetch_map(&map_a);
  if (MODE == kTwoA && threadIdx.x == 0) tma_prefetch_map(&map_a2);
  const int kb_seam = MODE == kTwoA ? (int)(a.x.k1 / kPK) : 0;  // first k block of A2
  if (a.p.prefetch_bytes && threadIdx.x == 64) {  // the next launch's weights (gemm_tc.cu)
    const uint64_t pf_policy = l2_policy_evict_first();
    const unsigned long long ctas = (unsigned long long)gridDim.x * gridDim.y * gridDim.z;
    const unsigned long long cta = blockIdx.x + (unsigned long long)gridDim.x * (blockIdx.y + (unsigned long long)gridDim.y * blockIdx.z);
    const unsigned long long share = ((a.p.prefetch_bytes + ctas - 1) / ctas + 127ull) & ~127ull;
    const unsigned long long lo = cta * share, hi = min(a.p.prefetch_bytes & ~15ull, lo + share);
    for (unsigned long long off = lo; off < hi; off += 16384ull) {
      const unsigned n = (unsigned)min(16384ull, hi - off);
      asm volatile("cp.async.bulk.prefetch.L2.global.L2::cache_hint [%0], %1, %2;"
                   ::"l"(a.p.prefetch + off), "r"(n), "l"(pf_policy) : "memory");
    }
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < a.stages_a; ++s) {
      mbar_init(bar_full_a + 8u * s, 1);
      mbar_init(bar_empty_a + 8u * s, 4);  // one arrival per warp of the converter set
    }
    for (int s = 0; s < a.stages_b; ++s) {
      mbar_init(bar_full_b + 8u * s, 1);
      mbar_init(bar_conv + 8u * s, 4);
      mbar_init(bar_empty_b + 8u * s, 1);
    }
    mbar_init(bar_accum, 1);
    mbar_init(bar_decide, 8);
    mbar_init(bar_final, 1);
    *abort_flag = 0;
    *redo_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x >= 64 && threadIdx.x < 64 + kBM) row_seen[threadIdx.x - 64] = 0u;
  if (warp == 1) tmem_alloc(smem_u32(tmem_slot), tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // Only now may the next kernel start: its CTAs must not take tensor memory that this one still has
  // to allocate (they give theirs back after waiting for this grid, so that would never end).
  pdl_launch_dependents();
  // Weights do not depend on the preceding kernel: the first stages are on their way while it drains.
  const int pre_b = min(a.stages_b, nkb);
  if (threadIdx.x == 0 && g_drop_loads != 1)
    for (int it = 0; it < pre_b; ++it) load_b(it, it);
  // vectors the epilogue will ask for, cold in HBM: into L2 now
  if (warp == 2) {
    const float *bp = a.p.bias && a.p.bias_sm == 0 && a.p.bias_sn == 1
                          ? a.p.bias + (int64_t)z0 * a.p.bias_b0 + (int64_t)z1 * a.p.bias_b1 : nullptr;
    for (int64_t n = (int64_t)tile_n * BN + lane * 8; n < min((int64_t)(tile_n + 1) * BN, a.p.N); n += 256) {
      if (bp) asm volatile("prefetch.global.L2 [%0];" ::"l"(bp + n));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(a.col_scale + n));
    }
  }
  pdl_wait();

  // A's ring in two parts, one per converter set (pair_stages)
  const int ring_0 = (a.stages_a + 1) >> 1, ring_1 = a.stages_a >> 1;
  TileEpilogue<ACT, kConvThreads, true, MODE == kProj> epi;
  float row_inv = 1.0f;  // converter threads: undoes the scale of this thread's row
  if (warp == 0) {
    // ------------------------------------------------------------ loads
    if (g_drop_loads != 1) {
      const int ca2 = a.p.a_b0 ? z0 : 0, ca3 = a.p.a_b1 ? z1 : 0;
      bool ok = true;
      int issued_0 = 0, issued_1 = 0, issued_b = pre_b;  // counted over both attempts: ring positions go on
      RingPos ra0, ra1, rb;
      for (int it = 0; it < pre_b; ++it) rb.step(a.stages_b);
      for (int attempt = 0; attempt < 2 && ok; ++attempt) {
        if (attempt) {
          ok = mbar_wait_warp(bar_decide, 0u, abort_flag);
          if (!ok || !*redo_flag || g_drop_loads) break;
        }
        int ia = 0, ib = attempt ? 0 : pre_b;
        uint32_t idle = 0;
        while (ia < nkb || ib < nkb) {  // whichever ring has room
          bool moved = false;
          const bool odd = ia & 1;
          const uint32_t sa = (uint32_t)(odd ? ring_0 + ra1.s : ra0.s);
          if (ia < nkb && mbar_test_warp(bar_empty_a + 8u * sa, (odd ? ra1.ph : ra0.ph) ^ 1u)) {
            const uint32_t bar = bar_full_a + 8u * sa;
            if (leader) {
              mbar_expect_tx(bar, kPairA);
              if (MODE == kTwoA && kb0 + ia >= kb_seam)
                tma_load_4d(ring_a + sa * kPairA, &map_a2, bar, (kb0 + ia - kb_seam) * kPK, tile_m * kBM, a.x.a2_b0 ? z0 : 0, a.x.a2_b1 ? z1 : 0);
              else
                tma_load_4d(ring_a + sa * kPairA, &map_a, bar, (kb0 + ia) * kPK, tile_m * kBM, ca2, ca3);
            }
            ++ia; moved = true;
            if (odd) { ++issued_1; ra1.step(ring_1); } else { ++issued_0; ra0.step(ring_0); }
          }
          if (ib < nkb && mbar_test_warp(bar_empty_b + 8u * rb.s, rb.ph ^ 1u)) {
            if (leader) load_b(ib, rb.s);
            ++ib; ++issued_b; moved = true;
            rb.step(a.stages_b);
          }
          if (moved) idle = 0;
          else if ((++idle & 255u) == 0 && (*abort_flag || idle >= 64u * g_wait_limit)) { ok = false; break; }
        }
      }
      if (!ok) {
        if (leader) atomicOr(a.status, kStatusTimeout);
        *abort_flag = 1;
        // bounded drain of the loads already in flight before the CTA may exit
        volatile int never = 0;
        for (int i = max(0, issued_0 - ring_0); i < issued_0; ++i)
          mbar_wait_warp(bar_full_a + 8u * (i % ring_0), (uint32_t)(i / ring_0) & 1u, &never);
        for (int i = max(0, issued_1 - ring_1); i < issued_1; ++i)
          mbar_wait_warp(bar_full_a + 8u * (ring_0 + i % ring_1), (uint32_t)(i / ring_1) & 1u, &never);
        for (int i = max(0, issued_b - a.stages_b); i < issued_b; ++i)
          mbar_wait_warp(bar_full_b + 8u * (i % a.stages_b), (uint32_t)(i / a.stages_b) & 1u, &never);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    const uint32_t idesc = instr_desc_f16(BN);
    const uint64_t desc_b = smem_desc(ring_b, 16u, 2 * kAtom, 4u);  // hi atoms (64-byte swizzle); lo one atom further
    RingPos rb;
    bool ok = true;
    for (int attempt = 0; attempt < 2 && ok; ++attempt) {
      if (attempt) {
        ok = mbar_wait_warp(bar_decide, 0u, abort_flag);
        if (!ok || !*redo_flag) break;
      }
      for (int it = 0; it < nkb; ++it) {
        ok = mbar_wait_warp(bar_full_b + 8u * rb.s, rb.ph, abort_flag) && mbar_wait_warp(bar_conv + 8u * rb.s, rb.ph, abort_flag);
        if (!ok) break;
        tc_fence_after();
        if (leader) {
          const uint64_t db0 = desc_b + (((uint32_t)rb.s * b_bytes) >> 4);
          const uint32_t ta = tmem_base + a_col0 + (uint32_t)rb.s * 32u;
#pragma unroll
          for (int j = 0; j < kPK / 16; ++j) {
            const uint32_t a_hi = ta + (uint32_t)j * 8u, a_lo = a_hi + 16u;
            const uint64_t db = db0 + (uint32_t)j * 2u, dbl = db + (kAtom >> 4);
            umma_f16_ts(tmem_base + small, a_lo, db, idesc, (it == 0 && j == 0) ? 0u : 1u);
            umma_f16_ts(tmem_base + small, a_hi, dbl, idesc, 1u);
            umma_f16_ts(tmem_base, a_hi, db, idesc, MODE == kTwoA && small && it == 0 && j == 0 ? 0u : 1u);
          }
          umma_commit(bar_empty_b + 8u * rb.s);  // B stage and TMEM stage reusable
        }
        __syncwarp();
        rb.step(a.stages_b);
      }
      if (ok && leader) umma_commit(bar_accum);  // with no MMA outstanding (nkb == 0) this arrives at once
      __syncwarp();
    }
    if (!ok) {
      if (leader) atomicOr(a.status, kStatusTimeout);
      *abort_flag = 1;
    }
    if (leader) umma_drain(bar_final);
    __syncwarp();
  } else {
    // ------------------------------------------------------------ converter
    const int q = warp & 3, row = q * 32 + lane, set = (warp - 2) >> 2, swz = row & 7;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
    const bool real_row = (int64_t)tile_m * kBM + row < a.p.M;
    bool ok = true;
    int k_row = 0;       // the row is scaled by 2^k_row
    auto load_row = [&](int slot, float4 *x) {  // 16-byte chunks swizzled by (row & 7)
      const float4 *src = reinterpret_cast<const float4 *>(smem + (size_t)slot * kPairA + row * 128);
#pragma unroll
      for (int c = 0; c < 8; ++c) x[c] = src[c ^ swz];
    };
    bool guess = false;  // this row's scale is the default one
    float seen = 0.0f;   // largest scaled magnitude this thread converted (kept while a row of its warp has the default scale)
    bool bad = false;    // this row needs a second attempt
    const float *const a_row = a.p.a + (int64_t)z0 * a.p.a_b0 + (int64_t)z1 * a.p.a_b1 + ((int64_t)tile_m * kBM + row) * a.p.a_sm;
    auto a2_row = [&](int r) { return a.x.a2 + (int64_t)z0 * a.x.a2_b0 + (int64_t)z1 * a.x.a2_b1 + ((int64_t)tile_m * kBM + r) * a.x.a2_sm; };
    float sampled = 0.0f;
    if (nkb >= kSampleBlocks && set == 0 && real_row) {
      float4 y[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int kb = kb0 + i * (nkb - 1) / 16;
        y[i] = *reinterpret_cast<const float4 *>(MODE == kTwoA && kb >= kb_seam ? a2_row(row) + (int64_t)(kb - kb_seam) * kPK : a_row + (int64_t)kb * kPK);
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) sampled = fmaxf(sampled, fmaxf(fmaxf(fabsf(y[i].x), fabsf(y[i].y)), fmaxf(fabsf(y[i].z), fabsf(y[i].w))));
    }
    __syncwarp();
    const int ring_n = set ? ring_1 : ring_0;
    const uint32_t slot0 = set ? (uint32_t)ring_0 : 0u;
    RingPos ma;  // within this set's part of A's ring
    for (int attempt = 0; attempt < 2 && ok; ++attempt) {
      // position of this set's block in B's ring (the second attempt's blocks follow the first's)
      const int at = attempt * nkb + set;
      RingPos mb{at % a.stages_b, (uint32_t)(at / a.stages_b) & 1u};
      float4 x[8];
      bool have = false;
      if (attempt) {
        // exact maxima of those rows over the CTA's k range, straight from global memory (rare)
        for (uint32_t left = __ballot_sync(0xffffffffu, bad); left; left &= left - 1) {
          const int r = __ffs((int)left) - 1;
          const float *src = a_row + (int64_t)(r - lane) * a.p.a_sm;
          const int64_t k_end = min((int64_t)kb1 * kPK, a.p.K);
          float m;
          if (MODE == kTwoA) {
            m = kb0 < kb_seam ? warp_row_max(src, (int64_t)kb0 * kPK, min(k_end, a.x.k1), lane) : 0.0f;
            if (kb1 > kb_seam) m = fmaxf(m, warp_row_max(a2_row(q * 32 + r), (int64_t)max(kb0 - kb_seam, 0) * kPK, k_end - a.x.k1, lane));
          } else {
            m = warp_row_max(src, (int64_t)kb0 * kPK, k_end, lane);
          }
          if (lane == r) k_row = scale_exponent(m, 14);
        }
      } else {
        // set 0 finds the scale in block 0, set 1 takes it over
        if (set == 0) {
          float m = sampled;
          if (nkb > 0) {
            ok = mbar_wait_warp(bar_full_a + 8u * (slot0 + ma.s), ma.ph, abort_flag);
            if (ok) {
              load_row(slot0 + ma.s, x);
              have = true;
#pragma unroll
              for (int c = 0; c < 8; ++c)
                m = fmaxf(m, fmaxf(fmaxf(fabsf(x[c].x), fabsf(x[c].y)), fmaxf(fabsf(x[c].z), fabsf(x[c].w))));
            }
          }
          guess = !(m > 0.0f);
          k_row = guess ? kDefaultExponent : scale_exponent(m, 3);
          row_exp[row] = (signed char)(guess ? -128 : k_row);
          named_barrier_arrive(1, 256);  // also when the wait gave up: set 1 must not be left behind
        } else {
          named_barrier_sync(1, 256);
          k_row = row_exp[row];
          guess = k_row == -128;
          if (guess) k_row = kDefaultExponent;
        }
      }
      const float s_mul = pow2(k_row);
      row_inv = pow2(-k_row);
      const bool watch = attempt == 0 && __any_sync(0xffffffffu, guess);
      for (int it = set; it < nkb && ok; it += 2) {
        if (!have) {
          ok = mbar_wait_warp(bar_full_a + 8u * (slot0 + ma.s), ma.ph, abort_flag);
          if (!ok) break;
          load_row(slot0 + ma.s, x);
        }
        if (watch) {
#pragma unroll
          for (int c = 0; c < 8; ++c)
            seen = fmaxf(seen, s_mul * fmaxf(fmaxf(fabsf(x[c].x), fabsf(x[c].y)), fmaxf(fabsf(x[c].z), fabsf(x[c].w))));
        }
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          split_pair(x[c].x, x[c].y, s_mul, hi[2 * c], lo[2 * c]);
          split_pair(x[c].z, x[c].w, s_mul, hi[2 * c + 1], lo[2 * c + 1]);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_empty_a + 8u * (slot0 + ma.s));  // the values are in registers
        ma.step(ring_n);
        // the MMAs that read this tensor-memory stage last are done
        ok = mbar_wait_warp(bar_empty_b + 8u * mb.s, mb.ph ^ 1u, abort_flag);
        if (!ok) break;
        tc_fence_after();
        const uint32_t t_hi = lane_addr + a_col0 + (uint32_t)mb.s * 32u;
        tmem_st16(t_hi, hi);
        tmem_st16(t_hi + 16u, lo);
        // the next block of this set, if it is there: its shared-memory latency runs under these stores
        have = it + 2 < nkb && __all_sync(0xffffffffu, mbar_test(bar_full_a + 8u * (slot0 + ma.s), ma.ph));
        if (have) load_row(slot0 + ma.s, x);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_conv + 8u * mb.s);
        mb.step(a.stages_b); mb.step(a.stages_b);
      }
      if (BULK) {
        const int64_t n = (int64_t)tile_n * BN + (threadIdx.x - 64);  // this thread's column (a tile has at most 256)
        if (!attempt) {  // (in registers that the other epilogue uses)
          const bool real = n < min((int64_t)(tile_n + 1) * BN, a.p.N);
          epi.cs.x = real ? a.col_scale[n] : 0.0f;
          epi.bvec.x = real && a.p.bias ? a.p.bias[(int64_t)z0 * a.p.bias_b0 + (int64_t)z1 * a.p.bias_b1 + n] : 0.0f;
        }
      } else if (!attempt) epi.preload(a.p, a.shape, BN, tile_m, tile_n, split, a.split_k, z0, z1, threadIdx.x - 64, a.col_scale);
      if (ok) ok = mbar_wait_warp(bar_accum, (uint32_t)attempt, abort_flag);
      if (attempt) break;
      // A row whose hi overflowed shows it in every column of the accumulator; one on the default scale
      // must have had a value that this scale resolves, unless it is all zero.
      tc_fence_after();
      const float v0 = ok && nkb > 0 ? tmem_ld1(lane_addr) : 0.0f;
      tc_fence_before();
      if (watch && guess && seen > 0.0f) atomicMax(&row_seen[row], __float_as_uint(seen));
      named_barrier_sync(2, 256);  // every converter warp comes here, whether its waits were met or not
      bad = !(fabsf(v0) <= 3.4028235e38f);
      if (watch && guess) {
        const float m = __uint_as_float(row_seen[row]);
        bad = bad || (m > 0.0f && m < 0.0625f);
      }
      if (__any_sync(0xffffffffu, bad) && lane == 0) *redo_flag = 1;
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_decide);
      ok = ok && mbar_wait_warp(bar_decide, 0u, abort_flag);
      if (!ok || !*redo_flag) break;
    }
    if (!ok) {
      atomicOr(a.status, kStatusTimeout);
      *abort_flag = 1;
    }
    tc_fence_after();  // the accumulator's loads stay behind the wait for the MMAs of the last attempt, in either ending
    if (BULK) {
      // behind the boxes, in what a staged tile's padding would take
      float *cols = reinterpret_cast<float *>(smem + (size_t)BN * kBM * 4);
      const int et = threadIdx.x - 64;
      if (et < BN) { cols[et] = epi.cs.x; cols[BN + et] = epi.bvec.x; }
      named_barrier_sync(3, kConvThreads);
      if (ok) store_tile_bulk<ACT, MODE == kProj>(a, &map_c, smem, lane_addr, row_inv, cols, cols + BN, tile_m, tile_n, set, q, lane, z0, z1);
    } else {
    // Accumulator row -> staging row; the rings are free (every load has been consumed).  The two
    // sets take alternate groups of 32 columns.
    float *dst = staging + (size_t)row * pitch;
    for (int c0 = set * 32; c0 < BN; c0 += 64) {
      float v[32];
      if (ok && nkb > 0) {
        tmem_ld32(lane_addr + (uint32_t)c0, v);
        if (MODE == kTwoA && small) {
          float w[32];
          tmem_ld32(lane_addr + small + (uint32_t)c0, w);
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] += w[i];
        }
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = 0.0f;
      }
#pragma unroll
      for (int i = 0; i < 32; i += 4)
        if (c0 + i < BN)
          *reinterpret_cast<float4 *>(dst + c0 + i) =
              make_float4(v[i] * row_inv, v[i + 1] * row_inv, v[i + 2] * row_inv, v[i + 3] * row_inv);
    }
    }
  }

  // ---------------------------------------------------------------- reduce + epilogue
  tc_fence_before();
  __syncthreads();
  const int S = a.split_k;
  if (S > 1) cluster_sync_all();
  if (warp >= 2 && !BULK)
    epi.finish(a.p, a.e, a.shape, staging, pitch, BN, tile_m, tile_n, split, S, z0, z1, threadIdx.x - 64, a.col_scale, a.x);
  if (S > 1) cluster_sync_relaxed();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, tmem_cols);
  }
}

// ---------------------------------------------------------------- packing
// One block per 8 columns: the columns' largest magnitudes, then their k blocks.
__global__ void __launch_bounds__(256) gemm_pack_kernel(const float *b, int64_t K, int64_t N, int64_t sk, int64_t sn,
                                                        char *packed, float *col_scale, int n_pad, int kb_total) {
  __shared__ unsigned m_bits[8];
  const int n0 = blockIdx.x * 8;
  if (threadIdx.x < 8) m_bits[threadIdx.x] = 0u;
  __syncthreads();
  const int r = threadIdx.x & 7;
  float m = 0.0f;
  if (n0 + r < N)
    for (int64_t k = threadIdx.x >> 3; k < K; k += 32) m = fmaxf(m, fabsf(b[k * sk + (n0 + r) * sn]));
  atomicMax(&m_bits[r], __float_as_uint(m));  // non-negative floats order as their bits
  __syncthreads();
  float s = 1.0f, inv = 1.0f;
  if (m_bits[r]) {
    const int e = scale_exponent(__uint_as_float(m_bits[r]), 14);
    s = pow2(e);
    inv = pow2(-e);
  }
  if (threadIdx.x < 8) col_scale[n0 + r] = inv;
  for (int64_t i = threadIdx.x >> 3; i < (int64_t)kb_total * 4; i += 32) {  // (k block, 16-byte chunk) of column r
    const int64_t kb = i >> 2;
    const int c = (int)(i & 3);
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t k = kb * kPK + c * 8 + j * 2;
      const float x0 = n0 + r < N && k < K ? b[k * sk + (n0 + r) * sn] : 0.0f;
      const float x1 = n0 + r < N && k + 1 < K ? b[(k + 1) * sk + (n0 + r) * sn] : 0.0f;
      split_pair(x0, x1, s, hi[j], lo[j]);
    }
    // 64-byte swizzle: the chunk index is XORed with bits 7-8 of the address, i.e. (row / 2) mod 4
    char *atom = packed + ((size_t)kb * n_pad + n0) * kPairB + r * (kPK * 2) + ((c ^ (r >> 1)) * 16);
    *reinterpret_cast<uint4 *>(atom) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4 *>(atom + kAtom) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
}

// ---------------------------------------------------------------- host side
int n_padded(int64_t n) { return (int)((n + 15) / 16 * 16); }
int k_blocks(int64_t k) { return (int)((k + kPK - 1) / kPK); }
size_t atoms_bytes(int64_t k, int64_t n) { return (size_t)k_blocks(k) * n_padded(n) * kPairB; }

size_t pair_smem(int tile_n, int stages_a, int stages_b) {
  const size_t ring = (size_t)stages_a * kPairA + (size_t)stages_b * tile_n * kPairB;
  const size_t staging = ((size_t)kBM * (tile_n + 4) * 4 + 1023) / 1024 * 1024;
  return std::max(ring, staging) + (2 * stages_a + 3 * stages_b + 3) * 8 + 16 + kBM * 5;
}

constexpr size_t kSmemSm = 228 * 1024, kSmemCta = 227 * 1024;
constexpr size_t kSmemHalf = kSmemSm / 2 - 1024;  // what lets two CTAs share an SM

// Ring depths for a tile width: the deepest that fits the budget and the 512 TMEM columns.
// A's ring is split between the converter sets, which take alternate blocks, so that a set sees every phase of
// its slots.  In one common ring of odd depth it would see every other one: loads land out of order, and while
// the other set's block is still on its way the parity of the phase before it reads as this set's own -- stale
// values would be converted and the slot given back a second time.  (B's barriers need no such care from two
// stages on: MMAs end in order, and a set's previous wait covers the phase before.)
bool pair_stages(int tile_n, int per, bool two_ctas, bool two_accs, int *stages_a, int *stages_b, size_t *smem) {
  const int acc = (tile_n + 31) / 32 * 32 * (two_accs ? 2 : 1);
  const size_t budget = two_ctas ? kSmemHalf : kSmemCta;
  const int tmem = two_ctas ? 256 : 512;
  int best_a = 0, best_b = 0;
  double best = 0.0;
  for (int sb = 1; sb <= 8 && acc + 32 * sb <= tmem; ++sb)
    for (int sa = 1; sa <= 8; ++sa) {
      if (pair_smem(tile_n, sa, sb) > budget) continue;
      if (sa > per || sb > per) continue;   // no deeper than the k loop
      if (std::min(sa, sb) == 1 && per > 1) continue;
      // both rings count; the shallower one limits
      const double score = std::min(sa, sb) * 8 + sa + sb;
      if (score > best) { best = score; best_a = sa; best_b = sb; }
    }
  if (!best_a) return false;
  if (two_ctas && per > 1 && std::min(best_a, best_b) < std::min(per, 3)) return false;
  *stages_a = best_a;
  *stages_b = best_b;
  size_t need = pair_smem(tile_n, best_a, best_b);
  // no more CTAs on an SM than its 512 TMEM columns serve at once (gemm_tc.cu)
  unsigned cols = 32;
  while ((int)cols < acc + 32 * best_b) cols <<= 1;
  need = std::max(need, kSmemSm / (512 / cols + 1) + 1024);
  *smem = need;
  return need <= kSmemCta;
}

}  // namespace

size_t pair_packed_bytes(int64_t K, int64_t N) { return atoms_bytes(K, N) + (size_t)n_padded(N) * sizeof(float); }

int pair_pack(const float *b, int64_t K, int64_t N, int64_t sk, int64_t sn, void *dst, cudaStream_t s) {
  const int np = n_padded(N), kb = k_blocks(K);
  char *packed = static_cast<char *>(dst);
  gemm_pack_kernel<<<np / 8, 256, 0, s>>>(b, K, N, sk, sn, packed, reinterpret_cast<float *>(packed + atoms_bytes(K, N)), np, kb);
  FML_CUDA(cudaGetLastError());
  return FML_OK;
}

bool pair_rotates(const GemmProblem &p, const GemmExtras &x, const PairPlan &plan) {
  if (!x.rot) return false;
  // groups of rot columns lie within a tile and, four columns to a lane, within a warp
  const bool pow2 = (x.rot & (x.rot - 1)) == 0;
  if (!pow2 || x.rot < 8 || x.rot > 128 || x.rot_head % x.rot || plan.tile_n % x.rot) return false;
  if (!aligned16(x.rot_cos) || !aligned16(x.rot_sin)) return false;
  // tiles of rotated columns take the epilogue's 16-byte path (TileEpilogue::Where), which a split of 3, 5, 6 or 7 does not
  // -- nor an activation from inside a group of four columns
  if ((plan.split_k & (plan.split_k - 1)) != 0 || x.act_from % 4 != 0) return false;
  if ((x.rot_cols + plan.tile_n - 1) / plan.tile_n * (int64_t)plan.tile_n > p.N) return false;
  if (p.c_sn != 1 || p.c_sm % 4 || p.c_b0 % 4 || p.c_b1 % 4 || !aligned16(p.c) || p.res) return false;
  return !p.bias || (p.bias_sn == 1 && p.bias_sm % 4 == 0 && p.bias_b0 % 4 == 0 && p.bias_b1 % 4 == 0 && aligned16(p.bias));
}

// Whether finished tiles may leave by bulk stores (store_tile_bulk): boxes of 32 columns, rows of C that begin and end on
// 16-byte boundaries, and an epilogue of column scale, per-column bias, rotation by 16 features and activation.
static bool bulk_stores(const GemmProblem &p, const GemmEpilogue &e, const GemmExtras &x, const PairPlan &plan) {
  if (plan.two_accs || plan.split_k != 1 || plan.tile_n % 32 || p.res || e.divisor != 1.0f || e.alpha != 1.0f || (p.bias && e.beta != 1.0f)) return false;
  // (a bulk store clips at 16-byte steps: with 50 columns it would write zeros into two more)
  if (p.N % 4 || p.c_sn != 1 || p.c_sm <= 0 || p.c_sm % 4 || !aligned16(p.c)) return false;
  if (p.c_b0 < 0 || p.c_b0 % 4 || p.c_b1 < 0 || p.c_b1 % 4 || (p.nb0 > 1 && !p.c_b0) || (p.nb1 > 1 && !p.c_b1)) return false;
  if (p.bias && (p.bias_sm != 0 || p.bias_sn != 1)) return false;
  return !x.rot || (x.rot == 16 && x.rot_head % 16 == 0);
}

// An accumulator is cut to 24 bits at every instruction, once or (one accumulator for all three products) three times per
// sixteen k values, and that is nearly all of a long product's error.  Joined products fill the SMs with fewer slices of k than
// they would apart, and a sum has the k range of both.  So a sum only takes splits that cut no more often than its longer
// half would be cut alone, in the split that fills the SMs with tiles of 256; products side by side as many slices, up to the four
// that they mostly have apart, as the SMs hold with tiles of 128, two to an SM.
// Error (relative 2-norm, rows x (1024 + 4096) x 1024, activations non-negative) and time, best tiles, of two launches / one with
// one accumulator / as chosen here: 77 rows 1.2e-6 21.1 us / 1.7e-6 14.8 / 6.0e-7 14.9; 308 2.2e-6 29.2 / 1.7e-6 20.6 / 1.2e-6 22.5;
// 1024 2.3e-6 39.5 / 3.4e-6 29.9 / 2.4e-6 38.0; 2048 4.6e-6 62.5 / 7.1e-6 55.3 / 3.4e-6 61.1 (four slices of tiles of 256, which
// leave no room for a second accumulator).  Side by side: 77 x 1024 x (3072 + 4096) takes tiles of 64 unsplit or of 128 in four
// slices within 2 %, and a whole model was off by 4.3e-6 with the former, 1.4e-6 with the latter; 512 rows, which fill the
// SMs unsplit, would pay 20 % of a pass for two slices (4.1e-6 -> 2.7e-6, 3.9e-6 with all products apart).
static int fill_slices(int64_t tiles) {
  int s = 1;
  while (s < 8 && tiles * s * 2 <= kSms) s *= 2;
  return s;
}
static int sum_slices(int64_t M, int64_t N, int64_t batch) { return fill_slices((M + kBM - 1) / kBM * ((N + 255) / 256) * batch); }
bool pair_exact(const GemmProblem &p, const GemmExtras &x, int split, bool two_accs) {
  const int64_t batch = p.nb0 * p.nb1, kb = k_blocks(p.K), per = (kb + split - 1) / split;
  if (x.summed) {
    const int64_t longer = k_blocks(std::max(x.k1, p.K - x.k1)), s = sum_slices(p.M, p.N, batch);
    return per * (two_accs ? 1 : 3) <= (longer + s - 1) / s * 3;
  }
  if (x.act_from) {
    const int64_t tiles = (p.M + kBM - 1) / kBM * ((p.N + 127) / 128) * batch, s = std::min(4, fill_slices((tiles + 1) / 2));  // (two CTAs to an SM)
    return per <= (kb + s - 1) / s;
  }
  return true;
}

bool plan_gemm_pair(const GemmProblem &p, const GemmExtras &x, const fml_gemm_params &gp, PairPlan &plan) {
  if (!gp.b_packed || gp.precision != FML_GEMM_AUTO) return false;
  // A goes through a tensor map (K contiguous, 16-byte aligned rows); fewer than 32 rows stay on the
  // weight-streaming fp32 kernel, as with the 3xTF32 kernel
  if (p.M < 32 || p.N < 16 || p.K < 16 || p.a_sk != 1 || !aligned16(p.a) || p.a_sm <= 0 || p.a_sm % 4) return false;
  auto stride_ok = [](int64_t s) { return s == 0 || (s > 0 && s % 4 == 0); };
  if (!stride_ok(p.a_b0) || !stride_ok(p.a_b1) || p.b_b0 || p.b_b1) return false;
  if (x.a2 && (!aligned16(x.a2) || x.a2_sm <= 0 || x.a2_sm % 4 || !stride_ok(x.a2_b0) || !stride_ok(x.a2_b1) || x.k1 % kPK)) return false;
  if ((x.act_from || x.rot) && gp.act != FML_ACT_GELU_ERF && gp.act != FML_ACT_NONE) return false;  // the instantiations there are
  if (x.a2 && gp.act != FML_ACT_NONE) return false;
  if ((x.act_from || x.rot) && x.a2) return false;
  if (p.M > (1ll << 30) || p.N > (1ll << 24) || p.K > (1ll << 30) || p.nb0 * p.nb1 > 65535) return false;
  if (!aligned16(gp.b_packed)) return false;
  const int kb_total = k_blocks(p.K);
  const int64_t tiles_m = (p.M + kBM - 1) / kBM, batch = p.nb0 * p.nb1;
  // Default tile and split (the tuner measures the alternatives): time of a CTA = set-up and epilogue
  // plus its k blocks at one SM's fill path (80 bytes per ns: slower than the block's 6 MMAs of N / 2 clocks
  // at every width); waves of CTAs at one or two per SM.  Against the best of all tiles and splits, over 23
  // products of 32 to 6144 rows in captured graphs: 1.27x in the geometric mean (77 x 1024 x 4096: 21.5 us
  // for 11.4, a wide tile split eight ways; from 1024 rows on within 1.06x).
  const int tn_opts[] = {32, 64, 96, 128, 192, 256};
  const int sk_opts[] = {1, 2, 4, 8};
  double best = 1e30;
  bool found = false;
  for (int tn : tn_opts) {
    if (gp.tile_n) tn = gp.tile_n;
    tn = std::min(tn, n_padded(p.N));
    tn = std::max(16, std::min(256, tn / 16 * 16));
    for (int sk : sk_opts) {
      if (gp.split_k) sk = gp.split_k;
      if (sk > 8 || sk > kb_total) { if (gp.split_k) break; continue; }
      const int per = (kb_total + sk - 1) / sk;
      for (int two = 1; two >= 0; --two) {
        if (gp.tile_n && gp.ctas_per_sm && gp.ctas_per_sm != two + 1) continue;
        int sa, sb;
        size_t smem;
        const bool accs = x.summed && pair_stages(tn, per, two != 0, true, &sa, &sb, &smem);
        if (!accs && !pair_stages(tn, per, two != 0, false, &sa, &sb, &smem)) continue;
        const int64_t ctas = tiles_m * ((p.N + tn - 1) / tn) * batch * sk;
        const int slots = (two ? 2 : 1) * kSms * (sk == 8 ? 0.87 : sk == 4 ? 0.97 : 1.0);
        const double waves = (double)((ctas + slots - 1) / slots);
        const double t_kb = (double)(kPairA + tn * kPairB) / 80e3;
        const double t_fixed = 3.0 + (double)kBM * tn / sk * 4.0 / 20e3 + (sk > 1 ? 0.6 : 0.0);
        const double inexact = gp.split_k || pair_exact(p, x, sk, accs) ? 0.0 : 1e9;  // only where there is nothing else
        const double t = waves * (t_fixed + per * t_kb * (two && ctas > kSms ? 2.0 : 1.0)) + inexact;
        if (t < best) {
          best = t;
          found = true;
          plan.tile_n = tn; plan.split_k = sk; plan.stages_a = sa; plan.stages_b = sb;
          plan.smem_bytes = smem; plan.ctas_per_sm = two + 1; plan.two_accs = accs;
        }
      }
      if (gp.split_k) break;
    }
    if (gp.tile_n) break;
  }
  return found;
}

int launch_gemm_pair(const GemmProblem &p, const GemmEpilogue &e, const GemmExtras &x, const PairPlan &plan, const void *packed, cudaStream_t s) {
  PairArgs a;
  a.p = p; a.e = e; a.x = x;
  const bool rotates = pair_rotates(p, x, plan);
  if (!rotates) a.x.rot = 0;
  const int mode = x.a2 ? kTwoA : x.act_from || rotates ? kProj : kPlain;
  a.shape = epilogue_shape(plan.tile_n, kConvThreads);
  a.packed = static_cast<const char *>(packed);
  a.col_scale = reinterpret_cast<const float *>(a.packed + atoms_bytes(p.K, p.N));
  a.n_pad = n_padded(p.N);
  a.tile_n = plan.tile_n; a.split_k = plan.split_k; a.stages_a = plan.stages_a; a.stages_b = plan.stages_b;
  a.two_accs = plan.two_accs;
  a.tiles_m = (int)((p.M + kBM - 1) / kBM);
  a.tiles_n = (int)((p.N + plan.tile_n - 1) / plan.tile_n);
  a.kb_total = k_blocks(p.K);
  a.kb_per_split = (a.kb_total + plan.split_k - 1) / plan.split_k;
  a.status = device_status_word();
  FML_REQUIRE(a.status, FML_CUDA_ERROR, "fml_gemm: no device status word");
  CUtensorMap map_a, map_a2;
  int st = make_gemm_map(&map_a, p.a, x.a2 ? x.k1 : p.K, p.M, p.a_sm, p.nb0, p.a_b0, p.nb1, p.a_b1, 32, kBM, CU_TENSOR_MAP_SWIZZLE_128B);
  if (st != FML_OK) return st;
  map_a2 = map_a;
  if (x.a2) {
    st = make_gemm_map(&map_a2, x.a2, p.K - x.k1, p.M, x.a2_sm, p.nb0, x.a2_b0, p.nb1, x.a2_b1, 32, kBM, CU_TENSOR_MAP_SWIZZLE_128B);
    if (st != FML_OK) return st;
  }
  CUtensorMap map_c = map_a;
  const bool bulk = bulk_stores(p, e, a.x, plan);
  if (bulk) {
    st = make_gemm_map(&map_c, p.c, p.N, p.M, p.c_sm, p.nb0, p.c_b0, p.nb1, p.c_b1, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B);
    if (st != FML_OK) return st;
  }
  using KernelFn = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const PairArgs);
#define FML_PAIR_PLAIN(B)                                                                                                        \
  gemm_pair_kernel<FML_ACT_NONE, kPlain, B>, gemm_pair_kernel<FML_ACT_GELU_ERF, kPlain, B>, gemm_pair_kernel<FML_ACT_RELU, kPlain, B>, \
  gemm_pair_kernel<FML_ACT_TANH, kPlain, B>, gemm_pair_kernel<FML_ACT_SIGMOID, kPlain, B>, gemm_pair_kernel<FML_ACT_SILU, kPlain, B>,  \
  gemm_pair_kernel<FML_ACT_NONE, kProj, B>, gemm_pair_kernel<FML_ACT_GELU_ERF, kProj, B>, gemm_pair_kernel<FML_ACT_NONE, kTwoA, B>
  static const KernelFn kernels[18] = {FML_PAIR_PLAIN(false), FML_PAIR_PLAIN(true)};
#undef FML_PAIR_PLAIN
  FML_REQUIRE(e.act >= 0 && e.act <= FML_ACT_SILU, FML_BAD_ARG, "fml_gemm: unknown activation %d", e.act);
  FML_REQUIRE(mode == kPlain || e.act == FML_ACT_NONE || (mode == kProj && e.act == FML_ACT_GELU_ERF), FML_UNSUPPORTED, "fml_gemm: activation %d in a joined product", e.act);
  const KernelFn kernel = kernels[(bulk ? 9 : 0) + (mode == kPlain ? e.act : mode == kTwoA ? 8 : e.act == FML_ACT_NONE ? 6 : 7)];
  static bool attr_set[64] = {false};
  int dev = 0;
  FML_CUDA(cudaGetDevice(&dev));
  if (!attr_set[dev & 63]) {
    for (KernelFn k : kernels) FML_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemCta));
    attr_set[dev & 63] = true;
  }
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(a.tiles_m * a.tiles_n), (unsigned)plan.split_k, (unsigned)(p.nb0 * p.nb1));
  cfg.blockDim = dim3(kPairThreads);
  cfg.dynamicSmemBytes = plan.smem_bytes;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = (unsigned)plan.split_k;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  FML_CUDA(cudaLaunchKernelEx(&cfg, kernel, map_a, map_a2, map_c, a));
  return x.rot && !rotates ? launch_rotary_in_place(p, x, s) : FML_OK;
}

}  // namespace fml

// Declared in fluidml_cuda.h: while the longer product would be split at all (sum_slices).  With more tiles two launches lose
// nothing and an exact sum does: 4000 x (1024 + 4096) x 1024 116 us, 107 as two.
extern "C" int fml_gemm_joins_sums(int64_t rows, int64_t n) { return rows >= 1 && n >= 1 && fml::sum_slices(rows, n, 1) > 1 ? 1 : 0; }

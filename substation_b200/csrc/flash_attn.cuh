// Attention without the score tensors in memory (included by gemm.cu; shares its TMA / tcgen05 helpers).
//
// Forward:  GAMMA[p,j] = sum_k mask[j,k] * ALPHA[j,k] * V[p,k],  ALPHA = softmax_k(scale * Q^T K)
//           (QKT, Softmax and gamma of pytorch_module/encoder.cu:112-125 in one kernel)
// Backward: dV, dK and dQ from DGAMMA, with ALPHA computed again from Q, K and the rows' log-sum-exp
//           (dX1gamma, dX2gamma, BackwardSoftmax, dX1QKT, dX2QKT of pytorch_module/encoder.cu:250-269)
//
// What bounded the operators these replace was the score tensor itself: at B=8, L=512 ALPHA and ATTN_DROP (67 MB
// each), DBETA (67 MB) and the mask bytes (34 MB) were written once and read one to two times each, and for lengths
// that are not a multiple of 128, or beyond 512, BETA and DATTN_DROP as well, by eight separate launches.  Here a
// pass keeps one float per row (log2 of the sum) and one BIT per score (the dropout mask) instead.  They are used
// where nobody can look at the intermediates of a pass (sb_encoder_forward_private).
//
// Scores are addressed by unit u = (head, sample), query row j and key column k.  Projections are 16-bit tensors with
// head size 64 and unit stride along either the rows ("jc") or the head dim; a tile is 128 rows x 64, 16 KiB in
// shared memory as two 64-row boxes with 128-byte swizzle, and the same bytes serve as an operand whose K index is
// the head dim (scores) and as one whose K index is the row (outputs): only the descriptors differ.

#pragma once

namespace flash {

constexpr int kTile = 16384;                         // 128 rows x 64, 16-bit
constexpr float kLazy = 8.f;                         // log2 units a row maximum may lag behind (see flash_fwd_kernel)

// ---- dropout masks as bits -------------------------------------------------------------------------------------
// 32 consecutive scores of a row are one word in "pair order": bit i is element 2i, bit 16 + i is element 2i + 1, so
// that one shift brings a pair's two flags to bits 15 and 31, where byte-permute can replicate them.
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, 0, %2;" : "=r"(d) : "r"(a), "r"(sel));
  return d;
}
__device__ __forceinline__ uint32_t pair_lanes(uint32_t word, int i) { return prmt(word << (15 - i), 0xBB99u); }
__device__ __forceinline__ uint32_t even_full(uint32_t word, int i) { return prmt(word << (15 - i), 0x9999u); }
__device__ __forceinline__ uint32_t odd_full(uint32_t word, int i) { return prmt(word << (15 - i), 0xBBBBu); }
// plain bit order -> pair order (even bits to the low half)
__device__ __forceinline__ uint32_t to_pairs(uint32_t x) {
  uint32_t t;
  t = (x ^ (x >> 1)) & 0x22222222u; x ^= t ^ (t << 1);
  t = (x ^ (x >> 2)) & 0x0C0C0C0Cu; x ^= t ^ (t << 2);
  t = (x ^ (x >> 4)) & 0x00F000F0u; x ^= t ^ (t << 4);
  t = (x ^ (x >> 8)) & 0x0000FF00u; x ^= t ^ (t << 8);
  return x;
}
// Philox flags of elements 8g .. 8g+31, pair order.  The generator's 16-bit lanes are compared with the threshold two
// at a time: with the top bits forced on (x) and off (thr) the subtraction cannot borrow across lanes, and x >= thr is
// the majority of x's top bit, thr's inverted one and the difference's.
__device__ __forceinline__ uint32_t philox_pairs32(const Rng& r, unsigned long long g) {
  const uint32_t thr2 = r.thr * 0x10001u, tl = thr2 & 0x7fff7fffu, nt = ~thr2;
  uint32_t bits = 0;
#pragma unroll
  for (int gi = 0; gi < 4; ++gi) {
    const unsigned long long gg = g + gi;
    const uint4 w = philox4x32_10(make_uint4((uint32_t)gg, (uint32_t)(gg >> 32), r.off_lo, r.off_hi), r.seed_lo, r.seed_hi);
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t t = (ww[i] | 0x80008000u) - tl;
      const uint32_t keep = (ww[i] & t) | (nt & (ww[i] | t));
      bits |= (keep >> (15 - (gi * 4 + i))) & (0x00010001u << (gi * 4 + i));
    }
  }
  return bits;
}
// The same for 32 elements that start anywhere.
__device__ __noinline__ uint32_t philox_pairs32_any(const Rng& r, unsigned long long e0) {
  unsigned long long v = 0;
  for (int gi = 0; gi < 5; ++gi) {
    uint32_t m[8];
    philox_keep8(r, (e0 >> 3) + gi, m);
    uint32_t b = 0;
#pragma unroll
    for (int t = 0; t < 8; ++t) b |= m[t] << t;
    v |= (unsigned long long)b << (8 * gi);
  }
  return to_pairs((uint32_t)(v >> (e0 & 7ull)));
}
// 32 mask bytes (0 or 1) of one row, n of them inside the row (the others read as 0), pair order.
__device__ __noinline__ uint32_t bytes_pairs32(const uint8_t* p, int n) {
  uint32_t plain = 0;
  if ((reinterpret_cast<uintptr_t>(p) & 15u) == 0 && n >= 32) {
    const uint4 a = reinterpret_cast<const uint4*>(p)[0], b = reinterpret_cast<const uint4*>(p)[1];
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) plain |= ((w[i] * 0x10204080u) >> 28) << (4 * i);
  } else {
    for (int i = 0; i < 32; ++i)
      if (i < n) plain |= (p[i] ? 1u : 0u) << i;
  }
  return to_pairs(plain);
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const sb_half2 h = sb_f2h2(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// NC accumulator columns -> alpha * value, 16-bit, at ptr[p * sP]
template <int NC>
__device__ __forceinline__ void store_cols(sb_half* ptr, long long sP, const uint32_t* r, float alpha) {
  if (sP == 1 && (reinterpret_cast<uintptr_t>(ptr) & 15u) == 0) {
#pragma unroll
    for (int v = 0; v < NC / 8; ++v) {
      uint4 o;
      uint32_t* w = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
      for (int e = 0; e < 4; ++e) w[e] = pack2(__uint_as_float(r[v * 8 + 2 * e]) * alpha, __uint_as_float(r[v * 8 + 2 * e + 1]) * alpha);
      reinterpret_cast<uint4*>(ptr)[v] = o;
    }
  } else {
#pragma unroll
    for (int e = 0; e < NC; ++e) ptr[e * sP] = sb_f2h(__uint_as_float(r[e]) * alpha);
  }
}

// A projection tile: rows r0 .. r0+127 of unit u (rows beyond the sequence arrive as zeros).
__device__ __forceinline__ void load_tile(uint32_t dst, const CUtensorMap* map, uint32_t bar, int jc, int swap, int r0, int u) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = r0 + 64 * h;
    const uint32_t d = dst + h * 8192;
    if (jc) {
      if (swap) tma_load_3d(d, map, bar, r, u, 0);
      else tma_load_3d(d, map, bar, r, 0, u);
    } else {
      if (swap) tma_load_3d(d, map, bar, 0, u, r);
      else tma_load_3d(d, map, bar, 0, r, u);
    }
  }
}
// D[128 x 128] = rows of tile a times rows of tile b over the head dim
__device__ __forceinline__ void mma_scores(uint32_t d, uint32_t a, uint32_t b, int a_jc, int b_jc) {
  const uint32_t idesc = (1u << 4) | SB_IDESC_AB_FMT | ((uint32_t)a_jc << 15) | ((uint32_t)b_jc << 16) | ((128u >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
  const uint32_t a_lbo = a_jc ? 8192u : 16u, a_step = a_jc ? 2048u : 32u, b_lbo = b_jc ? 8192u : 16u, b_step = b_jc ? 2048u : 32u;
  const uint64_t da = make_desc(a, a_lbo, 1024u), db = make_desc(b, b_lbo, 1024u);
#pragma unroll
  for (int k = 0; k < 4; ++k)
    umma_f16(d, da + (uint64_t)(k * a_step >> 4), db + (uint64_t)(k * b_step >> 4), idesc, k > 0 ? 1u : 0u);
}
// D[128 x 64] (+)= S * tile, S a [128 x 128] 16-bit tile in shared memory (two 64-column boxes) and the summed index
// its columns, or its rows when `transposed`; the tile's rows are the summed index.
__device__ __forceinline__ void mma_outputs(uint32_t d, uint32_t s, uint32_t tile, int jc, bool transposed, bool accumulate) {
  const uint32_t idesc = (1u << 4) | SB_IDESC_AB_FMT | (transposed ? 1u << 15 : 0u) | (jc ? 0u : 1u << 16) | ((64u >> 3) << 17) |
                         ((uint32_t)(kBM >> 4) << 24);
  const uint64_t da = transposed ? make_desc(s, 16384u, 1024u) : make_desc(s, 16u, 1024u);
  const uint64_t db = make_desc(tile, jc ? 16u : 8192u, 1024u);
  const uint32_t b_step = jc ? 2u : 128u;             // in 16-byte units, like the increments below
#pragma unroll
  for (int k = 0; k < 8; ++k)
    umma_f16(d, da + (uint64_t)(transposed ? k * 128 : (k >> 2) * 1024 + (k & 3) * 2), db + (uint64_t)((k >> 2) * 512 + (k & 3) * b_step),
             idesc, (accumulate || k > 0) ? 1u : 0u);
}

// One thread of a converged warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(pred));
  return pred != 0;
}

// After a wait ran out: give copies still in flight time to land before the CTA retires.
__device__ __forceinline__ void drain_after_error() {
  if (*reinterpret_cast<volatile int*>(&g_tc_error) != 0) {
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 1000000ull) __nanosleep(1000);
  }
}

// ---- forward ---------------------------------------------------------------------------------------------------
constexpr int kRing = 3;                             // key and value tiles in flight
constexpr int kFwdThreads = 192;                     // producer warp, MMA warp, four softmax warps
constexpr int kFwdSmem = (1 + kRing + 2) * kTile + 1024 + 256;

enum { kNoDrop = 0, kPhilox = 1, kAnyMask = 2 };     // masks: none dropped | drawn, rows 8-aligned | everything else

struct FwdParams {
  int L, nb;               // sequence length, ceil(L / 128)
  int items;               // units * nb
  int sweeps;              // 2: a first sweep over the keys finds maximum and sum, so that ALPHA itself is rounded to 16 bits
  int jc, q_swap, k_swap, v_swap;
  float c2;                // scale * log2(e)
  Rng rng;
  const uint8_t* mask;     // explicit masks, [unit][L][L]
  uint4* bits;             // [unit][nb][L] words of 128 flags, or null
  float* lse;              // [unit][L], or null
  sb_half* out;
  int B;                   // unit u is head u / B of sample u % B
  long long o_sH, o_sB, o_sRow, o_sP;
};

// One CTA: 128 query rows of one unit against all keys in tiles of 128; two CTAs per SM, so that one's tensor and
// copy work runs beside the other's softmax.  Tensor memory: scores [128 x 128] and the output [128 x 64].  Softmax
// warps: thread = row, online softmax with a lazily updated reference: exponentials are taken against a maximum that
// may lag up to 2^8 behind (they stay below 256, exact in every format involved up to the usual relative rounding),
// and only when some row of a warp exceeds it is the output rescaled.  The masks' generator runs while the tile's
// scores are still being multiplied.  With two sweeps the first one only keeps the running maximum and sum.
// Bound by issue slots (40 % of them the mask generator) and the special-function unit.  B=8, L=512 with masks: 43 us where
// the scores kernel and the gamma contraction took 62 + 18; B=64, L=256 without: 48 us for 122 + 42.
template <int MODE>
__global__ void __launch_bounds__(kFwdThreads, 2)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const FwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sq = (raw + 1023u) & ~1023u;
  const uint32_t ring = sq + kTile, sp = ring + kRing * kTile, bars = sp + 2 * kTile;
  const uint32_t q_full = bars, q_empty = bars + 8, s_full = bars + 16, p_full = bars + 24, p_free = bars + 32, o_empty = bars + 40;
  const uint32_t kv_full = bars + 48, kv_empty = kv_full + 8 * kRing;
  uint8_t* gen = smem_raw + (sq - raw);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen + (bars - sq) + 48 + 16 * kRing);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int L = p.L, nb = p.nb;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    mbar_init(s_full, 1);
    mbar_init(p_full, 4);
    mbar_init(p_free, 1);
    mbar_init(o_empty, 4);
    for (int i = 0; i < kRing; ++i) {
      mbar_init(kv_full + 8 * i, 1);
      mbar_init(kv_empty + 8 * i, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmQ) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmK) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmV) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(256u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  const uint32_t tmem_o = tmem + 128u;
  grid_dependency_sync();

  if (warp == 0) {
    // ---------------- TMA producer: Q of the item, then K, V of each key tile ----------------
    uint32_t it = 0, n = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < p.items && ok; item += gridDim.x, ++it) {
      const int u = item / nb, j0 = (item % nb) * 128;
      ok = __all_sync(0xffffffffu, mbar_wait(q_empty, (it & 1u) ^ 1u, 21));
      if (!ok) break;
      if (lane == 0) {
        mbar_expect_tx(q_full, kTile);
        load_tile(sq, &tmQ, q_full, p.jc, p.q_swap, j0, u);
      }
      __syncwarp();
      const int first = (p.sweeps - 1) * nb;               // a first sweep reads the keys alone
      for (int i = 0; i < first + 2 * nb; ++i, ++n) {
        const int x = i < first ? 2 * i : i - first;       // even: keys of tile x / 2, odd: values
        const uint32_t s = n % kRing, ph = (n / kRing) & 1u;
        ok = __all_sync(0xffffffffu, mbar_wait(kv_empty + 8 * s, ph ^ 1u, 21));
        if (!ok) break;
        if (lane == 0) {
          mbar_expect_tx(kv_full + 8 * s, kTile);
          if (x & 1) load_tile(ring + s * kTile, &tmV, kv_full + 8 * s, p.jc, p.v_swap, (x >> 1) * 128, u);
          else load_tile(ring + s * kTile, &tmK, kv_full + 8 * s, p.jc, p.k_swap, (x >> 1) * 128, u);
        }
        __syncwarp();
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer: scores of the next key tile before the output of this one ----------------
    uint32_t it = 0, n = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < p.items && ok; item += gridDim.x, ++it) {
      const int first = (p.sweeps - 1) * nb, tiles = first + nb;
      const uint32_t base = it * (uint32_t)(first + 2 * nb);
      auto scores = [&](int i) {                           // i-th score tile of the item
        const uint32_t x = base + (i < first ? i : first + 2 * (i - first)), s = x % kRing;
        ok = __all_sync(0xffffffffu, mbar_wait(kv_full + 8 * s, (x / kRing) & 1u, 22));
        if (!ok) return;
        tc_fence_after();
        if (elect_one()) {
          mma_scores(tmem, sq, ring + s * kTile, p.jc, p.jc);
          umma_commit(s_full);
          umma_commit(kv_empty + 8 * s);
          if (i == tiles - 1) umma_commit(q_empty);
        }
        __syncwarp();
      };
      ok = __all_sync(0xffffffffu, mbar_wait(q_full, it & 1u, 22));
      if (!ok) break;
      scores(0);
      for (int i = 0; i < tiles && ok; ++i, ++n) {
        ok = __all_sync(0xffffffffu, mbar_wait(p_full, n & 1u, 22));   // the scores have been read, their exponentials written
        if (!ok) break;
        tc_fence_after();
        if (i + 1 < tiles) scores(i + 1);
        if (!ok) break;
        if (i < first) continue;
        const int kb = i - first;
        const uint32_t x = base + first + 2u * kb + 1u, s = x % kRing;
        ok = __all_sync(0xffffffffu, mbar_wait(kv_full + 8 * s, (x / kRing) & 1u, 22));
        if (!ok) break;
        if (kb == 0) {
          ok = __all_sync(0xffffffffu, mbar_wait(o_empty, (it & 1u) ^ 1u, 24));
          if (!ok) break;
        }
        tc_fence_after();
        if (elect_one()) {
          mma_outputs(tmem_o, sp, ring + s * kTile, p.jc, false, kb > 0);
          umma_commit(kv_empty + 8 * s);
          umma_commit(p_free);
        }
        __syncwarp();
      }
    }
  } else {
    // ---------------- softmax warps: thread = one query row ----------------
    const int q = warp & 3;
    const int rt = q * 32 + lane;
    const uint32_t lanes = (uint32_t)(q * 32) << 16;
    uint8_t* prow = gen + (sp - sq) + rt * 128;
    uint32_t n = 0, v = 0;     // score tiles and output products so far
    bool ok = true;
    for (int item = blockIdx.x; item < p.items && ok; item += gridDim.x) {
      const int u = item / nb, j = (item % nb) * 128 + rt;
      const bool row = j < L;
      const long long row0 = ((long long)u * L + j) * (long long)L;   // linear index of the row's first score
      float m = -INFINITY, l = 0.f, ref = 0.f;
      // first sweep: maximum and sum of the row (scores read twice, nothing written)
      for (int kb = 0; kb < (p.sweeps - 1) * nb; ++kb, ++n) {
        const int rem = L - kb * 128;
        ok = __all_sync(0xffffffffu, mbar_wait(s_full, n & 1u, 23));
        if (!ok) break;
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t r[32];
          tmem_ld32_nowait(tmem + lanes + c * 32, r);
          attn::tmem_ld_wait32(r);
          float mx = m;
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            if (c * 32 + e >= rem) r[e] = 0xff800000u;
            mx = fmaxf(mx, __uint_as_float(r[e]));
          }
          const float ms = mx == -INFINITY ? 0.f : mx * p.c2;
          if (mx > m) l *= attn::ex2_approx((m - mx) * p.c2);
          m = mx;
#pragma unroll
          for (int e = 0; e < 32; ++e) l += attn::ex2_approx(fmaf(__uint_as_float(r[e]), p.c2, -ms));
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full);
      }
      if (!ok) break;
      if (p.sweeps == 2) ref = (m == -INFINITY ? 0.f : m * p.c2) + log2f(l);
      for (int kb = 0; kb < nb; ++kb, ++n, ++v) {
        const int rem = L - kb * 128;                                  // columns of this tile inside the row (may exceed 128)
        uint32_t keep[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          keep[c] = 0xffffffffu;
          if (MODE == kPhilox) keep[c] = philox_pairs32(p.rng, (unsigned long long)(row0 + kb * 128 + c * 32) >> 3);
          if (MODE == kAnyMask) {
            if (p.rng.philox) keep[c] = philox_pairs32_any(p.rng, (unsigned long long)(row0 + kb * 128 + c * 32));
            else keep[c] = row && rem > c * 32 ? bytes_pairs32(p.mask + row0 + kb * 128 + c * 32, rem - c * 32) : 0u;
          }
        }
        if (p.bits && row) p.bits[((long long)u * nb + kb) * L + j] = make_uint4(keep[0], keep[1], keep[2], keep[3]);
        ok = __all_sync(0xffffffffu, mbar_wait(s_full, n & 1u, 23));
        if (!ok) break;
        tc_fence_after();
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t r[64];
          tmem_ld32_nowait(tmem + lanes + h * 64, r);
          tmem_ld32_nowait(tmem + lanes + h * 64 + 32, r + 32);
          attn::tmem_ld_wait32(r);
          attn::tmem_ld_wait32(r + 32);
          if (rem < 128) {
#pragma unroll
            for (int e = 0; e < 64; ++e)
              if (h * 64 + e >= rem) r[e] = 0xff800000u;
          }
#pragma unroll
          for (int e = 0; e < 64; e += 4)
#pragma unroll
            for (int x = 0; x < 4; ++x) mx4[x] = fmaxf(mx4[x], __uint_as_float(r[e + x]));
        }
        const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
        if (v > 0) {                                   // the previous output multiplication has read its exponentials
          ok = __all_sync(0xffffffffu, mbar_wait(p_free, (v - 1u) & 1u, 25));
          if (!ok) break;
          tc_fence_after();
        }
        if (p.sweeps == 2) {
        } else if (kb == 0) {
          m = mx;
        } else {
          const bool raise = (mx - m) * p.c2 > kLazy;  // -inf so far: true as soon as a finite score comes
          if (__any_sync(0xffffffffu, raise)) {
            const float f = raise ? attn::ex2_approx((m - mx) * p.c2) : 1.f;
            if (raise) m = mx;
            l *= f;
            uint32_t r[64];
            tmem_ld32_nowait(tmem_o + lanes, r);
            tmem_ld32_nowait(tmem_o + lanes + 32, r + 32);
            attn::tmem_ld_wait32(r);
            attn::tmem_ld_wait32(r + 32);
#pragma unroll
            for (int e = 0; e < 64; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * f);
            attn::tmem_st32(tmem_o + lanes, r);
            attn::tmem_st32(tmem_o + lanes + 32, r + 32);
            attn::tmem_st_wait();
          }
        }
        const float ms = p.sweeps == 2 ? ref : m == -INFINITY ? 0.f : m * p.c2;
        uint32_t ra[32], rb[32];
        tmem_ld32_nowait(tmem + lanes, ra);
        float l0 = 0.f, l1 = 0.f;
        auto chunk = [&](int c, uint32_t* r) {
          if (rem < 128) {
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (c * 32 + e >= rem) r[e] = 0xff800000u;
          }
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            uint4 o;
            uint32_t* w = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float a = attn::ex2_approx(fmaf(__uint_as_float(r[v * 8 + 2 * e]), p.c2, -ms));
              const float b = attn::ex2_approx(fmaf(__uint_as_float(r[v * 8 + 2 * e + 1]), p.c2, -ms));
              l0 += a;
              l1 += b;
              w[e] = pack2(a, b);
              if (MODE != kNoDrop) w[e] &= pair_lanes(keep[c], v * 4 + e);
            }
            const int piece = (c & 1) * 4 + v;          // 16-byte piece of this row in its 64-column box
            *reinterpret_cast<uint4*>(prow + (c >> 1) * 16384 + ((piece ^ (lane & 7)) << 4)) = o;
          }
        };
        attn::tmem_ld_wait32(ra);
        tmem_ld32_nowait(tmem + lanes + 32, rb);
        chunk(0, ra);
        attn::tmem_ld_wait32(rb);
        tmem_ld32_nowait(tmem + lanes + 64, ra);
        chunk(1, rb);
        attn::tmem_ld_wait32(ra);
        tmem_ld32_nowait(tmem + lanes + 96, rb);
        chunk(2, ra);
        attn::tmem_ld_wait32(rb);
        chunk(3, rb);
        if (p.sweeps == 1) l += l0 + l1;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full);
      }
      if (!ok) break;
      ok = __all_sync(0xffffffffu, mbar_wait(p_free, (v - 1u) & 1u, 25));
      if (!ok) break;
      tc_fence_after();
      uint32_t r[64];
      tmem_ld32_nowait(tmem_o + lanes, r);
      tmem_ld32_nowait(tmem_o + lanes + 32, r + 32);
      attn::tmem_ld_wait32(r);
      attn::tmem_ld_wait32(r + 32);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(o_empty);
      if (row) {
        store_cols<64>(p.out + (u / p.B) * p.o_sH + (u % p.B) * p.o_sB + (long long)j * p.o_sRow, p.o_sP, r, p.sweeps == 2 ? 1.f : 1.f / l);
        if (p.lse) p.lse[(long long)u * L + j] = p.sweeps == 2 ? ref : (m == -INFINITY ? 0.f : m * p.c2) + log2f(l);
      }
    }
  }
  drain_after_error();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u) : "memory");
  }
}

// ---- backward --------------------------------------------------------------------------------------------------
constexpr int kSlots = 4;                            // tile pairs (Q and DGAMMA, or K and V) in shared memory
constexpr int kBwdThreads = 320;                     // producer warp, MMA warp, eight element warps
constexpr int kBwdSmem = kSlots * 2 * kTile + 4 * kTile + 1024 + 256;

struct BwdParams {
  int L, nb, units;
  int items, first_q;      // items below first_q compute dK and dV of a key tile, the others dQ of a query tile
  int both;                // one tile per unit (L <= 128): an item computes all three
  int jc, g_jc;            // Q, K, V | DGAMMA
  int q_swap, k_swap, v_swap, g_swap;
  float scale, c2;
  const uint4* bits;
  const float* lse;
  const float* dsum;       // [unit][L]: sum_p DGAMMA * GAMMA = sum_k ALPHA * dALPHA
  sb_half* dq; sb_half* dk; sb_half* dv;
  int B;
  long long d_sH, d_sB, d_sRow, d_sP;
};

// Which of the four tile-pair slots are used for what: one is held for a whole item, the other three take the tiles
// that stream past it in turn, and the next item's held pair is the next of the three.  Producer and MMA warp walk
// the same sequence.
struct SlotQueue {
  int held = -1, q0 = 0, q1 = 1, q2 = 2, spare = 3;
  __device__ __forceinline__ int hold() {
    const int s = q0;
    q0 = q1; q1 = q2; q2 = held < 0 ? spare : held;
    held = s;
    return s;
  }
  __device__ __forceinline__ int stream() {
    const int s = q0;
    q0 = q1; q1 = q2; q2 = s;
    return s;
  }
};

// One CTA per SM.  Work items hold one pair of tiles and stream the other pair past it: (K, V) held for dK and dV, (Q,
// DGAMMA) held for dQ.  Computing the scores twice costs less than what the alternatives do: dQ partial sums over key
// tiles in memory (4 bytes x 64 x L per key tile) or DBETA itself.  Per tile: scores and dALPHA into tensor memory (128
// columns each), eight element warps (thread = query row, 64 columns) turn them into mask * ALPHA and DBETA in
// registers, write both to shared memory as 16-bit [j x k] tiles, and these are operands as they lie: K-major
// for dQ, MN-major for dK and dV.  The next tile's scores are multiplied while this one's are turned, so in dQ items, whose
// 16-bit tiles alternate, the element warps can be done with tile n + 1 before the MMA warp has looked whether tile n was:
// two barriers (pd_full) say that a tile is written, n & 1, and neither can run a phase ahead of its waiter, because tile
// n + 2 needs scores which the MMA warp multiplies only after it has seen tile n.  Accumulators
// alternate between two sets so that an item's results are stored while the next item computes.  Bound by the element
// warps: special-function unit (16 exponentials per clock and SM) and the latencies of a tile's hand-overs, 3 700 clocks per
// tile.  B=8, L=512: 58 us and 5 for the row sums, where scores backward, dX2gamma and dX1QKT+dX2QKT took 41 + 21 + 23;
// B=96, L=128: 48 + 8 for 37 + 21 + 26; B=2, L=1024: 63 + 4 for eight launches of 160.
__global__ void __launch_bounds__(kBwdThreads, 1)
flash_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmG, const BwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t slots = (raw + 1023u) & ~1023u;
  const uint32_t sds = slots + kSlots * 2 * kTile, spm = sds + 2 * kTile, bars = spm + 2 * kTile;
  const uint32_t full = bars, empty = full + 8 * kSlots, sd_full = empty + 8 * kSlots, sd_empty = sd_full + 8;
  const uint32_t pd_full = sd_empty + 8, ds_empty = pd_full + 16, acc_full = ds_empty + 16, acc_empty = acc_full + 16;
  uint8_t* gen = smem_raw + (slots - raw);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen + (acc_empty + 16 - slots));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int L = p.L, nb = p.nb;
  const uint32_t sets = p.both ? 1u : 2u;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(full + 8 * i, 1);
      mbar_init(empty + 8 * i, 1);
    }
    mbar_init(sd_full, 1);
    mbar_init(sd_empty, 8);
    for (int i = 0; i < 2; ++i) {
      mbar_init(pd_full + 8 * i, 8);
      mbar_init(ds_empty + 8 * i, 1);
      mbar_init(acc_full + 8 * i, 1);
      mbar_init(acc_empty + 8 * i, 8);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmQ) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmK) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmV) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmG) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  const uint32_t tmem_acc = tmem + 256u;
  grid_dependency_sync();

  auto is_q = [&](int item) { return item >= p.first_q; };
  auto unit_of = [&](int item) { return (is_q(item) ? item - p.first_q : item) / nb; };
  auto block_of = [&](int item) { return (is_q(item) ? item - p.first_q : item) % nb; };

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    SlotQueue sq;
    uint32_t phase = 0;
    bool ok = true;
    auto load_pair = [&](int s, bool queries, int u, int r0) {
      ok = __all_sync(0xffffffffu, mbar_wait(empty + 8 * s, ((phase >> s) & 1u) ^ 1u, 31));
      if (!ok) return;
      phase ^= 1u << s;
      if (lane == 0) {
        const uint32_t bar = full + 8 * s, d = slots + s * 2 * kTile;
        mbar_expect_tx(bar, 2 * kTile);
        if (queries) {
          load_tile(d, &tmQ, bar, p.jc, p.q_swap, r0, u);
          load_tile(d + kTile, &tmG, bar, p.g_jc, p.g_swap, r0, u);
        } else {
          load_tile(d, &tmK, bar, p.jc, p.k_swap, r0, u);
          load_tile(d + kTile, &tmV, bar, p.jc, p.v_swap, r0, u);
        }
      }
      __syncwarp();
    };
    for (int item = blockIdx.x; item < p.items && ok; item += gridDim.x) {
      const int u = unit_of(item), b = block_of(item);
      const bool qi = is_q(item);
      load_pair(sq.hold(), qi, u, b * 128);
      for (int t = 0; t < nb && ok; ++t) load_pair(sq.stream(), !qi, u, t * 128);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    SlotQueue sq;
    uint32_t phase = 0, n = 0, it = 0;
    bool ok = true;
    struct Pending { int item, held, slot; uint32_t it, n; bool first, last; };
    Pending pend{-1, 0, 0, 0u, 0u, false, false};
    auto wait_slot = [&](int s) {
      ok = __all_sync(0xffffffffu, mbar_wait(full + 8 * s, (phase >> s) & 1u, 32)) && ok;
      phase ^= 1u << s;
    };
    auto outputs = [&](const Pending& d) {
      const bool qi = is_q(d.item);
      const uint32_t set = d.it % sets;
      ok = ok && __all_sync(0xffffffffu, mbar_wait(pd_full + 8 * (d.n & 1u), (d.n >> 1) & 1u, 33));
      if (ok && d.first) ok = __all_sync(0xffffffffu, mbar_wait(acc_empty + 8 * set, ((d.it / sets) & 1u) ^ 1u, 34));
      if (!ok) return;
      tc_fence_after();
      if (elect_one()) {
        const uint32_t held = slots + d.held * 2 * kTile, str = slots + d.slot * 2 * kTile;
        const uint32_t qt = qi ? held : str, kt = qi ? str : held;   // (Q, DGAMMA) and (K, V)
        const uint32_t acc = tmem_acc + set * 128u;
        if (!qi) {
          mma_outputs(acc, spm, qt + kTile, p.g_jc, true, !d.first);          // dV += (mask * ALPHA)^T DGAMMA
          umma_commit(ds_empty + 8);
          mma_outputs(acc + 64u, sds, qt, p.jc, true, !d.first);              // dK += DBETA^T Q
          if (p.both) mma_outputs(acc + 128u, sds, kt, p.jc, false, false);   // dQ  = DBETA K
        } else {
          mma_outputs(acc, d.n & 1u ? spm : sds, kt, p.jc, false, !d.first);  // dQ += DBETA K
        }
        umma_commit(qi && (d.n & 1u) ? ds_empty + 8 : ds_empty);
        umma_commit(empty + 8 * d.slot);
        if (d.last) {
          umma_commit(empty + 8 * d.held);
          umma_commit(acc_full + 8 * set);
        }
      }
      __syncwarp();
    };
    for (int item = blockIdx.x; item < p.items && ok; item += gridDim.x, ++it) {
      const bool qi = is_q(item);
      const int held = sq.hold();
      wait_slot(held);
      for (int t = 0; t < nb && ok; ++t, ++n) {
        const int s = sq.stream();
        wait_slot(s);
        ok = ok && __all_sync(0xffffffffu, mbar_wait(sd_empty, (n & 1u) ^ 1u, 35));
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
          const uint32_t hs = slots + held * 2 * kTile, ss = slots + s * 2 * kTile;
          const uint32_t qt = qi ? hs : ss, kt = qi ? ss : hs;
          mma_scores(tmem, qt, kt, p.jc, p.jc);
          mma_scores(tmem + 128u, qt + kTile, kt + kTile, p.g_jc, p.jc);
          umma_commit(sd_full);
        }
        __syncwarp();
        if (pend.item >= 0) outputs(pend);
        pend = Pending{item, held, s, it, n, t == 0, t == nb - 1};
      }
    }
    if (ok && pend.item >= 0) outputs(pend);
  } else {
    // ---------------- element warps: thread = one query row, 64 columns ----------------
    const int q = warp & 3, h = (warp - 2) >> 2;
    const int rt = q * 32 + lane;
    const uint32_t lanes = (uint32_t)(q * 32) << 16;
    uint8_t* drow = gen + (sds - slots) + h * 16384 + rt * 128;
    uint8_t* prow = gen + (spm - slots) + h * 16384 + rt * 128;
    uint32_t n = 0, it = 0;
    bool ok = true;
    // results of an item, stored once its last product is done (after the next item's first tile has been turned)
    auto finish = [&](int item, uint32_t i) {
      const uint32_t set = i % sets;
      ok = ok && __all_sync(0xffffffffu, mbar_wait(acc_full + 8 * set, (i / sets) & 1u, 36));
      if (!ok) return;
      tc_fence_after();
      const uint32_t acc = tmem_acc + set * 128u + lanes;
      const bool qi = is_q(item);
      const int u = unit_of(item), r0 = block_of(item) * 128 + rt;
      const long long off = (u / p.B) * p.d_sH + (u % p.B) * p.d_sB + (long long)r0 * p.d_sRow;
      // 32 columns at a time: two pieces of dV (h = 0) or dK (h = 1), one of dQ
#pragma unroll 1
      for (int c = qi ? 2 : 0; c < (qi || p.both ? 3 : 2); ++c) {
        uint32_t r[32];
        tmem_ld32_nowait(acc + (c < 2 ? h * 64 + c * 32 : (p.both ? 128 : 0) + h * 32), r);
        attn::tmem_ld_wait32(r);
        sb_half* out = c < 2 ? (h ? p.dk : p.dv) + c * 32 * p.d_sP : p.dq + h * 32 * p.d_sP;
        if (r0 < L) store_cols<32>(out + off, p.d_sP, r, c < 2 && !h ? 1.f : p.scale);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty + 8 * set);
    };
    // row inputs of a tile, asked for one tile ahead
    float lse = INFINITY, ds = 0.f;
    uint2 keep = make_uint2(0u, 0u);
    auto fetch = [&](bool qi, int u, int b, int t) {
      const int j = (qi ? b : t) * 128 + rt, kb = qi ? t : b;
      lse = INFINITY; ds = 0.f;
      keep = make_uint2(0u, 0u);
      if (j < L) {
        lse = p.lse[(long long)u * L + j];
        ds = p.dsum[(long long)u * L + j];
        keep = reinterpret_cast<const uint2*>(p.bits + ((long long)u * nb + kb) * L + j)[h];
      }
    };
    // the two 16-bit tiles of shared memory: dK/dV items fill DBETA (0) and mask * ALPHA (1), dQ items alternate between
    // them; `fills` counts the uses of each, and a tile is free once the products that read its last use are done
    uint32_t fills0 = 0, fills1 = 0;
    auto wait_tile = [&](int i) {
      uint32_t& f = i ? fills1 : fills0;
      if (f > 0) ok = __all_sync(0xffffffffu, mbar_wait(ds_empty + 8 * i, (f - 1u) & 1u, 38));
      ++f;
      return ok;
    };
    bool qi = false, next_qi = false;
    int u = 0, b = 0, next_u = 0, next_b = 0;
    if ((int)blockIdx.x < p.items) {
      next_qi = is_q(blockIdx.x); next_u = unit_of(blockIdx.x); next_b = block_of(blockIdx.x);
      fetch(next_qi, next_u, next_b, 0);
    }
    int prev = -1;
    for (int item = blockIdx.x; item < p.items && ok; item += gridDim.x, ++it) {
      qi = next_qi; u = next_u; b = next_b;
      const int next = item + (int)gridDim.x;
      const bool more = next < p.items;
      if (more) { next_qi = is_q(next); next_u = unit_of(next); next_b = block_of(next); }
      for (int t = 0; t < nb && ok; ++t, ++n) {
        const int rem = L - (qi ? t : b) * 128 - h * 64;
        ok = __all_sync(0xffffffffu, mbar_wait(sd_full, n & 1u, 37));
        if (!ok) break;
        tc_fence_after();
        // 32 columns at a time; pm[i], db[i] are the packed pairs i of mask * ALPHA and of DBETA
        uint32_t pm[32], db[32];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t rs[32], rg[32];
          tmem_ld32_nowait(tmem + lanes + h * 64 + c * 32, rs);
          tmem_ld32_nowait(tmem + 128u + lanes + h * 64 + c * 32, rg);
          attn::tmem_ld_wait32(rs);
          attn::tmem_ld_wait32(rg);
          if (c == 1) {                                 // the next tile's scores may be multiplied
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(sd_empty);
          }
          if (rem < 64) {
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (c * 32 + e >= rem) rs[e] = 0xff800000u;
          }
          const uint32_t w = c ? keep.y : keep.x;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float a0 = attn::ex2_approx(fmaf(__uint_as_float(rs[2 * i]), p.c2, -lse));
            const float a1 = attn::ex2_approx(fmaf(__uint_as_float(rs[2 * i + 1]), p.c2, -lse));
            const float m0 = __uint_as_float(__float_as_uint(a0) & even_full(w, i));
            const float m1 = __uint_as_float(__float_as_uint(a1) & odd_full(w, i));
            pm[c * 16 + i] = pack2(m0, m1);
            db[c * 16 + i] = pack2(fmaf(m0, __uint_as_float(rg[2 * i]), -ds * a0), fmaf(m1, __uint_as_float(rg[2 * i + 1]), -ds * a1));
          }
        }
        if (t + 1 < nb) fetch(qi, u, b, t + 1);
        else if (more) fetch(next_qi, next_u, next_b, 0);
        if (!qi) {
          if (!wait_tile(1)) break;
#pragma unroll
          for (int v = 0; v < 8; ++v)
            *reinterpret_cast<uint4*>(prow + ((v ^ (lane & 7)) << 4)) = make_uint4(pm[4 * v], pm[4 * v + 1], pm[4 * v + 2], pm[4 * v + 3]);
        }
        const bool alt = qi && (n & 1u);
        if (!wait_tile(alt ? 1 : 0)) break;
        uint8_t* dst = alt ? prow : drow;
#pragma unroll
        for (int v = 0; v < 8; ++v)
          *reinterpret_cast<uint4*>(dst + ((v ^ (lane & 7)) << 4)) = make_uint4(db[4 * v], db[4 * v + 1], db[4 * v + 2], db[4 * v + 3]);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(pd_full + 8 * (n & 1u));
        if (t == 0 && prev >= 0) finish(prev, it - 1u);
      }
      prev = item;
    }
    if (ok && prev >= 0) finish(prev, it - 1u);
  }
  drain_after_error();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// ---- small kernels around them ---------------------------------------------------------------------------------
// Row-contiguous projections whose rows do not start on 16-byte boundaries (L not a multiple of 8), or whose head and
// sample dims do not collapse, are copied to [p][unit][Lp] with Lp = L rounded up to 8, which tensor maps can address.
__global__ void __launch_bounds__(256)
pad_projections_kernel(const sb_half* src, long long slice, long long sP, long long sH, long long sB, int B, sb_half* dst, int units,
                       int L, int Lp) {
  grid_dependency_sync();
  const long long rows = 192ll * units;
  for (long long r = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += (long long)gridDim.x * 8) {
    const int pp = (int)(r / units), u = (int)(r % units);
    const sb_half* s = src + (pp >> 6) * slice + (pp & 63) * sP + (u / B) * sH + (u % B) * sB;
    sb_half* d = dst + r * Lp;
    for (int j = threadIdx.x & 31; j < L; j += 32) d[j] = s[j];
  }
}

// dsum[unit][j] = sum_p DGAMMA * GAMMA, 32 rows per block, eight head-dim indices per thread; with `pad`, DGAMMA is
// copied as above on the way.
struct DsumParams {
  const sb_half* g; long long g_sP, g_sH, g_sB, g_sRow;
  const sb_half* o; long long o_sP, o_sH, o_sB, o_sRow;
  float* dsum;
  sb_half* pad;
  int units, B, L, Lp, blocks_j;
};
__global__ void __launch_bounds__(256)
dsum_kernel(const DsumParams p) {
  __shared__ float part[8][33];
  grid_dependency_sync();
  const int u = (int)(blockIdx.x / p.blocks_j), j = (int)(blockIdx.x % p.blocks_j) * 32 + (threadIdx.x & 31);
  const int pg = threadIdx.x >> 5;
  const long long g0 = (u / p.B) * p.g_sH + (u % p.B) * p.g_sB + j * p.g_sRow, o0 = (u / p.B) * p.o_sH + (u % p.B) * p.o_sB + j * p.o_sRow;
  float acc = 0.f;
  if (j < p.L) {
    sb_half g[8], o[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      g[e] = p.g[(pg * 8 + e) * p.g_sP + g0];
      o[e] = p.o[(pg * 8 + e) * p.o_sP + o0];
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      acc = fmaf(sb_h2f(g[e]), sb_h2f(o[e]), acc);
      if (p.pad) p.pad[((long long)(pg * 8 + e) * p.units + u) * p.Lp + j] = g[e];
    }
  }
  part[pg][threadIdx.x & 31] = acc;
  __syncthreads();
  if (pg == 0 && j < p.L) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += part[i][threadIdx.x & 31];
    p.dsum[(long long)u * p.L + j] = s;
  }
}

// The same where rows are consecutive and 16-byte aligned in both (L a multiple of 8): eight rows per access, 128 rows per
// block, four head-dim indices per thread.  Two bytes at a time took 13.9 us for the 50 MB of B=96, L=128.
__global__ void __launch_bounds__(256)
dsum_vec_kernel(const DsumParams p) {
  __shared__ float part[16][128 + 4];
  grid_dependency_sync();
  const int u = (int)(blockIdx.x / p.blocks_j), oct = threadIdx.x & 15, j = (int)(blockIdx.x % p.blocks_j) * 128 + oct * 8;
  const int pg = threadIdx.x >> 4;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (j < p.L) {
    const long long g0 = (u / p.B) * p.g_sH + (u % p.B) * p.g_sB + j, o0 = (u / p.B) * p.o_sH + (u % p.B) * p.o_sB + j;
    uint4 g[4], o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      g[e] = *reinterpret_cast<const uint4*>(p.g + (pg * 4 + e) * p.g_sP + g0);
      o[e] = *reinterpret_cast<const uint4*>(p.o + (pg * 4 + e) * p.o_sP + o0);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float a[8], b[8];
      unpack8(g[e], a);
      unpack8(o[e], b);
#pragma unroll
      for (int x = 0; x < 8; ++x) acc[x] = fmaf(a[x], b[x], acc[x]);
    }
  }
#pragma unroll
  for (int x = 0; x < 8; x += 4) *reinterpret_cast<float4*>(&part[pg][oct * 8 + x]) = make_float4(acc[x], acc[x + 1], acc[x + 2], acc[x + 3]);
  __syncthreads();
  const int r = (int)(blockIdx.x % p.blocks_j) * 128 + threadIdx.x;
  if (threadIdx.x < 128 && r < p.L) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) s += part[i][threadIdx.x];
    p.dsum[(long long)u * p.L + r] = s;
  }
}

}  // namespace flash

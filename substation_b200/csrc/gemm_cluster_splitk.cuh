// Contractions with few rows or columns (a handful of short sequences): split-K inside a cluster of single CTAs
// (included by gemm.cu after gemm_pair_splitk.cuh, whose cluster helpers it shares).
//
// What bounds them is how fast the SMs that take part can pull in the weights: at 128 tokens and 1024 features the plain
// kernel runs 8 to 32 tiles of 128 x 128, so a fifth of the machine fetches everything (64 bytes per clock and SM) and the
// reduction over K is a second launch.  Here a tile is 128 x 64, SK CTAs (2 or 4) take a part of its K each, leave
// their fp32 partial in their own shared memory and add up a share of the rows each through distributed shared memory, in
// the fixed order 0..SK-1; the elementwise operator that would read C next is applied on the way out.  Two CTAs fit on an SM.
// Requirements: C with unit stride along N, its row pitch a multiple of 8, 16-byte aligned base, one batch.

#pragma once

namespace csk {

constexpr int kBN = 64;
constexpr int kStages = 4;
constexpr int kStageBytes = kABytes + kBN * kBK * 2;     // 24 KiB
constexpr int kPitch = kBN * 4 + 16;                     // fp32 partial row: spare bytes spread rows over the banks
constexpr int kSmemBytes = kStages * kStageBytes + 1024 + 256;
constexpr int kThreads = 192;                            // producer warp, MMA warp, four epilogue warps
static_assert(128 * kPitch <= kStages * kStageBytes, "the fp32 partial must fit into the operand ring");

__device__ __forceinline__ void store_piece(sb_half* dst, const uint4& v, int w) {
  if (w == 8) {
    *reinterpret_cast<uint4*>(dst) = v;
  } else {
    const sb_half* h = reinterpret_cast<const sb_half*>(&v);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < w) dst[k] = h[k];
  }
}

// Outputs of the fused epilogue (EpiParams::kind 0 to 3, arithmetic as in the paired kernel).
struct Outs { sb_half* c; sb_half* out2; sb_half* out3; };

template <int SK>
__global__ void __cluster_dims__(SK, 1, 1) __launch_bounds__(kThreads, 2)
gemm_cluster_splitk_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                           const TcParams p, const Outs o) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t tiles = (raw + 1023u) & ~1023u;
  const uint32_t bars = tiles + kStages * kStageBytes;
  const uint32_t bar_full = bars, bar_empty = bars + 8 * kStages, bar_accf = bars + 16 * kStages;
  uint8_t* gen = smem_raw + (tiles - raw);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen + (bars - tiles) + 16 * kStages + 8);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = pair::cluster_rank();
  const int t = (int)(blockIdx.x / SK);
  const int KT = (int)((p.K + kBK - 1) / kBK);
  const int kb_begin = min(KT, (int)rank * p.kt_per_split), kb_end = min(KT, kb_begin + p.kt_per_split);
  const int n0 = (t % p.tiles_n) * kBN, m0 = (t / p.tiles_n) * kBM;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    mbar_init(bar_accf, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmA) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmB) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)kBN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  grid_dependency_sync();

  if (warp == 0) {
    uint32_t it = 0;
    for (int kb = kb_begin; kb < kb_end; ++kb, ++it) {
      const uint32_t s = it % kStages, ph = (it / kStages) & 1u;
      if (!__all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * s, ph ^ 1u, 41))) break;
      if (lane == 0) {
        const uint32_t full = bar_full + 8 * s, sa = tiles + s * kStageBytes, sb_ = sa + kABytes;
        mbar_expect_tx(full, (uint32_t)kStageBytes);
        const int k0 = kb * kBK;
        if (!p.a_mn) {
          if (p.a_swap) tma_load_3d(sa, &tmA, full, k0, 0, m0);
          else tma_load_3d(sa, &tmA, full, k0, m0, 0);
        } else {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (p.a_swap) tma_load_3d(sa + h * 8192, &tmA, full, m0 + 64 * h, 0, k0);
            else tma_load_3d(sa + h * 8192, &tmA, full, m0 + 64 * h, k0, 0);
          }
        }
        const int c0 = p.b_mn ? n0 : k0, c1 = p.b_mn ? k0 : n0;
        if (p.b_swap) tma_load_3d(sb_, &tmB, full, c0, 0, c1);
        else tma_load_3d(sb_, &tmB, full, c0, c1, 0);
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    const uint32_t idesc = (1u << 4) | SB_IDESC_AB_FMT | ((uint32_t)(p.a_mn ? 1 : 0) << 15) | ((uint32_t)(p.b_mn ? 1 : 0) << 16) |
                           ((uint32_t)(kBN >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
    const uint64_t da0 = make_desc(tiles, p.a_mn ? 8192u : 16u, 1024u), db0 = make_desc(tiles + kABytes, p.b_mn ? 8192u : 16u, 1024u);
    const uint64_t a_inc = p.a_mn ? 128u : 2u, b_inc = p.b_mn ? 128u : 2u;
    uint32_t it = 0;
    bool ok = true;
    for (int kb = kb_begin; kb < kb_end; ++kb, ++it) {
      const uint32_t s = it % kStages, ph = (it / kStages) & 1u;
      ok = __all_sync(0xffffffffu, mbar_wait(bar_full + 8 * s, ph, 42));
      if (!ok) break;
      tc_fence_after();
      if (lane == 0) {
        const uint64_t off = (uint64_t)(s * (uint32_t)(kStageBytes >> 4));
#pragma unroll
        for (int k = 0; k < kBK / 16; ++k)
          umma_f16(tmem, da0 + off + k * a_inc, db0 + off + k * b_inc, idesc, (it > 0 || k > 0) ? 1u : 0u);
        umma_commit(bar_empty + 8 * s);
      }
      __syncwarp();
    }
    if (ok && lane == 0) umma_commit(bar_accf);
    __syncwarp();
  } else {
    // this CTA's 128 x 64 partial: tensor memory -> shared memory (the ring is free once the last product is done)
    const int q = warp & 3;
    const bool ok = __all_sync(0xffffffffu, mbar_wait(bar_accf, 0u, 43));
    tc_fence_after();
    uint8_t* prow = gen + (q * 32 + lane) * kPitch;
    uint32_t r[64];
    if (ok && kb_end > kb_begin) {
      const uint32_t tsrc = tmem + ((uint32_t)(q * 32) << 16);
      tmem_ld32_nowait(tsrc, r);
      tmem_ld32_nowait(tsrc + 32, r + 32);
      tmem_ld_wait();
    } else {
#pragma unroll
      for (int e = 0; e < 64; ++e) r[e] = 0u;
    }
#pragma unroll
    for (int v = 0; v < 16; ++v)
      *reinterpret_cast<uint4*>(prow + v * 16) = make_uint4(r[4 * v], r[4 * v + 1], r[4 * v + 2], r[4 * v + 3]);
  }
  tc_fence_before();
  pair::cluster_sync_all();   // every partial is in shared memory (release / acquire at cluster scope)
  if (warp >= 2 && *reinterpret_cast<volatile int*>(&g_tc_error) == 0) {
    // rows rank * 128 / SK .. of the tile, eight columns per thread and step
    const int tid = threadIdx.x - 64;
    uint32_t src[SK];
#pragma unroll
    for (int j = 0; j < SK; ++j) src[j] = pair::map_to_rank(tiles, (uint32_t)j);
    const EpiParams& e = p.epi;
#pragma unroll 1
    for (int i = tid; i < 128 / SK * (kBN / 8); i += 128) {
      const int row = (int)rank * (128 / SK) + i / (kBN / 8), col = (i % (kBN / 8)) * 8;
      const long long m = (long long)m0 + row, n = (long long)n0 + col;
      if (m >= p.M || n >= p.N) continue;
      float4 lo[SK], hi[SK];
      const uint32_t at = (uint32_t)(row * kPitch + col * 4);
#pragma unroll
      for (int j = 0; j < SK; ++j) {
        lo[j] = pair::ld_cluster_f4(src[j] + at);
        hi[j] = pair::ld_cluster_f4(src[j] + at + 16);
      }
      const long long off = m * p.sCm + n;
      uint4 side = make_uint4(0, 0, 0, 0);
      if (e.kind == 2) side = *reinterpret_cast<const uint4*>(e.resid + off);
      if (e.kind == 1 || e.kind == 3) {
        if (e.vec_along_m) {
          const sb_half2 b2 = sb_h2h2(e.vec[m]);
          const uint32_t w = *reinterpret_cast<const uint32_t*>(&b2);
          side = make_uint4(w, w, w, w);
        } else {
          side = *reinterpret_cast<const uint4*>(e.vec + n);
        }
      }
#pragma unroll
      for (int j = 1; j < SK; ++j) {
        lo[0].x += lo[j].x; lo[0].y += lo[j].y; lo[0].z += lo[j].z; lo[0].w += lo[j].w;
        hi[0].x += hi[j].x; hi[0].y += hi[j].y; hi[0].z += hi[j].z; hi[0].w += hi[j].w;
      }
      const float f[8] = {lo[0].x * p.alpha, lo[0].y * p.alpha, lo[0].z * p.alpha, lo[0].w * p.alpha,
                          hi[0].x * p.alpha, hi[0].y * p.alpha, hi[0].z * p.alpha, hi[0].w * p.alpha};
      uint4 v = pack8(f);
      const int w = (int)min(8ll, p.N - n);      // columns inside C (kinds 0 and 1 only may have fewer than eight)
      if (e.kind == 0 || !e.skip_c) store_piece(o.c + off, v, w);
      if (e.kind == 0) continue;
      v = hadd8(v, side);
      if (e.kind != 3) {
        store_piece(o.out2 + off, v, w);
        continue;
      }
      if (!e.skip_out2) *reinterpret_cast<uint4*>(o.out2 + off) = v;
      uint2 mk;
      if (e.rng.philox) {
        mk = philox_mask8(e.rng, (unsigned long long)off >> 3);
        if (e.mask) *reinterpret_cast<uint2*>(e.mask + off) = mk;
      } else {
        mk = *reinterpret_cast<const uint2*>(e.mask + off);
      }
      float x[8];
      unpack8(v, x);
#pragma unroll
      for (int k = 0; k < 8; ++k) x[k] = act_fwd(x[k], e.activation);
      *reinterpret_cast<uint4*>(o.out3 + off) = mask_apply(pack8(x), mk);
    }
    __syncwarp();
  }
  if (*reinterpret_cast<volatile int*>(&g_tc_error) != 0) {
    // a wait ran out somewhere: give copies still in flight time to land before the CTA retires
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 1000000ull) __nanosleep(1000);
  }
  tc_fence_before();
  pair::cluster_sync_all();   // no CTA leaves while a peer may still read its shared memory
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)kBN) : "memory");
  }
}

}  // namespace csk

// Tensor contractions of the encoder layer.
//
// plan_einsum() collapses an einsum over strided operands into one batched GEMM
//   C[b,m,n] = alpha * sum_k A[b,m,k] * B[b,n,k]
// with independent strides for every index of every operand.
//
// gemm_tc_kernel: the sm_100a path.  Persistent CTAs (one per SM) walk 128 x BN output tiles;
// two TMEM accumulators let the epilogue of one tile overlap the MMAs of the next:
//   warp 0   : TMA producer, cp.async.bulk.tensor into a ring of 128-byte-swizzled
//              shared-memory stages (every CTA fetches its own tiles), completion on
//              mbarriers;
//   warp 1   : allocates tensor memory and issues tcgen05.mma (fp16 x fp16 -> fp32
//              accumulator in TMEM) from shared-memory descriptors, one thread;
//   warps 2-5: epilogue, tcgen05.ld of the accumulator, alpha, fp16 stores.
// Either operand may be K-major or MN-major in global memory (the eight layout
// cases a BLAS expresses with op flags and operand swapping); that choice only
// changes the TMA box shape and the shared-memory descriptor.
// Every mbarrier wait is bounded: after ~2 s it records an error code, the CTA
// drains, frees its tensor memory and returns.
//
// gemm_simt_kernel: plain FMA fallback for operands TMA cannot address
// (strides that are not multiples of 16 bytes, or no unit-stride index).

#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

#include "ops.h"

namespace sb {

thread_local int g_last_gemm_impl = 0;

// ---------------------------------------------------------------------------
// Einsum -> GEMM
// ---------------------------------------------------------------------------
namespace {

struct Operand {
  const char* dims;
  const sb_tensor* t;
  int find(char c) const {
    const char* p = strchr(dims, c);
    return p ? (int)(p - dims) : -1;
  }
};

// Collapse the letters of `group`, taken in the order `order`, to (size, stride) in operand o.
bool collapse_in(const Operand& o, const std::string& order, long long* stride) {
  long long st = 0;
  bool first = true;
  long long expect = 0;
  for (int i = (int)order.size() - 1; i >= 0; --i) {
    const int d = o.find(order[i]);
    const long long sz = o.t->size[d];
    if (sz == 1) continue;
    if (first) {
      st = o.t->stride[d];
      expect = st * sz;
      first = false;
    } else {
      if (o.t->stride[d] != expect) return false;
      expect *= sz;
    }
  }
  *stride = first ? 0 : st;
  return true;
}

std::string order_in(const Operand& o, const std::string& group) {
  std::string r;
  for (const char* p = o.dims; *p; ++p)
    if (group.find(*p) != std::string::npos) r.push_back(*p);
  return r;
}

}  // namespace

int plan_einsum(const char* a_dims, const sb_tensor* a, const char* b_dims, const sb_tensor* b,
                const char* c_dims, const sb_tensor* c, float alpha, GemmProblem* g) {
  if (!a_dims || !b_dims || !c_dims || !a || !b || !c || !g)
    return fail(SB_ERR_ARG, "einsum: null argument");
  Operand A{a_dims, a}, B{b_dims, b}, C{c_dims, c};
  for (const Operand* o : {&A, &B, &C}) {
    const int n = (int)strlen(o->dims);
    if (n != o->t->ndim || n > SB_MAX_DIMS)
      return fail(SB_ERR_LAYOUT, std::string("einsum: dims string '") + o->dims +
                                     "' does not match the operand's rank");
    for (int i = 0; i < n; ++i) {
      if (strchr(o->dims + i + 1, o->dims[i]))
        return fail(SB_ERR_LAYOUT, std::string("einsum: repeated index in '") + o->dims + "'");
      if (o->t->size[i] <= 0) return fail(SB_ERR_ARG, "einsum: non-positive extent");
    }
    if (!o->t->ptr) return fail(SB_ERR_ARG, "einsum: null data pointer");
  }
  std::string batch, sum, aonly, bonly;
  long long nb = 1, nm = 1, nn = 1, nk = 1;
  auto size_of = [&](char ch, long long* out) -> bool {
    long long s = -1;
    for (const Operand* o : {&A, &B, &C}) {
      const int d = o->find(ch);
      if (d < 0) continue;
      if (s < 0) s = o->t->size[d];
      else if (s != o->t->size[d]) return false;
    }
    *out = s;
    return true;
  };
  std::string all = std::string(a_dims) + b_dims + c_dims, seen;
  for (char ch : all) {
    if (seen.find(ch) != std::string::npos) continue;
    seen.push_back(ch);
    const bool ia = A.find(ch) >= 0, ib = B.find(ch) >= 0, ic = C.find(ch) >= 0;
    long long s;
    if (!size_of(ch, &s))
      return fail(SB_ERR_ARG, std::string("einsum: extent of index '") + ch + "' differs between operands");
    if (ia && ib && ic) { batch.push_back(ch); nb *= s; }
    else if (ia && ib) { sum.push_back(ch); nk *= s; }
    else if (ia && ic) { aonly.push_back(ch); nm *= s; }
    else if (ib && ic) { bonly.push_back(ch); nn *= s; }
    else return fail(SB_ERR_UNSUPPORTED, std::string("einsum: index '") + ch + "' appears in only one operand");
  }
  // Find one index order per group under which the group collapses in every operand holding it.
  auto solve = [&](const std::string& group, std::initializer_list<const Operand*> ops,
                   long long* strides) -> bool {
    if (group.empty()) {
      int i = 0;
      for (const Operand* o : ops) { (void)o; strides[i++] = 0; }
      return true;
    }
    for (const Operand* cand : ops) {
      const std::string order = order_in(*cand, group);
      bool ok = true;
      int i = 0;
      for (const Operand* o : ops) ok = ok && collapse_in(*o, order, &strides[i++]);
      if (ok) return true;
    }
    return false;
  };
  long long sb3[3], sm2[2], sn2[2], sk2[2];
  if (!solve(batch, {&A, &B, &C}, sb3))
    return fail(SB_ERR_UNSUPPORTED, "einsum: batch indices do not collapse to one stride in every operand");
  if (!solve(aonly, {&A, &C}, sm2))
    return fail(SB_ERR_UNSUPPORTED, "einsum: A-only indices do not collapse to one stride");
  if (!solve(bonly, {&B, &C}, sn2))
    return fail(SB_ERR_UNSUPPORTED, "einsum: B-only indices do not collapse to one stride");
  if (!solve(sum, {&A, &B}, sk2))
    return fail(SB_ERR_UNSUPPORTED, "einsum: summed indices do not collapse to one stride");
  g->batch = nb; g->M = nm; g->N = nn; g->K = nk;
  g->sAb = sb3[0]; g->sBb = sb3[1]; g->sCb = sb3[2];
  g->sAm = sm2[0]; g->sCm = sm2[1];
  g->sBn = sn2[0]; g->sCn = sn2[1];
  g->sAk = sk2[0]; g->sBk = sk2[1];
  g->A = a->ptr; g->B = b->ptr; g->C = c->ptr;
  g->alpha = alpha;
  return SB_OK;
}

// ---------------------------------------------------------------------------
// SIMT fallback
// ---------------------------------------------------------------------------
namespace {

constexpr int kSt = 64, kSk = 16;

__global__ void __launch_bounds__(256)
gemm_simt_kernel(GemmProblem g) {
  grid_dependency_sync();
  __shared__ float As[kSk][kSt + 4];
  __shared__ float Bs[kSk][kSt + 4];
  const int tid = threadIdx.x;
  const int tx = tid % 16, ty = tid / 16;
  const long long m0 = (long long)blockIdx.y * kSt, n0 = (long long)blockIdx.x * kSt;
  const sb_half* A = reinterpret_cast<const sb_half*>(g.A);
  const sb_half* B = reinterpret_cast<const sb_half*>(g.B);
  sb_half* C = reinterpret_cast<sb_half*>(g.C);
  for (long long bt = blockIdx.z; bt < g.batch; bt += gridDim.z) {
    float acc[4][4] = {};
    for (long long k0 = 0; k0 < g.K; k0 += kSk) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int idx = tid + 256 * i;
        // consecutive threads follow the unit-stride index of each operand
        int am, ak, bn, bk;
        if (g.sAk == 1) { ak = idx % kSk; am = idx / kSk; } else { am = idx % kSt; ak = idx / kSt; }
        if (g.sBk == 1) { bk = idx % kSk; bn = idx / kSk; } else { bn = idx % kSt; bk = idx / kSt; }
        const long long m = m0 + am, ka = k0 + ak, n = n0 + bn, kb = k0 + bk;
        As[ak][am] = (m < g.M && ka < g.K) ? sb_h2f(A[bt * g.sAb + m * g.sAm + ka * g.sAk]) : 0.f;
        Bs[bk][bn] = (n < g.N && kb < g.K) ? sb_h2f(B[bt * g.sBb + n * g.sBn + kb * g.sBk]) : 0.f;
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < kSk; ++k) {
        float a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) { a[i] = As[k][ty * 4 + i]; b[i] = Bs[k][tx * 4 + i]; }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] += a[i] * b[j];
      }
      __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const long long m = m0 + ty * 4 + i, n = n0 + tx * 4 + j;
        if (m < g.M && n < g.N) C[bt * g.sCb + m * g.sCm + n * g.sCn] = sb_f2h(acc[i][j] * g.alpha);
      }
  }
}

}  // namespace

int launch_gemm_simt(cudaStream_t s, const GemmProblem& g) {
  if (g.batch == 0 || g.M == 0 || g.N == 0) return SB_OK;
  dim3 grid((unsigned)((g.N + kSt - 1) / kSt), (unsigned)((g.M + kSt - 1) / kSt),
            (unsigned)std::min<long long>(g.batch, 65535));
  SB_LAUNCH_OK(launch_k(gemm_simt_kernel, grid, 256, 0, s, g));
  SB_CUDA_OK(cudaGetLastError());
  g_last_gemm_impl = SB_GEMM_SIMT;
  return SB_OK;
}

// ---------------------------------------------------------------------------
// tcgen05 path
// ---------------------------------------------------------------------------
namespace {

constexpr int kBM = 128;                 // UMMA M
constexpr int kBK = 64;                  // one 128-byte swizzle span of fp16
constexpr int kTcThreads = 192;          // 6 warps
constexpr int kABytes = kBM * kBK * 2;   // 16 KiB per 64-wide K block
constexpr int kStageOutBytes = 4 * 2 * 4096;  // epilogue staging: 4 warps x 2 buffers x (32 rows x 128 B)
constexpr unsigned long long kWaitNs = 2000000000ull;

__device__ int g_tc_error = 0;  // first failure code of any tcgen05 kernel on this device since the last reset

// Work fused behind a contraction's epilogue (paired-CTA kernel, TMA-store mode).  All extra tensors have C's
// geometry; the arithmetic on the stored fp16 values is the flat elementwise kernels', so results are identical
// to running those kernels on C afterwards.
//   kind 1: out2 = C + bias                        (attention input biases)
//   kind 2: out2 = C + resid                       (encoder-input gradient)
//   kind 3: out2 = C + bias, out3 = mask * act(out2)   (bias + activation + dropout)
//   kind 4: out2 = act'(resid) * mask * C, and its column sums per 32 rows   (dropout + activation backward, bias
//           gradient); C itself is never stored.  Contraction and separate operator 57 -> 43 + 4 us at B=8, L=512 (58 MB
//           less traffic), 142 -> 97 + 8 at B=96, L=128
struct EpiParams {
  int kind;
  int vec_along_m;       // bias indexed by the row (m) instead of the column (n)
  const sb_half* vec;
  const sb_half* resid;   // [M][N], row stride sCm
  uint8_t* mask;         // [M][N] bytes, row stride sCm; read, or written when rng.philox
  int activation;
  int skip_c;            // C itself is not stored (nothing reads it once the fused outputs exist)
  int skip_out2;         // kind 3: the pre-activation and (mask == null) the generated mask are not stored either
  Rng rng;
  float* partial;        // kind 4: column sums, one row of N floats per 32 rows of C
};

struct TcParams {
  long long M, N, K;
  long long sCb, sCm, sCn;
  void* C;             // fp16 output, or fp32 split-K partials [split][batch][M][N]
  float alpha;
  int a_mn, b_mn;      // operand is MN-major in global memory
  int a_swap, b_swap;  // tensor-map dims 1 and 2 are exchanged (kept in increasing-stride order)
  int c_swap;
  int c_mode;          // 0: scalar fp16 stores, 1: 128-bit fp16 stores, 2: TMA stores, 3: fp32 partials
  int tiles_m, tiles_n, batch;
  int splits, kt_per_split;  // split-K: K stages per split
  long long tiles;     // tiles_m * tiles_n * batch * splits
  EpiParams epi;       // paired-CTA kernel only
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// Bounded wait: gives up after kWaitNs, or earlier when another CTA already failed.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int code) {
  unsigned long long t0 = 0;
  for (uint32_t it = 1;; ++it) {
    if (mbar_try(bar, parity)) return true;
    if ((it & 0x3ffu) == 0) {
      if (*reinterpret_cast<volatile int*>(&g_tc_error) != 0) return false;
      const unsigned long long now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > kWaitNs) { atomicCAS(&g_tc_error, 0, code); return false; }
    }
  }
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar,
                                            int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
      ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor, 128-byte swizzle.  lbo/sbo in bytes.
__device__ __forceinline__ uint64_t make_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3ffffu) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3fffu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3fffu) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version of this architecture
  d |= (uint64_t)2 << 61;  // SWIZZLE_128B
  return d;
}
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// 32 consecutive accumulator columns of this thread's TMEM lane (no wait)
__device__ __forceinline__ void tmem_ld32_nowait(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// KS: 64-wide K blocks per pipeline stage (2 halves the number of passes over a K-major
// operand's rows, which matters when the operand streams from HBM).
template <int BN, int KS>
struct TcCfg {
  static constexpr int kBBytes = BN * kBK * 2;                 // per K block
  static constexpr int kStageBytes = KS * (kABytes + kBBytes);
  static constexpr int kStages = (196608 / kStageBytes) > 8 ? 8 : (196608 / kStageBytes);
  static constexpr int kTileBytes = kStages * kStageBytes;
  static constexpr int kTmemCols = 2 * BN;  // two accumulators: the epilogue of one tile overlaps the next tile's MMAs
  static constexpr int kSmemBytes = kTileBytes + kStageOutBytes + 1024 /*alignment slack*/ + 256 /*barriers*/;
};

// Persistent: CTA c works on items c, c + gridDim.x, ...; item = (split, batch, m tile, n tile), n fastest.
template <int BN, int KS>
__global__ void __launch_bounds__(kTcThreads, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               const __grid_constant__ CUtensorMap tmC, const TcParams p) {
  using Cfg = TcCfg<BN, KS>;
  constexpr int S = Cfg::kStages;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t tiles = (raw + 1023u) & ~1023u;
  const uint32_t stage_out = tiles + Cfg::kTileBytes;  // 1024-aligned
  const uint32_t bars = stage_out + kStageOutBytes;    // full[S], empty[S], acc_full[2], acc_empty[2]
  const uint32_t bar_full = bars, bar_empty = bars + 8 * S;
  const uint32_t bar_accf = bars + 16 * S, bar_acce = bars + 16 * S + 16;
  uint8_t* gen_base = smem_raw + (tiles - raw);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen_base + Cfg::kTileBytes + kStageOutBytes + 16 * S + 32);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int KT = (int)((p.K + kBK - 1) / kBK);        // 64-wide K blocks in total
  const long long per_split = (long long)p.tiles_n * p.tiles_m * p.batch;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_accf + 8 * b, 1);
      mbar_init(bar_acce + 8 * b, 4);  // one arrival per epilogue warp
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmA) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmB) : "memory");
    if (p.c_mode == 2) asm volatile("prefetch.tensormap [%0];" ::"l"(&tmC) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)Cfg::kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  grid_dependency_sync();  // barriers, tensor memory and tensor maps were set up while the previous kernel drained

  if (warp == 0) {
    // ---------------- TMA producer (whole warp walks the loop, lane 0 issues) ----------------
    uint32_t it = 0;
    bool ok = true;
    for (long long t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
      const long long tt = t % per_split;
      const int split = (int)(t / per_split);
      const int n0 = (int)(tt % p.tiles_n) * BN;
      const int m0 = (int)((tt / p.tiles_n) % p.tiles_m) * kBM;
      const int bt = (int)(tt / ((long long)p.tiles_n * p.tiles_m));
      const int kb_begin = split * p.kt_per_split;
      const int kb_end = min(KT, kb_begin + p.kt_per_split);
      for (int kb = kb_begin; kb < kb_end; kb += KS, ++it) {
        const int s = it % S;
        const uint32_t ph = (it / S) & 1u;
        ok = __all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * s, ph ^ 1u, 1));
        if (!ok) break;
        if (lane == 0) {
          const uint32_t full = bar_full + 8 * s;
          mbar_expect_tx(full, (uint32_t)Cfg::kStageBytes);
          const uint32_t sa0 = tiles + s * Cfg::kStageBytes;
          const uint32_t sb0 = sa0 + KS * kABytes;
#pragma unroll
          for (int ks = 0; ks < KS; ++ks) {
            // blocks past the end of K are fetched out of range: zero filled, no memory traffic
            const int k0 = (kb + ks) * kBK;
            const uint32_t sa = sa0 + ks * kABytes, sb_ = sb0 + ks * Cfg::kBBytes;
            if (!p.a_mn) {
              // dims (k, m, batch), box 64 x 128
              if (p.a_swap) tma_load_3d(sa, &tmA, full, k0, bt, m0);
              else tma_load_3d(sa, &tmA, full, k0, m0, bt);
            } else {
              // dims (m, k, batch), two boxes of 64 (m) x 64 (k)
#pragma unroll
              for (int h = 0; h < kBM / 64; ++h) {
                if (p.a_swap) tma_load_3d(sa + h * 8192, &tmA, full, m0 + 64 * h, bt, k0);
                else tma_load_3d(sa + h * 8192, &tmA, full, m0 + 64 * h, k0, bt);
              }
            }
            if (!p.b_mn) {
              if (p.b_swap) tma_load_3d(sb_, &tmB, full, k0, bt, n0);
              else tma_load_3d(sb_, &tmB, full, k0, n0, bt);
            } else {
#pragma unroll
              for (int h = 0; h < BN / 64; ++h) {
                if (p.b_swap) tma_load_3d(sb_ + h * 8192, &tmB, full, n0 + 64 * h, bt, k0);
                else tma_load_3d(sb_ + h * 8192, &tmB, full, n0 + 64 * h, k0, bt);
              }
            }
          }
        }
        __syncwarp();
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (whole warp walks the loop, lane 0 issues) ----------------
    // instruction descriptor: fp32 accumulate, fp16 A and B, operand majors, N, M
    const uint32_t idesc = (1u << 4) | SB_IDESC_AB_FMT | ((uint32_t)(p.a_mn ? 1 : 0) << 15) |
                           ((uint32_t)(p.b_mn ? 1 : 0) << 16) | ((uint32_t)(BN >> 3) << 17) |
                           ((uint32_t)(kBM >> 4) << 24);
    // K-major: 8-row groups 1024 B apart, 32 B per K step of 16.
    // MN-major: 64-wide MN blocks 8192 B apart (LBO), 8-row K groups 1024 B apart, 2048 B per K step.
    const uint32_t a_lbo = p.a_mn ? 8192u : 16u, b_lbo = p.b_mn ? 8192u : 16u;
    const uint32_t a_step = p.a_mn ? 2048u : 32u, b_step = p.b_mn ? 2048u : 32u;
    uint32_t it = 0, lt = 0;
    bool ok = true;
    for (long long t = blockIdx.x; t < p.tiles && ok; t += gridDim.x, ++lt) {
      const int split = (int)(t / per_split);
      const int kb_begin = split * p.kt_per_split;
      const int kb_end = min(KT, kb_begin + p.kt_per_split);
      const uint32_t buf = lt & 1u, aph = (lt >> 1) & 1u;
      // the epilogue must have drained this accumulator (passes at once for its first use)
      ok = __all_sync(0xffffffffu, mbar_wait(bar_acce + 8 * buf, aph ^ 1u, 4));
      if (!ok) break;
      tc_fence_after();
      const uint32_t tmem_d = tmem_base + buf * BN;
      for (int kb = kb_begin; kb < kb_end; kb += KS, ++it) {
        const int s = it % S;
        const uint32_t ph = (it / S) & 1u;
        ok = __all_sync(0xffffffffu, mbar_wait(bar_full + 8 * s, ph, 2));
        if (!ok) break;
        tc_fence_after();
        if (lane == 0) {
          const uint32_t sa0 = tiles + s * Cfg::kStageBytes;
          const uint32_t sb0 = sa0 + KS * kABytes;
#pragma unroll
          for (int ks = 0; ks < KS; ++ks) {
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k) {
              const uint64_t da = make_desc(sa0 + ks * kABytes + k * a_step, a_lbo, 1024u);
              const uint64_t db = make_desc(sb0 + ks * Cfg::kBBytes + k * b_step, b_lbo, 1024u);
              umma_f16(tmem_d, da, db, idesc, (kb > kb_begin || ks > 0 || k > 0) ? 1u : 0u);
            }
          }
          umma_commit(bar_empty + 8 * s);  // frees the stage once these MMAs have read it
        }
        __syncwarp();
      }
      if (ok && lane == 0) umma_commit(bar_accf + 8 * buf);
      __syncwarp();
    }
  } else {
    // ---------------- epilogue (4 warps; warp w reads TMEM lanes 32*(w%4)..+31) ----------------
    const int q = warp & 3;
    const uint32_t my_stage = stage_out + (uint32_t)(warp - 2) * 8192u;  // two 4 KiB buffers
    uint8_t* my_stage_gen = gen_base + Cfg::kTileBytes + (warp - 2) * 8192;
    uint32_t lt = 0, nstore = 0;
    bool ok = true;
    for (long long t = blockIdx.x; t < p.tiles && ok; t += gridDim.x, ++lt) {
      const long long tt = t % per_split;
      const int split = (int)(t / per_split);
      const int n0 = (int)(tt % p.tiles_n) * BN;
      const int m0 = (int)((tt / p.tiles_n) % p.tiles_m) * kBM;
      const long long bt = tt / ((long long)p.tiles_n * p.tiles_m);
      const uint32_t buf = lt & 1u, aph = (lt >> 1) & 1u;
      ok = __all_sync(0xffffffffu, mbar_wait(bar_accf + 8 * buf, aph, 3));
      if (!ok) break;
      tc_fence_after();
      const long long m = (long long)m0 + q * 32 + lane;
      const uint32_t tsrc = tmem_base + buf * BN + ((uint32_t)(q * 32) << 16);
      if (p.c_mode == 2) {
        // 64 columns at a time: TMEM -> registers -> fp16 -> swizzled staging row -> TMA store
#pragma unroll 1
        for (int c = 0; c < BN / 64; ++c) {
          uint32_t r[64];
          tmem_ld32_nowait(tsrc + (uint32_t)(c * 64), r);
          tmem_ld32_nowait(tsrc + (uint32_t)(c * 64 + 32), r + 32);
          tmem_ld_wait();
          if (c == BN / 64 - 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_acce + 8 * buf);
          }
          const uint32_t sbuf = nstore & 1u;
          // the store issued two chunks ago must have finished reading this buffer
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
          __syncwarp();
          uint8_t* row = my_stage_gen + sbuf * 4096 + lane * 128;
#pragma unroll
          for (int v = 0; v < 8; ++v) {
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(r[v * 8 + e]) * p.alpha;
            *reinterpret_cast<uint4*>(row + ((v ^ (lane & 7)) << 4)) = pack8(f);
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          const int nc = n0 + c * 64, mc = m0 + q * 32;
          if (lane == 0 && nc < p.N && mc < p.M) {
            if (p.c_swap) tma_store_3d(&tmC, my_stage + sbuf * 4096, nc, (int)bt, mc);
            else tma_store_3d(&tmC, my_stage + sbuf * 4096, nc, mc, (int)bt);
          }
          if (lane == 0) asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          ++nstore;
        }
      } else if (p.c_mode == 3) {
        float* crow = reinterpret_cast<float*>(p.C) + ((long long)split * p.batch + bt) * p.M * p.N + m * p.N;
#pragma unroll 1
        for (int c = 0; c < BN / 32; ++c) {
          uint32_t r[32];
          tmem_ld32_nowait(tsrc + (uint32_t)(c * 32), r);
          tmem_ld_wait();
          if (c == BN / 32 - 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_acce + 8 * buf);
          }
          if (m < p.M) {
            const long long nb = (long long)n0 + c * 32;
#pragma unroll
            for (int v = 0; v < 8; ++v)
              if (nb + v * 4 < p.N)  // N % 4 == 0 in this mode
                *reinterpret_cast<uint4*>(crow + nb + v * 4) = make_uint4(r[v * 4], r[v * 4 + 1], r[v * 4 + 2], r[v * 4 + 3]);
          }
        }
      } else {
        sb_half* crow = reinterpret_cast<sb_half*>(p.C) + bt * p.sCb + m * p.sCm;
#pragma unroll 1
        for (int c = 0; c < BN / 32; ++c) {
          uint32_t r[32];
          tmem_ld32_nowait(tsrc + (uint32_t)(c * 32), r);
          tmem_ld_wait();
          if (c == BN / 32 - 1) {
            // accumulator fully read into registers: hand it back to the MMA warp
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_acce + 8 * buf);
          }
          if (m < p.M) {
            const long long nb = (long long)n0 + c * 32;
            if (p.c_mode == 1) {
#pragma unroll
              for (int v = 0; v < 4; ++v) {
                if (nb + v * 8 < p.N) {
                  float f[8];
#pragma unroll
                  for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(r[v * 8 + e]) * p.alpha;
                  *reinterpret_cast<uint4*>(crow + nb + v * 8) = pack8(f);
                }
              }
            } else {
#pragma unroll
              for (int e = 0; e < 32; ++e)
                if (nb + e < p.N) crow[(nb + e) * p.sCn] = sb_f2h(__uint_as_float(r[e]) * p.alpha);
            }
          }
        }
      }
    }
    // all bulk stores of this thread must be complete before the CTA's shared memory goes away
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    __syncwarp();
  }
  if (*reinterpret_cast<volatile int*>(&g_tc_error) != 0) {
    // failure path: give bulk copies already in flight time to land before the CTA's memory is reused
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 1000000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)Cfg::kTmemCols) : "memory");
  }
}

// out = alpha * sum over splits of the fp32 partials [split][batch][M][N] (fixed order)
__global__ void __launch_bounds__(256)
splitk_reduce_kernel(const float* __restrict__ ws, int splits, long long batch, long long M, long long N,
                     sb_half* out, long long sCb, long long sCm, long long sCn, float alpha) {
  grid_dependency_sync();
  const long long total4 = batch * M * N / 4;  // N % 4 == 0
  const long long plane = batch * M * N;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < total4; i += (long long)gridDim.x * 256) {
    // all partials of this element are requested before any is added (splits <= 4), then added in split order
    float4 part[4];
#pragma unroll
    for (int s = 0; s < 4; ++s)
      part[s] = s < splits ? __ldcs(reinterpret_cast<const float4*>(ws + s * plane) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 acc = part[0];
#pragma unroll
    for (int s = 1; s < 4; ++s) {
      acc.x += part[s].x; acc.y += part[s].y; acc.z += part[s].z; acc.w += part[s].w;
    }
    const long long e = i * 4;
    const long long n = e % N, m = (e / N) % M, b = e / (N * M);
    sb_half* o = out + b * sCb + m * sCm + n * sCn;
    if (sCn == 1 && ((reinterpret_cast<uintptr_t>(o) & 7u) == 0)) {
      sb_half2 lo = sb_f2h2(acc.x * alpha, acc.y * alpha), hi = sb_f2h2(acc.z * alpha, acc.w * alpha);
      uint2 u;
      u.x = *reinterpret_cast<uint32_t*>(&lo);
      u.y = *reinterpret_cast<uint32_t*>(&hi);
      *reinterpret_cast<uint2*>(o) = u;
    } else {
      o[0] = sb_f2h(acc.x * alpha);
      o[sCn] = sb_f2h(acc.y * alpha);
      o[2 * sCn] = sb_f2h(acc.z * alpha);
      o[3 * sCn] = sb_f2h(acc.w * alpha);
    }
  }
}

#include "gemm_pair.cuh"
#include "gemm_pair_splitk.cuh"
#include "gemm_cluster_splitk.cuh"
#include "attn_fused.cuh"
#include "score_contract.cuh"
#include "flash_attn.cuh"
#include "peak_probe.cuh"

// ---- host side ------------------------------------------------------------
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
std::once_flag g_encode_once;

void load_encode() {
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
      q == cudaDriverEntryPointSuccess)
    g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
}

struct OperandMap {
  CUtensorMap map;
  int mn;    // MN-major
  int swap;  // dims 1 and 2 exchanged
};

// 3-D tensor map over dims (inner, d1, d2) with element strides (1, s1, s2) and box (b0, b1, 1);
// dims 1 and 2 are exchanged when needed to keep strides increasing.  fp16 elements with 128-byte
// swizzle, or (bytes = true) single bytes with 64-byte swizzle.
bool encode_map(const void* ptr, cuuint64_t n0, cuuint64_t n1, cuuint64_t n2, long long s1, long long s2,
                cuuint32_t b0, cuuint32_t b1, CUtensorMap* map, int* swapped, std::string* why, bool bytes = false) {
  const long long esize = bytes ? 1 : 2;
  if (reinterpret_cast<uintptr_t>(ptr) & 15u) { *why = "base is not 16-byte aligned"; return false; }
  cuuint64_t dim[3] = {n0, n1, n2};
  long long str[3] = {1, s1, s2};
  cuuint32_t box[3] = {b0, b1, 1};
  // extent-1 dims: any legal stride (a multiple of 8 elements)
  const long long unit = 16 / esize;
  if (dim[1] == 1) str[1] = ((long long)dim[0] + unit - 1) / unit * unit;
  if (dim[2] == 1) str[2] = std::max(str[1] * (long long)dim[1], ((long long)dim[0] + unit - 1) / unit * unit);
  *swapped = 0;
  if (str[2] < str[1]) {
    std::swap(dim[1], dim[2]);
    std::swap(str[1], str[2]);
    std::swap(box[1], box[2]);
    *swapped = 1;
  }
  for (int i = 1; i < 3; ++i)
    if (str[i] <= 0 || (str[i] * esize) % 16 != 0) { *why = "stride is not a positive multiple of 16 bytes"; return false; }
  for (int i = 0; i < 3; ++i)
    if (dim[i] == 0 || dim[i] > 0xffffffffull) { *why = "extent out of range"; return false; }
  cuuint64_t gstr[2] = {(cuuint64_t)(str[1] * esize), (cuuint64_t)(str[2] * esize)};
  cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = g_encode(map, bytes ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : SB_TMAP_DTYPE, 3,
                              const_cast<void*>(ptr), dim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              bytes ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { *why = "cuTensorMapEncodeTiled rejected it (code " + std::to_string((int)r) + ")"; return false; }
  return true;
}

// Operand X[batch][r][k] (r = m or n) with strides (sb, sr, sk); tile = rows x 64 (k).
bool make_operand_map(const void* ptr, long long R, long long K, long long batch, long long sr,
                      long long sk, long long sb, int rows, OperandMap* out, std::string* why) {
  if (sk == 1 || K == 1) {  // K-major (a single K column is K-major with any stride)
    out->mn = 0;
    return encode_map(ptr, (cuuint64_t)K, (cuuint64_t)R, (cuuint64_t)batch, sr, sb, kBK, (cuuint32_t)rows,
                      &out->map, &out->swap, why);
  }
  if (sr == 1) {
    out->mn = 1;
    return encode_map(ptr, (cuuint64_t)R, (cuuint64_t)K, (cuuint64_t)batch, sk, sb, 64, kBK, &out->map,
                      &out->swap, why);
  }
  *why = "operand has no unit-stride index";
  return false;
}

int g_sm_budget = 0;  // 0: all SMs; otherwise the persistent grid leaves the rest to concurrent kernels

int device_sms() {
  static thread_local int cached_dev = -1, cached = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev != cached_dev) {
    cudaDeviceGetAttribute(&cached, cudaDevAttrMultiProcessorCount, dev);
    cached_dev = dev;
  }
  return cached > 0 ? cached : 148;
}
int sm_count() {
  const int n = device_sms();
  return (g_sm_budget > 0 && g_sm_budget < n) ? g_sm_budget : n;
}

// Split K only when the output tiles cover less than a third of the SMs: the fp32 partials cost
// 2 * splits * M * N * 4 bytes of extra traffic, which a fuller grid does not win back.
int pick_splits(long long tiles, int KT, int ks, long long out_elems, size_t ws_bytes) {
  const int sms = sm_count();
  if (tiles * 3 > sms) return 1;
  int best = 1;
  for (int s : {2, 3, 4}) {
    if (KT / s < 8 * ks) break;  // keep at least 8 stages per item
    if ((size_t)s * out_elems * sizeof(float) > ws_bytes) break;
    if (tiles * s > sms) break;
    best = s;
  }
  return best;
}

template <int BN, int KS>
int launch_tc(cudaStream_t s, const GemmProblem& g, const OperandMap& a, const OperandMap& b, void* ws,
              size_t ws_bytes) {
  using Cfg = TcCfg<BN, KS>;
  // per-device attribute; setting it is cheap and idempotent
  SB_CUDA_OK(ensure_dynamic_smem(reinterpret_cast<const void*>(gemm_tc_kernel<BN, KS>), Cfg::kSmemBytes));
  TcParams p;
  memset(&p.epi, 0, sizeof(p.epi));
  p.M = g.M; p.N = g.N; p.K = g.K;
  p.sCb = g.sCb; p.sCm = g.sCm; p.sCn = g.sCn;
  p.C = g.C;
  p.alpha = g.alpha;
  p.a_mn = a.mn; p.b_mn = b.mn; p.a_swap = a.swap; p.b_swap = b.swap; p.c_swap = 0;
  p.tiles_n = (int)((g.N + BN - 1) / BN);
  p.tiles_m = (int)((g.M + kBM - 1) / kBM);
  p.batch = (int)g.batch;
  const int KT = (int)((g.K + kBK - 1) / kBK);
  const long long base_tiles = (long long)p.tiles_m * p.tiles_n * g.batch;
  p.splits = 1;
  if (ws && g.N % 4 == 0) p.splits = pick_splits(base_tiles, KT, KS, g.batch * g.M * g.N, ws_bytes);
  p.kt_per_split = ((KT + p.splits - 1) / p.splits + KS - 1) / KS * KS;
  p.splits = (KT + p.kt_per_split - 1) / p.kt_per_split;  // no split may be left without work
  p.tiles = base_tiles * p.splits;
  CUtensorMap cmap;
  memset(&cmap, 0, sizeof(cmap));
  // tensor-map stores clip at N; the plain 128-bit ones need it to be a multiple of 8
  const bool c_tma = g.sCn == 1 && g.sCm % 8 == 0 && (g.batch == 1 || g.sCb % 8 == 0) && (reinterpret_cast<uintptr_t>(g.C) & 15u) == 0;
  if (p.splits > 1) {
    p.c_mode = 3;
    p.C = ws;
  } else {
    p.c_mode = c_tma && g.N % 8 == 0 ? 1 : 0;
    if (c_tma) {
      std::string why;
      int swapped = 0;
      if (encode_map(g.C, (cuuint64_t)g.N, (cuuint64_t)g.M, (cuuint64_t)g.batch, g.sCm, g.sCb, 64, 32, &cmap, &swapped, &why)) {
        p.c_mode = 2;
        p.c_swap = swapped;
      }
    }
  }
  const unsigned grid = (unsigned)std::min<long long>(p.tiles, sm_count());
  SB_LAUNCH_OK(launch_k(gemm_tc_kernel<BN, KS>, grid, kTcThreads, Cfg::kSmemBytes, s, a.map, b.map, cmap, p));
  SB_CUDA_OK(cudaGetLastError());
  if (p.splits > 1) {
    const long long total4 = g.batch * g.M * g.N / 4;
    const unsigned blocks = (unsigned)std::min<long long>((total4 + 255) / 256, (long long)sm_count() * 8);
    SB_LAUNCH_OK(launch_k(splitk_reduce_kernel, blocks, 256, 0, s, reinterpret_cast<const float*>(ws), p.splits, g.batch, g.M, g.N,
                                                reinterpret_cast<sb_half*>(g.C), g.sCb, g.sCm, g.sCn, g.alpha));
    SB_CUDA_OK(cudaGetLastError());
  }
  return SB_OK;
}

// Epilogue warps per CTA of the paired kernel: 8 unless the environment asks for 4 (see pair::Cfg).
int pair_epi_warps() {
  static const int ew = [] {
    const char* e = getenv("SUBSTATION_B200_EPI_WARPS");
    return (e && e[0] == '4') ? 4 : 8;
  }();
  return ew;
}

// Paired-CTA launch: 256 x 256 tiles, one cluster of two CTAs per tile.
int pair_clusters() {
  static thread_local int cached_dev = -1, cached = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev != cached_dev) {
    cached_dev = dev;
    cached = 0;
    const bool ew8 = pair_epi_warps() == 8;
    const void* fn = ew8 ? reinterpret_cast<const void*>(pair::gemm_tc_pair_kernel<0, 8>)
                         : reinterpret_cast<const void*>(pair::gemm_tc_pair_kernel<0, 4>);
    const int smem = ew8 ? pair::Cfg<8>::kSmemBytes : pair::Cfg<4>::kSmemBytes;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess) {
      cudaLaunchConfig_t cfg;
      memset(&cfg, 0, sizeof(cfg));
      cfg.gridDim = dim3(2 * 74);
      cfg.blockDim = dim3(ew8 ? pair::Cfg<8>::kThreads : pair::Cfg<4>::kThreads);
      cfg.dynamicSmemBytes = smem;
      cudaLaunchAttribute attr;
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = 2; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
      cfg.attrs = &attr;
      cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess) cached = n;
      else cudaGetLastError();
    } else {
      cudaGetLastError();
    }
  }
  return cached;
}

bool pair_enabled() {
  static const bool on = [] {
    const char* e = getenv("SUBSTATION_B200_PAIR");
    return !(e && e[0] == '0');
  }();
  return on;
}

int launch_tc_pair(cudaStream_t s, const GemmProblem& g, const OperandMap& a, const OperandMap& b, int clusters,
                   const GemmEpilogue* epi = nullptr, bool vec_flipped = false) {
  TcParams p;
  memset(&p.epi, 0, sizeof(p.epi));
  p.M = g.M; p.N = g.N; p.K = g.K;
  p.sCb = g.sCb; p.sCm = g.sCm; p.sCn = g.sCn;
  p.C = g.C;
  p.alpha = g.alpha;
  p.a_mn = a.mn; p.b_mn = b.mn; p.a_swap = a.swap; p.b_swap = b.swap; p.c_swap = 0;
  p.tiles_n = (int)((g.N + 255) / 256);
  p.tiles_m = (int)((g.M + 255) / 256);
  p.batch = (int)g.batch;
  p.splits = 1;
  p.kt_per_split = (int)((g.K + kBK - 1) / kBK);
  p.tiles = (long long)p.tiles_m * p.tiles_n * g.batch;
  CUtensorMap cmap;
  memset(&cmap, 0, sizeof(cmap));
  const bool c_tma = g.sCn == 1 && g.sCm % 8 == 0 && (g.batch == 1 || g.sCb % 8 == 0) && (reinterpret_cast<uintptr_t>(g.C) & 15u) == 0;
  p.c_mode = c_tma && g.N % 8 == 0 ? 1 : 0;
  if (c_tma) {
    std::string why;
    int swapped = 0;
    if (encode_map(g.C, (cuuint64_t)g.N, (cuuint64_t)g.M, (cuuint64_t)g.batch, g.sCm, g.sCb, 64, 32, &cmap, &swapped, &why)) {
      p.c_mode = 2;
      p.c_swap = swapped;
    }
  }
  const int budget = sm_count() / 2;
  const unsigned nclusters = (unsigned)std::max<long long>(1, std::min<long long>(p.tiles, std::min(clusters, budget)));
  CUtensorMap cmap2, cmap3;
  memset(&cmap2, 0, sizeof(cmap2));
  memset(&cmap3, 0, sizeof(cmap3));
  if (epi) {
    // fused epilogue work needs the TMA-store path, and whole 64-column blocks where it reads anything along them
    const bool along_m = vec_flipped ? !epi->vec_along_m : epi->vec_along_m;
    if (p.c_mode != 2 || (g.N % 64 != 0 && !(epi->kind == 1 && along_m)))
      return fail(SB_ERR_UNSUPPORTED, "fused epilogue: output rows must be TMA-addressable with N a multiple of 64");
    std::string why;
    int sw = 0;
    if (!encode_map(epi->out2, (cuuint64_t)g.N, (cuuint64_t)g.M, (cuuint64_t)g.batch, g.sCm, g.sCb, 64, 32, &cmap2, &sw, &why) ||
        sw != p.c_swap)
      return fail(SB_ERR_UNSUPPORTED, "fused epilogue, second output: " + why);
    if (epi->kind == 3 && (!encode_map(epi->out3, (cuuint64_t)g.N, (cuuint64_t)g.M, (cuuint64_t)g.batch, g.sCm, g.sCb, 64, 32, &cmap3,
                                       &sw, &why) || sw != p.c_swap))
      return fail(SB_ERR_UNSUPPORTED, "fused epilogue, third output: " + why);
    p.epi.kind = epi->kind;
    p.epi.vec_along_m = vec_flipped ? !epi->vec_along_m : epi->vec_along_m;
    // the epilogue reads its side inputs with 128-bit accesses at (row * sCm + 64-column block)
    auto misaligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) != 0; };
    if ((epi->kind == 1 || epi->kind == 3) && !p.epi.vec_along_m && misaligned(epi->vec))
      return fail(SB_ERR_ALIGNMENT, "fused epilogue: a bias along the columns must be 16-byte aligned");
    if ((epi->kind == 2 || epi->kind == 4) && misaligned(epi->resid))
      return fail(SB_ERR_ALIGNMENT, "fused epilogue: the residual must be 16-byte aligned");
    if ((epi->kind == 3 || epi->kind == 4) && (misaligned(epi->mask) || g.sCm % 16 != 0))
      return fail(SB_ERR_ALIGNMENT, "fused epilogue: the mask must be 16-byte aligned with a row pitch that is a multiple of 16");
    p.epi.vec = reinterpret_cast<const sb_half*>(epi->vec);
    p.epi.resid = reinterpret_cast<const sb_half*>(epi->resid);
    p.epi.mask = reinterpret_cast<uint8_t*>(epi->mask);
    p.epi.activation = epi->activation;
    p.epi.skip_c = epi->skip_c;
    p.epi.skip_out2 = epi->skip_out2;
    p.epi.rng = epi->rng;
    p.epi.partial = epi->partial;
  }
  const int kind = epi ? epi->kind : 0;
  auto launch = [&](auto kernel, int threads, int smem) {
    // per-device attribute; setting it is cheap and idempotent
    const cudaError_t ea = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
    if (ea != cudaSuccess) return ea;
    return launch_k(kernel, 2 * nclusters, threads, smem, s, a.map, b.map, cmap, cmap2, cmap3, p);
  };
  if (kind < 0 || kind > 4) return fail(SB_ERR_ARG, "fused epilogue: unknown kind");
#define SB_PAIR_CASE(K, EW)                                                                             \
  if (kind == K && ew == EW)                                                                            \
    SB_LAUNCH_OK(launch(pair::gemm_tc_pair_kernel<K, EW>, pair::Cfg<EW>::kThreads, pair::Cfg<EW>::kSmemBytes))
  const int ew = pair_epi_warps();
  SB_PAIR_CASE(0, 4); SB_PAIR_CASE(1, 4); SB_PAIR_CASE(2, 4); SB_PAIR_CASE(3, 4); SB_PAIR_CASE(4, 4);
  SB_PAIR_CASE(0, 8); SB_PAIR_CASE(1, 8); SB_PAIR_CASE(2, 8); SB_PAIR_CASE(3, 8); SB_PAIR_CASE(4, 8);
#undef SB_PAIR_CASE
  SB_CUDA_OK(cudaGetLastError());
  return SB_OK;
}

// Split-K clusters (SK CTA pairs per 256 x 256 tile, partials reduced through distributed shared memory).
// SUBSTATION_B200_PAIR_SPLITK: 0 switches the form off, 2..4 force that many pairs; unset, the launcher takes the
// largest number of pairs whose clusters are all resident at once.
int pair_splitk_forced() {
  static const int sk = [] {
    const char* e = getenv("SUBSTATION_B200_PAIR_SPLITK");
    if (!e) return -1;
    const int v = atoi(e);
    return (v >= 2 && v <= 4) ? v : 0;
  }();
  return sk;
}

template <int SK>
int splitk_clusters_resident() {
  static thread_local int cached_dev = -1, cached = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev != cached_dev) {
    cached_dev = dev;
    cached = 0;
    const void* fn = reinterpret_cast<const void*>(pair::gemm_tc_pair_splitk_kernel<8, SK>);
    const int smem = pair::Cfg<8>::kSmemBytes;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess) {
      cudaLaunchConfig_t cfg;
      memset(&cfg, 0, sizeof(cfg));
      cfg.gridDim = dim3(2 * SK * 16);
      cfg.blockDim = dim3(pair::Cfg<8>::kThreads);
      cfg.dynamicSmemBytes = smem;
      cudaLaunchAttribute attr;
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = 2 * SK; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
      cfg.attrs = &attr;
      cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess) cached = n;
      else cudaGetLastError();
    } else {
      cudaGetLastError();
    }
  }
  return cached;
}

template <int SK>
int launch_tc_pair_splitk(cudaStream_t s, const GemmProblem& g, const OperandMap& a, const OperandMap& b) {
  TcParams p;
  memset(&p.epi, 0, sizeof(p.epi));
  p.M = g.M; p.N = g.N; p.K = g.K;
  p.sCb = g.sCb; p.sCm = g.sCm; p.sCn = g.sCn;
  p.C = g.C;
  p.alpha = g.alpha;
  p.a_mn = a.mn; p.b_mn = b.mn; p.a_swap = a.swap; p.b_swap = b.swap; p.c_swap = 0;
  p.tiles_n = (int)((g.N + 255) / 256);
  p.tiles_m = (int)((g.M + 255) / 256);
  p.batch = (int)g.batch;
  const int KT = (int)((g.K + kBK - 1) / kBK);
  p.splits = SK;
  p.kt_per_split = (KT + SK - 1) / SK;
  p.tiles = (long long)p.tiles_m * p.tiles_n * g.batch;
  p.c_mode = 1;
  const void* fn = reinterpret_cast<const void*>(pair::gemm_tc_pair_splitk_kernel<8, SK>);
  SB_CUDA_OK(ensure_dynamic_smem(fn, pair::Cfg<8>::kSmemBytes));
  SB_LAUNCH_OK(launch_k(pair::gemm_tc_pair_splitk_kernel<8, SK>, (unsigned)(2 * SK * p.tiles), pair::Cfg<8>::kThreads,
                        pair::Cfg<8>::kSmemBytes, s, a.map, b.map, p));
  SB_CUDA_OK(cudaGetLastError());
  return SB_OK;
}

// Single-CTA split-K clusters for problems with a short side: how many CTAs share a tile's K (0: not this kernel).
// Up to 256 rows or columns: beyond that the paired kernel and its split-K form have tiles enough (at 512 tokens they are
// as fast).  Two CTAs fit on an SM, every CTA keeps two K blocks, and clusters of eight were slower than of four whenever
// both fit (barriers and remote reads: 10.5 against 6.8 us for `out` at 256 tokens, 15.7 against 12.3 us for dXlin1).
// Contractions and elementwise operators of an inference pass at 1024 features, together: 40.3 -> 35.4 us at 128 tokens,
// 58.4 -> 37.0 at 200, 46.4 -> 37.6 at 256; of a training step 104.8 -> 95.5, 135 -> 106, 118.8 -> 105.6 us.
// The device's SMs count here and not the budget: the number of parts is an order of summation, and results must not
// depend on the budget.  (Nor does the kernel hold SMs from a collective: its CTAs have one tile each and are gone in 5 to 12 us.)
int cluster_splits(const GemmProblem& g) {
  if (g.batch != 1 || g.sCn != 1 || std::min(g.M, g.N) > 256 || g.sCm % 8 != 0 || (reinterpret_cast<uintptr_t>(g.C) & 15u))
    return 0;
  const long long tiles = ((g.M + kBM - 1) / kBM) * ((g.N + csk::kBN - 1) / csk::kBN), KT = (g.K + kBK - 1) / kBK;
  const int sms = device_sms();
  for (int sk : {4, 2})
    if (tiles * sk <= 2 * sms && KT >= 2 * sk) return sk;
  return 0;
}

// C^T = B^T A^T
void transpose_problem(GemmProblem* g) {
  std::swap(g->M, g->N);
  std::swap(g->A, g->B);
  std::swap(g->sAb, g->sBb);
  std::swap(g->sAm, g->sBn);
  std::swap(g->sAk, g->sBk);
  std::swap(g->sCm, g->sCn);
}

template <int SK>
int launch_cluster_splitk(cudaStream_t s, const GemmProblem& g, const OperandMap& a, const OperandMap& b, const GemmEpilogue* epi,
                          bool vec_flipped) {
  TcParams p;
  memset(&p, 0, sizeof(p));
  p.M = g.M; p.N = g.N; p.K = g.K;
  p.sCm = g.sCm; p.sCn = 1;
  p.C = g.C;
  p.alpha = g.alpha;
  p.a_mn = a.mn; p.b_mn = b.mn; p.a_swap = a.swap; p.b_swap = b.swap;
  p.tiles_n = (int)((g.N + csk::kBN - 1) / csk::kBN);
  p.tiles_m = (int)((g.M + kBM - 1) / kBM);
  p.batch = 1;
  p.kt_per_split = (int)(((g.K + kBK - 1) / kBK + SK - 1) / SK);
  p.tiles = (long long)p.tiles_m * p.tiles_n;
  csk::Outs o{reinterpret_cast<sb_half*>(g.C), nullptr, nullptr};
  if (epi) {
    auto misaligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) != 0; };
    p.epi.kind = epi->kind;
    p.epi.vec_along_m = vec_flipped ? !epi->vec_along_m : epi->vec_along_m;
    if (epi->kind < 1 || epi->kind > 3 || (g.N % 8 != 0 && !(epi->kind == 1 && p.epi.vec_along_m)) || misaligned(epi->out2) || (epi->kind == 3 && misaligned(epi->out3)) ||
        (epi->kind != 2 && !p.epi.vec_along_m && misaligned(epi->vec)) || (epi->kind == 2 && misaligned(epi->resid)) ||
        (epi->kind == 3 && (reinterpret_cast<uintptr_t>(epi->mask) & 7u)))
      return fail(SB_ERR_UNSUPPORTED, "fused epilogue: not one the split-K cluster kernel takes");
    p.epi.vec = reinterpret_cast<const sb_half*>(epi->vec);
    p.epi.resid = reinterpret_cast<const sb_half*>(epi->resid);
    p.epi.mask = reinterpret_cast<uint8_t*>(epi->mask);
    p.epi.activation = epi->activation;
    p.epi.skip_c = epi->skip_c;
    p.epi.skip_out2 = epi->skip_out2;
    p.epi.rng = epi->rng;
    o.out2 = reinterpret_cast<sb_half*>(epi->out2);
    o.out3 = reinterpret_cast<sb_half*>(epi->out3);
  }
  const auto kernel = csk::gemm_cluster_splitk_kernel<SK>;
  SB_CUDA_OK(ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), csk::kSmemBytes));
  SB_LAUNCH_OK(launch_k(kernel, (unsigned)(p.tiles * SK), csk::kThreads, csk::kSmemBytes, s, a.map, b.map, p, o));
  return SB_OK;
}

int pick_bn(long long M, long long N, long long batch) {
  // 128 x 256 moves the fewest operand bytes per flop (each CTA fetches its own tiles), so it is
  // used whenever N fills most of it and the persistent grid still covers about half the SMs
  // (split-K can recover the rest when K is long).
  const long long mt = (M + kBM - 1) / kBM;
  if (N <= 64) return 64;
  if (N <= 128) return 128;
  const long long t256 = mt * ((N + 255) / 256) * batch;
  const bool fills = (N % 256 == 0) || (N % 256 > 128) || N >= 1024;
  if (fills && t256 >= 24) return 256;
  const long long t128 = mt * ((N + 127) / 128) * batch;
  if (t128 >= 64 || N % 128 == 0 || N % 128 > 64) return 128;
  return 64;
}

long long padded_work(long long M, long long N) {
  const long long mp = (M + kBM - 1) / kBM * kBM;
  const long long np = (N + 63) / 64 * 64;
  return mp * np;
}

}  // namespace

bool tcgen05_supported(const GemmProblem& g, std::string* why) {
  if (g.K < 1 || g.M < 1 || g.N < 1) { *why = "empty problem"; return false; }
  if (g.batch > 0x7fffffffLL) { *why = "too many batches"; return false; }
  if (!(g.sAk == 1 || g.sAm == 1 || g.K == 1)) { *why = "A has no unit-stride index"; return false; }
  if (!(g.sBk == 1 || g.sBn == 1 || g.K == 1)) { *why = "B has no unit-stride index"; return false; }
  return true;
}

int launch_gemm_tcgen05_epi(cudaStream_t s, const GemmProblem& g0, void* ws, size_t ws_bytes, const GemmEpilogue* epi) {
  std::string why;
  if (!tcgen05_supported(g0, &why)) return fail(SB_ERR_UNSUPPORTED, "tcgen05 contraction: " + why);
  std::call_once(g_encode_once, load_encode);
  if (!g_encode) return fail(SB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  OperandMap a, b;
  {
    GemmProblem gs = g0;                       // C's rows are the stored lines
    const bool flip = g0.sCn != 1 && g0.sCm == 1;
    if (flip) transpose_problem(&gs);
    if (const int sk = epi && !epi->few_tiles ? 0 : cluster_splits(gs)) {
      if (make_operand_map(gs.A, gs.M, gs.K, 1, gs.sAm, gs.sAk, gs.sAb, kBM, &a, &why) &&
          make_operand_map(gs.B, gs.N, gs.K, 1, gs.sBn, gs.sBk, gs.sBb, csk::kBN, &b, &why)) {
        const int st2 = sk == 4 ? launch_cluster_splitk<4>(s, gs, a, b, epi, flip) : launch_cluster_splitk<2>(s, gs, a, b, epi, flip);
        if (st2 == SB_OK) g_last_gemm_impl = SB_GEMM_TCGEN05;
        if (st2 != SB_ERR_UNSUPPORTED) return st2;
      }
    }
  }
  // C^T = B^T A^T: use the orientation that wastes fewer padded tile elements
  // (ties: keep N as the unit-stride index of C so rows are stored as full lines).
  GemmProblem g = g0;
  const long long w0 = padded_work(g.M, g.N), w1 = padded_work(g.N, g.M);
  // With fused epilogue work the rows of C have to be the stored lines.
  const bool swap = epi ? g.sCn != 1 && g.sCm == 1 : (w1 < w0) || (w1 == w0 && g.sCn != 1 && g.sCm == 1);
  if (swap) transpose_problem(&g);
  const int bn = pick_bn(g.M, g.N, g.batch);
  // Large single-batch problems go to the paired-CTA kernel (256 x 256 tiles) when enough of its
  // clusters fit on the device and there are enough tiles to keep them busy.
  if (bn == 256 && g.batch == 1 && g.M >= 256 && g.N >= 256 && g.K >= 256 && pair_enabled()) {
    const int clusters = pair_clusters();
    const long long tiles2 = ((g.M + 255) / 256) * ((g.N + 255) / 256);
    if (clusters >= 32 && tiles2 * 2 >= clusters) {
      if (!make_operand_map(g.A, g.M, g.K, g.batch, g.sAm, g.sAk, g.sAb, kBM, &a, &why))
        return fail(SB_ERR_ALIGNMENT, "tcgen05 contraction, operand A: " + why);
      if (!make_operand_map(g.B, g.N, g.K, g.batch, g.sBn, g.sBk, g.sBb, 128, &b, &why))
        return fail(SB_ERR_ALIGNMENT, "tcgen05 contraction, operand B: " + why);
      const int st2 = launch_tc_pair(s, g, a, b, clusters, epi, swap);
      if (st2 == SB_OK) g_last_gemm_impl = SB_GEMM_TCGEN05;
      return st2;
    }
  }
  if (epi) return fail(SB_ERR_UNSUPPORTED, "fused epilogue: only the paired-CTA kernel (large single-batch problems) has it");
  // Few output tiles and a long K: several CTA pairs per tile share K and add their partials up inside the
  // cluster.  Every cluster must be resident at once (a second round would double the time): on a B200, 22 clusters
  // of six CTAs are, 15 of eight, 33 of four.
  if (bn == 256 && g.batch == 1 && g.M >= 256 && g.N >= 256 && pair_enabled() && pair_splitk_forced() != 0) {
    const long long tiles2 = ((g.M + 255) / 256) * ((g.N + 255) / 256);
    const long long KT = (g.K + kBK - 1) / kBK;
    const bool c_ok = g.sCn == 1 && g.N % 4 == 0 && g.sCm % 4 == 0 && (reinterpret_cast<uintptr_t>(g.C) & 7u) == 0;
    int sk = 0;
    if (c_ok && tiles2 * 4 <= sm_count()) {
      for (int cand : {4, 3, 2}) {
        if (pair_splitk_forced() > 0 && cand != pair_splitk_forced()) continue;
        const int resident = cand == 4 ? splitk_clusters_resident<4>() : cand == 3 ? splitk_clusters_resident<3>()
                                                                                   : splitk_clusters_resident<2>();
        if (KT >= 8 * cand && tiles2 * 2 * cand <= sm_count() && resident >= tiles2) {
          sk = cand;
          break;
        }
      }
    }
    if (sk && make_operand_map(g.A, g.M, g.K, g.batch, g.sAm, g.sAk, g.sAb, kBM, &a, &why) &&
        make_operand_map(g.B, g.N, g.K, g.batch, g.sBn, g.sBk, g.sBb, 128, &b, &why)) {
      const int st2 = sk == 4 ? launch_tc_pair_splitk<4>(s, g, a, b)
                              : sk == 3 ? launch_tc_pair_splitk<3>(s, g, a, b) : launch_tc_pair_splitk<2>(s, g, a, b);
      if (st2 == SB_OK) g_last_gemm_impl = SB_GEMM_TCGEN05;
      return st2;
    }
  }
  if (!make_operand_map(g.A, g.M, g.K, g.batch, g.sAm, g.sAk, g.sAb, kBM, &a, &why))
    return fail(SB_ERR_ALIGNMENT, "tcgen05 contraction, operand A: " + why);
  if (!make_operand_map(g.B, g.N, g.K, g.batch, g.sBn, g.sBk, g.sBb, bn, &b, &why))
    return fail(SB_ERR_ALIGNMENT, "tcgen05 contraction, operand B: " + why);
  int st;
  if (bn == 256) st = launch_tc<256, 1>(s, g, a, b, ws, ws_bytes);
  else if (bn == 128) st = launch_tc<128, 2>(s, g, a, b, ws, ws_bytes);
  else st = launch_tc<64, 2>(s, g, a, b, ws, ws_bytes);
  if (st == SB_OK) g_last_gemm_impl = SB_GEMM_TCGEN05;
  return st;
}

int launch_gemm_tcgen05(cudaStream_t s, const GemmProblem& g, void* ws, size_t ws_bytes) {
  return launch_gemm_tcgen05_epi(s, g, ws, ws_bytes, nullptr);
}

int run_gemm_fused(cudaStream_t s, const GemmProblem& g, const GemmEpilogue& epi) {
  return launch_gemm_tcgen05_epi(s, g, nullptr, 0, &epi);
}

int run_gemm(cudaStream_t s, const GemmProblem& g, int impl, void* ws, size_t ws_bytes) {
  if (impl == SB_GEMM_SIMT) return launch_gemm_simt(s, g);
  if (impl == SB_GEMM_TCGEN05) return launch_gemm_tcgen05(s, g, ws, ws_bytes);
  if (impl != SB_GEMM_AUTO) return fail(SB_ERR_ARG, "einsum: unknown implementation selector");
  const int st = launch_gemm_tcgen05(s, g, ws, ws_bytes);
  if (st == SB_ERR_UNSUPPORTED || st == SB_ERR_ALIGNMENT) return launch_gemm_simt(s, g);
  return st;
}

void set_gemm_sm_budget(int n) { g_sm_budget = n; }
int gemm_sm_budget() { return g_sm_budget; }

namespace {

bool dense_scores(const View4& v, const Dims4& d) {
  return v.sK == 1 && v.sJ == d.K && v.sB == (long long)d.J * d.K && (d.H == 1 || v.sH == (long long)d.B * d.J * d.K) &&
         (reinterpret_cast<uintptr_t>(v.p) & 15u) == 0;
}

// Shared launcher: operands a [P,H,B,rows] (queries / DGAMMA) and b [P,H,B,rows] (keys / values).
template <bool BWD>
int launch_attn_scores(cudaStream_t s, Dims4 d, int P, const void* a_ptr, long long aP, long long aH, long long aB,
                       long long aJ, const void* b_ptr, long long bP, long long bH, long long bB, long long bJ,
                       void* o0, void* o1, void* o2, const void* alpha_in, const void* mask_in, attn::Params p) {
  std::call_once(g_encode_once, load_encode);
  if (!g_encode) return fail(SB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const int L = d.K;
  if (P != 64 || d.J != d.K || L % 64 != 0 || L > attn::kMaxL)
    return fail(SB_ERR_UNSUPPORTED, "fused attention scores need head size 64 and a sequence length that is a multiple of 64, at most 512");
  if ((d.H > 1 && d.B > 1) && (aH != aB * d.B || bH != bB * d.B))
    return fail(SB_ERR_UNSUPPORTED, "fused attention scores: head and sample dims of the projections do not collapse");
  const long long batch = (long long)d.H * d.B;
  const long long sAb = d.B > 1 ? aB : aH, sBb = d.B > 1 ? bB : bH;
  std::string why;
  OperandMap a, b;
  if (!make_operand_map(a_ptr, L, P, batch, aJ, aP, sAb, kBM, &a, &why))
    return fail(SB_ERR_UNSUPPORTED, "fused attention scores, first operand: " + why);
  const int brows = std::min(256, L);
  if (!make_operand_map(b_ptr, L, P, batch, bJ, bP, sBb, brows, &b, &why))
    return fail(SB_ERR_UNSUPPORTED, "fused attention scores, second operand: " + why);
  CUtensorMap m0, m1, m2, mi, mm;
  memset(&m0, 0, sizeof(m0));
  memset(&m2, 0, sizeof(m2));
  memset(&mi, 0, sizeof(mi));
  memset(&mm, 0, sizeof(mm));
  int sw0 = 0, sw1 = 0, sw2 = 0, swi = 0, swm = 0;
  // o0 (BETA forward, DATTN_DROP backward) may be absent: the kernel then never stores it
  if ((o0 && !encode_map(o0, (cuuint64_t)L, (cuuint64_t)L, (cuuint64_t)batch, L, (long long)L * L, 64, 32, &m0, &sw0, &why)) ||
      !encode_map(o1, (cuuint64_t)L, (cuuint64_t)L, (cuuint64_t)batch, L, (long long)L * L, 64, 32, &m1, &sw1, &why) ||
      (o2 && !encode_map(o2, (cuuint64_t)L, (cuuint64_t)L, (cuuint64_t)batch, L, (long long)L * L, 64, 32, &m2, &sw2, &why)))
    return fail(SB_ERR_UNSUPPORTED, "fused attention scores, output: " + why);
  if ((alpha_in && !encode_map(alpha_in, (cuuint64_t)L, (cuuint64_t)L, (cuuint64_t)batch, L, (long long)L * L, 64, 32, &mi, &swi, &why)) ||
      (mask_in && !encode_map(mask_in, (cuuint64_t)L, (cuuint64_t)L, (cuuint64_t)batch, L, (long long)L * L, 64, 32, &mm, &swm, &why, true)))
    return fail(SB_ERR_UNSUPPORTED, "fused attention scores, row inputs: " + why);
  // measured: the L2 prefetch of the next tile's mask rows helps the forward kernel; in the backward kernel the
  // extra requests (ALPHA too) queue in front of the slot fetches and cost more than they save
  p.prefetch = BWD ? 0 : 1;
  p.L = L;
  p.tiles_j = (L + 127) / 128;
  if ((long long)p.tiles_j * batch > 0x7fffffffLL) return fail(SB_ERR_UNSUPPORTED, "fused attention scores: too many tiles");
  p.tiles = (int)(p.tiles_j * batch);
  p.a_mn = a.mn; p.b_mn = b.mn; p.a_swap = a.swap; p.b_swap = b.swap;
  p.swap_o = sw1;      // every score tensor has the same geometry
  p.skip_o0 = o0 ? 0 : 1;
  p.b_bytes = b.mn ? L * 128 : ((L + 255) / 256) * brows * 128;
  constexpr int smem = attn::Cfg<BWD>::kSmemBytes;
  static_assert(smem <= 232448, "shared memory of the fused attention kernel");
  SB_CUDA_OK(ensure_dynamic_smem(reinterpret_cast<const void*>(attn::attn_scores_kernel<BWD>), smem));
  const unsigned grid = (unsigned)std::min<long long>(p.tiles, sm_count());
  SB_LAUNCH_OK(launch_k(attn::attn_scores_kernel<BWD>, grid, attn::kThreads, smem, s, a.map, b.map, m0, m1, m2, mi, mm, p));
  return SB_OK;
}

}  // namespace

int launch_attn_scores_fwd(cudaStream_t s, Dims4 d, int P, View4 qq, View4 kk, View4 beta, View4 alpha, View4 mask,
                           View4 drop, float scale, Rng rng) {
  if ((long long)d.H * d.B * d.J == 0) return SB_OK;
  if ((beta.p && !dense_scores(beta, d)) || !dense_scores(alpha, d) || !dense_scores(drop, d) || !dense_scores(mask, d))
    return fail(SB_ERR_UNSUPPORTED, "fused attention scores need score tensors dense as [H,B,J,K]");
  if (!(scale > 0.f)) return fail(SB_ERR_UNSUPPORTED, "fused attention scores need a positive scale");
  attn::Params p{};
  p.scale = scale;
  p.rng = rng;
  p.mask = reinterpret_cast<uint8_t*>(mask.p);
  // projections arrive as [P,H,B,rows] views: sH/sB/sJ/sK of the View4 hold the P,H,B,row strides
  return launch_attn_scores<false>(s, d, P, qq.p, qq.sH, qq.sB, qq.sJ, qq.sK, kk.p, kk.sH, kk.sB, kk.sJ, kk.sK, beta.p,
                                   alpha.p, drop.p, nullptr, rng.philox ? nullptr : mask.p, p);
}

int launch_attn_scores_bwd(cudaStream_t s, Dims4 d, int P, View4 dgamma, View4 vv, View4 alpha, View4 mask,
                           View4 dattn_drop, View4 dbeta) {
  if ((long long)d.H * d.B * d.J == 0) return SB_OK;
  if (!dense_scores(alpha, d) || (dattn_drop.p && !dense_scores(dattn_drop, d)) || !dense_scores(dbeta, d) || !dense_scores(mask, d))
    return fail(SB_ERR_UNSUPPORTED, "fused attention scores need score tensors dense as [H,B,J,K]");
  attn::Params p{};
  p.scale = 1.f;
  p.mask = reinterpret_cast<uint8_t*>(mask.p);
  return launch_attn_scores<true>(s, d, P, dgamma.p, dgamma.sH, dgamma.sB, dgamma.sJ, dgamma.sK, vv.p, vv.sH, vv.sB,
                                  vv.sJ, vv.sK, dattn_drop.p, dbeta.p, nullptr, alpha.p, mask.p, p);
}

int launch_score_contract(cudaStream_t s, Dims4 d, int P, View4 scores, const View4* x, const View4* out_r, const View4* y,
                          const View4* out_c, float alpha) {
  if ((long long)d.H * d.B * d.J == 0) return SB_OK;
  if (!x && !y) return SB_OK;
  std::call_once(g_encode_once, load_encode);
  if (!g_encode) return fail(SB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const int L = d.K;
  if (P != 64 || d.J != d.K || L % 128 != 0 || L > 512)
    return fail(SB_ERR_UNSUPPORTED, "score contractions need head size 64 and a sequence length that is a multiple of 128, at most 512");
  if (!dense_scores(scores, d)) return fail(SB_ERR_UNSUPPORTED, "score contractions need the score tensor dense as [H,B,J,K]");
  const long long batch = (long long)d.H * d.B;
  if (batch > 0x7fffffffLL) return fail(SB_ERR_UNSUPPORTED, "score contractions: too many (head, sample) pairs");
  // projections are [P,H,B,rows] views: sH/sB/sJ/sK of the View4 hold the (P,H,B,row) strides
  auto unit_stride = [&](const View4& v, long long* su) {
    if (d.H > 1 && d.B > 1 && v.sB != v.sJ * d.B) return false;
    *su = d.B > 1 ? v.sJ : v.sB;
    return true;
  };
  scon::Params p{};
  p.L = L; p.nt = L / 128; p.units = (int)batch; p.alpha = alpha;
  p.has_r = x ? 1 : 0; p.has_c = y ? 1 : 0;
  std::string why;
  CUtensorMap ms, mx, my;
  memset(&mx, 0, sizeof(mx));
  memset(&my, 0, sizeof(my));
  if (!encode_map(scores.p, (cuuint64_t)L, (cuuint64_t)L, (cuuint64_t)batch, L, (long long)L * L, 64, 128, &ms, &p.s_swap, &why))
    return fail(SB_ERR_UNSUPPORTED, "score contractions, scores: " + why);
  long long su = 0;
  if (x) {
    OperandMap m;
    if (!unit_stride(*x, &su) || !make_operand_map(x->p, 64, L, batch, x->sH, x->sK, su, 64, &m, &why))
      return fail(SB_ERR_UNSUPPORTED, "score contractions, row operand: " + why);
    mx = m.map; p.x_mn = m.mn; p.x_swap = m.swap;
    if (!unit_stride(*out_r, &su)) return fail(SB_ERR_UNSUPPORTED, "score contractions: head and sample dims of the row output do not collapse");
    p.out_r = reinterpret_cast<sb_half*>(out_r->p); p.r_sU = su; p.r_sRow = out_r->sK; p.r_sP = out_r->sH;
  }
  if (y) {
    OperandMap m;
    if (!unit_stride(*y, &su) || !make_operand_map(y->p, 64, L, batch, y->sH, y->sK, su, 64, &m, &why))
      return fail(SB_ERR_UNSUPPORTED, "score contractions, column operand: " + why);
    my = m.map; p.y_mn = m.mn; p.y_swap = m.swap;
    if (!unit_stride(*out_c, &su)) return fail(SB_ERR_UNSUPPORTED, "score contractions: head and sample dims of the column output do not collapse");
    p.out_c = reinterpret_cast<sb_half*>(out_c->p); p.c_sU = su; p.c_sRow = out_c->sK; p.c_sP = out_c->sH;
  }
  // two sets of projections and column accumulators when they fit (L <= 256): the next (head, sample) loads
  // while this one computes, which is what matters when a unit is only one or four tiles long
  p.nbuf = L <= 256 ? 2 : 1;
  const int proj = p.nbuf * (p.has_r + p.has_c) * L * 128;
  p.nstages = std::min(scon::kMaxStages, (232448 - 1280 - proj) / scon::kStageBytes);
  const int smem = proj + p.nstages * scon::kStageBytes + 1024 + 256;
  SB_CUDA_OK(ensure_dynamic_smem(reinterpret_cast<const void*>(scon::score_contract_kernel), 232448));
  const unsigned grid = (unsigned)std::min<long long>(batch, sm_count());
  SB_LAUNCH_OK(launch_k(scon::score_contract_kernel, grid, kTcThreads, smem, s, ms, mx, my, p));
  return SB_OK;
}

namespace {

// [P,H,B,rows] projection (View4 fields hold the P,H,B,row strides): rows of units h * B + b, sU apart if they collapse.
struct UnitView { long long sP, sH, sB, sU, sRow; bool collapses; };
UnitView unit_view(const View4& v, int H, int B) {
  UnitView o;
  o.sP = v.sH; o.sH = v.sB; o.sB = v.sJ; o.sRow = v.sK;
  o.collapses = H == 1 || B == 1 || v.sB == v.sJ * B;
  o.sU = B > 1 ? v.sJ : v.sB;
  return o;
}
// Tensor map of a projection the flash kernels read in 64 x 64 boxes: `jc` when the rows are the unit-stride index.
bool flash_map(const void* ptr, const UnitView& v, int units, int L, CUtensorMap* map, int* jc, int* swap, std::string* why) {
  OperandMap m;
  if (!make_operand_map(ptr, L, 64, units, v.sRow, v.sP, v.sU, 64, &m, why)) return false;
  *map = m.map; *jc = m.mn; *swap = m.swap;
  return true;
}
long long pad8(long long n) { return (n + 7) / 8 * 8; }
size_t align256(size_t n) { return (n + 255) / 256 * 256; }
// what a padded copy looks like
void padded_view(UnitView* v, int units, int L) {
  v->sRow = 1; v->sU = pad8(L); v->sP = v->sU * units;
}

}  // namespace

// The rows are the projections' unit-stride index and units are not 16 bytes apart, or not in one sequence: the kernels
// read a padded copy.
bool flash_padded(const View4& v, int H, int B, int L) {
  return v.sK == 1 && v.sH != 1 && (L % 8 != 0 || !unit_view(v, H, B).collapses);
}

int flash_supported(int H, int B, int L, int P, View4 proj, View4 dgamma) {
  for (const View4* v : {&proj, &dgamma}) {
    if (v->sH != 1 && v->sK != 1) return SB_ERR_UNSUPPORTED;
    if (v->sH == 1 && (((v->sK | v->sJ | v->sB) & 7) || !unit_view(*v, H, B).collapses)) return SB_ERR_UNSUPPORTED;
  }
  // (rows beyond 2048 are refused by the operators of a pass that keeps its scores; a pass that is looked at and one that is
  // not accept the same calls)
  if (P != 64 || L < 1 || L > 2048 || (long long)H * B * ((L + 31) / 32) > 0x3fffffffLL) return SB_ERR_UNSUPPORTED;
  return SB_OK;
}

void flash_scratch(int H, int B, int L, bool pad_proj, bool pad_dgamma, FlashScratch* f) {
  const size_t units = (size_t)H * B, nb = (L + 127) / 128;
  f->bits = align256(units * L * sizeof(float));
  f->pad = f->bits + align256(units * nb * L * 16);
  f->fwd_bytes = f->pad + (pad_proj ? align256(192 * units * pad8(L) * 2) : 0);
  f->dpad = align256(units * L * sizeof(float));
  f->bwd_bytes = f->dpad + (pad_dgamma ? align256(64 * units * pad8(L) * 2) : 0);
}

int launch_flash_fwd(cudaStream_t s, int H, int B, int L, const void* kqv, long long slice, View4 proj, void* gamma, View4 gv,
                     const void* mask, float scale, Rng rng, void* scratch, bool keep, bool relu) {
  std::call_once(g_encode_once, load_encode);
  if (!g_encode) return fail(SB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const int units = H * B;
  FlashScratch f;
  const bool pad = flash_padded(proj, H, B, L);
  flash_scratch(H, B, L, pad, false, &f);
  char* sc = reinterpret_cast<char*>(scratch);
  UnitView v = unit_view(proj, H, B);
  const UnitView o = unit_view(gv, H, B);
  const sb_half* base = reinterpret_cast<const sb_half*>(kqv);
  if (pad) {
    sb_half* dst = reinterpret_cast<sb_half*>(sc + f.pad);
    const unsigned grid = (unsigned)std::min<long long>((192ll * units + 7) / 8, (long long)sm_count() * 8);
    SB_LAUNCH_OK(launch_k(flash::pad_projections_kernel, grid, 256, 0, s, base, slice, v.sP, v.sH, v.sB, B, dst, units, L, (int)pad8(L)));
    base = dst;
    padded_view(&v, units, L);
    slice = 64 * v.sP;
  }
  flash::FwdParams p;
  memset(&p, 0, sizeof(p));
  std::string why;
  CUtensorMap mk, mq, mv;
  if (!flash_map(base, v, units, L, &mk, &p.jc, &p.k_swap, &why) || !flash_map(base + slice, v, units, L, &mq, &p.jc, &p.q_swap, &why) ||
      !flash_map(base + 2 * slice, v, units, L, &mv, &p.jc, &p.v_swap, &why))
    return fail(SB_ERR_UNSUPPORTED, "attention, projections: " + why);
  p.L = L; p.nb = (L + 127) / 128; p.items = units * p.nb;
  // ReLU layers over few tokens round ALPHA as passes that keep it do, at the price of a second look at the keys (0.5 to 1 us).
  // This is agreement with those passes and not accuracy: against float64 both forms are alike (Y, DX and the gradients of
  // WO, WKQV and LINW1, means over ten seeds at 16 to 1024 tokens: 0.95 to 1.20 of one sweep's error in ReLU layers, 1.00 to
  // 1.04 with GELU).  But where ReLU's sign hangs on how attention rounded, whole elements of a gradient move, and few tokens
  // do not average them out: at B=2, L=128 a step's gradients are within 6e-3 of a keeping pass with two sweeps and
  // within 1e-2 with one, single elements 0.9 and 1.1 times the root mean square apart; at 1024 tokens 0.36 and 0.53.  GELU
  // has no such step.  With and without gradients the form is the same, so that both have the same bits.
  p.sweeps = relu && (long long)B * L <= 1024 ? 2 : 1;
  p.c2 = scale * 1.4426950408889634f;
  p.rng = rng;
  p.mask = reinterpret_cast<const uint8_t*>(mask);
  if (keep) { p.lse = reinterpret_cast<float*>(sc); p.bits = reinterpret_cast<uint4*>(sc + f.bits); }
  p.out = reinterpret_cast<sb_half*>(gamma);
  p.B = B;
  p.o_sH = o.sH; p.o_sB = o.sB; p.o_sRow = o.sRow; p.o_sP = o.sP;
  const bool none = rng.philox && rng.thr == 0;
  auto kernel = none ? flash::flash_fwd_kernel<flash::kNoDrop>
                     : rng.philox && L % 8 == 0 ? flash::flash_fwd_kernel<flash::kPhilox> : flash::flash_fwd_kernel<flash::kAnyMask>;
  SB_CUDA_OK(ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), flash::kFwdSmem));
  // Two CTAs per SM, but the machine may place one on each SM first: within a budget there is one for every SM of it.
  const unsigned grid = (unsigned)std::min<long long>(p.items, sm_count() < device_sms() ? sm_count() : 2 * sm_count());
  SB_LAUNCH_OK(launch_k(kernel, grid, flash::kFwdThreads, flash::kFwdSmem, s, mq, mk, mv, p));
  return SB_OK;
}

int launch_flash_bwd(cudaStream_t s, int H, int B, int L, const void* kqv, long long slice, View4 proj, const void* gamma, View4 gv,
                     const void* dgamma, View4 dgv, void* dkqv, long long dslice, View4 dproj, float scale, const void* fwd_scratch,
                     void* bwd_scratch) {
  std::call_once(g_encode_once, load_encode);
  if (!g_encode) return fail(SB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const int units = H * B;
  FlashScratch f;
  const bool pad = flash_padded(proj, H, B, L), dpad = flash_padded(dgv, H, B, L);
  flash_scratch(H, B, L, pad, dpad, &f);
  const char* fs = reinterpret_cast<const char*>(fwd_scratch);
  char* bs = reinterpret_cast<char*>(bwd_scratch);
  UnitView v = unit_view(proj, H, B), g = unit_view(dgv, H, B);
  const UnitView o = unit_view(gv, H, B), d = unit_view(dproj, H, B);
  const sb_half* base = reinterpret_cast<const sb_half*>(kqv);
  if (pad) {
    base = reinterpret_cast<const sb_half*>(fs + f.pad);
    padded_view(&v, units, L);
    slice = 64 * v.sP;
  }
  flash::DsumParams q;
  memset(&q, 0, sizeof(q));
  q.g = reinterpret_cast<const sb_half*>(dgamma); q.g_sP = g.sP; q.g_sH = g.sH; q.g_sB = g.sB; q.g_sRow = g.sRow;
  q.o = reinterpret_cast<const sb_half*>(gamma); q.o_sP = o.sP; q.o_sH = o.sH; q.o_sB = o.sB; q.o_sRow = o.sRow;
  q.dsum = reinterpret_cast<float*>(bs);
  q.pad = dpad ? reinterpret_cast<sb_half*>(bs + f.dpad) : nullptr;
  q.units = units; q.B = B; q.L = L; q.Lp = (int)pad8(L);
  auto rows_of_eight = [&](const void* ptr, const UnitView& w) {
    return w.sRow == 1 && !((w.sP | w.sH | w.sB) & 7) && !(reinterpret_cast<uintptr_t>(ptr) & 15u);
  };
  const bool vec = L % 8 == 0 && !dpad && rows_of_eight(dgamma, g) && rows_of_eight(gamma, o);
  q.blocks_j = vec ? (L + 127) / 128 : (L + 31) / 32;
  SB_LAUNCH_OK(launch_k(vec ? flash::dsum_vec_kernel : flash::dsum_kernel, (unsigned)((long long)units * q.blocks_j), 256, 0, s, q));
  const void* gptr = dgamma;
  if (dpad) {
    gptr = q.pad;
    padded_view(&g, units, L);
  }
  flash::BwdParams p;
  memset(&p, 0, sizeof(p));
  std::string why;
  CUtensorMap mk, mq, mv, mg;
  if (!flash_map(base, v, units, L, &mk, &p.jc, &p.k_swap, &why) || !flash_map(base + slice, v, units, L, &mq, &p.jc, &p.q_swap, &why) ||
      !flash_map(base + 2 * slice, v, units, L, &mv, &p.jc, &p.v_swap, &why) || !flash_map(gptr, g, units, L, &mg, &p.g_jc, &p.g_swap, &why))
    return fail(SB_ERR_UNSUPPORTED, "attention backward, operands: " + why);
  p.L = L; p.nb = (L + 127) / 128; p.units = units;
  p.both = p.nb == 1 ? 1 : 0;
  p.first_q = units * p.nb;
  p.items = p.both ? p.first_q : 2 * p.first_q;
  p.scale = scale;
  p.c2 = scale * 1.4426950408889634f;
  p.lse = reinterpret_cast<const float*>(fs);
  p.bits = reinterpret_cast<const uint4*>(fs + f.bits);
  p.dsum = q.dsum;
  sb_half* dk = reinterpret_cast<sb_half*>(dkqv);
  p.dk = dk; p.dq = dk + dslice; p.dv = dk + 2 * dslice;
  p.B = B;
  p.d_sH = d.sH; p.d_sB = d.sB; p.d_sRow = d.sRow; p.d_sP = d.sP;
  static_assert(flash::kBwdSmem <= 232448, "shared memory of the attention backward kernel");
  SB_CUDA_OK(ensure_dynamic_smem(reinterpret_cast<const void*>(flash::flash_bwd_kernel), flash::kBwdSmem));
  const unsigned grid = (unsigned)std::min<long long>(p.items, sm_count());
  SB_LAUNCH_OK(launch_k(flash::flash_bwd_kernel, grid, flash::kBwdThreads, flash::kBwdSmem, s, mq, mk, mv, mg, p));
  return SB_OK;
}

int gemm_device_error(cudaStream_t s, int* code) {
  int v = 0;
  SB_CUDA_OK(cudaMemcpyFromSymbolAsync(&v, g_tc_error, sizeof(int), 0, cudaMemcpyDeviceToHost, s));
  SB_CUDA_OK(cudaStreamSynchronize(s));
  *code = v;
  return SB_OK;
}

int run_mma_peak_probe(cudaStream_t s, int k_blocks, int bf16, double* flops) {
  if (k_blocks < 1 || k_blocks > (1 << 24)) return fail(SB_ERR_ARG, "peak probe: K-block count out of range");
  const int clusters = std::min(pair_clusters(), sm_count() / 2);
  if (clusters < 1) return fail(SB_ERR_UNSUPPORTED, "peak probe: no cluster of two CTAs fits on this device");
  SB_CUDA_OK(ensure_dynamic_smem(reinterpret_cast<const void*>(probe::mma_peak_kernel), probe::kSmemBytes));
  SB_LAUNCH_OK(launch_k(probe::mma_peak_kernel, 2 * clusters, probe::kThreads, probe::kSmemBytes, s, k_blocks, bf16 ? 1 : 0));
  SB_CUDA_OK(cudaGetLastError());
  if (flops) *flops = (double)clusters * k_blocks * 4.0 * 2.0 * 256.0 * 256.0 * 16.0;
  return SB_OK;
}

int gemm_device_error_reset(cudaStream_t s) {
  const int zero = 0;
  SB_CUDA_OK(cudaStreamSynchronize(s));
  SB_CUDA_OK(cudaMemcpyToSymbol(g_tc_error, &zero, sizeof(int), 0, cudaMemcpyHostToDevice));
  return SB_OK;
}

}  // namespace sb

// K2 (tensor cores) — TMA-fed tcgen05 GEMM with the accumulator in TMEM, kind::tf32.
//
//   C (M×N, column-major) = Σ_p  A_p ᵀ · B_p      over 1 or 3 operand pairs p
//
// Both operands are K-major (the contraction index contiguous), which is the layout the
// contraction planner produces with the permutation kernel.  Precision modes:
//   * TF32      — one pass (A, B), FP32 accumulation;
//   * 3×TF32    — three passes A_hi·B_hi + (A_hi·B_lo + A_lo·B_hi), where x_hi is x
//                 rounded to nearest TF32 and x_lo = x − x_hi exactly; the hi·hi pass and
//                 the two small correction passes accumulate in separate TMEM
//                 accumulators (the corrections would otherwise be lost to the large
//                 accumulator's alignment) and are summed in the epilogue: FP32-grade
//                 products from the TF32 tensor pipe.
// Complex operands use the real 4M form as one real GEMM of twice the size:
//   [Re C; Im C] = [[Ar, −Ai], [Ai, Ar]] · [Br; Bi]
// built by a prep kernel that also does the hi/lo split, with an epilogue that writes the
// two row blocks back as interleaved complex.
//
// CTA (128 threads) per 128×256 output tile, tiles visited in bands of 8 row tiles so
// the resident CTAs share their operand panels in L2.  Thread 0 issues TMA loads
// (128-byte swizzle, 4-stage ring of 48 KB stages with full/empty mbarriers), thread 32
// issues tcgen05.mma (M=128, N=256, K=8 per instruction; accumulator = 256 TMEM
// columns) and commits each stage back to its empty barrier; all four warps then drain
// TMEM with tcgen05.ld (warp w owns accumulator rows 32w…32w+31).  Every mbarrier wait is bounded: on timeout the kernel records an error
// word, skips the remaining work, and still releases its TMEM.
#include <cuda.h>

#include <algorithm>
#include <cstring>

#include "tn_internal.cuh"

namespace {

constexpr int BM = 128, BN = 256, BKB = 128;  // tile: 128×256 outputs, 128 bytes of K
constexpr int STAGES = 4;
constexpr int A_BYTES = BM * BKB, B_BYTES = BN * BKB;
constexpr int SMEM_BYTES = STAGES * (A_BYTES + B_BYTES) + 1024 /*align*/ + 256 /*barriers*/;
constexpr long long kSpinLimit = 1ll << 28;
constexpr int kGroupM = 8;

struct Maps {
  CUtensorMap a[2];  // A_hi, A_lo
  CUtensorMap b[2];  // B_hi, B_lo
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait: false (and the error word set) if the phase never completes
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* err) {
  for (long long i = 0; i < kSpinLimit; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  atomicExch(err, 1);
  return false;
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
// shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1024 B apart
__device__ __forceinline__ uint64_t sdesc(const void* p) {
  const uint64_t addr = (uint64_t)smem_u32(p);
  uint64_t d = (addr & 0x3FFFFull) >> 4;  // start address
  d |= 1ull << 16;                        // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;       // stride byte offset: 8 rows × 128 B
  d |= 1ull << 46;                        // descriptor version for tcgen05
  d |= 2ull << 61;                        // 128-byte swizzle
  return d;
}
// instruction descriptor: D f32, A/B tf32, both K-major, N = BN, M = BM
constexpr uint32_t kIdescTF32 = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(BN >> 3) << 17) |
                                ((uint32_t)(BM >> 4) << 24);

__device__ __forceinline__ void mma_tf32(uint32_t dtmem, uint64_t a, uint64_t b, uint32_t accum) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n" ::"r"(
          dtmem),
      "l"(a), "l"(b), "r"(kIdescTF32), "r"(accum)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

template <int EPI>  // 0: real C (float); 1: complex interleaved from [Re; Im] row blocks
__global__ void __launch_bounds__(128, 1)
    k_gemm_tf32(const __grid_constant__ Maps maps, int passes, int M, int N, int K, float* __restrict__ C,
                int64_t ldc, int Mh, float alpha, float beta, int* err) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t base_u = smem_u32(smem_raw);
  unsigned char* smem = smem_raw + ((1024 - (base_u & 1023)) & 1023);
  unsigned char* sA = smem;
  unsigned char* sB = smem + STAGES * A_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * (A_BYTES + B_BYTES));
  uint64_t* full = bars;
  uint64_t* empty = bars + STAGES;
  uint64_t* done = bars + 2 * STAGES;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // grouped tile order: consecutive CTAs sweep the N tiles of a band of kGroupM row tiles,
  // so the CTAs resident at one time share their A and B panels in L2
  const int tiles_m = (M + BM - 1) / BM, tiles_n = (N + BN - 1) / BN;
  const int per_group = kGroupM * tiles_n;
  const int grp = (int)blockIdx.x / per_group, first_m = grp * kGroupM;
  const int gsize = min(kGroupM, tiles_m - first_m);
  const int in_grp = (int)blockIdx.x % per_group;
  const int m0 = (first_m + in_grp % gsize) * BM, n0 = (in_grp / gsize) * BN;
  const uint32_t tcols = passes > 1 ? 2 * BN : BN;  // hi·hi accumulator [+ corrections]
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(tcols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 32) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tslot;

  const int nk = (K + 31) / 32;  // 32 fp32 = 128 bytes of K per tile
  const int total = passes * nk;
  if (tid == 0) {
    // producer
    for (int t = 0; t < total; ++t) {
      const int s = t % STAGES;
      if (t >= STAGES && !mbar_wait(&empty[s], ((t / STAGES) & 1) ^ 1, err)) break;
      const int pass = t / nk, kt = t % nk;
      const CUtensorMap* am = &maps.a[pass == 2 ? 1 : 0];
      const CUtensorMap* bm = &maps.b[pass == 1 ? 1 : 0];
      mbar_expect_tx(&full[s], A_BYTES + B_BYTES);
      tma_load_2d(sA + s * A_BYTES, am, &full[s], kt * 32, m0);
      tma_load_2d(sB + s * B_BYTES, bm, &full[s], kt * 32, n0);
    }
  } else if (tid == 32) {
    // MMA issuer
    bool ok = true;
    for (int t = 0; t < total && ok; ++t) {
      const int s = t % STAGES;
      ok = mbar_wait(&full[s], (t / STAGES) & 1, err);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int pass = t / nk;
      const uint32_t acc = tmem + (pass > 0 ? (uint32_t)BN : 0u);  // corrections: their own accumulator
      const bool first = (t % nk == 0) && pass <= 1;
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {  // 4 × (K = 8 tf32 = 32 bytes)
        const uint64_t a = sdesc(sA + s * A_BYTES) + (uint64_t)((kk * 32) >> 4);
        const uint64_t b = sdesc(sB + s * B_BYTES) + (uint64_t)((kk * 32) >> 4);
        mma_tf32(acc, a, b, (first && kk == 0) ? 0u : 1u);
      }
      mma_commit(&empty[s]);
    }
    mma_commit(done);
  }
  __syncwarp();
  // epilogue: all 4 warps
  const bool ok = mbar_wait(done, 0, err);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (ok) {
    const int row = m0 + warp * 32 + lane;
#pragma unroll 1
    for (int c0 = 0; c0 < BN; c0 += 16) {
      uint32_t r[16];
      const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0;
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
          : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
            "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
          : "r"(taddr));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (passes > 1) {  // add the correction accumulator
        uint32_t q[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]), "=r"(q[4]), "=r"(q[5]), "=r"(q[6]), "=r"(q[7]),
              "=r"(q[8]), "=r"(q[9]), "=r"(q[10]), "=r"(q[11]), "=r"(q[12]), "=r"(q[13]), "=r"(q[14]), "=r"(q[15])
            : "r"(taddr + (uint32_t)BN));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(q[j]));
      }
      if (row < M) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int col = n0 + c0 + j;
          if (col >= N) break;
          float v = alpha * __uint_as_float(r[j]);
          float* dst;
          if (EPI == 0)
            dst = C + row + (int64_t)col * ldc;
          else
            dst = C + 2 * ((int64_t)(row % Mh) + (int64_t)col * ldc) + (row >= Mh ? 1 : 0);
          if (beta != 0.f) v += beta * *dst;
          *dst = v;
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tcols) : "memory");
}

// ---------------------------------------------------------------------------------
// tall complex products with a short contraction (k ≤ 64): C[m, n] = α Σ_k A[m, k]·B[k, n] + β C
//
// Bound: HBM.  The general path expands A fourfold (the 4M form's two row blocks, hi and lo)
// in a pass of its own and reads it back; for a lattice's boundary tensor (2²⁴ entries, k = n =
// 64) that is 1 GB beside the product's own 0.27 GB.  Here A is read once, through a strided
// view, and split on the way into shared memory; the real form doubles B's columns instead
// of A's rows:  [Re C | Im C] = [Re A | Im A] · [[Br, Bi], [−Bi, Br]].
// A CTA keeps its 64 columns of B (128 real ones, hi and lo, 128 KB) for all its row tiles.
// 8 producer warps load 128 rows × 16 k (four stages ahead in registers), split them and write
// the K-major 128-byte-swizzled tiles of a two-slot ring; one thread issues tcgen05.mma
// (M = 128, N = 128, K = 8: hi·hi in one TMEM accumulator, lo·hi and hi·lo in another, as the
// general kernel); 4 epilogue warps drain one pair of accumulators while the next fills.
// Every mbarrier wait is bounded (error word, the remaining work is skipped, TMEM released).
// ---------------------------------------------------------------------------------
constexpr int TALL_KT = 4;                       // K tiles of 16 complex (32 real) entries
constexpr int TALL_THREADS = 13 * 32;            // 8 producer, 4 epilogue, 1 issuing warp
constexpr int TALL_TILE = 128 * 128;             // bytes of a 128-row tile
constexpr int TALL_SMEM = 2 * TALL_KT * TALL_TILE + 2 * 2 * TALL_TILE + 1024 + 256;
constexpr long long kTallSpin = 1ll << 24;

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool tall_wait(uint64_t* bar, uint32_t parity, int* err);
// one lane waits for its warp, so that the warp's lanes go on or give up together
__device__ __forceinline__ bool tall_wait_warp(uint64_t* bar, uint32_t parity, int* err) {
  int ok = 1;
  if ((threadIdx.x & 31) == 0) ok = tall_wait(bar, parity, err);
  return __shfl_sync(0xffffffffu, ok, 0) != 0;
}
__device__ __forceinline__ bool tall_wait(uint64_t* bar, uint32_t parity, int* err) {
  for (long long i = 0; i < kTallSpin; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  atomicExch(err, 1);
  return false;
}
// x rounded to the nearest TF32 value, ties away from zero
__device__ __forceinline__ float to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}
// byte offset of element (row, j) of a K-major tile of 32 floats per row, 128-byte swizzle
__device__ __forceinline__ uint32_t tall_at(int row, int j) {
  return (uint32_t)((row >> 3) * 1024 + (row & 7) * 128 + ((j * 4) ^ ((row & 7) << 4)));
}
__device__ __forceinline__ int64_t view_offset(const IndexView& v, int64_t i) {
  if (v.outer == 0) return i * v.inner;
  const unsigned n = (unsigned)v.extent, q = (unsigned)i / n;
  return (int64_t)((unsigned)i - q * n) * v.inner + (int64_t)q * v.outer;
}
constexpr uint32_t kIdescTall = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(128 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
__device__ __forceinline__ void mma_tall(uint32_t d, uint64_t a, uint64_t b, uint32_t accum) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
               "l"(a), "l"(b), "r"(kIdescTall), "r"(accum)
               : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                 "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

// grid: (CTAs per column block, column blocks of 64)
__global__ void __launch_bounds__(TALL_THREADS, 1)
    k_gemm_tf32_tall(int64_t m, int64_t n, int k, int passes, const cxf* __restrict__ A, GemmView va, const cxf* __restrict__ B,
                     GemmView vb, float alpha, float beta, cxf* __restrict__ C, int64_t ldc, int* err) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ int64_t s_koff[16 * TALL_KT];
  const uint32_t base_u = smem_u32(smem_raw);
  unsigned char* smem = smem_raw + ((1024 - (base_u & 1023)) & 1023);
  unsigned char* sB = smem;                                    // hi: KT tiles, lo: KT tiles
  unsigned char* sA = smem + 2 * TALL_KT * TALL_TILE;          // 2 slots × (hi, lo)
  uint64_t* bars = reinterpret_cast<uint64_t*>(sA + 4 * TALL_TILE);
  uint64_t *full = bars, *empty = bars + 2, *tfull = bars + 4, *tempty = bars + 6;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 8);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t j0 = (int64_t)blockIdx.y * 64, tiles = (m + 127) / 128;
  const int KT = (k + 15) / 16;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 32) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&full[s], 8);
      mbar_init(&empty[s], 1);
      mbar_init(&tfull[s], 1);
      mbar_init(&tempty[s], 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int kk = tid; kk < k; kk += TALL_THREADS) s_koff[kk] = view_offset(va.col, kk);
  // B's real form, rows c (Re C) and 64 + c (Im C); K tile t holds Re then Im of entries 16t…16t+15
  for (int e = tid; e < KT * 16 * 64; e += TALL_THREADS) {
    const int c = e & 63, kk = e >> 6;
    cxf b = mkcx<float>(0.f, 0.f);
    if (kk < k && j0 + c < n) b = B[view_offset(vb.row, kk) + view_offset(vb.col, j0 + c)];
    if (vb.conj) b.y = -b.y;
    const float v[4] = {b.x, -b.y, b.y, b.x};  // (Re row, Re k), (Re row, Im k), (Im row, Re k), (Im row, Im k)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t at = (uint32_t)(kk >> 4) * TALL_TILE + tall_at(c + (q >> 1) * 64, (kk & 15) + (q & 1) * 16);
      const float h = to_tf32(v[q]);
      *reinterpret_cast<float*>(sB + at) = h;
      *reinterpret_cast<float*>(sB + TALL_KT * TALL_TILE + at) = v[q] - h;
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tslot;

  if (warp < 8) {
    // producers: thread = (row of the tile, 8 of the stage's 16 entries)
    const int row = tid & 127, hf = tid >> 7;
    const int64_t stages = tiles > (int64_t)blockIdx.x ? ((tiles - blockIdx.x + gridDim.x - 1) / gridDim.x) * KT : 0;
    cxf r[4][8];  // stages in flight
    int64_t ftile = blockIdx.x;  // the next stage to fetch: its tile, row pointer and K tile
    int fkt = 0;
    const cxf* fp = nullptr;
    auto fetch = [&](cxf* v) {
      if (fkt == 0) fp = ftile * 128 + row < m ? A + view_offset(va.row, ftile * 128 + row) : nullptr;
      const int k0 = fkt * 16 + hf * 8;
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = (fp && k0 + j < k) ? fp[s_koff[k0 + j]] : mkcx<float>(0.f, 0.f);
      if (++fkt == KT) {
        fkt = 0;
        ftile += gridDim.x;
      }
    };
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (u < stages) fetch(r[u]);
    bool ok = true;
    for (int64_t st = 0; st < stages && ok; st += 4) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (st + u >= stages) break;
        const int64_t g = st + u;
        const int slot = u & 1;  // g mod 2
        if (g >= 2 && !(ok = tall_wait_warp(&empty[slot], (uint32_t)(((g >> 1) & 1) ^ 1), err))) break;
        unsigned char* hi = sA + slot * 2 * TALL_TILE;
        unsigned char* lo = hi + TALL_TILE;
#pragma unroll
        for (int part = 0; part < 2; ++part)
#pragma unroll
          for (int q = 0; q < 8; q += 4) {
            float x[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) x[j] = part ? (va.conj ? -r[u][q + j].y : r[u][q + j].y) : r[u][q + j].x;
            const uint32_t at = tall_at(row, part * 16 + hf * 8 + q);
            const float4 h = make_float4(to_tf32(x[0]), to_tf32(x[1]), to_tf32(x[2]), to_tf32(x[3]));
            *reinterpret_cast<float4*>(hi + at) = h;
            if (passes > 1) *reinterpret_cast<float4*>(lo + at) = make_float4(x[0] - h.x, x[1] - h.y, x[2] - h.z, x[3] - h.w);
          }
        if (g + 4 < stages) fetch(r[u]);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[slot]);
      }
    }
  } else if (warp == 12) {
    if (lane == 0) {
      int64_t g = 0, it = 0;
      bool ok = true;
      for (int64_t tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, ++it) {
        const int ab = (int)(it & 1);
        if (it >= 2 && !(ok = tall_wait(&tempty[ab], (uint32_t)(((it >> 1) & 1) ^ 1), err))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d = tmem + (uint32_t)(ab * 256);
        for (int kt = 0; kt < KT; ++kt, ++g) {
          const int slot = (int)(g & 1);
          if (!(ok = tall_wait(&full[slot], (uint32_t)((g >> 1) & 1), err))) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t ah = sdesc(sA + slot * 2 * TALL_TILE), al = sdesc(sA + slot * 2 * TALL_TILE + TALL_TILE);
          const uint64_t bh = sdesc(sB + kt * TALL_TILE), bl = sdesc(sB + (TALL_KT + kt) * TALL_TILE);
#pragma unroll
          for (int q = 0; q < 4; ++q) mma_tall(d, ah + 2 * q, bh + 2 * q, (kt > 0 || q > 0) ? 1u : 0u);
          if (passes > 1) {
#pragma unroll
            for (int q = 0; q < 4; ++q) mma_tall(d + 128, al + 2 * q, bh + 2 * q, (kt > 0 || q > 0) ? 1u : 0u);
#pragma unroll
            for (int q = 0; q < 4; ++q) mma_tall(d + 128, ah + 2 * q, bl + 2 * q, 1u);
          }
          mma_commit(&empty[slot]);
        }
        if (ok) mma_commit(&tfull[ab]);
      }
    }
  } else {
    // epilogue: warps 8-11, TMEM lanes 32·(warp mod 4)…
    const uint32_t tl = (uint32_t)((warp & 3) * 32) << 16;
    int64_t it = 0;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++it) {
      const int ab = (int)(it & 1);
      if (!tall_wait_warp(&tfull[ab], (uint32_t)((it >> 1) & 1), err)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int64_t i = tile * 128 + (warp & 3) * 32 + lane;
      const uint32_t d = tmem + tl + (uint32_t)(ab * 256);
#pragma unroll 1
      for (int c0 = 0; c0 < 64; c0 += 16) {
        if (j0 + c0 >= n) break;
        float re[16], im[16];
        tmem_ld16(d + c0, re);
        tmem_ld16(d + 64 + c0, im);
        if (passes > 1) {
          float q[16];
          tmem_ld16(d + 128 + c0, q);
#pragma unroll
          for (int j = 0; j < 16; ++j) re[j] += q[j];
          tmem_ld16(d + 192 + c0, q);
#pragma unroll
          for (int j = 0; j < 16; ++j) im[j] += q[j];
        }
        if (i < m) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (j0 + c0 + j >= n) break;
            cxf* dst = C + i + (j0 + c0 + j) * ldc;
            cxf v = mkcx<float>(alpha * re[j], alpha * im[j]);
            if (beta != 0.f) {
              v.x += beta * dst->x;
              v.y += beta * dst->y;
            }
            *dst = v;
          }
        }
        __syncwarp();
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[ab]);
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

// ---------------------------------------------------------------------------------
// operand preparation: K-major real planes (hi, lo) with K padded to Kp (multiple of 32)
// ---------------------------------------------------------------------------------
// x rounded to the nearest TF32 value (10-bit mantissa, ties away from zero): the
// remainder x − hi is exact in FP32 and at most half a TF32 unit
__device__ __forceinline__ float tf32_hi(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

// element (r, c) of op(X) for a column-major complex X with leading dimension ld
__device__ __forceinline__ cxf ld_op(const cxf* X, int64_t ld, char op, int64_t r, int64_t c) {
  if (op == 'N') return X[r + c * ld];
  cxf v = X[c + r * ld];
  if (op == 'C') v.y = -v.y;
  return v;
}

// A' (rows i' < 2M, K-major, pitch Kp): i' < M → [Ar, −Ai], i' ≥ M → [Ai, Ar]
__global__ void k_prep_a_cx(int64_t M, int64_t K, int64_t Kp, const cxf* A, int64_t lda, char op, float* hi, float* lo) {
  const int64_t total = 2 * M * Kp;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t kp = t % Kp, ip = t / Kp;
    float v = 0.f;
    if (kp < 2 * K) {
      const int64_t i = ip % M, k = kp % K;
      const cxf a = ld_op(A, lda, op, i, k);
      const bool top = ip < M, left = kp < K;
      v = top ? (left ? a.x : -a.y) : (left ? a.y : a.x);
    }
    const float h = tf32_hi(v);
    hi[t] = h;
    if (lo) lo[t] = v - h;
  }
}
// A' for op(A) = A (M-major source): 32×32 tiles of A staged through shared memory so
// that both the reads (along i) and the K-major writes (along k) are coalesced; the four
// quadrants [Ar, −Ai; Ai, Ar] of the tile are written from the staged tile.  Columns
// kp ≥ 2K of A' (the padding) are written by k_prep_a_pad.
__global__ void __launch_bounds__(256) k_prep_a_cx_n(int64_t M, int64_t K, int64_t Kp, const cxf* __restrict__ A,
                                                     int64_t lda, float* __restrict__ hi, float* __restrict__ lo) {
  __shared__ cxf tile[32][33];
  const int64_t i0 = (int64_t)blockIdx.x * 32, k0 = (int64_t)blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 × 8
  for (int r = ty; r < 32; r += 8) {
    const int64_t i = i0 + tx, k = k0 + r;
    tile[r][tx] = (i < M && k < K) ? A[i + k * lda] : mkcx(0.f, 0.f);
  }
  __syncthreads();
  for (int r = ty; r < 32; r += 8) {
    const int64_t i = i0 + r, k = k0 + tx;
    if (i >= M || k >= K) continue;
    const cxf a = tile[tx][r];
    const float q[4] = {a.x, -a.y, a.y, a.x};  // (top,left) (top,right) (bottom,left) (bottom,right)
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int64_t ip = i + (u >= 2 ? M : 0), kp = k + ((u & 1) ? K : 0);
      const float v = q[u], h = tf32_hi(v);
      hi[ip * Kp + kp] = h;
      if (lo) lo[ip * Kp + kp] = v - h;
    }
  }
}
__global__ void k_prep_a_pad(int64_t M2, int64_t K2, int64_t Kp, float* hi, float* lo) {
  const int64_t w = Kp - K2, total = M2 * w;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t ip = t / w, kp = K2 + t % w;
    hi[ip * Kp + kp] = 0.f;
    if (lo) lo[ip * Kp + kp] = 0.f;
  }
}
// B' (columns j < N, K-major, pitch Kp): [Br; Bi]
__global__ void k_prep_b_cx(int64_t N, int64_t K, int64_t Kp, const cxf* B, int64_t ldb, char op, float* hi, float* lo) {
  const int64_t total = N * Kp;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t kp = t % Kp, j = t / Kp;
    float v = 0.f;
    if (kp < 2 * K) {
      const cxf b = ld_op(B, ldb, op, kp % K, j);
      v = kp < K ? b.x : b.y;
    }
    const float h = tf32_hi(v);
    hi[t] = h;
    if (lo) lo[t] = v - h;
  }
}
// real: A' (M rows, K-major) from op(A); B' (N columns, K-major) from op(B)
__global__ void k_prep_re(int64_t R, int64_t K, int64_t Kp, const float* X, int64_t ld, bool kmajor_src, float* hi,
                          float* lo) {
  const int64_t total = R * Kp;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t kp = t % Kp, r = t / Kp;
    float v = 0.f;
    if (kp < K) v = kmajor_src ? X[kp + r * ld] : X[r + kp * ld];
    const float h = tf32_hi(v);
    hi[t] = h;
    if (lo) lo[t] = v - h;
  }
}

EncodeTiledFn encode_fn(tn_ctx* ctx) { return tn_encode_tiled_fn(ctx); }

// K-major operand: rows × Kp floats, row pitch Kp·4 bytes; box 32 floats × box_rows
tn_status_t make_map(tn_ctx* ctx, CUtensorMap* map, const float* base, int64_t rows, int64_t Kp, uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn(ctx);
  if (!fn) return TN_ECUDA;
  cuuint64_t dims[2] = {(cuuint64_t)Kp, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(Kp * 4)};
  cuuint32_t box[2] = {32, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void*)base, dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return tn_set_error(ctx, TN_ECUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return TN_OK;
}

unsigned blocks_for(tn_ctx* ctx, int64_t n) {
  int64_t b = (n + 255) / 256;
  int64_t cap = (int64_t)ctx->num_sms * 16;
  return (unsigned)std::max<int64_t>(1, std::min(b, cap));
}

}  // namespace

// the driver's cuTensorMapEncodeTiled, looked up once through the runtime
EncodeTiledFn tn_encode_tiled_fn(tn_ctx* ctx) {
  static EncodeTiledFn fn = nullptr;
  if (fn) return fn;
  void* p = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess || !p) {
    tn_set_error(ctx, TN_ECUDA, "cuTensorMapEncodeTiled unavailable");
    return nullptr;
  }
  fn = (EncodeTiledFn)p;
  return fn;
}

// Workspace (bytes) for tc_gemm on the given shape.
// K-major operands are stored with K padded to a multiple of 4 floats (the 16-byte TMA
// pitch rule) and at least one 32-float box; the last box reads past K as zeros.
static inline int64_t padded_k(bool complex_in, int64_t k) {
  int64_t kk = complex_in ? 2 * k : k;
  kk = (kk + 3) / 4 * 4;
  return kk < 32 ? 32 : kk;
}

size_t tc_gemm_workspace(bool complex_in, int passes, int64_t m, int64_t n, int64_t k) {
  const int64_t Kp = padded_k(complex_in, k);
  const int64_t Ma = complex_in ? 2 * m : m;
  const int copies = passes > 1 ? 2 : 1;
  return copies * (ws_round(4 * (size_t)(Ma * Kp)) + ws_round(4 * (size_t)(n * Kp))) + ws_round(sizeof(int) * 4);
}

// C (m×n) = op(A)·op(B) on the TF32 tensor pipe (passes: 1 = TF32, 3 = 3×TF32).
// complex_in: A, B, C are interleaved complex (C64 data must be converted by the caller);
// otherwise real float.  beta applies to C (real).  Workspace reserved by the caller.
tn_status_t tc_gemm(tn_ctx* ctx, bool complex_in, int passes, char opa, char opb, int64_t m, int64_t n, int64_t k,
                    float alpha, const void* A, int64_t lda, const void* B, int64_t ldb, float beta, void* C, int64_t ldc) {
  if (m == 0 || n == 0) return TN_OK;
  const int64_t Kp = padded_k(complex_in, k);
  const int64_t Ma = complex_in ? 2 * m : m;
  if (Ma > (1ll << 31) - 128 || n > (1ll << 31) - 128) return tn_set_error(ctx, TN_EUNSUPPORTED, "tc_gemm: too large");
  const bool split = passes > 1;
  float* Ahi = ws_take<float>(ctx, (size_t)(Ma * Kp));
  float* Bhi = ws_take<float>(ctx, (size_t)(n * Kp));
  float* Alo = split ? ws_take<float>(ctx, (size_t)(Ma * Kp)) : nullptr;
  float* Blo = split ? ws_take<float>(ctx, (size_t)(n * Kp)) : nullptr;
  int* err = ws_take<int>(ctx, 4);
  TN_CHECK_CUDA(ctx, cudaMemsetAsync(err, 0, sizeof(int), ctx->stream));
  if (complex_in) {
    if (opa == 'N') {
      k_prep_a_cx_n<<<dim3(cdiv(m, 32), cdiv(k, 32)), 256, 0, ctx->stream>>>(m, k, Kp, (const cxf*)A, lda, Ahi, Alo);
      TN_LAUNCHED(ctx);
      if (Kp > 2 * k) {
        k_prep_a_pad<<<blocks_for(ctx, Ma * (Kp - 2 * k)), 256, 0, ctx->stream>>>(Ma, 2 * k, Kp, Ahi, Alo);
        TN_LAUNCHED(ctx);
      }
    } else {
      k_prep_a_cx<<<blocks_for(ctx, Ma * Kp), 256, 0, ctx->stream>>>(m, k, Kp, (const cxf*)A, lda, opa, Ahi, Alo);
      TN_LAUNCHED(ctx);
    }
    k_prep_b_cx<<<blocks_for(ctx, n * Kp), 256, 0, ctx->stream>>>(n, k, Kp, (const cxf*)B, ldb, opb, Bhi, Blo);
    TN_LAUNCHED(ctx);
  } else {
    // A' rows are the m rows of op(A): K-major source when op(A) = Aᵀ
    k_prep_re<<<blocks_for(ctx, m * Kp), 256, 0, ctx->stream>>>(m, k, Kp, (const float*)A, lda, opa != 'N', Ahi, Alo);
    TN_LAUNCHED(ctx);
    k_prep_re<<<blocks_for(ctx, n * Kp), 256, 0, ctx->stream>>>(n, k, Kp, (const float*)B, ldb, opb == 'N', Bhi, Blo);
    TN_LAUNCHED(ctx);
  }
  Maps maps;
  memset(&maps, 0, sizeof(maps));
  TN_RETURN_IF(make_map(ctx, &maps.a[0], Ahi, Ma, Kp, BM));
  TN_RETURN_IF(make_map(ctx, &maps.b[0], Bhi, n, Kp, BN));
  if (split) {
    TN_RETURN_IF(make_map(ctx, &maps.a[1], Alo, Ma, Kp, BM));
    TN_RETURN_IF(make_map(ctx, &maps.b[1], Blo, n, Kp, BN));
  } else {
    maps.a[1] = maps.a[0];
    maps.b[1] = maps.b[0];
  }
  const int64_t tiles = (int64_t)cdiv(Ma, BM) * cdiv(n, BN);
  if (tiles > 0x7fffffffll) return tn_set_error(ctx, TN_EUNSUPPORTED, "tc_gemm: too many tiles");
  const dim3 grid((unsigned)tiles);
  if (complex_in) {
    TN_CHECK_CUDA(ctx, cudaFuncSetAttribute(k_gemm_tf32<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
    k_gemm_tf32<1><<<grid, 128, SMEM_BYTES, ctx->stream>>>(maps, passes, (int)Ma, (int)n, (int)Kp, (float*)C, ldc,
                                                           (int)m, alpha, beta, err);
  } else {
    TN_CHECK_CUDA(ctx, cudaFuncSetAttribute(k_gemm_tf32<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
    k_gemm_tf32<0><<<grid, 128, SMEM_BYTES, ctx->stream>>>(maps, passes, (int)Ma, (int)n, (int)Kp, (float*)C, ldc,
                                                           (int)m, alpha, beta, err);
  }
  TN_LAUNCHED(ctx);
  int* hp = reinterpret_cast<int*>(ctx->pinned);
  TN_CHECK_CUDA(ctx, cudaMemcpyAsync(hp, err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  TN_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (hp[0]) return tn_set_error(ctx, TN_ETIMEOUT, "tc_gemm: a pipeline wait timed out");
  return TN_OK;
}

// Tall products with k ≤ 64 whose rows are contiguous in A: at least one 128-row tile per SM for
// every column block of 64, and enough contraction and columns that the tensor pipe pays
// (the general path's own bounds).
bool tc_gemm_tall_fits(tn_ctx* ctx, int64_t m, int64_t n, int64_t k, const GemmView& va) {
  return k >= 32 && k <= 16 * TALL_KT && n >= 48 && va.row.inner == 1 &&
         (va.row.outer == 0 || va.row.extent >= 32) && (m + 127) / 128 * ((n + 63) / 64) >= ctx->num_sms && (n + 63) / 64 <= 65535;
}

tn_status_t tc_gemm_tall(tn_ctx* ctx, int passes, int64_t m, int64_t n, int64_t k, float alpha, const cxf* A,
                         const GemmView& va, const cxf* B, const GemmView& vb, float beta, cxf* C, int64_t ldc) {
  int* err = nullptr;
  TN_RETURN_IF(wait_error_word(ctx, &err));
  const int64_t blocks = (n + 63) / 64, tiles = (m + 127) / 128;
  const int64_t gx = std::min<int64_t>(tiles, std::max<int64_t>(1, ctx->num_sms / blocks));
  TN_CHECK_CUDA(ctx, cudaFuncSetAttribute(k_gemm_tf32_tall, cudaFuncAttributeMaxDynamicSharedMemorySize, TALL_SMEM));
  k_gemm_tf32_tall<<<dim3((unsigned)gx, (unsigned)blocks), TALL_THREADS, TALL_SMEM, ctx->stream>>>(
      m, n, (int)k, passes, A, va, B, vb, alpha, beta, C, ldc, err);
  TN_LAUNCHED(ctx);
  return TN_OK;
}

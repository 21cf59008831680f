// K2c — ComplexF64 GEMM from exact BF16 digit planes on the tcgen05 tensor pipe
// (an error-free splitting in the manner of Ozaki, Ogita, Oishi & Rump, "Error-free
// transformations of matrix multiplication by using fast routines of matrix
// multiplication and its applications", Numer. Algorithms 59 (2012)).
//
//   C = alpha · op(A) · op(B) + beta · C          (A, B, C ComplexF64, column-major)
//
// Splitting.  Every row i of op(A) gets a power-of-two scale σ_i ≥ max_k(|Re a_ik|,
// |Im a_ik|) and every column j of op(B) a scale τ_j.  Each real part v of an entry is
// cut into S signed digits of b bits (b ≤ 8):
//     v = σ · 2^{2-b} · Σ_{p=0}^{S-1} d_p · 2^{-bp} + r,   |d_p| ≤ 2^{b-1} integers,
//     |r| ≤ 2^{1-bS} σ,
// computed exactly (the top digit rint(2^{b-2}·v/σ) in FP64 — one bit of headroom, so the
// carry from the lower digits keeps it within 2^{b-1} — the others as balanced base-2^b
// digits of the remainder held as one int64).  Every digit is an integer of magnitude
// ≤ 2^{b-1} ≤ 128, exactly representable in BF16.
//
// Products.  Complex arithmetic uses the real 4M form with Re/Im rows interleaved:
//     A''[2i]   = [Re a_i·, −Im a_i·],  A''[2i+1] = [Im a_i·, Re a_i·]   (2m × 2k)
//     B''[j]    = [Re b_·j,  Im b_·j]                                      (n × 2k)
// so that (A''·B''ᵀ)[2i + c, j] is Re (c = 0) or Im (c = 1) of (op(A)·op(B))_ij.  The
// digit planes D^A_p, D^B_q (p, q < S) are multiplied on the tensor pipe (kind::f16,
// BF16 inputs, FP32 accumulation) for every pair with p + q < S, and all pairs of one
// level L = p + q accumulate into one TMEM accumulator.  A level holds at most S pairs
// of K = 2k products of magnitude ≤ 2^{2b-2}, so its sum is an integer ≤ S·K·2^{2b-2};
// b is the widest digit with S·K·2^{2b-2} ≤ 2^24, which keeps the FP32 accumulation
// exact, and contractions too long for b = 7 are split on the host into chunks that
// accumulate into C.  The epilogue combines the levels exactly in int64 (the FP64 pipe
// is the scarce one on this part) and applies σ_i τ_j 2^{4-2b} in FP64:
//     c_ij = σ_i τ_j 2^{4-2b} Σ_L 2^{-bL} acc_L.
// The only approximation is the dropped pairs (p + q ≥ S) and the digit remainders, of
// relative size ~S·2^{1-bS} per product: S = 8, b = 7 gives ~52 bits, FP64-grade products.
//
// Kernel.  One persistent CTA (6 warps) per SM takes 128×64 tiles of the real 4M product of all
// batch instances in turn.  Warp 4 lane 0 issues TMA loads: a K stage is 32 BF16 (64 bytes,
// 64-byte swizzle) of all S digit planes of both tiles, two stages in shared memory.  Warp 5
// lane 0 issues tcgen05.mma (M=128, N=256, K=16): plane p of A against four planes of B at a time,
// every plane q < S − p into level p + q (TMEM columns 64·(p+q)…).  After plane 3 of A, the first four
// of A and the last four of B are not needed again in this stage, and their place goes back to the
// producer one stage ahead of its next use.  Warps 0-3 read the S level accumulators with
// tcgen05.ld (warp w owns rows 32w…32w+31) into int64 sums in registers, give the accumulators
// back to warp 5, and finish and write C while the next tile is multiplied.
// Every mbarrier wait is bounded: on timeout the kernel records an error word, skips the
// remaining work and still releases its TMEM.
//
// What bounds it: the tensor pipe.  The S planes of B lie one after the other and so do the
// levels, so four planes of B are one operand of N = 256: a tile of k = 256 takes 47 thousand clocks of
// tensor pipe (a product per pair of planes, N = 64, took 81 clocks each, 90 thousand).  Its planes come
// four to a TMA load; one load each, 16 a stage, took 53 thousand clocks to issue and complete.
// Reading the accumulators takes 12 thousand more; the rest of the epilogue (3 thousand; with 14
// FP64 operations of 64 clocks per column 88 to 129) runs beside the next tile.
// 16 products of 512 × 512 × 512: 1.97 → 0.77 ms, of it the operand preparation 0.54 → 0.24.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cstring>

#include "tn_internal.cuh"

namespace {

constexpr int OZ_BM = 128, OZ_BN = 64, OZ_BK = 32;  // tile 128×64, 32 BF16 (64 B) of K per stage
constexpr int OZ_MAX_S = 8;
constexpr int OZ_WIN = 4;  // levels of one accumulator, planes of B in one product (N = 256)
constexpr int OZ_A_TILE = OZ_BM * OZ_BK * 2;  // 8 KB
constexpr int OZ_B_TILE = OZ_BN * OZ_BK * 2;  // 4 KB
constexpr int OZ_THREADS = 192;
constexpr long long kOzSpin = 1ll << 24;

// planes that a stage has room for: a multiple of OZ_WIN, those beyond S are filled with zeros
__host__ __device__ inline int oz_planes(int S) { return S <= OZ_WIN ? OZ_WIN : 2 * OZ_WIN; }
inline int oz_smem_bytes(int S) {  // (three planes of zeros before B's)
  return 2 * (oz_planes(S) * OZ_A_TILE + (oz_planes(S) + OZ_WIN - 1) * OZ_B_TILE) + 1024 + 512;
}

struct OzMaps {
  CUtensorMap a;  // digit planes of A'': (2k, 2m, batch, S)
  CUtensorMap b;  // digit planes of B'': (2k, n, batch, S)
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
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
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* err) {
  for (long long i = 0; i < kOzSpin; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  atomicExch(err, 1);
  return false;
}
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::
          "r"(smem_u32(dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}
// shared-memory matrix descriptor: K-major, 64-byte swizzle, 8-row groups 512 B apart
__device__ __forceinline__ uint64_t sdesc(const void* p) {
  const uint64_t addr = (uint64_t)smem_u32(p);
  uint64_t d = (addr & 0x3FFFFull) >> 4;
  d |= 1ull << 16;
  d |= (uint64_t)(512 >> 4) << 32;
  d |= 1ull << 46;
  d |= 4ull << 61;
  return d;
}
// instruction descriptor, kind::f16: D f32, A and B bf16, both K-major, M = 128, N = 256
constexpr uint32_t kIdescBF16 =
    (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(OZ_WIN * OZ_BN >> 3) << 17) | ((uint32_t)(OZ_BM >> 4) << 24);

__device__ __forceinline__ void mma_bf16(uint32_t dtmem, uint64_t a, uint64_t b, uint32_t accum) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
          dtmem),
      "l"(a), "l"(b), "r"(kIdescBF16), "r"(accum)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr)
      : "memory");
}

// x · 2^e by an addition to the exponent (the FP64 pipe takes 64 clocks for a product), for x and
// results that are 0 or normal numbers
__device__ __forceinline__ double times_pow2(double x, int e) {
  const int hi = __double2hiint(x);
  return __hiloint2double((hi & 0x7ff00000) ? hi + (e << 20) : hi, __double2loint(x));
}
// the exponent of a power of two (1024 stands for what is none)
__device__ __forceinline__ int exponent_of(double pow2) { return ((__double2hiint(pow2) >> 20) & 0x7ff) - 1023; }

// grid: at most one CTA per SM; 192 threads
__global__ void __launch_bounds__(OZ_THREADS, 1)
    k_gemm_oz(const __grid_constant__ OzMaps maps, int S, int bits, int M2, int N, int K2, int batch, cxd* __restrict__ C,
              int64_t ldc, int64_t sC, const double* __restrict__ sig, const double* __restrict__ tau, cxd alpha,
              cxd beta, int m_complex, int upper, int* err) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t base_u = smem_u32(smem_raw);
  unsigned char* smem = smem_raw + ((1024 - (base_u & 1023)) & 1023);
  unsigned char* sA = smem;                          // 2 stages × SP planes
  const int SP = oz_planes(S), b_planes = SP + OZ_WIN - 1;
  unsigned char* sZ = smem + 2 * SP * OZ_A_TILE;     // 2 stages × (3 planes of zeros and SP of B)
  unsigned char* sB = sZ + (OZ_WIN - 1) * OZ_B_TILE;
  uint64_t* full = reinterpret_cast<uint64_t*>(sZ + 2 * b_planes * OZ_B_TILE);  // [2]
  uint64_t* empty = full + 2;                                            // [2][2]
  uint64_t* acc_full = empty + 4;
  uint64_t* acc_empty = acc_full + 1;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(acc_empty + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles_m = (M2 + OZ_BM - 1) / OZ_BM;
  const int per = upper ? tiles_m * (tiles_m + 1) / 2 : tiles_m * ((N + OZ_BN - 1) / OZ_BN);
  const int64_t tiles = (int64_t)per * batch;
  // a tile's first real row and its column; upper: the tiles on and above the diagonal, column by column
  auto place = [&](int w, int& m0, int& n0) {
    int ti = w % tiles_m, tj = w / tiles_m;
    if (upper) {
      tj = (int)((sqrtf(8.0f * (float)w + 1.0f) - 1.0f) * 0.5f);
      while (tj * (tj + 1) / 2 > w) --tj;
      while ((tj + 1) * (tj + 2) / 2 <= w) ++tj;
      ti = w - tj * (tj + 1) / 2;
    }
    m0 = ti * OZ_BM;
    n0 = tj * OZ_BN;
  };
  const uint32_t tcols = S <= 4 ? 256u : 512u;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(tcols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 32) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(&full[b], 1);
      for (int p = 0; p < 2; ++p) mbar_init(&empty[b * 2 + p], 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 4);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int t = tid; t < 2 * b_planes * (OZ_B_TILE / 16); t += OZ_THREADS)  // (also what no plane is loaded to)
    reinterpret_cast<uint4*>(sZ)[t] = make_uint4(0, 0, 0, 0);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tslot;
  const int nks = (K2 + OZ_BK - 1) / OZ_BK;

  if (warp == 4) {
    if (lane == 0) {
      // producer: four planes of A from the first and of B from the last, as the stage before last
      // gives their place back
      long long g = 0;
      bool ok = true;
      for (int64_t tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const int bidx = (int)(tile / per);
        int m0, n0;
        place((int)(tile % per), m0, n0);
        for (int ks = 0; ks < nks && ok; ++ks, ++g) {
          const int kb = (int)(g & 1);
          const uint32_t parity = (uint32_t)((g >> 1) & 1) ^ 1;
          for (int p = 0; p < SP / OZ_WIN; ++p) {
            if (g >= 2 && !(ok = mbar_wait(&empty[kb * 2 + p], parity, err))) break;
            if (p == 0) mbar_expect_tx(&full[kb], (uint32_t)(SP * (OZ_A_TILE + OZ_B_TILE)));
            tma_load_4d(sA + (kb * SP + p * OZ_WIN) * OZ_A_TILE, &maps.a, &full[kb], ks * OZ_BK, m0, bidx, p * OZ_WIN);
            const int q = SP - (p + 1) * OZ_WIN;
            tma_load_4d(sB + (kb * b_planes + q) * OZ_B_TILE, &maps.b, &full[kb], ks * OZ_BK, n0, bidx, q);
          }
        }
      }
    }
  } else if (warp == 5) {
    if (lane == 0) {
      // MMA issuer: plane p of A against every plane q < S - p of B, level p + q
      long long g = 0;
      int it = 0;
      bool ok = true;
      for (int64_t tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, ++it) {
        if (it > 0 && !(ok = mbar_wait(acc_empty, (uint32_t)(it - 1) & 1, err))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int ks = 0; ks < nks; ++ks, ++g) {
          const int kb = (int)(g & 1);
          if (!(ok = mbar_wait(&full[kb], (uint32_t)(g >> 1) & 1, err))) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          for (int p = 0; p < S; ++p) {
            // The planes of B lie one after the other, and so do the levels: four planes are one operand
            // of N = 256 for the levels 0 … 3 or 4 … 7, planes before the first are zeros.  (All
            // products into an accumulator have one shape: only those are executed in the order
            // of issue.)
            const uint64_t a0 = sdesc(sA + (kb * SP + p) * OZ_A_TILE), b0 = sdesc(sB + kb * b_planes * OZ_B_TILE);
            for (int w = p < OZ_WIN ? 0 : OZ_WIN; w < SP; w += OZ_WIN) {
#pragma unroll
              for (int kk = 0; kk < OZ_BK / 16; ++kk)  // K = 16 BF16 = 32 bytes
                mma_bf16(tmem + (uint32_t)(w * OZ_BN), a0 + (uint64_t)kk * 2,
                         b0 + (uint64_t)((int64_t)(w - p) * (OZ_B_TILE >> 4) + kk * 2), (ks > 0 || p > 0 || kk > 0) ? 1u : 0u);
            }
            // (planes 0 … 3 of A and the last four of B are done with after group 3)
            if (p % OZ_WIN == OZ_WIN - 1 || p == S - 1) mma_commit(&empty[kb * 2 + p / OZ_WIN]);
          }
        }
        if (ok) mma_commit(acc_full);
      }
    }
  } else {
    // epilogue: warps 0-3
    // The levels are recombined exactly in int64 on the integer pipe (GB300's FP64 pipe
    // is ~1/70 of its FP32 pipe): H = Σ_L acc_L · 2^{b(S−1−L)−D}, each acc_L an
    // integer of magnitude ≤ 2^24 (exact in FP32), D = max(0, b(S−1) − 37) so that
    // |H| < 2^62; the levels below 2^D are rounded to nearest (an error of at most
    // S/2 units of 2^{D−b(S−1)} relative to acc_0, below 2^-60 of the largest term).
    // The scales σ_i τ_j 2^{4−2b+D−b(S−1)} are powers of two: a lane writes its own component, and
    // for alpha = ±1 and beta = 0 or 1 the only FP64 operation left is the sum with C.
    const int D = bits * (S - 1) > 37 ? bits * (S - 1) - 37 : 0, shift = 4 - 2 * bits + D - bits * (S - 1);
    const bool plain = alpha.y == 0.0 && (alpha.x == 1.0 || alpha.x == -1.0) && beta.y == 0.0 && (beta.x == 0.0 || beta.x == 1.0);
    const bool beta_zero = beta.x == 0.0 && beta.y == 0.0;
    int it = 0;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++it) {
      const int bidx = (int)(tile / per);
      int m0, n0;
      place((int)(tile % per), m0, n0);
      const bool mirror = upper && m0 != 2 * n0;  // a tile above the diagonal writes the one below it as well
      if (!mbar_wait(acc_full, (uint32_t)it & 1, err)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      long long h[OZ_BN];
#pragma unroll
      for (int j = 0; j < OZ_BN; ++j) h[j] = 0;
#pragma unroll 1
      for (int L = 0; L < S; ++L) {
        const int sh = bits * (S - 1 - L) - D;
        const int up = max(sh - 32, 0), mul = 1 << max(0, min(30, sh)), twice = sh == 31 ? 1 : 0;
        const int rs = sh < 0 ? min(-sh, 31) : 0, half = sh < 0 ? 1 << (rs - 1) : 0;
#pragma unroll
        for (int cb = 0; cb < OZ_BN; cb += 32) {
          uint32_t v[32];
          tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(L * OZ_BN + cb), v);
          if (sh >= 32) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              h[cb + j] += (long long)((unsigned long long)(unsigned)(__float2int_rn(__uint_as_float(v[j])) << up) << 32);
          } else if (sh >= 0) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              h[cb + j] += (long long)(__float2int_rn(__uint_as_float(v[j])) << twice) * (long long)mul;
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) h[cb + j] += (long long)((__float2int_rn(__uint_as_float(v[j])) + half) >> rs);
          }
        }
      }
      // the accumulators are read: the next tile's products may begin
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty);
      const int row = m0 + warp * 32 + lane;  // real row of the 4M product: 2i + (0 Re | 1 Im)
      const int i = row >> 1;
      const bool live = row < M2;
      cxd* Cb = C + (int64_t)bidx * sC;
      const double si = live ? sig[(int64_t)bidx * m_complex + i] : 1.0;
      const int ei = exponent_of(si);
      // the tile's column scales: one exponent per lane and half
      const double t0 = n0 + lane < N ? tau[(int64_t)bidx * N + n0 + lane] : 1.0;
      const double t1 = n0 + 32 + lane < N ? tau[(int64_t)bidx * N + n0 + 32 + lane] : 1.0;
      const int e0 = exponent_of(t0), e1 = exponent_of(t1);
      double* Cr = reinterpret_cast<double*>(Cb + (int64_t)n0 * ldc) + row;
      // (the code of the 64 columns is kept short: it runs once a tile, and its fetching would
      // otherwise take longer than its execution)
      const int base = ei + shift;
      const int lowest = base + __reduce_min_sync(0xffffffffu, min(e0, e1)), highest = base + __reduce_max_sync(0xffffffffu, max(e0, e1));
      // (|h| is 0 or between 1 and 2^62)
      const bool normal = __all_sync(0xffffffffu, lowest > -1022 && highest < 960);
      if (plain && normal) {
        const unsigned flip = alpha.x < 0.0 ? 0x80000000u : 0u;
#pragma unroll
        for (int c = 0; c < OZ_BN; c += 16) {
          double old[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) old[j] = !beta_zero && live && n0 + c + j < N ? Cr[2 * (int64_t)(c + j) * ldc] : 0.0;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int ej = __shfl_sync(0xffffffffu, c + j < 32 ? e0 : e1, (c + j) & 31);
            const double x = times_pow2((double)h[c + j], base + ej);
            const double y = __hiloint2double(__double2hiint(x) ^ flip, __double2loint(x));
            const double z = beta_zero ? y : y + old[j];
            if (live && n0 + c + j < N) {
              Cr[2 * (int64_t)(c + j) * ldc] = z;
              if (mirror) reinterpret_cast<double*>(Cb + (n0 + c + j) + (int64_t)i * ldc)[row & 1] = (row & 1) ? -z : z;
            }
          }
        }
      } else {
        // any alpha and beta, and scales whose products may not be normal numbers
#pragma unroll
        for (int j = 0; j < OZ_BN; ++j) {
          const double tj = __shfl_sync(0xffffffffu, j < 32 ? t0 : t1, j & 31);
          const double x = ldexp(si, shift) * tj * (double)h[j], y = __shfl_xor_sync(0xffffffffu, x, 1);
          if (live && n0 + j < N && !(lane & 1)) {
            cxd* dst = Cb + i + (int64_t)(n0 + j) * ldc;
            cxd out = alpha * mkcx(x, y);
            if (!beta_zero) out = out + beta * *dst;
            *dst = out;
            if (mirror) Cb[(n0 + j) + (int64_t)i * ldc] = conjg(out);
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tcols) : "memory");
}

// ---------------------------------------------------------------------------------
// operand preparation
// ---------------------------------------------------------------------------------
// op(X) as a K-major "row" matrix X̃ (rows r, contraction index c): X̃(r, c) =
// base[r + c·ld] (r_contig) or base[c + r·ld], conjugated when conj.
struct OpView {
  const cxd* base;
  int64_t ld, stride;  // leading dimension, instance stride
  bool r_contig, conj;
};
__device__ __forceinline__ cxd view_at(const OpView& v, int64_t b, int64_t r, int64_t c) {
  cxd x = v.r_contig ? v.base[b * v.stride + r + c * v.ld] : v.base[b * v.stride + c + r * v.ld];
  if (v.conj) x.y = -x.y;
  return x;
}

// the larger of two |Re|, |Im| bit patterns (ordered like the values; a NaN counts as 0)
__device__ __forceinline__ unsigned long long larger_abs(unsigned long long m, cxd x) {
  const unsigned long long a = (unsigned long long)__double_as_longlong(fabs(x.x)), b = (unsigned long long)__double_as_longlong(fabs(x.y));
  m = a > m && a <= 0x7ff0000000000000ull ? a : m;
  return b > m && b <= 0x7ff0000000000000ull ? b : m;
}
__device__ __forceinline__ double scale_of(unsigned long long m) {
  const double mx = __longlong_as_double((long long)m);
  double s = 1.0;
  if (mx > 0.0) {
    int e;
    const double f = frexp(mx, &e);  // mx = f·2^e, f ∈ [0.5, 1)
    s = ldexp(1.0, f == 0.5 ? e - 1 : e);
  }
  return s;
}

// σ_r = the smallest power of two ≥ max_c max(|Re X̃(r,c)|, |Im X̃(r,c)|) (1 for a zero row).
// Contiguous rows: 32 rows per block, a warp reads them side by side; otherwise one warp per row.
__global__ void __launch_bounds__(256) k_oz_scales(OpView v, int64_t R, int64_t K, int64_t batch, double* __restrict__ out) {
  __shared__ unsigned long long part[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (v.r_contig) {
    const int64_t blocks = (R + 31) / 32;
    for (int64_t w = blockIdx.x; w < blocks * batch; w += gridDim.x) {
      const int64_t b = w / blocks, r = w % blocks * 32 + lane;
      unsigned long long mx = 0;
      if (r < R)
        for (int64_t c = warp; c < K; c += 8) mx = larger_abs(mx, view_at(v, b, r, c));
      part[warp][lane] = mx;
      __syncthreads();
      if (warp == 0 && r < R) {
#pragma unroll
        for (int u = 1; u < 8; ++u) mx = part[u][lane] > mx ? part[u][lane] : mx;
        out[b * R + r] = scale_of(mx);
      }
      __syncthreads();
    }
    return;
  }
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t w = blockIdx.x * (int64_t)(blockDim.x >> 5) + warp; w < R * batch; w += warps) {
    const int64_t b = w / R, r = w % R;
    unsigned long long mx = 0;
    for (int64_t c = lane; c < K; c += 32) mx = larger_abs(mx, view_at(v, b, r, c));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long u = __shfl_xor_sync(0xffffffffu, mx, o);
      mx = u > mx ? u : mx;
    }
    if (lane == 0) out[b * R + r] = scale_of(mx);
  }
}

// v·2^ex rounded to the nearest integer (even on a tie), |v·2^ex| ≤ 2^62
__device__ __forceinline__ long long fixed_of(double v, int ex) {
  const long long bits = __double_as_longlong(v);
  const int e = (int)((unsigned long long)bits >> 52) & 0x7ff, s = e - 1075 + ex;
  if (e == 0 || e == 0x7ff) return v == 0.0 ? 0 : llrint(ldexp(v, ex));
  const unsigned long long m = ((unsigned long long)bits & 0xfffffffffffffull) | 0x10000000000000ull;
  unsigned long long q;
  if (s >= 0) {
    q = m << min(s, 10);
  } else if (s < -54) {
    q = 0;
  } else {
    const unsigned long long half = 1ull << (-s - 1), rem = m & (2 * half - 1);
    q = m >> -s;
    q += rem > half || (rem == half && (q & 1)) ? 1 : 0;
  }
  return bits < 0 ? -(long long)q : (long long)q;
}
// an integer of magnitude ≤ 2^22 as a float, by additions (its BF16 form is the upper half)
__device__ __forceinline__ unsigned digit_bits(int d) { return __float_as_uint(__int_as_float(0x4B400000 + d) - 12582912.0f); }

// digit planes of one operand.  a_form: A'' rows 2r (Re) / 2r+1 (Im) with columns
// [Re | −Im] / [Im | Re]; otherwise B'' rows r with columns [Re | Im].  Planes are
// stored plane-major: out[(p·batch + b)·rows'·pitch + row'·pitch + col].  32×32 tiles of
// X̃ are staged through shared memory so that reads follow the source's contiguous index
// and writes the contraction index, two entries per thread.  All arithmetic is on integers: an
// entry becomes round(x·2^{bS−2}/σ) and its balanced base-2^b digits are peeled off from the bottom
// (in FP64, with a conversion per digit, the FP64 pipe took 0.27 ms for 16 × 512² where the
// planes' 200 MB take 0.05; now 0.12).
__global__ void __launch_bounds__(256)
    k_oz_split(OpView v, int64_t R, int64_t K, int64_t batch, int S, int bits, bool a_form, const double* __restrict__ scale,
               int64_t pitch, unsigned short* __restrict__ out) {
  __shared__ cxd tile[32][33];
  const int64_t r0 = (int64_t)blockIdx.x * 32, c0 = (int64_t)blockIdx.y * 32, b = blockIdx.z;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 × 8
  for (int u = ty; u < 32; u += 8) {
    // tile[c][r]; the fast thread index follows the source's contiguous dimension
    const int64_t r = v.r_contig ? r0 + tx : r0 + u, c = v.r_contig ? c0 + u : c0 + tx;
    const cxd x = (r < R && c < K) ? view_at(v, b, r, c) : mkcx(0.0, 0.0);
    if (v.r_contig)
      tile[u][tx] = x;
    else
      tile[tx][u] = x;
  }
  __syncthreads();
  const int64_t rows_out = a_form ? 2 * R : R;
  const int64_t plane = rows_out * pitch;
  const long long half = 1ll << (bits - 1), mask = (1ll << bits) - 1;
  const bool pairs = (K & 1) == 0;
  for (int u = threadIdx.x >> 4; u < 32; u += 16) {
    const int64_t r = r0 + u, c = c0 + 2 * (threadIdx.x & 15);
    if (r >= R || c >= K) continue;
    const int ex = bits * S - 2 - exponent_of(scale[b * R + r]);
    long long X[4];  // Re, Im of entry c, Re, Im of entry c + 1 (0 beyond K: the tile's padding)
#pragma unroll
    for (int z = 0; z < 2; ++z) {
      const cxd x = tile[2 * (threadIdx.x & 15) + z][u];
      X[2 * z] = fixed_of(x.x, ex);
      X[2 * z + 1] = fixed_of(x.y, ex);
    }
    unsigned short* o = out + ((int64_t)(S - 1) * batch + b) * plane + (a_form ? 2 * r : r) * pitch + c;
    for (int p = S - 1; p >= 0; --p, o -= (int64_t)batch * plane) {
      unsigned f[4];
#pragma unroll
      for (int z = 0; z < 4; ++z) {
        const long long d = p > 0 ? ((X[z] + half) & mask) - half : X[z];
        X[z] = (X[z] - d) >> bits;
        f[z] = digit_bits((int)d);
      }
      const unsigned re = __byte_perm(f[0], f[2], 0x7632), im = __byte_perm(f[1], f[3], 0x7632);
      if (pairs) {
        *reinterpret_cast<unsigned*>(o) = re;
        *reinterpret_cast<unsigned*>(o + K) = a_form ? im ^ 0x80008000u : im;
        if (a_form) {
          *reinterpret_cast<unsigned*>(o + pitch) = im;
          *reinterpret_cast<unsigned*>(o + pitch + K) = re;
        }
      } else {
        const int two = c + 1 < K ? 2 : 1;
        for (int z = 0; z < two; ++z) {
          const unsigned short dr = (unsigned short)(z ? re >> 16 : re), di = (unsigned short)(z ? im >> 16 : im);
          o[z] = dr;
          o[z + K] = a_form ? di ^ 0x8000 : di;
          if (a_form) {
            o[z + pitch] = di;
            o[z + pitch + K] = dr;
          }
        }
      }
    }
  }
}

// planes of rows × K2 BF16 per instance: a row `pitch` and an instance `matrix` elements after the one
// before, the planes batch instances apart; a box is `box_rows` rows of 64 bytes of OZ_WIN planes
tn_status_t make_map4(tn_ctx* ctx, CUtensorMap* map, const void* base, int64_t K2, int64_t rows, int64_t batch, int64_t planes,
                      int64_t pitch, int64_t matrix, uint32_t box_rows) {
  EncodeTiledFn fn = tn_encode_tiled_fn(ctx);
  if (!fn) return TN_ECUDA;
  cuuint64_t dims[4] = {(cuuint64_t)K2, (cuuint64_t)rows, (cuuint64_t)batch, (cuuint64_t)planes};
  cuuint64_t strides[3] = {(cuuint64_t)(pitch * 2), (cuuint64_t)(matrix * 2), (cuuint64_t)(matrix * 2 * batch)};
  cuuint32_t box[4] = {(cuuint32_t)OZ_BK, box_rows, 1, (cuuint32_t)OZ_WIN};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, (void*)base, dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return tn_set_error(ctx, TN_ECUDA, "cuTensorMapEncodeTiled (split GEMM) failed (%d)", (int)r);
  return TN_OK;
}

OpView make_view(const cxd* base, int64_t ld, int64_t stride, char op, bool is_a) {
  OpView v;
  v.base = base;
  v.ld = ld;
  v.stride = stride;
  v.conj = op == 'C';
  // A: X̃ = op(A) (rows i): 'N' → A[i + c·lda] (r-contiguous).  B: X̃ = op(B)ᵀ (rows j):
  // 'N' → B[c + j·ldb] (c-contiguous); 'T'/'C' → B[j + c·ldb].
  v.r_contig = is_a ? (op == 'N') : (op != 'N');
  return v;
}

// the split GEMM's error word (sticky until split_gemm_check reads it)
tn_status_t oz_error_word(tn_ctx* ctx, int** out) {
  if (!ctx->oz_err) {
    void* p = nullptr;
    TN_RETURN_IF(tn_dev_alloc(ctx, 256, &p));
    TN_CHECK_CUDA(ctx, cudaMemsetAsync(p, 0, sizeof(int), ctx->stream));
    ctx->oz_err = static_cast<int*>(p);
  }
  *out = ctx->oz_err;
  return TN_OK;
}

// the split GEMM's operand planes, kept in a scratch of the context's own: grown (after
// the stream has drained) when a larger product needs it
tn_status_t oz_scratch(tn_ctx* ctx, size_t bytes, char** out) {
  if (bytes > ctx->oz_cap) {
    if (ctx->oz_ws) {
      TN_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
      TN_RETURN_IF(tn_dev_free(ctx, ctx->oz_ws));
      ctx->oz_ws = nullptr;
      ctx->oz_cap = 0;
    }
    void* p = nullptr;
    TN_RETURN_IF(tn_dev_alloc(ctx, bytes, &p));
    ctx->oz_ws = static_cast<char*>(p);
    ctx->oz_cap = bytes;
  }
  *out = ctx->oz_ws;
  return TN_OK;
}

}  // namespace

tn_status_t gemm_c64_split(tn_ctx* ctx, int S, char opa, char opb, int64_t m, int64_t n, int64_t k, cxd alpha,
                           const cxd* A, int64_t lda, int64_t sA, const cxd* B, int64_t ldb, int64_t sB, cxd beta,
                           cxd* C, int64_t ldc, int64_t sC, int64_t batch, bool hermitian) {
  if (m == 0 || n == 0 || batch == 0) return TN_OK;
  if (S < 2 || S > OZ_MAX_S) return tn_set_error(ctx, TN_EINVAL, "split GEMM: slices must be in [2, %d]", OZ_MAX_S);
  if (batch > 65535) return tn_set_error(ctx, TN_EUNSUPPORTED, "split GEMM: batch > 65535");
  if (k == 0) return gemm_cx<double>(ctx, opa, opb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch);
  // Aᴴ·A: B'' is the even rows of A'', so its planes need not be cut, and with a real alpha the
  // product is Hermitian: for beta = 0, or where C is known to be, the tiles above the diagonal
  // are enough (16 × 512³: 0.78 → 0.46 ms)
  const bool gram = opa == 'C' && opb == 'N' && A == B && lda == ldb && (sA == sB || batch == 1) && m == n;
  const bool upper = gram && alpha.y == 0.0 && ((beta.x == 0.0 && beta.y == 0.0) || (hermitian && beta.y == 0.0));
  // a level's FP32 sum is exact while S·(2k)·2^{2b-2} ≤ 2^24: the widest such digit b
  // (at most 8); contractions that would need b < 7 run in chunks of k sized for b = 7,
  // the later chunks accumulating into C (beta = 1)
  int bits = 8;
  while (bits > 1 && (double)S * (double)(2 * k) * ldexp(1.0, 2 * bits - 2) > 16777216.0) --bits;
  const int64_t kmax = std::max<int64_t>(32, (4096 / S) / 2 / 32 * 32);
  if (bits < 7 && k > kmax) {
    for (int64_t k0 = 0; k0 < k; k0 += kmax) {
      const int64_t kc = std::min(kmax, k - k0);
      const cxd* Ac = (opa == 'N') ? A + k0 * lda : A + k0;
      const cxd* Bc = (opb == 'N') ? B + k0 : B + k0 * ldb;
      TN_RETURN_IF(gemm_c64_split(ctx, S, opa, opb, m, n, kc, alpha, Ac, lda, sA, Bc, ldb, sB,
                                  k0 == 0 ? beta : mkcx(1.0, 0.0), C, ldc, sC, batch, upper));
    }
    return TN_OK;
  }
  const int64_t M2 = 2 * m, K2 = 2 * k, pitch = (K2 + 7) / 8 * 8;
  if (M2 > (1ll << 30) || n > (1ll << 30)) return tn_set_error(ctx, TN_EUNSUPPORTED, "split GEMM: too large");
  const size_t bytesA = ws_round(2 * (size_t)(S * batch * M2 * pitch));
  const size_t bytesB = gram ? 0 : ws_round(2 * (size_t)(S * batch * n * pitch));
  const size_t bytesS = ws_round(sizeof(double) * (size_t)(batch * m)) + ws_round(sizeof(double) * (size_t)(batch * n));
  char* ws = nullptr;
  int* err = nullptr;
  TN_RETURN_IF(oz_error_word(ctx, &err));
  TN_RETURN_IF(oz_scratch(ctx, bytesA + bytesB + bytesS, &ws));
  unsigned short* dA = reinterpret_cast<unsigned short*>(ws);
  unsigned short* dB = reinterpret_cast<unsigned short*>(ws + bytesA);
  double* sig = reinterpret_cast<double*>(ws + bytesA + bytesB);
  double* tau = gram ? sig : sig + ws_round(sizeof(double) * (size_t)(batch * m)) / sizeof(double);
  const OpView va = make_view(A, lda, sA, opa, true), vb = make_view(B, ldb, sB, opb, false);
  const int prep_slot = prof_begin(ctx);
  {
    auto scale_blocks = [&](const OpView& v, int64_t R) {
      const int64_t want = v.r_contig ? (R + 31) / 32 * batch : (R * batch + 7) / 8;
      return (unsigned)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)ctx->num_sms * 16));
    };
    k_oz_scales<<<scale_blocks(va, m), 256, 0, ctx->stream>>>(va, m, k, batch, sig);
    TN_LAUNCHED(ctx);
    if (!gram) {
      k_oz_scales<<<scale_blocks(vb, n), 256, 0, ctx->stream>>>(vb, n, k, batch, tau);
      TN_LAUNCHED(ctx);
    }
    k_oz_split<<<dim3(cdiv(m, 32), cdiv(k, 32), (unsigned)batch), 256, 0, ctx->stream>>>(va, m, k, batch, S, bits, true,
                                                                                       sig, pitch, dA);
    TN_LAUNCHED(ctx);
    if (!gram) {
      k_oz_split<<<dim3(cdiv(n, 32), cdiv(k, 32), (unsigned)batch), 256, 0, ctx->stream>>>(vb, n, k, batch, S, bits,
                                                                                         false, tau, pitch, dB);
      TN_LAUNCHED(ctx);
    }
  }
  if (prep_slot >= 0)  // read op(A), op(B) once, write their digit planes and scales
    prof_end(ctx, prep_slot, TN_PROF_SPLIT_PREP, gram ? 2 : 4, 0.0,
             2.0 * 16.0 * ((double)m * k + (gram ? 0.0 : (double)k * n)) * batch +
                 2.0 * S * ((double)M2 + (gram ? 0 : n)) * K2 * batch);
  OzMaps maps;
  memset(&maps, 0, sizeof(maps));
  TN_RETURN_IF(make_map4(ctx, &maps.a, dA, K2, M2, batch, S, pitch, M2 * pitch, OZ_BM));
  if (gram)
    TN_RETURN_IF(make_map4(ctx, &maps.b, dA, K2, n, batch, S, 2 * pitch, M2 * pitch, OZ_BN));
  else
    TN_RETURN_IF(make_map4(ctx, &maps.b, dB, K2, n, batch, S, pitch, n * pitch, OZ_BN));
  const int64_t tiles_m = cdiv(M2, OZ_BM), tiles = upper ? tiles_m * (tiles_m + 1) / 2 : tiles_m * cdiv(n, OZ_BN);
  if (tiles > 0x7fffffffll) return tn_set_error(ctx, TN_EUNSUPPORTED, "split GEMM: too many tiles");
  const int smem = oz_smem_bytes(S);
  TN_CHECK_CUDA(ctx, cudaFuncSetAttribute(k_gemm_oz, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const bool beta_zero = beta.x == 0.0 && beta.y == 0.0;
  const int slot = prof_begin(ctx);
  k_gemm_oz<<<(unsigned)std::min<int64_t>(tiles * batch, ctx->num_sms), OZ_THREADS, smem, ctx->stream>>>(
      maps, S, bits, (int)M2, (int)n, (int)K2, (int)batch, C, ldc, sC, sig, tau, alpha, beta, (int)m, upper ? 1 : 0, err);
  TN_LAUNCHED(ctx);
  if (slot >= 0)  // tensor-pipe flops of the S(S+1)/2 real products it issues; planes read once, C written
    prof_end(ctx, slot, TN_PROF_GEMM_SPLIT, 1, S * (S + 1) / 2 * 2.0 * M2 * n * K2 * batch * (upper ? (tiles_m + 1.0) / (2.0 * tiles_m) : 1.0),
             (2.0 * S * ((double)M2 + n) * K2 + 16.0 * m * n * (beta_zero ? 1 : 2)) * batch);
  return TN_OK;
}

// Shapes below these bounds stay on the FP64 CUDA cores: the split path's operand
// preparation and 128×64 tiles cost more than they save there.
static bool split_pays(int64_t m, int64_t n, int64_t k) { return m >= 32 && n >= 32 && k >= 32 && m * n >= 8192; }

tn_status_t gemm_c64(tn_ctx* ctx, tn_precision_t prec, char opa, char opb, int64_t m, int64_t n, int64_t k, cxd alpha,
                     const cxd* A, int64_t lda, int64_t sA, const cxd* B, int64_t ldb, int64_t sB, cxd beta, cxd* C,
                     int64_t ldc, int64_t sC, int64_t batch) {
  if ((prec == TN_PREC_MIXED || prec == TN_PREC_SPLIT_BF16) && split_pays(m, n, k))
    return gemm_c64_split(ctx, ctx->split_slices, opa, opb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC,
                          batch);
  return gemm_cx<double>(ctx, opa, opb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch);
}

// status of the split GEMMs enqueued since the last check: a pipeline wait that ran out
// is reported here (after the stream has drained)
tn_status_t split_gemm_check(tn_ctx* ctx) {
  if (!ctx->oz_err) return TN_OK;
  int* hp = reinterpret_cast<int*>(ctx->pinned);
  TN_CHECK_CUDA(ctx, cudaMemcpyAsync(hp, ctx->oz_err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  TN_RETURN_IF(read_back_sync(ctx));
  if (hp[0]) {
    TN_CHECK_CUDA(ctx, cudaMemsetAsync(ctx->oz_err, 0, sizeof(int), ctx->stream));
    return tn_set_error(ctx, TN_ETIMEOUT, "split GEMM: a pipeline wait timed out");
  }
  return TN_OK;
}

extern "C" tn_status_t tn_set_split_slices(tn_ctx* ctx, int32_t slices) {
  if (!ctx) return TN_EINVAL;
  TN_ARG(ctx, slices >= 2 && slices <= OZ_MAX_S, "tn_set_split_slices: slices must be in [2, 8]");
  ctx->split_slices = slices;
  return TN_OK;
}

// K2 (native arithmetic) — batched strided complex GEMM on the CUDA cores.
//
//   C = alpha · op(A) · op(B) + beta · C,  op ∈ {N, T, C}, column-major.
//
// This is the plain-form contraction GEMM (ComplexF64 in FP64, ComplexF32 in FP32).  It
// replaces the BLAS zgemm/cgemm inside Muscle.binary_einsum.  On GB300 the FP64 pipe is
// the bound for this kernel, so the design goal is to keep every SM's DFMA units fed:
// register tiles of 4×4 (or 2×2 for small grids) complex accumulators per thread,
// A/B tiles staged through shared memory, and a tile size chosen so the grid covers
// all 152 SMs even for the small bond-dimension GEMMs of an MPS sweep (k_gemm_fine below
// is the kernel for grids that 64×64 tiles leave partly idle).
#include <cooperative_groups.h>

#include "tn_internal.cuh"

namespace {

template <typename T>
__device__ __forceinline__ cx<T> load_op(const cx<T>* __restrict__ X, int64_t ld, char op,
                                         int64_t r, int64_t c) {
  // element (r, c) of op(X)
  if (op == 'N') return X[r + c * ld];
  cx<T> v = X[c + r * ld];
  if (op == 'C') v.y = -v.y;
  return v;
}

template <typename T, int BM, int BN, int BK, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
    k_gemm_cx(char opa, char opb, int64_t m, int64_t n, int64_t k, cx<T> alpha,
              const cx<T>* __restrict__ A, int64_t lda, int64_t sA, const cx<T>* __restrict__ B,
              int64_t ldb, int64_t sB, cx<T> beta, cx<T>* __restrict__ C, int64_t ldc, int64_t sC,
              int64_t batch, bool upper) {
  constexpr int NT = (BM / TM) * (BN / TN);
  constexpr int RX = BN / TN;  // threads along n
  constexpr int RY = BM / TM;  // threads along m
  __shared__ cx<T> As[BK][BM + 1];
  __shared__ cx<T> Bs[BK][BN + 1];
  const int tid = threadIdx.x;
  const int tx = tid % RX, ty = tid / RX;
  const int64_t i0 = (int64_t)blockIdx.x * BM;
  const int64_t j0 = (int64_t)blockIdx.y * BN;
  if (upper && i0 >= j0 + BN) return;  // Hermitian product: tiles below the diagonal are mirrored
  for (int64_t bz = blockIdx.z; bz < batch; bz += gridDim.z) {
    const cx<T>* Ab = A + bz * sA;
    const cx<T>* Bb = B + bz * sB;
    cx<T>* Cb = C + bz * sC;
    cx<T> acc[TM][TN];
#pragma unroll
    for (int a = 0; a < TM; ++a)
#pragma unroll
      for (int b = 0; b < TN; ++b) acc[a][b] = mkcx<T>(0, 0);

    for (int64_t p0 = 0; p0 < k; p0 += BK) {
      // stage A tile (BM × BK)
      for (int t = tid; t < BM * BK; t += NT) {
        int ii, pp;
        if (opa == 'N') {
          ii = t % BM;
          pp = t / BM;
        } else {
          pp = t % BK;
          ii = t / BK;
        }
        int64_t gi = i0 + ii, gp = p0 + pp;
        As[pp][ii] = (gi < m && gp < k) ? load_op(Ab, lda, opa, gi, gp) : mkcx<T>(0, 0);
      }
      // stage B tile (BK × BN)
      for (int t = tid; t < BK * BN; t += NT) {
        int pp, jj;
        if (opb == 'N') {
          pp = t % BK;
          jj = t / BK;
        } else {
          jj = t % BN;
          pp = t / BN;
        }
        int64_t gp = p0 + pp, gj = j0 + jj;
        Bs[pp][jj] = (gp < k && gj < n) ? load_op(Bb, ldb, opb, gp, gj) : mkcx<T>(0, 0);
      }
      __syncthreads();
#pragma unroll
      for (int pp = 0; pp < BK; ++pp) {
        cx<T> a[TM], b[TN];
#pragma unroll
        for (int r = 0; r < TM; ++r) a[r] = As[pp][ty + r * RY];
#pragma unroll
        for (int c = 0; c < TN; ++c) b[c] = Bs[pp][tx + c * RX];
#pragma unroll
        for (int r = 0; r < TM; ++r)
#pragma unroll
          for (int c = 0; c < TN; ++c) cfma(acc[r][c], a[r], b[c]);
      }
      __syncthreads();
    }
    const bool beta0 = beta.x == T(0) && beta.y == T(0);
#pragma unroll
    for (int r = 0; r < TM; ++r) {
      int64_t gi = i0 + ty + r * RY;
      if (gi >= m) continue;
#pragma unroll
      for (int c = 0; c < TN; ++c) {
        int64_t gj = j0 + tx + c * RX;
        if (gj >= n) continue;
        cx<T> v = alpha * acc[r][c];
        if (!beta0) v = v + beta * Cb[gi + gj * ldc];
        Cb[gi + gj * ldc] = v;
      }
    }
  }
}

template <typename T, int BM, int BN, int BK, int TM, int TN>
tn_status_t launch(tn_ctx* ctx, char opa, char opb, int64_t m, int64_t n, int64_t k, cx<T> alpha,
                   const cx<T>* A, int64_t lda, int64_t sA, const cx<T>* B, int64_t ldb, int64_t sB,
                   cx<T> beta, cx<T>* C, int64_t ldc, int64_t sC, int64_t batch, bool upper = false) {
  dim3 grid(cdiv(m, BM), cdiv(n, BN), (unsigned)(batch < 65535 ? batch : 65535));
  if (grid.x > 0x7fffffffu || grid.y > 65535u) return tn_set_error(ctx, TN_EINVAL, "gemm: grid too large");
  const int slot = sizeof(T) == 8 ? prof_begin(ctx) : -1;
  k_gemm_cx<T, BM, BN, BK, TM, TN><<<grid, (BM / TM) * (BN / TN), 0, ctx->stream>>>(
      opa, opb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, upper);
  TN_LAUNCHED(ctx);
  if (slot >= 0) {
    const bool b0 = beta.x == T(0) && beta.y == T(0);
    prof_end(ctx, slot, TN_PROF_GEMM_F64, 1, 8.0 * m * n * k * batch,
             sizeof(cx<T>) * ((double)m * k + (double)k * n + (double)m * n * (b0 ? 1 : 2)) * batch);
  }
  return TN_OK;
}

// Fine-grained GEMM: one output per thread and K group, tiles of BM·BN ≤ 64 outputs.
//
// Bound: the FP64 pipe retires 2 DFMA per clock and SM (64 clocks per warp instruction,
// measured), so a 32×32 tile with k = 64 holds one SM for 70 µs while the chip's rate for the
// whole 64×128×64 product is 4 µs: what counts for an MPS-sized product is that every SM has
// work.  8×8 tiles keep 128 of 152 SMs busy there; operand traffic (32 bytes per 4 DFMA)
// stays two orders below the L2 rate.  Measured (GB300): the overlap of two L = 64, χ = 256 MPS
// (256×512×256 and 256×256×512 products) 49.2 → 27.8 ms, 24.7 ms being the FP64 pipe's time;
// a served burst of 64 queries (L ≤ 48, χ ≤ 128) 18.9 → 7.5 ms; one two-site DMRG sweep
// (L = 24, χ = 32) 297 → 258 ms.  K goes in stages of 32 prefetched to registers, split
// over KS thread groups inside the CTA and over a cluster of CS CTAs (summed through
// distributed shared memory) when the columns alone leave SMs idle.
//
// The sum over k is the same sequence for every tile shape: 16 interleaved accumulators
// (k mod 16) per cluster rank, added in a fixed order, and CS depends on n and k only.  A
// row of C is therefore bit-identical whatever number of rows it is computed with, as long
// as this kernel serves both products.
constexpr int kFineBK = 32, kFineAcc = 16, kFineThreads = 256;

template <typename T, int BM, int BN>
__global__ void __launch_bounds__(kFineThreads)
    k_gemm_fine(char opa, char opb, int64_t m, int64_t n, int64_t k, cx<T> alpha, const cx<T>* __restrict__ A, int64_t lda,
                int64_t sA, const cx<T>* __restrict__ B, int64_t ldb, int64_t sB, cx<T> beta, cx<T>* __restrict__ C,
                int64_t ldc, int64_t sC, int64_t batch, int CS) {
  namespace cg = cooperative_groups;
  constexpr int KS = kFineThreads / (BM * BN), NA = kFineAcc / KS;
  constexpr int LA = (BM * kFineBK + kFineThreads - 1) / kFineThreads, LB = (BN * kFineBK + kFineThreads - 1) / kFineThreads;
  static_assert(KS * NA == kFineAcc, "accumulators must divide among the K groups");
  __shared__ cx<T> As[kFineBK][BM + 1];
  __shared__ cx<T> Bs[kFineBK][BN + 1];
  __shared__ cx<T> part[kFineAcc][BM * BN];
  __shared__ cx<T> total[BM * BN];
  const int tid = threadIdx.x, out = tid % (BM * BN), kg = tid / (BM * BN);
  const int ti = out % BM, tj = out / BM;
  const int rank = (int)(blockIdx.x % (unsigned)CS);
  const int64_t i0 = (int64_t)(blockIdx.x / (unsigned)CS) * BM, j0 = (int64_t)blockIdx.y * BN;
  // this rank's part of K, a whole number of stages
  const int64_t stages = (k + kFineBK - 1) / kFineBK, per = (stages + CS - 1) / CS;
  const int64_t kb = min((int64_t)rank * per * kFineBK, k), ke = min((int64_t)(rank + 1) * per * kFineBK, k);
  for (int64_t bz = blockIdx.z; bz < batch; bz += gridDim.z) {
    const cx<T>* Ab = A + bz * sA;
    const cx<T>* Bb = B + bz * sB;
    cx<T> acc[NA], ra[LA], rb[LB];
#pragma unroll
    for (int a = 0; a < NA; ++a) acc[a] = mkcx<T>(0, 0);
    auto fetch = [&](int64_t p0) {
#pragma unroll
      for (int u = 0; u < LA; ++u) {
        const int t = tid + u * kFineThreads;
        const int ii = opa == 'N' ? t % BM : t / kFineBK, pp = opa == 'N' ? t / BM : t % kFineBK;
        ra[u] = (t < BM * kFineBK && i0 + ii < m && p0 + pp < ke) ? load_op(Ab, lda, opa, i0 + ii, p0 + pp) : mkcx<T>(0, 0);
      }
#pragma unroll
      for (int u = 0; u < LB; ++u) {
        const int t = tid + u * kFineThreads;
        const int pp = opb == 'N' ? t % kFineBK : t / BN, jj = opb == 'N' ? t / kFineBK : t % BN;
        rb[u] = (t < BN * kFineBK && p0 + pp < ke && j0 + jj < n) ? load_op(Bb, ldb, opb, p0 + pp, j0 + jj) : mkcx<T>(0, 0);
      }
    };
    if (kb < ke) fetch(kb);
    for (int64_t p0 = kb; p0 < ke; p0 += kFineBK) {
#pragma unroll
      for (int u = 0; u < LA; ++u) {
        const int t = tid + u * kFineThreads;
        if (t < BM * kFineBK) As[opa == 'N' ? t / BM : t % kFineBK][opa == 'N' ? t % BM : t / kFineBK] = ra[u];
      }
#pragma unroll
      for (int u = 0; u < LB; ++u) {
        const int t = tid + u * kFineThreads;
        if (t < BN * kFineBK) Bs[opb == 'N' ? t % kFineBK : t / BN][opb == 'N' ? t / kFineBK : t % BN] = rb[u];
      }
      __syncthreads();
      if (p0 + kFineBK < ke) fetch(p0 + kFineBK);
      const int kk = (int)min((int64_t)kFineBK, ke - p0);
      // k = p0 + pp + a·KS + kg: accumulator (k mod 16) = a·KS + kg
#pragma unroll
      for (int pp = 0; pp < kFineBK; pp += kFineAcc)
#pragma unroll
        for (int a = 0; a < NA; ++a) {
          const int q = pp + a * KS + kg;
          if (q < kk) cfma(acc[a], As[q][ti], Bs[q][tj]);
        }
      __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < NA; ++a) part[a * KS + kg][out] = acc[a];
    __syncthreads();
    cx<T> v = mkcx<T>(0, 0);
    if (tid < BM * BN) {
      v = part[0][tid];
#pragma unroll
      for (int g = 1; g < kFineAcc; ++g) v = v + part[g][tid];
    }
    if (CS > 1) {
      cg::cluster_group cl = cg::this_cluster();
      if (tid < BM * BN) total[tid] = v;
      cl.sync();
      if (rank == 0 && tid < BM * BN)
        for (int c = 1; c < CS; ++c) v = v + cl.map_shared_rank(total, c)[tid];
      cl.sync();
    }
    const int64_t gi = i0 + tid % BM, gj = j0 + tid / BM;
    if (rank == 0 && tid < BM * BN && gi < m && gj < n) {
      cx<T>* dst = C + bz * sC + gi + gj * ldc;
      cx<T> r = alpha * v;
      if (!(beta.x == T(0) && beta.y == T(0))) r = r + beta * *dst;
      *dst = r;
    }
    __syncthreads();
  }
}

// K split over a cluster while the 8-wide column tiles leave SMs idle and a rank keeps a
// whole stage: a function of n and k only (see the kernel)
int fine_ranks(int64_t n, int64_t k, int64_t sms) {
  int CS = 1;
  while (CS < 8 && (int64_t)cdiv(n, 8) * CS * 2 <= sms && k >= (int64_t)kFineBK * CS * 2) CS *= 2;
  return CS;
}

// Whether FP64 products of these sizes take less time in k_gemm_fine, which spends a whole stage of
// 32 on what is left of k and 16 accumulators' sums per output and rank (some 16 of k; 36 and 22 with
// the tiles of one and two rows): both times in outputs·k of one SM, 2 clocks of its FP64 pipe each.
// 3000 products of sizes from 1 to 20000: of 880 in which k_gemm_fine was slower by more than 6 %, up to
// 5 times, 12 are left, and the sum of all is 0.1 % above that of the faster kernel of each.  Measured,
// µs, register tiles / fine: 64×1000×1 ×200 814 / 4213, 2000×64×4 12.6 / 49.7, 20000×64×4 114 / 431,
// 2000×128×200 ×16 5643 / 9065, 64×128×200 ×200 2466 / 3636; 256×256×512 ×1 1.4 times faster fine.
bool fine_pays(int64_t m, int64_t n, int64_t k, int64_t batch, int64_t bm, int64_t bn, int64_t sms) {
  int64_t tm = 32, tn = 32;  // the register tile that would serve
  if (m <= 8 && n >= 64)
    tm = 8;
  else if (m <= 16 && n >= 64)
    tm = 16;
  else if ((int64_t)cdiv(m, 64) * cdiv(n, 64) * batch >= sms)
    tm = tn = 64;
  // (in 0.95 of k, rounded up to the 8 that are staged together; 0.97 of it in a single wave of 32×32 tiles)
  const int64_t waves = cdiv((int64_t)cdiv(m, tm) * cdiv(n, tn) * batch, sms);
  const double spent = (tm == 32 && waves == 1 && k > 24 ? 0.97 : 0.95) * 8.0 * (double)cdiv(k, 8);
  const int CS = fine_ranks(n, k, sms);
  const double stages = (double)cdiv(k, kFineBK), sums = bm == 1 ? 36 : bm == 2 ? 22 : 16;
  const double fine = (double)cdiv((int64_t)cdiv(m, bm) * cdiv(n, bn) * batch * CS, sms) * (double)(bm * bn);
  return fine * (kFineBK * stages / CS + sums) + 900 < (double)(waves * tm * tn) * spent;
}

template <typename T, int BM, int BN>
tn_status_t launch_fine(tn_ctx* ctx, char opa, char opb, int64_t m, int64_t n, int64_t k, cx<T> alpha, const cx<T>* A,
                        int64_t lda, int64_t sA, const cx<T>* B, int64_t ldb, int64_t sB, cx<T> beta, cx<T>* C,
                        int64_t ldc, int64_t sC, int64_t batch) {
  const int CS = fine_ranks(n, k, ctx->num_sms);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cdiv(m, BM) * (unsigned)CS, cdiv(n, BN), (unsigned)(batch < 65535 ? batch : 65535));
  cfg.blockDim = dim3(kFineThreads);
  cfg.stream = ctx->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)CS;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const int slot = sizeof(T) == 8 ? prof_begin(ctx) : -1;
  TN_CHECK_CUDA(ctx, cudaLaunchKernelEx(&cfg, k_gemm_fine<T, BM, BN>, opa, opb, m, n, k, alpha, A, lda, sA, B, ldb, sB,
                                        beta, C, ldc, sC, batch, CS));
  TN_LAUNCHED(ctx);
  if (slot >= 0) {
    const bool b0 = beta.x == T(0) && beta.y == T(0);
    prof_end(ctx, slot, TN_PROF_GEMM_F64, 1, 8.0 * m * n * k * batch,
             sizeof(cx<T>) * ((double)m * k + (double)k * n + (double)m * n * (b0 ? 1 : 2)) * batch);
  }
  return TN_OK;
}

// C(i, j) = conj(C(j, i)) for i > j (n × n, batched)
template <typename T>
__global__ void k_mirror_lower(int64_t n, cx<T>* C, int64_t ldc, int64_t sC, int64_t batch) {
  const int64_t total = n * n;
  for (int64_t b = blockIdx.y; b < batch; b += gridDim.y)
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
      const int64_t i = t % n, j = t / n;
      if (i > j) C[b * sC + i + j * ldc] = conjg(C[b * sC + j + i * ldc]);
    }
}

}  // namespace

template <typename T>
tn_status_t gemm_cx(tn_ctx* ctx, char opa, char opb, int64_t m, int64_t n, int64_t k, cx<T> alpha,
                    const cx<T>* A, int64_t lda, int64_t sA, const cx<T>* B, int64_t ldb,
                    int64_t sB, cx<T> beta, cx<T>* C, int64_t ldc, int64_t sC, int64_t batch) {
  if (m == 0 || n == 0 || batch == 0) return TN_OK;
  // Which kernel: the SM with the most tiles sets the time, (tiles per SM) × (outputs per
  // tile) in units of k/2 clocks per output.  64×64 tiles reuse operands best and are kept
  // where their last wave is nearly full; 8×8 tiles (5 % overhead assumed) elsewhere.
  // FP32 has 64 times the lanes, so there the small tiles only pay where 32×32 tiles leave
  // three quarters of the SMs idle.
  const int64_t sms = ctx->num_sms;
  const int64_t tiles64 = (int64_t)cdiv(m, 64) * cdiv(n, 64) * batch, tiles32 = (int64_t)cdiv(m, 32) * cdiv(n, 32) * batch;
  const int64_t bm = m <= 1 ? 1 : m <= 2 ? 2 : m <= 4 ? 4 : 8, bn = bm < 8 ? 16 : 8;
  const int64_t tiles_f = (int64_t)cdiv(m, bm) * cdiv(n, bn) * batch;
  const bool fits = cdiv(n, bn) <= 65535u && (int64_t)cdiv(m, bm) * 8 <= 0x7fffffff;
  bool fine = sizeof(T) == 8 ? cdiv(tiles64, sms) * 4096.0 > cdiv(tiles_f, sms) * (double)(bm * bn) * 1.05
                             : 4 * tiles32 <= sms;
  if (sizeof(T) == 8 && fine) fine = fine_pays(m, n, k, batch, bm, bn, sms);
  if (fine && fits) {
    if (bm == 1)
      return launch_fine<T, 1, 16>(ctx, opa, opb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch);
    if (bm == 2)
      return launch_fine<T, 2, 16>(ctx, opa, opb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch);
    if (bm == 4)
      return launch_fine<T, 4, 16>(ctx, opa, opb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch);
    return launch_fine<T, 8, 8>(ctx, opa, opb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch);
  }
  if constexpr (sizeof(T) == 4) {
    if (gemm_f32_views_pays(ctx, m, n, batch))
      return gemm_f32_views(ctx, m, n, k, alpha, A, matrix_view(opa, lda), sA, B, matrix_view(opb, ldb), sB, beta, C, ldc,
                            sC, batch);
  }
  // a few rows against wide operands (batched amplitudes, environment rows): row tiles
  // of 8 / 16 so the DFMA work is not spent on padding
  if (m <= 8 && n >= 64)
    return launch<T, 8, 32, 8, 1, 1>(ctx, opa, opb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch);
  if (m <= 16 && n >= 64)
    return launch<T, 16, 32, 8, 2, 1>(ctx, opa, opb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch);
  if (tiles64 >= sms)
    return launch<T, 64, 64, 8, 4, 4>(ctx, opa, opb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C,
                                      ldc, sC, batch);
  return launch<T, 32, 32, 8, 2, 2>(ctx, opa, opb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C,
                                    ldc, sC, batch);
}

// C = Aᴴ A (k × n input, n × n Hermitian output, batched): the tiles on and above the
// diagonal by the GEMM kernel, the rest mirrored
template <typename T>
tn_status_t herk_cx(tn_ctx* ctx, int64_t n, int64_t k, const cx<T>* A, int64_t lda, int64_t sA, cx<T>* C, int64_t ldc,
                    int64_t sC, int64_t batch) {
  if (n == 0 || batch == 0) return TN_OK;
  const cx<T> one = mkcx<T>(1, 0), zero = mkcx<T>(0, 0);
  const int64_t tiles64 = (int64_t)cdiv(n, 64) * cdiv(n, 64) * batch;
  if (tiles64 >= 2 * ctx->num_sms)
    TN_RETURN_IF((launch<T, 64, 64, 8, 4, 4>(ctx, 'C', 'N', n, n, k, one, A, lda, sA, A, lda, sA, zero, C, ldc, sC,
                                              batch, true)));
  else
    TN_RETURN_IF((launch<T, 32, 32, 8, 2, 2>(ctx, 'C', 'N', n, n, k, one, A, lda, sA, A, lda, sA, zero, C, ldc, sC,
                                              batch, true)));
  const int64_t blocks = std::min<int64_t>((n * n + 255) / 256, 2048);
  k_mirror_lower<T><<<dim3((unsigned)blocks, (unsigned)(batch < 65535 ? batch : 65535)), 256, 0, ctx->stream>>>(
      n, C, ldc, sC, batch);
  TN_LAUNCHED(ctx);
  return TN_OK;
}
template tn_status_t herk_cx<double>(tn_ctx*, int64_t, int64_t, const cxd*, int64_t, int64_t, cxd*, int64_t, int64_t,
                                     int64_t);

template tn_status_t gemm_cx<double>(tn_ctx*, char, char, int64_t, int64_t, int64_t, cxd,
                                     const cxd*, int64_t, int64_t, const cxd*, int64_t, int64_t,
                                     cxd, cxd*, int64_t, int64_t, int64_t);
template tn_status_t gemm_cx<float>(tn_ctx*, char, char, int64_t, int64_t, int64_t, cxf,
                                    const cxf*, int64_t, int64_t, const cxf*, int64_t, int64_t,
                                    cxf, cxf*, int64_t, int64_t, int64_t);

// real GEMMs reuse the complex kernel through a zero-imaginary copy would waste half the
// work; they go through a dedicated real kernel below.
namespace {
template <typename T, int BM, int BN, int BK, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
    k_gemm_re(char opa, char opb, int64_t m, int64_t n, int64_t k, T alpha, const T* __restrict__ A,
              int64_t lda, int64_t sA, const T* __restrict__ B, int64_t ldb, int64_t sB, T beta,
              T* __restrict__ C, int64_t ldc, int64_t sC, int64_t batch) {
  constexpr int NT = (BM / TM) * (BN / TN);
  constexpr int RX = BN / TN, RY = BM / TM;
  __shared__ T As[BK][BM + 1];
  __shared__ T Bs[BK][BN + 1];
  const int tid = threadIdx.x, tx = tid % RX, ty = tid / RX;
  const int64_t i0 = (int64_t)blockIdx.x * BM, j0 = (int64_t)blockIdx.y * BN;
  for (int64_t bz = blockIdx.z; bz < batch; bz += gridDim.z) {
    const T* Ab = A + bz * sA;
    const T* Bb = B + bz * sB;
    T* Cb = C + bz * sC;
    T acc[TM][TN] = {};
    for (int64_t p0 = 0; p0 < k; p0 += BK) {
      for (int t = tid; t < BM * BK; t += NT) {
        int ii = opa == 'N' ? t % BM : t / BK, pp = opa == 'N' ? t / BM : t % BK;
        int64_t gi = i0 + ii, gp = p0 + pp;
        As[pp][ii] = (gi < m && gp < k) ? (opa == 'N' ? Ab[gi + gp * lda] : Ab[gp + gi * lda]) : T(0);
      }
      for (int t = tid; t < BK * BN; t += NT) {
        int pp = opb == 'N' ? t % BK : t / BN, jj = opb == 'N' ? t / BK : t % BN;
        int64_t gp = p0 + pp, gj = j0 + jj;
        Bs[pp][jj] = (gp < k && gj < n) ? (opb == 'N' ? Bb[gp + gj * ldb] : Bb[gj + gp * ldb]) : T(0);
      }
      __syncthreads();
#pragma unroll
      for (int pp = 0; pp < BK; ++pp)
#pragma unroll
        for (int r = 0; r < TM; ++r)
#pragma unroll
          for (int c = 0; c < TN; ++c) acc[r][c] = fma(As[pp][ty + r * RY], Bs[pp][tx + c * RX], acc[r][c]);
      __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < TM; ++r) {
      int64_t gi = i0 + ty + r * RY;
      if (gi >= m) continue;
#pragma unroll
      for (int c = 0; c < TN; ++c) {
        int64_t gj = j0 + tx + c * RX;
        if (gj >= n) continue;
        T v = alpha * acc[r][c];
        if (beta != T(0)) v += beta * Cb[gi + gj * ldc];
        Cb[gi + gj * ldc] = v;
      }
    }
  }
}
}  // namespace

template <typename T>
static tn_status_t gemm_re(tn_ctx* ctx, char opa, char opb, int64_t m, int64_t n, int64_t k, T alpha,
                           const T* A, int64_t lda, int64_t sA, const T* B, int64_t ldb, int64_t sB,
                           T beta, T* C, int64_t ldc, int64_t sC, int64_t batch) {
  if (m == 0 || n == 0 || batch == 0) return TN_OK;
  dim3 grid(cdiv(m, 64), cdiv(n, 64), (unsigned)(batch < 65535 ? batch : 65535));
  k_gemm_re<T, 64, 64, 16, 4, 4><<<grid, 256, 0, ctx->stream>>>(opa, opb, m, n, k, alpha, A, lda, sA, B,
                                                                ldb, sB, beta, C, ldc, sC, batch);
  TN_LAUNCHED(ctx);
  return TN_OK;
}

static bool valid_op(char c) { return c == 'N' || c == 'T' || c == 'C'; }

// The tensor path pays an operand-preparation pass (split + 4M expansion) and 128×128
// tiles; skinny GEMMs (any of m, n < 64 or k < 32) are HBM-bound and stay on the FP32
// CUDA cores, which are also the more accurate choice.
bool gemm_on_tensor_pipe(tn_dtype_t dt, tn_precision_t prec, int64_t m, int64_t n, int64_t k) {
  return (dt == TN_C32 || dt == TN_F32) && prec != TN_PREC_NATIVE && m >= 64 && n >= 64 && k >= 32;
}

size_t gemm_any_workspace(tn_dtype_t dt, tn_precision_t prec, int64_t m, int64_t n, int64_t k) {
  if (gemm_on_tensor_pipe(dt, prec, m, n, k)) return tc_gemm_workspace(dt == TN_C32, prec == TN_PREC_TF32 ? 1 : 3, m, n, k);
  return 0;
}

tn_status_t gemm_any(tn_ctx* ctx, tn_dtype_t dtype, tn_precision_t prec, char opa, char opb, int64_t m, int64_t n,
                     int64_t k, const double* alpha, const void* A, int64_t lda, int64_t strideA, const void* B,
                     int64_t ldb, int64_t strideB, const double* beta, void* C, int64_t ldc, int64_t strideC,
                     int64_t batch) {
  const bool tc = gemm_on_tensor_pipe(dtype, prec, m, n, k);
  if (tc) {
    if (dtype == TN_C32 && (alpha[1] != 0.0 || beta[1] != 0.0))
      return tn_set_error(ctx, TN_EUNSUPPORTED, "tensor-core GEMM: complex alpha/beta not supported");
    const int passes = prec == TN_PREC_TF32 ? 1 : 3;
    const size_t es = dtype == TN_C32 ? 8 : 4;
    const size_t top = ctx->ws_top;
    const GemmView va = matrix_view(opa, lda), vb = matrix_view(opb, ldb);
    // (read in place: C over an operand of its product is left to the general path, which copies)
    const size_t na = es * (size_t)(opa == 'N' ? (k - 1) * lda + m : (m - 1) * lda + k),
                 nb = es * (size_t)(opb == 'N' ? (n - 1) * ldb + k : (k - 1) * ldb + n), nc = es * (size_t)((n - 1) * ldc + m);
    bool apart = true;
    for (int64_t b = 0; b < batch && apart; ++b) {
      const char *a = (const char*)A + es * (size_t)(b * strideA), *x = (const char*)B + es * (size_t)(b * strideB),
                 *c = (const char*)C + es * (size_t)(b * strideC);
      apart = !ranges_meet(c, nc, a, na) && !ranges_meet(c, nc, x, nb);
    }
    if (dtype == TN_C32 && apart && tc_gemm_tall_fits(ctx, m, n, k, va)) {
      for (int64_t b = 0; b < batch; ++b)
        TN_RETURN_IF(tc_gemm_tall(ctx, passes, m, n, k, (float)alpha[0], (const cxf*)A + b * strideA, va,
                                  (const cxf*)B + b * strideB, vb, (float)beta[0], (cxf*)C + b * strideC, ldc));
      return TN_OK;
    }
    for (int64_t b = 0; b < batch; ++b) {
      ctx->ws_top = top;
      TN_RETURN_IF(tc_gemm(ctx, dtype == TN_C32, passes, opa, opb, m, n, k, (float)alpha[0],
                           (const char*)A + es * b * strideA, lda, (const char*)B + es * b * strideB, ldb, (float)beta[0],
                           (char*)C + es * b * strideC, ldc));
    }
    ctx->ws_top = top;
    return TN_OK;
  }
  switch (dtype) {
    case TN_C64: {
      cxd a = mkcx(alpha[0], alpha[1]), b = mkcx(beta[0], beta[1]);
      return gemm_c64(ctx, prec, opa, opb, m, n, k, a, (const cxd*)A, lda, strideA, (const cxd*)B, ldb, strideB, b,
                      (cxd*)C, ldc, strideC, batch);
    }
    case TN_C32: {
      cxf a = mkcx((float)alpha[0], (float)alpha[1]), b = mkcx((float)beta[0], (float)beta[1]);
      return gemm_cx<float>(ctx, opa, opb, m, n, k, a, (const cxf*)A, lda, strideA, (const cxf*)B, ldb, strideB, b,
                            (cxf*)C, ldc, strideC, batch);
    }
    case TN_F64:
      return gemm_re<double>(ctx, opa, opb, m, n, k, alpha[0], (const double*)A, lda, strideA, (const double*)B, ldb,
                             strideB, beta[0], (double*)C, ldc, strideC, batch);
    case TN_F32:
      return gemm_re<float>(ctx, opa, opb, m, n, k, (float)alpha[0], (const float*)A, lda, strideA, (const float*)B,
                            ldb, strideB, (float)beta[0], (float*)C, ldc, strideC, batch);
  }
  return tn_set_error(ctx, TN_EINVAL, "gemm: bad dtype");
}

extern "C" tn_status_t tn_gemm(tn_ctx* ctx, tn_dtype_t dtype, tn_precision_t prec, char opa, char opb,
                               int64_t m, int64_t n, int64_t k, const double* alpha, const void* A,
                               int64_t lda, int64_t strideA, const void* B, int64_t ldb,
                               int64_t strideB, const double* beta, void* C, int64_t ldc,
                               int64_t strideC, int64_t batch) {
  if (!ctx) return TN_EINVAL;
  TN_ARG(ctx, valid_op(opa) && valid_op(opb), "tn_gemm: op must be 'N', 'T' or 'C'");
  TN_ARG(ctx, m >= 0 && n >= 0 && k >= 0 && batch >= 0, "tn_gemm: negative size");
  TN_ARG(ctx, alpha && beta, "tn_gemm: null alpha/beta");
  TN_ARG(ctx, (m == 0 || n == 0 || batch == 0) || (A && B && C), "tn_gemm: null matrix");
  TN_ARG(ctx, dtype_complex(dtype) || (opa != 'C' && opb != 'C'), "tn_gemm: 'C' needs a complex dtype");
  int64_t ra = opa == 'N' ? m : k, rb = opb == 'N' ? k : n;
  TN_ARG(ctx, lda >= (ra > 1 ? ra : 1) && ldb >= (rb > 1 ? rb : 1) && ldc >= (m > 1 ? m : 1),
         "tn_gemm: leading dimension too small");
  TN_RETURN_IF(ws_reserve(ctx, gemm_any_workspace(dtype, prec, m, n, k)));
  TN_RETURN_IF(gemm_any(ctx, dtype, prec, opa, opb, m, n, k, alpha, A, lda, strideA, B, ldb, strideB, beta, C, ldc,
                        strideC, batch));
  return split_gemm_check(ctx);
}

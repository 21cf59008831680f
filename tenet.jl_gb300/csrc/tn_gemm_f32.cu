// K2d — ComplexF32 GEMM on the FP32 pipe for products with tall outputs, operands read through
// strided views.
//
//   C[m, n] = alpha · Σ_k A[m, k]·B[k, n] + beta · C     (C column-major, A and B views)
//
// Bound: FP32 issue.  A 64×64 tile with 4×4 outputs per thread (k_gemm_cx) spends as many
// instructions on shared-memory loads and scalar FMAs as the pipe has slots; here a thread
// holds 8×8 outputs of a 128×64 tile (with 8×4 the shared-memory loads took as long as the
// FMAs), rows in pairs, so one fma.rn.f32x2 does two rows, operands
// sit in shared memory as the instruction wants them (A split into Re and Im planes, B's
// parts doubled), and the next stage of K is fetched to registers under the current one.
// A view maps an index to an offset by two levels (inner extent, inner and outer stride), so
// a tensor whose contracted legs lie between free ones is read in place instead of being
// permuted first: two legs fused are one level.
// The sum over k runs in index order with the same two FMAs per part as k_gemm_cx: the
// results are the same bits.
#include <algorithm>

#include "tn_internal.cuh"

namespace {

typedef unsigned long long f2;
__device__ __forceinline__ f2 f2_pack(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2_unpack(f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

constexpr int BM = 128, BN = 64, BK = 8, NT = 128;
constexpr int LA = BM * BK / NT, LB = BN * BK / NT;  // entries a thread stages

__device__ __forceinline__ int64_t at(const IndexView& v, int64_t i) {
  if (v.outer == 0) return i * v.inner;
  const unsigned n = (unsigned)v.extent, q = (unsigned)i / n;  // (extents below 2³¹ with an outer level)
  return (int64_t)((unsigned)i - q * n) * v.inner + (int64_t)q * v.outer;
}

__global__ void __launch_bounds__(NT, 2)
    k_gemm_f32_views(int64_t m, int64_t n, int64_t k, cxf alpha, const cxf* __restrict__ A, GemmView va, int64_t sA,
                     const cxf* __restrict__ B, GemmView vb, int64_t sB, cxf beta, cxf* __restrict__ C, int64_t ldc,
                     int64_t sC, int64_t batch) {
  __shared__ __align__(16) float Ar[2][BK][BM], Ai[2][BK][BM];
  __shared__ float4 Bs[2][BK][BN];  // (Re, Re, Im, Im)
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
  const int64_t i0 = (int64_t)blockIdx.x * BM, j0 = (int64_t)blockIdx.y * BN;
  // staging: along the index that is contiguous in memory
  const bool a_rows = va.row.inner == 1, b_cols = vb.col.inner == 1 && vb.row.inner != 1;
  for (int64_t bz = blockIdx.z; bz < batch; bz += gridDim.z) {
    const cxf* Ab = A + bz * sA;
    const cxf* Bb = B + bz * sB;
    int64_t ao[LA], bo[LB];
    auto a_i = [&](int u) { return a_rows ? tid : tid / BK + u * (NT / BK); };
    auto a_p = [&](int u) { return a_rows ? u : tid % BK; };
    auto b_j = [&](int u) { return b_cols ? tid % BN : tid / BK + u * (NT / BK); };
    auto b_p = [&](int u) { return b_cols ? tid / BN + u * (NT / BN) : tid % BK; };
#pragma unroll
    for (int u = 0; u < LA; ++u) ao[u] = i0 + a_i(u) < m ? at(va.row, i0 + a_i(u)) : -1;  // (one value when a_rows)
#pragma unroll
    for (int u = 0; u < LB; ++u) bo[u] = j0 + b_j(u) < n ? at(vb.col, j0 + b_j(u)) : -1;
    cxf ra[LA], rb[LB];
    auto fetch = [&](int64_t p0) {
      if (a_rows) {
#pragma unroll
        for (int u = 0; u < LA; ++u)
          ra[u] = (ao[0] >= 0 && p0 + u < k) ? Ab[ao[0] + at(va.col, p0 + u)] : mkcx<float>(0.f, 0.f);
      } else {
        const bool in = p0 + a_p(0) < k;
        const int64_t o = in ? at(va.col, p0 + a_p(0)) : 0;
#pragma unroll
        for (int u = 0; u < LA; ++u) ra[u] = (in && ao[u] >= 0) ? Ab[ao[u] + o] : mkcx<float>(0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < LB; ++u)
        rb[u] = (bo[u] >= 0 && p0 + b_p(u) < k) ? Bb[bo[u] + at(vb.row, p0 + b_p(u))] : mkcx<float>(0.f, 0.f);
    };
    auto stage = [&](int s) {
#pragma unroll
      for (int u = 0; u < LA; ++u) {
        Ar[s][a_p(u)][a_i(u)] = ra[u].x;
        Ai[s][a_p(u)][a_i(u)] = va.conj ? -ra[u].y : ra[u].y;
      }
#pragma unroll
      for (int u = 0; u < LB; ++u) {
        const float y = vb.conj ? -rb[u].y : rb[u].y;
        Bs[s][b_p(u)][b_j(u)] = make_float4(rb[u].x, rb[u].x, y, y);
      }
    };
    f2 re[4][8], im[4][8];  // [row pair][column]
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 8; ++c) re[r][c] = im[r][c] = 0ull;
    if (k > 0) {
      fetch(0);
      stage(0);
    }
    __syncthreads();
    int s = 0;
    for (int64_t p0 = 0; p0 < k; p0 += BK, s ^= 1) {
      const bool more = p0 + BK < k;
      if (more) fetch(p0 + BK);
#pragma unroll
      for (int pp = 0; pp < BK; ++pp) {
        f2 ar[4], ay[4], an[4];
        const float4 r0 = *reinterpret_cast<const float4*>(&Ar[s][pp][ty * 8]), r1 = *reinterpret_cast<const float4*>(&Ar[s][pp][ty * 8 + 4]);
        const float4 y0 = *reinterpret_cast<const float4*>(&Ai[s][pp][ty * 8]), y1 = *reinterpret_cast<const float4*>(&Ai[s][pp][ty * 8 + 4]);
        ar[0] = f2_pack(r0.x, r0.y);
        ar[1] = f2_pack(r0.z, r0.w);
        ar[2] = f2_pack(r1.x, r1.y);
        ar[3] = f2_pack(r1.z, r1.w);
        ay[0] = f2_pack(y0.x, y0.y);
        ay[1] = f2_pack(y0.z, y0.w);
        ay[2] = f2_pack(y1.x, y1.y);
        ay[3] = f2_pack(y1.z, y1.w);
#pragma unroll
        for (int r = 0; r < 4; ++r) an[r] = ay[r] ^ 0x8000000080000000ull;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float4 b = Bs[s][pp][tx + 8 * c];
          const f2 br = f2_pack(b.x, b.y), bi = f2_pack(b.z, b.w);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            re[r][c] = f2_fma(ar[r], br, re[r][c]);
            re[r][c] = f2_fma(an[r], bi, re[r][c]);
            im[r][c] = f2_fma(ar[r], bi, im[r][c]);
            im[r][c] = f2_fma(ay[r], br, im[r][c]);
          }
        }
      }
      if (more) stage(s ^ 1);
      __syncthreads();
    }
    const bool beta0 = beta.x == 0.f && beta.y == 0.f;
    cxf* Cb = C + bz * sC;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int64_t gj = j0 + tx + 8 * c;
      if (gj >= n) continue;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        cxf v[2];
        f2_unpack(re[r][c], v[0].x, v[1].x);
        f2_unpack(im[r][c], v[0].y, v[1].y);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int64_t gi = i0 + ty * 8 + 2 * r + h;
          if (gi >= m) continue;
          cxf o = alpha * v[h];
          if (!beta0) o = o + beta * Cb[gi + gj * ldc];
          Cb[gi + gj * ldc] = o;
        }
      }
    }
    __syncthreads();
  }
}

}  // namespace

// Enough 128 × 64 tiles to occupy the chip, and not mostly padding; below that the 64 × 64 and
// smaller tiles of gemm_cx spread the product further.
bool gemm_f32_views_pays(tn_ctx* ctx, int64_t m, int64_t n, int64_t batch) {
  return m >= 96 && n >= 32 && (int64_t)cdiv(m, BM) * cdiv(n, BN) * batch >= 2 * ctx->num_sms;
}

tn_status_t gemm_f32_views(tn_ctx* ctx, int64_t m, int64_t n, int64_t k, cxf alpha, const cxf* A, const GemmView& va,
                           int64_t sA, const cxf* B, const GemmView& vb, int64_t sB, cxf beta, cxf* C, int64_t ldc,
                           int64_t sC, int64_t batch) {
  if (m == 0 || n == 0 || batch == 0) return TN_OK;
  const int64_t gx = (m + BM - 1) / BM, gy = (n + BN - 1) / BN;
  if (gx > 0x7fffffff || gy > 65535) return tn_set_error(ctx, TN_EINVAL, "gemm: grid too large");
  const dim3 grid((unsigned)gx, (unsigned)gy, (unsigned)std::min<int64_t>(batch, 65535));
  k_gemm_f32_views<<<grid, NT, 0, ctx->stream>>>(m, n, k, alpha, A, va, sA, B, vb, sB, beta, C, ldc, sC, batch);
  TN_LAUNCHED(ctx);
  return TN_OK;
}

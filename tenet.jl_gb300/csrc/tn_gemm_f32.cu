// K2d — ComplexF32 GEMM on the FP32 pipe for products with tall outputs, operands read through
// strided views.
//
//   C[m, n] = alpha · Σ_k A[m, k]·B[k, n] + beta · C     (C column-major, A and B views)
//
// Bound: FP32 issue.  A 64×64 tile with 4×4 outputs per thread (k_gemm_cx) spends as many
// instructions on shared-memory loads and scalar FMAs as the pipe has slots; here a thread
// holds 4 rows, in pairs, × 4 to 8 columns, so one fma.rn.f32x2 does two rows, operands sit in
// shared memory as the instruction wants them (A split into Re and Im planes, B's parts doubled),
// and the next stage of K is fetched to registers under the current one.  256 threads of at
// most 128 registers keep four warps on a scheduler; with 8 × 8 outputs, 255 registers and half the
// warps, the shared-memory latency showed (117649 × 49 × 49: 128 → 97 µs).  The columns per thread
// are the fewest that hold n in as many tiles as 64 would take, and the last stage of K
// runs over what is left of k only, so that a bond of 7 pays for 56 columns, not 64, and no padded k.
// A view maps an index to an offset by two levels (inner extent, inner and outer stride), so a
// tensor whose contracted legs lie between free ones is read in place instead of being permuted
// first: two legs fused are one level.  The offsets of the contracted index come from a table in
// shared memory, KT at a time.
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

constexpr int BM = 128, BK = 8, NT = 256;
constexpr int LA = BM * BK / NT;  // entries of A a thread stages
constexpr int KT = 256;           // (a multiple of BK)

__device__ __forceinline__ int64_t at(const IndexView& v, int64_t i) {
  if (v.outer == 0) return i * v.inner;
  const unsigned n = (unsigned)v.extent, q = (unsigned)i / n;  // (extents below 2³¹ with an outer level)
  return (int64_t)((unsigned)i - q * n) * v.inner + (int64_t)q * v.outer;
}

template <int CC>
__global__ void __launch_bounds__(NT, 2)
    k_gemm_f32_views(int64_t m, int64_t n, int64_t k, cxf alpha, const cxf* __restrict__ A, GemmView va, int64_t sA,
                     const cxf* __restrict__ B, GemmView vb, int64_t sB, cxf beta, cxf* __restrict__ C, int64_t ldc,
                     int64_t sC, int64_t batch) {
  constexpr int BN = 8 * CC, LB = (BN * BK + NT - 1) / NT;
  // (a row of 4 floats or one entry more than the tile: staged along k, 8 rows fall on 8 banks)
  __shared__ __align__(16) float Ar[2][BK][BM + 4], Ai[2][BK][BM + 4];
  __shared__ float4 Bs[2][BK][BN + 1];  // (Re, Re, Im, Im)
  __shared__ int64_t ka[KT], kb[KT];  // the offsets of KT contracted indices (−1 beyond k)
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
  const int64_t i0 = (int64_t)blockIdx.x * BM, j0 = (int64_t)blockIdx.y * BN;
  // staging: along the index that is contiguous in memory
  const bool a_rows = va.row.inner == 1, b_cols = vb.col.inner == 1 && vb.row.inner != 1;
  for (int64_t bz = blockIdx.z; bz < batch; bz += gridDim.z) {
    const cxf* Ab = A + bz * sA;
    const cxf* Bb = B + bz * sB;
    int64_t ao[LA], bo[LB];
    auto a_i = [&](int u) { return a_rows ? tid % BM : tid / BK + u * (NT / BK); };
    auto a_p = [&](int u) { return a_rows ? tid / BM + u * (NT / BM) : tid % BK; };
    auto b_j = [&](int u) { return b_cols ? (tid + u * NT) % BN : tid / BK + u * (NT / BK); };
    auto b_p = [&](int u) { return b_cols ? (tid + u * NT) / BN : tid % BK; };
#pragma unroll
    for (int u = 0; u < LA; ++u) ao[u] = i0 + a_i(u) < m ? at(va.row, i0 + a_i(u)) : -1;  // (one value when a_rows)
#pragma unroll
    for (int u = 0; u < LB; ++u) bo[u] = (b_j(u) < BN && b_p(u) < BK && j0 + b_j(u) < n) ? at(vb.col, j0 + b_j(u)) : -1;
    cxf ra[LA], rb[LB];
    auto fetch = [&](int64_t p0) {
      const int t = (int)(p0 % KT);
      if (t == 0) {
        __syncthreads();
        for (int q = tid; q < KT; q += NT) {
          ka[q] = p0 + q < k ? at(va.col, p0 + q) : -1;
          kb[q] = p0 + q < k ? at(vb.row, p0 + q) : -1;
        }
        __syncthreads();
      }
#pragma unroll
      for (int u = 0; u < LA; ++u) {
        const int64_t o = ka[t + a_p(u)], r = ao[a_rows ? 0 : u];
        ra[u] = (o >= 0 && r >= 0) ? Ab[r + o] : mkcx<float>(0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < LB; ++u) {
        const int64_t o = bo[u] >= 0 ? kb[t + b_p(u)] : -1;
        rb[u] = o >= 0 ? Bb[bo[u] + o] : mkcx<float>(0.f, 0.f);
      }
    };
    auto stage = [&](int s) {
#pragma unroll
      for (int u = 0; u < LA; ++u) {
        Ar[s][a_p(u)][a_i(u)] = ra[u].x;
        Ai[s][a_p(u)][a_i(u)] = va.conj ? -ra[u].y : ra[u].y;
      }
#pragma unroll
      for (int u = 0; u < LB; ++u)
        if (b_j(u) < BN && b_p(u) < BK) {
          const float y = vb.conj ? -rb[u].y : rb[u].y;
          Bs[s][b_p(u)][b_j(u)] = make_float4(rb[u].x, rb[u].x, y, y);
        }
    };
    f2 re[2][CC], im[2][CC];  // [row pair][column]
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int c = 0; c < CC; ++c) re[r][c] = im[r][c] = 0ull;
    if (k > 0) {
      fetch(0);
      stage(0);
    }
    __syncthreads();
    auto step = [&](int s, int pp) {
      const float4 x = *reinterpret_cast<const float4*>(&Ar[s][pp][ty * 4]), y = *reinterpret_cast<const float4*>(&Ai[s][pp][ty * 4]);
      const f2 ar[2] = {f2_pack(x.x, x.y), f2_pack(x.z, x.w)}, ay[2] = {f2_pack(y.x, y.y), f2_pack(y.z, y.w)};
      const f2 an[2] = {ay[0] ^ 0x8000000080000000ull, ay[1] ^ 0x8000000080000000ull};
#pragma unroll
      for (int c = 0; c < CC; ++c) {
        const float4 b = Bs[s][pp][tx + 8 * c];
        const f2 br = f2_pack(b.x, b.y), bi = f2_pack(b.z, b.w);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          re[r][c] = f2_fma(ar[r], br, re[r][c]);
          re[r][c] = f2_fma(an[r], bi, re[r][c]);
          im[r][c] = f2_fma(ar[r], bi, im[r][c]);
          im[r][c] = f2_fma(ay[r], br, im[r][c]);
        }
      }
    };
    int s = 0;
    for (int64_t p0 = 0; p0 < k; p0 += BK, s ^= 1) {
      const bool more = p0 + BK < k;
      if (more) fetch(p0 + BK);
      if (p0 + BK <= k) {
#pragma unroll
        for (int pp = 0; pp < BK; ++pp) step(s, pp);
      } else {  // what is left of k, without its padding
#pragma unroll 1
        for (int pp = 0; pp < (int)(k - p0); ++pp) step(s, pp);
      }
      if (more) stage(s ^ 1);
      __syncthreads();
    }
    const bool beta0 = beta.x == 0.f && beta.y == 0.f;
    cxf* Cb = C + bz * sC;
#pragma unroll
    for (int c = 0; c < CC; ++c) {
      const int64_t gj = j0 + tx + 8 * c;
      if (gj >= n) continue;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        cxf v[2];
        f2_unpack(re[r][c], v[0].x, v[1].x);
        f2_unpack(im[r][c], v[0].y, v[1].y);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int64_t gi = i0 + ty * 4 + 2 * r + h;
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

// columns a thread holds (4 … 8, tiles of 32 … 64): as many tiles as with 64 columns, of the
// fewest columns that hold n
int columns_per_thread(int64_t n) {
  const int64_t tiles = (n + 63) / 64;
  return (int)std::max<int64_t>(4, ((n + tiles - 1) / tiles + 7) / 8);
}

}  // namespace

// Enough 128 × 64 tiles to occupy the chip, and not mostly padding; below that the 64 × 64 and
// smaller tiles of gemm_cx spread the product further.
bool gemm_f32_views_pays(tn_ctx* ctx, int64_t m, int64_t n, int64_t batch) {
  return m >= 96 && n >= 32 && (int64_t)cdiv(m, BM) * cdiv(n, 64) * batch >= 2 * ctx->num_sms;
}

tn_status_t gemm_f32_views(tn_ctx* ctx, int64_t m, int64_t n, int64_t k, cxf alpha, const cxf* A, const GemmView& va,
                           int64_t sA, const cxf* B, const GemmView& vb, int64_t sB, cxf beta, cxf* C, int64_t ldc,
                           int64_t sC, int64_t batch) {
  if (m == 0 || n == 0 || batch == 0) return TN_OK;
  const int64_t gx = (m + BM - 1) / BM, gy = (n + 63) / 64;
  if (gx > 0x7fffffff || gy > 65535) return tn_set_error(ctx, TN_EINVAL, "gemm: grid too large");
  const dim3 grid((unsigned)gx, (unsigned)gy, (unsigned)std::min<int64_t>(batch, 65535));
  auto* kernel = k_gemm_f32_views<8>;
  switch (columns_per_thread(n)) {
    case 4: kernel = k_gemm_f32_views<4>; break;
    case 5: kernel = k_gemm_f32_views<5>; break;
    case 6: kernel = k_gemm_f32_views<6>; break;
    case 7: kernel = k_gemm_f32_views<7>; break;
  }
  kernel<<<grid, NT, 0, ctx->stream>>>(m, n, k, alpha, A, va, sA, B, vb, sB, beta, C, ldc, sC, batch);
  TN_LAUNCHED(ctx);
  return TN_OK;
}

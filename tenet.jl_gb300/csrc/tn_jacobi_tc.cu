// K4f — block round of the FP32 pre-pass on the tensor pipe (truncated and untruncated mixed
// SVD; n, m ≤ 512).
//
// What bounds the register form (k_jacobi_block_f32): every pair of a 16-column block pair is
// an inner product over all rows, a block-wide barrier and a rotation of all rows of W and V,
// a chain of 8 such steps per 64 pairs, 63 launches per sweep at n = 512.  Here a block pair
// has 32 columns and the rows are touched by matrix products only:
//   G = WᴴW (32 × 32),  J = the unitary of one cyclic sweep over G's pairs,  W ← W·J,  V ← V·J.
// The rotations are formed and applied on G in shared memory, by the same rules (threshold,
// truncation-aware tail, numerically zero columns, counters) as the other FP32 rounds; each
// column pair is visited once per sweep.  31 launches per sweep at n = 512, and a block pair
// in which nothing rotates leaves W and V untouched.
//
// Products.  kind::tf32 with operands split x = hi + lo (hi: x rounded to TF32, lo the exact
// remainder), FP32 accumulation in TMEM.  The rows are taken 128 at a time; a thread owns a row
// and half of the columns (warp w reads the TMEM lanes of its own rows) and writes the
// operand tiles itself, K-major with the 128-byte swizzle:
//  * G: per 128 rows a tile of 128 × 128 whose rows 0-63 are the hi parts of the 64 real
//    columns [Re | Im] and rows 64-127 the lo parts, multiplied by its own first 64 rows:
//    one M = 128, N = 64 product gives hi·hi and lo·hi, and G = HH + LH + LHᵀ.  Each 128 rows
//    have their own accumulator; they are added in FP32.
//  * W·J, V·J: per 128 rows A (rows × 64 real columns) hi and lo against the 64 × 64 real form
//    of J: hi·[hi | lo] and lo·[hi | lo] as products of N = 128, the halves added in FP32 (products of
//    N = 64 take the tensor pipe nearly as long).  All products into an accumulator have one
//    shape: only those are executed in the order of issue.
// One 64 KB operand buffer, which between the products also holds G and J, leaves room for two
// CTAs per SM: one's rotations run under the other's products and memory traffic.
// A round of 16 matrices of n = 512 takes 44 µs (47 with J's hi and lo parts as products of their
// own); of a CTA's 73 thousand clocks the products of W and V take 35, the rotations 21, G 15.
// Error: ~1e-6 of ‖wᵢ‖‖wⱼ‖ in G, below the pre-pass's rotation threshold (4√m·2⁻²³, 1e-5 at
// m = 512); what it leaves is removed by the FP64 stage that follows every pre-pass.
#include <cuda.h>

#include <algorithm>

#include "tn_internal.cuh"

namespace {

constexpr int kC = 32;  // columns of a block pair
constexpr int kNT = 256;
constexpr int kBufBytes = 64 * 1024;
constexpr long long kSpin = 1ll << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity, int* err) {  // bounded
  for (long long i = 0; i < kSpin; ++i) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok)
                 : "r"(smem_u32(bar)), "r"(parity)
                 : "memory");
    if (ok) return;
  }
  atomicExch(err, 1);
}
// shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1024 B apart
__device__ __forceinline__ uint64_t sdesc(uint32_t addr) {
  uint64_t d = (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= 1ull << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= 1ull << 46;
  d |= 2ull << 61;
  return d;
}
// D f32, A and B tf32, both K-major, M = 128, N = 64 or 128
constexpr uint32_t kIdesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(64 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
constexpr uint32_t kIdesc128 = kIdesc + ((uint32_t)(64 >> 3) << 17);
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t accum, uint32_t idesc = kIdesc) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
               "l"(a), "l"(b), "r"(idesc), "r"(accum)
               : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
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
__device__ __forceinline__ float tf32_hi(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}
// byte offset of element (row, k) in a K-major tile of 32 floats per row, 128-byte swizzle
__device__ __forceinline__ uint32_t tile_at(int row, int k) {
  return (uint32_t)((row >> 3) * 1024 + (row & 7) * 128 + ((k * 4) ^ ((row & 7) << 4)));
}
__device__ __forceinline__ void pair_of(int N, int r, int k, int& i, int& j) {
  if (k == 0) {
    i = r % (N - 1);
    j = N - 1;
  } else {
    i = (r + k) % (N - 1);
    j = (r - k + (N - 1)) % (N - 1);
  }
  if (i > j) {
    const int t = i;
    i = j;
    j = t;
  }
}

__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

struct Rot {
  float c, sx, sy, monitor;
  int apply;
};
// The rotation that diagonalises [[α, γ], [γ*, β]] in FP32: with ρ = γ/√(αβ) and
// δ = (β − α)/√(αβ), t = 2|ρ|·sgn(δ)/(|δ| + √(δ² + 4|ρ|²)) from approximate roots and quotients,
// then c and s scaled by 1 − (c² + |s|² − 1)/2, whose residual is formed exactly enough by FMAs
// to leave no drift of the columns' norms.
__device__ __forceinline__ Rot rotation(float al, float be, float gx, float gy, float tol, float negl) {
  Rot R = {1.f, 0.f, 0.f, 0.f, 0};
  const float fl = fmaxf(negl, 1e-32f);
  if (!(al > fl) || !(be > fl)) return R;
  const float ra = rsqrt_approx(al), rb = rsqrt_approx(be);
  const float px = gx * ra * rb, py = gy * ra * rb;
  const float rho2 = fmaf(px, px, py * py);
  if (!(rho2 > 1.2e-38f)) return R;  // (below: no normal number, and nothing the threshold would see)
  const float irho = rsqrt_approx(rho2), rho = rho2 * irho;
  R.monitor = rho;
  if (!(rho > tol)) return R;
  const float d = (be - al) * ra * rb, q = fmaf(d, d, 4.f * rho2);
  const float t = copysignf(__fdividef(2.f * rho, fabsf(d) + q * rsqrt_approx(q)), d);
  if (!(fabsf(t) > 0.f)) return R;
  float c = rsqrt_approx(fmaf(t, t, 1.f));
  const float s = c * t * irho;
  float sx = s * px, sy = s * py;
  const float e = -0.5f * fmaf(sy, sy, fmaf(sx, sx, fmaf(c, c, -1.f)));
  R.c = fmaf(c, e, c);
  R.sx = fmaf(sx, e, sx);
  R.sy = fmaf(sy, e, sy);
  R.apply = 1;
  return R;
}

struct Shared {
  uint64_t bar;
  uint32_t tslot;
  int col[kC];
  unsigned char tail[kC];
  int cnt;
};

__global__ void __launch_bounds__(kNT, 2)
    k_jacobi_block_tc(int m, int n, int NB, int R, cxf* __restrict__ W, cxf* __restrict__ V, const float* __restrict__ nrm,
                      const int* __restrict__ active, int* __restrict__ cnt, float tol, const unsigned char* __restrict__ tail,
                      int* err) {
  const int64_t b = blockIdx.y, nmat = gridDim.y;
  if (!active[b]) return;
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* buf = smem;               // operand tiles, 64 KB
  unsigned char* bj = smem + kBufBytes;    // J: hi 2 tiles, lo 2 tiles of 8 KB
  // between the products the operand buffer holds G's parts, G (two copies) and J's rotations
  float* hh = reinterpret_cast<float*>(buf);
  float2(*G)[kC][kC + 1] = reinterpret_cast<float2(*)[kC][kC + 1]>(buf + 2 * 64 * 65 * sizeof(float) + 256);
  float2(*Q)[kC + 1] = G[2];
  Shared& S = *reinterpret_cast<Shared*>(bj + 32768);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, hf = tid >> 7, rloc = tid & 127;
  int P, Qb;
  pair_of(NB, R, blockIdx.x, P, Qb);
  if (tid < kC) {
    const int c = tid < 16 ? P * 16 + tid : Qb * 16 + (tid - 16);
    S.col[tid] = c < n ? c : -1;
    S.tail[tid] = (tail && c < n) ? tail[b * n + c] : 0;
  }
  const int CHm = (m + 127) / 128, CHn = (n + 127) / 128;  // chunks of 128 rows of W, of V (n ≤ m)
  const uint32_t tcols = CHm <= 2 ? 128 : 256;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tslot)), "r"(tcols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 32) {
    mbar_init(&S.bar);
    S.cnt = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = S.tslot;
  const uint32_t tlane = (uint32_t)((warp & 3) * 32) << 16;
  uint32_t parity = 0;  // of the next commit on S.bar (one product in flight at a time)
  cxf* Wb = W + b * (int64_t)m * n;
  cxf* Vb = V + b * (int64_t)n * n;
  // this thread's row and 16 columns of 128 rows of X
  float xr[16], xi[16];
  auto load = [&](const cxf* X, int rows, int chunk) {
    const int row = chunk * 128 + rloc;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const int col = S.col[hf * 16 + c];
      cxf v = mkcx<float>(0.f, 0.f);
      if (col >= 0 && row < rows) v = X[(int64_t)col * rows + row];
      xr[c] = v.x;
      xi[c] = v.y;
    }
  };
  // operand tiles written by all threads → one product by thread 0 → all threads wait
  auto publish = [&]() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  };
  auto finish = [&]() {
    mbar_wait(&S.bar, parity, err);
    parity ^= 1;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  };

  // ---- G: 128 rows as a 128 (hi | lo of the 64 real columns) × 128 operand ----
  load(Wb, m, 0);
  for (int ch = 0; ch < CHm; ++ch) {
    unsigned char* t = buf + (rloc >> 5) * 16384;  // 32 rows of W = one 32-deep K tile
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const int cc = hf * 16 + c;
      const float h = tf32_hi(xr[c]), g = tf32_hi(xi[c]);
      *reinterpret_cast<float*>(t + tile_at(cc, lane)) = h;
      *reinterpret_cast<float*>(t + tile_at(32 + cc, lane)) = g;
      *reinterpret_cast<float*>(t + tile_at(64 + cc, lane)) = xr[c] - h;
      *reinterpret_cast<float*>(t + tile_at(96 + cc, lane)) = xi[c] - g;
    }
    publish();
    if (tid == 0) {
      const uint32_t d = tmem + (uint32_t)(ch * 64);
#pragma unroll 1
      for (int kt = 0; kt < 4; ++kt) {
        const uint64_t a = sdesc(smem_u32(buf + kt * 16384));
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) mma(d, a + 2 * kk, a + 2 * kk, (kt > 0 || kk > 0) ? 1u : 0u);
      }
      mma_commit(&S.bar);
    }
    __syncwarp();
    if (ch + 1 < CHm) load(Wb, m, ch + 1);  // under the product
    finish();
  }
  // HH (lanes 0-63) and LH (lanes 64-127), the chunks' accumulators added; each half of the
  // warps takes 32 of the 64 columns
  {
    const int a = (warp & 3) * 32 + lane;
#pragma unroll 1
    for (int c0 = hf * 32; c0 < hf * 32 + 32; c0 += 16) {
      float s[16], v[16];
      tmem_ld16(tmem + tlane + (uint32_t)c0, s);
      for (int q = 1; q < CHm; ++q) {
        tmem_ld16(tmem + tlane + (uint32_t)(q * 64 + c0), v);
#pragma unroll
        for (int j = 0; j < 16; ++j) s[j] += v[j];
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) hh[(a >> 6) * 64 * 65 + (a & 63) * 65 + c0 + j] = s[j];
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  {
    const float* lh = hh + 64 * 65;
    auto T = [&](int a, int c) { return hh[a * 65 + c] + (lh[a * 65 + c] + lh[c * 65 + a]); };
    for (int e = tid; e < kC * kC; e += kNT) {
      const int i = e & 31, j = e >> 5;
      G[0][i][j] = make_float2(T(i, j) + T(32 + i, 32 + j), T(i, 32 + j) - T(32 + i, j));
      Q[i][j] = make_float2(i == j ? 1.f : 0.f, 0.f);
    }
  }
  __syncthreads();

  // ---- one cyclic sweep over G's pairs (all of them in outer round 0, the cross pairs after):
  // one barrier per round, G alternating between two copies ----
  const float negl = 1.1920929e-7f * 1.1920929e-7f * nrm[n * nmat + b];
  const int rounds = R == 0 ? kC - 1 : 16;
  const unsigned there = __ballot_sync(0xffffffffu, S.col[lane] >= 0), tails = __ballot_sync(0xffffffffu, S.tail[lane] != 0);
  float worst = 0.f;
  int mine = 0, cur = 0;
#pragma unroll 1
  for (int r = 0; r < rounds; ++r) {
    // lanes k and k + 16 of every warp: the rotation of pair k
    Rot rt = {1.f, 0.f, 0.f, 0.f, 0};
    int pi, pj;
    const int k = lane & 15;
    if (R == 0) {
      pair_of(kC, r, k, pi, pj);
    } else {
      pi = k;
      pj = 16 + ((k + r) & 15);
    }
    const bool ti = (tails >> pi) & 1, tj = (tails >> pj) & 1;
    if (((there >> pi) & (there >> pj) & 1) && !(ti && tj)) {
      const float al = G[cur][pi][pi].x, be = G[cur][pj][pj].x;
      const float2 g = G[cur][pi][pj];
      rt = rotation(al, be, g.x, g.y, tol, negl);
      if (ti != tj && al > 0.f && be > 0.f) {
        const float ak = ti ? be : al, at = ti ? al : be;
        rt.monitor *= at / ak;
        if (!(rt.monitor > tol)) {
          rt.apply = 0;
          rt.c = 1.f;
          rt.sx = rt.sy = 0.f;
        }
      }
      if (al > 0.f && be > 0.f) worst = fmaxf(worst, rt.monitor);
      mine += rt.apply;
    }
    if (__ballot_sync(0xffffffffu, rt.apply) != 0) {  // the same in every warp
      const float2(*from)[kC + 1] = G[cur];
      float2(*to)[kC + 1] = G[cur ^ 1];
      // pair q = lane & 15 of this thread: columns a' = c·a − conj(s)·b, b' = s·a + c·b
      auto cols = [&](float2& a, float2& c) {
        const float2 u = make_float2(rt.c * a.x - (rt.sx * c.x + rt.sy * c.y), rt.c * a.y - (rt.sx * c.y - rt.sy * c.x));
        const float2 w = make_float2((rt.sx * a.x - rt.sy * a.y) + rt.c * c.x, (rt.sx * a.y + rt.sy * a.x) + rt.c * c.y);
        a = u;
        c = w;
      };
      {  // G ← Jᴴ G J by 2 × 2 blocks: rows of pair p = tid / 16, columns of pair q
        const int p = tid >> 4;
        const float pc = __shfl_sync(0xffffffffu, rt.c, p), px = __shfl_sync(0xffffffffu, rt.sx, p),
                    py = __shfl_sync(0xffffffffu, rt.sy, p);
        const int p0 = __shfl_sync(0xffffffffu, pi, p), p1 = __shfl_sync(0xffffffffu, pj, p);
        float2 g00 = from[p0][pi], g01 = from[p0][pj], g10 = from[p1][pi], g11 = from[p1][pj];
        cols(g00, g01);
        cols(g10, g11);
        // rows: a' = c·a − s·b, b' = conj(s)·a + c·b
        auto rows = [&](float2& a, float2& c) {
          const float2 u = make_float2(pc * a.x - (px * c.x - py * c.y), pc * a.y - (px * c.y + py * c.x));
          const float2 w = make_float2((px * a.x + py * a.y) + pc * c.x, (px * a.y - py * a.x) + pc * c.y);
          a = u;
          c = w;
        };
        rows(g00, g10);
        rows(g01, g11);
        to[p0][pi] = g00;
        to[p0][pj] = g01;
        to[p1][pi] = g10;
        to[p1][pj] = g11;
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {  // Q ← Q J by rows and pairs
        const int rq = (tid >> 4) + u * 16;
        float2 a = Q[rq][pi], c = Q[rq][pj];
        cols(a, c);
        Q[rq][pi] = a;
        Q[rq][pj] = c;
      }
      cur ^= 1;
      __syncthreads();
    }
  }
  if (warp == 0) {
    int total = lane < 16 ? mine : 0;
    total = (int)__reduce_add_sync(0xffffffffu, (unsigned)total);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) worst = fmaxf(worst, __shfl_xor_sync(0xffffffffu, worst, o));
    if (lane == 0) {
      S.cnt = total;
      if (total) atomicAdd(&cnt[b], total);
      if (worst > 0.f) atomicMax(&cnt[nmat + b], __float_as_int(worst));
    }
  }
  __syncthreads();
  if (S.cnt > 0) {
    load(Wb, m, 0);
    // ---- J in its real 64 × 64 form, B[n][k]: k < 32 and k ≥ 32, of each the hi parts of all n, then lo ----
    for (int e = tid; e < 64 * 64; e += kNT) {
      const int k = e & 63, nn = e >> 6;
      const float2 q = Q[k & 31][nn & 31];
      const float v = (k < 32) == (nn < 32) ? q.x : (nn < 32 ? -q.y : q.y);
      const float h = tf32_hi(v);
      const uint32_t at = (uint32_t)(k >> 5) * 16384 + tile_at(nn, k & 31);
      *reinterpret_cast<float*>(bj + at) = h;
      *reinterpret_cast<float*>(bj + 8192 + at) = v - h;
    }
    __syncthreads();  // Q's place becomes the operand buffer again
    // X ← X·J, 128 rows at a time: W, then V
    const int steps = CHm + CHn;
#pragma unroll 1
    for (int st = 0; st < steps; ++st) {
      const bool is_v = st >= CHm;
      const int ch = is_v ? st - CHm : st;
#pragma unroll
      for (int c = 0; c < 16; c += 4) {
        const uint32_t at = tile_at(rloc, hf * 16 + c);
        float4 h, l;
        h = make_float4(tf32_hi(xr[c]), tf32_hi(xr[c + 1]), tf32_hi(xr[c + 2]), tf32_hi(xr[c + 3]));
        l = make_float4(xr[c] - h.x, xr[c + 1] - h.y, xr[c + 2] - h.z, xr[c + 3] - h.w);
        *reinterpret_cast<float4*>(buf + at) = h;
        *reinterpret_cast<float4*>(buf + 32768 + at) = l;
        h = make_float4(tf32_hi(xi[c]), tf32_hi(xi[c + 1]), tf32_hi(xi[c + 2]), tf32_hi(xi[c + 3]));
        l = make_float4(xi[c] - h.x, xi[c + 1] - h.y, xi[c + 2] - h.z, xi[c + 3] - h.w);
        *reinterpret_cast<float4*>(buf + 16384 + at) = h;
        *reinterpret_cast<float4*>(buf + 49152 + at) = l;
      }
      publish();
      if (tid == 0) {
#pragma unroll
        for (int kt = 0; kt < 2; ++kt) {
          const uint64_t h = sdesc(smem_u32(buf + kt * 16384)), l = sdesc(smem_u32(buf + 32768 + kt * 16384));
          const uint64_t q = sdesc(smem_u32(bj + kt * 16384));
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            mma(tmem, h + 2 * kk, q + 2 * kk, (kt > 0 || kk > 0) ? 1u : 0u, kIdesc128);  // hi·hi | hi·lo
            mma(tmem, l + 2 * kk, q + 2 * kk, 1u, kIdesc128);                             // lo·hi | lo·lo
          }
        }
        mma_commit(&S.bar);
      }
      __syncwarp();
      if (st + 1 < steps) {  // the next rows, under the product
        if (st + 1 < CHm)
          load(Wb, m, st + 1);
        else
          load(Vb, n, st + 1 - CHm);
      }
      finish();
      cxf* X = is_v ? Vb : Wb;
      const int rows = is_v ? n : m, row = ch * 128 + rloc;
      float re[16], im[16], lo[16];
      tmem_ld16(tmem + tlane + (uint32_t)(hf * 16), re);
      tmem_ld16(tmem + tlane + (uint32_t)(64 + hf * 16), lo);
#pragma unroll
      for (int j = 0; j < 16; ++j) re[j] += lo[j];
      tmem_ld16(tmem + tlane + (uint32_t)(32 + hf * 16), im);
      tmem_ld16(tmem + tlane + (uint32_t)(96 + hf * 16), lo);
#pragma unroll
      for (int j = 0; j < 16; ++j) im[j] += lo[j];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int col = S.col[hf * 16 + j];
        if (col >= 0 && row < rows) X[(int64_t)col * rows + row] = mkcx<float>(re[j], im[j]);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tcols) : "memory");
}

constexpr int kSmem = kBufBytes + 32768 + 512;
static_assert(sizeof(Shared) <= 512 && 2 * 64 * 65 * 4 + 256 + 3 * kC * (kC + 1) * 8 <= kBufBytes, "shared memory layout");

}  // namespace

bool jacobi_block_tc_fits(int64_t m, int64_t n) { return m <= 512 && n <= m; }

// outer round r of a sweep over blocks of 16 columns (NB even, ≥ n/16); enqueued on the stream
tn_status_t jacobi_block_tc(tn_ctx* ctx, cudaStream_t stream, int64_t m, int64_t n, int NB, int r, cxf* W, cxf* V,
                            const float* nrm, const int* active, int* rotated, float tol, int64_t batch,
                            const unsigned char* tail) {
  int* err = nullptr;
  TN_RETURN_IF(wait_error_word(ctx, &err));
  const dim3 grid((unsigned)(NB / 2), (unsigned)batch);
  TN_CHECK_CUDA(ctx, cudaFuncSetAttribute(k_jacobi_block_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  k_jacobi_block_tc<<<grid, kNT, kSmem, stream>>>((int)m, (int)n, NB, r, W, V, nrm, active, rotated, tol, tail, err);
  TN_LAUNCHED(ctx);
  return TN_OK;
}

// K3b — thin QR of few matrices, complex FP64: one CTA per column, reflectors handed on as
// flagged packets.
//
// What bounds it.  The FP64 pipe retires 2 DFMA per clock and SM, so a panel factored by one
// CTA (k_qr_panel) runs at 1/152 of the chip and a bond-sized QR is a chain of such panels:
// 128×64 took 795 µs where the chip's FP64 rate for it is 7 µs.  The chain that cannot be
// avoided is one step per column: reflector j in, inner product with column j+1, update,
// norm, reflector j+1 out.  Here every column has its own CTA and stays in registers:
//  * the entries below the diagonal of an updated column are its reflector as they are
//    (u = x − β e₁ is not normalised; H = I − κ u uᴴ), so they are sent at once, and the
//    receivers form uᴴc while the sender still reduces ‖x‖² and forms β and κ;
//  * entries travel as packets of two 64-bit words with 32 data bits and a flag each, polled
//    by the receivers directly: no fence, no barrier between CTAs, and they stay in place as
//    the stored reflectors;
//  * Q is formed in one of two ways.  With CTAs to spare, m more of them carry the rows: row i
//    of Q is (Qᴴeᵢ)ᴴ, the reflectors applied to eᵢ in the order in which they appear, so Q is
//    ready one step after R (64×64 255 → 174 µs, 128×128 498 → 394).  At more than two CTAs
//    an SM the FP64 pipe is what they wait for (256×256 1158 → 1400, 512×64 361 → 521), and
//    column q of Q = H₀…H_{k−1}, which needs reflectors q…0 only, is formed by its column's CTA
//    as soon as column q is done, with half the products.
//  * u₁ is sent before κ, so that the receivers' wᴴ = uᴴc is complete when κ arrives.
// A step takes 2.0 µs with a column per SM: a packet's 0.4 µs, two reductions of 0.4 µs, the
// scalars of 0.5 µs and the updates, in FP64 operations of 64 clocks' latency each.
// Reflectors and signs are LAPACK's (H = I − τ v vᴴ, v₁ = 1, τ v vᴴ = κ u uᴴ, R_jj real with
// the sign opposite to Re x₁).  Every wait is bounded: a CTA whose wait ran out records an
// error and leaves.
// A column whose ‖x‖² leaves the range in which squares and their inverses are normal numbers is
// taken in units of its largest entry: u₁ and κ are sent in those units, with the exponent as u₁'s
// flag, and the receivers bring the entries, sent already, to them (kUnits).
#include <algorithm>
#include <vector>

#include "tn_fixed_sum.cuh"
#include "tn_internal.cuh"
#include "tn_newton.cuh"

namespace {

constexpr int kNT = 128;
static_assert(kQrColsMaxRows == 4 * kNT);
constexpr long long kSpinLimit = 1ll << 22;
// A column or row far from its turn leaves the memory to the ones whose turn it is: asleep for
// 1 µs between looks at a packet (a step is 2 µs) instead of 64 ns, 128 × 128 took 398 µs, not 443 (299 by
// now).
constexpr unsigned kFarSleep = 1000;

struct QMat {
  const cxd* A;
  cxd *Q, *R;       // Q m × k (ld m), R k × n (ld k)
  ulonglong2* box;  // k reflectors × (2m + 4) packets
  const int* perm;  // column c of the factored matrix is column perm[c] of op(A); null: c
  const int* expo;  // A is read in units of 2^expo (one of each matrix); null: as it is
  int64_t lda;
  int m, n, k;        // m × n: the factored matrix
  int rows;           // CTAs that form rows of Q (m or 0)
  int adj;            // bit 0: op(A) = Aᴴ (A n × m); bit 1: Rᴴ (n × k, ld n) is stored for R;
                      // bit 2: Qᴴ (k × m, ld k) is stored for Q
};

__device__ __forceinline__ void put(ulonglong2* p, double v, unsigned flag = 1) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v), f = (unsigned long long)flag << 32;
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"((b & 0xffffffffull) | f), "l"((b >> 32) | f)
               : "memory");
}
__device__ __forceinline__ ulonglong2 get_raw(const ulonglong2* p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ bool arrived(ulonglong2 v) { return (v.x >> 32) != 0 && (v.y >> 32) != 0; }
__device__ __forceinline__ double value_of(ulonglong2 v) {
  return __longlong_as_double((long long)((v.x & 0xffffffffull) | (v.y << 32)));
}

// ‖x‖² between these: ‖x‖ and 1/(‖x‖·|u₁|²), |u₁| ≤ 2‖x‖, by Newton's iteration, as they are in the chain of
// every step (CUDA's rsqrt and divide take up to 600 clocks each).  One reciprocal in place of 1/‖x‖
// and 1/|u₁|²: 31 QRs of bond 64 5.07 → 4.97 ms.  What lies outside is brought into the range by a
// power of two first: u₁'s flag is then kUnits + e with the entries in units of 2^e, 1 otherwise.
// (compared as exponent fields: 2^±600, integers beside FP64 comparisons of 64 clocks)
constexpr int kNormLo = 1023 - 600, kNormHi = 1023 + 600;
constexpr int kUnits = 4096;
// v · 2^k, |k| ≤ 1074, by two factors that are normal numbers
__device__ __forceinline__ double times_pow2(double v, int k) {
  const int h = k >> 1;
  return v * __hiloint2double((1023 + h) << 20, 0) * __hiloint2double((1023 + k - h) << 20, 0);
}
__device__ __forceinline__ cxd times_pow2(cxd v, int k) { return mkcx(times_pow2(v.x, k), times_pow2(v.y, k)); }
__device__ __forceinline__ bool is_zero(double v) { return (((unsigned)__double2hiint(v) << 1) | (unsigned)__double2loint(v)) == 0; }

__device__ __forceinline__ double block_sum(double v, long long* part, int* exps) {  // one barrier
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned e = __reduce_max_sync(0xffffffffu, exponent_field(v));
  const long long s = fixed_warp_sum(v, e);
  if (lane == 0) {
    part[warp] = s;
    exps[warp] = (int)e;
  }
  __syncthreads();
  int E;
  const long long total = fixed_sum4(part, exps, E);
  return fixed_value(total, E);
}

// β = −sgn(Re α)·‖x‖, u₁ = α − β, conj(κ) = −1/(β·u₁) = −(conj(u₁)/|u₁|²)/β from α = (ax, ay), s2 = ‖x‖² − |α|²
// and n2 = ‖x‖²: the scalar packets p, unless ‖x‖² is out of range.  Returns β
__device__ __forceinline__ double send_scalars(ulonglong2* p, double ax, double ay, double s2, double n2, unsigned flag, bool out) {
  const int tid = threadIdx.x;
  const bool none = is_zero(s2) && is_zero(ay);  // H = I
  // (signs are turned and zeros found as bits: an FP64 operation is 64 clocks of the chain; 31 QRs of
  // bond 64 5.08 → 4.72 ms)
  const int flip = __double2hiint(ax) < 0 && !is_zero(ax) ? 0 : (int)0x80000000;
  const double nrm = newton_root(n2), refl = __hiloint2double(__double2hiint(nrm) ^ flip, __double2loint(nrm));
  const double d = ax - refl, ux = none ? 0.0 : d, uy = ay;
  if (tid < 2 && !out) put(p + tid, tid == 0 ? ux : uy, flag);  // κ follows
  const double r = newton_reciprocal(nrm * fma(d, d, uy * uy));
  const double q = none ? 0.0 : __hiloint2double(__double2hiint(r) ^ (~flip & (int)0x80000000), __double2loint(r));
  if (tid < 2 && !out) put(p + 2 + tid, (tid == 0 ? ux : -uy) * q);
  return none ? ax : refl;
}

// the same for a column x (rows tid + q·kNT) whose ‖x‖² is out of range, in units of its largest
// entry.  A function of its own, called behind the chain's code: in its place before the root it made 31
// QRs of bond 64 take 5.23 ms, here 5.08
__device__ __noinline__ double send_in_units(const cxd* x, int R, int col, int m, double ax, double ay, ulonglong2* p,
                                             long long* part, int* exps, int* tops) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // the largest entry's high word; 1 where only low words are left
  unsigned top = 0;
  for (int q = 0; q < R; ++q) {
    const int t = tid + q * kNT;
    if (t < col || t >= m) continue;
    const unsigned hx = (unsigned)__double2hiint(x[q].x) & 0x7fffffffu, hy = (unsigned)__double2hiint(x[q].y) & 0x7fffffffu;
    top = max(top, max(max(hx, hy), (__double2loint(x[q].x) | __double2loint(x[q].y)) != 0 ? 1u : 0u));
  }
  top = __reduce_max_sync(0xffffffffu, top);
  __syncthreads();
  if (lane == 0) tops[warp] = (int)top;
  __syncthreads();
  top = (unsigned)max(max(tops[0], tops[1]), max(tops[2], tops[3]));
  // (zeros, and what is not finite, stay as they are)
  const int e = top == 0 || top >= 0x7ff00000u ? 0 : top < 0x100000u ? -1060 : (int)(top >> 20) - 1023;
  double s2 = 0;
  for (int q = 0; q < R; ++q) {
    const int t = tid + q * kNT;
    if (t <= col || t >= m) continue;
    const cxd v = times_pow2(x[q], -e);
    s2 = fma(v.x, v.x, fma(v.y, v.y, s2));
  }
  s2 = block_sum(s2, part, exps);
  __syncthreads();
  ax = times_pow2(ax, -e);
  ay = times_pow2(ay, -e);
  return times_pow2(send_scalars(p, ax, ay, s2, fma(ax, ax, fma(ay, ay, s2)), (unsigned)(kUnits + e), false), e);
}

// a batch of equal matrices: the first one and the strides to the next; or a list of matrices
// of falling n, whose columns are taken in the order 0 of all, 1 of all, …
struct QBatch {
  QMat first;
  int64_t sA, sQ, sR, sBox;
  const QMat* list;
  const int* level;  // levels + 1: the columns before column c of the first matrix
  int levels;
  int* ticket;
};

template <int R>
__global__ void __launch_bounds__(kNT, 4) k_qr_cols(QBatch batch, int* err) {
  QMat M;
  int index;
  if (batch.list) {
    __shared__ int s_t;
    if (threadIdx.x == 0) s_t = atomicAdd(batch.ticket, 1);
    __syncthreads();
    const int t = s_t;
    int lo = 0, hi = batch.levels;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      (batch.level[mid] <= t ? lo : hi) = mid;
    }
    index = lo;
    M = batch.list[t - batch.level[lo]];
  } else {
    M = batch.first;
    const int b = (int)blockIdx.x / (M.n + M.rows);
    index = (int)blockIdx.x - b * (M.n + M.rows);
    M.A += b * batch.sA;
    if (M.Q) M.Q += b * batch.sQ;
    M.R += b * batch.sR;
    M.box += b * batch.sBox;
    if (M.perm) M.perm += b * M.n;
    if (M.expo) M.expo += b;
  }
  const int m = M.m, k = M.k;
  const bool row = index >= M.n;         // a CTA that forms a row of Q
  const int col = row ? m + k : index;  // (rows wait for all reflectors)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, half = lane >> 4;
  const int64_t stride = 2 * (int64_t)m + 4;
  __shared__ __align__(16) long long fix[2][2][4];  // parity, Re or Im, warp: partial sums in fixed point
  __shared__ __align__(16) int fix_e[2][4];
  __shared__ double s_row[2][2];  // this column's entry in the pivot row
  // whether a wait ran out, and the flag of a reflector that came in units (0: none did); looked at
  // together behind the one barrier of a step, of either parity
  __shared__ __align__(8) int2 s_state[2];
  if (tid < 2) s_state[tid] = make_int2(0, 0);
  cxd x[R];
  const int64_t src = row ? 0 : (M.perm ? M.perm[col] : col);
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int64_t t = tid + q * kNT;
    x[q] = mkcx(row && t == index - M.n ? 1.0 : 0.0, 0.0);
    if (!row && t < m) x[q] = (M.adj & 1) ? conjg(M.A[src + t * M.lda]) : M.A[src * M.lda + t];
  }
  if (!row && M.expo && *M.expo != 0) {
    const int e = -*M.expo;
#pragma unroll
    for (int q = 0; q < R; ++q) x[q] = times_pow2(x[q], e);
  }
  int buf = 0;
  // whether a warp's 32 rows of group q meet the reflector's, j … m − 1: what lies outside is zeros, and
  // not a turn in the FP64 pipe (a group of 16 up to 144×72: 46.1 → 44.4 ms)
  auto warp_row = [&](int q, int j) { return q * kNT + warp * 32 + 31 >= j && q * kNT + warp * 32 < m; };
  // x ← (I − f-form of reflector j) x: rows > j of u from the packets, u₁ and conj(κ) from the
  // scalar packets; adj: the factorisation's Hᴴ, otherwise H
  auto reflect = [&](int j, bool adj) -> bool {
    const ulonglong2* b = M.box + (int64_t)j * stride;
    cxd u[R];
    long long spins = 0;
    bool ok;
    ulonglong2 p0, p1, p2, p3;
    do {
      ok = true;
      ulonglong2 p[2 * R];
      p0 = get_raw(b + 2 * m);
      p1 = get_raw(b + 2 * m + 1);
      p2 = get_raw(b + 2 * m + 2);
      p3 = get_raw(b + 2 * m + 3);
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const int t = tid + q * kNT;
        if (t > j && t < m) {
          p[2 * q] = get_raw(b + t);
          p[2 * q + 1] = get_raw(b + m + t);
        }
      }
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const int t = tid + q * kNT;
        u[q] = mkcx(0.0, 0.0);
        if (t > j && t < m) {
          ok = ok && arrived(p[2 * q]) && arrived(p[2 * q + 1]);
          u[q] = mkcx(value_of(p[2 * q]), value_of(p[2 * q + 1]));
        }
      }
      if (!ok && adj && col > j + 8) __nanosleep(kFarSleep);
    } while (!ok && ++spins < kSpinLimit);
    const bool far = adj && col > j + 8;
    // (a second time round for a reflector in units)
    for (bool again = false;; again = true) {
      double wx = 0, wy = 0;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        if (!warp_row(q, j)) continue;
        wx = fma(u[q].x, x[q].x, fma(u[q].y, x[q].y, wx));
        wy = fma(u[q].x, x[q].y, fma(-u[q].y, x[q].x, wy));
        if (tid + q * kNT == j) {
          s_row[buf][0] = x[q].x;
          s_row[buf][1] = x[q].y;
        }
      }
      {
        const unsigned e = __reduce_max_sync(0xffffffffu, max(exponent_field(wx), exponent_field(wy)));
        const long long s0 = fixed_warp_sum(wx, e), s1 = fixed_warp_sum(wy, e);
        if (lane == 0) {
          fix[buf][0][warp] = s0;
          fix[buf][1][warp] = s1;
          fix_e[buf][warp] = (int)e;
        }
      }
      while (!(arrived(p0) && arrived(p1)) && ++spins < kSpinLimit) {
        if (far) __nanosleep(kFarSleep);
        p0 = get_raw(b + 2 * m);
        p1 = get_raw(b + 2 * m + 1);
        p2 = get_raw(b + 2 * m + 2);
        p3 = get_raw(b + 2 * m + 3);
      }
      if (spins >= kSpinLimit) {
        atomicExch(err, 1);
        s_state[0].x = s_state[1].x = 1;
      }
      if ((unsigned)(p0.x >> 32) > 1 && !again) s_state[buf].y = (int)(unsigned)(p0.x >> 32);
      __syncthreads();
      const int2 state = s_state[buf];
      if ((state.x | state.y) == 0) break;
      if (state.x) return false;
      // u₁ and κ are in units of 2^e: the other entries, and their products, in the same
#pragma unroll
      for (int q = 0; q < R; ++q) u[q] = times_pow2(u[q], kUnits - state.y);
      __syncthreads();
      if (tid == 0) s_state[buf].y = 0;
    }
    int E;
    const long long total = fixed_sum4(fix[buf][half], fix_e[buf], E);
    const double d = fixed_value(total, E);
    const double ux = value_of(p0), uy = value_of(p1);
    // w = uᴴx + conj(u₁)·x_j, f = κ'·w (κ' = conj(κ) for Hᴴ): Re in lanes 0-15, Im in 16-31
    const double cx_ = s_row[buf][0], cy_ = s_row[buf][1];
    const double w = fma(ux, half ? cy_ : cx_, fma(uy, half ? -cx_ : cy_, d));
    while (!(arrived(p2) && arrived(p3)) && ++spins < kSpinLimit) {
      p2 = get_raw(b + 2 * m + 2);
      p3 = get_raw(b + 2 * m + 3);
    }
    if (spins >= kSpinLimit) {  // (seen after the next reflector's barrier)
      atomicExch(err, 1);
      s_state[0].x = s_state[1].x = 1;
    }
    const double kx = value_of(p2), ky = adj ? value_of(p3) : -value_of(p3);
    const double wo = __shfl_xor_sync(0xffffffffu, w, 16);
    const double f = fma(kx, w, (half ? ky : -ky) * wo);
    const double fx = __shfl_sync(0xffffffffu, f, 0), fy = __shfl_sync(0xffffffffu, f, 16);
#pragma unroll
    for (int q = 0; q < R; ++q) {
      if (!warp_row(q, j)) continue;
      const cxd v = tid + q * kNT == j ? mkcx(ux, uy) : u[q];
      x[q].x = fma(-fx, v.x, fma(fy, v.y, x[q].x));
      x[q].y = fma(-fx, v.y, fma(-fy, v.x, x[q].y));
    }
    buf ^= 1;
    return true;
  };

  const int steps = min(col, k);
  for (int j = 0; j < steps; ++j)
    if (!reflect(j, true)) return;
  if (row) {
    // x = Qᴴ e_i: row i of Q is its conjugate
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int t = tid + q * kNT;
      if (t >= k) continue;
      if (M.adj & 4)
        M.Q[(int64_t)(index - M.n) * k + t] = x[q];
      else
        M.Q[(int64_t)t * m + index - M.n] = conjg(x[q]);
    }
    return;
  }
  if (col < k) {
    // this column's reflector: the entries below the pivot go out first
    ulonglong2* b = M.box + (int64_t)col * stride;
    double s2 = 0;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int t = tid + q * kNT;
      if (t > col && t < m) {
        put(b + t, x[q].x);
        put(b + m + t, x[q].y);
        s2 = fma(x[q].x, x[q].x, fma(x[q].y, x[q].y, s2));
      }
      if (t == col) {
        s_row[buf][0] = x[q].x;
        s_row[buf][1] = x[q].y;
      }
    }
    s2 = block_sum(s2, fix[buf][0], fix_e[buf]);
    const double ax = s_row[buf][0], ay = s_row[buf][1];
    buf ^= 1;
    const double n2 = fma(ax, ax, fma(ay, ay, s2));
    const int n2_field = __double2hiint(n2) >> 20;
    const bool out = n2_field < kNormLo || n2_field > kNormHi;
    double beta = send_scalars(b + 2 * m, ax, ay, s2, n2, 1, out);
    if (out) {
      cxd y[R];
#pragma unroll
      for (int q = 0; q < R; ++q) y[q] = x[q];
      beta = send_in_units(y, R, col, m, ax, ay, b + 2 * m, fix[buf][0], fix_e[buf], fix_e[buf ^ 1]);
    }
#pragma unroll
    for (int q = 0; q < R; ++q)
      if (tid + q * kNT == col) x[q] = mkcx(beta, 0.0);
  }
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int t = tid + q * kNT;
    if (t >= k) continue;
    const cxd v = t <= col ? x[q] : mkcx(0.0, 0.0);
    if (M.adj & 2)
      M.R[(int64_t)t * M.n + col] = conjg(v);
    else
      M.R[(int64_t)col * k + t] = v;
  }
  if (col >= k || !M.Q || M.rows) return;
#pragma unroll
  for (int q = 0; q < R; ++q) x[q] = mkcx(tid + q * kNT == col ? 1.0 : 0.0, 0.0);
  for (int j = col; j >= 0; --j)
    if (!reflect(j, false)) return;
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int t = tid + q * kNT;
    if (t >= m) continue;
    if (M.adj & 4)
      M.Q[(int64_t)t * k + col] = conjg(x[q]);
    else
      M.Q[(int64_t)col * m + t] = x[q];
  }
}

const void* kernel_for(int64_t m) {
  return m <= kNT ? (const void*)k_qr_cols<1> : (m <= 2 * kNT ? (const void*)k_qr_cols<2> : (const void*)k_qr_cols<4>);
}

size_t boxes_bytes(int64_t m, int64_t k) { return (size_t)k * (size_t)(2 * m + 4) * sizeof(ulonglong2); }

}  // namespace

size_t qr_cols_workspace(int64_t m, int64_t n, int64_t batch) {
  return ws_round((size_t)batch * boxes_bytes(m, std::min(m, n)));
}

// whether the one-CTA-per-column kernel takes these matrices: rows in the registers of one
// CTA, and every column of every matrix resident at once
tn_status_t qr_cols_takes(tn_ctx* ctx, int64_t m, int64_t columns, bool* out) {
  static int per_sm[3] = {};
  *out = false;
  if (m > kQrColsMaxRows) return TN_OK;
  int& p = per_sm[m <= kNT ? 0 : (m <= 2 * kNT ? 1 : 2)];
  int q = p;
  if (q == 0) {
    TN_CHECK_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&q, kernel_for(m), kNT, 0));
    p = q;
  }
  *out = columns <= (int64_t)q * ctx->num_sms;
  return TN_OK;
}

// thin QR of a batch of m × n matrices op(A)·Π (the caller asked qr_cols_takes with n·batch).
// Q null: not formed.  perm (n per matrix): the column order Π, null for none.  expo (one per
// matrix): A is read, and R is left, in units of 2^expo.
tn_status_t qr_cols_batch(tn_ctx* ctx, int64_t m, int64_t n, const cxd* A, int64_t lda, int64_t sA, cxd* Q, int64_t sQ,
                          cxd* R, int64_t sR, int64_t batch, const int* perm, bool adj_in, bool adj_r, bool adj_q,
                          const int* expo) {
  const int64_t k = std::min(m, n);
  const size_t one = boxes_bytes(m, k);
  char* box = ws_take<char>(ctx, one * (size_t)batch);
  TN_CHECK_CUDA(ctx, cudaMemsetAsync(box, 0, one * (size_t)batch, ctx->stream));
  const int64_t rows = Q && (n + m) * batch <= 2 * (int64_t)ctx->num_sms ? m : 0;
  QBatch b = {QMat{A, Q, R, reinterpret_cast<ulonglong2*>(box), perm, expo, lda, (int)m, (int)n, (int)k, (int)rows,
                   (adj_in ? 1 : 0) + (adj_r ? 2 : 0) + (adj_q ? 4 : 0)},
              sA, sQ, sR, (int64_t)(one / sizeof(ulonglong2)), nullptr, nullptr, 0, nullptr};
  int* err = nullptr;
  TN_RETURN_IF(wait_error_word(ctx, &err));
  void* args[] = {&b, &err};
  TN_CHECK_CUDA(ctx, cudaLaunchCooperativeKernel(kernel_for(m), dim3((unsigned)((n + rows) * batch)), dim3(kNT), args, 0,
                                                 ctx->stream));
  TN_LAUNCHED(ctx);
  return TN_OK;
}

size_t qr_cols_list_workspace(const std::vector<QrColsMat>& mats) {
  size_t boxes = 256;
  int64_t nmax = 0;
  for (auto& q : mats) {
    boxes += boxes_bytes(q.m, std::min(q.m, q.n));
    nmax = std::max<int64_t>(nmax, q.n);
  }
  return ws_round(boxes) + ws_round(sizeof(QMat) * mats.size()) + ws_round(sizeof(int) * (size_t)(nmax + 1));
}

// thin QR of matrices of different sizes (rows ≤ kQrColsMaxRows) in one launch.  Their columns
// need not be resident together: a CTA takes the next column of the order from a counter, so
// whatever it waits for has been taken by a CTA that runs or has finished.  One column of every
// matrix after the other keeps the matrices' chains running side by side.
tn_status_t qr_cols_list(tn_ctx* ctx, std::vector<QrColsMat> mats) {
  if (mats.empty()) return TN_OK;
  std::stable_sort(mats.begin(), mats.end(), [](const QrColsMat& a, const QrColsMat& b) { return a.n > b.n; });
  const int nmax = mats[0].n;
  std::vector<QMat> list;
  std::vector<int> level(nmax + 1, 0);
  size_t boxes = 256;  // the counter
  int64_t total = 0, mmax = 1;
  for (auto& q : mats) {
    boxes += boxes_bytes(q.m, std::min(q.m, q.n));
    total += q.n;
    mmax = std::max<int64_t>(mmax, q.m);
  }
  if (total > 0x7fffffffll) return tn_set_error(ctx, TN_EUNSUPPORTED, "qr: too many columns in a group");
  char* box = ws_take<char>(ctx, boxes);
  size_t at = 256;
  for (auto& q : mats) {
    const int k = std::min(q.m, q.n);
    list.push_back(QMat{q.A, q.Q, q.R, reinterpret_cast<ulonglong2*>(box + at), nullptr, nullptr, q.lda, q.m, q.n, k, 0,
                        q.adjoint ? 5 : 0});
    at += boxes_bytes(q.m, k);
  }
  for (int c = 0, live = (int)mats.size(); c < nmax; ++c) {
    while (live > 0 && mats[live - 1].n <= c) --live;
    level[c + 1] = level[c] + live;
  }
  QMat* d_list = ws_take<QMat>(ctx, list.size());
  int* d_level = ws_take<int>(ctx, level.size());
  TN_CHECK_CUDA(ctx, cudaMemcpyAsync(d_list, list.data(), sizeof(QMat) * list.size(), cudaMemcpyHostToDevice, ctx->stream));
  TN_CHECK_CUDA(ctx, cudaMemcpyAsync(d_level, level.data(), sizeof(int) * level.size(), cudaMemcpyHostToDevice, ctx->stream));
  TN_CHECK_CUDA(ctx, cudaMemsetAsync(box, 0, boxes, ctx->stream));
  QBatch b = {QMat{}, 0, 0, 0, 0, d_list, d_level, nmax, reinterpret_cast<int*>(box)};
  int* err = nullptr;
  TN_RETURN_IF(wait_error_word(ctx, &err));
  void* args[] = {&b, &err};
  TN_CHECK_CUDA(ctx, cudaLaunchKernel(kernel_for(mmax), dim3((unsigned)total), dim3(kNT), args, 0, ctx->stream));
  TN_LAUNCHED(ctx);
  return TN_OK;
}

// K4c — persistent FP64 one-sided Jacobi: a column pair per CTA, columns handed from CTA to
// CTA through flagged packets.
//
// What bounds it.  GB300 retires 2 DFMA per clock and SM (a warp's DFMA occupies its
// scheduler for 64 clocks, which is also its latency), an FP64 division or square root takes
// ~580 clocks, and one column pair of a 256-row matrix is only ~2000 clocks of FP64 work.
// A round of the circle ordering is therefore a latency chain: columns in, inner product,
// rotation, columns out.  The chain here:
//  * the columns stay in registers and travel as packets of two 64-bit words, each carrying
//    32 data bits and the number of the round it is meant for: the receiver polls the data
//    itself, so there is no fence, no separate flag and no barrier between rounds (one way
//    555 clocks on the same die, 970 across, measured);
//  * wᵢᴴwⱼ is reduced by a butterfly that carries Re in one half warp and Im in the other
//    (5 DADD instead of 10), then across warps with one barrier per round; every warp forms
//    the rotation itself from the same numbers;
//  * the rotation's angle and phase come from FP32 (4 approximate MUFU operations instead of
//    6 FP64 divisions and roots) and are made unitary to FP64 by one scaling (unit_rotation):
//    the angle's 1e-7 relative error leaves 1e-7 of the coupling, which a later sweep
//    removes (the stop test counts on it), while W, V and the inner products stay FP64;
//  * V has CTAs of its own, which get each rotation as packets from the CTA that formed it, so
//    its half of the FP64 work is off the chain and on other SMs;
//  * the column norms (cached as unevaluated FP32 sums, updated by t|γ|, recomputed exactly in
//    FP64 at the start of every sweep) travel with the columns; the stop test is one barrier among a matrix's CTAs per
//    sweep, so the matrices of a batch converge independently.
// Every wait is bounded: a CTA that waited kSpinLimit polls records an error and leaves, and
// so do, one limit later each, the CTAs that wait for it.
#include <algorithm>
#include <cstring>

#include "tn_internal.cuh"

namespace {

constexpr int kNT = 128;
constexpr long long kSpinLimit = 1ll << 22;
constexpr int kSweepMax = 80;
// control words of a matrix: barrier arrivals, sweeps run, 1 while unconverged, then per
// sweep the largest ratio (float bits) and the rotation count
constexpr int kCtl = 4 + 2 * kSweepMax;

struct Mat {
  cxd* W;             // m × n, dense
  cxd* V;             // n × n, dense, or null
  double* nrm;        // n
  ulonglong2* box;    // 2 × N × (2m + 1) packets
  ulonglong2* vbox;   // 2 × N × 2n packets (with V)
  ulonglong2* rot;    // (N − 1) × N/2 × 3 packets: the rotations of a sweep (with V)
  int* ctl;           // kCtl
  int m, n, N, cta0;  // cta0: the first CTA of this matrix
};

// circle method: players 0..N-1 (N even), round r in 0..N-2, pair k in 0..N/2-1
__device__ __forceinline__ void circle_pair(int N, int r, int k, int& i, int& j) {
  if (k == 0) {
    i = r;
    j = N - 1;
  } else {
    i = r + k;
    if (i >= N - 1) i -= N - 1;
    j = r - k;
    if (j < 0) j += N - 1;
  }
  if (i > j) {
    const int t = i;
    i = j;
    j = t;
  }
}

__device__ __forceinline__ void put(ulonglong2* p, double v, unsigned flag) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v), f = (unsigned long long)flag << 32;
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"((b & 0xffffffffull) | f), "l"((b >> 32) | f)
               : "memory");
}
__device__ __forceinline__ ulonglong2 get_raw(const ulonglong2* p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ bool arrived(ulonglong2 v, unsigned flag) {
  return (unsigned)(v.x >> 32) == flag && (unsigned)(v.y >> 32) == flag;
}
__device__ __forceinline__ double value_of(ulonglong2 v) {
  return __longlong_as_double((long long)((v.x & 0xffffffffull) | (v.y << 32)));
}

// barrier among the CTAs of one matrix (co-resident: cooperative launch), bounded
__device__ __forceinline__ bool mat_barrier(int* ctr, int target, int* err) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(ctr, 1);
    int v = 0;
    long long spins = 0;
    do {
      asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
    } while (v < target && ++spins < kSpinLimit);
    if (v < target) atomicExch(err, 1);
    s_ok = v >= target;
    __threadfence();
  }
  __syncthreads();
  return s_ok != 0;
}

// Σ over the warp of (a, b): lanes 0-15 end with Σa, lanes 16-31 with Σb
__device__ __forceinline__ double warp_sum2(double a, double b, int lane) {
  double keep = (lane & 16) ? b : a;
  const double send = (lane & 16) ? a : b;
  keep += __shfl_xor_sync(0xffffffffu, send, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) keep += __shfl_xor_sync(0xffffffffu, keep, o);
  return keep;
}

// float → double and (shifted) double → float by integer operations: the conversion
// instructions share the FP64 pipe.  Values below the normal range become 0.
__device__ __forceinline__ double widen(float f) {
  const unsigned b = __float_as_uint(f);
  const int hi = (int)((b & 0x80000000u) | (((b >> 3) & 0x0fffffffu) + 0x38000000u));
  return (b & 0x7f800000u) ? __hiloint2double(hi, (int)(b << 29)) : 0.0;
}
// v · 2^s, truncated to float
__device__ __forceinline__ float narrow(double v, int s) {
  const int hi = __double2hiint(v), lo = __double2loint(v);
  const int e = ((hi >> 20) & 0x7ff) + s - 896;
  const unsigned m = ((unsigned)(hi & 0xfffff) << 3) | ((unsigned)lo >> 29);
  const unsigned r = e <= 0 ? 0u : (e >= 255 ? 0x7f800000u : ((unsigned)e << 23) | m);
  return __uint_as_float(r | (hi & 0x80000000));
}
// f · 2^s for a normal f whose result is normal
__device__ __forceinline__ float shifted(float f, int s) { return __int_as_float(__float_as_int(f) + (s << 23)); }

// (c, s) in FP32 with c² + |s|² = 1 + δ, |δ| ~ 1e-7, made unitary to FP64:
// (1 + δ)^{-1/2} = 1 − δ/2 + 3δ²/8 + O(δ³), δ exact to one rounding each
__device__ __forceinline__ void unit_rotation(float cf, float sxf, float syf, double& c, cxd& se) {
  const double c0 = widen(cf), sx = widen(sxf), sy = widen(syf);
  const double d = fma(sy, sy, fma(sx, sx, fma(c0, c0, -1.0)));
  const double h = d * fma(0.375, d, -0.5);
  c = fma(c0, h, c0);
  se.x = fma(sx, h, sx);
  se.y = fma(sy, h, sy);
}

// a squared column norm relative to ‖W‖²_F as an unevaluated FP32 sum: FP64's 64-clock
// additions stay off the chain
struct Norm {
  float hi, lo;
};
__device__ __forceinline__ Norm norm_add(Norm a, float d) {
  const float s = a.hi + d, b = s - a.hi;
  const float lo = a.lo + ((a.hi - (s - b)) + (d - b));
  Norm r;
  r.hi = s + lo;
  r.lo = lo - (r.hi - s);
  return r;
}
__device__ __forceinline__ void put_norm(ulonglong2* p, Norm v, unsigned flag) {
  const unsigned long long f = (unsigned long long)flag << 32;
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(__float_as_uint(v.hi) | f),
               "l"(__float_as_uint(v.lo) | f)
               : "memory");
}

// x' = c·x − conj(se)·y, y' = se·x + c·y
__device__ __forceinline__ void rotate(double c, cxd se, cxd& x, cxd& y) {
  const cxd a = mkcx(fma(c, x.x, fma(-se.x, y.x, -se.y * y.y)), fma(c, x.y, fma(-se.x, y.y, se.y * y.x)));
  const cxd b = mkcx(fma(c, y.x, fma(se.x, x.x, -se.y * x.y)), fma(c, y.y, fma(se.x, x.y, se.y * x.x)));
  x = a;
  y = b;
}

// the same, or with two threads per row only the output column of this one's side
template <bool SPLIT>
__device__ __forceinline__ void rotate_side(double c, cxd se, cxd& x, cxd& y, int side) {
  if (!SPLIT) {
    rotate(c, se, x, y);
  } else if (side == 0) {
    x = mkcx(fma(c, x.x, fma(-se.x, y.x, -se.y * y.y)), fma(c, x.y, fma(-se.x, y.y, se.y * y.x)));
  } else {
    y = mkcx(fma(c, y.x, fma(se.x, x.x, -se.y * x.y)), fma(c, y.y, fma(se.x, x.y, se.y * x.x)));
  }
}

// V's half of a pair: the rotations come from the CTA that holds the pair's W columns, V's
// columns travel like W's.  Nothing waits for this CTA but the next holders of its columns.
template <int R, bool SPLIT>
__device__ __forceinline__ void v_role(const Mat& M, int k, bool v_given, int max_sweeps, float stop_ratio, int* err) {
  const int n = M.n, N = M.N, pairs = N / 2, tid = threadIdx.x;
  const int side = SPLIT ? tid >> 6 : 0;
  const int64_t colp = 2 * (int64_t)n;
  __shared__ int s_vfail;
  if (tid == 0) s_vfail = 0;
  int i, j;
  circle_pair(N, 0, k, i, j);
  cxd x[R], y[R];
  auto row = [&](int q) { return SPLIT ? tid & 63 : tid + q * kNT; };
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int t = row(q);
    if (v_given) {
      x[q] = t < n ? M.V[(int64_t)i * n + t] : mkcx(0.0, 0.0);
      y[q] = (t < n && j < n) ? M.V[(int64_t)j * n + t] : mkcx(0.0, 0.0);
    } else {
      x[q] = mkcx(t == i ? 1.0 : 0.0, 0.0);
      y[q] = mkcx(t == j ? 1.0 : 0.0, 0.0);
    }
  }
  unsigned flag = 0;
  int arrivals = 2 * pairs;
  if (!mat_barrier(M.ctl, arrivals, err)) return;  // the norms' barrier
  bool more = true;
  for (int sweep = 0; more && sweep < max_sweeps; ++sweep) {
#pragma unroll 1
    for (int r = 0; r < N - 1; ++r, ++flag) {
      circle_pair(N, r, k, i, j);
      const bool two = j < n;
      const ulonglong2* bi = M.vbox + ((int64_t)(flag & 1) * N + i) * colp;
      const ulonglong2* bj = M.vbox + ((int64_t)(flag & 1) * N + (two ? j : i)) * colp;
      const ulonglong2* br = M.rot + ((int64_t)r * pairs + k) * 3;
      double c;
      cxd se;
      long long spins = 0;
      bool ok;
      do {
        const ulonglong2 r0 = get_raw(br), r1 = get_raw(br + 1), r2 = get_raw(br + 2);
        ok = arrived(r0, flag + 1) && arrived(r1, flag + 1) && arrived(r2, flag + 1);
        c = value_of(r0);
        se = mkcx(value_of(r1), value_of(r2));
      } while (!ok && ++spins < kSpinLimit);
      if (flag > 0) {
        constexpr int RC = R < 2 ? R : 2;
#pragma unroll
        for (int q0 = 0; q0 < R; q0 += RC) {
          bool got;
          do {
            ulonglong2 p[4 * RC];
            got = true;
#pragma unroll
            for (int q = 0; q < RC; ++q) {
              const int t = row(q0 + q);
              if (t < n) {
                p[4 * q] = get_raw(bi + t);
                p[4 * q + 1] = get_raw(bi + n + t);
                p[4 * q + 2] = get_raw(bj + t);
                p[4 * q + 3] = get_raw(bj + n + t);
              }
            }
#pragma unroll
            for (int q = 0; q < RC; ++q)
              if (row(q0 + q) < n) {
                got = got && arrived(p[4 * q], flag) && arrived(p[4 * q + 1], flag) && arrived(p[4 * q + 2], flag) &&
                      arrived(p[4 * q + 3], flag);
                x[q0 + q] = mkcx(value_of(p[4 * q]), value_of(p[4 * q + 1]));
                y[q0 + q] = mkcx(value_of(p[4 * q + 2]), value_of(p[4 * q + 3]));
              }
          } while (!got && ++spins < kSpinLimit);
          ok = ok && got;
        }
      }
      if (!ok) {
        atomicExch(err, 1);
        s_vfail = 1;
      }
      // two threads per row: the one that sends a column must not do so before the other has
      // read the packets that the column's next holder will overwrite
      if (SPLIT) __syncthreads();
      if (SPLIT ? s_vfail != 0 : !ok) return;
      if (se.x != 0.0 || se.y != 0.0) {
#pragma unroll
        for (int q = 0; q < R; ++q) rotate_side<SPLIT>(c, se, x[q], y[q], side);
      }
      const unsigned next = flag + 1;
      ulonglong2* oi = M.vbox + ((int64_t)(next & 1) * N + i) * colp;
      ulonglong2* oj = M.vbox + ((int64_t)(next & 1) * N + j) * colp;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const int t = row(q);
        if (t >= n) continue;
        if (!SPLIT || side == 0) {
          put(oi + t, x[q].x, next);
          put(oi + n + t, x[q].y, next);
        }
        if (two && (!SPLIT || side == 1)) {
          put(oj + t, y[q].x, next);
          put(oj + n + t, y[q].y, next);
        }
      }
    }
    arrivals += 2 * pairs;
    if (!mat_barrier(M.ctl, arrivals, err)) return;
    more = __ldcg(&M.ctl[4 + kSweepMax + sweep]) > 0 && __int_as_float(__ldcg(&M.ctl[4 + sweep])) > stop_ratio;
  }
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int t = row(q);
    if (t >= n) continue;
    if (!SPLIT || side == 0) M.V[(int64_t)i * n + t] = x[q];
    if (j < n && (!SPLIT || side == 1)) M.V[(int64_t)j * n + t] = y[q];
  }
}

// CTAs 0 … N/2 − 1 of a matrix hold W's pairs, the next N/2 (with V) V's.  SPLIT (m ≤ 64): two
// threads per row, one for each output column, so that all four schedulers have work.
template <int R, bool SPLIT>
__global__ void __launch_bounds__(kNT, 4)
    k_jacobi_pairs(const Mat* __restrict__ mats, const int* __restrict__ owner, bool v_given, double tol_rel, int max_sweeps,
                   int* err) {
  static_assert(!SPLIT || R == 1, "two threads per row cover 64 rows");
  const Mat M = mats[owner[blockIdx.x]];
  const int m = M.m, n = M.n, N = M.N, pairs = N / 2;
  // A pair above 2u is rotated (the angle's FP32 error leaves couplings of 1e-7 of what they
  // were: none of those above rounding are left standing), and the sweeps end after one whose
  // largest ratio was at most stop_ratio, so that what it left, by either rule (its square or
  // 1e-7 of it), is below rounding
  constexpr float kTwoU = 2.220446e-16f;
  const float tol2 = kTwoU * kTwoU;
  const float stop_ratio = (float)fmin(sqrt(tol_rel * sqrt((double)(m > 1 ? m : 1)) * 0.1), 1e-9);
  if ((int)blockIdx.x - M.cta0 >= pairs) {
    v_role<R, SPLIT>(M, (int)blockIdx.x - M.cta0 - pairs, v_given, max_sweeps, stop_ratio, err);
    return;
  }
  const int k = (int)blockIdx.x - M.cta0, ctas = M.V ? 2 * pairs : pairs;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, half = lane >> 4, side = SPLIT ? tid >> 6 : 0;
  __shared__ double red[2][4][2];
  __shared__ int s_fail;
  const int64_t colp = 2 * (int64_t)m + 1;
  if (tid == 0) s_fail = 0;
  auto row = [&](int q) { return SPLIT ? tid & 63 : tid + q * kNT; };

  int i, j, buf = 0;
  circle_pair(N, 0, k, i, j);
  cxd x[R], y[R];
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int t = row(q);
    x[q] = t < m ? M.W[(int64_t)i * m + t] : mkcx(0.0, 0.0);
    y[q] = (t < m && j < n) ? M.W[(int64_t)j * m + t] : mkcx(0.0, 0.0);
  }
  // Σ over the CTA of (a, b): lanes 0-15 get Σa, lanes 16-31 Σb.  SPLIT: the threads of side 0
  // bring a, those of side 1 b.  One barrier; `between` runs before it.
  auto block_sum2 = [&](double a, double b, auto between) -> double {
    if (SPLIT) {
      const double s = warp_sum(side ? b : a);
      if (lane == 0) red[buf][warp & 1][side] = s;
    } else {
      const double s = warp_sum2(a, b, lane);
      if ((lane & 15) == 0) red[buf][warp][half] = s;
    }
    between();
    __syncthreads();
    double v = red[buf][lane & (SPLIT ? 1 : 3)][half];
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    if (!SPLIT) v += __shfl_xor_sync(0xffffffffu, v, 2);
    buf ^= 1;
    return v;
  };
  // exact ‖x‖², ‖y‖² of the pair held
  auto exact_norms = [&](double& al, double& be) {
    double a = 0, b = 0;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      a = fma(x[q].x, x[q].x, fma(x[q].y, x[q].y, a));
      b = fma(y[q].x, y[q].x, fma(y[q].y, y[q].y, b));
    }
    const double v = block_sum2(a, b, [] {});
    al = __shfl_sync(0xffffffffu, v, 0);
    be = __shfl_sync(0xffffffffu, v, 16);
  };
  double al, be;
  exact_norms(al, be);
  // ‖W‖²_F: columns at or below ε²‖W‖²_F are numerically zero and left alone
  if (tid == 0) {
    M.nrm[i] = al;
    if (j < n) M.nrm[j] = be;
  }
  int arrivals = ctas;
  if (!mat_barrier(M.ctl, arrivals, err)) return;
  double fro = 0;
  for (int c = tid; c < n; c += kNT) fro += __ldcg(&M.nrm[c]);
  fro = warp_sum(fro);
  if (lane == 0) red[buf][warp][0] = fro;
  __syncthreads();
  fro = (red[buf][0][0] + red[buf][1][0]) + (red[buf][2][0] + red[buf][3][0]);
  buf ^= 1;
  constexpr double kEps = 2.220446049250313e-16;
  int ex = 0;
  frexp(fro, &ex);
  ex = max(min(ex, 1000), -1000);
  const double scale = ldexp(1.0, -ex);  // norms are kept relative to 2^ex ≈ ‖W‖²_F
  const float floor2 = fmaxf((float)(fmax(kEps * kEps * fro, 1e-290) * scale), 1.2e-37f);
  auto as_norm = [&](double v) {
    const double s = v * scale;
    Norm r;
    r.hi = (float)s;
    r.lo = (float)(s - (double)r.hi);
    return r;
  };
  Norm na = as_norm(al), nb = as_norm(be);

  unsigned flag = 0;  // the round counter carried by the packets, over all sweeps
  int sweep = 0;
  bool more = true;
  while (more && sweep < max_sweeps) {
    float worst = 0.f;
    int count = 0;
#pragma unroll 1
    for (int r = 0; r < N - 1; ++r, ++flag) {
      if (flag > 0) {
        circle_pair(N, r, k, i, j);
        const bool two = j < n;
        const ulonglong2* bi = M.box + ((int64_t)(flag & 1) * N + i) * colp;
        const ulonglong2* bj = M.box + ((int64_t)(flag & 1) * N + (two ? j : i)) * colp;
        // (two rows of both columns at a time: more packets in flight cost the registers that
        // keep four CTAs of 512 rows on an SM)
        constexpr int RC = R < 2 ? R : 2;
        long long spins = 0;
        bool ok = true;
#pragma unroll
        for (int q0 = 0; q0 < R; q0 += RC) {
          bool got;
          do {
            ulonglong2 p[4 * RC];
#pragma unroll
            for (int q = 0; q < RC; ++q) {
              const int t = row(q0 + q);
              if (t < m) {
                p[4 * q] = get_raw(bi + t);
                p[4 * q + 1] = get_raw(bi + m + t);
                p[4 * q + 2] = get_raw(bj + t);
                p[4 * q + 3] = get_raw(bj + m + t);
              }
            }
            got = true;
            if (q0 == 0) {
              const ulonglong2 pa = get_raw(bi + 2 * m), pb = get_raw(bj + 2 * m);
              got = arrived(pa, flag) && arrived(pb, flag);
              na.hi = __uint_as_float((unsigned)pa.x);
              na.lo = __uint_as_float((unsigned)pa.y);
              nb.hi = __uint_as_float((unsigned)pb.x);
              nb.lo = __uint_as_float((unsigned)pb.y);
            }
#pragma unroll
            for (int q = 0; q < RC; ++q)
              if (row(q0 + q) < m) {
                got = got && arrived(p[4 * q], flag) && arrived(p[4 * q + 1], flag) && arrived(p[4 * q + 2], flag) &&
                      arrived(p[4 * q + 3], flag);
                x[q0 + q] = mkcx(value_of(p[4 * q]), value_of(p[4 * q + 1]));
                y[q0 + q] = mkcx(value_of(p[4 * q + 2]), value_of(p[4 * q + 3]));
              }
          } while (!got && ++spins < kSpinLimit);
          ok = ok && got;
        }
        if (!ok) {
          atomicExch(err, 1);
          s_fail = 1;
        }
        if (r == 0) {
          exact_norms(al, be);
          na = as_norm(al);
          nb = as_norm(be);
        }
      }
      const bool two = j < n;
      // γ = xᴴy
      double gx = 0, gy = 0;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        if (!SPLIT || side == 0) gx = fma(x[q].x, y[q].x, fma(x[q].y, y[q].y, gx));
        if (!SPLIT || side == 1) gy = fma(x[q].x, y[q].y, fma(-x[q].y, y[q].x, gy));
      }
      // what needs only the norms is formed while the partial sums settle: the pair's scale
      // 2^e ≈ √(αβ), 2^e/√(αβ) and (β − α)/√(αβ)
      const bool live = two && na.hi > floor2 && nb.hi > floor2;
      int e = 0;
      float sa = 1.f, sb = 1.f, isab = 1.f, dif = 0.f;
      const double v = block_sum2(gx, gy, [&] {
        if (live) {
          e = (((__float_as_int(na.hi) >> 23) + (__float_as_int(nb.hi) >> 23)) >> 1) - 127;
          const float a = shifted(na.hi, -e), b = shifted(nb.hi, -e);
          const float ra = rsqrtf(a), rb = rsqrtf(b);
          sa = a * ra;
          sb = b * rb;
          isab = ra * rb;
          const float d = (nb.hi - na.hi) + (nb.lo - na.lo);
          dif = d * shifted(1.f, -e) * isab;
        }
      });
      if (s_fail) return;  // (set before the barrier by a thread whose wait ran out)
      // ρ = γ/√(αβ)
      const float rl = narrow(v, -ex - e) * isab;
      const float rx = __shfl_sync(0xffffffffu, rl, 0), ry = __shfl_sync(0xffffffffu, rl, 16);
      const float rho2 = rx * rx + ry * ry;
      const bool apply = live && rho2 > tol2;
      if (live) worst = fmaxf(worst, rho2);
      double c = 1.0;
      cxd se = mkcx(0.0, 0.0);
      if (apply) {
        ++count;
        // t = sgn(ζ)/(|ζ| + √(1 + ζ²)), ζ = (β − α)/(2|γ|), without forming the quotient
        const float irho = rsqrtf(rho2), rho = rho2 * irho;
        const float q2 = fmaf(dif, dif, 4.f * rho2);
        const float t = copysignf(__fdividef(2.f * rho, fabsf(dif) + q2 * rsqrtf(q2)), dif);
        const float cf = rsqrtf(fmaf(t, t, 1.f)), sf = cf * t * irho;
        unit_rotation(cf, sf * rx, sf * ry, c, se);
        // α − t|γ|, β + t|γ|
        const float tag = t * rho * (sa * shifted(1.f, e)) * sb;
        na = norm_add(na, -tag);
        nb = norm_add(nb, tag);
#pragma unroll
        for (int q = 0; q < R; ++q) rotate_side<SPLIT>(c, se, x[q], y[q], side);
      }
      const unsigned next = flag + 1;
      ulonglong2* oi = M.box + ((int64_t)(next & 1) * N + i) * colp;
      ulonglong2* oj = M.box + ((int64_t)(next & 1) * N + j) * colp;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const int t = row(q);
        if (t >= m) continue;
        if (!SPLIT || side == 0) {
          put(oi + t, x[q].x, next);
          put(oi + m + t, x[q].y, next);
        }
        if (two && (!SPLIT || side == 1)) {
          put(oj + t, y[q].x, next);
          put(oj + m + t, y[q].y, next);
        }
      }
      if (tid == 0) put_norm(oi + 2 * m, na, next);
      if (tid == 32 && two) put_norm(oj + 2 * m, nb, next);
      if (M.V && tid >= 96 && tid < 99) {
        const int w = tid - 96;
        put(M.rot + ((int64_t)r * pairs + k) * 3 + w, w == 0 ? c : (w == 1 ? se.x : se.y), next);
      }
    }
    // stop test: a sweep whose largest ratio is ρ leaves ~ρ² for the next one
    if (tid == 0) {
      atomicMax(&M.ctl[4 + sweep], __float_as_int(sqrtf(worst)));
      if (count) atomicAdd(&M.ctl[4 + kSweepMax + sweep], count);
    }
    arrivals += ctas;
    if (!mat_barrier(M.ctl, arrivals, err)) return;
    more = __ldcg(&M.ctl[4 + kSweepMax + sweep]) > 0 && __int_as_float(__ldcg(&M.ctl[4 + sweep])) > stop_ratio;
    ++sweep;
  }
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int t = row(q);
    if (t >= m) continue;
    if (!SPLIT || side == 0) M.W[(int64_t)i * m + t] = x[q];
    if (j < n && (!SPLIT || side == 1)) M.W[(int64_t)j * m + t] = y[q];
  }
  if (k == 0 && tid == 0) {
    M.ctl[1] = sweep;
    M.ctl[2] = more ? 1 : 0;
  }
}

// (rows: the larger of m and, with V, n)
const void* kernel_for(int64_t rows) {
  return rows <= kNT / 2 ? (const void*)k_jacobi_pairs<1, true>
                         : (rows <= kNT ? (const void*)k_jacobi_pairs<1, false>
                                        : (rows <= 2 * kNT ? (const void*)k_jacobi_pairs<2, false>
                                                           : (const void*)k_jacobi_pairs<4, false>));
}

inline int even(int n) { return n + (n & 1); }
// most CTAs of one launch the workspace is sized for (the occupancy may allow fewer)
constexpr int64_t kMaxCtas = 152 * 6;
// packets of a matrix: W's columns and norms, V's columns, the rotations of a sweep
size_t packets(int64_t m, int64_t n, bool with_v) {
  const int64_t N = n + (n & 1);
  return (size_t)(2 * N * (2 * m + 1) + (with_v ? 2 * N * 2 * n + (N - 1) * (N / 2) * 3 : 0));
}

}  // namespace

// workspace of jacobi_pairs for `count` matrices of at most m × n
size_t jacobi_pairs_workspace(int64_t m, int64_t n, int64_t count, bool with_v) {
  const int64_t each = (n + 1) / 2 * (with_v ? 2 : 1);
  const int64_t at_once = std::min(count, kMaxCtas / each + 1);
  return ws_round((size_t)at_once * packets(m, n, with_v) * sizeof(ulonglong2) + sizeof(int) * (size_t)(kCtl * count + 64) + 512) +
         ws_round(sizeof(Mat) * (size_t)count + sizeof(int) * (size_t)(at_once * each) + 512);
}

bool jacobi_pairs_fits(int64_t m, int64_t n) { return m <= 4 * kNT && n >= 2 && n <= m; }

// CTAs that one launch keeps resident for matrices of m rows
tn_status_t jacobi_pairs_resident(tn_ctx* ctx, int64_t m, int64_t* out) {
  static int per_sm[4] = {};
  int& p = per_sm[m <= kNT / 2 ? 0 : (m <= kNT ? 1 : (m <= 2 * kNT ? 2 : 3))];
  int q = p;
  if (q == 0) {
    TN_CHECK_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&q, kernel_for(m), kNT, 0));
    p = q;
  }
  *out = std::min<int64_t>((int64_t)q * ctx->num_sms, kMaxCtas);
  return TN_OK;
}

// One-sided Jacobi of every matrix (W m × n, m ≥ n, m ≤ 512; all with V or all without) until
// it converges or max_sweeps: as many matrices per launch as fit on the chip at once.
// Reports the most sweeps a matrix took and whether one did not converge.
tn_status_t jacobi_pairs(tn_ctx* ctx, const std::vector<JacobiMat>& mats, bool v_given, int max_sweeps, int* sweeps_out,
                         bool* noconv_out) {
  *sweeps_out = 0;
  *noconv_out = false;
  if (mats.empty()) return TN_OK;
  max_sweeps = std::min(max_sweeps, kSweepMax);
  const bool with_v = mats[0].V != nullptr;
  int64_t mmax = 1, nmax = 2;
  for (const JacobiMat& q : mats) {
    mmax = std::max<int64_t>(mmax, q.m);
    nmax = std::max<int64_t>(nmax, q.n);
  }
  int64_t resident = 0;
  TN_RETURN_IF(jacobi_pairs_resident(ctx, mmax, &resident));
  auto ctas_of = [&](const JacobiMat& q) { return (int64_t)even(q.n) / 2 * (with_v ? 2 : 1); };
  // the launches, and the largest of each buffer over them
  std::vector<size_t> starts;
  size_t zero_bytes = 0, table_bytes = 0;
  for (size_t first = 0; first < mats.size();) {
    size_t last = first, pk = 0;
    int64_t g = 0;
    while (last < mats.size() && (last == first || g + ctas_of(mats[last]) <= resident)) {
      pk += packets(mats[last].m, mats[last].n, with_v);
      g += ctas_of(mats[last++]);
    }
    if (g > resident) return tn_set_error(ctx, TN_EUNSUPPORTED, "svd: the Jacobi pairs do not fit the device");
    zero_bytes = std::max(zero_bytes, pk * sizeof(ulonglong2) + (sizeof(int) * (kCtl * (last - first) + 1) + 255) / 256 * 256);
    table_bytes = std::max(table_bytes, sizeof(Mat) * (last - first) + sizeof(int) * (size_t)g);
    starts.push_back(first);
    first = last;
  }
  starts.push_back(mats.size());
  char* zeroed = ws_take<char>(ctx, zero_bytes);
  char* table = ws_take<char>(ctx, table_bytes);
  std::vector<char> host;
  std::vector<int> h_ctl;
  for (int s = 0; s < 64; ++s) {
    ctx->sweep_ratio[s] = 0.f;
    ctx->sweep_rotations[s] = 0;
  }
  for (size_t part = 0; part + 1 < starts.size(); ++part) {
    const size_t first = starts[part], count = starts[part + 1] - first, owner_at = sizeof(Mat) * count;
    int64_t g = 0;
    for (size_t q = 0; q < count; ++q) g += ctas_of(mats[first + q]);
    host.assign(owner_at + sizeof(int) * (size_t)g, 0);
    Mat* hm = reinterpret_cast<Mat*>(host.data());
    int* ho = reinterpret_cast<int*>(host.data() + owner_at);
    int* ctl = reinterpret_cast<int*>(zeroed);
    int* err = ctl + kCtl * count;
    ulonglong2* box = reinterpret_cast<ulonglong2*>(zeroed + (sizeof(int) * (kCtl * count + 1) + 255) / 256 * 256);
    int cta = 0;
    for (size_t q = 0; q < count; ++q) {
      const JacobiMat& src = mats[first + q];
      const int N = even(src.n);
      Mat& M = hm[q];
      M.W = src.W;
      M.V = src.V;
      M.nrm = src.nrm;
      M.m = src.m;
      M.n = src.n;
      M.N = N;
      M.cta0 = cta;
      M.ctl = ctl + kCtl * q;
      M.box = box;
      M.vbox = M.box + (size_t)2 * N * (2 * src.m + 1);
      M.rot = M.vbox + (size_t)2 * N * 2 * src.n;
      box += packets(src.m, src.n, with_v);
      for (int64_t c = 0; c < ctas_of(src); ++c) ho[cta++] = (int)q;
    }
    TN_CHECK_CUDA(ctx, cudaMemsetAsync(zeroed, 0, (size_t)(reinterpret_cast<char*>(box) - zeroed), ctx->stream));
    TN_CHECK_CUDA(ctx, cudaMemcpyAsync(table, host.data(), host.size(), cudaMemcpyHostToDevice, ctx->stream));
    const Mat* dm = reinterpret_cast<const Mat*>(table);
    const int* down = reinterpret_cast<const int*>(table + owner_at);
    double tol_rel = 4.0 * 2.220446049250313e-16;
    void* args[] = {&dm, &down, &v_given, &tol_rel, &max_sweeps, &err};
    const int slot = prof_begin(ctx);
    TN_CHECK_CUDA(ctx, cudaLaunchCooperativeKernel(kernel_for(mmax), dim3((unsigned)g), dim3(kNT), args, 0, ctx->stream));
    TN_LAUNCHED(ctx);
    h_ctl.resize(kCtl * count + 1);
    TN_CHECK_CUDA(ctx, cudaMemcpyAsync(h_ctl.data(), ctl, sizeof(int) * h_ctl.size(), cudaMemcpyDeviceToHost, ctx->stream));
    TN_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    double flops = 0;
    for (size_t q = 0; q < count; ++q) {
      const int* h = &h_ctl[kCtl * q];
      *sweeps_out = std::max(*sweeps_out, h[1]);
      *noconv_out = *noconv_out || h[2] != 0;
      for (int s = 0; s < 64; ++s) {
        float ratio;
        memcpy(&ratio, &h[4 + s], sizeof(float));
        if (ratio > ctx->sweep_ratio[s]) {
          ctx->sweep_ratio[s] = ratio;
          ctx->sweep_rotations[s] = h[4 + kSweepMax + s];
        }
      }
      const double mm = hm[q].m, nn = hm[q].n;
      flops += h[1] * nn * (nn - 1) / 2 * (32.0 * mm + (with_v ? 24.0 * nn : 0.0));
    }
    if (slot >= 0) prof_end(ctx, slot, TN_PROF_JACOBI_COOP, 1, flops, 0.0);
    if (h_ctl[kCtl * count]) return tn_set_error(ctx, TN_ETIMEOUT, "svd: a wait of the Jacobi rounds exceeded its limit");
  }
  return TN_OK;
}

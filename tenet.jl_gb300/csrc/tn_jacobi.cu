// K4 — persistent FP64 one-sided Jacobi: a column pair per CTA, columns handed from CTA to
// CTA through flagged packets.
//
// What bounds it.  GB300 retires 2 DFMA per clock and SM (a warp's DFMA occupies its
// scheduler for 64 clocks, which is also its latency), an FP64 division or square root takes
// ~580 clocks, and one column pair of a 256-row matrix is only ~2000 clocks of FP64 work.
// A round of the circle ordering is therefore a latency chain: columns in, inner product,
// rotation, columns out.  The chain here:
//  * the columns stay in registers and travel as packets of two 64-bit words, each carrying
//    32 data bits and the number of the round it is meant for: the receiver polls the data
//    itself, so there is no fence, no separate flag and no barrier between rounds;
//  * columns are held as w = √D·x (Pair): a rotation is 8 products per row, not 12, and needs
//    neither the cosine nor a unitary correction on the chain; the new D follows its column as a
//    packet of its own;
//  * wᵢᴴwⱼ is added up in fixed point (fixed_warp_sum): integers take the place of 7 dependent
//    DADDs; one barrier per round, after which every warp forms the rotation itself from the
//    same numbers;
//  * the tangent comes from FP32 (approximate MUFU operations instead of 6 FP64 divisions and
//    roots); the rotation is unitary to FP64 for any tangent, whose 1e-7 relative error leaves
//    1e-7 of the coupling, which a later sweep removes (the stop test counts on it);
//  * V has CTAs of its own, which get each rotation as packets from the CTA that formed it, so
//    its half of the FP64 work is off the chain and on other SMs;
//  * the column norms (cached as unevaluated FP32 sums, updated by t|γ|, recomputed exactly in
//    FP64 at the start of every sweep, when the scales are taken into the columns) travel with
//    the columns; the stop test is one barrier among a matrix's CTAs per sweep, so the matrices of a
//    batch converge independently.
// A round of 64 to 128 rows is 1.9 µs (2.2 with 12 products, DADD sums and a corrected cosine), of
// 256 rows 2.6 (3.1), 512 rows 5.8 (7.2); of 1.9 µs the hop is 0.85 (a look at packets in L2 takes
// ~1000 clocks, 1.3 looks on average), the FP64 products 0.45, and the sums and the angle 0.5.
// Every wait is bounded: a CTA that waited kSpinLimit polls records an error and leaves, and
// so do, one limit later each, the CTAs that wait for it.
#include <algorithm>
#include <cstring>

#include "tn_fixed_sum.cuh"
#include "tn_internal.cuh"
#include "tn_newton.cuh"

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
  double* nrm;        // n: ‖wᵢ‖² at the start, Dᵢ at the end of a sweep
  ulonglong2* box;    // 2 × N × (2m + 2) packets
  ulonglong2* vbox;   // 2 × N × 2n packets (with V)
  ulonglong2* rot;    // (N − 1) × N/2 × 3 packets: the rotations of a sweep (with V), and N/2 × 2: the scales
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
// f · 2^s for a normal f whose result is normal
__device__ __forceinline__ float shifted(float f, int s) { return __int_as_float(__float_as_int(f) + (s << 23)); }

__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// √D = s·2^e for a normal D, s in FP32
__device__ __forceinline__ void root_of(double D, float& s, int& e) {
  const int hi = __double2hiint(D), ef = (hi >> 20) - 1023;
  const float v = __int_as_float(((127 + (ef & 1)) << 23) | ((hi & 0xfffff) << 3) | (int)((unsigned)__double2loint(D) >> 29));
  s = v * rsqrt_approx(v);
  e = ef >> 1;
}
// 2^K, 0 below the normal range
__device__ __forceinline__ float pow2(int K) { return K < -126 ? 0.f : __int_as_float((min(K, 127) + 127) << 23); }

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
__device__ __forceinline__ void put_words(ulonglong2* p, unsigned x, unsigned y, unsigned flag) {
  const unsigned long long f = (unsigned long long)flag << 32;
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(x | f), "l"(y | f) : "memory");
}

// Columns are held as w = √D·x.  With a any complex number, q = Dx/Dy, b = q·a and
// w = 1 + Re(ā b),   x ← x − ā y,  y ← y + b x,  D ← D/w
// is a unitary rotation of the columns by the tangent a√q: 8 products per row instead of 12,
// and no square root; the scales are off the chain of the columns.
struct Pair {
  double ax, ay, bx, by;
};
__device__ __forceinline__ cxd turned_x(const Pair& p, cxd x, cxd y) {
  return mkcx(fma(-p.ax, y.x, fma(-p.ay, y.y, x.x)), fma(-p.ax, y.y, fma(p.ay, y.x, x.y)));
}
__device__ __forceinline__ cxd turned_y(const Pair& p, cxd x, cxd y) {
  return mkcx(fma(p.bx, x.x, fma(-p.by, x.y, y.x)), fma(p.bx, x.y, fma(p.by, x.x, y.y)));
}
// with two threads per row only the output column of this one's side, by one expression
template <bool SPLIT>
__device__ __forceinline__ void rotate_side(const Pair& p, cxd& x, cxd& y, int side) {
  if (!SPLIT) {
    const cxd old = x;
    x = turned_x(p, old, y);
    y = turned_y(p, old, y);
  } else {
    const double c1 = side ? p.bx : -p.ax, c2 = side ? -p.by : -p.ay;
    const cxd o = side ? y : x, z = side ? x : y;
    const cxd v = mkcx(fma(c1, z.x, fma(c2, z.y, o.x)), fma(c1, z.y, fma(-c2, z.x, o.y)));
    if (side)
      y = v;
    else
      x = v;
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
      Pair p;
      double fx = 1.0, fy = 1.0;
      long long spins = 0;
      bool ok;
      do {
        const ulonglong2 r0 = get_raw(br), r1 = get_raw(br + 1), r2 = get_raw(br + 2);
        ok = arrived(r0, flag + 1) && arrived(r1, flag + 1) && arrived(r2, flag + 1);
        p.ax = widen(__uint_as_float((unsigned)r0.x));
        p.ay = widen(__uint_as_float((unsigned)r0.y));
        p.bx = value_of(r1);
        p.by = value_of(r2);
      } while (!ok && ++spins < kSpinLimit);
      if (r == 0 && flag > 0) {  // the scales are taken into the columns once a sweep
        const ulonglong2* bs = M.rot + ((int64_t)(N - 1) * pairs) * 3 + 2 * k;
        bool got;
        do {
          const ulonglong2 r0 = get_raw(bs), r1 = get_raw(bs + 1);
          got = arrived(r0, flag + 1) && arrived(r1, flag + 1);
          fx = value_of(r0);
          fy = value_of(r1);
        } while (!got && ++spins < kSpinLimit);
        ok = ok && got;
      }
      if (flag > 0) {
        constexpr int RC = R < 2 ? R : 2;
#pragma unroll
        for (int q0 = 0; q0 < R; q0 += RC) {
          bool got;
          do {
            ulonglong2 u[4 * RC];
            got = true;
#pragma unroll
            for (int q = 0; q < RC; ++q) {
              const int t = row(q0 + q);
              if (t < n) {
                u[4 * q] = get_raw(bi + t);
                u[4 * q + 1] = get_raw(bi + n + t);
                u[4 * q + 2] = get_raw(bj + t);
                u[4 * q + 3] = get_raw(bj + n + t);
              }
            }
#pragma unroll
            for (int q = 0; q < RC; ++q)
              if (row(q0 + q) < n) {
                got = got && arrived(u[4 * q], flag) && arrived(u[4 * q + 1], flag) && arrived(u[4 * q + 2], flag) &&
                      arrived(u[4 * q + 3], flag);
                x[q0 + q] = mkcx(value_of(u[4 * q]), value_of(u[4 * q + 1]));
                y[q0 + q] = mkcx(value_of(u[4 * q + 2]), value_of(u[4 * q + 3]));
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
      if (r == 0 && flag > 0) {
#pragma unroll
        for (int q = 0; q < R; ++q) {
          x[q] = mkcx(x[q].x * fx, x[q].y * fx);
          y[q] = mkcx(y[q].x * fy, y[q].y * fy);
        }
      }
      if (p.ax != 0.0 || p.ay != 0.0) {
#pragma unroll
        for (int q = 0; q < R; ++q)
          if (R == 1 || q * kNT + (tid & ~31) < n) rotate_side<SPLIT>(p, x[q], y[q], side);
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
  const double fx = sqrt(__ldcg(&M.nrm[i])), fy = j < n ? sqrt(__ldcg(&M.nrm[j])) : 0.0;
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int t = row(q);
    if (t >= n) continue;
    if (!SPLIT || side == 0) M.V[(int64_t)i * n + t] = mkcx(x[q].x * fx, x[q].y * fx);
    if (j < n && (!SPLIT || side == 1)) M.V[(int64_t)j * n + t] = mkcx(y[q].x * fy, y[q].y * fy);
  }
}

// CTAs 0 … N/2 − 1 of a matrix hold W's pairs, the next N/2 (with V) V's.  SPLIT (m ≤ 64): two
// threads per row, one for each output column, so that all four schedulers have work.
template <int R, bool SPLIT>
__global__ void __launch_bounds__(kNT, 4)
    k_jacobi_pairs(const Mat* __restrict__ mats, const int* __restrict__ owner, bool v_given, double tol_rel, int max_sweeps,
                   int first, int* err) {
  static_assert(!SPLIT || R == 1, "two threads per row cover 64 rows");
  // (block `first` is CTA 0, and so on around)
  const int cta = (int)blockIdx.x >= first ? (int)blockIdx.x - first : (int)(blockIdx.x + gridDim.x) - first;
  const Mat M = mats[owner[cta]];
  const int m = M.m, n = M.n, N = M.N, pairs = N / 2;
  // A pair above 2u is rotated (the angle's FP32 error leaves couplings of 1e-7 of what they
  // were: none of those above rounding are left standing), and the sweeps end after one whose
  // largest ratio was at most stop_ratio, so that what it left, by either rule (its square or
  // 1e-7 of it), is below rounding
  constexpr float kTwoU = 2.220446e-16f;
  const float tol2 = kTwoU * kTwoU;
  // (1e-9 for every m that this kernel takes; as a constant the 512-row kernel came out 0.6 % slower,
  // 78.4 → 78.9 ms of two 512 × 512 SVDs and a TEBD layer around them)
  const float stop_ratio = (float)fmin(sqrt(tol_rel * sqrt((double)(m > 1 ? m : 1)) * 0.1), 1e-9);
  if (cta - M.cta0 >= pairs) {
    v_role<R, SPLIT>(M, cta - M.cta0 - pairs, v_given, max_sweeps, stop_ratio, err);
    return;
  }
  const int k = cta - M.cta0, ctas = M.V ? 2 * pairs : pairs;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, half = lane >> 4, side = SPLIT ? tid >> 6 : 0;
  __shared__ double red[2][4][2];
  __shared__ __align__(16) long long fix[2][2][4];  // parity, Re or Im, warp
  __shared__ __align__(16) int fix_e[2][2][4];
  __shared__ int s_fail;
  const int64_t colp = 2 * (int64_t)m + 2;
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
  // bring a, those of side 1 b. One barrier.
  auto block_sum2 = [&](double a, double b) -> double {
    if (SPLIT) {
      const double s = warp_sum(side ? b : a);
      if (lane == 0) red[buf][warp & 1][side] = s;
    } else {
      const double s = warp_sum2(a, b, lane);
      if ((lane & 15) == 0) red[buf][warp][half] = s;
    }
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
    const double v = block_sum2(a, b);
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
  ex = max(min(ex, 1000), -1000) >> 1;
  // the columns are kept relative to 2^ex ≈ ‖W‖_F, their norms to its square
  const double scale = ldexp(1.0, -2 * ex), scale1 = ldexp(1.0, -ex);
  const float floor2 = fmaxf((float)(fmax(kEps * kEps * fro, 1e-290) * scale), 1.2e-37f);
  auto as_norm = [&](double v) {
    Norm r;
    r.hi = (float)v;
    r.lo = (float)(v - (double)r.hi);
    return r;
  };
  auto take_scales = [&](double fx, double fy) {
#pragma unroll
    for (int q = 0; q < R; ++q) {
      x[q] = mkcx(x[q].x * fx, x[q].y * fx);
      y[q] = mkcx(y[q].x * fy, y[q].y * fy);
    }
  };
  take_scales(scale1, scale1);
  Norm na = as_norm(al * scale), nb = as_norm(be * scale);
  double Dx = 1.0, Dy = 1.0;
  // The scales D/w that a round leaves, x's in lanes 0-15 of the last warp, y's in lanes 16-31.  With
  // four rows per thread they are formed while the next round's first look at the packets is on its
  // way (512 rows: 6.0 → 5.8 µs a round); with fewer they would arrive too late for their reader
  // (64 rows: 1.92 → 2.02).
  constexpr bool kScalesLater = R == 4;
  Pair p = {0.0, 0.0, 0.0, 0.0};
  bool turned = false, pending = false;
  ulonglong2* dst = nullptr;
  auto send_scales = [&](unsigned f) -> double {
    double D = half ? Dy : Dx;
    if (turned) D *= newton_reciprocal(fma(p.ax, p.bx, fma(p.ay, p.by, 1.0)));
    if (dst) put(dst, D, f);
    pending = false;
    return D;
  };

  unsigned flag = 0;  // the round counter carried by the packets, over all sweeps
  int sweep = 0;
  bool more = true;
  while (more && sweep < max_sweeps) {
    float worst = 0.f;
    int count = 0;
#pragma unroll 1
    for (int r = 0; r < N - 1; ++r, ++flag) {
      long long spins = 0;
      const ulonglong2 *bD = nullptr, *bE = nullptr;
      ulonglong2 d0, d1;
      auto scales_in = [&] {
        while (!(arrived(d0, flag) && arrived(d1, flag)) && ++spins < kSpinLimit) {
          d0 = get_raw(bD);
          d1 = get_raw(bE);
        }
        if (spins >= kSpinLimit) {
          atomicExch(err, 1);
          s_fail = 1;
        }
        Dx = value_of(d0);
        Dy = value_of(d1);
      };
      if (flag > 0) {
        circle_pair(N, r, k, i, j);
        const bool two = j < n;
        const ulonglong2* bi = M.box + ((int64_t)(flag & 1) * N + i) * colp;
        const ulonglong2* bj = M.box + ((int64_t)(flag & 1) * N + (two ? j : i)) * colp;
        // (two rows of both columns at a time: more packets in flight cost the registers that
        // keep four CTAs of 512 rows on an SM)
        constexpr int RC = R < 2 ? R : 2;
        spins = 0;
        bool ok = true;
        struct Look {
          ulonglong2 p[4 * RC], a, b;
        };
        auto look = [&](Look& l, int q0) {
#pragma unroll
          for (int q = 0; q < RC; ++q) {
            const int t = row(q0 + q);
            if (t < m) {
              l.p[4 * q] = get_raw(bi + t);
              l.p[4 * q + 1] = get_raw(bi + m + t);
              l.p[4 * q + 2] = get_raw(bj + t);
              l.p[4 * q + 3] = get_raw(bj + m + t);
            }
          }
          if (q0 == 0) {
            l.a = get_raw(bi + 2 * m);
            l.b = get_raw(bj + 2 * m);
          }
        };
        auto take = [&](const Look& l, int q0) -> bool {
          bool got = true;
          if (q0 == 0) {
            got = arrived(l.a, flag) && arrived(l.b, flag);
            na.hi = __uint_as_float((unsigned)l.a.x);
            na.lo = __uint_as_float((unsigned)l.a.y);
            nb.hi = __uint_as_float((unsigned)l.b.x);
            nb.lo = __uint_as_float((unsigned)l.b.y);
          }
#pragma unroll
          for (int q = 0; q < RC; ++q)
            if (row(q0 + q) < m) {
              got = got && arrived(l.p[4 * q], flag) && arrived(l.p[4 * q + 1], flag) && arrived(l.p[4 * q + 2], flag) &&
                    arrived(l.p[4 * q + 3], flag);
              x[q0 + q] = mkcx(value_of(l.p[4 * q]), value_of(l.p[4 * q + 1]));
              y[q0 + q] = mkcx(value_of(l.p[4 * q + 2]), value_of(l.p[4 * q + 3]));
            }
          return got;
        };
#pragma unroll
        for (int q0 = 0; q0 < R; q0 += RC) {
          bool got;
          do {
            Look l;
            look(l, q0);
            if (kScalesLater && q0 == 0 && pending) send_scales(flag);
            got = take(l, q0);
          } while (!got && ++spins < kSpinLimit);
          ok = ok && got;
        }
        if (!ok) {
          atomicExch(err, 1);
          s_fail = 1;
        }
        // the scales follow their columns; they are looked for now and looked at before the barrier
        bD = bi + 2 * m + 1;
        bE = bj + 2 * m + 1;
        d0 = get_raw(bD);
        d1 = get_raw(bE);
        if (r == 0) {  // once a sweep they are taken into the columns
          scales_in();
          const double fx = sqrt(Dx), fy = sqrt(Dy);
          take_scales(fx, fy);
          if (M.V && tid < 2) put(M.rot + ((int64_t)(N - 1) * pairs) * 3 + 2 * k + tid, tid ? fy : fx, flag + 1);
          exact_norms(al, be);
          na = as_norm(al);
          nb = as_norm(be);
          Dx = Dy = 1.0;
        }
      }
      const bool two = j < n;
      const unsigned next = flag + 1;
      ulonglong2* oi = M.box + ((int64_t)(next & 1) * N + i) * colp;
      ulonglong2* oj = M.box + ((int64_t)(next & 1) * N + j) * colp;
      // what needs only the norms: the pair's scale 2^e ≈ √(αβ), 2^e/√(αβ) and (β − α)/√(αβ) (of no
      // meaning unless live; without a branch they fit between the FP64 products that follow)
      const bool live = two && na.hi > floor2 && nb.hi > floor2 && na.hi < 3e38f && nb.hi < 3e38f;
      const int e = (((__float_as_int(na.hi) >> 23) + (__float_as_int(nb.hi) >> 23)) >> 1) - 127;
      const float fa = shifted(na.hi, -e), fb = shifted(nb.hi, -e);
      const float ra = rsqrt_approx(fa), rb = rsqrt_approx(fb), sa = fa * ra, sb = fb * rb, isab = ra * rb;
      const float dif = ((nb.hi - na.hi) + (nb.lo - na.lo)) * shifted(1.f, -e) * isab;
      // γ = xᴴy (of the columns as held)
      double gx = 0, gy = 0;
      if (SPLIT) {
        gx = gy = fma(x[0].x, side ? y[0].y : y[0].x, x[0].y * (side ? -y[0].x : y[0].y));
      } else {
#pragma unroll
        for (int q = 0; q < R; ++q) {
          if (R > 1 && q * kNT + warp * 32 >= m) continue;
          gx = fma(x[q].x, y[q].x, fma(x[q].y, y[q].y, gx));
          gy = fma(x[q].x, y[q].y, fma(-x[q].y, y[q].x, gy));
        }
      }
      // (SPLIT: a warp has one of the two)
      const unsigned we = __reduce_max_sync(0xffffffffu, max(exponent_field(gx), exponent_field(gy)));
      if (SPLIT) {
        const long long s = fixed_warp_sum(side ? gy : gx, we);
        if (lane == 0) {
          fix[buf][side][warp & 1] = s;
          fix_e[buf][side][warp & 1] = (int)we;
        }
      } else {
        const long long s0 = fixed_warp_sum(gx, we), s1 = fixed_warp_sum(gy, we);
        if (lane == 0) {
          fix[buf][0][warp] = s0;
          fix[buf][1][warp] = s1;
          fix_e[buf][0][warp] = fix_e[buf][1][warp] = (int)we;
        }
      }
      if (flag > 0 && r > 0) scales_in();
      __syncthreads();
      // √D = s·2^se as floats for the angle
      float sx, sy;
      int ex_x, ex_y;
      root_of(Dx, sx, ex_x);
      root_of(Dy, sy, ex_y);
      // (a ratio of scales beyond 2^±60 waits for the next sweep's columns of scale 1)
      const float ratio = abs(ex_y - ex_x) > 60 ? 0.f : __fdividef(sy, sx) * pow2(ex_y - ex_x);
      const double q = Dx * newton_reciprocal(Dy);
      long long total;
      int E;
      if (SPLIT) {
        const int e0 = fix_e[buf][half][0], e1 = fix_e[buf][half][1];
        E = max(e0, e1);
        total = (fix[buf][half][0] >> min(E - e0, 63)) + (fix[buf][half][1] >> min(E - e1, 63));
      } else {
        total = fixed_sum4(fix[buf][half], fix_e[buf][half], E);
      }
      buf ^= 1;
      // ρ = γ/√(αβ)
      const float rl = fixed_to_float(total) * (sx * sy * isab) * pow2(E - 1077 + ex_x + ex_y - e);
      const float rx = __shfl_sync(0xffffffffu, rl, 0), ry = __shfl_sync(0xffffffffu, rl, 16);
      const float rho2 = rx * rx + ry * ry;
      const bool apply = live && rho2 > tol2;
      if (live) worst = fmaxf(worst, rho2);
      p = {0.0, 0.0, 0.0, 0.0};
      float axf = 0.f, ayf = 0.f;
      if (apply) {
        ++count;
        // t = sgn(ζ)/(|ζ| + √(1 + ζ²)), ζ = (β − α)/(2|γ|), without forming the quotient
        const float irho = rsqrt_approx(rho2), rho = rho2 * irho;
        const float q2 = fmaf(dif, dif, 4.f * rho2);
        float t = copysignf(__fdividef(2.f * rho, fabsf(dif) + q2 * rsqrt_approx(q2)), dif);
        if (ratio == 0.f) t = 0.f;
        const float g = t * irho * ratio;
        axf = g * rx;
        ayf = g * ry;
        p.ax = widen(axf);
        p.ay = widen(ayf);
        if (!SPLIT || side) {
          p.bx = p.ax * q;
          p.by = p.ay * q;
        }
#pragma unroll
        for (int u = 0; u < R; ++u)
          if (R == 1 || u * kNT + warp * 32 < m) rotate_side<SPLIT>(p, x[u], y[u], side);
        // α − t|γ|, β + t|γ|
        const float tag = t * rho * (sa * shifted(1.f, e)) * sb;
        na = norm_add(na, -tag);
        nb = norm_add(nb, tag);
      }
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const int t = row(u);
        if (t >= m) continue;
        if (!SPLIT || side == 0) {
          put(oi + t, x[u].x, next);
          put(oi + m + t, x[u].y, next);
        }
        if (two && (!SPLIT || side == 1)) {
          put(oj + t, y[u].x, next);
          put(oj + m + t, y[u].y, next);
        }
      }
      if (warp == 3) {
        turned = apply;
        pending = true;
        dst = (lane & 15) == 0 && (two || half == 0) ? (half ? oj : oi) + 2 * m + 1 : nullptr;
        if (!kScalesLater || r == N - 2) {
          const double D = send_scales(next);
          if (dst && r == N - 2) M.nrm[half ? j : i] = D;
        }
      } else if (lane == 0 && warp < 2 && (two || warp == 0)) {
        const Norm v = warp ? nb : na;
        put_words((warp ? oj : oi) + 2 * m, __float_as_uint(v.hi), __float_as_uint(v.lo), next);
      } else if (warp == 2 && M.V && lane < 3) {
        ulonglong2* o = M.rot + ((int64_t)r * pairs + k) * 3 + lane;
        if (lane == 0)
          put_words(o, __float_as_uint(axf), __float_as_uint(ayf), next);
        else
          put(o, lane == 1 ? p.bx : p.by, next);
      }
      if (s_fail) return;  // (set before the barrier by a thread whose wait ran out)
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
  const double back = ldexp(1.0, ex);
  take_scales(sqrt(__ldcg(&M.nrm[i])) * back, j < n ? sqrt(__ldcg(&M.nrm[j])) * back : 0.0);
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
  return (size_t)(2 * N * (2 * m + 2) + (with_v ? 2 * N * 2 * n + (N - 1) * (N / 2) * 3 + N : 0));
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
  const size_t top = ctx->ws_top;
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
      M.vbox = M.box + (size_t)2 * N * (2 * src.m + 2);
      M.rot = M.vbox + (size_t)2 * N * 2 * src.n;
      box += packets(src.m, src.n, with_v);
      for (int64_t c = 0; c < ctas_of(src); ++c) ho[cta++] = (int)q;
    }
    TN_CHECK_CUDA(ctx, cudaMemsetAsync(zeroed, 0, (size_t)(reinterpret_cast<char*>(box) - zeroed), ctx->stream));
    TN_CHECK_CUDA(ctx, cudaMemcpyAsync(table, host.data(), host.size(), cudaMemcpyHostToDevice, ctx->stream));
    const Mat* dm = reinterpret_cast<const Mat*>(table);
    const int* down = reinterpret_cast<const int*>(table + owner_at);
    double tol_rel = 4.0 * 2.220446049250313e-16;
    // One matrix with V on slightly more CTAs than SMs: the blocks beyond one per SM share the SMs of
    // the first ones, so those are given to V, which has time to spare, as long as W's
    // CTAs then have an SM each (200 × 200: 3.2 → 3.0 µs a round).  Where blocks really lie only
    // matters for the time.
    const int64_t extra = g - ctx->num_sms;
    int turn = with_v && count == 1 && extra > 0 && extra + g / 2 <= ctx->num_sms ? (int)extra : 0;
    void* args[] = {&dm, &down, &v_given, &tol_rel, &max_sweeps, &turn, &err};
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
      // a pair's row: 8 operations of wᵢᴴwⱼ, 16 of the scaled rotation of W [16 of V's]
      flops += h[1] * nn * (nn - 1) / 2 * (24.0 * mm + (with_v ? 16.0 * nn : 0.0));
    }
    if (slot >= 0) prof_end(ctx, slot, TN_PROF_JACOBI_COOP, 1, flops, 0.0);
    if (h_ctl[kCtl * count]) return tn_set_error(ctx, TN_ETIMEOUT, "svd: a wait of the Jacobi rounds exceeded its limit");
  }
  ctx->ws_top = top;
  return TN_OK;
}

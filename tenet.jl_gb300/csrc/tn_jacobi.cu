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
//    the angle's 1e-7 relative error leaves 1e-7 of the coupling, which the next sweep
//    removes, while W, V and the inner products stay FP64 throughout;
//  * V is received, rotated and sent after W's columns have left, off the chain;
//  * the column norms (cached, updated by t|γ|, recomputed exactly at the start of every
//    sweep) travel with the columns; the stop test is one barrier among a matrix's CTAs per
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

// (c, s) in FP32 with c² + |s|² = 1 + δ, |δ| ~ 1e-7, made unitary to FP64:
// (1 + δ)^{-1/2} = 1 − δ/2 + 3δ²/8 + O(δ³), δ exact to one rounding each
__device__ __forceinline__ void unit_rotation(float cf, float sxf, float syf, double& c, cxd& se) {
  const double c0 = cf, sx = sxf, sy = syf;
  const double d = fma(sy, sy, fma(sx, sx, fma(c0, c0, -1.0)));
  const double h = d * fma(0.375, d, -0.5);
  c = fma(c0, h, c0);
  se.x = fma(sx, h, sx);
  se.y = fma(sy, h, sy);
}

// x' = c·x − conj(se)·y, y' = se·x + c·y
__device__ __forceinline__ void rotate(double c, cxd se, cxd& x, cxd& y) {
  const cxd a = mkcx(fma(c, x.x, fma(-se.x, y.x, -se.y * y.y)), fma(c, x.y, fma(-se.x, y.y, se.y * y.x)));
  const cxd b = mkcx(fma(c, y.x, fma(se.x, x.x, -se.y * x.y)), fma(c, y.y, fma(se.x, x.y, se.y * x.x)));
  x = a;
  y = b;
}

template <int R, bool VACC>
__global__ void __launch_bounds__(kNT, R == 1 ? 4 : (R == 2 ? 3 : 2))
    k_jacobi_pairs(const Mat* __restrict__ mats, const int* __restrict__ owner, bool v_given, double tol_rel, int max_sweeps,
                   int* err) {
  const Mat M = mats[owner[blockIdx.x]];
  const int m = M.m, n = M.n, N = M.N, k = (int)blockIdx.x - M.cta0, pairs = N / 2;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NW = kNT / 32;
  static_assert(NW == 4, "the cross-warp sum below adds four partials");
  __shared__ double red[2][NW][2];
  __shared__ double red_n[NW][2];
  __shared__ int s_fail;
  const int64_t colp = 2 * (int64_t)m + 1, vcolp = 2 * (int64_t)n;
  const double tol = tol_rel * sqrt((double)(m > 1 ? m : 1));
  const float tol2 = (float)(tol * tol), stop_ratio = (float)sqrt(tol * 0.1);
  if (tid == 0) s_fail = 0;

  int i, j;
  circle_pair(N, 0, k, i, j);
  cxd x[R], y[R], vx[VACC ? R : 1], vy[VACC ? R : 1];
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int t = tid + q * kNT;
    x[q] = t < m ? M.W[(int64_t)i * m + t] : mkcx(0.0, 0.0);
    y[q] = (t < m && j < n) ? M.W[(int64_t)j * m + t] : mkcx(0.0, 0.0);
    if (VACC) {
      if (v_given) {
        vx[VACC ? q : 0] = t < n ? M.V[(int64_t)i * n + t] : mkcx(0.0, 0.0);
        vy[VACC ? q : 0] = (t < n && j < n) ? M.V[(int64_t)j * n + t] : mkcx(0.0, 0.0);
      } else {
        vx[VACC ? q : 0] = mkcx(t == i ? 1.0 : 0.0, 0.0);
        vy[VACC ? q : 0] = mkcx(t == j ? 1.0 : 0.0, 0.0);
      }
    }
  }
  double al = 0, be = 0;
  // exact ‖x‖², ‖y‖² of the pair held (all threads get both)
  auto exact_norms = [&]() {
    double a = 0, b = 0;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      a = fma(x[q].x, x[q].x, fma(x[q].y, x[q].y, a));
      b = fma(y[q].x, y[q].x, fma(y[q].y, y[q].y, b));
    }
    const double s = warp_sum2(a, b, lane);
    if ((lane & 15) == 0) red_n[warp][lane >> 4] = s;
    __syncthreads();
    double v = red_n[lane & 3][lane >> 4];
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    al = __shfl_sync(0xffffffffu, v, 0);
    be = __shfl_sync(0xffffffffu, v, 16);
    __syncthreads();
  };
  exact_norms();
  // ‖W‖²_F: columns at or below ε²‖W‖²_F are numerically zero and left alone
  if (tid == 0) {
    M.nrm[i] = al;
    if (j < n) M.nrm[j] = be;
  }
  int arrivals = pairs;
  if (!mat_barrier(M.ctl, arrivals, err)) return;
  double fro = 0;
  for (int c = tid; c < n; c += kNT) fro += __ldcg(&M.nrm[c]);
  {
    const double s = warp_sum2(fro, 0.0, lane);
    if (lane == 0) red_n[warp][0] = s;
    __syncthreads();
    fro = (red_n[0][0] + red_n[1][0]) + (red_n[2][0] + red_n[3][0]);
  }
  constexpr double kEps = 2.220446049250313e-16;
  const double floor2 = fmax(kEps * kEps * fro, 1e-290);
  // norms enter the FP32 angle relative to ‖W‖²_F (a power of two near it)
  int ex = 0;
  frexp(fro, &ex);
  const double scale = ldexp(1.0, -max(min(ex, 1000), -1000));

  const double unscale = ldexp(1.0, max(min(ex, 1000), -1000));

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
        long long spins = 0;
        bool ok;
        do {
          ulonglong2 pi[2 * R + 1], pj[2 * R + 1];
          ok = true;
#pragma unroll
          for (int q = 0; q < R; ++q) {
            const int t = tid + q * kNT;
            if (t < m) {
              pi[2 * q] = get_raw(bi + t);
              pi[2 * q + 1] = get_raw(bi + m + t);
              pj[2 * q] = get_raw(bj + t);
              pj[2 * q + 1] = get_raw(bj + m + t);
            }
          }
          pi[2 * R] = get_raw(bi + 2 * m);
          pj[2 * R] = get_raw(bj + 2 * m);
#pragma unroll
          for (int q = 0; q < R; ++q)
            if (tid + q * kNT < m) {
              ok = ok && arrived(pi[2 * q], flag) && arrived(pi[2 * q + 1], flag) && arrived(pj[2 * q], flag) &&
                   arrived(pj[2 * q + 1], flag);
              x[q] = mkcx(value_of(pi[2 * q]), value_of(pi[2 * q + 1]));
              y[q] = mkcx(value_of(pj[2 * q]), value_of(pj[2 * q + 1]));
            }
          ok = ok && arrived(pi[2 * R], flag) && arrived(pj[2 * R], flag);
          al = value_of(pi[2 * R]);
          be = value_of(pj[2 * R]);
        } while (!ok && ++spins < kSpinLimit);
        if (!ok) {
          atomicExch(err, 1);
          s_fail = 1;
        }
        if (r == 0) exact_norms();
      }
      const bool two = j < n;
      // γ = xᴴy
      double gx = 0, gy = 0;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        gx = fma(x[q].x, y[q].x, fma(x[q].y, y[q].y, gx));
        gy = fma(x[q].x, y[q].y, fma(-x[q].y, y[q].x, gy));
      }
      const int rb = (int)(flag & 1);
      {
        const double s = warp_sum2(gx, gy, lane);
        if ((lane & 15) == 0) red[rb][warp][lane >> 4] = s;
      }
      // the part of the angle that needs only the norms, while the partial sums settle
      const bool live = two && al > floor2 && be > floor2;
      const float alf = live ? (float)(al * scale) : 1.f, bef = live ? (float)(be * scale) : 1.f;
      const float isab = rsqrtf(alf) * rsqrtf(bef);  // 1/√(αβ), scaled
      const float dif = (float)((be - al) * scale) * isab;
      const double gs = scale * (double)isab;
      __syncthreads();
      if (s_fail) return;  // (set before the barrier by a thread whose wait ran out)
      double v = red[rb][lane & 3][lane >> 4];
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      // ρ = γ/√(αβ)
      const float rl = (float)(v * gs);
      const float rx = __shfl_sync(0xffffffffu, rl, 0), ry = __shfl_sync(0xffffffffu, rl, 16);
      const float rho2 = rx * rx + ry * ry;
      const bool apply = live && rho2 > tol2;
      if (live) worst = fmaxf(worst, sqrtf(rho2));
      double c = 1.0;
      cxd se = mkcx(0.0, 0.0);
      if (apply) {
        ++count;
        // t = sgn(ζ)/(|ζ| + √(1 + ζ²)), ζ = (β − α)/(2|γ|), without forming the quotient
        const float irho = rsqrtf(rho2), rho = rho2 * irho;
        const float t = copysignf(__fdividef(2.f * rho, fabsf(dif) + sqrtf(fmaf(dif, dif, 4.f * rho2))), dif);
        const float cf = rsqrtf(fmaf(t, t, 1.f)), sf = cf * t * irho;
        unit_rotation(cf, sf * rx, sf * ry, c, se);
        const double tag = (double)__fdividef(t * rho, isab);  // t|γ|, scaled
        al = fma(-tag, unscale, al);
        be = fma(tag, unscale, be);
#pragma unroll
        for (int q = 0; q < R; ++q) rotate(c, se, x[q], y[q]);
      }
      const unsigned next = flag + 1;
      ulonglong2* oi = M.box + ((int64_t)(next & 1) * N + i) * colp;
      ulonglong2* oj = M.box + ((int64_t)(next & 1) * N + j) * colp;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const int t = tid + q * kNT;
        if (t < m) {
          put(oi + t, x[q].x, next);
          put(oi + m + t, x[q].y, next);
          if (two) {
            put(oj + t, y[q].x, next);
            put(oj + m + t, y[q].y, next);
          }
        }
      }
      if (tid == 0) {
        put(oi + 2 * m, al, next);
        if (two) put(oj + 2 * m, be, next);
      }
      if (VACC) {
        constexpr int RV = VACC ? R : 1;
        if (flag > 0) {
          const ulonglong2* bi = M.vbox + ((int64_t)(flag & 1) * N + i) * vcolp;
          const ulonglong2* bj = M.vbox + ((int64_t)(flag & 1) * N + (two ? j : i)) * vcolp;
          long long spins = 0;
          bool ok;
          do {
            ok = true;
#pragma unroll
            for (int q = 0; q < RV; ++q) {
              const int t = tid + q * kNT;
              if (t < n) {
                const ulonglong2 p0 = get_raw(bi + t), p1 = get_raw(bi + n + t), p2 = get_raw(bj + t), p3 = get_raw(bj + n + t);
                ok = ok && arrived(p0, flag) && arrived(p1, flag) && arrived(p2, flag) && arrived(p3, flag);
                vx[q] = mkcx(value_of(p0), value_of(p1));
                vy[q] = mkcx(value_of(p2), value_of(p3));
              }
            }
          } while (!ok && ++spins < kSpinLimit);
          if (!ok) {
            atomicExch(err, 1);
            s_fail = 1;  // seen at the next round's barrier
          }
        }
        if (apply) {
#pragma unroll
          for (int q = 0; q < RV; ++q) rotate(c, se, vx[q], vy[q]);
        }
        ulonglong2* pi = M.vbox + ((int64_t)(next & 1) * N + i) * vcolp;
        ulonglong2* pj = M.vbox + ((int64_t)(next & 1) * N + j) * vcolp;
#pragma unroll
        for (int q = 0; q < RV; ++q) {
          const int t = tid + q * kNT;
          if (t < n) {
            put(pi + t, vx[q].x, next);
            put(pi + n + t, vx[q].y, next);
            if (two) {
              put(pj + t, vy[q].x, next);
              put(pj + n + t, vy[q].y, next);
            }
          }
        }
      }
    }
    // stop test: a sweep whose largest ratio is ρ leaves ~ρ² for the next one
    if (tid == 0) {
      atomicMax(&M.ctl[4 + sweep], __float_as_int(worst));
      if (count) atomicAdd(&M.ctl[4 + kSweepMax + sweep], count);
    }
    arrivals += pairs;
    if (!mat_barrier(M.ctl, arrivals, err)) return;
    more = __ldcg(&M.ctl[4 + kSweepMax + sweep]) > 0 && __int_as_float(__ldcg(&M.ctl[4 + sweep])) > stop_ratio;
    ++sweep;
  }
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int t = tid + q * kNT;
    if (t < m) {
      M.W[(int64_t)i * m + t] = x[q];
      if (j < n) M.W[(int64_t)j * m + t] = y[q];
    }
    if (VACC && t < n) {
      M.V[(int64_t)i * n + t] = vx[VACC ? q : 0];
      if (j < n) M.V[(int64_t)j * n + t] = vy[VACC ? q : 0];
    }
  }
  if (k == 0 && tid == 0) {
    M.ctl[1] = sweep;
    M.ctl[2] = more ? 1 : 0;
  }
}

template <int R>
const void* kernel_of(bool v) {
  return v ? (const void*)k_jacobi_pairs<R, true> : (const void*)k_jacobi_pairs<R, false>;
}
const void* kernel_for(int rows, bool v) {
  return rows <= kNT ? kernel_of<1>(v) : (rows <= 2 * kNT ? kernel_of<2>(v) : kernel_of<4>(v));
}

inline int even(int n) { return n + (n & 1); }
// most CTAs of one launch the workspace is sized for (the occupancy may allow fewer)
constexpr int64_t kMaxCtas = 152 * 6;

}  // namespace

// workspace of jacobi_pairs for matrices of at most m × n, `ctas` = Σ pairs in all of them
size_t jacobi_pairs_workspace(int64_t m, int64_t n, int64_t count, int64_t ctas, bool with_v) {
  const int64_t at_once = std::min<int64_t>(ctas, std::max<int64_t>(kMaxCtas, (n + 1) / 2));
  return ws_round((size_t)at_once * 4 * sizeof(ulonglong2) * (size_t)(2 * m + 1 + (with_v ? 2 * n : 0)) +
                  sizeof(int) * (size_t)(kCtl * count + 64)) +
         ws_round(sizeof(Mat) * (size_t)count + sizeof(int) * (size_t)ctas + 256) + 1024;
}

bool jacobi_pairs_fits(int64_t m, int64_t n) { return m <= 4 * kNT && n >= 2 && n <= m; }

// CTAs that one launch keeps resident for these sizes
tn_status_t jacobi_pairs_resident(tn_ctx* ctx, int64_t m, bool with_v, int64_t* out) {
  static int per_sm[3][2] = {};
  int& p = per_sm[m <= kNT ? 0 : (m <= 2 * kNT ? 1 : 2)][with_v ? 1 : 0];
  int q = p;
  if (q == 0) {
    TN_CHECK_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&q, kernel_for((int)m, with_v), kNT, 0));
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
  int64_t mmax = 1, nmax = 2, ctas = 0;
  for (const JacobiMat& q : mats) {
    mmax = std::max<int64_t>(mmax, q.m);
    nmax = std::max<int64_t>(nmax, q.n);
    ctas += even(q.n) / 2;
  }
  int64_t resident = 0;
  TN_RETURN_IF(jacobi_pairs_resident(ctx, mmax, with_v, &resident));
  if (even((int)nmax) / 2 > resident) return tn_set_error(ctx, TN_EUNSUPPORTED, "svd: the Jacobi pairs do not fit the device");
  const size_t boxes = (size_t)std::min<int64_t>(ctas, std::max<int64_t>(kMaxCtas, (nmax + 1) / 2)) * 4 * sizeof(ulonglong2) *
                       (size_t)(2 * mmax + 1 + (with_v ? 2 * nmax : 0));
  const size_t ctl_bytes = sizeof(int) * (size_t)(kCtl * mats.size() + 64);
  char* zeroed = ws_take<char>(ctx, boxes + ctl_bytes);
  char* table = ws_take<char>(ctx, sizeof(Mat) * mats.size() + sizeof(int) * (size_t)ctas + 256);
  std::vector<char> host;
  std::vector<int> h_ctl;
  for (int s = 0; s < 64; ++s) {
    ctx->sweep_ratio[s] = 0.f;
    ctx->sweep_rotations[s] = 0;
  }
  for (size_t first = 0; first < mats.size();) {
    // the matrices of this launch
    size_t last = first;
    int64_t g = 0;
    while (last < mats.size() && (last == first || g + even(mats[last].n) / 2 <= resident)) g += even(mats[last++].n) / 2;
    const size_t count = last - first, owner_at = sizeof(Mat) * count;
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
      hm[q].W = src.W;
      hm[q].V = src.V;
      hm[q].nrm = src.nrm;
      hm[q].m = src.m;
      hm[q].n = src.n;
      hm[q].N = N;
      hm[q].cta0 = cta;
      hm[q].ctl = ctl + kCtl * q;
      hm[q].box = box;
      box += (size_t)2 * N * (2 * src.m + 1);
      hm[q].vbox = box;
      if (with_v) box += (size_t)2 * N * 2 * src.n;
      for (int k = 0; k < N / 2; ++k) ho[cta++] = (int)q;
    }
    TN_CHECK_CUDA(ctx, cudaMemsetAsync(zeroed, 0, (size_t)(reinterpret_cast<char*>(box) - zeroed), ctx->stream));
    TN_CHECK_CUDA(ctx, cudaMemcpyAsync(table, host.data(), host.size(), cudaMemcpyHostToDevice, ctx->stream));
    const Mat* dm = reinterpret_cast<const Mat*>(table);
    const int* down = reinterpret_cast<const int*>(table + owner_at);
    double tol_rel = 4.0 * 2.220446049250313e-16;
    void* args[] = {&dm, &down, &v_given, &tol_rel, &max_sweeps, &err};
    const int slot = prof_begin(ctx);
    TN_CHECK_CUDA(ctx, cudaLaunchCooperativeKernel(kernel_for((int)mmax, with_v), dim3((unsigned)g), dim3(kNT), args, 0,
                                                   ctx->stream));
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
    first = last;
  }
  return TN_OK;
}

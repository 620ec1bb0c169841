// Persistent one-sided Jacobi: every sweep of a large problem in one
// cooperative launch.
//
// The per-step formulation (one launch per round-robin step, 2n launches per
// sweep) is bound by launch latency and by re-fetching the pair's columns
// cold each step.  Here one launch runs all sweeps: the steps are separated
// by a grid-wide barrier, and the kernel leaves when a sweep rotated nothing.
// CTAs own column pairs (CTA b takes pairs b, b + gridDim.x, ... of the
// step; a pair's columns are cached in registers between the dot products and
// the rotation).  Same pairing (Brent-Luk round robin), rotation formula and
// skip rule as the one-CTA and per-step kernels of itg_factor.cu:
//   zeta = (b - a) / (2g), t = sign(zeta) / (|zeta| + sqrt(1 + zeta^2)),
//   c = 1/sqrt(1 + t^2), s = c t;  skip when |g| <= tol sqrt(a) sqrt(b); a
//   sweep has converged when no rotated pair had |g| > conv_tol(tol) sqrt(a b).
//
// Columns move between SMs from step to step, so every load of W and V goes
// through L2 (ld.global.cg) and stores bypass L1 (st.global.cg); the barrier
// fences before arriving and after leaving.  The barrier wait is bounded by
// %globaltimer (the handle's wait limit, 4 s by default): a block that times
// out raises a status word that makes every other waiting block leave too,
// and the host reports ITG_ERR_TIMEOUT.
#include "itg_internal.cuh"

#include <cmath>
#include <cstdint>
#include <type_traits>

namespace {

constexpr int JP_THREADS = 256;
constexpr int JP_WARPS = JP_THREADS / 32;

__device__ __forceinline__ unsigned long long jp_timer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ int jp_player(int pos, int step, int np) {
  if (pos == 0) return 0;
  return ((pos - 1 + step) % (np - 1)) + 1;
}

template <class T>
__device__ __forceinline__ T jp_warp_sum(T v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Grid-wide barrier over `nblocks` co-resident blocks (count / generation
// words in global memory).  Returns false for every thread of the block when
// the wait timed out or another block reported a timeout.
__device__ bool jp_grid_sync(unsigned* count, unsigned* gen, int* status, unsigned nblocks,
                             unsigned long long wait_ns) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int good = 1;
    const unsigned g = *(volatile unsigned*)gen;
    __threadfence();
    const unsigned arrived = atomicAdd(count, 1u);
    if (arrived == nblocks - 1) {
      atomicExch(count, 0u);
      __threadfence();
      atomicAdd(gen, 1u);
    } else {
      const unsigned long long t0 = jp_timer();
      while (*(volatile unsigned*)gen == g) {
        if (*(volatile int*)status) {
          good = 0;
          break;
        }
        if (jp_timer() - t0 > wait_ns) {
          atomicExch(status, 1);
          good = 0;
          break;
        }
        __nanosleep(64);
      }
    }
    __threadfence();
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

// Block-wide sums of three values (every thread gets the same totals: the
// per-warp partials are added in a fixed order).
template <class T>
__device__ __forceinline__ void jp_block_sum3(T& a, T& b, T& g, T (*sh)[JP_WARPS]) {
  a = jp_warp_sum(a);
  b = jp_warp_sum(b);
  g = jp_warp_sum(g);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
    sh[0][warp] = a;
    sh[1][warp] = b;
    sh[2][warp] = g;
  }
  __syncthreads();
  a = 0;
  b = 0;
  g = 0;
#pragma unroll
  for (int w = 0; w < JP_WARPS; ++w) {
    a += sh[0][w];
    b += sh[1][w];
    g += sh[2][w];
  }
  __syncthreads();  // sh is reused by the next pair
}

// aux (ints, zeroed by the host): [0] barrier count, [1] generation,
// [2] timeout status, [3] sweeps run (max_sweeps + 1: limit hit, -1: timed
// out), [8 + s] "sweep s rotated".
// One CTA per column pair (CTA b takes pairs b, b + gridDim.x, ... of the
// step).  RC = column elements cached per thread (m <= JP_THREADS * RC), so a
// pair's columns are read once per step; RC = 0 streams them (any m).
template <class T, int RC>
__global__ void __launch_bounds__(JP_THREADS)
k_jacobi_persist(T* __restrict__ W, int64_t m, int n, T* __restrict__ V, T tol, T tol_conv, T amin, T amin_conv,
                 int max_sweeps,
                 int* aux, unsigned long long wait_ns) {
  __shared__ T sh[3][JP_WARPS];
  unsigned* count = (unsigned*)aux;
  unsigned* gen = (unsigned*)aux + 1;
  int* status = aux + 2;
  int* rot = aux + 8;
  const int np = n + (n & 1), npairs = np / 2;
  const int t = threadIdx.x;
  int done = max_sweeps + 1;  // not converged within max_sweeps
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    for (int step = 0; step < np - 1; ++step) {
      for (int pi = blockIdx.x; pi < npairs; pi += gridDim.x) {
        int p = jp_player(pi, step, np), q = jp_player(np - 1 - pi, step, np);
        if (p >= n || q >= n) continue;  // block-uniform
        if (p > q) {
          const int tmp = p;
          p = q;
          q = tmp;
        }
        T* wp = W + (int64_t)p * m;
        T* wq = W + (int64_t)q * m;
        T a = 0, b = 0, g = 0;
        T xr[RC > 0 ? RC : 1], yr[RC > 0 ? RC : 1];
        if (RC > 0) {
#pragma unroll
          for (int r = 0; r < RC; ++r) {
            const int64_t i = t + (int64_t)r * JP_THREADS;
            xr[r] = i < m ? __ldcg(wp + i) : T(0);
            yr[r] = i < m ? __ldcg(wq + i) : T(0);
          }
#pragma unroll
          for (int r = 0; r < RC; ++r) {
            a = fma(xr[r], xr[r], a);
            b = fma(yr[r], yr[r], b);
            g = fma(xr[r], yr[r], g);
          }
        } else {
          for (int64_t i = t; i < m; i += JP_THREADS) {
            const T x = __ldcg(wp + i), y = __ldcg(wq + i);
            a = fma(x, x, a);
            b = fma(y, y, b);
            g = fma(x, y, g);
          }
        }
        jp_block_sum3(a, b, g, sh);
        if (a <= amin || b <= amin || fabs(g) <= tol * sqrt(a) * sqrt(b)) continue;  // block-uniform
        const T zeta = (b - a) / (T(2) * g);
        const T tt = copysign(T(1), zeta) / (fabs(zeta) + sqrt(T(1) + zeta * zeta));
        const T c = T(1) / sqrt(T(1) + tt * tt), s = c * tt;
        if (RC > 0) {
#pragma unroll
          for (int r = 0; r < RC; ++r) {
            const int64_t i = t + (int64_t)r * JP_THREADS;
            if (i < m) {
              __stcg(wp + i, c * xr[r] - s * yr[r]);
              __stcg(wq + i, s * xr[r] + c * yr[r]);
            }
          }
        } else {
          for (int64_t i = t; i < m; i += JP_THREADS) {
            const T x = __ldcg(wp + i), y = __ldcg(wq + i);
            __stcg(wp + i, c * x - s * y);
            __stcg(wq + i, s * x + c * y);
          }
        }
        T* vp = V + (int64_t)p * n;
        T* vq = V + (int64_t)q * n;
        for (int i = t; i < n; i += JP_THREADS) {
          const T x = __ldcg(vp + i), y = __ldcg(vq + i);
          __stcg(vp + i, c * x - s * y);
          __stcg(vq + i, s * x + c * y);
        }
        if (t == 0 && a > amin_conv && b > amin_conv && fabs(g) > tol_conv * sqrt(a) * sqrt(b))
          __stcg(rot + sweep, 1);
      }
      if (!jp_grid_sync(count, gen, status, gridDim.x, wait_ns)) {
        done = -1;
        break;
      }
    }
    if (done < 0) break;
    if (__ldcg(rot + sweep) == 0) {
      done = sweep + 1;
      break;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) aux[3] = done;
}

// ------------------------------------------------------ blocked step
// Block-cyclic one-sided Jacobi: the columns form blocks of WB; step `step`
// of a sweep pairs the blocks round robin (nbp slots), one CTA per block
// pair.  The CTA stages the pair's 2 WB columns in shared memory, rotates
// every cross pair (i in block I, j in block J; WB rounds of WB disjoint
// pairs), accumulates the rotations into a 2WB x 2WB matrix Q, writes the
// columns back and applies Q to the pair's columns of V.  The first step of
// a sweep also rotates the pairs inside each block (a full round robin over
// the 2 WB columns), so every column pair is visited once per sweep.  Same
// rotation formula and skip rule as the element-wise kernels; a step moves
// 2 WB columns per CTA through shared memory instead of two per CTA.
constexpr int JB_THREADS = 512;

// Convergence threshold of a sweep (see the element-wise FP64 kernels): in
// FP64, pairs rotated with |g| <= 4 tol sqrt(a b) sit at the rounding floor of
// the dot product and do not keep the sweep loop running.  The FP32 start of
// the mixed method keeps its plain rule (its tol is far above FP32 rounding).
template <class T>
__host__ __device__ inline T conv_tol(T tol) {
  return sizeof(T) == 8 ? T(4) * tol : tol;
}

template <class T, int WB, int THREADS>
__global__ void __launch_bounds__(THREADS)
k_jacobi_block_step(T* __restrict__ W, int64_t m, int n, T* __restrict__ V, T tol, T tol_conv, T amin,
                    T amin_conv, int step, int first, int* __restrict__ rotated) {
  constexpr int C2 = 2 * WB;              // local columns
  constexpr int TP = THREADS / WB;        // threads per pair
  constexpr int WPG = TP / 32;            // warps per pair group
  extern __shared__ __align__(16) unsigned char jb_smem[];
  T* cols = (T*)jb_smem;                  // [C2][m]
  T* Q = cols + (int64_t)C2 * m;          // [C2][C2], column-major
  T* red = Q + C2 * C2;                   // [WB][WPG][3]
  __shared__ int any, major;
  const int nb = (n + WB - 1) / WB, nbp = nb + (nb & 1);
  const int bi = jp_player(blockIdx.x, step, nbp), bj = jp_player(nbp - 1 - blockIdx.x, step, nbp);
  const int t = threadIdx.x;
  auto gcol = [&](int c) -> int {  // global column of local c, or -1
    const int blk = c < WB ? bi : bj;
    const int gc = blk * WB + (c < WB ? c : c - WB);
    return (blk < nb && gc < n) ? gc : -1;
  };
  if (t == 0) any = major = 0;
  int gcs[C2];
#pragma unroll
  for (int c = 0; c < C2; ++c) gcs[c] = gcol(c);
  // Stage the pair's columns: a thread issues its loads of all 2 WB columns
  // (two rows at a time) before storing any of them, so the L2 latency is paid
  // once per 4 WB loads instead of once per element.
  for (int64_t i0 = t; i0 < m; i0 += 2 * THREADS) {
    const int64_t i1 = i0 + THREADS;
    T v0[C2], v1[C2];
#pragma unroll
    for (int c = 0; c < C2; ++c) {
      v0[c] = gcs[c] >= 0 ? W[(int64_t)gcs[c] * m + i0] : T(0);
      v1[c] = (gcs[c] >= 0 && i1 < m) ? W[(int64_t)gcs[c] * m + i1] : T(0);
    }
#pragma unroll
    for (int c = 0; c < C2; ++c) {
      cols[(int64_t)c * m + i0] = v0[c];
      if (i1 < m) cols[(int64_t)c * m + i1] = v1[c];
    }
  }
  for (int i = t; i < C2 * C2; i += THREADS) Q[i] = (i % (C2 + 1) == 0) ? T(1) : T(0);
  __syncthreads();
  const int g = t / TP, lt = t % TP, wg = lt / 32, lane = t & 31;
  const int rounds = first ? C2 - 1 : WB;
  for (int r = 0; r < rounds; ++r) {
    int p, q;
    if (first) {
      p = jp_player(g, r, C2);
      q = jp_player(C2 - 1 - g, r, C2);
    } else {
      p = g;
      q = WB + (g + r) % WB;
    }
    if (p > q) {
      const int tmp = p;
      p = q;
      q = tmp;
    }
    T* xp = cols + (int64_t)p * m;
    T* xq = cols + (int64_t)q * m;
    // the pair's column slices: four independent loads per iteration, two
    // accumulator sets (m fits in shared memory, so 32-bit indices)
    const int mi = (int)m;
    T a = 0, b = 0, gg = 0, a1 = 0, b1 = 0, g1 = 0;
    int i = lt;
    for (; i + 3 * TP < mi; i += 4 * TP) {
      const T x0 = xp[i], y0 = xq[i], x1 = xp[i + TP], y1 = xq[i + TP];
      const T x2 = xp[i + 2 * TP], y2 = xq[i + 2 * TP], x3 = xp[i + 3 * TP], y3 = xq[i + 3 * TP];
      a = fma(x0, x0, a);
      b = fma(y0, y0, b);
      gg = fma(x0, y0, gg);
      a1 = fma(x1, x1, a1);
      b1 = fma(y1, y1, b1);
      g1 = fma(x1, y1, g1);
      a = fma(x2, x2, a);
      b = fma(y2, y2, b);
      gg = fma(x2, y2, gg);
      a1 = fma(x3, x3, a1);
      b1 = fma(y3, y3, b1);
      g1 = fma(x3, y3, g1);
    }
    for (; i < mi; i += TP) {
      const T x = xp[i], y = xq[i];
      a = fma(x, x, a);
      b = fma(y, y, b);
      gg = fma(x, y, gg);
    }
    a += a1;
    b += b1;
    gg += g1;
    a = jp_warp_sum(a);
    b = jp_warp_sum(b);
    gg = jp_warp_sum(gg);
    if constexpr (WPG > 1) {
      if (lane == 0) {
        red[(g * WPG + wg) * 3 + 0] = a;
        red[(g * WPG + wg) * 3 + 1] = b;
        red[(g * WPG + wg) * 3 + 2] = gg;
      }
      __syncthreads();
      a = 0;
      b = 0;
      gg = 0;
#pragma unroll
      for (int w = 0; w < WPG; ++w) {
        a += red[(g * WPG + w) * 3 + 0];
        b += red[(g * WPG + w) * 3 + 1];
        gg += red[(g * WPG + w) * 3 + 2];
      }
    }
    const bool rot = !(a <= amin || b <= amin || fabs(gg) <= tol * sqrt(a) * sqrt(b));
    if (rot) {
      const T zeta = (b - a) / (T(2) * gg);
      const T tt = copysign(T(1), zeta) / (fabs(zeta) + sqrt(T(1) + zeta * zeta));
      const T c = T(1) / sqrt(T(1) + tt * tt), sn = c * tt;
      int j = lt;
      for (; j + 3 * TP < mi; j += 4 * TP) {
        T x[4], y[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          x[u] = xp[j + u * TP];
          y[u] = xq[j + u * TP];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          xp[j + u * TP] = c * x[u] - sn * y[u];
          xq[j + u * TP] = sn * x[u] + c * y[u];
        }
      }
      for (; j < mi; j += TP) {
        const T x = xp[j], y = xq[j];
        xp[j] = c * x - sn * y;
        xq[j] = sn * x + c * y;
      }
      if (lt < C2) {
        const T x = Q[lt + p * C2], y = Q[lt + q * C2];
        Q[lt + p * C2] = c * x - sn * y;
        Q[lt + q * C2] = sn * x + c * y;
      }
      if (lt == 0) {
        any = 1;
        if (a > amin_conv && b > amin_conv && fabs(gg) > tol_conv * sqrt(a) * sqrt(b)) major = 1;
      }
    }
    __syncthreads();  // columns, Q and red are reused by the next round
  }
  if (!any) return;  // block-uniform (read after the last barrier)
  for (int c = 0; c < C2; ++c) {
    const int gc = gcol(c);
    if (gc < 0) continue;
    const T* src = cols + (int64_t)c * m;
    T* dst = W + (int64_t)gc * m;
    for (int64_t i = t; i < m; i += THREADS) dst[i] = src[i];
  }
  // V[:, cols] <- V[:, cols] Q, one row per thread; the next row's loads are
  // issued before the current row is combined and stored
  int row = t;
  T v[C2];
#pragma unroll
  for (int c = 0; c < C2; ++c) v[c] = (gcs[c] >= 0 && row < n) ? V[row + (int64_t)gcs[c] * n] : T(0);
  for (; row < n; row += THREADS) {
    const int nrow = row + THREADS;
    T vn[C2];
#pragma unroll
    for (int c = 0; c < C2; ++c) vn[c] = (gcs[c] >= 0 && nrow < n) ? V[nrow + (int64_t)gcs[c] * n] : T(0);
#pragma unroll
    for (int c = 0; c < C2; ++c) {
      if (gcs[c] < 0) continue;
      T s = 0;
#pragma unroll
      for (int d = 0; d < C2; ++d) s = fma(v[d], Q[d + c * C2], s);
      V[row + (int64_t)gcs[c] * n] = s;
    }
#pragma unroll
    for (int c = 0; c < C2; ++c) v[c] = vn[c];
  }
  if (t == 0 && major) *rotated = 1;
}

// ------------------------------------------- register-resident block step
// The same block-cyclic step with the pair's columns held in registers: thread
// t keeps RPT rows of all 2 WB columns (rows t, t + threads, ..., or four
// consecutive ones with 16-byte accesses, VEC), so a rotation round touches
// no shared memory but for its sums.  A round's WB dot products are reduced
// together (a transposing butterfly: 9 shuffles for 8 values instead of 40)
// and the squared norms are carried along (a' = a - t g, b' = b + t g;
// computed afresh at the start of a step and whenever one shrank to less than
// a quarter, where the difference has cancelled).  The rotations of all rounds
// are kept and replayed on the rows of V afterwards.
//
// What bounds it: FP32, the issue of its FMAs (5 a row, pair and round, 4 more
// for V) and the latency of a round's reduction and angle; FP64,
// the FP64 pipe (a warp instruction takes 64 clocks of its quarter of the SM),
// so there the divisions and square roots of the angle are taken in FP32 and
// corrected by Newton steps in FP64 (15 FP64 instructions instead of several
// hundred), and a problem runs on few warps with many rows each.  Blocks of 8
// columns in FP32 and 4 in FP64 (fewer pairs wait for one SM's FP64 pipe).
// Measured: a step of the FP32 sweeps 27 -> 19 us at n = 2048 and 15.5 -> 9 us
// at n = 366; FP64, n = 120: 14 us a step where one CTA needed 9 ms a sweep
// (the 150 x 120 SVD 153 -> 6 ms together with the QR before it), and errors of
// 6e-16 |W| instead of 2e-14 |W| in the singular values.
// Sums of NV values over the warp's lanes: afterwards lane l holds the sum of
// value l >> (5 - log2 NV).
template <class T, int NV>
__device__ __forceinline__ T jp_transpose_sum(T (&v)[NV], int lane) {
  int o = 16;
#pragma unroll
  for (int n = NV; n > 1; n >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      const T send = up ? v[i] : v[i + n / 2];
      const T keep = up ? v[i + n / 2] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
    o >>= 1;
  }
#pragma unroll
  for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}

// A rotation is applied as w_p -= s (w_q + u w_p), w_q += s (w_p - u w_q) with
// u = tan(theta / 2) = s / (1 + c): two FMAs a column like the plain form, but
// its rounding is proportional to s, so the many small rotations of the late
// sweeps leave no trace in the columns' norms (Rutishauser, "The Jacobi method
// for real symmetric matrices", Numer. Math. 9 (1966)).  It is orthogonal to
// rounding for any u as long as s = 2 u / (1 + u^2).
//
// jp_angle: the rotation of a pair from its squared norms and dot product;
// true when the pair is rotated.  t = tan(theta), for the norms' update; major:
// it counts against convergence.  FAR (FP64): the pair's norms may be any factor
// apart, see below.
__device__ __forceinline__ float jp_sqrt1p2(float x) {  // sqrt(1 + x^2), a few ulp
  const float y = fmaf(x, x, 1.f);
  return y * rsqrtf(y);
}
template <bool FAR>
__device__ __forceinline__ bool jp_angle(float a, float b, float g, float tol, float tol_conv, float amin,
                                         float amin_conv, float& t, float& u, float& s, bool& major) {
  const float cosine = fabsf(g) * rsqrtf(a) * rsqrtf(b);  // NaN for a zero column
  major = a > amin_conv && b > amin_conv && cosine > tol_conv;
  t = u = s = 0.f;
  if (a <= amin || b <= amin || !(cosine > tol)) return false;
  const float zeta = __fdividef(b - a, 2.f * g);
  const float az = fabsf(zeta);
  t = copysignf(__fdividef(az > 1e9f ? 0.5f : 1.f, az > 1e9f ? az : az + jp_sqrt1p2(az)), zeta);
  u = __fdividef(t, 1.f + jp_sqrt1p2(t));
  const float x = fmaf(u, u, 1.f);
  const float r = __fdividef(1.f, x);
  s = 2.f * u * fmaf(r, fmaf(-x, r, 1.f), r);
  return true;
}

// x 2^-(e - 1023) as a float, truncated, and a float as a double, by integer
// instructions: an FP64 conversion occupies a quarter of an SM for 64 clocks.
// Zero and subnormal numbers (exponent field 0, no leading one) give zero.
__device__ __forceinline__ float jp_to_float(double x, int e) {
  const int hi = __double2hiint(x), field = (hi >> 20) & 0x7FF;
  const int ex = field == 0 ? 0 : field - e + 127;
  const int bits = (ex << 23) | ((hi & 0xFFFFF) << 3) | (int)((unsigned)__double2loint(x) >> 29);
  return ex <= 0 ? 0.f : __int_as_float((hi & 0x80000000) | (ex >= 255 ? 0x7F800000 : bits));
}
__device__ __forceinline__ double jp_to_double(float x) {  // normal numbers; below that zero
  const int b = __float_as_int(x), ex = (b >> 23) & 0xFF;
  return ex == 0 ? 0.0 : __hiloint2double((b & 0x80000000) | ((ex + 896) << 20) | ((b & 0x7FFFFF) >> 3), b << 29);
}
__device__ __forceinline__ bool jp_less(double x, double y) {  // x < y for non-negative x and y
  return __double_as_longlong(x) < __double_as_longlong(y);
}
template <bool FAR>
__device__ __forceinline__ bool jp_angle(double a, double b, double g, float tol, float tol_conv, double amin,
                                         double amin_conv, double& t, double& u, double& s, bool& major) {
  // scaled by a power of two so that max(a, b) is in [1, 2)
  const int ea = (__double2hiint(a) >> 20) & 0x7FF, eb = (__double2hiint(b) >> 20) & 0x7FF;
  const int e = ea > eb ? ea : eb;
  const double d = b - a;
  const float fg = jp_to_float(g, e), fa = jp_to_float(a, e), fb = jp_to_float(b, e), fd = jp_to_float(d, e);
  float cosine = fabsf(fg) * rsqrtf(fa) * rsqrtf(fb);
  // Norms more than 2^55 apart (a graded matrix): the squares and g leave FP32's
  // range, so the cosine takes each number by its own exponent; the angle is g / d
  // to the last bit.  (In every sweep it would cost 1 to 2 % of an SVD.)
  const int lo = ea < eb ? ea : eb;
  const bool far = FAR && lo + 110 < e;
  if (far)
    cosine = fabsf(jp_to_float(g, (ea + eb) >> 1)) * rsqrtf(jp_to_float(a, ea)) * rsqrtf(jp_to_float(b, eb)) *
             ((ea + eb) & 1 ? 0.70710678f : 1.f);
  major = (!FAR || lo > 0) && jp_less(amin_conv, a) && jp_less(amin_conv, b) && cosine > tol_conv;
  // (a column with NaN or infinity is left alone)
  const bool rot = e < 2047 && jp_less(amin, a) && jp_less(amin, b) && cosine > tol;
  const float zeta = __fdividef(fd, 2.f * fg);
  const float az = fabsf(zeta);
  const float tf = copysignf(__fdividef(az > 1e9f ? 0.5f : 1.f, az > 1e9f ? az : az + jp_sqrt1p2(az)), zeta);
  t = jp_to_double(tf);
  // one Newton step of g t^2 + d t - g = 0 (its derivative is at least 2 |g|),
  // the residual in FP64, the step in FP32
  const double f = fma(t, fma(g, t, d), -g);
  // u = t / (1 + q), q = sqrt(1 + t^2), to FP32 accuracy and corrected to first
  // order for its rounding, found from (u^2 - 1) t + 2 u = 0 (derivative
  // 2 (1 + t u)), and for the Newton step, du = dt / (q (1 + q))
  const float q = jp_sqrt1p2(tf);
  const float uf = __fdividef(tf, 1.f + q);
  const double ud = jp_to_double(uf);
  const double w = fma(ud, fma(t, ud, 2.0), -t);
  const float dt = -__fdividef(jp_to_float(f, e), fmaf(2.f * fg, tf, fd));
  u = ud + jp_to_double(__fdividef(dt, q * (1.f + q)) -
                        __fdividef(jp_to_float(w, 1023), 2.f * fmaf(tf, uf, 1.f)));
  // s = 2 u / (1 + u^2): the reciprocal from FP32, its error removed to second order
  const double x = fma(u, u, 1.0);
  const double r = jp_to_double(__fdividef(1.f, fmaf(uf, uf, 1.f)));
  const double s0 = (u + u) * r;
  const double er = fma(-x, r, 1.0);
  s = fma(s0, fma(er, er, er), s0);
  if (far) {
    const double p = __hiloint2double((2046 - ((__double2hiint(d) >> 20) & 0x7FF)) << 20, 0), dm = d * p;
    const double r0 = jp_to_double(__fdividef(1.f, jp_to_float(dm, 1023)));
    t = s = g * p * fma(r0, fma(-dm, r0, 1.0), r0);
    u = 0.5 * t;
  }
  if (!rot) t = u = s = 0.0;
  return rot;
}
// A squared norm that shrank to less than about a quarter (or cancelled to a
// negative number) is computed afresh.
__device__ __forceinline__ bool jp_shrunk(float now, float before) { return now < 0.25f * before; }
__device__ __forceinline__ bool jp_shrunk(double now, double before) {
  return (__double2hiint(now) >> 20) + 2 <= (__double2hiint(before) >> 20);
}

constexpr int64_t JR_MAX_M = 2048;  // rows held in registers: 8 for each of 256 threads

// `prev`: nullptr, or the rotated flag of the sweep before (the step does
// nothing when that sweep had converged; lets several sweeps be queued).
template <class T, int WB, int RPT, bool VEC, bool FIRST, int MAXT, bool FAR>
__global__ void __launch_bounds__(MAXT)
k_jacobi_reg_step(T* __restrict__ W, int64_t m, int n, T* __restrict__ V, float tol, float tol_conv, T amin,
                  T amin_conv, int step, const int* prev, int* rotated) {
  constexpr int C2 = 2 * WB;                 // columns of the pair
  constexpr int NR = FIRST ? C2 - 1 : WB;    // rounds
  constexpr int MAXW = MAXT / 32;
  struct __align__(2 * sizeof(T)) Rot {
    T u, s;
  };
  __shared__ T red[2][MAXW][WB];
  __shared__ T nred[MAXW][C2];
  __shared__ Rot rots[NR][WB];           // all rounds, for V
  __shared__ Rot rotw[MAXW][WB];         // the current round, one copy a warp
  __shared__ unsigned rmask[NR];
  // the previous step's kernel must be done before its columns are read
  itg_grid_wait();
  if (prev && *(const volatile int*)prev == 0) return;
  const int nb = (n + WB - 1) / WB, nbp = nb + (nb & 1);
  const int bi = jp_player(blockIdx.x, step, nbp), bj = jp_player(nbp - 1 - blockIdx.x, step, nbp);
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, nw = blockDim.x >> 5;
  const int64_t c0 = (int64_t)bi * WB, c1 = (int64_t)bj * WB;
  const int nI = bi < nb ? (n - c0 < WB ? (int)(n - c0) : WB) : 0;  // columns of each block
  const int nJ = bj < nb ? (n - c1 < WB ? (int)(n - c1) : WB) : 0;
  const int bd = (int)blockDim.x;

  T x[C2][RPT];
  // row of this thread's element k, counted from r0
  auto row = [&](int k) { return VEC ? 4 * (int64_t)(t + (k >> 2) * bd) + (k & 3) : t + (int64_t)k * bd; };
  // rows r0 + ... of the pair's columns of X (leading dimension and row count ld)
  auto load = [&](const T* X, int64_t ld, int64_t r0) {
#pragma unroll
    for (int c = 0; c < C2; ++c) {
      const bool in = c < WB ? c < nI : c - WB < nJ;
      const T* col = X + (c < WB ? c0 + c : c1 + c - WB) * ld + r0;
      const int64_t left = in ? ld - r0 : 0;
      if constexpr (VEC) {
#pragma unroll
        for (int k = 0; k < RPT; k += 4) {
          float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
          if (row(k) < left) v = *reinterpret_cast<const float4*>(col + row(k));
          x[c][k] = v.x;
          x[c][k + 1] = v.y;
          x[c][k + 2] = v.z;
          x[c][k + 3] = v.w;
        }
      } else {
#pragma unroll
        for (int k = 0; k < RPT; ++k) x[c][k] = row(k) < left ? col[row(k)] : T(0);
      }
    }
  };
  auto store = [&](T* X, int64_t ld, int64_t r0) {
#pragma unroll
    for (int c = 0; c < C2; ++c) {
      const bool in = c < WB ? c < nI : c - WB < nJ;
      T* col = X + (c < WB ? c0 + c : c1 + c - WB) * ld + r0;
      const int64_t left = in ? ld - r0 : 0;
      if constexpr (VEC) {
#pragma unroll
        for (int k = 0; k < RPT; k += 4)
          if (row(k) < left)
            *reinterpret_cast<float4*>(col + row(k)) = make_float4(x[c][k], x[c][k + 1], x[c][k + 2], x[c][k + 3]);
      } else {
#pragma unroll
        for (int k = 0; k < RPT; ++k)
          if (row(k) < left) col[row(k)] = x[c][k];
      }
    }
  };
  auto rotate = [&](int p, int q, const Rot& o) {
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      const T y = x[p][k], z = x[q][k];
      x[p][k] = fma(-o.s, fma(o.u, y, z), y);
      x[q][k] = fma(o.s, fma(-o.u, z, y), z);
    }
  };
  // A round always rotates the same register columns (position g with partner(g));
  // the columns move one position on between rounds and are back in place after
  // the last, so the rounds are one loop: unrolled, they ran once each from a
  // cold instruction cache (FP64, n = 120: 4 us of a 5 us round).
  auto partner = [](int g) { return FIRST ? C2 - 1 - g : WB + g; };
  auto advance = [&]() {
    constexpr int lo = FIRST ? 1 : WB;
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      const T y = x[lo][k];
#pragma unroll
      for (int c = lo; c + 1 < C2; ++c) x[c][k] = x[c + 1][k];
      x[C2 - 1][k] = y;
    }
  };
  const int next_lane = FIRST ? (lane == 0 ? 0 : (lane == C2 - 1 ? 1 : lane + 1))
                              : (lane < WB ? lane : (lane == C2 - 1 ? WB : lane + 1));

  load(W, m, 0);
  // every warp computes the angles of a round (one barrier a round; shuffles
  // inside a branch for one warp cost about 500 clocks each)
  T norm = T(0);  // lane c < C2: squared norm of the column at position c
  bool dirty = true;
  unsigned any = 0, any_major = 0;
#pragma unroll 1
  for (int r = 0; r < NR; ++r) {
    if (dirty) {  // block-uniform
      T v[C2];
#pragma unroll
      for (int c = 0; c < C2; ++c) {
        v[c] = x[c][0] * x[c][0];
#pragma unroll
        for (int k = 1; k < RPT; ++k) v[c] = fma(x[c][k], x[c][k], v[c]);
      }
      constexpr int SH = C2 == 32 ? 0 : (C2 == 16 ? 1 : 2);  // 5 - log2 C2
      const T sum = jp_transpose_sum<T, C2>(v, lane);
      if ((lane & ((1 << SH) - 1)) == 0) nred[warp][lane >> SH] = sum;
      __syncthreads();
      T a = nred[0][lane & (C2 - 1)];
      for (int w = 1; w < nw; ++w) a += nred[w][lane & (C2 - 1)];
      norm = a;
      // nred is rewritten only after later barriers of this loop
    }
    {
      T v[WB];
#pragma unroll
      for (int g = 0; g < WB; ++g) {
        v[g] = x[g][0] * x[partner(g)][0];
#pragma unroll
        for (int k = 1; k < RPT; ++k) v[g] = fma(x[g][k], x[partner(g)][k], v[g]);
      }
      constexpr int SH = WB == 16 ? 1 : (WB == 8 ? 2 : 3);  // 5 - log2 WB
      const T sum = jp_transpose_sum<T, WB>(v, lane);
      if ((lane & ((1 << SH) - 1)) == 0) red[r & 1][warp][lane >> SH] = sum;
    }
    __syncthreads();
    const int pr = lane & (WB - 1);
    T g = T(0);
#pragma unroll
    for (int w0 = 0; w0 < MAXW; w0 += 32 / WB) {
      const int w = w0 + lane / WB;
      const T part = red[r & 1][w < MAXW ? w : 0][pr];  // rows of absent warps are never written
      g += w < nw ? part : T(0);
    }
#pragma unroll
    for (int o = WB; o < 32; o <<= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
    const T a = __shfl_sync(0xffffffffu, norm, pr), b = __shfl_sync(0xffffffffu, norm, partner(pr));
    T tt, u, s;
    bool major;
    const bool rot = jp_angle<FAR>(a, b, g, tol, tol_conv, amin, amin_conv, tt, u, s, major);
    const T an = a - tt * g, bn = b + tt * g;
    const unsigned mask = __ballot_sync(0xffffffffu, rot) & ((1u << WB) - 1u);
    any_major |= __ballot_sync(0xffffffffu, rot && major);
    dirty = __any_sync(0xffffffffu, rot && (jp_shrunk(an, a) || jp_shrunk(bn, b)));
    // lane c takes the new norm of position c from its pair's lane, then the
    // norms move on with the columns
    const int src = lane < WB ? lane : (FIRST ? C2 - 1 - lane : lane - WB) & (WB - 1);
    const T na = __shfl_sync(0xffffffffu, an, src), nb2 = __shfl_sync(0xffffffffu, bn, src);
    norm = __shfl_sync(0xffffffffu, lane < WB ? na : nb2, next_lane & 31);
    if (lane < WB) {
      const Rot o{u, s};
      rotw[warp][lane] = o;
      if (warp == 0) {
        rots[r][lane] = o;
        if (lane == 0) rmask[r] = mask;
      }
    }
    __syncwarp();
    any |= mask;
    if (mask) {
#pragma unroll
      for (int g = 0; g < WB; ++g) rotate(g, partner(g), rotw[warp][g]);
    }
    advance();
    __syncwarp();  // rotw is rewritten by the next round
  }
  if (!any) return;  // block-uniform
  store(W, m, 0);
  __syncthreads();  // rots and rmask of the last round (written by warp 0)
  for (int64_t r0 = 0; r0 < n; r0 += (int64_t)RPT * bd) {
    load(V, n, r0);
#pragma unroll 1
    for (int r = 0; r < NR; ++r) {
      if (rmask[r]) {
#pragma unroll
        for (int g = 0; g < WB; ++g) rotate(g, partner(g), rots[r][g]);
      }
      advance();
    }
    store(V, n, r0);
  }
  if (t == 0 && any_major) *rotated = 1;
}

// All FP32 sweeps of a small start in one launch: n <= 48 columns of W (m <= 32 RPT
// rows, FP64, times a power of two `scale`) and of V in shared memory, a warp a
// pair of the element-wise round robin, one barrier a round.  V goes out in FP64.
// Bound by a round's latency (sums over a warp, angle, barrier: 0.45 us); the
// blocked steps above take 8 us for eight rounds and a launch each, and the host
// has to wait for their flags: n = 48 (all of the start but its products) 390 -> 177
// us, n = 20 250 -> 52; n = 64 no longer gains.
constexpr int JS_MAX_N = 48, JS_V = 64;  // columns; rows kept of V
template <int RPT>
__global__ void __launch_bounds__(JS_MAX_N / 2 * 32)
k_jacobi32_small(const double* __restrict__ W, int m, int n, double scale, float tol, float amin,
                 float amin_conv, int max_sweeps, double* __restrict__ V) {
  constexpr int ROWS = 32 * RPT;
  extern __shared__ float js_smem[];
  float* w = js_smem;                  // [n][ROWS]
  float* v = js_smem + n * ROWS;       // [n][JS_V]
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, bd = (int)blockDim.x, np = n + (n & 1);
  for (int i = t; i < n * ROWS; i += bd) {
    const int c = i / ROWS, r = i % ROWS;
    w[i] = r < m ? (float)(W[(int64_t)c * m + r] * scale) : 0.f;
  }
  for (int i = t; i < n * JS_V; i += bd) v[i] = i / JS_V == i % JS_V ? 1.f : 0.f;
  __syncthreads();
  int p = warp, q = np - 1 - warp;
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    int major_any = 0;
    for (int step = 0; step < np - 1; ++step) {
      if (p < n && q < n) {  // warp-uniform
        float *wp = w + p * ROWS + lane, *wq = w + q * ROWS + lane;
        float *vp = v + p * JS_V + lane, *vq = v + q * JS_V + lane;
        float x[RPT], y[RPT], a = 0.f, b = 0.f, g = 0.f;
#pragma unroll
        for (int k = 0; k < RPT; ++k) {
          x[k] = wp[32 * k];
          y[k] = wq[32 * k];
          a = fmaf(x[k], x[k], a);
          b = fmaf(y[k], y[k], b);
          g = fmaf(x[k], y[k], g);
        }
        const float v0 = vp[0], v1 = vp[32], u0 = vq[0], u1 = vq[32];
        // the three sums in one tree: lanes 0-7 end with a, 8-15 with b, 16-23 with g
        const bool hi = lane & 16, mid = lane & 8;
        const float e = (hi ? g : a) + __shfl_xor_sync(0xffffffffu, hi ? a : g, 16);
        const float f = (hi ? 0.f : b) + __shfl_xor_sync(0xffffffffu, hi ? b : 0.f, 16);
        float d = (mid ? f : e) + __shfl_xor_sync(0xffffffffu, mid ? e : f, 8);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        a = __shfl_sync(0xffffffffu, d, 0);
        b = __shfl_sync(0xffffffffu, d, 8);
        g = __shfl_sync(0xffffffffu, d, 16);
        float tt, u, s;
        bool major;
        if (jp_angle<false>(a, b, g, tol, tol, amin, amin_conv, tt, u, s, major)) {
#pragma unroll
          for (int k = 0; k < RPT; ++k) {
            wp[32 * k] = fmaf(-s, fmaf(u, x[k], y[k]), x[k]);
            wq[32 * k] = fmaf(s, fmaf(-u, y[k], x[k]), y[k]);
          }
          vp[0] = fmaf(-s, fmaf(u, v0, u0), v0);
          vq[0] = fmaf(s, fmaf(-u, u0, v0), u0);
          vp[32] = fmaf(-s, fmaf(u, v1, u1), v1);
          vq[32] = fmaf(s, fmaf(-u, u1, v1), u1);
          major_any |= major;
        }
      }
      // the players of the next step (0 keeps its place)
      if (p > 0 && ++p == np) p = 1;
      if (++q == np) q = 1;
      __syncthreads();
    }
    if (!__syncthreads_or(major_any)) break;
  }
  for (int i = t; i < n * n; i += bd) V[i] = (double)v[i / n * JS_V + i % n];
}

// Self-test of the grid barrier's timeout path: every block arrives at a
// barrier that counts one participant more than the grid has, so the count
// is never met; each block waits until the limit, the first to give up raises
// the status word and all of them leave.  No block spins past the limit.
__global__ void k_grid_barrier_selftest(int* aux, unsigned long long wait_ns) {
  const bool ok = jp_grid_sync((unsigned*)aux, (unsigned*)aux + 1, aux + 2, gridDim.x + 1, wait_ns);
  if (threadIdx.x == 0 && !ok) atomicAdd(aux + 3, 1);
}

}  // namespace

namespace itg {

int grid_barrier_selftest(itg_handle* h, int* status, int* blocks_out) {
  ITG_TRY(itg_scratch_reserve(h, 8 * sizeof(int)));
  int* aux = (int*)h->scratch;
  ITG_CUDA(h, cudaMemsetAsync(aux, 0, 8 * sizeof(int), h->stream));
  k_grid_barrier_selftest<<<2, 32, 0, h->stream>>>(aux, (unsigned long long)h->wait_ns);
  ITG_CHECK_LAUNCH(h);
  int* hp = (int*)h->pinned;
  ITG_CUDA(h, cudaMemcpyAsync(hp, aux, 4 * sizeof(int), cudaMemcpyDeviceToHost, h->stream));
  ITG_TRY(itg_wait_stream(h));
  *status = hp[2];
  *blocks_out = hp[3];
  return ITG_OK;
}

int jacobi_aux_ints(int max_sweeps) { return 8 + max_sweeps; }

// The rotations V (n x n) of the FP32 start of W (m x n); false when it is too
// large for the one-launch kernel.
bool jacobi32_small_fits(const itg_handle* h, int64_t m, int64_t n) {
  return h->jacobi_mode == 0 && n >= 2 && n <= JS_MAX_N && m <= 128;
}
int jacobi32_small(itg_handle* h, const double* W, int64_t m, int64_t n, double scale, float tol, float amin,
                   float amin_conv, int max_sweeps, double* V) {
  const bool tall = m > 64;
  const size_t smem = sizeof(float) * (size_t)n * ((tall ? 128 : 64) + JS_V);
  const int threads = 32 * (int)((n + 1) / 2);
  static bool attr = false;
  if (!attr) {
    ITG_CUDA(h, cudaFuncSetAttribute(k_jacobi32_small<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024));
    ITG_CUDA(h, cudaFuncSetAttribute(k_jacobi32_small<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024));
    attr = true;
  }
  if (tall)
    k_jacobi32_small<4><<<1, threads, smem, h->stream>>>(W, (int)m, (int)n, scale, tol, amin, amin_conv, max_sweeps, V);
  else
    k_jacobi32_small<2><<<1, threads, smem, h->stream>>>(W, (int)m, (int)n, scale, tol, amin, amin_conv, max_sweeps, V);
  ITG_CHECK_LAUNCH(h);
  return ITG_OK;
}

// Runs up to max_sweeps sweeps on W (m x n) accumulating into V (n x n, set
// by the caller).  *sweeps = sweeps run; ITG_ERR_NOTCONVERGED when the limit
// was hit (results usable), ITG_ERR_UNSUPPORTED when the device cannot run a
// cooperative launch (the caller then uses per-step launches).
template <class T, int RC>
int launch_persist(itg_handle* h, T* W, int64_t m, int n, T* V, T tol, T amin, T amin_conv, int max_sweeps,
                   int* aux) {
  const T tol_conv = conv_tol(tol);
  int per_sm = 0;
  ITG_CUDA(h, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_jacobi_persist<T, RC>, JP_THREADS, 0));
  if (per_sm < 1) return ITG_ERR_UNSUPPORTED;
  if (per_sm > 4) per_sm = 4;  // fewer arrivals per barrier
  const int np = n + (n & 1);
  int64_t grid = (int64_t)h->num_sms * per_sm;
  if ((int64_t)np / 2 < grid) grid = np / 2;
  if (grid < 1) grid = 1;
  unsigned long long wait_ns = h->wait_ns;
  void* args[] = {(void*)&W,          (void*)&m,          (void*)&n,    (void*)&V,
                  (void*)&tol,        (void*)&tol_conv,   (void*)&amin, (void*)&amin_conv,
                  (void*)&max_sweeps, (void*)&aux,        (void*)&wait_ns};
  ITG_CUDA(h, cudaLaunchCooperativeKernel((const void*)k_jacobi_persist<T, RC>, dim3((unsigned)grid),
                                          dim3(JP_THREADS), args, 0, h->stream));
  return ITG_OK;
}

template <class T>
int jacobi_persistent(itg_handle* h, T* W, int64_t m, int n, T* V, T tol, T amin, int max_sweeps, int* aux,
                      int* sweeps, T amin_conv) {
  int coop = 0;
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, h->device);
  if (!coop) return ITG_ERR_UNSUPPORTED;
  ITG_CUDA(h, cudaMemsetAsync(aux, 0, sizeof(int) * jacobi_aux_ints(max_sweeps), h->stream));
  int st;
  if (m <= 4 * JP_THREADS) st = launch_persist<T, 4>(h, W, m, n, V, tol, amin, amin_conv, max_sweeps, aux);
  else if (m <= 8 * JP_THREADS) st = launch_persist<T, 8>(h, W, m, n, V, tol, amin, amin_conv, max_sweeps, aux);
  else if (m <= 16 * JP_THREADS) st = launch_persist<T, 16>(h, W, m, n, V, tol, amin, amin_conv, max_sweeps, aux);
  else st = launch_persist<T, 0>(h, W, m, n, V, tol, amin, amin_conv, max_sweeps, aux);
  if (st != ITG_OK) return st;
  int* hp = (int*)h->pinned;
  ITG_CUDA(h, cudaMemcpyAsync(hp, aux, sizeof(int) * 4, cudaMemcpyDeviceToHost, h->stream));
  ITG_TRY(itg_wait_stream(h));
  if (hp[2] != 0 || hp[3] < 0)
    return itg_fail(h, ITG_ERR_TIMEOUT, "Jacobi grid barrier timed out (n=%d)", n);
  *sweeps = hp[3] > max_sweeps ? max_sweeps : hp[3];
  return hp[3] > max_sweeps ? ITG_ERR_NOTCONVERGED : ITG_OK;
}

template <class T, int WB>
size_t jb_smem_bytes(int64_t m) {
  return sizeof(T) * ((size_t)2 * WB * m + (size_t)4 * WB * WB + (size_t)WB * (JB_THREADS / WB / 32) * 3);
}

// Sweeps of a block-cyclic kernel: launch(sweep, step) enqueues one step whose
// rotations raise flag[sweep].  Up to `chunk` sweeps are queued between two
// reads of the flags (the steps of a sweep after a converged one return at
// once), so that small problems do not wait for the host after every sweep.
template <class F>
int jb_sweeps(itg_handle* h, int steps, int max_sweeps, int chunk, int* flag, int* sweeps, F&& launch) {
  int* hp = (int*)h->pinned;
  ITG_CUDA(h, cudaMemsetAsync(flag, 0, sizeof(int) * max_sweeps, h->stream));
  for (int sw = 0; sw < max_sweeps;) {
    const int end = sw + chunk < max_sweeps ? sw + chunk : max_sweeps;
    for (int q = sw; q < end; ++q)
      for (int step = 0; step < steps; ++step) ITG_TRY(launch(q, step, q > sw ? flag + q - 1 : nullptr, flag + q));
    ITG_CUDA(h, cudaMemcpyAsync(hp, flag + sw, sizeof(int) * (end - sw), cudaMemcpyDeviceToHost, h->stream));
    ITG_TRY(itg_wait_stream(h));
    for (int q = sw; q < end; ++q)
      if (hp[q - sw] == 0) {
        *sweeps = q + 1;
        return ITG_OK;
      }
    sw = end;
  }
  *sweeps = max_sweeps;
  return ITG_ERR_NOTCONVERGED;
}

template <class T, int WB>
int jb_run(itg_handle* h, T* W, int64_t m, int n, T* V, T tol, T amin, T amin_conv, int max_sweeps, int* flag,
           int* sweeps) {
  const size_t smem = jb_smem_bytes<T, WB>(m);
  static bool attr = false;
  if (!attr) {
    ITG_CUDA(h, cudaFuncSetAttribute(k_jacobi_block_step<T, WB, JB_THREADS>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    attr = true;
  }
  const int nb = (n + WB - 1) / WB, nbp = nb + (nb & 1);
  return jb_sweeps(h, nbp - 1, max_sweeps, 1, flag, sweeps, [&](int, int step, const int*, int* rot) -> int {
    k_jacobi_block_step<T, WB, JB_THREADS><<<nbp / 2, JB_THREADS, smem, h->stream>>>(
        W, m, n, V, tol, conv_tol(tol), amin, amin_conv, step, step == 0, rot);
    ITG_CHECK_LAUNCH(h);
    return ITG_OK;
  });
}

// Register-resident steps (m <= JR_MAX_M), each launched so that it may start
// while its predecessor drains (it waits for its results itself).
template <class T, int WB, int RPT, bool VEC, int MAXT, bool FAR = false>
int jr_run_t(itg_handle* h, T* W, int64_t m, int n, T* V, T tol, T amin, T amin_conv, int max_sweeps, int* flag,
             int* sweeps) {
  const int nb = (n + WB - 1) / WB, nbp = nb + (nb & 1);
  const int threads = (int)((m + RPT - 1) / RPT + 31) / 32 * 32;
  // a queued step costs about 1 us when it has nothing to do, a look at the flags
  // about 25: FP32 takes seven sweeps and more (all seven are queued where they are
  // cheap), FP64 (after the FP32 start, which smaller problems do not take) mostly one
  const int chunk = sizeof(T) == 4 ? (n <= 160 ? 7 : (n <= 512 ? 4 : 1)) : (n < 16 ? 5 : 1);
  const dim3 grid((unsigned)(nbp / 2));
  const float tolf = (float)tol, tolc = (float)conv_tol(tol);
  return jb_sweeps(h, nbp - 1, max_sweeps, chunk, flag, sweeps, [&](int, int step, const int* prev, int* rot) {
    auto kernel = step == 0 ? k_jacobi_reg_step<T, WB, RPT, VEC, true, MAXT, FAR>
                            : k_jacobi_reg_step<T, WB, RPT, VEC, false, MAXT, FAR>;
    return itg_launch_after(h, true, grid, threads, 0, kernel, W, m, n, V, tolf, tolc, amin, amin_conv, step, prev, rot);
  });
}

// FP32: 8-column blocks, at most eight warps (each computes the angles again);
// 16-column blocks for up to 256 rows: half as many steps of twice the rounds,
// which saves their hand-over while four warps hold the pair (FP64 SVD n = 96
// 2.25 -> 2.14 ms, 150 x 120 2.76 -> 2.53, 192 4.07 -> 3.86; n = 48, an odd number of
// blocks, 1.29 -> 1.39 and n = 300, five warps, 7.3 -> 8.0).
// FP64: 4-column blocks and, up to
// 1024 rows, four warps (one for each quarter of the SM, whose FP64 pipes are
// separate).
template <class T>
int jr_run(itg_handle* h, T* W, int64_t m, int n, T* V, T tol, T amin, T amin_conv, int max_sweeps, int* flag,
           int* sweeps) {
  if constexpr (sizeof(T) == 4) {
    const bool vec = m % 4 == 0 && n % 4 == 0 && ((uintptr_t)W % 16) == 0 && ((uintptr_t)V % 16) == 0;
    if (n >= 64 && m <= 256)
      return jr_run_t<T, 16, 2, false, 128>(h, W, m, n, V, tol, amin, amin_conv, max_sweeps, flag, sweeps);
    if (m <= 1024) {
      if (vec) return jr_run_t<T, 8, 4, true, 256>(h, W, m, n, V, tol, amin, amin_conv, max_sweeps, flag, sweeps);
      return jr_run_t<T, 8, 4, false, 256>(h, W, m, n, V, tol, amin, amin_conv, max_sweeps, flag, sweeps);
    }
    if (vec) return jr_run_t<T, 8, 8, true, 256>(h, W, m, n, V, tol, amin, amin_conv, max_sweeps, flag, sweeps);
    return jr_run_t<T, 8, 8, false, 256>(h, W, m, n, V, tol, amin, amin_conv, max_sweeps, flag, sweeps);
  } else {
    auto run = [&](auto far) {
      constexpr bool F = decltype(far)::value;
      if (m <= 128) return jr_run_t<T, 4, 1, false, 128, F>(h, W, m, n, V, tol, amin, amin_conv, max_sweeps, flag, sweeps);
      if (m <= 256) return jr_run_t<T, 4, 2, false, 128, F>(h, W, m, n, V, tol, amin, amin_conv, max_sweeps, flag, sweeps);
      if (m <= 512) return jr_run_t<T, 4, 4, false, 128, F>(h, W, m, n, V, tol, amin, amin_conv, max_sweeps, flag, sweeps);
      return jr_run_t<T, 4, 8, false, 256, F>(h, W, m, n, V, tol, amin, amin_conv, max_sweeps, flag, sweeps);
    };
    // columns of any size count: a graded matrix
    if (amin_conv == T(0)) return run(std::true_type());
    return run(std::false_type());
  }
}

// Blocked Jacobi with the widest block whose column pair fits in 200 KB of
// shared memory; ITG_ERR_UNSUPPORTED when not even 2 + 2 columns fit.
template <class T>
int jacobi_blocked(itg_handle* h, T* W, int64_t m, int n, T* V, T tol, T amin, int max_sweeps, int* flag,
                   int* sweeps, T amin_conv) {
  constexpr size_t LIM = 200 * 1024;
  if (n < 2) {
    *sweeps = 0;
    return ITG_OK;
  }
  if (h->jacobi_mode == 0 && m <= JR_MAX_M)
    return jr_run<T>(h, W, m, n, V, tol, amin, amin_conv, max_sweeps, flag, sweeps);
  // jacobi_mode 3 keeps the blocks at 4 columns (half the shared memory per CTA, more CTAs per SM)
  if (h->jacobi_mode != 3 && jb_smem_bytes<T, 8>(m) <= LIM && n >= 64)
    return jb_run<T, 8>(h, W, m, n, V, tol, amin, amin_conv, max_sweeps, flag, sweeps);
  if (jb_smem_bytes<T, 4>(m) <= LIM) return jb_run<T, 4>(h, W, m, n, V, tol, amin, amin_conv, max_sweeps, flag, sweeps);
  if (jb_smem_bytes<T, 2>(m) <= LIM) return jb_run<T, 2>(h, W, m, n, V, tol, amin, amin_conv, max_sweeps, flag, sweeps);
  return ITG_ERR_UNSUPPORTED;
}

template int jacobi_blocked<float>(itg_handle*, float*, int64_t, int, float*, float, float, int, int*, int*, float);
template int jacobi_blocked<double>(itg_handle*, double*, int64_t, int, double*, double, double, int, int*, int*,
                                     double);

template int jacobi_persistent<float>(itg_handle*, float*, int64_t, int, float*, float, float, int, int*, int*,
                                       float);
template int jacobi_persistent<double>(itg_handle*, double*, int64_t, int, double*, double, double, int, int*,
                                        int*, double);

}  // namespace itg

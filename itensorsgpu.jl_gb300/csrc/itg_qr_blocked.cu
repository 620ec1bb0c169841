// Blocked Householder QR and the application of its Q, with the trailing
// updates as matrix products by kernels of their own (compact WY form
// of Schreiber & Van Loan, "A storage-efficient WY representation for
// products of Householder transformations", SIAM J. Sci. Stat. Comput. 10
// (1989); the T recurrence is LAPACK's larft, restated).
//
// Panel of QR_NB columns: the column steps of k_house_step (itg_factor.cu)
// restricted to the panel, then T (upper triangular, Q_p = I - V T V^T) from
// Y = V^T V, then the trailing columns A_t <- (I - V T^T V^T) A_t: the partial
// sums of Z = V^T A_t over chunks of K, Z2 = T^T Z together with their
// reduction, A_t -= V Z2.  Q [X; 0] applies the panels in reverse order with
// Y <- Y - V (T (V^T Y)).  All of it is FP64.
#include "itg_internal.cuh"

#include <utility>

namespace itg {
int house_panel(itg_handle* h, bool fast, double* A, int64_t m, int64_t j0, int64_t count, int64_t jend, double* Vh,
                double* tau, double* rdiag);
}  // namespace itg

namespace {

// T (32 x 32, upper triangular) from the partial sums of Y = V^T V (column c
// of chunk q at part[32 (q bw + c)]): LAPACK's larft,
//   T(j,j) = tau_j, T(0:j, j) = -tau_j T(0:j, 0:j) Y(0:j, j),
// with its sums formed one term a step for all elements at once (lane i of warp
// j % 8 adds T(i,l) Y(l,j) as soon as column l is final: the order of the
// recurrence, bw steps instead of a chain of 500 FP64 instructions).  Bound by
// a step's latency (a product, a barrier, a sum of up to four columns a warp);
// eight warps instead of 32 shorten its barrier (21 -> 14 us at bw = 32).
__global__ void __launch_bounds__(256)
k_larft(const double* __restrict__ part, int nchunk, const double* __restrict__ tau, int bw, double* __restrict__ T) {
  constexpr int NB = QR_NB, NW = 8, CW = NB / NW;
  __shared__ double Y[NB][NB + 1], col[2][NB];  // Y[column][row]; column l of T
  itg_grid_wait();
  const int i = threadIdx.x % NB, w = threadIdx.x / NB;
  double tj[CW], s[CW], t[CW];
#pragma unroll
  for (int c = 0; c < CW; ++c) {
    const int j = w + NW * c;
    tj[c] = j < bw ? tau[j] : 0.0;
    s[c] = t[c] = 0.0;
    double y = 0.0;
    if (i < j && j < bw)
      for (int q = 0; q < nchunk; ++q) y += part[((int64_t)q * bw + j) * NB + i];
    Y[j][i] = y;
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < CW; ++c) {
    const int end = bw < NW * (c + 1) ? bw : NW * (c + 1);
    for (int l = NW * c; l < end; ++l) {
      if (w == l % NW) {
        t[c] = i < l ? -tj[c] * s[c] : (i == l ? tj[c] : 0.0);
        col[l & 1][i] = t[c];
      }
      __syncthreads();
      if (i <= l) {
        const double x = col[l & 1][i];
#pragma unroll
        for (int d = c; d < CW; ++d)
          if (w + NW * d > l) s[d] = fma(x, Y[w + NW * d][l], s[d]);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < CW; ++c) T[(w + NW * c) * NB + i] = t[c];
}

// Partial sums of V_p^T B for the panel's reflectors V_p (columns jb..jb+bw of
// Vh, rows jb..m) and N columns of B (ld ldb, rows jb..m): bw <= 32 rows of
// dot products of length K = m - jb.  The product is too thin for the tiled
// GEMM (it would run N / 64 CTAs), so the K range is split over gridDim.y
// chunks whose partial results are summed in chunk order by the consumer, and
// the 32 rows over gridDim.z: FP64 runs at 2 FMAs a clock and SM whatever the
// tile, so a tile is one element a thread (8 rows by 32 columns, a warp a row).
// With 32 rows a block (four elements a thread) a panel's 32 columns at K = 378
// took 18.7 us on 6 SMs; now 7 on 24, the same sums.
constexpr int SK_TILE_K = 64, SK_ROWS = 8;
constexpr int QR_PART_CHUNKS = 16;  // K chunks of the thin products (partials: 16 x 32 x N)
__global__ void __launch_bounds__(256)
k_skinny_partial(const double* __restrict__ Vh, int64_t m, int64_t jb, int bw, const double* __restrict__ B,
                 int64_t ldb, int64_t b0, int64_t N, int64_t kchunk, double* __restrict__ part) {
  __shared__ double vs[SK_ROWS][SK_TILE_K];
  __shared__ double bs[32][SK_TILE_K + 1];
  itg_grid_wait();
  const int t = threadIdx.x, r = t / 32, c = t % 32, r0 = blockIdx.z * SK_ROWS;
  const int64_t c0 = (int64_t)blockIdx.x * 32;
  const int64_t K = m - jb;
  const int64_t k_lo = (int64_t)blockIdx.y * kchunk;
  const int64_t k_hi = k_lo + kchunk < K ? k_lo + kchunk : K;
  double acc = 0.0;
  for (int64_t k0 = k_lo; k0 < k_hi; k0 += SK_TILE_K) {
#pragma unroll
    for (int i = t; i < SK_ROWS * SK_TILE_K; i += 256) {
      const int col = i / SK_TILE_K, kk = i % SK_TILE_K;
      vs[col][kk] = (k0 + kk < k_hi && r0 + col < bw) ? Vh[(jb + r0 + col) * m + jb + k0 + kk] : 0.0;
    }
#pragma unroll
    for (int i = t; i < 32 * SK_TILE_K; i += 256) {
      const int col = i / SK_TILE_K, kk = i % SK_TILE_K;
      bs[col][kk] = (k0 + kk < k_hi && c0 + col < N) ? B[(b0 + c0 + col) * ldb + jb + k0 + kk] : 0.0;
    }
    __syncthreads();
#pragma unroll 16
    for (int kk = 0; kk < SK_TILE_K; ++kk) acc = fma(vs[r][kk], bs[c][kk], acc);
    __syncthreads();
  }
  if (c0 + c < N) part[((int64_t)blockIdx.y * N + c0 + c) * 32 + r0 + r] = acc;
}

// Z2 (32 x N) = op(T) Z with Z the sum of the partial results in chunk order,
// op(T) = T^T or T; rows bw.. of Z2 are zero.  One thread an element, eight
// columns a block.
template <bool TRANS>
__global__ void __launch_bounds__(256)
k_skinny_t(const double* __restrict__ part, int nchunk, int bw, int64_t N, const double* __restrict__ T,
           double* __restrict__ Z2) {
  constexpr int NB = QR_NB;
  __shared__ double z[8][NB], Ts[NB][NB + 1];
  const int t = threadIdx.x, r = t % NB, cl = t / NB;
  const int64_t c = (int64_t)blockIdx.x * 8 + cl;
  itg_grid_wait();
  for (int i = t; i < NB * NB; i += 256) Ts[i / NB][i % NB] = T[i];  // [column][row]
  double s = 0.0;
  if (c < N && r < bw)
    for (int q = 0; q < nchunk; ++q) s += part[((int64_t)q * N + c) * NB + r];
  z[cl][r] = s;
  __syncthreads();
  if (c >= N) return;
  double a = 0.0;
  if (TRANS) {
    for (int l = 0; l <= r; ++l) a = fma(Ts[r][l], z[cl][l], a);
  } else {
    for (int l = r; l < NB; ++l) a = fma(Ts[l][r], z[cl][l], a);
  }
  Z2[c * NB + r] = r < bw ? a : 0.0;
}

// C(jb:m, c0 : c0 + N) -= V_p Z2 (C of leading dimension m).  Like every FP64
// product here bound by the FP64 pipe whatever its tile: 32 x 16 tiles of four
// elements a thread, or 16 x 8 of one (HALF) when those would leave SMs idle.
// One panel's columns at m = 378: 9.7 -> 7 us.
template <bool HALF>
__global__ void __launch_bounds__(128)
k_wy_update(const double* __restrict__ Vh, int64_t m, int64_t jb, int bw, const double* __restrict__ Z2, int64_t N,
            double* __restrict__ C, int64_t c0) {
  constexpr int NB = QR_NB, TM = HALF ? 16 : 32, TN = HALF ? 8 : 16, U = HALF ? 1 : 2;
  __shared__ double vs[NB][TM + 1], zs[TN][NB + 1];
  itg_grid_wait();
  const int t = threadIdx.x;
  const int64_t r0 = jb + (int64_t)blockIdx.x * TM, n0 = (int64_t)blockIdx.y * TN;
#pragma unroll
  for (int i = t; i < TM * NB; i += 128) {
    const int k = i / TM, r = i % TM;
    vs[k][r] = (k < bw && r0 + r < m) ? Vh[(jb + k) * m + r0 + r] : 0.0;
  }
#pragma unroll
  for (int i = t; i < TN * NB; i += 128) {
    const int c = i / NB, k = i % NB;
    zs[c][k] = n0 + c < N ? Z2[(n0 + c) * NB + k] : 0.0;
  }
  const int tr = t % 16, tc = t / 16;
  double acc[U][U], old[U][U];
#pragma unroll
  for (int a = 0; a < U; ++a)
#pragma unroll
    for (int b = 0; b < U; ++b) {
      const int64_t r = r0 + tr + 16 * a, c = n0 + tc + 8 * b;
      old[a][b] = (r < m && c < N) ? C[(c0 + c) * m + r] : 0.0;
      acc[a][b] = 0.0;
    }
  __syncthreads();
#pragma unroll 8
  for (int k = 0; k < NB; ++k)
#pragma unroll
    for (int a = 0; a < U; ++a)
#pragma unroll
      for (int b = 0; b < U; ++b) acc[a][b] = fma(vs[k][tr + 16 * a], zs[tc + 8 * b][k], acc[a][b]);
#pragma unroll
  for (int a = 0; a < U; ++a)
#pragma unroll
    for (int b = 0; b < U; ++b) {
      const int64_t r = r0 + tr + 16 * a, c = n0 + tc + 8 * b;
      if (r < m && c < N) C[(c0 + c) * m + r] = old[a][b] - acc[a][b];
    }
}

// Partial sums of V_p^T B into part; nchunk: how many.
int skinny_vt_b(itg_handle* h, const double* Vh, int64_t m, int64_t jb, int bw, const double* B,
                int64_t ldb, int64_t b0, int64_t N, double* part, int64_t part_doubles, int* nchunk_out) {
  const int64_t K = m - jb;
  const int64_t ntile = (N + 31) / 32;
  int64_t nchunk = (4 * (int64_t)h->num_sms + ntile - 1) / ntile;
  const int64_t maxc = (K + SK_TILE_K - 1) / SK_TILE_K;
  if (nchunk > maxc) nchunk = maxc;
  if (nchunk > part_doubles / (32 * N)) nchunk = part_doubles / (32 * N);
  if (nchunk < 1) return itg_fail(h, ITG_ERR_INVALID, "skinny product: partial buffer too small");
  const int64_t kchunk = ((K + nchunk - 1) / nchunk + SK_TILE_K - 1) / SK_TILE_K * SK_TILE_K;
  nchunk = (K + kchunk - 1) / kchunk;
  const dim3 grid((unsigned)ntile, (unsigned)nchunk, 32 / SK_ROWS);
  ITG_TRY(itg_launch_after(h, true, grid, 256, 0, k_skinny_partial, Vh, m, jb, bw, B, ldb, b0, N, kchunk,
                           part));
  *nchunk_out = (int)nchunk;
  return ITG_OK;
}

// C(jb:m, c0 : c0 + N) -= V_p (op(T_p) (V_p^T C(jb:m, c0 : c0 + N))) on the
// handle's current stream; Z2 holds 32 N doubles.
template <bool TRANS>
int wy_apply(itg_handle* h, double* C, int64_t m, int64_t jb, int bw, const double* Vh,
             const double* Tp, int64_t c0, int64_t N, double* Z2, double* part, int64_t part_doubles) {
  if (N <= 0) return ITG_OK;
  int nchunk = 0;
  ITG_TRY(skinny_vt_b(h, Vh, m, jb, bw, C, m, c0, N, part, part_doubles, &nchunk));
  ITG_TRY(itg_launch_after(h, true, dim3((unsigned)((N + 7) / 8)), 256, 0, k_skinny_t<TRANS>, part, nchunk, bw, N, Tp,
                           Z2));
  const bool half = ((m - jb + 31) / 32) * ((N + 15) / 16) < h->num_sms;
  const int tm = half ? 16 : 32, tn = half ? 8 : 16;
  const int64_t gx = (m - jb + tm - 1) / tm, gy = (N + tn - 1) / tn;
  for (int64_t y = 0; y < gy; y += 65535) {  // the grid's y limit
    const dim3 grid((unsigned)gx, (unsigned)(gy - y < 65535 ? gy - y : 65535));
    ITG_TRY(itg_launch_after(h, true, grid, 128, 0, half ? k_wy_update<true> : k_wy_update<false>, Vh, m, jb, bw,
                             Z2 + y * tn * QR_NB, N - y * tn, C, c0 + y * tn));
  }
  return ITG_OK;
}

}  // namespace

namespace itg {

// Blocked Householder QR (fast: with the column steps of house_panel's fast
// form) of W (m x n, ld m) in place with nref <= min(m, n)
// reflectors (nref = n for the tall case, m for a wide matrix): reflectors in
// Vh (m x nref, explicit unit diagonal, zeros above), tau, R's diagonal in rd,
// the rest of R's rows above the diagonal in W; Tbuf holds QR_NB^2 doubles
// per panel of reflectors and ws qr_blocked_ws_doubles(n) doubles.
//
// Look-ahead: the column steps of a panel are bound by their serial FP64
// scalar work and occupy few SMs.  They run on a stream of the greatest
// priority (qr_stream), so that their blocks are scheduled ahead of the
// trailing updates' product blocks, which run on the handle's stream: once
// panel p's reflectors and T are final, the panel stream updates the columns
// of panel p + 1 by them and factors panel p + 1 at once, while the handle's
// stream updates the rest of the trailing matrix by panel p.  The panel stream
// waits for that update before it applies the next panel's reflectors to the
// columns the update covers.  Each stream has its own Z2 and partial-sum
// buffers.  Results are deterministic (the split of V^T A's K
// range into chunks depends only on the column counts).
namespace {
// The handle's stream is swapped for the panel stream while this lives, and with
// it whether the stream's last thing is a kernel (chained: the panel stream's).
struct OnStream {
  itg_handle* h;
  cudaStream_t saved;
  bool& chained;
  OnStream(itg_handle* hh, cudaStream_t s, bool& c) : h(hh), saved(hh->stream), chained(c) {
    h->stream = s;
    std::swap(h->chained, chained);
  }
  ~OnStream() {
    h->stream = saved;
    std::swap(h->chained, chained);
  }
};

int qr_lookahead_init(itg_handle* h) {
  if (h->qr_stream) return ITG_OK;
  int least = 0, greatest = 0;
  ITG_CUDA(h, cudaDeviceGetStreamPriorityRange(&least, &greatest));
  ITG_CUDA(h, cudaStreamCreateWithPriority(&h->qr_stream, cudaStreamNonBlocking, greatest));
  ITG_CUDA(h, cudaEventCreateWithFlags(&h->qr_ev_ready, cudaEventDisableTiming));
  ITG_CUDA(h, cudaEventCreateWithFlags(&h->qr_ev_done, cudaEventDisableTiming));
  return ITG_OK;
}
}  // namespace

int qr_blocked(itg_handle* h, double* W, int64_t m, int64_t n, int64_t nref, double* Vh, double* tau, double* rd,
               double* Tbuf, double* ws, bool fast) {
  const int NB = QR_NB;
  const int64_t part_doubles = QR_PART_CHUNKS * 32 * n;
  double *Zp = ws, *partp = Zp + (int64_t)NB * n;                          // panel stream
  double *Zu = partp + part_doubles, *partu = Zu + (int64_t)NB * n;        // the handle's stream
  ITG_TRY(qr_lookahead_init(h));
  cudaStream_t main_stream = h->stream;
  bool chained = false;  // of the panel stream
  // the panel stream starts after everything already queued on the handle's stream
  ITG_CUDA(h, cudaEventRecord(h->qr_ev_done, main_stream));
  {
    OnStream on(h, h->qr_stream, chained);
    ITG_CUDA(h, cudaStreamWaitEvent(h->stream, h->qr_ev_done, 0));
    if (nref > 0) {
      const int64_t w = nref < NB ? nref : NB;
      ITG_TRY(house_panel(h, fast, W, m, 0, w, w, Vh, tau, rd));
    }
  }
  for (int64_t jb = 0, panel = 0; jb < nref; jb += NB, ++panel) {
    const int64_t bw = (nref - jb < NB) ? nref - jb : NB;
    const int64_t nt = n - jb - bw;
    double* Tp = Tbuf + panel * NB * NB;
    const int64_t jn = jb + bw;
    const int64_t nnext = nt > 0 && jn < nref ? ((nref - jn < NB) ? nref - jn : NB) : 0;
    const int64_t nrest = nt > 0 ? nt - nnext : 0;
    {
      OnStream on(h, h->qr_stream, chained);
      int nchunk = 0;
      ITG_TRY(skinny_vt_b(h, Vh, m, jb, (int)bw, Vh, m, jb, bw, partp, part_doubles, &nchunk));
      ITG_TRY(itg_launch_after(h, true, dim3(1), 256, 0, k_larft, partp, nchunk, tau + jb, (int)bw, Tp));
      if (nt <= 0) continue;
      // V_p and T_p are final: the handle's stream may update the rest
      ITG_CUDA(h, cudaEventRecord(h->qr_ev_ready, h->stream));
      // panel p + 1's columns got panel p - 1's update on the handle's stream
      if (panel > 0) ITG_CUDA(h, cudaStreamWaitEvent(h->stream, h->qr_ev_done, 0));
      ITG_TRY(wy_apply<true>(h, W, m, jb, (int)bw, Vh, Tp, jn, nnext, Zp, partp, part_doubles));
    }
    if (nrest > 0) {
      ITG_CUDA(h, cudaStreamWaitEvent(main_stream, h->qr_ev_ready, 0));
      ITG_TRY(wy_apply<true>(h, W, m, jb, (int)bw, Vh, Tp, jn + nnext, nrest, Zu, partu, part_doubles));
    }
    ITG_CUDA(h, cudaEventRecord(h->qr_ev_done, main_stream));
    if (nnext > 0) {
      OnStream on(h, h->qr_stream, chained);
      ITG_TRY(house_panel(h, fast, W, m, jn, nnext, jn + nnext, Vh, tau, rd));
    }
  }
  // the handle's stream continues after the last panel's work
  ITG_CUDA(h, cudaEventRecord(h->qr_ev_ready, h->qr_stream));
  ITG_CUDA(h, cudaStreamWaitEvent(main_stream, h->qr_ev_ready, 0));
  return ITG_OK;
}

// Y <- Q Y on the first ncols columns of Y (m rows, ld m), Q from qr_blocked of
// n reflectors; ws: qr_blocked_ws_doubles(ncols) doubles.
int q_apply_blocked(itg_handle* h, double* Y, int64_t m, int64_t n, int64_t ncols, const double* Vh,
                    const double* Tbuf, double* ws) {
  if (ncols <= 0) return ITG_OK;
  const int NB = QR_NB;
  double *Z2 = ws, *part = Z2 + (int64_t)NB * ncols;
  const int64_t npanel = (n + NB - 1) / NB;
  for (int64_t panel = npanel - 1; panel >= 0; --panel) {
    const int64_t jb = panel * NB;
    const int64_t bw = (n - jb < NB) ? n - jb : NB;
    ITG_TRY(wy_apply<false>(h, Y, m, jb, (int)bw, Vh, Tbuf + panel * NB * NB, 0, ncols, Z2, part,
                            QR_PART_CHUNKS * 32 * ncols));
  }
  return ITG_OK;
}

// Z2 and the partial sums of the panel stream, then those of the handle's.
size_t qr_blocked_ws_doubles(int64_t n) { return 2 * ((size_t)QR_NB * n + (size_t)QR_PART_CHUNKS * 32 * n); }
size_t qr_blocked_t_doubles(int64_t n) { return (size_t)((n + QR_NB - 1) / QR_NB) * QR_NB * QR_NB; }

}  // namespace itg

// Tensor permutation and permuted axpby (K2, K3).
//
// B[perm(i)] = alpha * A[i] (+ beta * Bin) for column-major tensors.  The host
// side first fuses modes that stay adjacent in both layouts, then picks one of
// two HBM-bound kernels:
//   * row copy  — A's fastest mode is also B's fastest: both sides stream
//                 contiguous rows, several short ones or a segment of a long
//                 one per CTA.
//   * transpose — different fastest modes: tiles staged through shared memory
//                 so that reads of A and writes of B are both coalesced.
// Both take items of about 4096 elements (fewer where there are few) with eight
// loads of every thread in flight, or the transpose 32 x 32 tiles with four
// (perm_tiles32, perm_few_tiles).
#include "itg_internal.cuh"

#include <algorithm>
#include <type_traits>

namespace {

struct PermDesc {
  int rank;                        // after fusion
  int64_t dims[ITG_MAX_RANK];      // in A's order
  int64_t strA[ITG_MAX_RANK];      // stride of A's mode i in A
  int64_t strB[ITG_MAX_RANK];      // stride of A's mode i in B
};

// Remaining-mode decomposition used by both kernels: modes listed in `idx`.
struct RestDesc {
  int n;
  int64_t dims[ITG_MAX_RANK];
  int64_t strA[ITG_MAX_RANK];
  int64_t strB[ITG_MAX_RANK];
};

__device__ __forceinline__ void rest_offsets(const RestDesc& r, int64_t lin, int64_t& oa,
                                             int64_t& ob) {
  oa = 0;
  ob = 0;
  for (int i = 0; i < r.n; ++i) {
    int64_t d = r.dims[i];
    int64_t q;
    if (((lin | d) >> 32) == 0) q = (int64_t)((uint32_t)lin / (uint32_t)d);
    else q = lin / d;
    int64_t c = lin - q * d;
    lin = q;
    oa += c * r.strA[i];
    ob += c * r.strB[i];
  }
}

// x / d for x, d <= 2^16: the upper half of x * ceil(2^32 / d)
struct FastDiv {
  uint32_t d, m;
  __device__ __forceinline__ uint32_t div(uint32_t x) const { return d == 1 ? x : __umulhi(x, m); }
};
inline FastDiv fast_div(uint32_t d) {
  return {d, d == 1 ? 0u : (uint32_t)(((1ull << 32) + d - 1) / d)};
}

constexpr int PERM_THREADS = 256;
constexpr int PERM_ITEM = 4096;  // elements per item
constexpr int PERM_FLIGHT = 8;   // loads of a thread in flight
constexpr int PERM_ROWS = 256;   // rows per item at most

// B = alpha A + beta Bin element by element.  The FP64 pipe (two operations a
// clock and SM, 0.6 of HBM's rate in 16-byte element copies) is spared where
// the scalars allow: a copy with alpha = +-1 takes no FP64 operation, a sum
// with beta = 1 and alpha = +-1 one, each with the bits of the general form.
enum PermOp { PERM_COPY, PERM_SCALE, PERM_ADD, PERM_AXPBY };
struct PermScalars {
  double alpha, beta;
  long long flip;  // sign bit of alpha (PERM_COPY, PERM_ADD)
};
template <int OP>
__device__ __forceinline__ double perm_op(const PermScalars& s, double a, double b) {
  if (OP == PERM_COPY || OP == PERM_ADD) {
    const double x = __longlong_as_double(__double_as_longlong(a) ^ s.flip);
    return OP == PERM_COPY ? x : x + b;
  }
  return OP == PERM_SCALE ? s.alpha * a : fma(s.beta, b, s.alpha * a);
}
constexpr bool perm_reads_b(int op) { return op == PERM_ADD || op == PERM_AXPBY; }

// Item: `rows` rows of length d0 (stride 1 in A and B), or (nseg > 1) one
// segment of seg elements of a row.  The rows' offsets are decomposed once per
// item, one row a thread.  Bin may be B: every element is read before it is
// written, by the same thread.  Measured: (d0, d2, d1, d3) of 129 x 250 x 64 x 63
// 767 -> 322 us (95% of measured HBM); a sum of 2^26 elements in one order, which
// is a single row, 110 ms (one CTA) -> 0.27 ms.
template <int OP>
__global__ void __launch_bounds__(PERM_THREADS, 4)
k_perm_rows(const double* __restrict__ A, double* B, const double* Bin, PermScalars sc, int64_t d0, int64_t nrows,
            int rows, int64_t seg, int64_t nseg, FastDiv by_d0, int64_t items, RestDesc rest) {
  __shared__ int64_t oa[PERM_ROWS], ob[PERM_ROWS];
  for (int64_t it = blockIdx.x; it < items; it += gridDim.x) {
    const int64_t row0 = nseg > 1 ? it / nseg : it * rows;
    const int64_t i0 = nseg > 1 ? (it - row0 * nseg) * seg : 0;
    const int nr = (int)(nrows - row0 < rows ? nrows - row0 : rows);
    __syncthreads();  // the offsets of the item before
    if ((int)threadIdx.x < nr) {
      int64_t x, y;
      rest_offsets(rest, row0 + threadIdx.x, x, y);
      oa[threadIdx.x] = x + i0;
      ob[threadIdx.x] = y + i0;
    }
    __syncthreads();
    const int len = (int)(nseg > 1 ? (d0 - i0 < seg ? d0 - i0 : seg) : d0);
    const int total = nr * len;
    for (int e0 = threadIdx.x; e0 < total; e0 += PERM_THREADS * PERM_FLIGHT) {
      double v[PERM_FLIGHT], w[PERM_FLIGHT];
      int64_t o[PERM_FLIGHT];
#pragma unroll
      for (int u = 0; u < PERM_FLIGHT; ++u) {
        const int e = e0 + u * PERM_THREADS;
        o[u] = -1;
        if (e < total) {
          const int r = nseg > 1 ? 0 : (int)by_d0.div(e);
          const int i = e - r * len;
          v[u] = A[oa[r] + i];
          o[u] = ob[r] + i;
          if (perm_reads_b(OP)) w[u] = Bin[o[u]];
        }
      }
#pragma unroll
      for (int u = 0; u < PERM_FLIGHT; ++u) {
        if (e0 - (int)threadIdx.x + u * PERM_THREADS >= total) break;  // the block's: no products for nobody
        if (o[u] >= 0) B[o[u]] = perm_op<OP>(sc, v[u], perm_reads_b(OP) ? w[u] : 0.0);
      }
    }
  }
}

// Tiled transpose between A's mode 0 (size n0, stride 1 in A, stride s0B in B)
// and A's mode q (size nq, stride sqA in A, stride 1 in B): e0 x eq tiles,
// equal within a mode, so a length just above a multiple leaves no sliver (129
// = 3 x 43); up to 64 wide, so that a tile row is 512 contiguous bytes on both
// sides.  Lanes run along the contiguous mode in two halves, 2^l0 (2^lq) of
// them to a row where the mode is short.  Four CTAs to an SM (at 78 registers,
// three, sums ran at 86 instead of 94% of HBM).  Measured against 32 x 32
// tiles with the general scalars: 129 x 250 x 64 x 63 reversed 495 -> 365 us,
// 128 x 256 x 64 x 64 reversed 392 -> 340 us (94% of measured HBM), its sum 625
// -> 530 us.
template <int OP>
__global__ void __launch_bounds__(PERM_THREADS, 4)
k_perm_transpose(const double* __restrict__ A, double* B, const double* Bin, PermScalars sc, int64_t n0, int64_t nq,
                 int64_t sqA, int64_t s0B, int e0, int eq, int l0, int lq, int64_t t0, int64_t tq, int64_t items,
                 RestDesc rest) {
  extern __shared__ double tile[];  // [eq][pitch], the pitch odd: no bank conflicts along either side
  const int pitch = e0 | 1;
  const int rx = threadIdx.x & ((1 << l0) - 1), ry = threadIdx.x >> l0, rstep = PERM_THREADS >> l0;
  const int wx = threadIdx.x & ((1 << lq) - 1), wy = threadIdx.x >> lq, wstep = PERM_THREADS >> lq;
  for (int64_t it = blockIdx.x; it < items; it += gridDim.x) {
    const int64_t tiles = t0 * tq;
    int64_t b, r, iq;
    if ((items >> 32) == 0) {
      b = (uint32_t)it / (uint32_t)tiles;
      r = it - b * tiles;
      iq = (uint32_t)r / (uint32_t)t0;
    } else {
      b = it / tiles;
      r = it - b * tiles;
      iq = r / t0;
    }
    const int64_t i0 = (r - iq * t0) * e0, k0 = iq * eq;
    int64_t oa, ob;
    rest_offsets(rest, b, oa, ob);
    const int w0 = (int)(n0 - i0 < e0 ? n0 - i0 : e0), wq = (int)(nq - k0 < eq ? nq - k0 : eq);
    // read along mode 0 (contiguous in A): rows ry, ry + rstep, ..., lanes rx and rx + 2^l0, ...
    {
      const double* a = A + oa + i0 + k0 * sqA;
      for (int x = rx; x < w0; x += 2 << l0) {
        const bool two = x + (1 << l0) < w0;
        for (int k = ry; k < wq; k += 4 * rstep) {
          double v[4][2];
          const double* p = a + x + k * sqA;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (k + j * rstep < wq) {
              v[j][0] = p[j * rstep * sqA];
              if (two) v[j][1] = p[j * rstep * sqA + (1 << l0)];
            }
          double* q = tile + k * pitch + x;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (k + j * rstep < wq) {
              q[j * rstep * pitch] = v[j][0];
              if (two) q[j * rstep * pitch + (1 << l0)] = v[j][1];
            }
        }
      }
    }
    __syncthreads();
    // write along mode q (contiguous in B)
    {
      const int64_t o0 = ob + k0 + i0 * s0B;
      for (int x = wx; x < wq; x += 2 << lq) {
        const bool two = x + (1 << lq) < wq;
        for (int i = wy; i < w0; i += 4 * wstep) {
          double v[4][2], w[4][2];
          const double* q = tile + x * pitch + i;
          double* p = B + o0 + x + i * s0B;
          const double* pb = Bin + o0 + x + i * s0B;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (i + j * wstep < w0) {
              if (perm_reads_b(OP)) {
                w[j][0] = pb[j * wstep * s0B];
                if (two) w[j][1] = pb[j * wstep * s0B + (1 << lq)];
              }
              v[j][0] = q[j * wstep];
              if (two) v[j][1] = q[j * wstep + (pitch << lq)];
            }
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (i + j * wstep < w0) {
              p[j * wstep * s0B] = perm_op<OP>(sc, v[j][0], perm_reads_b(OP) ? w[j][0] : 0.0);
              if (two)
                p[j * wstep * s0B + (1 << lq)] = perm_op<OP>(sc, v[j][1], perm_reads_b(OP) ? w[j][1] : 0.0);
            }
        }
      }
    }
    __syncthreads();
  }
}

// The transpose by 32 x 32 tiles, blockIdx.y over the batches: four loads a
// thread and eight CTAs an SM instead of eight and four.  It is the better one
// where the scalars need FP64 instructions (they run between the loads of more
// CTAs: 1.5 A - 0.5 B of 100 x 90 x 80 x 70 0.40 -> 0.32 ms), where modes are short or
// equal tiles leave lanes idle that these fill (perm_tiles32), and where there are
// few tiles at all (perm_few_tiles).
template <int OP>
__global__ void __launch_bounds__(256)
k_perm_transpose32(const double* __restrict__ A, double* B, const double* Bin, PermScalars sc, int64_t n0, int64_t nq,
                   int64_t sqA, int64_t s0B, int64_t nbatch, RestDesc rest) {
  constexpr int TP = 32;
  __shared__ double tile[TP][TP + 1];
  const int t0 = (int)((n0 + TP - 1) / TP), tq = (int)((nq + TP - 1) / TP), tiles = t0 * tq;
  for (int64_t b = blockIdx.y; b < nbatch; b += gridDim.y) {
    int64_t oa, ob;
    rest_offsets(rest, b, oa, ob);
    for (int r = blockIdx.x; r < tiles; r += gridDim.x) {
      const int iq = r / t0, i0 = r - iq * t0;
      const int64_t base0 = (int64_t)i0 * TP, baseq = (int64_t)iq * TP;
      // read along mode 0 (contiguous in A), all loads first
      double v[TP / 8];
#pragma unroll
      for (int j = 0; j < TP / 8; ++j) {
        const int64_t i = base0 + threadIdx.x, k = baseq + threadIdx.y + 8 * j;
        v[j] = (i < n0 && k < nq) ? A[oa + i + k * sqA] : 0.0;
      }
#pragma unroll
      for (int j = 0; j < TP / 8; ++j) tile[threadIdx.y + 8 * j][threadIdx.x] = v[j];
      __syncthreads();
      // write along mode q (contiguous in B)
#pragma unroll
      for (int j = 0; j < TP / 8; ++j) {
        const int y = threadIdx.y + 8 * j;
        const int64_t k = baseq + threadIdx.x, i = base0 + y;
        if (i < n0 && k < nq) {
          const int64_t o = ob + k + i * s0B;
          B[o] = perm_op<OP>(sc, tile[threadIdx.x][y], perm_reads_b(OP) ? Bin[o] : 0.0);
        }
      }
      __syncthreads();
    }
  }
}

// Tile of the transpose: about 64 x 64, the other side longer where one mode
// is short, and equal tiles within each mode; padded rows fit in 35 KB (of the
// four CTAs of an SM 140).  l0, lq: log2 of the lanes along each mode.
void perm_tile(int64_t n0, int64_t nq, int& e0, int& eq, int& l0, int& lq) {
  auto even = [](int64_t n, int64_t cap) { return (int)((n + (n + cap - 1) / cap - 1) / ((n + cap - 1) / cap)); };
  int64_t c0 = 64, cq = 64;
  if (n0 < 64) cq = 4352 / (n0 | 1);
  else if (nq < 64) c0 = 4352 / nq - 1;
  e0 = even(n0, c0);
  eq = even(nq, cq);
  auto lanes = [](int e) {
    int l = 0;
    while (l < 5 && (1 << l) < e) ++l;
    return l;
  };
  l0 = lanes(e0);
  lq = lanes(eq);
}

template <int OP>
void perm_launch_rows(int blocks, cudaStream_t st, const double* A, double* B, const double* Bin, PermScalars sc,
                      int64_t d0, int64_t nrows, int rows, int64_t seg, int64_t nseg, int64_t items,
                      const RestDesc& rest) {
  k_perm_rows<OP><<<blocks, PERM_THREADS, 0, st>>>(A, B, Bin, sc, d0, nrows, rows, seg, nseg,
                                                   fast_div(nseg > 1 ? 1 : (uint32_t)d0), items, rest);
}

// Whether 32 x 32 tiles take the transpose.  Their time over that of equal tiles
// for copy, sum and general sum of 2^24 elements, n0 x batches x nq reversed:
//   both modes up to 32: an equal tile is then no larger than theirs, and twice as
//     many of theirs share an SM.  2 x 2 0.66, 0.53, 0.53; 16 x 16 0.61, 0.61, 0.61;
//     32 x 32 0.64, 0.68, 0.55; only 32 x 2 1.12 for the general sum.
//   one of 17 to 32: half of the wide lanes' loads are idle on that side.  20 x 64
//     0.77, 0.85, 0.76; on the side of the writes 64 x 20 0.91, 0.75, 0.58 but, for
//     copies, 128 x 20 1.04.
//   one of 9 to 16: where the writes or the scalars count, 12 x 80 1.02, 0.90, 0.81;
//     16 x 48 1.01, 0.95, 0.85; 16 x 160 1.08, 0.99, 0.85; 64 x 12 1.10, 1.03, 0.95;
//     128 x 12 1.38, 1.14, 1.06 (0.85 of 2^20 elements).
//   longer ones: by the share of working lanes against theirs, below 0.745 (160 x 160,
//     0.71: 0.85, 0.92; 129 x 129, 0.69: 0.94, 0.93; 65 x 33, 0.75: 1.47, 1.31) or,
//     where theirs are full, 0.8 (128 x 96, 0.75: 0.91, 0.94; but 64 x 160, 0.84: 0.94,
//     and 1.13 of 2^22 elements), with general scalars below 1.3 (64 x 64, 1: 0.94; 100 x 100, 1: 0.98; above
//     it a mode is short: 128 x 8 1.70).
bool perm_tiles32(int op, int64_t n0, int64_t nq, int e0, int eq, int l0, int lq) {
  const bool general = op == PERM_SCALE || op == PERM_AXPBY;
  if (n0 <= 32 && nq <= 32) return op != PERM_AXPBY || n0 < 32 || nq > 8;
  if (n0 > 16 && n0 <= 32) return true;
  if (nq > (op == PERM_COPY ? 24 : 16) && nq <= 32) return true;
  if (n0 > 8 && n0 <= 16 && (op == PERM_AXPBY || (nq <= 96 && (general || (op == PERM_ADD && nq > 64))))) return true;
  if (general && nq > 8 && nq <= 16) return true;
  auto share = [](int64_t n, int e, int l) {
    const int lanes = (e + (1 << l) - 1) >> l << l;
    return (double)n / ((double)((n + e - 1) / e) * lanes);
  };
  const double theirs = share(n0, 32, 5) * share(nq, 32, 5), r = share(n0, e0, l0) * share(nq, eq, lq) / theirs;
  return r < (general ? 1.3 : (theirs > 0.95 ? 0.8 : 0.745));
}

// Whether 32 x 32 tiles take a transpose that is too small to fill the GPU.  As long
// as the equal tiles fit on it at once (four to an SM) their number does not count,
// but the rounds of loads of one of them, about 0.3 us each for a copy and 0.4 to 0.5
// with Bin, beside 1.9 us; the 32 x 32 ones take one round each, and eight share an SM
// (2^16 elements, 16 x 16 x 256, eight rounds: copy 4.7 -> 2.1 us, sum 6.5 -> 2.5;
// 1000 x 2: 7.0 -> 1.8; but 2^18, 256 x 512 x 2, six rounds: 4.4 against 10.7 us).
bool perm_few_tiles(int sms, int op, int64_t n0, int64_t nq, int64_t nbatch, int e0, int eq, int l0, int lq) {
  auto up = [](int64_t n, int64_t d) { return (n + d - 1) / d; };
  const int64_t equal = up(n0, e0) * up(nq, eq) * nbatch, by32 = up(n0, 32) * up(nq, 32) * nbatch;
  const int64_t rounds = up(e0, 2 << l0) * up(eq, 4 * (PERM_THREADS >> l0)) + up(eq, 2 << lq) * up(e0, 4 * (PERM_THREADS >> lq));
  return equal <= 4 * (int64_t)sms && (double)by32 <= sms * (0.6 + (op == PERM_COPY ? 1.0 : 1.3) * rounds);
}

// Resolve modesB as a permutation of modesA.  perm[j] = A-position of B's mode j.
int make_perm(itg_handle* h, int rank, const int32_t* modesA, const int32_t* modesB, int* perm) {
  for (int j = 0; j < rank; ++j) {
    perm[j] = -1;
    for (int i = 0; i < rank; ++i)
      if (modesA[i] == modesB[j]) {
        if (perm[j] >= 0) return itg_fail(h, ITG_ERR_SHAPE, "repeated mode %d", modesB[j]);
        perm[j] = i;
      }
    if (perm[j] < 0) return itg_fail(h, ITG_ERR_SHAPE, "mode %d of B not found in A", modesB[j]);
  }
  for (int i = 0; i < rank; ++i)
    for (int j = i + 1; j < rank; ++j)
      if (modesA[i] == modesA[j]) return itg_fail(h, ITG_ERR_SHAPE, "repeated mode %d in A", modesA[i]);
  return ITG_OK;
}

}  // namespace

// Shared host routine: Bin may be null (pure permute) or alias B.
static int permute_axpby(itg_handle* h, double alpha, const double* A, int rank,
                         const int64_t* dimsA, const int32_t* modesA, double beta,
                         const double* Bin, const int32_t* modesB, double* B) {
  if (rank < 0 || rank > ITG_MAX_RANK)
    return itg_fail(h, ITG_ERR_UNSUPPORTED, "rank %d outside 0..%d", rank, ITG_MAX_RANK);
  int perm[ITG_MAX_RANK];
  ITG_TRY(make_perm(h, rank, modesA, modesB, perm));
  int64_t total = 1;
  for (int i = 0; i < rank; ++i) {
    if (dimsA[i] < 0) return itg_fail(h, ITG_ERR_SHAPE, "negative dimension");
    total *= dimsA[i];
  }
  if (total == 0) return ITG_OK;
  // strides of A's modes in A and in B
  int64_t sA[ITG_MAX_RANK], sB[ITG_MAX_RANK];
  {
    int64_t s = 1;
    for (int i = 0; i < rank; ++i) { sA[i] = s; s *= dimsA[i]; }
    s = 1;
    for (int j = 0; j < rank; ++j) { sB[perm[j]] = s; s *= dimsA[perm[j]]; }
  }
  // Fuse: drop unit modes, then merge A-adjacent modes that are B-adjacent.
  PermDesc d;
  d.rank = 0;
  for (int i = 0; i < rank; ++i) {
    if (dimsA[i] == 1) continue;
    if (d.rank > 0) {
      int p = d.rank - 1;
      if (sA[i] == d.strA[p] * d.dims[p] && sB[i] == d.strB[p] * d.dims[p]) {
        d.dims[p] *= dimsA[i];
        continue;
      }
    }
    d.dims[d.rank] = dimsA[i];
    d.strA[d.rank] = sA[i];
    d.strB[d.rank] = sB[i];
    d.rank++;
  }
  const double* bin = (beta == 0.0) ? nullptr : Bin;
  const bool unit = alpha == 1.0 || alpha == -1.0;
  const int op = !bin ? (unit ? PERM_COPY : PERM_SCALE) : (unit && beta == 1.0 ? PERM_ADD : PERM_AXPBY);
  const PermScalars sc{alpha, beta, alpha < 0.0 ? (long long)(1ull << 63) : 0ll};
  if (d.rank == 0) {  // single element
    d.rank = 1;
    d.dims[0] = 1;
    d.strA[0] = 1;
    d.strB[0] = 1;
  }
  // find the fused mode that is fastest in B (strB == 1)
  int q = 0;
  for (int i = 0; i < d.rank; ++i)
    if (d.strB[i] == 1) q = i;
  RestDesc rest;
  if (q == 0) {
    rest.n = 0;
    for (int i = 1; i < d.rank; ++i) {
      rest.dims[rest.n] = d.dims[i];
      rest.strA[rest.n] = d.strA[i];
      rest.strB[rest.n] = d.strB[i];
      rest.n++;
    }
    const int64_t d0 = d.dims[0], nrows = total / d0;
    // short rows share an item, long ones are cut into segments; smaller items
    // where those of PERM_ITEM would leave SMs idle (24 x 96 x 3, a copy 3.7 -> 2.1 us)
    const int64_t share = (total + 4 * h->num_sms - 1) / (4 * h->num_sms);
    const int64_t seg = std::min<int64_t>(PERM_ITEM, (share + PERM_THREADS - 1) / PERM_THREADS * PERM_THREADS);
    const int64_t nseg = d0 > 2 * seg ? (d0 + seg - 1) / seg : 1;
    int64_t rows = nseg > 1 ? 1 : std::min<int64_t>(std::max<int64_t>(1, seg / d0), PERM_ROWS);
    const int64_t items = nseg > 1 ? nrows * nseg : (nrows + rows - 1) / rows;
    const int blocks = (int)std::min<int64_t>(items, (int64_t)h->num_sms * 64);
    auto run = [&](auto tag) {
      perm_launch_rows<decltype(tag)::value>(blocks, h->stream, A, B, bin, sc, d0, nrows, (int)rows, seg, nseg, items,
                                             rest);
    };
    if (op == PERM_COPY) run(std::integral_constant<int, PERM_COPY>());
    else if (op == PERM_SCALE) run(std::integral_constant<int, PERM_SCALE>());
    else if (op == PERM_ADD) run(std::integral_constant<int, PERM_ADD>());
    else run(std::integral_constant<int, PERM_AXPBY>());
  } else {
    rest.n = 0;
    for (int i = 1; i < d.rank; ++i) {
      if (i == q) continue;
      rest.dims[rest.n] = d.dims[i];
      rest.strA[rest.n] = d.strA[i];
      rest.strB[rest.n] = d.strB[i];
      rest.n++;
    }
    // batches next to each other in B first: a tile row of A is 512 bytes of its
    // own whatever the order, while B's rows then continue one another
    // (129 x 250 x 64 x 63 reversed 412 -> 365 us, no order slower)
    for (int i = 1; i < rest.n; ++i)
      for (int j = i; j > 0 && rest.strB[j] < rest.strB[j - 1]; --j) {
        std::swap(rest.dims[j], rest.dims[j - 1]);
        std::swap(rest.strA[j], rest.strA[j - 1]);
        std::swap(rest.strB[j], rest.strB[j - 1]);
      }
    int64_t n0 = d.dims[0], nq = d.dims[q];
    int64_t nbatch = total / (n0 * nq);
    int e0, eq, l0, lq;
    perm_tile(n0, nq, e0, eq, l0, lq);
    const int64_t sqA = d.strA[q], s0B = d.strB[0];
    const bool small = perm_few_tiles(h->num_sms, op, n0, nq, nbatch, e0, eq, l0, lq) ||
                       perm_tiles32(op, n0, nq, e0, eq, l0, lq);
    const int64_t t0 = (n0 + (small ? 32 : e0) - 1) / (small ? 32 : e0);
    const int64_t tq = (nq + (small ? 32 : eq) - 1) / (small ? 32 : eq);
    if (t0 * tq > (int64_t)INT32_MAX) return itg_fail(h, ITG_ERR_UNSUPPORTED, "permute: transpose too large");
    auto run = [&](auto tag) {
      constexpr int OP = decltype(tag)::value;
      if (small) {
        const int64_t want = (int64_t)h->num_sms * 32, gx = std::min<int64_t>(t0 * tq, want);
        const int64_t gy = std::min<int64_t>(std::min<int64_t>(nbatch, std::max<int64_t>(1, want / gx)), 65535);
        k_perm_transpose32<OP><<<dim3((unsigned)gx, (unsigned)gy), dim3(32, 8), 0, h->stream>>>(A, B, bin, sc, n0, nq, sqA,
                                                                                               s0B, nbatch, rest);
      } else {
        const int64_t items = t0 * tq * nbatch;
        const int blocks = (int)std::min<int64_t>(items, (int64_t)h->num_sms * 48);
        k_perm_transpose<OP><<<blocks, PERM_THREADS, sizeof(double) * (size_t)eq * (e0 | 1), h->stream>>>(
            A, B, bin, sc, n0, nq, sqA, s0B, e0, eq, l0, lq, t0, tq, items, rest);
      }
    };
    if (op == PERM_COPY) run(std::integral_constant<int, PERM_COPY>());
    else if (op == PERM_SCALE) run(std::integral_constant<int, PERM_SCALE>());
    else if (op == PERM_ADD) run(std::integral_constant<int, PERM_ADD>());
    else run(std::integral_constant<int, PERM_AXPBY>());
  }
  ITG_CHECK_LAUNCH(h);
  return ITG_OK;
}

namespace {
// Complex tensors (ITG_C64, interleaved re/im) are permuted as real tensors
// with one leading mode of length 2 that stays first.
struct C64View {
  int rank;
  int64_t dims[ITG_MAX_RANK];
  int32_t ma[ITG_MAX_RANK], mb[ITG_MAX_RANK];
};

int c64_view(itg_handle* h, int rank, const int64_t* dimsA, const int32_t* modesA, const int32_t* modesB,
             C64View& v) {
  if (rank + 1 > ITG_MAX_RANK) return itg_fail(h, ITG_ERR_UNSUPPORTED, "complex rank above %d", ITG_MAX_RANK - 1);
  int32_t c = 0;
  for (int i = 0; i < rank; ++i) c = modesA[i] > c ? modesA[i] : c;
  ++c;
  v.rank = rank + 1;
  v.dims[0] = 2;
  v.ma[0] = v.mb[0] = c;
  for (int i = 0; i < rank; ++i) {
    v.dims[i + 1] = dimsA[i];
    v.ma[i + 1] = modesA[i];
    v.mb[i + 1] = modesB[i];
  }
  return ITG_OK;
}
}  // namespace

extern "C" int itg_permute(itg_handle* h, int dtype, double alpha, const void* A, int rank,
                           const int64_t* dimsA, const int32_t* modesA, void* B,
                           const int32_t* modesB) {
  if (!h) return ITG_ERR_INVALID;
  if (dtype != ITG_F64 && dtype != ITG_C64) return itg_fail(h, ITG_ERR_UNSUPPORTED, "dtype %d", dtype);
  if (rank > 0 && (!dimsA || !modesA || !modesB)) return itg_fail(h, ITG_ERR_INVALID, "null array");
  if (!A || !B) return itg_fail(h, ITG_ERR_INVALID, "null tensor");
  if (dtype == ITG_C64) {
    C64View v;
    ITG_TRY(c64_view(h, rank, dimsA, modesA, modesB, v));
    return permute_axpby(h, alpha, (const double*)A, v.rank, v.dims, v.ma, 0.0, nullptr, v.mb, (double*)B);
  }
  return permute_axpby(h, alpha, (const double*)A, rank, dimsA, modesA, 0.0, nullptr, modesB,
                       (double*)B);
}

extern "C" int itg_axpby_permuted(itg_handle* h, int dtype, double alpha, const void* A, int rank,
                                  const int64_t* dimsA, const int32_t* modesA, double beta,
                                  const void* B, const int32_t* modesB, void* C) {
  if (!h) return ITG_ERR_INVALID;
  if (dtype != ITG_F64 && dtype != ITG_C64) return itg_fail(h, ITG_ERR_UNSUPPORTED, "dtype %d", dtype);
  if (rank > 0 && (!dimsA || !modesA || !modesB)) return itg_fail(h, ITG_ERR_INVALID, "null array");
  if (!A || !C || (beta != 0.0 && !B)) return itg_fail(h, ITG_ERR_INVALID, "null tensor");
  if (A == C) return itg_fail(h, ITG_ERR_INVALID, "C must not alias A");
  if (dtype == ITG_C64) {
    C64View v;
    ITG_TRY(c64_view(h, rank, dimsA, modesA, modesB, v));
    return permute_axpby(h, alpha, (const double*)A, v.rank, v.dims, v.ma, beta, (const double*)B, v.mb,
                         (double*)C);
  }
  return permute_axpby(h, alpha, (const double*)A, rank, dimsA, modesA, beta, (const double*)B,
                       modesB, (double*)C);
}

namespace itg {
int transpose(itg_handle* h, int64_t m, int64_t n, const double* in, int64_t lda, double* out) {
  if (lda != m) return itg_fail(h, ITG_ERR_UNSUPPORTED, "transpose needs lda == m");
  int64_t dims[2] = {m, n};
  int32_t ma[2] = {0, 1}, mb[2] = {1, 0};
  return permute_axpby(h, 1.0, in, 2, dims, ma, 0.0, nullptr, mb, out);
}
}  // namespace itg

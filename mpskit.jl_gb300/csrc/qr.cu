// Positive QR of a tall matrix by Cholesky factors of Gram matrices.
//
// A = Q R with R upper triangular and diag(R) > 0 is unique, so it need not come from
// Householder reflections, whose column-by-column panels keep one SM busy: G = A' A = R1' R1,
// Q1 = A R1^-1, and -- since rounding leaves Q1' Q1 = 1 + E with E ~ eps cond(A)^2 -- a second
// step that makes Q1 orthonormal to rounding (CholeskyQR2: Yamamoto, Nakatsukasa, Yanagisawa &
// Fukaya, ETNA 44 (2015) 306-326).  With |E| small the Cholesky factor of 1 + E is 1 + u to
// first order, u the upper triangle of E with half its diagonal, and its inverse 1 - u: the
// second step is a product and no factorisation; it is repeated while E^2 is not yet rounding.
// R is then the upper triangle of Q' A.  (The product of the passes' factors (1 + u) R1 is not:
// (1 - u)(1 + u) = 1 - u^2, and the u^2 of the first pass, up to 1e-2, stays in Q R for good --
// a residual of 2e-10 |A| at a condition number of 1e8, 2e-16 here.)  A matrix whose Gram matrix
// has no Cholesky factor, or whose E exceeds 0.1, is left to the caller's Householder routine.
//
// The columns are first brought to one scale, by powers of two and therefore exactly.  Site
// tensors have columns graded by Schmidt values, and the digits of the products hold a row of A
// to 2^-55 of its largest entry: unscaled, a column 1e-8 of the largest is kept to 1e-9 of its
// own norm (Householder and scaled columns: 1e-15), and E sees the grading as a condition.
//
// The products run as the plain-precision GEMMs (gemm_f64.cu).  gram_chol_kernel does the rest
// in one cooperative launch: the Cholesky factor of G and its inverse, by eliminating [G | 1]
// in block rows of 8.  Its chain is the 8 x 8 diagonal blocks (a scheduler issues an FP64 warp
// instruction in 64 clocks: eleven of them a column), hidden behind the other SMs' update of the
// remaining rows once these are long, and two grid barriers per block.
//
// Measured (QR and LQ of a 256 x 2 x 256 complex tensor): 11.9 ms with the library's Householder
// routines, 1.14 ms here; one complex 512 x 256 factorisation 5.9 ms before, 0.52 ms here (0.31 ms
// of it the factor; R from Q' A and the scaled copy of A are 10 us each).  Blocks of 16 took 0.84 ms (the chain through a diagonal block grows with its
// square, the grid barriers saved are 3 k clocks each), updates of one column at a time 0.59.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "gb_common.h"
#include "recip.cuh"
#include "tc_ptx.cuh"

namespace gb {

namespace {

constexpr int NB = 8;     // rows of a block
constexpr int NC = 32 / NB;  // columns of a warp beside each other
constexpr int QT = 256;   // threads per block: two warps per scheduler
constexpr int QW = QT / 32;

template <bool CX>
struct Sc;
template <>
struct Sc<false> {
  using T = double;
};
template <>
struct Sc<true> {
  using T = double2;
};
__device__ __forceinline__ double real_of(double a) { return a; }
__device__ __forceinline__ double real_of(double2 a) { return a.x; }
__device__ __forceinline__ double from_real(double, double r) { return r; }
__device__ __forceinline__ double2 from_real(double2, double r) { return make_double2(r, 0.0); }
__device__ __forceinline__ double times(double a, double s) { return a * s; }
__device__ __forceinline__ double2 times(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
// c - conj(a) b,  c + a b
__device__ __forceinline__ void sub_cmul(double& c, double a, double b) { c = fma(-a, b, c); }
__device__ __forceinline__ void sub_cmul(double2& c, double2 a, double2 b) {
  c.x = fma(-a.x, b.x, fma(-a.y, b.y, c.x));
  c.y = fma(-a.x, b.y, fma(a.y, b.x, c.y));
}
__device__ __forceinline__ void add_mul(double& c, double a, double b) { c = fma(a, b, c); }
__device__ __forceinline__ void add_mul(double2& c, double2 a, double2 b) {
  c.x = fma(a.x, b.x, fma(-a.y, b.y, c.x));
  c.y = fma(a.x, b.y, fma(a.y, b.x, c.y));
}

struct CholArgs {
  int n;
  void* A;      // n x 2n column-major: [G | 1] on entry (G: upper triangle), R^-H in the right
                // half on exit
  void* Z;      // NB x NB: inverse of the current diagonal block's (lower) factor
  int* fail;    // set when a pivot is not positive, or when a wait ran out
  const int* skip;  // nonzero: a column is zero or not finite, there is nothing to factor
  unsigned int* bar;
  int* status;
  unsigned long long wait_ns;
};

// added to the arrivals by the first block when a pivot is not positive: every block stops at its
// next barrier
constexpr unsigned int CHOL_STOP = 1u << 30;

__device__ bool chol_barrier(const CholArgs& g, unsigned int target) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&g.bar[0], 1u);
    ok = 1;
    const unsigned long long t0 = globaltimer();
    unsigned int arrived;
    while ((arrived = *(volatile unsigned int*)&g.bar[0]) < target) {
      if (globaltimer() - t0 > g.wait_ns) {
        atomicExch(g.status, GB_ERR_TIMEOUT);
        ok = 0;
        break;
      }
    }
    if (arrived >= CHOL_STOP) ok = 0;
    __threadfence();
  }
  __syncthreads();
  return ok != 0;
}

// Factor of the block at rows/columns k0..k0+nb-1: the first four warps eliminate
// [block | 1], a warp holding four of the 16 columns, a lane one entry.  The rows stay unscaled
// (a reciprocal per pivot); their factors 1 / sqrt(pivot) come in at the end.
template <typename T>
__device__ void diag_block(const CholArgs& g, int k0, int nb, T (*row)[2 * NB + 1]) {
  T* A = (T*)g.A;
  const int64_t ld = g.n;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int i = lane % NB, j = NC * warp + lane / NB;
  const T none = T{};
  T a = none;
  if (warp < 2 * NB / NC) {
    if (j < NB) {
      if (i < nb && j < nb && i <= j) a = A[k0 + i + ld * (k0 + j)];
      if (i >= nb && i == j) a = from_real(none, 1.0);  // pad: identity
    } else if (j - NB == i) {
      a = from_real(none, 1.0);
    }
    if (i == 0) row[0][j] = a;
  }
  bool bad = false;
  double mine = 1.0;  // pivot of this lane's row
  for (int k = 0; k < NB; ++k) {
    __syncthreads();
    if (warp < 2 * NB / NC) {
      const double d = real_of(row[k][k]);
      bad |= !(d > 0.0);
      if (i == k) mine = d;
      if (k + 1 < NB) {
        const double q = inverse(d);
        if (i > k) sub_cmul(a, times(row[k][i], q), row[k][j]);
        if (i == k + 1) row[k + 1][j] = a;
      }
    }
  }
  if (warp < 2 * NB / NC) {
    const double r = inv_sqrt(mine);
    T* Z = (T*)g.Z;
    const bool left = j < NB;
    const int jj = left ? j : j - NB;
    a = times(a, r);
    if (left && i == jj) a = from_real(none, real_of(a));
    if (left ? i > jj : jj > i) a = none;
    if (!left) Z[i + NB * jj] = a;
    if (i < nb && jj < nb && (!left || i <= jj))
      A[k0 + i + ld * ((left ? k0 : g.n + k0) + jj)] = a;
    if (bad && threadIdx.x == 0) {
      atomicExch(g.fail, 1);
      atomicAdd(&g.bar[0], CHOL_STOP);
    }
  }
  __syncthreads();
}

// A(r, c) -= sum_k conj(P(k, r)) P(k, c) over the block row k0..k0+nb-1, for the 32 rows from r0 and
// columns q0..q1-1 of the list cl..n-1 (left part, only the upper triangle), n.. (right part).  Two
// columns at a time, all their loads ahead of the arithmetic.
template <typename T>
__device__ __forceinline__ void update_columns(const CholArgs& g, int k0, int nb, int r0, int rend,
                                               int cl, int q0, int q1, int lane) {
  T* A = (T*)g.A;
  const int64_t ld = g.n;
  const int r = r0 + lane, nl = g.n - cl;
  T p[NB];
#pragma unroll
  for (int k = 0; k < NB; ++k) p[k] = (r < rend && k < nb) ? A[k0 + k + ld * r] : T{};
  for (int qq = q0; qq < q1; qq += 2) {
    T v[2], w[2][NB];
    T* at[2];
    bool live[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int q = min(qq + u, q1 - 1), c = q < nl ? cl + q : g.n + (q - nl);
      at[u] = A + ld * c;
      live[u] = qq + u < q1 && r < rend && (c >= g.n || r <= c);
      v[u] = live[u] ? at[u][r] : T{};
#pragma unroll
      for (int k = 0; k < NB; ++k) w[u][k] = at[u][k0 + min(k, nb - 1)];
    }
    // p is zero from nb on
#pragma unroll
    for (int u = 0; u < 2; ++u) {
#pragma unroll
      for (int k = 0; k < NB; ++k) sub_cmul(v[u], p[k], w[u][k]);
      if (live[u]) at[u][r] = v[u];
    }
  }
}

template <bool CX>
__global__ void __launch_bounds__(QT, 1) gram_chol_kernel(CholArgs g) {
  using T = typename Sc<CX>::T;
  __shared__ T row[NB + 1][2 * NB + 1];
  T* A = (T*)g.A;
  T* Z = (T*)g.Z;
  const int64_t ld = g.n;
  const int n = g.n, steps = (n + NB - 1) / NB;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int gw = blockIdx.x + warp * gridDim.x, nw = gridDim.x * QW;  // one warp per SM first
  unsigned int target = 0;
  bool ok = *(volatile const int*)g.skip == 0;
  if (ok && blockIdx.x == 0) diag_block<T>(g, 0, min(NB, n), row);
  for (int j = 0; j < steps && ok; ++j) {
    const int k0 = j * NB, nb = min(NB, n - k0), k1 = k0 + nb;
    target += gridDim.x;
    ok = chol_barrier(g, target);
    if (!ok) break;
    // the block row: Z times columns k1..n-1 of G and 0..k0-1 of the right part
    {
      const int i = lane % NB, h = lane / NB;
      const int left = n - k1, cols = left + k0;
      T z[NB];
      bool have = false;
      for (int p = gw; NC * p < cols; p += nw) {
        if (!have) {
#pragma unroll
          for (int k = 0; k < NB; ++k) z[k] = __ldcg(Z + i + NB * k);
          have = true;
        }
        const int q = NC * p + h;
        const int c = q < left ? k1 + q : n + (q - left);
        T v = (q < cols && i < nb) ? A[k0 + i + ld * c] : T{};
        T s = T{};
#pragma unroll
        for (int k = 0; k < NB; ++k) {
          T b;
          if constexpr (CX) {
            b.x = __shfl_sync(0xffffffffu, v.x, k + NB * h);
            b.y = __shfl_sync(0xffffffffu, v.y, k + NB * h);
          } else {
            b = __shfl_sync(0xffffffffu, v, k + NB * h);
          }
          add_mul(s, z[k], b);
        }
        if (q < cols && i < nb) A[k0 + i + ld * c] = s;
      }
    }
    if (k1 >= n) break;
    target += gridDim.x;
    ok = chol_barrier(g, target);
    if (!ok) break;
    // the rows below; the first block updates and factors the next diagonal block meanwhile
    const int nb2 = min(NB, n - k1);
    if (blockIdx.x == 0) {
      if (warp < NB / NC) {
        const int i = lane % NB, c = NC * warp + lane / NB;
        if (i <= c && c < nb2) {
          const T* p = A + k0 + ld * (k1 + i);
          const T* q = A + k0 + ld * (k1 + c);
          T v = A[k1 + i + ld * (k1 + c)];
#pragma unroll
          for (int k = 0; k < NB; ++k) sub_cmul(v, p[k], q[k]);  // every block but the last is full
          A[k1 + i + ld * (k1 + c)] = v;
        }
      }
      __syncthreads();
      diag_block<T>(g, k1, nb2, row);
    } else if (gridDim.x > 1) {
      const int w = (int)(blockIdx.x - 1) + warp * (int)(gridDim.x - 1);
      const int ws = (int)(gridDim.x - 1) * QW;
      // items: a group of rows and a run of four of its columns, of two while that leaves warps
      // idle; the first group is the next block row (its own diagonal block apart), the others 32
      // rows each
      const int groups = 1 + (n - k1 - nb2 + 31) / 32;
      const int run = groups * ((n + 3) / 4) > ws ? 4 : 2;
      int done = 0;
      for (int gr = 0; gr < groups; ++gr) {
        const int r0 = gr ? k1 + nb2 + 32 * (gr - 1) : k1;
        const int rend = gr ? min(n, r0 + 32) : k1 + nb2;
        const int cl = gr ? r0 : k1 + nb2;         // first left column
        const int cols = (n - cl) + k1;            // left columns, then right columns 0..k1-1
        const int items = (cols + run - 1) / run;
        for (int it = ((w - done) % ws + ws) % ws; it < items; it += ws)
          update_columns<T>(g, k0, nb, r0, rend, cl, run * it, min(cols, run * it + run), lane);
        done = (done + items) % ws;
      }
    }
  }
  if (!ok && threadIdx.x == 0) atomicExch(g.fail, 1);
  // the last block to leave makes the counters ready for the next launch
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(&g.bar[1], 1u) == gridDim.x - 1) {
    g.bar[0] = 0;
    __threadfence();
    g.bar[1] = 0;
  }
}

// the right half of the elimination's matrix: 1
template <bool CX>
__global__ void unit_kernel(int n, typename Sc<CX>::T* X) {
  using T = typename Sc<CX>::T;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < (int64_t)n * n;
       e += (int64_t)gridDim.x * blockDim.x)
    X[e] = e % n == e / n ? from_real(T{}, 1.0) : T{};
}

// As = A with column j scaled by 2^(1023 - ex[j]), ex[j] the largest biased exponent of its parts
// (columns of zeros or with Inf or NaN: 2^0, and *skip is set).  A block per column.  Bound by its latency (2 MB of
// a 512 x 256 complex matrix).
template <bool CX>
__global__ void __launch_bounds__(QT)
    equilibrate_kernel(int64_t m, int64_t n, const double* A, double* As, int* ex, int* skip) {
  chain_release();
  chain_wait();
  __shared__ int most;
  const int64_t len = CX ? 2 * m : m;  // reals of a column
  for (int64_t j = blockIdx.x; j < n; j += gridDim.x) {
    const double* a = A + j * len;
    if (threadIdx.x == 0) most = 0;
    __syncthreads();
    int e = 0;
    for (int64_t i = threadIdx.x; i < len; i += QT)
      e = max(e, (__double2hiint(a[i]) >> 20) & 0x7ff);
    e = __reduce_max_sync(0xffffffffu, e);
    if (threadIdx.x % 32 == 0) atomicMax(&most, e);
    __syncthreads();
    e = most == 0 || most == 0x7ff ? 1023 : min(most, 2045);
    const double s = __hiloint2double((2046 - e) << 20, 0);
    for (int64_t i = threadIdx.x; i < len; i += QT) As[j * len + i] = a[i] * s;
    if (threadIdx.x == 0) {
      ex[j] = e;
      if (most == 0 || most == 0x7ff) atomicExch(skip, 1);
    }
    __syncthreads();
  }
}

// R = upper triangle of P, the columns scaled back, the diagonal real
template <bool CX>
__global__ void upper_kernel(int n, const typename Sc<CX>::T* P, const int* ex,
                             typename Sc<CX>::T* R) {
  using T = typename Sc<CX>::T;
  chain_release();
  chain_wait();
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < (int64_t)n * n;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(e % n), c = (int)(e / n);
    T v = T{};
    if (r <= c) v = times(P[e], __hiloint2double(ex[c] << 20, 0));
    R[e] = r == c ? from_real(T{}, real_of(v)) : v;
  }
}

// E = G - 1 (G Hermitian): um = 1 - u with u the upper triangle of E and half its diagonal;
// *worst = bits of max |E|
template <bool CX>
__global__ void correction_kernel(int n, const typename Sc<CX>::T* __restrict__ G,
                                  typename Sc<CX>::T* __restrict__ um,
                                  unsigned long long* worst) {
  using T = typename Sc<CX>::T;
  unsigned long long m = 0;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < (int64_t)n * n;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(e % n), c = (int)(e / n);
    T a = T{};
    if (r == c) {
      const double d = real_of(G[e]) - 1.0;
      m = max(m, (unsigned long long)__double_as_longlong(d) & ~(1ull << 63));
      a = from_real(T{}, fma(-0.5, d, 1.0));
    } else if (r < c) {
      const T b = G[e];
      if constexpr (CX) {
        m = max(m, (unsigned long long)__double_as_longlong(b.x) & ~(1ull << 63));
        m = max(m, (unsigned long long)__double_as_longlong(b.y) & ~(1ull << 63));
        a = make_double2(-b.x, -b.y);
      } else {
        m = max(m, (unsigned long long)__double_as_longlong(b) & ~(1ull << 63));
        a = -b;
      }
    }
    um[e] = a;
  }
  for (int o = 16; o > 0; o >>= 1)
    m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (threadIdx.x % 32 == 0) atomicMax(worst, m);
}

struct WorkBuf {
  gb_ctx* ctx;
  char* p = nullptr;
  WorkBuf(gb_ctx* c, size_t bytes) : ctx(c) {
    void* q = nullptr;
    if (cudaMallocAsync(&q, bytes, c->stream) != cudaSuccess) {
      cudaGetLastError();
      q = nullptr;
    }
    p = (char*)q;
  }
  ~WorkBuf() {
    if (p) cudaFreeAsync(p, ctx->stream);
  }
  WorkBuf(const WorkBuf&) = delete;
  WorkBuf& operator=(const WorkBuf&) = delete;
};

size_t up256(size_t b) { return (b + 255) & ~(size_t)255; }

}  // namespace

bool qr_gram(gb_ctx* ctx, int dtype, int64_t m, int64_t n, const void* M, void* Q, void* R) {
  if (n < 1 || m < n || n > QR_GRAM_MAX) return false;
  const bool cx = is_cplx(dtype);
  // products that neither small tiles nor digits take (more than 262144 rows, half of that complex,
  // or FMAs on request) are slower than the panels: complex 200000 x 4 153 ms against 5.9
  if ((double)m * (double)n * (double)n * (cx ? 4 : 1) >= F64_SMALL_MAX_MAC &&
      !gemm_sliced_wanted(ctx, dtype, n, n, m, 1))
    return false;
  const size_t es = elem_size(dtype);
  const size_t nn = up256((size_t)n * n * es), mn = up256((size_t)m * n * es);
  WorkBuf w(ctx, 256 + up256(n * sizeof(int)) + up256(NB * NB * es) +
                     up256(2 * (size_t)n * n * es) + nn + 3 * mn);
  if (!w.p) return false;
  // [0] max |E|, [1] failed pivots (int), [2] columns without a scale (int)
  unsigned long long* res = (unsigned long long*)w.p;
  int* ex = (int*)(w.p + 256);
  char* Z = w.p + 256 + up256(n * sizeof(int));
  char* A = Z + up256(NB * NB * es);
  char* um = A + up256(2 * (size_t)n * n * es);
  char* As = um + nn;
  char* Q1 = As + mn;
  char* Q2 = Q1 + mn;
  const cplx one{1, 0}, none{0, 0};
  const int sms = std::max(1, ctx->num_sms);
  GB_CHECK_CUDA(cudaMemsetAsync(res, 0, 256, ctx->stream));
  const unsigned eb = (unsigned)std::min<int64_t>((n * n + 255) / 256, 4 * sms);
  launch_chained(cx ? equilibrate_kernel<true> : equilibrate_kernel<false>,
                 dim3((unsigned)std::min<int64_t>(n, 8 * sms)), QT, 0, ctx->stream, 1, 1, m, n,
                 (const double*)M, (double*)As, ex, (int*)(res + 2));
  gemm_fp64(ctx, dtype, 'C', 'N', n, n, m, one, As, m, 0, As, m, 0, none, A, n, 0, 1);
  char* X = A + (size_t)n * n * es;
  if (cx) unit_kernel<true><<<eb, 256, 0, ctx->stream>>>((int)n, (double2*)X);
  else unit_kernel<false><<<eb, 256, 0, ctx->stream>>>((int)n, (double*)X);
  GB_CHECK_CUDA(cudaGetLastError());
  CholArgs a{};
  a.n = (int)n;
  a.A = A;
  a.Z = Z;
  a.fail = (int*)(res + 1);
  a.skip = (int*)(res + 2);
  a.bar = (unsigned int*)((char*)ctx->d_status + 96);
  a.status = ctx->d_status;
  a.wait_ns = ctx->wait_ns;
  // a block per 64 columns and rows of the update, on a lane a share of the chip
  const int most = ctx->lane ? std::max(2, sms / 8) : sms;
  const int64_t half = (n + NB - 1) / NB;
  const int blocks = (int)std::max<int64_t>(2, std::min<int64_t>(most, half * half / 8 + 1));
  void* args[] = {&a};
  GB_CHECK_CUDA(cudaLaunchCooperativeKernel(
      cx ? (const void*)gram_chol_kernel<true> : (const void*)gram_chol_kernel<false>, dim3(blocks),
      dim3(QT), args, 0, ctx->stream));
  // Q1 = A R1^-1 (the right half holds R1^-H)
  gemm_fp64(ctx, dtype, 'N', 'C', m, n, n, one, As, m, 0, X, n, 0, none, Q1, m, 0, 1);
  count_launch_n(ctx, 3);
  // orthonormal to first order, until the second order is rounding: |E^2| <= (n max |E|)^2, which
  // is to stay below n eps / 4
  const double done = std::sqrt(0x1p-54 / (double)n);
  char *q = Q1, *qn = Q2;
  for (int pass = 0; pass < 5; ++pass) {
    gemm_fp64(ctx, dtype, 'C', 'N', n, n, m, one, q, m, 0, q, m, 0, none, A, n, 0, 1);
    if (cx)
      correction_kernel<true><<<eb, 256, 0, ctx->stream>>>((int)n, (const double2*)A, (double2*)um,
                                                           res);
    else
      correction_kernel<false><<<eb, 256, 0, ctx->stream>>>((int)n, (const double*)A, (double*)um,
                                                            res);
    GB_CHECK_CUDA(cudaGetLastError());
    // the outputs directly, in the hope that this pass is the last
    gemm_fp64(ctx, dtype, 'N', 'N', m, n, n, one, q, m, 0, um, n, 0, none, Q, m, 0, 1);
    gemm_fp64(ctx, dtype, 'C', 'N', n, n, m, one, Q, m, 0, As, m, 0, none, A, n, 0, 1);
    if (cx)
      launch_chained(upper_kernel<true>, dim3(eb), 256, 0, ctx->stream, 1, 1, (int)n,
                     (const double2*)A, (const int*)ex, (double2*)R);
    else
      launch_chained(upper_kernel<false>, dim3(eb), 256, 0, ctx->stream, 1, 1, (int)n,
                     (const double*)A, (const int*)ex, (double*)R);
    count_launch_n(ctx, 2);
    double* host = host_results(ctx, 512);
    GB_CHECK_CUDA(cudaMemcpyAsync(host, res, 16, cudaMemcpyDeviceToHost, ctx->stream));
    GB_CHECK_CUDA(cudaStreamSynchronize(ctx->stream));
    int failed = 0;
    std::memcpy(&failed, host + 1, sizeof(int));
    const double worst = host[0];
    if (failed || !(worst < 0.1)) return false;
    if (worst <= done) return true;
    GB_CHECK_CUDA(cudaMemcpyAsync(qn, Q, (size_t)m * n * es, cudaMemcpyDeviceToDevice, ctx->stream));
    GB_CHECK_CUDA(cudaMemsetAsync(res, 0, 8, ctx->stream));
    std::swap(q, qn);
  }
  return false;
}

}  // namespace gb

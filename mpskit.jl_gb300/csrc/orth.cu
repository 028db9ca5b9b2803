// One Krylov step after the matvec, in one launch.
//
// krylov_orth_kernel orthogonalises w against k basis vectors and writes the next one,
// v = w / |w|, entirely on the device; the projections and the norm go straight to pinned host
// memory.  The blocks hold their piece of the vectors between grid-wide barriers (cooperative
// launch), so a step is one launch and at most one host wait instead of 5-10 launches and
// three waits.
//
// Passes of classical Gram-Schmidt against all vectors, each with |w|^2 of its input: a pass
// that leaves at least half of |w|^2 met no cancellation and is the last one ("twice is
// enough", Giraud, Langou, Rozloznik & van den Eshof, Numer. Math. 101 (2005) 87-100, with the
// usual 1/sqrt(2)), and |w|^2 - sum |c|^2 is the norm it leaves.  A Lanczos step first takes
// out what the recurrence predicts -- the last projection on the last vector, the last norm on
// the one before -- which is where the cancellation of its first pass would be: one pass then
// does for nearly every step.
//
// Bound by the FP64 pipe of short vectors' few blocks and of long vectors alike: a scheduler
// issues one FP64 warp instruction in 64 clocks, however many lanes take part, so the kernel
// counts them (lists of sums reduced together, scalars by one warp while the others work) and
// spreads them over the four schedulers.  Then by two barriers and the sums between them.
// Measured, all of a Lanczos iteration but its matvec, means over 20 and 30 vectors: 16384
// complex entries 188 us before, 34 us with this kernel (12-16 us) and its host side; 131072
// complex entries 470 / 62 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>

#include "gb_common.h"
#include "tc_ptx.cuh"

namespace gb {

namespace {

constexpr int OT = 512;              // threads per block
constexpr int OW = OT / 32;          // warps
constexpr int OKMAX = 128;           // basis vectors
constexpr int LONG_PIECE = 1024;     // entries of a block's piece
constexpr size_t OPIECE = 192 * 1024;  // bytes of a piece kept in shared memory

struct OrthArgs {
  int64_t n, ld;
  int k;
  int predict;     // a Lanczos step: prev holds the last step's projection and norm
  int in_smem;     // the block's piece of w fits in shared memory
  int cluster;     // the blocks are one cluster: its barrier instead of a grid-wide one
  double* prev;
  const double* V;
  double* w;
  double* vnext;   // null: w is left orthogonalised in place
  double* part;    // [2][OKMAX + 1][blocks] complex partial sums, the sets by turns: a block may
                   // write those of the next pass while another still adds this one's
  double* coef;    // [OKMAX + 1] complex sums
  double* out;     // pinned host: k projections (complex), then the norm
  double* gave_up; // pinned host: set by a block whose wait ran out (null: nobody reads it)
  unsigned int* bar;  // [0] arrivals, [1] blocks that have left
  int* status;
  unsigned long long wait_ns;
};

template <bool CPLX>
struct Num;
template <>
struct Num<false> {
  using T = double;
  static __device__ double zero() { return 0.0; }
};
template <>
struct Num<true> {
  using T = double2;
  static __device__ double2 zero() { return make_double2(0.0, 0.0); }
};
__device__ __forceinline__ void acc_dot(double& r, double&, double v, double w) { r = fma(v, w, r); }
__device__ __forceinline__ void acc_dot(double& r, double& i, double2 v, double2 w) {
  r = fma(v.x, w.x, fma(v.y, w.y, r));
  i = fma(v.x, w.y, fma(-v.y, w.x, i));
}
__device__ __forceinline__ void sub_mul(double& a, double v, double2 c) { a = fma(-v, c.x, a); }
__device__ __forceinline__ void sub_mul(double2& a, double2 v, double2 c) {
  a.x = fma(-v.x, c.x, fma(v.y, c.y, a.x));
  a.y = fma(-v.x, c.y, fma(-v.y, c.x, a.y));
}
__device__ __forceinline__ void sub_mul_real(double& a, double v, double c) { a = fma(-v, c, a); }
__device__ __forceinline__ void sub_mul_real(double2& a, double2 v, double c) {
  a.x = fma(-v.x, c, a.x);
  a.y = fma(-v.y, c, a.y);
}
__device__ __forceinline__ double2 as_double2(double a) { return make_double2(a, 0.0); }
__device__ __forceinline__ double2 as_double2(double2 a) { return a; }
__device__ __forceinline__ void add_to(double& a, double2 b) { a += b.x; }
__device__ __forceinline__ void add_to(double2& a, double2 b) {
  a.x += b.x;
  a.y += b.y;
}
__device__ __forceinline__ double scaled(double a, double s) { return a * s; }
__device__ __forceinline__ double2 scaled(double2 a, double s) { return make_double2(a.x * s, a.y * s); }

// all blocks of the launch; false when the bounded wait gave up
__device__ bool grid_barrier(const OrthArgs& g, unsigned int target) {
  __shared__ int ok;
  if (g.cluster) {
    __threadfence();
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    return true;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&g.bar[0], 1u);
    ok = 1;
    const unsigned long long t0 = globaltimer();
    while (*(volatile unsigned int*)&g.bar[0] < target) {
      if (globaltimer() - t0 > g.wait_ns) {
        atomicExch(g.status, GB_ERR_TIMEOUT);
        ok = 0;
        break;
      }
    }
    __threadfence();
  }
  __syncthreads();
  return ok != 0;
}

// the last block to leave makes the counters ready for the next launch
__device__ void grid_leave(const OrthArgs& g) {
  if (g.cluster) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    if (atomicAdd(&g.bar[1], 1u) == gridDim.x - 1) {
      g.bar[0] = 0;
      __threadfence();
      g.bar[1] = 0;
    }
  }
}

// Sums over the lanes of v[0..N): afterwards lane l holds the sum of v[l / (32 / N)] in v[0].
// Halving the list while exchanging takes N + log2(32 / N) additions instead of 5 N.
template <int N>
__device__ __forceinline__ void lane_sums(double (&v)[N], int lane) {
  int o = 16;
#pragma unroll
  for (int h = N / 2; h >= 1; h /= 2, o /= 2) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const double keep = up ? v[i + h] : v[i], send = up ? v[i] : v[i + h];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  for (; o >= 1; o /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
}

// part[t][block] = this block's share of <V_t, w> for t < cnt, and of <w, w> at t = cnt.  A
// warp takes four vectors (and a share of the block's piece, so that every scheduler has work
// for short lists of vectors).
constexpr int JB = 4;
// four sums per task: as many tasks as lists of four vectors, or two rounds of the warps
constexpr int DOT_SUMS = JB * (OKMAX / JB + 1 > 2 * OW ? OKMAX / JB + 1 : 2 * OW);
// Shares of the piece per four vectors.  Short pieces: eight tasks, two per scheduler (more only
// add reductions).  Long ones: one or two full rounds of the warps, whichever leaves fewer idle --
// with eight tasks half of them waited for the others' loads (3.5 M real entries, 12 vectors:
// 472 us, 281 us with 16 to 32 tasks, the piece of w in shared memory and pairs of entries below;
// pieces of up to 860 entries: the same either way).
__device__ __forceinline__ int dot_shares(int groups, int len) {
  if (len < LONG_PIECE) return groups >= 8 ? 1 : max(1, min(8 / groups, (len + 31) / 32));
  const int a = max(1, OW / groups), b = max(1, 2 * OW / groups);
  // tasks per round: a against b in rounds of OW
  const int ra = (groups * a + OW - 1) / OW, rb = (groups * b + OW - 1) / OW;
  return a * rb >= b * ra ? a : b;
}
template <bool CPLX, typename T>
__device__ void block_dots(const OrthArgs& g, const T* V, const T* w, int64_t c0, int len, int cnt,
                           double2* sred) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int tot = cnt + 1;
  const int groups = (tot + JB - 1) / JB;
  const int P = dot_shares(groups, len);
  for (int t = warp; t < groups * P; t += OW) {
    const int j1 = t / P * JB, p = t % P;
    const int nj = tot - j1;
    const T* v[JB];
#pragma unroll
    for (int j = 0; j < JB; ++j) v[j] = j1 + j < cnt ? V + (int64_t)(j1 + j) * g.ld + c0 : w;
    double acc[CPLX ? 2 * JB : JB];
#pragma unroll
    for (int j = 0; j < (CPLX ? 2 * JB : JB); ++j) acc[j] = 0.0;
    double none = 0.0;
#pragma unroll(CPLX ? 2 : 4)
    for (int i = p * 32 + lane; i < len; i += 32 * P) {
      const T b = w[i];
      T a[JB];
#pragma unroll
      for (int j = 0; j < JB; ++j)
        if (j < nj) a[j] = v[j][i];
#pragma unroll
      for (int j = 0; j < JB; ++j)
        if (j < nj) acc_dot(acc[CPLX ? 2 * j : j], CPLX ? acc[CPLX ? 2 * j + 1 : 0] : none, a[j], b);
    }
    lane_sums(acc, lane);
    if (CPLX) {
      if (lane % 4 == 0) ((double*)sred)[2 * (t * JB) + lane / 4] = acc[0];
    } else if (lane % 8 == 0) {
      sred[t * JB + lane / 8] = make_double2(acc[0], 0.0);
    }
  }
  __syncthreads();
  for (int j = threadIdx.x; j < tot; j += OT) {
    const int t0 = j / JB * P;
    double2 s = sred[t0 * JB + j % JB];
    for (int p = 1; p < P; ++p) {
      const double2 q = sred[(t0 + p) * JB + j % JB];
      s.x += q.x;
      if (CPLX) s.y += q.y;
    }
    ((double2*)g.part)[(int64_t)j * gridDim.x + blockIdx.x] = s;
  }
}

// sum over the blocks of part[t], by one warp, in block order
__device__ __forceinline__ double2 sum_parts(const OrthArgs& g, int t, int lane) {
  double2 s = make_double2(0.0, 0.0);
  for (int b = lane; b < (int)gridDim.x; b += 32) {
    const double2 v = __ldcg((const double2*)g.part + (int64_t)t * gridDim.x + b);
    s.x += v.x;
    s.y += v.y;
  }
  for (int o = 16; o > 0; o >>= 1) {
    s.x += __shfl_down_sync(0xffffffffu, s.x, o);
    s.y += __shfl_down_sync(0xffffffffu, s.y, o);
  }
  return s;
}

// the sums of `tot` partial vectors to sc[0..tot) of every block.  Few: every block adds them
// itself (one barrier); many: one warp of the grid per sum and a second barrier -- adding all
// of them in every block keeps each SM's FP64 pipe busy for longer than the barrier takes
// (32 blocks, 15 sums: 14 k clocks instead of 9 k)
template <bool CPLX>
__device__ bool all_sums(const OrthArgs& g, int tot, double2* sc, unsigned int& target) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (gridDim.x == 1) {
    __syncthreads();
    for (int t = threadIdx.x; t < tot; t += OT) sc[t] = ((const double2*)g.part)[t];
    __syncthreads();
    return true;
  }
  target += gridDim.x;
  if (!grid_barrier(g, target)) return false;
  if (gridDim.x <= 16) {
    // half a warp per sum
    for (int t0 = 2 * warp; t0 < tot; t0 += 2 * OW) {
      const int t = t0 + lane / 16, b = lane % 16;
      double2 s = make_double2(0.0, 0.0);
      if (t < tot && b < (int)gridDim.x)
        s = __ldcg((const double2*)g.part + (int64_t)t * gridDim.x + b);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
        if (CPLX) s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
      }
      if (t < tot && b == 0) sc[t] = s;
    }
    __syncthreads();
    return true;
  }
  if (tot <= 4) {
    if (warp < tot) {
      const double2 s = sum_parts(g, warp, lane);
      if (lane == 0) sc[warp] = s;
    }
    __syncthreads();
    return true;
  }
  for (int t = blockIdx.x + warp * gridDim.x; t < tot; t += gridDim.x * OW) {
    const double2 s = sum_parts(g, t, lane);
    if (lane == 0) ((double2*)g.coef)[t] = s;
  }
  target += gridDim.x;
  if (!grid_barrier(g, target)) return false;
  for (int t = threadIdx.x; t < tot; t += OT) sc[t] = __ldcg((const double2*)g.coef + t);
  __syncthreads();
  return true;
}

template <bool CPLX>
__global__ void __launch_bounds__(OT, 1) krylov_orth_kernel(OrthArgs g) {
  using T = typename Num<CPLX>::T;
  extern __shared__ __align__(16) unsigned char piece[];
  __shared__ double2 sred[DOT_SUMS];
  __shared__ double2 sc[OKMAX + 1], sh[OKMAX + 1];
  __shared__ double2 spart[96];
  __shared__ double sinv, sleft;
  __shared__ int slast;
  const T* V = (const T*)g.V;
  const int64_t per = ((g.n + gridDim.x - 1) / gridDim.x + 31) / 32 * 32;
  const int64_t c0 = min(g.n, per * blockIdx.x);
  const int len = (int)(min(g.n, c0 + per) - c0);
  T* wg = (T*)g.w + c0;
  T* w = g.in_smem ? (T*)piece : wg;
  unsigned int target = 0;
  const int tid = threadIdx.x;
  chain_release();
  chain_wait();
  for (int j = tid; j < g.k; j += OT) sh[j] = make_double2(0.0, 0.0);
  if (g.predict) {
    // what the recurrence predicts: the last projection and the last norm
    const double2 a = make_double2(g.prev[0], 0.0), b = make_double2(g.prev[1], 0.0);
    const T* v1 = V + (int64_t)(g.k - 1) * g.ld + c0;
    const T* v2 = v1 - g.ld;
    for (int i = tid; i < len; i += OT) {
      T x = wg[i];
      sub_mul_real(x, v1[i], a.x);
      sub_mul_real(x, v2[i], b.x);
      w[i] = x;
    }
    __syncthreads();
    if (tid == 0) {
      sh[g.k - 1] = a;
      sh[g.k - 2] = b;
    }
  } else if (g.in_smem) {
    for (int i = tid; i < len; i += OT) w[i] = wg[i];
  }
  __syncthreads();
  bool ok = true;
  double* const parts = g.part;
  for (int pass = 0; pass < 3; ++pass) {
    g.part = parts + (pass & 1) * (2 * (OKMAX + 1) * (int64_t)gridDim.x);
    block_dots<CPLX>(g, V, w, c0, len, g.k, sred);
    ok = all_sums<CPLX>(g, g.k + 1, sc, target);
    if (!ok) break;
    if (tid >= OT - 32) {  // scalars by one warp, while the others go on
      const int lane = tid % 32;
      double sub = 0.0;
      for (int j = lane; j < g.k; j += 32) sub = fma(sc[j].x, sc[j].x, fma(sc[j].y, sc[j].y, sub));
      for (int o = 16; o > 0; o >>= 1) sub += __shfl_xor_sync(0xffffffffu, sub, o);
      if (lane == 0) {
        const double all = sc[g.k].x, rest = all - sub;
        slast = pass == 2 || !(rest < 0.5 * all);
        // a NaN stays one; a sum that rounding made negative is zero
        sleft = rest < 0.0 ? 0.0 : sqrt(rest);
        sinv = 1.0 / sleft;
      }
    }
    // one element per thread stays in a register until the norm is known
    const int rounds = (len + OT - 1) / OT;
    T keep = Num<CPLX>::zero();
    if (len <= 64 && len > 0) {
      // a piece of one or two warps: the vectors are dealt to four or two groups of threads,
      // so that every scheduler works
      const int L = len <= 32 ? 32 : 64, Q = 128 / L;
      const int i = tid % L, q = tid / L;
      T a = Num<CPLX>::zero();
      if (q < Q && i < len) {
        const T* v = V + c0 + i;
#pragma unroll 4
        for (int j = q; j < g.k; j += Q) sub_mul(a, v[(int64_t)j * g.ld], sc[j]);
        if (q) spart[(q - 1) * L + i] = as_double2(a);
      }
      __syncthreads();
      if (tid < len) {
        keep = w[tid];
        add_to(keep, as_double2(a));
        for (int p = 0; p < Q - 1; ++p) add_to(keep, spart[p * L + tid]);
      }
    } else {
      // pairs of entries, for twice the loads in flight
      int r = 0;
      for (; (r + 2) * OT <= len; r += 2) {
        const int i = r * OT + tid;
        T a = w[i], b = w[i + OT];
        const T* v = V + c0 + i;
#pragma unroll 8
        for (int j = 0; j < g.k; ++j) {
          const T* vj = v + (int64_t)j * g.ld;
          const T x = vj[0], y = vj[OT];
          sub_mul(a, x, sc[j]);
          sub_mul(b, y, sc[j]);
        }
        w[i] = a;
        w[i + OT] = b;
      }
      for (; r < rounds; ++r) {
        const int i = r * OT + tid;
        if (i < len) {
          T a = w[i];
          const T* v = V + c0 + i;
#pragma unroll 8
          for (int j = 0; j < g.k; ++j) sub_mul(a, v[(int64_t)j * g.ld], sc[j]);
          keep = a;
          if (rounds > 1) w[i] = a;
        }
      }
    }
    __syncthreads();
    for (int j = tid; j < g.k; j += OT) {
      sh[j].x += sc[j].x;
      sh[j].y += sc[j].y;
    }
    const bool last = slast;
    const double inv = sinv;
    T* dst = !last ? w : g.vnext ? (T*)g.vnext + c0 : wg;
    const bool scale = last && g.vnext;
    for (int r = 0; r < rounds; ++r) {
      const int i = r * OT + tid;
      if (i < len) {
        const T a = rounds > 1 ? w[i] : keep;
        dst[i] = scale ? scaled(a, inv) : a;
      }
    }
    __syncthreads();
    if (last) break;
  }
  if (!ok) {
    // any block may give up, and the others may not notice: the host is told beside the numbers
    if (tid == 0) {
      *g.gave_up = 1.0;
      sleft = __longlong_as_double(0x7ff8000000000000ll);
    }
    __syncthreads();
  }
  if (blockIdx.x == 0) {
    for (int j = tid; j < g.k; j += OT) ((double2*)g.out)[j] = sh[j];
    if (tid == 0) {
      g.out[2 * g.k] = sleft;
      g.prev[0] = sh[g.k - 1].x;
      g.prev[1] = sleft;
    }
  }
  grid_leave(g);
}

struct CombineArgs {
  OrthArgs g;
  double c[2 * 64];
  int normalize;
};

// dst = sum_j c_j V_j, normalised; without basis vectors (k = 0) dst = w / |w|
template <bool CPLX>
__global__ void __launch_bounds__(OT) krylov_combine_kernel(CombineArgs a) {
  using T = typename Num<CPLX>::T;
  const OrthArgs& g = a.g;
  __shared__ double2 sc[1];
  const int64_t per = ((g.n + gridDim.x - 1) / gridDim.x + 31) / 32 * 32;
  const int64_t c0 = min(g.n, per * blockIdx.x);
  const int len = (int)(min(g.n, c0 + per) - c0);
  T* dst = (T*)g.vnext + c0;
  const T* src = g.k ? dst : (const T*)g.w + c0;
  chain_release();
  chain_wait();
  for (int i = threadIdx.x; g.k && i < len; i += OT) {
    T s = Num<CPLX>::zero();
    const T* v = (const T*)g.V + c0 + i;
#pragma unroll 8
    for (int j = 0; j < g.k; ++j)
      sub_mul(s, v[(int64_t)j * g.ld], make_double2(-a.c[2 * j], -a.c[2 * j + 1]));
    dst[i] = s;
  }
  if (a.normalize) {
    __syncthreads();
    unsigned int target = 0;
    __shared__ double2 sred[DOT_SUMS];
    block_dots<CPLX>(g, (const T*)nullptr, src, c0, len, 0, sred);
    __shared__ double sinv;
    const bool ok = all_sums<CPLX>(g, 1, sc, target);
    if (threadIdx.x == 0) {
      // NaN where the wait ran out: a piece without its norm must not pass for a result
      const double nrm = ok ? sqrt(sc[0].x) : __longlong_as_double(0x7ff8000000000000ll);
      sinv = 1.0 / nrm;
      if (blockIdx.x == 0 && g.out) g.out[0] = nrm;
      if (!ok && g.gave_up) *g.gave_up = 1.0;
    }
    __syncthreads();
    const double inv = sinv;
    for (int i = threadIdx.x; i < len; i += OT) dst[i] = scaled(src[i], inv);
    grid_leave(g);
  }
}

// clusters of more than eight blocks need a device that grants them
bool orth_cluster_fits(int device) {
  static DeviceOnce once;
  static std::mutex mu;
  static std::map<int, bool> granted;
  once(device, [device] {
    bool fits = true;
    auto allow = [&](const void* kernel) {
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
          cudaSuccess) {
        cudaGetLastError();
        fits = false;
        return;
      }
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(16);
      cfg.blockDim = dim3(OT);
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim = {16, 1, 1};
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) cudaGetLastError();
      if (n < 1) fits = false;
    };
    allow((const void*)krylov_orth_kernel<true>);
    allow((const void*)krylov_orth_kernel<false>);
    allow((const void*)krylov_combine_kernel<true>);
    allow((const void*)krylov_combine_kernel<false>);
    std::lock_guard<std::mutex> lk(mu);
    granted[device] = fits;
  });
  std::lock_guard<std::mutex> lk(mu);
  return granted[device];
}

// blocks of a launch: one per SM at most, pieces of 64 entries at least.  Up to 128 complex (256
// real) entries for each of 16 blocks they are one cluster: a hardware barrier instead of one
// through memory (300 clocks and 3000), sums over 16 parts that every block adds itself, and a
// launch that can join the chain.  With the host's wait for the kernel in place of a system-wide
// fence, a D = 32 time step of 1100 such steps goes from 31.5 to 27.0 ms.
constexpr int OCLUSTER = 16;
int orth_blocks(gb_ctx* ctx, int dtype, int64_t n, bool* cluster) {
  const int64_t most = std::max(1, ctx->num_sms);
  const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>(most, (n + 63) / 64));
  *cluster = blocks > 1 && n <= OCLUSTER * (is_cplx(dtype) ? 128 : 256) && orth_cluster_fits(ctx->device);
  return (int)(*cluster ? std::min<int64_t>(blocks, OCLUSTER) : blocks);
}

template <typename A>
void orth_launch(gb_ctx* ctx, void (*kernel)(A), int blocks, bool cluster, size_t smem, A args) {
  if (cluster) {
    launch_chained(kernel, dim3(blocks), OT, smem, ctx->stream, blocks, 1, args);
  } else {
    void* p[] = {&args};
    GB_CHECK_CUDA(cudaLaunchCooperativeKernel((const void*)kernel, dim3(blocks), dim3(OT), p, smem,
                                              ctx->stream));
  }
  count_launch(ctx);
}

OrthArgs orth_args(gb_ctx* ctx, int64_t n, int blocks) {
  OrthArgs g{};
  g.n = n;
  const size_t part = 2 * (size_t)(OKMAX + 1) * blocks * 16;
  char* s = (char*)scratch(ctx, SLOT_RED, part + (OKMAX + 1) * 16 + 256);
  g.part = (double*)s;
  g.coef = (double*)(s + part);
  g.bar = (unsigned int*)((char*)ctx->d_status + 64);
  g.prev = (double*)((char*)ctx->d_status + 80);
  g.status = ctx->d_status;
  g.wait_ns = ctx->wait_ns;
  return g;
}

}  // namespace

// pinned host memory that kernels write scalar results to
double* host_results(gb_ctx* ctx, size_t elems) {
  if (ctx->h_pinned_elems < elems) {
    GB_CHECK_CUDA(cudaStreamSynchronize(ctx->stream));
    if (ctx->h_pinned) cudaFreeHost(ctx->h_pinned);
    ctx->h_pinned = nullptr;
    ctx->h_pinned_elems = 0;
    const size_t n = std::max<size_t>(elems, 512);
    GB_CHECK_CUDA(cudaMallocHost(&ctx->h_pinned, sizeof(double) * n));
    ctx->h_pinned_elems = n;
  }
  return ctx->h_pinned;
}

bool krylov_orth_fits(int k) { return k <= OKMAX; }

// doubles of one step's results; the last one: a block gave up
constexpr size_t OSLOT = 2 * (OKMAX + 1) + 2;

void krylov_orth_start(gb_ctx* ctx, int dtype, int64_t n, int k, bool predict, const void* V,
                       void* w, void* vnext, int slot) {
  GB_REQUIRE(k >= 1 && k <= OKMAX && n > 0 && slot >= 0 && slot < ORTH_SLOTS,
             "krylov_orth: shape");
  bool cluster = false;
  const int blocks = orth_blocks(ctx, dtype, n, &cluster);
  OrthArgs g = orth_args(ctx, n, blocks);
  g.cluster = cluster;
  g.ld = n;
  g.k = k;
  g.predict = predict && k >= 2;
  g.V = (const double*)V;
  g.w = (double*)w;
  g.vnext = (double*)vnext;
  const int64_t per = ((n + blocks - 1) / blocks + 31) / 32 * 32;
  const size_t bytes = (size_t)per * elem_size(dtype);
  g.in_smem = bytes <= OPIECE;
  g.out = host_results(ctx, OSLOT * ORTH_SLOTS) + OSLOT * slot;
  g.gave_up = g.out + OSLOT - 1;
  *g.gave_up = 0.0;
  if (!ctx->orth_done[slot])
    GB_CHECK_CUDA(cudaEventCreateWithFlags(&ctx->orth_done[slot], cudaEventDisableTiming));
  static DeviceOnce once;
  once(ctx->device, [] {
    GB_CHECK_CUDA(cudaFuncSetAttribute(krylov_orth_kernel<true>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)OPIECE));
    GB_CHECK_CUDA(cudaFuncSetAttribute(krylov_orth_kernel<false>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)OPIECE));
  });
  orth_launch(ctx, is_cplx(dtype) ? krylov_orth_kernel<true> : krylov_orth_kernel<false>, blocks,
              cluster, g.in_smem ? bytes : 0, g);
  GB_CHECK_CUDA(cudaEventRecord(ctx->orth_done[slot], ctx->stream));
}

void krylov_orth_wait(gb_ctx* ctx, int k, int slot, cplx* h, double* norm) {
  GB_CHECK_CUDA(cudaEventSynchronize(ctx->orth_done[slot]));
  const double* out = ctx->h_pinned + OSLOT * slot;
  if (out[OSLOT - 1] != 0.0) throw Error(GB_ERR_TIMEOUT, "Krylov step: a device wait ran out");
  for (int j = 0; j < k; ++j) h[j] = cplx{out[2 * j], out[2 * j + 1]};
  *norm = out[2 * k];
}

void krylov_orth(gb_ctx* ctx, int dtype, int64_t n, int k, const void* V, void* w, void* vnext,
                 cplx* h, double* norm) {
  krylov_orth_start(ctx, dtype, n, k, false, V, w, vnext, 0);
  krylov_orth_wait(ctx, k, 0, h, norm);
}

// dst = sum_{j < k} coef_j V_j, divided by its norm when normalize is set (real coefficients
// only then).  k = 0: dst = src / |src|, the norm to *norm (waits)
void krylov_combine(gb_ctx* ctx, int dtype, int64_t n, int k, const void* V, const cplx* coef,
                    const void* src, void* dst, bool normalize, double* norm) {
  GB_REQUIRE(k >= 0 && k <= 64 && n > 0, "krylov_combine: shape");
  bool cluster = false;
  const int blocks = orth_blocks(ctx, dtype, n, &cluster);
  CombineArgs a{};
  a.g = orth_args(ctx, n, blocks);
  a.g.cluster = cluster;
  a.g.ld = n;
  a.g.k = k;
  a.g.V = (const double*)V;
  a.g.w = (double*)src;
  a.g.vnext = (double*)dst;
  a.g.out = norm ? host_results(ctx, OSLOT * ORTH_SLOTS) : nullptr;
  if (norm) {
    a.g.gave_up = a.g.out + OSLOT - 1;
    *a.g.gave_up = 0.0;
  }
  a.normalize = normalize;
  for (int j = 0; j < k; ++j) {
    a.c[2 * j] = coef[j].re;
    a.c[2 * j + 1] = coef[j].im;
  }
  orth_launch(ctx, is_cplx(dtype) ? krylov_combine_kernel<true> : krylov_combine_kernel<false>,
              blocks, cluster, 0, a);
  if (norm) {
    GB_CHECK_CUDA(cudaStreamSynchronize(ctx->stream));
    if (*a.g.gave_up != 0.0) throw Error(GB_ERR_TIMEOUT, "Krylov vector: a device wait ran out");
    *norm = a.g.out[0];
  }
}

}  // namespace gb

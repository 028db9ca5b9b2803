// FP64 GEMMs that do not run at the FP64 pipe's pace.
//
// GB300 issues two FP64 FMAs per clock and SM, so a 64 x 64 x 64 tile is 70 us of one SM's
// time.  Two kernels replace the 64 x 64-tile SIMT GEMM where they win:
//
//  * gemm_sliced_kernel -- the product in exact integer arithmetic on the tensor cores.
//    Every row of op(A) and every column of op(B) is scaled by a power of two so that its
//    largest entry fills 55 bits, rounded to an integer of 56 bits, and written as seven
//    signed 8-bit digits (error-free slicing as in Ozaki, Ogita, Oishi & Rump, "Error-free
//    transformations of matrix multiplication by using fast routines of matrix
//    multiplication and its applications", Numer. Algorithms 59 (2012) 95-118; on tensor
//    cores: Mukunoki, Ozaki, Ogita & Imamura, ISC 2020).  A digit is an integer of magnitude
//    <= 128, which BF16 holds exactly; products of digits are <= 2^14, and the sum over 128
//    contraction indices of at most seven of them stays below 2^24, so the FP32 accumulators
//    of tcgen05 hold it exactly.  The 34 digit products with i + j <= 7 are kept (the
//    dropped ones are 2^-8 of the rounding of the digits themselves); the eight accumulators,
//    one per i + j, are added into 96-bit integers after every 128 contraction indices, and
//    the only rounding besides the slicing is the final one to FP64.
//
//    Measured (one product, operands cut included; SIMT tiles / here): complex 256 x 256 x 256
//    531 / 21 us, complex 512 x 512 x 256 530 / 39 us, real 2048^3 8.6 / 0.58 ms = 30 TFLOP/s.
//    Its error against extended precision at K = 128..256 is 5.7e-17 of the result (the FMAs':
//    3.8e-16).  That is norm by norm.  The bound of an entry is one of its row and column,
//    2 K 2^-54 max |a| max |b| (four times that when complex), where the FMAs' is
//    K 2^-53 sum |a_k| |b_k|: terms far below the largest entries of the row and the column keep
//    fewer bits, and those below 2^-55 of them vanish ((1, 1e-10) times (1e-10, 1)' is off by 1e-7
//    of itself).  Krylov vectors, environments and Gram matrices are used by norms; the positive QR
//    scales its columns first; other callers have GB_OPT_FP64_FMA.
//
//  * gemm_small_kernel -- plain FP64 FMAs in tiles small enough that a product of a few
//    million FMAs is spread over all SMs (complex 22 x 69 x 23: 240 / 3.6 us).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "gb_common.h"
#include "tc_ptx.cuh"

namespace gb {

CUtensorMap make_slice_map(void* data, int64_t kdim, int64_t rows, int64_t planes, int box_rows,
                           int box_planes);

// ------------------------------------------------------------------ slicing
constexpr int SL = F64_SLICES;   // digits per entry
constexpr int DG = SL + 1;       // accumulators: i + j = 0 .. 7
constexpr int SL_SHIFT = 2;      // 53-bit mantissas are shifted to 55 bits at the row maximum

// one operand of a sliced GEMM: the logical R x K matrix (rows of op(A), columns of op(B))
struct SliceArgs {
  const double* src;
  int64_t ld, stride;  // elements
  int64_t R, K, Kh, Kp;
  int64_t rows;        // packed rows per batch entry
  int64_t imrow;       // first packed row of the imaginary parts (complex B)
  int rowfast;         // R is the contiguous index of src
  int cplx, conj, isB;
  int batch;
  int nchunk, kchunk;  // row maxima are taken over chunks of kchunk contraction indices
  int* part;           // [batch][nchunk][R] maxima of the biased exponent
  int* exps;           // [batch][R]
  __nv_bfloat16* planes;  // [batch][SL][rows][Kp]
  uint32_t* nz;        // [batch][groups][Kp / 64]: a 32-row x 64-k block holds a nonzero (a
                       // byte for each 8 rows)
  int64_t groups;
  int rblk;            // row blocks of 32
  int nblk;            // blocks of this operand in the launch
};

__device__ __forceinline__ int biased_exp(double v) {
  return (__double2hiint(v) >> 20) & 0x7ff;
}

// part[b][chunk][r] = max over the chunk of the biased exponents of row r.  Block: 32 rows.
// Bound by reading the operand once; a row of blocks per chunk keeps the chip busy when R is
// small.  Latency-sized operands dominate, so both operands share one launch.
__global__ void __launch_bounds__(256) slice_max_kernel(SliceArgs a, SliceArgs b) {
  chain_release();
  chain_wait();
  const bool second = (int)blockIdx.x >= a.nblk;
  const SliceArgs& p = second ? b : a;
  int blk = second ? (int)blockIdx.x - a.nblk : (int)blockIdx.x;
  const int c = blk % p.nchunk;
  blk /= p.nchunk;
  const int rb = blk % p.rblk, z = blk / p.rblk;
  const int lane = threadIdx.x % 32, w = threadIdx.x / 32;
  const int64_t k0 = (int64_t)c * p.kchunk, k1 = min(p.K, k0 + p.kchunk);
  const double* src = p.src + (int64_t)z * p.stride * (p.cplx ? 2 : 1);
  __shared__ int red[8][33];
  int* out = p.part + ((int64_t)z * p.nchunk + c) * p.R;
  if (p.rowfast) {
    const int64_t r = (int64_t)rb * 32 + lane;
    int m = 0;
    if (r < p.R) {
      if (p.cplx) {
        const double2* s = (const double2*)src + r;
#pragma unroll 4
        for (int64_t k = k0 + w; k < k1; k += 8) {
          const double2 v = s[k * p.ld];
          m = max(m, max(biased_exp(v.x), biased_exp(v.y)));
        }
      } else {
        const double* s = src + r;
#pragma unroll 4
        for (int64_t k = k0 + w; k < k1; k += 8) m = max(m, biased_exp(s[k * p.ld]));
      }
    }
    red[w][lane] = m;
    __syncthreads();
    if (w == 0 && r < p.R) {
      for (int i = 1; i < 8; ++i) m = max(m, red[i][lane]);
      out[r] = m;
    }
  } else {
    for (int i = w; i < 32; i += 8) {
      const int64_t r = (int64_t)rb * 32 + i;
      if (r >= p.R) break;
      int m = 0;
      if (p.cplx) {
        const double2* s = (const double2*)src + r * p.ld;
#pragma unroll 2
        for (int64_t k = k0 + lane; k < k1; k += 32) {
          const double2 v = s[k];
          m = max(m, max(biased_exp(v.x), biased_exp(v.y)));
        }
      } else {
        const double* s = src + r * p.ld;
#pragma unroll 4
        for (int64_t k = k0 + lane; k < k1; k += 32) m = max(m, biased_exp(s[k]));
      }
      m = __reduce_max_sync(0xffffffffu, m);
      if (lane == 0) out[r] = m;
    }
  }
}

// biased fixed-point image of v in a row whose largest biased exponent is E:
// Y = round(v 2^(1075 + SL_SHIFT - E)) + 0x80808080808080, whose bytes are digit + 128
__device__ __forceinline__ unsigned long long slice_bits(double v, int E) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(v);
  const int e = (int)(u >> 52) & 0x7ff;
  unsigned long long m = u & 0xfffffffffffffull;
  m |= e ? (1ull << 52) : 0ull;
  const int sh = E - max(e, 1) - SL_SHIFT;  // right shift (negative: left)
  if (sh <= 0) {
    m <<= -sh;
  } else {
    m = sh < 64 ? (m + (1ull << (sh - 1))) >> sh : 0ull;
  }
  const unsigned long long bias = 0x80808080808080ull;
  return (long long)u < 0 ? bias - m : bias + m;
}
__device__ __forceinline__ uint32_t digit_pair(uint32_t b0, uint32_t b1) {
  // byte b holds digit + 128; the float of an integer of magnitude <= 128 has its BF16 image
  // in its upper half
  const float f0 = __uint_as_float(0x4B000000u | b0) - 8388736.0f;
  const float f1 = __uint_as_float(0x4B000000u | b1) - 8388736.0f;
  return __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632);
}

// digits of an RB-row x 64-k block: the source block goes through shared memory (its contiguous
// index is R or K), each warp then writes whole 128-byte K lines of the planes.
template <int RB>
struct SliceSmem {
  double re[RB][65], im[RB][65];
  int e[RB];       // largest biased exponents of the rows: this CTA's k-blocks
  int all[RB];     // of the whole rows
};

template <int RB>
__device__ __forceinline__ void slice_load(const SliceArgs& p, SliceSmem<RB>& s, const double* src,
                                           int64_t r0, int64_t k0, int& nz, bool maxima) {
  const int tid = threadIdx.x;
  const long long flip = p.conj ? (long long)(1ull << 63) : 0;
  int m = 0;
  double re[RB / 4], im[RB / 4];
#pragma unroll
  for (int i = 0; i < RB / 4; ++i) {
    const int e = tid + 256 * i;
    const int rr = p.rowfast ? e % RB : e / 64, kk = p.rowfast ? e / RB : e % 64;
    const int64_t r = r0 + rr, k = k0 + kk;
    re[i] = im[i] = 0.0;
    if (r < p.R && k < p.K) {
      const int64_t ad = p.rowfast ? r + p.ld * k : k + p.ld * r;
      if (p.cplx) {
        const double2 v = ((const double2*)src)[ad];
        re[i] = v.x;
        im[i] = __longlong_as_double(__double_as_longlong(v.y) ^ flip);
      } else {
        re[i] = src[ad];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < RB / 4; ++i) {
    const int e = tid + 256 * i;
    const int rr = p.rowfast ? e % RB : e / 64, kk = p.rowfast ? e / RB : e % 64;
    // zero tests and sign flips on the bits: comparisons run on the FP64 pipe
    nz |= ((__double_as_longlong(re[i]) | __double_as_longlong(im[i])) << 1) != 0;
    s.re[rr][kk] = re[i];
    if (p.cplx) s.im[rr][kk] = im[i];
    if (maxima) {
      const int x = max(biased_exp(re[i]), biased_exp(im[i]));
      if (p.rowfast) {
        m = max(m, x);
      } else {
        const int w = __reduce_max_sync(0xffffffffu, x);
        if (tid % 32 == 0) atomicMax(&s.e[rr], w);
      }
    }
  }
  if (maxima && p.rowfast) atomicMax(&s.e[tid % RB], m);
}

template <int RB>
__device__ __forceinline__ void slice_store(const SliceArgs& p, const SliceSmem<RB>& s, int z,
                                            int64_t r0, int64_t k0) {
  const int lane = threadIdx.x % 32, w = threadIdx.x / 32;
  const int64_t plane = p.rows * p.Kp;
  __nv_bfloat16* base = p.planes + (int64_t)z * SL * plane;
  auto put = [&](int64_t row, int64_t k, unsigned long long y0, unsigned long long y1) {
    uint32_t* d = (uint32_t*)(base + row * p.Kp + k) + lane;
#pragma unroll
    for (int i = 0; i < SL; ++i) {
      const int sh = 8 * (SL - 1 - i);
      const uint32_t mask = i == 0 ? 0x1ffu : 0xffu;  // the top digit may be +128
      *d = digit_pair((uint32_t)(y0 >> sh) & mask, (uint32_t)(y1 >> sh) & mask);
      d += plane / 2;
    }
  };
  const unsigned long long two_bias = 2ull * 0x80808080808080ull;
#pragma unroll 1
  for (int rr = w; rr < RB; rr += 8) {
    const int64_t r = r0 + rr;
    if (r >= (p.isB && p.cplx ? p.imrow : p.R)) break;  // complex B: pad rows are written too
    const int E = max(s.all[rr], 1);
    const unsigned long long y0 = slice_bits(s.re[rr][2 * lane], E),
                             y1 = slice_bits(s.re[rr][2 * lane + 1], E);
    put(r, k0, y0, y1);
    if (p.cplx) {
      const unsigned long long w0 = slice_bits(s.im[rr][2 * lane], E),
                               w1 = slice_bits(s.im[rr][2 * lane + 1], E);
      if (!p.isB) {
        put(r, p.Kh + k0, w0, w1);
      } else {
        // bytes of bias - m are those of 2 bias - (bias + m)
        put(r, p.Kh + k0, two_bias - w0, two_bias - w1);
        put(p.imrow + r, k0, w0, w1);
        put(p.imrow + r, p.Kh + k0, y0, y1);
      }
    }
  }
}

// flag of the RB-row x 64-k block at rows r0 (an 8-row piece writes its byte)
template <int RB>
__device__ __forceinline__ void slice_flags(const SliceArgs& p, int z, int64_t r0, int kb, int nz) {
  const int64_t kbs = p.Kh / 64, kbp = p.Kp / 64;
  uint32_t* nzb = p.nz + (int64_t)z * p.groups * kbp;
  auto put = [&](int64_t i) {
    if (RB == 32) nzb[i] = nz ? 1u : 0u;
    else ((uint8_t*)(nzb + i))[r0 % 32 / 8] = nz ? 1 : 0;
  };
  const int64_t rb = r0 / 32;
  put(rb * kbp + kb);
  if (p.cplx) {
    put(rb * kbp + kbs + kb);
    if (p.isB) {
      const int64_t ri = p.imrow / 32 + rb;
      put(ri * kbp + kb);
      put(ri * kbp + kbs + kb);
    }
  }
}

// Row maxima and digits in one launch: the CTAs of a cluster share a block of rows, each takes
// every cs-th 64-k block, and the maxima meet in distributed shared memory.  A row's first pass
// leaves the CTA's last k-block in shared memory; the others are read again (from L2).  Bound by
// the writes: 14 bytes per real entry (28 per complex entry of A, 56 of B); below a few million
// entries by its latency, which is why operands of few blocks are cut into 8-row pieces and why it
// is one launch: complex 256 x 256, 16.5 us as
// a launch for the maxima and one for the digits, 8.8 us here.
template <int RB>
__global__ void __launch_bounds__(256) slice_cluster_kernel(SliceArgs a, SliceArgs b, int cs,
                                                            double* zero, int64_t nzero) {
  __shared__ SliceSmem<RB> s;
  const int rank = (int)blockIdx.x % cs;  // clusters are runs of cs CTAs
  int blk = (int)blockIdx.x / cs;
  const bool second = blk >= a.nblk;
  const SliceArgs& p = second ? b : a;
  if (second) blk -= a.nblk;
  const int kbs = (int)(p.Kh / 64);
  const int per = p.rblk * (32 / RB), rb = blk % per, z = blk / per;
  const int64_t r0 = (int64_t)rb * RB;
  const double* src = p.src + (int64_t)z * p.stride * (p.cplx ? 2 : 1);
  const int tid = threadIdx.x;
  if (tid < RB) s.e[tid] = 0;
  chain_release();
  chain_wait();
  for (int64_t i = blockIdx.x * (int64_t)256 + tid; i < nzero; i += (int64_t)gridDim.x * 256)
    zero[i] = 0.0;
  const int mine = rank < kbs ? (kbs - rank + cs - 1) / cs : 0;
  int nz = 0;
  for (int i = 0; i < mine; ++i) {
    __syncthreads();
    nz = 0;
    slice_load<RB>(p, s, src, r0, (int64_t)(rank + i * cs) * 64, nz, true);
  }
  __syncwarp();
  if (cs > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
  if (tid < RB) {
    int m = 0;
    for (int c = 0; c < cs; ++c) {
      uint32_t at;
      int v;
      asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_u32(&s.e[tid])), "r"(c));
      asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
      m = max(m, v);
    }
    s.all[tid] = m;
    if (rank == 0 && r0 + tid < p.R) p.exps[(int64_t)z * p.R + r0 + tid] = m;
  }
  // no CTA leaves while another reads its maxima
  __syncwarp();
  if (cs > 1) asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
  for (int i = mine - 1; i >= 0; --i) {
    const int kb = rank + i * cs;
    if (i < mine - 1) {
      __syncthreads();
      nz = 0;
      slice_load<RB>(p, s, src, r0, (int64_t)kb * 64, nz, false);
    }
    nz = __syncthreads_or(nz);
    if (tid == 0) slice_flags<RB>(p, z, r0, kb, nz);
    slice_store<RB>(p, s, z, r0, (int64_t)kb * 64);
  }
  if (cs > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
}

// The digits alone, the row maxima being in p.part (few rows and a long contraction: a CTA per
// 64-k block)
__global__ void __launch_bounds__(256) slice_kernel(SliceArgs a, SliceArgs b) {
  __shared__ SliceSmem<32> s;
  const bool second = (int)blockIdx.x >= a.nblk;
  const SliceArgs& p = second ? b : a;
  int blk = second ? (int)blockIdx.x - a.nblk : (int)blockIdx.x;
  const int kbs = (int)(p.Kh / 64);
  const int kb = blk % kbs;
  blk /= kbs;
  const int rb = blk % p.rblk, z = blk / p.rblk;
  const int64_t r0 = (int64_t)rb * 32, k0 = (int64_t)kb * 64;
  const double* src = p.src + (int64_t)z * p.stride * (p.cplx ? 2 : 1);
  const int tid = threadIdx.x;
  chain_release();
  chain_wait();
  if (tid < 32) {
    int m = 0;
    if (r0 + tid < p.R) {
      for (int c = 0; c < p.nchunk; ++c)
        m = max(m, p.part[((int64_t)z * p.nchunk + c) * p.R + r0 + tid]);
      if (kb == 0) p.exps[(int64_t)z * p.R + r0 + tid] = m;
    }
    s.all[tid] = m;
  }
  int nz = 0;
  slice_load<32>(p, s, src, r0, k0, nz, false);
  nz = __syncthreads_or(nz);
  if (tid == 0) slice_flags<32>(p, z, r0, kb, nz);
  slice_store<32>(p, s, z, r0, k0);
}

// ------------------------------------------------------------------ the GEMM
constexpr int SG_THREADS = 320;     // producer, MMA and eight epilogue warps
constexpr int SG_CHUNK = 2;         // 64-wide k-blocks whose sums are exact in FP32
constexpr int SG_MAX_KB = 4096;     // k-blocks of one tile (list in shared memory)
constexpr int SG_A_BYTES = 128 * 128;

struct SGArgs {
  int64_t M, N;      // logical
  int cplx;
  int64_t imrow;     // packed row of B where the imaginary parts begin
  int nkb;           // Kp / 64
  int batchA, batchB;
  const uint32_t *nzA, *nzB;
  int64_t grpA, grpB;
  const int *eA, *eB;
  double alpha, beta;
  double* C;
  int64_t ldc, sC;
  int splits;        // CTAs of a cluster that share a tile's k-blocks
  int mt, nt;
  int* status;
  unsigned long long wait_ns;
  // rows with Inf or NaN: their entries are recomputed from the operands themselves
  const double *A, *B;
  int64_t lda, sA, ldb, sB, K;
  int opA, opB;      // 0 'N', 1 'T', 2 'C'
  int add;           // C += by atomics: two products of one launch share an output
};
// one product, or two whose blocks along x follow one another
template <int PRODUCTS>
struct SGLaunch {
  CUtensorMap a[PRODUCTS], b[PRODUCTS];
  SGArgs g[PRODUCTS];
  int first;         // blocks of the first
};

// products of one digit of A with n digits of B (adjacent rows, adjacent accumulators)
template <int BN>
__device__ __forceinline__ void issue_digits(uint32_t d, uint64_t da, uint64_t db, int n,
                                             uint32_t acc) {
  constexpr int PER = 256 / BN;
  for (int j = 0; j < n; j += PER)
    mma_bf16(d + j * BN, da, db + (uint64_t)(j * BN * 8),
             idesc_bf16(128, (n - j < PER ? n - j : PER) * BN), acc);
}

template <int BN>
struct SGShape {
  static constexpr int B_BYTES = SL * BN * 128;
  static constexpr int BST = BN == 64 ? 2 : 3;   // B stages (all digits of a k-block)
  static constexpr int AST = BN == 64 ? 6 : 7;   // A stages (one digit of a k-block)
  static constexpr int BUFS = BN == 64 ? 1 : 2;  // accumulator sets in TMEM
  static constexpr int SMEM = BST * B_BYTES + AST * SG_A_BYTES + SG_MAX_KB * 2 + 1024 + 1280;
};

#define TMEM_LD16(taddr, r)                                                                    \
  asm volatile(                                                                                \
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13," \
      "%14,%15}, [%16];"                                                                       \
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),   \
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),            \
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15])                                                  \
      : "r"(taddr))

// results outside the normal range (kept out of line: if-converted into the common path its
// FP64 instructions cost more than the whole product)
__device__ __noinline__ long long out_of_range(unsigned long long r, int e) {
  return __double_as_longlong(scalbn((double)(long long)r, e));
}

// bits of (hi 2^32 + lo) 2^T rounded to FP64, with integer instructions: the FP64 pipe issues
// one warp instruction in 16 clocks.  64 leading bits are kept before the rounding.  Free of
// branches, so that the conversions of several entries overlap; *be outside 1..2045 (with
// *r the 53 leading bits) leaves the entry to out_of_range.
__device__ __forceinline__ long long fixed_to_double(long long hi, long long lo, int T,
                                                     unsigned long long* r, int* be) {
  hi += lo >> 32;
  const uint32_t sign = (uint32_t)(hi >> 63);
  uint32_t w0 = (uint32_t)lo ^ sign, w1 = (uint32_t)hi ^ sign, w2 = (uint32_t)(hi >> 32) ^ sign;
  // two's complement of the 96-bit value: + 1 when negative
  w0 -= sign;
  const uint32_t c0 = sign & (uint32_t)(w0 == 0);
  w1 += c0;
  w2 += c0 & (uint32_t)(w1 == 0);
  // the leading nonzero word first
  const bool z2 = w2 == 0, z1 = z2 && w1 == 0;
  const uint32_t a2 = z1 ? w0 : z2 ? w1 : w2, a1 = z1 ? 0u : z2 ? w0 : w1, a0 = z2 ? 0u : w0;
  const int ex = z1 ? -32 : z2 ? 0 : 32;
  const int sh = __clz((int)a2) & 31;
  const uint32_t m1 = __funnelshift_l(a1, a2, sh), m0 = __funnelshift_l(a0, a1, sh);
  const unsigned long long m = ((unsigned long long)m1 << 32) | m0;
  *r = (m >> 11) + ((m >> 10) & 1);
  const bool zero = a2 == 0;
  *be = zero ? 1 : 63 + ex - sh + T + 1023;
  const unsigned long long v = ((unsigned long long)(uint32_t)(*be - 1) << 52) + *r;  // hidden bit
  return (long long)(zero ? 0ull : v | ((unsigned long long)(sign & 1) << 63));
}

// one entry of op(A) op(B) by FP64 FMAs (rows or columns with Inf or NaN)
__device__ __noinline__ void plain_entry(const SGArgs& g, int z, int64_t m, int64_t n, double* re,
                                         double* im) {
  const int c = g.cplx ? 2 : 1;
  const double* A = g.A + (int64_t)z * g.sA * c;
  const double* B = g.B + (int64_t)z * g.sB * c;
  double xr = 0.0, xi = 0.0;
  for (int64_t k = 0; k < g.K; ++k) {
    const double* a = A + c * (g.opA ? k + g.lda * m : m + g.lda * k);
    const double* b = B + c * (g.opB ? n + g.ldb * k : k + g.ldb * n);
    if (g.cplx) {
      const double ar = a[0], ai = g.opA == 2 ? -a[1] : a[1];
      const double br = b[0], bi = g.opB == 2 ? -b[1] : b[1];
      xr = fma(ar, br, fma(-ai, bi, xr));
      xi = fma(ar, bi, fma(ai, br, xi));
    } else {
      xr = fma(a[0], b[0], xr);
    }
  }
  *re = xr;
  *im = xi;
}

// One CTA per 128 x BN tile (and split of its k-blocks).  Warp 0 streams, by TMA, all seven
// digits of a 64-wide k-block of B (one box) and the digits of A one at a time; warp 1 issues
// for digit i of A the products with the digits 0..min(6, 7-i) of B -- they are adjacent rows
// in shared memory, and the accumulators i + j = i..7 adjacent TMEM columns, so one or two
// instructions of N up to 256 cover them; warps 2-9 add the accumulators of every 128
// contraction indices into 96-bit integers.  Blocks of zeros (block-sparse operands stored
// densely) are left out.  A tile grid under half the chip splits the k-blocks over the CTAs of
// a cluster; each then adds the integer sums of all of them for its share of the columns
// (through distributed shared memory: exact, so the result does not depend on the split).
template <int BN, int PRODUCTS>
__global__ void __launch_bounds__(SG_THREADS, 1)
    gemm_sliced_kernel(const __grid_constant__ SGLaunch<PRODUCTS> L) {
  const int which = PRODUCTS > 1 && (int)blockIdx.x >= L.first ? 1 : 0;
  const int block = (int)blockIdx.x - (which ? L.first : 0);
  const SGArgs& g = L.g[which];
  const CUtensorMap &mapA = L.a[which], &mapB = L.b[which];
  using S = SGShape<BN>;
  constexpr int HC = BN / 2;  // columns per epilogue thread
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sB = smem;
  uint8_t* sA = smem + S::BST * S::B_BYTES;
  uint16_t* list = (uint16_t*)(sA + S::AST * SG_A_BYTES);
  uint64_t* bars = (uint64_t*)(list + SG_MAX_KB);
  uint64_t *fullA = bars, *emptyA = fullA + S::AST, *fullB = emptyA + S::AST,
           *emptyB = fullB + S::BST, *tfull = emptyB + S::BST, *tempty = tfull + S::BUFS,
           *done = tempty + S::BUFS;
  int* scnt = (int*)(done + 1);
  int* sfail = scnt + 1;
  uint32_t* tmem_slot = (uint32_t*)(sfail + 1);
  int* seb = (int*)(tmem_slot + 1);  // [BN] column exponents
  int* sea = seb + BN;               // [128] row exponents

  const int warp = warp_index(), lane = threadIdx.x % 32;
  const int mi = block % g.mt, rest = block / g.mt;
  const int ni = rest % g.nt, z = rest / g.nt;
  const int split = blockIdx.y;
  const int64_t m0 = (int64_t)mi * 128, n0 = (int64_t)ni * BN;
  const int zA = g.batchA > 1 ? z : 0, zB = g.batchB > 1 ? z : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::AST; ++s) {
      mbar_init(smem_u32(&fullA[s]), 1);
      mbar_init(smem_u32(&emptyA[s]), 1);
    }
    for (int s = 0; s < S::BST; ++s) {
      mbar_init(smem_u32(&fullB[s]), 1);
      mbar_init(smem_u32(&emptyB[s]), 1);
    }
    for (int s = 0; s < S::BUFS; ++s) {
      mbar_init(smem_u32(&tfull[s]), 1);
      mbar_init(smem_u32(&tempty[s]), 8);
    }
    mbar_init(smem_u32(done), 1);
    *sfail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&mapA) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&mapB) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  chain_release();
  chain_wait();
  if (warp == 3) {
    for (int i = lane; i < 128; i += 32)
      sea[i] = m0 + i < g.M ? g.eA[(int64_t)zA * g.M + m0 + i] : 0;
  }
  if (warp >= 4) {
    // row and column exponents, read once per tile
    const int64_t np = n0 + threadIdx.x - 128;
    if (threadIdx.x - 128 < BN) {
      const int64_t n = g.cplx && np >= g.imrow ? np - g.imrow : np;
      seb[threadIdx.x - 128] = n < g.N ? g.eB[(int64_t)zB * g.N + n] : 0;
    }
  }
  if (warp == 2) {
    // the k-blocks in which both operands hold a nonzero, in order
    const uint32_t* za = g.nzA + ((int64_t)zA * g.grpA + m0 / 32) * g.nkb;
    const uint32_t* zb = g.nzB + ((int64_t)zB * g.grpB + n0 / 32) * g.nkb;
    const int ga = (int)min((int64_t)4, g.grpA - m0 / 32);
    const int gb_ = (int)min((int64_t)(BN / 32), g.grpB - n0 / 32);
    int cnt = 0;
    for (int k0 = 0; k0 < g.nkb; k0 += 32) {
      const int kb = k0 + lane;
      int fa = 0, fb = 0;
      if (kb < g.nkb) {
        for (int q = 0; q < ga; ++q) fa |= za[(int64_t)q * g.nkb + kb];
        for (int q = 0; q < gb_; ++q) fb |= zb[(int64_t)q * g.nkb + kb];
      }
      const unsigned v = __ballot_sync(0xffffffffu, fa && fb);
      if ((v >> lane) & 1u) list[cnt + __popc(v & ((1u << lane) - 1u))] = (uint16_t)kb;
      cnt += __popc(v);
    }
    if (lane == 0) *scnt = cnt;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const int cnt = *scnt;
  const int b0 = (int)((int64_t)cnt * split / g.splits);
  const int b1 = (int)((int64_t)cnt * (split + 1) / g.splits);
  const int nb = b1 - b0;

  if (warp == 0 && elect_one()) {
    // ---------------- TMA producer
    uint32_t ia = 0, ib = 0;
    bool ok = true;
    for (int t = 0; t < nb && ok; ++t) {
      const int kb = list[b0 + t];
      const int sb = ib % S::BST;
      ok = mbar_wait_bounded(smem_u32(&emptyB[sb]), ((ib / S::BST) & 1) ^ 1, g.status, g.wait_ns);
      if (!ok) break;
      mbar_expect_tx(smem_u32(&fullB[sb]), S::B_BYTES);
      tma_load_3d(smem_u32(sB + sb * S::B_BYTES), &mapB, smem_u32(&fullB[sb]), kb * 64, (int)n0,
                 zB * SL);
      ++ib;
      for (int i = 0; i < SL; ++i) {
        const int sa = ia % S::AST;
        ok = mbar_wait_bounded(smem_u32(&emptyA[sa]), ((ia / S::AST) & 1) ^ 1, g.status,
                               g.wait_ns);
        if (!ok) break;
        mbar_expect_tx(smem_u32(&fullA[sa]), SG_A_BYTES);
        tma_load_3d(smem_u32(sA + sa * SG_A_BYTES), &mapA, smem_u32(&fullA[sa]), kb * 64, (int)m0,
                    zA * SL + i);
        ++ia;
      }
    }
    if (!ok) {
      // drain the copies still in flight before this CTA may exit
      for (uint32_t t = ia > (uint32_t)S::AST ? ia - S::AST : 0; t < ia; ++t)
        mbar_wait_bounded(smem_u32(&fullA[t % S::AST]), (t / S::AST) & 1, g.status, DRAIN_WAIT_NS);
      for (uint32_t t = ib > (uint32_t)S::BST ? ib - S::BST : 0; t < ib; ++t)
        mbar_wait_bounded(smem_u32(&fullB[t % S::BST]), (t / S::BST) & 1, g.status, DRAIN_WAIT_NS);
    }
  } else if (warp == 1 && elect_one()) {
    // ---------------- MMA issuer
    uint32_t ia = 0, ib = 0;
    bool ok = true;
    for (int t = 0; t < nb && ok; ++t) {
      const int chunk = t / SG_CHUNK, buf = chunk % S::BUFS;
      if (t % SG_CHUNK == 0) {
        ok = mbar_wait_bounded(smem_u32(&tempty[buf]), ((chunk / S::BUFS) & 1) ^ 1, g.status,
                               g.wait_ns);
        if (!ok) break;
        tc_fence_after();
      }
      const int sb = ib % S::BST;
      ok = mbar_wait_bounded(smem_u32(&fullB[sb]), (ib / S::BST) & 1, g.status, g.wait_ns);
      if (!ok) break;
      const uint64_t db = smem_desc_sw128(smem_u32(sB + sb * S::B_BYTES));
      const uint32_t d0 = tmem + buf * (DG * BN);
#pragma unroll
      for (int i = 0; i < SL; ++i) {
        const int sa = ia % S::AST;
        ok = mbar_wait_bounded(smem_u32(&fullA[sa]), (ia / S::AST) & 1, g.status, g.wait_ns);
        if (!ok) break;
        tc_fence_after();
        const uint64_t da = smem_desc_sw128(smem_u32(sA + sa * SG_A_BYTES));
        // digits 0..nj-1 of B into accumulators i..i+nj-1; the first k-step of a chunk
        // overwrites: digit 0 of A starts accumulators 0..6, digit 1 starts the last one
        const int nj = i == 0 ? SL : SL + 1 - i;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const bool first = t % SG_CHUNK == 0 && k == 0;
          const int head = first && i == 1 ? nj - 1 : nj;
          const uint32_t acc = first && i == 0 ? 0u : 1u;
          issue_digits<BN>(d0 + i * BN, da + 2 * k, db + 2 * k, head, acc);
          if (head < nj)
            issue_digits<BN>(d0 + (i + head) * BN, da + 2 * k, db + 2 * k + head * BN * 8, 1, 0u);
        }
        mma_commit(smem_u32(&emptyA[sa]));
        ++ia;
      }
      if (!ok) break;
      mma_commit(smem_u32(&emptyB[sb]));
      ++ib;
      if (t % SG_CHUNK == SG_CHUNK - 1 || t == nb - 1) mma_commit(smem_u32(&tfull[buf]));
    }
    mma_commit(smem_u32(done));
    mbar_wait_bounded(smem_u32(done), 0, g.status, DRAIN_WAIT_NS);
  } else if (warp >= 2) {
    // ---------------- integer accumulation and output
    const int q = warp % 4, half = (warp - 2) / 4;
    const int et = threadIdx.x - 64;
    long long hi[HC], lo[HC];
#pragma unroll
    for (int j = 0; j < HC; ++j) hi[j] = lo[j] = 0;
    bool ok = true;
    const int nchunk = (nb + SG_CHUNK - 1) / SG_CHUNK;
    for (int c = 0; c < nchunk; ++c) {
      const int buf = c % S::BUFS;
      ok = mbar_wait_bounded(smem_u32(&tfull[buf]), (c / S::BUFS) & 1, g.status, g.wait_ns);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const uint32_t base = tmem + ((uint32_t)(32 * q) << 16) + buf * (DG * BN) + half * HC;
#pragma unroll
      for (int d = 0; d < DG; ++d) {
        const int wgt = 1 << (8 * (3 - d % 4));
#pragma unroll
        for (int j0 = 0; j0 < HC; j0 += 16) {
          uint32_t v[16];
          TMEM_LD16(base + d * BN + j0, v);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int a = __float2int_rn(__uint_as_float(v[j]));
            if (d < 4) hi[j0 + j] += (long long)a * wgt;
            else lo[j0 + j] += (long long)a * wgt;
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&tempty[buf]));
    }
    // the sums go through shared memory (the operand stages are free: every MMA has retired),
    // for the other CTAs of the cluster and so that the conversion is a rolled loop: unrolled
    // over the registers it is tens of kilobytes of straight-line code, fetched once per tile
    if (ok) {
      long long* st = (long long*)smem + et;
#pragma unroll
      for (int j = 0; j < HC; ++j) {
        st[(2 * j) * 256] = hi[j];
        st[(2 * j + 1) * 256] = lo[j];
      }
    } else if (lane == 0) {
      *sfail = 1;
    }
  }
  __syncwarp();
  if (g.splits > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
  if (warp >= 2 && !*sfail) {
    const int q = warp % 4, half = (warp - 2) / 4;
    const int et = threadIdx.x - 64;
    const int64_t m = m0 + 32 * q + lane;
    if (m < g.M) {
      const int ea = sea[32 * q + lane];
      const uint32_t st = smem_u32(smem) + 8 * et;
      const int j0 = HC * split / g.splits, j1 = HC * (split + 1) / g.splits;
      // column j of every CTA of the cluster
      auto sums = [&](int j, long long& hi, long long& lo) {
        if (g.splits == 1) {
          asm volatile("ld.shared.b64 %0, [%1];" : "=l"(hi) : "r"(st + j * 4096));
          asm volatile("ld.shared.b64 %0, [%1];" : "=l"(lo) : "r"(st + j * 4096 + 2048));
          return;
        }
        hi = lo = 0;
        for (int c = 0; c < g.splits; ++c) {
          uint32_t ad;
          long long h, l;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ad) : "r"(st + j * 4096), "r"(c));
          asm volatile("ld.shared::cluster.b64 %0, [%1];" : "=l"(h) : "r"(ad));
          asm volatile("ld.shared::cluster.b64 %0, [%1];" : "=l"(l) : "r"(ad + 2048));
          hi += h;
          lo += l;
        }
      };
      // the columns of this thread are real or imaginary parts as a whole (imrow is a
      // multiple of 32)
      const int64_t np0 = n0 + half * HC;
      const bool im = g.cplx && np0 >= g.imrow;
      const int64_t n00 = im ? np0 - g.imrow : np0;
      const int jn = (int)min((int64_t)j1, g.N - n00);
      double* C = g.C + (int64_t)z * g.sC * (g.cplx ? 2 : 1);
      C += g.cplx ? 2 * (m + g.ldc * n00) + (im ? 1 : 0) : m + g.ldc * n00;
      const int64_t step = g.cplx ? 2 * g.ldc : g.ldc;
      const int T0 = 8 * (2 * (SL - 1) - (DG - 1)) + max(ea, 1) - 2 * (1075 + SL_SHIFT);
      // one loop per form of the update: a conditional FP64 instruction in a common loop is
      // executed and selected, and each costs as much as the conversion
      uint32_t slow = 0;  // entries that the conversion does not cover
      auto update = [&](auto form, double* p, double v) {
        if constexpr (form.value == 3) {
          atomicAdd(p, v);
          return;
        }
        if constexpr (form.value == 1) v += *p;
        if constexpr (form.value == 2) {
          v *= g.alpha;
          if (g.beta != 0.0) v = fma(g.beta, *p, v);
        }
        *p = v;
      };
      auto store = [&](auto form) {
#pragma unroll 4
        for (int j = j0; j < jn; ++j) {
          // entries have units 2^(E - 1075 - SL_SHIFT), accumulator d units 256^(12 - d)
          const int eb = seb[half * HC + j];
          long long hi, lo;
          sums(j, hi, lo);
          unsigned long long r;
          int be;
          const long long bits = fixed_to_double(hi, lo, T0 + max(eb, 1), &r, &be);
          const bool odd = ea == 0x7ff || eb == 0x7ff || (unsigned)(be - 1) >= 2045u;
          slow |= (uint32_t)odd << j;
          if (!odd) update(form, C + step * j, __longlong_as_double(bits));
        }
        while (slow) {
          const int j = __ffs(slow) - 1;
          slow &= slow - 1;
          const int eb = seb[half * HC + j];
          double v;
          if (ea == 0x7ff || eb == 0x7ff) {
            double xr, xi;
            plain_entry(g, z, m, n00 + j, &xr, &xi);
            v = im ? xi : xr;
          } else {
            long long hi, lo;
            sums(j, hi, lo);
            unsigned long long r;
            int be;
            fixed_to_double(hi, lo, T0 + max(eb, 1), &r, &be);
            const bool neg = hi + (lo >> 32) < 0;
            v = __longlong_as_double(out_of_range(r, be - 1075) |
                                     (long long)((unsigned long long)neg << 63));
          }
          update(form, C + step * j, v);
        }
      };
      if (g.add) store(std::integral_constant<int, 3>{});
      else if (g.alpha == 1.0 && g.beta == 0.0) store(std::integral_constant<int, 0>{});
      else if (g.alpha == 1.0 && g.beta == 1.0) store(std::integral_constant<int, 1>{});
      else store(std::integral_constant<int, 2>{});
    }
  }
  tc_fence_before();
  __syncwarp();
  if (g.splits > 1) {  // no CTA leaves while another reads its sums
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

// ------------------------------------------------------------------ small products
// TM x TN outputs per CTA of 128 threads, KG adjacent lanes share an output's contraction: the FP64
// pipe is the bound (two FMAs per clock and SM) together with the latency of one pass through the
// operands, so the tile is chosen to put work on every SM rather than for operand reuse, and the
// next piece of the operands is loaded while one is used.  Two products may add up in one output
// (y = x R + L x), one launch
// instead of two of 4.5 us for complex 32 x 64 x 64 and 64 x 32 x 64.
template <typename T>
struct SmallOps;
template <>
struct SmallOps<double> {
  static __device__ double zero() { return 0.0; }
  static __device__ double fma_(double a, double b, double c) { return fma(a, b, c); }
  static __device__ double add(double a, double b) { return a + b; }
  static __device__ double conj(double a) { return a; }
  static __device__ double shfl_xor(double a, int d) { return __shfl_xor_sync(0xffffffffu, a, d); }
};
template <>
struct SmallOps<double2> {
  static __device__ double2 zero() { return make_double2(0.0, 0.0); }
  static __device__ double2 fma_(double2 a, double2 b, double2 c) {
    return make_double2(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
  }
  static __device__ double2 add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
  static __device__ double2 conj(double2 a) { return make_double2(a.x, -a.y); }
  static __device__ double2 shfl_xor(double2 a, int d) {
    return make_double2(__shfl_xor_sync(0xffffffffu, a.x, d), __shfl_xor_sync(0xffffffffu, a.y, d));
  }
};

template <typename T>
struct SmallProduct {
  const T *A, *B;
  int64_t lda, sA, ldb, sB, K;
  int opA, opB;  // 0 'N', 1 'T', 2 'C'
};
template <typename T>
struct SmallArgs {
  int64_t M, N, ldc, sC, kchunk;
  T alpha, beta;
  int use_beta, products;
  T* C;
  SmallProduct<T> p[2];
};

template <typename T, int TM, int TN>
__global__ void __launch_bounds__(128) gemm_small_kernel(const __grid_constant__ SmallArgs<T> g) {
  using O = SmallOps<T>;
  constexpr int KG = 128 / (TM * TN);  // lanes of an output
  constexpr int KB = KG > 1 ? 64 : 32;
  constexpr int LD = KB + (KG > 1 ? KG : 1);  // rows of neighbouring outputs in other banks
  constexpr int NA = TM * KB / 128, NB = TN * KB / 128;
  __shared__ T As[TM * LD], Bs[TN * LD];
  const int64_t bz = blockIdx.z;
  const int64_t m0 = (int64_t)blockIdx.x * TM, n0 = (int64_t)blockIdx.y * TN;
  const int tid = threadIdx.x, kg = tid % KG, o = tid / KG;
  const int tm = o % TM, tn = o / TM;
  const bool live = m0 + tm < g.M && n0 + tn < g.N;
  T a[NA], b[NB];
  // the piece of product q that starts at kb
  auto load = [&](int q, int64_t kb, int64_t k1) {
    const SmallProduct<T>& p = g.p[q];
    const T *A = p.A + (g.kchunk ? 0 : bz * p.sA), *Bq = p.B + (g.kchunk ? 0 : bz * p.sB);
#pragma unroll
    for (int i = 0; i < NA; ++i) {
      const int e = tid + 128 * i;
      const int r = p.opA ? e / KB : e % TM, c = p.opA ? e % KB : e / TM;
      a[i] = O::zero();
      if (m0 + r < g.M && kb + c < k1)
        a[i] = p.opA ? A[kb + c + p.lda * (m0 + r)] : A[m0 + r + p.lda * (kb + c)];
      if (p.opA == 2) a[i] = O::conj(a[i]);
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const int e = tid + 128 * i;
      const int c = p.opB ? e % TN : e / KB, r = p.opB ? e / TN : e % KB;
      b[i] = O::zero();
      if (n0 + c < g.N && kb + r < k1)
        b[i] = p.opB ? Bq[n0 + c + p.ldb * (kb + r)] : Bq[kb + r + p.ldb * (n0 + c)];
      if (p.opB == 2) b[i] = O::conj(b[i]);
    }
  };
  int64_t kb = g.kchunk ? bz * g.kchunk : 0, k1 = g.kchunk ? min(g.p[0].K, kb + g.kchunk) : g.p[0].K;
  int q = 0;
  T acc = O::zero();
  chain_release();
  chain_wait();
  load(0, kb, k1);
  for (;;) {
    {
      const SmallProduct<T>& p = g.p[q];
#pragma unroll
      for (int i = 0; i < NA; ++i) {
        const int e = tid + 128 * i;
        As[p.opA ? (e / KB) * LD + e % KB : (e % TM) * LD + e / TM] = a[i];
      }
#pragma unroll
      for (int i = 0; i < NB; ++i) {
        const int e = tid + 128 * i;
        Bs[p.opB ? (e % TN) * LD + e / TN : (e / KB) * LD + e % KB] = b[i];
      }
    }
    __syncthreads();
    const int kn = (int)min((int64_t)KB, k1 - kb);
    kb += KB;
    bool more = kb < k1;
    if (!more && q + 1 < g.products) {
      ++q;
      kb = 0;
      k1 = g.p[q].K;
      more = k1 > 0;
    }
    if (more) load(q, kb, k1);
    if (live) {
#pragma unroll 4
      for (int k = kg; k < kn; k += KG) acc = O::fma_(As[tm * LD + k], Bs[tn * LD + k], acc);
    }
    if (!more) break;
    __syncthreads();
  }
  // the lanes' sums, by one warp: four from shared memory each, then across the 32 / (TM TN) lanes
  // of an output (exchanging them in every warp is up to five times the FP64 instructions)
  int out = o;
  if (KG > 1) {
    constexpr int LP = KG > 1 ? KG / 4 : 1;
    __shared__ T red[KG > 1 ? 128 : 1];
    red[tid] = acc;
    __syncthreads();
    if (tid >= 32) return;
    out = tid / LP;
    const T* part = red + out * KG + tid % LP;
    acc = part[0];
#pragma unroll
    for (int i = 1; i < 4; ++i) acc = O::add(acc, part[i * LP]);
#pragma unroll
    for (int d = 1; d < LP; d *= 2) acc = O::add(acc, O::shfl_xor(acc, d));
    if (tid % LP) return;
  }
  const int64_t m = m0 + out % TM, n = n0 + out / TM;
  if (m >= g.M || n >= g.N) return;
  T* C = g.C + bz * g.sC + m + g.ldc * n;
  T v = O::fma_(g.alpha, acc, O::zero());
  if (g.use_beta) v = O::fma_(g.beta, *C, v);
  *C = v;
}

// ------------------------------------------------------------------ host side
static inline int64_t rup(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

size_t sliced_bytes(int64_t R, int64_t K, bool cx, int role, int64_t batch) {
  const int64_t Kp = rup(K, 64) * (cx ? 2 : 1);
  const bool dbl = cx && role == PACK_AS_B;
  const int64_t rows = dbl ? 2 * rup(R, 32) : R;
  const int64_t groups = (rows + 31) / 32;
  return (size_t)rup(batch * SL * rows * Kp * 2, 256) + (size_t)rup(batch * groups * (Kp / 64) * 4, 256) +
         (size_t)rup(batch * R * 4, 256) + (size_t)rup(batch * 16 * R * 4, 256);
}

static SliceArgs slice_args(gb_ctx* ctx, int dtype, int role, char op, int64_t R, int64_t K,
                            const void* src, int64_t ld, int64_t stride, int64_t batch, void* dst,
                            Packed& out) {
  const bool cx = is_cplx(dtype);
  SliceArgs a{};
  a.src = (const double*)src;
  a.ld = ld;
  a.stride = stride;
  a.R = R;
  a.K = K;
  a.Kh = rup(K, 64);
  a.Kp = cx ? 2 * a.Kh : a.Kh;
  a.isB = role == PACK_AS_B;
  a.cplx = cx;
  a.conj = op == 'C';
  a.imrow = rup(R, 32);
  a.rows = cx && a.isB ? 2 * a.imrow : R;
  a.rowfast = (role == PACK_AS_A) == (op == 'N');
  a.batch = (int)batch;
  a.groups = (a.rows + 31) / 32;
  a.rblk = (int)((R + 31) / 32);
  // enough blocks to fill the chip, chunks of at least 64 contraction indices, 16 at most
  const int64_t want = (2 * std::max(1, ctx->num_sms)) / std::max<int64_t>(1, a.rblk * batch);
  a.nchunk = (int)std::max<int64_t>(1, std::min<int64_t>({want, (K + 63) / 64, 16}));
  a.kchunk = (int)((K + a.nchunk - 1) / a.nchunk);
  char* d = (char*)dst;
  a.planes = (__nv_bfloat16*)d;
  d += rup(batch * SL * a.rows * a.Kp * 2, 256);
  a.nz = (uint32_t*)d;
  d += rup(batch * a.groups * (a.Kp / 64) * 4, 256);
  a.exps = (int*)d;
  d += rup(batch * R * 4, 256);
  a.part = (int*)d;
  out = Packed();
  out.data = dst;
  out.rows = a.rows;
  out.K = K;
  out.Kh = a.Kh;
  out.Kp = a.Kp;
  out.batch = batch;
  out.cplx = cx;
  out.slices = SL;
  out.nz = a.nz;
  out.exps = a.exps;
  out.mrows = a.groups;
  return a;
}

// also sets `zero` to zero, the output that products of the cut operands add up in
static void slice_launch(gb_ctx* ctx, SliceArgs a, SliceArgs b, double* zero = nullptr,
                         int64_t nzero = 0) {
  auto blocks = [](SliceArgs& s, int64_t per) {
    const int64_t n = s.src ? (int64_t)s.rblk * s.batch * per : 0;
    GB_REQUIRE(n < (int64_t)1 << 30, "gemm: operand too large to slice");
    s.nblk = (int)n;
    return n;
  };
  const int64_t ka = a.Kh / 64, kb = b.src ? b.Kh / 64 : 0, kbs = std::max(ka, kb);
  const int64_t sms = std::max(1, ctx->num_sms);
  const int64_t rows = blocks(a, 1) + blocks(b, 1);
  // One launch unless a cluster's CTAs would each walk many k-blocks while SMs stand idle (real
  // 128 x 2000: 12.7 us in one launch, 14.5 in two; 128 x 4000: 19 both; 128 x 8000: 30 and 23;
  // 64 k-blocks a CTA and more: 1.4 times the two launches).  Blocks of 8 rows where those of 32
  // would leave SMs idle (complex 256 x 512: 10.5 us against 12.6); beyond that they only cost
  // reads (real 1024 x 512: 16.5 against 12.5).
  const int cs = (int)std::min<int64_t>(8, kbs);
  if (kbs <= 32 || rows * cs >= sms) {
    const bool small = rows * cs <= sms;
    if (small) {
      blocks(a, 4);
      blocks(b, 4);
    }
    GB_REQUIRE((int64_t)(a.nblk + b.nblk) * cs < (int64_t)1 << 31,
               "gemm: operand too large to slice");
    launch_chained(small ? slice_cluster_kernel<8> : slice_cluster_kernel<32>,
                   dim3((unsigned)(a.nblk + b.nblk) * cs), 256, 0, ctx->stream, cs, 1, a, b, cs,
                   zero, nzero);
    count_launch(ctx);
    return;
  }
  if (nzero) fill_zero(ctx, zero, (size_t)nzero * 8);
  blocks(a, a.nchunk);
  blocks(b, b.nchunk);
  launch_chained(slice_max_kernel, dim3(a.nblk + b.nblk), 256, 0, ctx->stream, 1, 1, a, b);
  blocks(a, ka);
  blocks(b, kb);
  launch_chained(slice_kernel, dim3(a.nblk + b.nblk), 256, 0, ctx->stream, 1, 1, a, b);
  count_launch_n(ctx, 2);
}

void slice_operand(gb_ctx* ctx, int dtype, int role, char op, int64_t R, int64_t K,
                   const void* src, int64_t ld, int64_t stride, int64_t batch, Packed& out,
                   void* dst) {
  SliceArgs a = slice_args(ctx, dtype, role, op, R, K, src, ld, stride, batch, dst, out);
  SliceArgs none{};
  slice_launch(ctx, a, none);
}

// x as the left operand of one product (R1 x K1) and the right operand of another (K2 x R2), cut in
// one launch; both stay in the context's scratch.  False when that does not fit.
static bool slice_both(gb_ctx* ctx, int dtype, const void* x, int64_t R1, int64_t K1, int64_t R2,
                int64_t K2, Packed& a, Packed& b, double* zero, int64_t nzero) {
  const bool cx = is_cplx(dtype);
  void *da = nullptr, *db = nullptr;
  try {
    da = scratch(ctx, SLOT_PACK_A, sliced_bytes(R1, K1, cx, PACK_AS_A, 1));
    db = scratch(ctx, SLOT_PACK_B, sliced_bytes(R2, K2, cx, PACK_AS_B, 1));
  } catch (const Error& e) {
    if (e.code != GB_ERR_OOM) throw;
    cudaGetLastError();
    return false;
  }
  const SliceArgs aa = slice_args(ctx, dtype, PACK_AS_A, 'N', R1, K1, x, R1, 0, 1, da, a);
  const SliceArgs ab = slice_args(ctx, dtype, PACK_AS_B, 'N', R2, K2, x, K2, 0, 1, db, b);
  slice_launch(ctx, aa, ab, zero, nzero);
  return true;
}

bool gemm_sliced_wanted(gb_ctx* ctx, int dtype, int64_t M, int64_t N, int64_t K, int64_t batch,
                        double min_mac) {
  const double mac = (double)M * (double)N * (double)K * (double)batch * (is_cplx(dtype) ? 4 : 1);
  const int64_t nkb = rup(K, 64) * (is_cplx(dtype) ? 2 : 1) / 64;
  return !ctx->fp64_fma && mac >= min_mac && nkb <= SG_MAX_KB && M < (int64_t)1 << 30 &&
         N < (int64_t)1 << 29 && tc_available(ctx);
}

static int opcode(char op) { return op == 'N' ? 0 : op == 'T' ? 1 : 2; }

// one product, or two that add up in one output
template <int BN, int PRODUCTS>
static void launch_sliced(gb_ctx* ctx, const Packed* const* a, const Packed* const* b,
                          const SGArgs* g, int64_t batch) {
  using S = SGShape<BN>;
  static DeviceOnce once;
  once(ctx->device, [] {
    GB_CHECK_CUDA(cudaFuncSetAttribute(gemm_sliced_kernel<BN, PRODUCTS>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM));
  });
  SGLaunch<PRODUCTS> L{};
  int64_t tiles = 0;
  for (int i = 0; i < PRODUCTS; ++i) {
    L.a[i] = make_slice_map(a[i]->data, a[i]->Kp, a[i]->rows, a[i]->batch * SL, 128, 1);
    L.b[i] = make_slice_map(b[i]->data, b[i]->Kp, b[i]->rows, b[i]->batch * SL, BN, SL);
    L.g[i] = g[i];
    tiles += (int64_t)g[i].mt * g[i].nt * batch;
    GB_REQUIRE(tiles < (int64_t)1 << 31, "gemm: too many tiles");
    if (i == 0) L.first = (int)tiles;
  }
  launch_chained(gemm_sliced_kernel<BN, PRODUCTS>, dim3((unsigned)tiles, (unsigned)g[0].splits),
                 SG_THREADS, S::SMEM, ctx->stream, 1, g[0].splits, L);
  count_launch(ctx);
}

// digits of an operand of one product; on a lane (work items of many sizes, where a growing
// scratch slot would synchronise the device) from the stream-ordered pool
struct DigitBuf {
  gb_ctx* ctx;
  void* p = nullptr;
  bool own = false;
  explicit DigitBuf(gb_ctx* c) : ctx(c) {}
  bool get(int slot, size_t bytes) {
    if (ctx->lane) {
      own = cudaMallocAsync(&p, bytes, ctx->stream) == cudaSuccess;
      if (!own) p = nullptr;
    } else {
      try {
        p = scratch(ctx, slot, bytes);
      } catch (const Error& e) {
        if (e.code != GB_ERR_OOM) throw;
      }
    }
    if (!p) cudaGetLastError();
    return p != nullptr;
  }
  ~DigitBuf() {
    if (own) cudaFreeAsync(p, ctx->stream);
  }
  DigitBuf(const DigitBuf&) = delete;
  DigitBuf& operator=(const DigitBuf&) = delete;
};

static SGArgs sliced_args(gb_ctx* ctx, int dtype, char opA, char opB, int64_t M, int64_t N,
                          int64_t K, double alpha, const void* A, int64_t lda, int64_t sA,
                          const void* B, int64_t ldb, int64_t sB, double beta, void* C,
                          int64_t ldc, int64_t sC, const Packed& a, const Packed& b) {
  const bool cx = is_cplx(dtype);
  SGArgs g{};
  g.M = M;
  g.N = N;
  g.cplx = cx;
  g.imrow = cx ? rup(N, 32) : 0;
  g.nkb = (int)(a.Kp / 64);
  g.batchA = (int)a.batch;
  g.batchB = (int)b.batch;
  g.nzA = a.nz;
  g.nzB = b.nz;
  g.grpA = a.mrows;
  g.grpB = b.mrows;
  g.eA = a.exps;
  g.eB = b.exps;
  g.alpha = alpha;
  g.beta = beta;
  g.C = (double*)C;
  g.ldc = ldc;
  g.sC = sC;
  g.status = ctx->d_status;
  g.wait_ns = ctx->wait_ns;
  g.A = (const double*)A;
  g.B = (const double*)B;
  g.lda = lda;
  g.sA = sA;
  g.ldb = ldb;
  g.sB = sB;
  g.K = K;
  g.opA = opcode(opA);
  g.opB = opcode(opB);
  g.mt = (int)((M + 127) / 128);
  return g;
}

// Tile width and split by a model of the measured clocks.  A k-block moves its digits into and out
// of shared memory at 128 bytes a clock (388 KB at 32 columns, 616 KB at 64, which read A half as
// often); measured 3300 and 4900.  A tile has 7500 of start-up and pipeline ends, its output 110
// per column of a thread, adding the partial sums of a split 1000.  With a second product (mt2 > 0)
// for both in one launch.
struct SGPlan {
  double clocks = 1e300;
  bool wide = false;
  int nt[2] = {0, 0}, splits = 1;
};
static SGPlan sliced_plan(int sms, int mt, int64_t rows, int nkb, int64_t batch, int mt2 = 0,
                          int64_t rows2 = 0, int nkb2 = 0) {
  SGPlan p;
  for (int w = 0; w < 2; ++w) {
    const int64_t nt = (rows + (w ? 63 : 31)) / (w ? 64 : 32);
    const int64_t nt2 = (rows2 + (w ? 63 : 31)) / (w ? 64 : 32);
    const int64_t tiles = (int64_t)mt * nt * batch + (int64_t)mt2 * nt2;
    const int least = mt2 ? std::min(nkb, nkb2) : nkb, most = std::max(nkb, nkb2);
    for (int sp = 1; sp <= 8 && (sp == 1 || (tiles * sp <= sms && sp * 2 <= least)); sp *= 2) {
      const double waves = (double)((tiles * sp + sms - 1) / sms);
      const double kb = (double)((most + sp - 1) / sp);
      const double t = waves * (kb * (w ? 4900.0 : 3300.0) + 7500.0 + (w ? 3520.0 : 1760.0) / sp) +
                       (sp > 1 ? 1000.0 : 0.0);
      if (t < p.clocks) {
        p.clocks = t;
        p.wide = w;
        p.nt[0] = (int)nt;
        p.nt[1] = (int)nt2;
        p.splits = sp;
      }
    }
  }
  return p;
}

bool gemm_fp64_sliced(gb_ctx* ctx, int dtype, char opA, char opB, int64_t M, int64_t N, int64_t K,
                      double alpha, const void* A, int64_t lda, int64_t sA, const void* B,
                      int64_t ldb, int64_t sB, double beta, void* C, int64_t ldc, int64_t sC,
                      int64_t batch, const Packed* pA, const Packed* pB) {
  const bool cx = is_cplx(dtype);
  const int64_t bA = sA ? batch : 1, bB = sB ? batch : 1;
  Packed a, b;
  DigitBuf da(ctx), db(ctx);
  if (!pA && !da.get(SLOT_PACK_A, sliced_bytes(M, K, cx, PACK_AS_A, bA))) return false;
  if (!pB && !db.get(SLOT_PACK_B, sliced_bytes(N, K, cx, PACK_AS_B, bB))) return false;
  SliceArgs aa{}, ab{};
  if (pA) a = *pA;
  else aa = slice_args(ctx, dtype, PACK_AS_A, opA, M, K, A, lda, sA, bA, da.p, a);
  if (pB) b = *pB;
  else ab = slice_args(ctx, dtype, PACK_AS_B, opB, N, K, B, ldb, sB, bB, db.p, b);
  if (!pA && !pB) slice_launch(ctx, aa, ab);
  else if (!pA) slice_launch(ctx, aa, SliceArgs{});
  else if (!pB) slice_launch(ctx, ab, SliceArgs{});
  SGArgs g = sliced_args(ctx, dtype, opA, opB, M, N, K, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc,
                         sC, a, b);
  const int sms = std::max(1, ctx->num_sms);
  const SGPlan p = sliced_plan(sms, g.mt, b.rows, g.nkb, batch);
  g.nt = p.nt[0];
  g.splits = p.splits;
  const Packed *pa = &a, *pb = &b;
  if (p.wide) launch_sliced<64, 1>(ctx, &pa, &pb, &g, batch);
  else launch_sliced<32, 1>(ctx, &pa, &pb, &g, batch);
  return true;
}

// y = x R + L x, x and the constants cut into digits: both products in one launch when
// together they leave fewer SMs idle than one after the other; their outputs meet by atomic adds of
// two values on a cleared y, whose sum does not depend on the order (that of three would).  An apply of two complex products of 128 x
// 256 x 256: 31.0 us one by one, 20.9 us; of 256 x 512 x 512: 58 and 49 us.
bool gemm_sliced_pair(gb_ctx* ctx, int dtype, const void* x, int64_t M1, int64_t N1, int64_t K1,
                      const Packed& R, const void* Rsrc, int64_t ldr, int64_t M2, int64_t N2,
                      int64_t K2, const Packed& Lp, const void* Lsrc, int64_t ldl, void* y) {
  const bool cx = is_cplx(dtype);
  const int sms = std::max(1, ctx->num_sms);
  const int mt[2] = {(int)((M1 + 127) / 128), (int)((M2 + 127) / 128)};
  const int64_t rows[2] = {R.rows, cx ? 2 * rup(N2, 32) : N2};
  const int nkb[2] = {(int)(R.Kp / 64), (int)(Lp.Kp / 64)};
  const SGPlan p = sliced_plan(sms, mt[0], rows[0], nkb[0], 1, mt[1], rows[1], nkb[1]);
  const SGPlan p0 = sliced_plan(sms, mt[0], rows[0], nkb[0], 1);
  const SGPlan p1 = sliced_plan(sms, mt[1], rows[1], nkb[1], 1);
  Packed xa, xb;
  const bool together = p.clocks < p0.clocks + p1.clocks;
  const int64_t n = M1 * N1 * (cx ? 2 : 1);
  if (!slice_both(ctx, dtype, x, M1, K1, N2, K2, xa, xb, (double*)y,
                  together ? n : 0))
    return false;
  if (!together)
    return gemm_fp64_sliced(ctx, dtype, 'N', 'N', M1, N1, K1, 1.0, x, M1, 0, Rsrc, ldr, 0,
                            0.0, y, M1, 0, 1, &xa, &R) &&
           gemm_fp64_sliced(ctx, dtype, 'N', 'N', M2, N2, K2, 1.0, Lsrc, ldl, 0, x, K2, 0, 1.0, y,
                            M2, 0, 1, &Lp, &xb);
  SGArgs g[2] = {sliced_args(ctx, dtype, 'N', 'N', M1, N1, K1, 1.0, x, M1, 0, Rsrc, ldr, 0, 1.0, y,
                             M1, 0, xa, R),
                 sliced_args(ctx, dtype, 'N', 'N', M2, N2, K2, 1.0, Lsrc, ldl, 0, x, K2, 0, 1.0, y,
                             M2, 0, Lp, xb)};
  for (int i = 0; i < 2; ++i) {
    g[i].nt = p.nt[i];
    g[i].splits = p.splits;
    g[i].add = 1;
  }
  const Packed* pa[2] = {&xa, &Lp};
  const Packed* pb[2] = {&R, &xb};
  if (p.wide) launch_sliced<64, 2>(ctx, pa, pb, g, 1);
  else launch_sliced<32, 2>(ctx, pa, pb, g, 1);
  return true;
}

template <typename T>
static void small_launch(cudaStream_t st, const SmallPlan& p, const SmallArgs<T>& g,
                         int64_t batch) {
  void (*kernel)(SmallArgs<T>) = p.tm == 16   ? gemm_small_kernel<T, 16, 8>
                                 : p.tn == 8  ? gemm_small_kernel<T, 4, 8>
                                 : p.tm == 4  ? gemm_small_kernel<T, 4, 4>
                                              : gemm_small_kernel<T, 2, 4>;
  const dim3 grid((unsigned)((g.M + p.tm - 1) / p.tm), (unsigned)((g.N + p.tn - 1) / p.tn),
                  (unsigned)batch);
  launch_chained(kernel, grid, 128, 0, st, 1, 1, g);
}

// The tile (and split of the contraction) whose busiest SM is done first, by a model fitted to
// measured times: the FP64 pipe's clocks (real: two FMAs a clock), 0.6 of what a tile costs
// besides (some 320 clocks, 500 complex, and 250 for every further 64 contraction indices; the rest
// hides behind other tiles), 900 clocks of latency per 64 contraction indices at least.  The 16 x 8
// tile has one lane per output and needs many tiles per SM to hide its chain of additions.  In us
// for tiles of 16 x 8, 4 x 8, 4 x 4, 2 x 4: real 600 x 8 x 600: 8.1, 14, 24, 47; real 200 x 200 x
// 150: 28, 23, 17, 16; complex 32 x 32 x 160: 7.2, 5.4, 5.6, 7.7; complex 128^3: -, 30, 30, 22.
SmallPlan gemm_small_plan(int sms, int64_t M, int64_t N, int64_t K, int64_t batch, bool cx) {
  static const int tile[4][2] = {{16, 8}, {4, 8}, {4, 4}, {2, 4}};
  SmallPlan p;
  double best = 1e300;
  for (const auto& t : tile) {
    const int64_t n = ((M + t[0] - 1) / t[0]) * ((N + t[1] - 1) / t[1]) * batch;
    int64_t sp = 1;  // splits cost the launch that adds them up
    if (batch == 1 && K >= 512)
      sp = std::max<int64_t>(1, std::min<int64_t>({32, K / 256, 4 * (int64_t)sms / n}));
    const int64_t pieces = ((K + sp - 1) / sp + 63) / 64;
    const double waves = (double)((n * sp + sms - 1) / sms);
    const double work = t[0] * t[1] * (double)K / sp * (cx ? 2.0 : 0.5) *
                        (t[0] == 16 && n * sp < 8 * (int64_t)sms ? 2.0 : 1.0);
    const double rest = (cx ? 500.0 : 320.0) + 250.0 * (double)(pieces - 1);
    const double clk =
        std::max(waves * (work + 0.6 * rest), 900.0 * (double)pieces) + (sp > 1 ? 4000.0 : 0.0);
    if (clk < best) {
      best = clk;
      p.tm = t[0];
      p.tn = t[1];
      p.splits = (int)sp;
    }
  }
  p.ok = (M + p.tm - 1) / p.tm < (int64_t)1 << 31 && (N + p.tn - 1) / p.tn <= 65535 &&
         batch <= 65535;
  return p;
}

template <typename T>
static SmallProduct<T> small_product(char opA, char opB, int64_t K, const void* A, int64_t lda,
                                     int64_t sA, const void* B, int64_t ldb, int64_t sB) {
  return SmallProduct<T>{(const T*)A, (const T*)B, lda, sA, ldb, sB, K, opcode(opA), opcode(opB)};
}

void gemm_small(cudaStream_t st, const SmallPlan& p, int dtype, char opA, char opB, int64_t M,
                int64_t N, int64_t K, cplx alpha, const void* A, int64_t lda, int64_t sA,
                const void* B, int64_t ldb, int64_t sB, cplx beta, bool use_beta, void* C,
                int64_t ldc, int64_t sC, int64_t batch, int64_t kchunk) {
  auto run = [&](auto al, auto be) {
    using T = decltype(al);
    SmallArgs<T> g{M, N, ldc, sC, kchunk, al, be, use_beta ? 1 : 0, 1, (T*)C, {}};
    g.p[0] = small_product<T>(opA, opB, K, A, lda, sA, B, ldb, sB);
    small_launch(st, p, g, batch);
  };
  if (is_cplx(dtype)) run(make_double2(alpha.re, alpha.im), make_double2(beta.re, beta.im));
  else run(alpha.re, beta.re);
}

// y[l, s, r] = sum_k x[l, k] R[k, (s, r)] + sum_k L[(l, s), k] x[k, r] (+ y): one launch where both
// products are small.  x is contiguous: Ml x K1 for the first product, K2 x Nr for the second.
bool gemm_small_dual(gb_ctx* ctx, int dtype, int64_t Ml, int64_t d, int64_t Nr, int64_t K1,
                     const void* R, int64_t ldr, int64_t K2, const void* L, int64_t ldl,
                     const void* x, bool accumulate, void* y) {
  const bool cx = is_cplx(dtype);
  const double mac = (double)Ml * (double)d * (double)Nr * (cx ? 4 : 1);
  // each by itself would be a small product
  if (mac * (double)std::max(K1, K2) >= F64_SLICED_MIN_MAC_CUT) return false;
  const SmallPlan p = gemm_small_plan(std::max(1, ctx->num_sms), Ml, Nr, K1 + K2, d, cx);
  if (!p.ok) return false;
  auto run = [&](auto one) {
    using T = decltype(one);
    SmallArgs<T> g{Ml, Nr, Ml * d, Ml, 0, one, one, accumulate ? 1 : 0, 2, (T*)y, {}};
    // column (s, r) of R is its column s + d r; row (l, s) of L its row l + Ml s
    g.p[0] = small_product<T>('N', 'N', K1, x, Ml, 0, R, ldr * d, ldr);
    g.p[1] = small_product<T>('N', 'N', K2, L, ldl, Ml, x, K2, 0);
    small_launch(ctx->stream, p, g, d);
  };
  if (cx) run(make_double2(1.0, 0.0));
  else run(1.0);
  count_launch(ctx);
  return true;
}

}  // namespace gb

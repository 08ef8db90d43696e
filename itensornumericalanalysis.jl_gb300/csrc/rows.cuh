// Device code of the row-gather contractions of batched evaluation: digit
// codes, the one-child contraction over gathered rows, permuted tensor
// copies, and the dot product at the centre.
#pragma once
#include <climits>

#include "evaluate.cuh"

namespace tnfa {

// ------------------------------------------------------------- digits ----
// The digit map of the reference subtracts the largest v * base^-d that fits,
// digit after digit.  In base 2 the digits of x in [0, 1) are the leading bits
// of x, and all ones for x >= 1, so a run of digits that feeds one code with
// strides w, 2w, 4w, ... (or the reverse) is a bit field taken with integer
// operations (GB300 executes FP64 at 1/64 of the FP32 rate: the subtraction
// loop costs 2 FP64 operations per digit).  Other bases run the loop.
struct DigitRun {
  int col;       // column of X
  int slot;      // code it adds to
  int w;         // stride of the last digit of the run (first when reversed)
  short first;   // first digit, 1-based
  short n;       // digits in the run
  short base;
  short bits;    // a bit field (base 2); else one greedy digit
  short start;   // first run of its column: (re)load x
  short rev;     // the first digit has the smallest stride
  double invb;   // greedy: base^-first
};

__device__ __forceinline__ unsigned long long unit_fraction(double x) {
  // floor(x * 2^64) for x in [0, 1), all ones from 1 on
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int e = (int)((b >> 52) & 0x7FF) - 1023;
  if ((long long)b < 0) return 0;  // -0.0
  if (e >= 0) return ~0ull;
  const unsigned long long m = (b & 0xFFFFFFFFFFFFFull) | (1ull << 52);
  const int sh = 12 + e;
  if (sh >= 0) return m << sh;
  return sh > -53 ? m >> -sh : 0ull;
}

// Sets the error word (which may lie in host memory: one lane asks for the
// warp, and writes only until the word is seen set).
__device__ __noinline__ void raise_domain(int* err) {
  if ((int)(threadIdx.x & 31) == __ffs(__activemask()) - 1 && !(*(volatile int*)err & 1)) atomicOr(err, 1);
}

// Adds every run to codes[slot * ld] for the slots [s0, s1).
__device__ __forceinline__ void digit_codes(const double* __restrict__ Xp, const DigitRun* runs, int nruns,
                                            int* codes, int ld, int s0, int s1, int* err) {
  double xr = 0.0;
  unsigned long long u = 0;
  for (int e = 0; e < nruns; ++e) {
    const DigitRun d = runs[e];
    if (d.start) {
      xr = Xp[d.col];
      const unsigned long long xb = (unsigned long long)__double_as_longlong(xr);
      // negative (not -0), infinite or NaN
      if (xb > 0x8000000000000000ull || (xb & 0x7FF0000000000000ull) == 0x7FF0000000000000ull) {
        raise_domain(err);
        xr = 0.0;
      }
      u = unit_fraction(xr);
    }
    int add;
    if (d.bits) {
      unsigned f = (unsigned)((u << (d.first - 1)) >> 32);  // the run's digits at the top
      if (d.rev) f = __brev(f) & (0xFFFFFFFFu >> (32 - d.n));
      else f >>= 32 - d.n;
      add = (int)f * d.w;
    } else {
      int dig = 0;
      for (int v = d.base - 1; v >= 1; --v) {
        const double t = (double)v * d.invb;
        if (xr >= t) {
          dig = v;
          xr -= t;
          break;
        }
      }
      add = dig * d.w;
    }
    if (d.slot >= s0 && d.slot < s1) codes[(d.slot - s0) * ld] += add;
  }
}

// Codes of every point: C[slot * ldC + p].  Accumulated in shared memory, one
// column per thread; a program with more slots than fit runs in several
// launches over slot ranges.
__global__ void k_digitize(const double* __restrict__ X, int ncols, int Pc, const DigitRun* __restrict__ runs,
                           int nruns, int* __restrict__ C, int64_t ldC, int s0, int s1, int* __restrict__ err) {
  extern __shared__ int dig_sh[];
  const int n = s1 - s0;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < Pc; p += gridDim.x * blockDim.x) {
    int* c = dig_sh + threadIdx.x;
    for (int s = 0; s < n; ++s) c[s * blockDim.x] = 0;
    digit_codes(X + (int64_t)p * ncols, runs, nruns, c, blockDim.x, s0, s1, err);
    for (int s = 0; s < n; ++s) C[(int64_t)(s0 + s) * ldC + p] = c[s * blockDim.x];
  }
}

// ----------------------------------------------------------- grouping ----
// Points grouped by an integer key: counts, then offsets, tile starts and
// scatter cursors from the counts, then the permutation.  Up to GROUP_SMEM
// keys are counted in shared memory; more keys means few points each, and the
// global counters see little contention.
constexpr int GROUP_SMEM = 2048;

__global__ void k_group_count(const int* __restrict__ key, int Pc, int ng, int* __restrict__ cnt) {
  extern __shared__ int grp_sh[];
  if (ng > GROUP_SMEM) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < Pc; p += gridDim.x * blockDim.x)
      atomicAdd(&cnt[key[p]], 1);
    return;
  }
  for (int i = threadIdx.x; i < ng; i += blockDim.x) grp_sh[i] = 0;
  __syncthreads();
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < Pc; p += gridDim.x * blockDim.x)
    atomicAdd(&grp_sh[key[p]], 1);
  __syncthreads();
  for (int i = threadIdx.x; i < ng; i += blockDim.x)
    if (grp_sh[i]) atomicAdd(&cnt[i], grp_sh[i]);
}

// One block of 1024 threads: [off | cnt | tile_start (ng + 1) | cursor].
__global__ void __launch_bounds__(1024) k_group_scan(int* meta, int ng, int tp) {
  int* off = meta;
  int* cnt = meta + ng;
  int* ts = meta + 2 * ng;
  int* cur = meta + 3 * ng + 1;
  __shared__ int2 wsum[32];
  __shared__ int2 carry;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = make_int2(0, 0);
  __syncthreads();
  for (int g0 = 0; g0 < ng; g0 += 1024) {
    const int g = g0 + threadIdx.x;
    const int c = g < ng ? cnt[g] : 0, t = (c + tp - 1) / tp;
    int2 s = make_int2(c, t);
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, s.x, o), b = __shfl_up_sync(0xffffffffu, s.y, o);
      if (lane >= o) s.x += a, s.y += b;
    }
    if (lane == 31) wsum[warp] = s;
    __syncthreads();
    if (warp == 0) {
      int2 w = wsum[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, w.x, o), b = __shfl_up_sync(0xffffffffu, w.y, o);
        if (lane >= o) w.x += a, w.y += b;
      }
      wsum[lane] = w;
    }
    __syncthreads();
    const int2 base = warp ? wsum[warp - 1] : make_int2(0, 0);
    if (g < ng) {
      off[g] = cur[g] = carry.x + base.x + s.x - c;
      ts[g] = carry.y + base.y + s.y - t;
    }
    __syncthreads();
    if (threadIdx.x == 0) carry.x += wsum[31].x, carry.y += wsum[31].y;
    __syncthreads();
  }
  if (threadIdx.x == 0) ts[ng] = carry.y;
}

// Identity grouping (one group).
__global__ void k_group_identity(int* meta, int Pc, int tp) {
  meta[0] = 0;
  meta[1] = Pc;
  meta[2] = 0;
  meta[3] = (Pc + tp - 1) / tp;
  meta[4] = 0;
}

constexpr int SCATTER_ITEMS = 8;
__global__ void k_group_scatter(const int* __restrict__ key, int Pc, int ng, int* __restrict__ cur,
                                int* __restrict__ perm) {
  extern __shared__ int grp_sh[];
  const int p0 = blockIdx.x * blockDim.x * SCATTER_ITEMS;
  if (ng > GROUP_SMEM) {
    for (int i = 0; i < SCATTER_ITEMS; ++i) {
      const int p = p0 + i * blockDim.x + threadIdx.x;
      if (p < Pc) perm[atomicAdd(&cur[key[p]], 1)] = p;
    }
    return;
  }
  int* h = grp_sh;
  int* base = grp_sh + ng;
  for (int i = threadIdx.x; i < ng; i += blockDim.x) h[i] = 0;
  __syncthreads();
  int loc[SCATTER_ITEMS];
  int grp[SCATTER_ITEMS];
#pragma unroll
  for (int i = 0; i < SCATTER_ITEMS; ++i) {
    const int p = p0 + i * blockDim.x + threadIdx.x;
    grp[i] = -1;
    if (p < Pc) {
      grp[i] = key[p];
      loc[i] = atomicAdd(&h[grp[i]], 1);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < ng; i += blockDim.x) base[i] = h[i] ? atomicAdd(&cur[i], h[i]) : 0;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < SCATTER_ITEMS; ++i) {
    const int p = p0 + i * blockDim.x + threadIdx.x;
    if (grp[i] >= 0) perm[base[grp[i]] + loc[i]] = p;
  }
}

// Largest g with start[g] <= b (start ascending, start[0] = 0, b < start[ng]);
// among empty groups with equal starts the last, which is the one that has b.
__device__ __forceinline__ int find_group(const int* __restrict__ start, int ng, int b) {
  int lo = 0, hi = ng;  // start[lo] <= b < start[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (start[mid] <= b) lo = mid;
    else hi = mid;
  }
  return lo;
}

// --------------------------------------------------- exponent helpers ----
// Exponent e of frexp (2^(e-1) <= |x| < 2^e) from the bit pattern; 0 for zero,
// infinities and NaN, which are left unscaled.
__device__ __forceinline__ int exponent_of(float m) {
  if (!(m > 0.f) || m > 3.4028234663852886e38f) return 0;
  const int b = (int)(__float_as_uint(m) >> 23) & 0xFF;
  return b ? b - 126 : ilogbf(m) + 1;
}
__device__ __forceinline__ int exponent_of(double m) {
  const unsigned hi = (unsigned)((unsigned long long)__double_as_longlong(m) >> 32) & 0x7FFFFFFFu;
  const int b = (int)(hi >> 20);
  if (b == 0x7FF) return 0;
  if (b) return b - 1022;
  return m != 0.0 ? ilogb(m) + 1 : 0;
}
// x * 2^e, exact unless the result leaves the normal range.
__device__ __forceinline__ float scale_pow2(float x, int e) { return scalbnf(x, e); }
__device__ __forceinline__ double scale_pow2(double x, int e) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int be = (int)((b >> 52) & 0x7FF);
  if (be != 0 && be != 0x7FF && be + e > 0 && be + e < 0x7FF)
    return __longlong_as_double((long long)(b + ((unsigned long long)(long long)e << 52)));
  return scalbn(x, e);
}
__device__ __forceinline__ cplx scale_pow2(cplx z, int e) { return {scale_pow2(z.re, e), scale_pow2(z.im, e)}; }
// max of magnitudes without the FP64 pipe: doubles compare as their bits
__device__ __forceinline__ float mag_max(float m, float x) { return fmaxf(m, fabsf(x)); }
__device__ __forceinline__ double mag_max(double m, double x) {
  const long long a = __double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFll, b = __double_as_longlong(m);
  return __longlong_as_double(a > b ? a : b);
}
__device__ __forceinline__ double mag_max(double m, cplx z) { return mag_max(mag_max(m, z.re), z.im); }
template <class T> struct Real { using t = T; };
template <> struct Real<cplx> { using t = double; };

// ------------------------------------------------ row-gather products ----
// out[q][n] = sum_k A[row(q)][k] B[g(q)][n][k] over items q, each of one
// group g: the contraction of a vertex with one child (A its rows, B the
// vertex tensor, groups = site values), the absorption of a child's table
// into the tensor (N = the other axes), and the contraction with an absorbed
// tensor (groups = site value and absorbed row).  Groups are runs of rpg
// consecutive items, or given by a permutation (perm, grp_off, ...).  Rows of
// A are scaled by a power of two as they are read and the exponents of the
// row, the scaling and the group add up in out_exp.
template <class T>
struct RowJob {
  const T* A;
  const int* Aexp;  // null: zero
  RowIdx aidx;
  const T* B;
  const int* gexp;  // exponent of B[g], null: zero
  T* out;
  int* out_exp;
  int* rex;         // receives the scaling exponent of every row of A, null: not kept
  int K, N, rows;
  int rpg;  // > 0: uniform groups, and row(q) = q % rpg
  const int* perm;  // null: identity
  const int* grp_off;
  const int* grp_cnt;
  const int* tile_start;
  int ngroups;
};

// Up to ROW_PACK jobs travel in the launch's parameters (no load stands before
// a job's own operands); longer lists are read from the job table.
constexpr int ROW_PACK = 8;
template <class T>
struct RowPack {
  const RowJob<T>* jobs;
  const int* first;  // first block of every job, and the end
  int n;             // 0: in the table
  int total;         // jobs
  RowJob<T> j[ROW_PACK];
  int f[ROW_PACK + 1];
};
template <class T>
__device__ __forceinline__ int find_job(const RowPack<T>& p, int b, RowJob<T>& j) {
  if (p.n) {
    int i = 0;
    while (i + 1 < p.n && p.f[i + 1] <= b) ++i;
    j = p.j[i];
    return b - p.f[i];
  }
  const int i = find_group(p.first, p.total, b);
  j = p.jobs[i];
  return b - p.first[i];
}

// A block: TM = 8 RM rows x TN = 32 CN columns, 8 warps of RM rows each (a
// warp without valid rows skips the products, so short groups cost their own
// rows only), a lane CN neighbouring columns; K in chunks of 32 through shared
// memory.  On the FP64 pipe (2 multiply-adds per clock per SM) any tile is
// compute bound and small ones spread over more SMs; FP32 takes 64 x 128
// (8 x 4 accumulators per thread: 12 shared-memory words per 32 FMAs).
template <class T, int RM, int CN>
__global__ void __launch_bounds__(256) k_rows_gemm(const __grid_constant__ RowPack<T> pack) {
  constexpr int TM = 8 * RM, TN = 32 * CN, KC = 32;
  constexpr int LA = TM + (sizeof(T) == 4 ? 4 : 2), LB = TN + (sizeof(T) == 4 ? 4 : 2);
  __shared__ __align__(16) T As[KC * LA];
  __shared__ __align__(16) T Bs[KC * LB];
  __shared__ int arow[TM], item[TM], rex[TM];
  RowJob<T> j;
  const int b = find_job(pack, blockIdx.x, j);
  const int nbn = (j.N + TN - 1) / TN;
  const int n0 = (b % nbn) * TN, bm = b / nbn;
  int g, q0, nrows;
  if (j.rpg > 0) {
    const int tpg = (j.rpg + TM - 1) / TM;
    g = bm / tpg;
    const int r = (bm - g * tpg) * TM;
    q0 = g * j.rpg + r;
    nrows = min(TM, j.rpg - r);
    if (q0 >= j.rows) return;
  } else {
    if (bm >= j.tile_start[j.ngroups]) return;
    g = find_group(j.tile_start, j.ngroups, bm);
    const int r = (bm - j.tile_start[g]) * TM;
    q0 = j.grp_off[g] + r;
    nrows = min(TM, j.grp_cnt[g] - r);
    if (nrows <= 0) return;
  }
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < TM) {
    const int q = tid < nrows ? (j.perm ? j.perm[q0 + tid] : q0 + tid) : 0;
    item[tid] = q;
    arow[tid] = tid < nrows ? j.aidx(q) : 0;
    rex[tid] = 0;
  }
  __syncthreads();
  for (int r = warp; r < nrows; r += 8) {
    const T* row = j.A + (int64_t)arow[r] * j.K;
    typename Real<T>::t m = 0;
    for (int k = lane; k < j.K; k += 32) m = mag_max(m, row[k]);
    for (int o = 16; o; o >>= 1) m = mag_max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) rex[r] = exponent_of(m);
  }
  __syncthreads();
  const T* Bg = j.B + (int64_t)g * j.N * j.K;
  T acc[RM][CN];
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int c = 0; c < CN; ++c) acc[i][c] = Sc<T>::zero();
  const bool mine = warp * RM < nrows;
  for (int k0 = 0; k0 < j.K; k0 += KC) {
    const int kn = min(KC, j.K - k0);
#pragma unroll
    for (int it = 0; it < TM * KC / 256; ++it) {
      const int r = it * 8 + warp, k = lane;
      T v = Sc<T>::zero();
      if (r < nrows && k < kn) {
        v = j.A[(int64_t)arow[r] * j.K + k0 + k];
        if (rex[r]) v = scale_pow2(v, -rex[r]);
      }
      As[k * LA + r] = v;
    }
#pragma unroll
    for (int it = 0; it < TN * KC / 256; ++it) {
      const int n = it * 8 + warp, k = lane;
      T v = Sc<T>::zero();
      if (n0 + n < j.N && k < kn) v = Bg[(int64_t)(n0 + n) * j.K + k0 + k];
      Bs[k * LB + n] = v;
    }
    __syncthreads();
    if (mine) {
#pragma unroll 8
      for (int k = 0; k < KC; ++k) {
        if (k >= kn) break;
        T a[RM], x[CN];
#pragma unroll
        for (int i = 0; i < RM; ++i) a[i] = As[k * LA + warp * RM + i];
#pragma unroll
        for (int c = 0; c < CN; ++c) x[c] = Bs[k * LB + lane * CN + c];
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
          for (int c = 0; c < CN; ++c) acc[i][c] = Sc<T>::fma(a[i], x[c], acc[i][c]);
      }
    }
    __syncthreads();
  }
  if (mine) {
#pragma unroll
    for (int i = 0; i < RM; ++i) {
      const int r = warp * RM + i;
      if (r >= nrows) break;
      T* o = j.out + (int64_t)item[r] * j.N + n0;
#pragma unroll
      for (int c = 0; c < CN; ++c)
        if (n0 + lane * CN + c < j.N) o[lane * CN + c] = acc[i][c];
    }
  }
  if (n0 == 0 && tid < nrows && j.rex) j.rex[arow[tid]] = rex[tid];
  if (n0 == 0 && tid < nrows)
    j.out_exp[item[tid]] = rex[tid] + (j.Aexp ? j.Aexp[arow[tid]] : 0) + (j.gexp ? j.gexp[g] : 0);
}

// The same products for short rows (K <= 32): one thread per row and chunk of
// 4 columns, the row in registers and scaled there.  A tile of k_rows_gemm
// would leave most of its 32 column lanes idle below N = 32.
template <class T, int KM>
__device__ __forceinline__ void small_row(const RowJob<T>& j, unsigned it, unsigned nc) {
  const int q = nc == 1 ? (int)it : (int)(it / nc), n0 = (int)(it - (unsigned)q * nc) * 4;
  const int g = (int)((unsigned)q / (unsigned)j.rpg), ar = q - g * j.rpg;
  const T* A = j.A + (int64_t)ar * j.K;
  const T* B = j.B + ((int64_t)g * j.N + n0) * j.K;
  T a[KM];
  typename Real<T>::t m = 0;
#pragma unroll
  for (int k = 0; k < KM; ++k) a[k] = k < j.K ? A[k] : Sc<T>::zero();
  int ex = n0 == 0 ? (j.Aexp ? j.Aexp[ar] : 0) + (j.gexp ? j.gexp[g] : 0) : 0;
#pragma unroll
  for (int k = 0; k < KM; ++k) m = mag_max(m, a[k]);
  const int e = exponent_of(m);
  ex += e;
  if (e)
#pragma unroll
    for (int k = 0; k < KM; ++k) a[k] = scale_pow2(a[k], -e);
  T* o = j.out + (int64_t)q * j.N + n0;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    if (n0 + c >= j.N) break;
    T s = Sc<T>::zero();
#pragma unroll
    for (int k = 0; k < KM; ++k)
      if (k < j.K) s = Sc<T>::fma(a[k], B[c * j.K + k], s);
    o[c] = s;
  }
  if (n0 == 0) {
    j.out_exp[q] = ex;
    if (j.rex) j.rex[ar] = e;
  }
}
template <class T, int KM>
__global__ void __launch_bounds__(128) k_rows_small(const __grid_constant__ RowPack<T> pack) {
  RowJob<T> j;
  const int b = find_job(pack, blockIdx.x, j);
  const unsigned nc = (j.N + 3) / 4, it = (unsigned)b * 128 + threadIdx.x;
  if (it < (unsigned)j.rows * nc) small_row<T, KM>(j, it, nc);
}

// --------------------------------------------------- permuted tensors ----
constexpr int MOVE_MAXD = 20;
struct MoveJob {
  const void* src;
  void* dst;
  int64_t n;
  int nd;
  int dim[MOVE_MAXD];      // of dst
  int64_t str[MOVE_MAXD];  // strides of those axes in src
};
template <class T>
__device__ __forceinline__ void move_run(const MoveJob& j, int64_t i0, int64_t step) {
  const bool small = j.n < (int64_t(1) << 31);
  for (int64_t i = i0; i < j.n; i += step) {
    int64_t s = 0;
    if (small) {
      unsigned q = (unsigned)i;
      for (int d = j.nd - 1; d >= 0; --d) {
        const unsigned t = q / (unsigned)j.dim[d];
        s += (int64_t)(q - t * (unsigned)j.dim[d]) * j.str[d];
        q = t;
      }
    } else {
      int64_t q = i;
      for (int d = j.nd - 1; d >= 0; --d) {
        const int64_t t = q / j.dim[d];
        s += (q - t * j.dim[d]) * j.str[d];
        q = t;
      }
    }
    ((T*)j.dst)[i] = ((const T*)j.src)[s];
  }
}
template <class T>
__global__ void k_move(const MoveJob* __restrict__ jobs) {
  move_run<T>(jobs[blockIdx.y], blockIdx.x * (int64_t)blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x);
}

// ------------------------------------------------------------- centre ----
// One component of the forest: the two sides that meet at its centre edge
// (B null: a vertex centre, the value is the one entry of row A).
template <class T>
struct CentreSide {
  const T* ptr;
  const int* exps;  // null: zero
  RowIdx idx;
  int slot;   // >= 0: the row is this digit code of the point
  int scale;  // nonzero: scale the row by a power of two as it is read
};
template <class T>
struct CentreJob {
  CentreSide<T> a, b;
  int chi;
};

template <class T>
__device__ inline void write_out(void* out, int kind, int64_t p, int64_t P, T v, int e);
template <>
__device__ inline void write_out<double>(void* out, int kind, int64_t p, int64_t P, double v, int e) {
  if (kind == TNFA_OUT_F64) {
    ((double*)out)[p] = e ? scale_pow2(v, e) : v;
  } else if (kind == TNFA_OUT_F32) {
    ((float*)out)[p] = (float)scale_pow2(v, e);
  } else {  // scaled f32
    int ex = 0;
    double m = frexp(v, &ex);
    ((float*)out)[p] = (float)m;
    ((int*)((float*)out + P))[p] = (v == 0.0) ? 0 : e + ex;
  }
}
template <>
__device__ inline void write_out<float>(void* out, int kind, int64_t p, int64_t P, float v, int e) {
  write_out<double>(out, kind, p, P, (double)v, e);
}
template <>
__device__ inline void write_out<cplx>(void* out, int kind, int64_t p, int64_t P, cplx v, int e) {
  ((cplx*)out)[p] = scale_pow2(v, e);
}

__device__ __forceinline__ float shfl_x(float v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ double shfl_x(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ cplx shfl_x(cplx v, int o) {
  return {__shfl_xor_sync(0xffffffffu, v.re, o), __shfl_xor_sync(0xffffffffu, v.im, o)};
}

__device__ __forceinline__ float shfl_i(float v, int i) { return __shfl_sync(0xffffffffu, v, i); }
__device__ __forceinline__ double shfl_i(double v, int i) { return __shfl_sync(0xffffffffu, v, i); }
__device__ __forceinline__ cplx shfl_i(cplx v, int i) {
  return {__shfl_sync(0xffffffffu, v.re, i), __shfl_sync(0xffffffffu, v.im, i)};
}

// f(p) = prod over components of sum_c A[c] B[c].  The block digitizes its
// 256 points into shared memory (when the sides are codes), then G lanes per
// point take the dot products, VEC elements (16 bytes) per load, and the
// values go out through shared memory.  Bound by the row gathers (L2) and, for
// short rows, by HBM: 8 bytes per coordinate in, 8 out.
template <class T, int G, int VEC>
__global__ void __launch_bounds__(256) k_centre(const double* __restrict__ X, int ncols, int Pc,
                                                const DigitRun* __restrict__ runs, int nruns, int nslots,
                                                const CentreJob<T>* __restrict__ jobs, int njobs, void* out,
                                                int kind, int64_t P, int64_t p0, int* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char centre_sh[];
  T* val = (T*)centre_sh;                 // [256]
  int* vex = (int*)(val + 256);           // [256]
  int* codes = vex + 256;                 // [nslots][256]
  DigitRun* rs = (DigitRun*)(codes + nslots * 256);
  const int tid = threadIdx.x, l = tid % G, gi = tid / G;
  if (nslots > 0)
    for (int i = tid; i < nruns * (int)(sizeof(DigitRun) / 4); i += 256) ((int*)rs)[i] = ((const int*)runs)[i];
  for (int base = blockIdx.x * 256; base < Pc; base += gridDim.x * 256) {
    __syncthreads();
    if (nslots > 0) {
      for (int s = 0; s < nslots; ++s) codes[s * 256 + tid] = 0;
      if (base + tid < Pc)
        digit_codes(X + (int64_t)(base + tid) * ncols, rs, nruns, codes + tid, 256, 0, nslots, err);
      __syncthreads();
    }
#pragma unroll 1
    for (int t = gi; t < 256; t += 256 / G) {
      const int p = min(base + t, Pc - 1);  // the padding points repeat the last one
      T v = Sc<T>::one();
      int e = 0;
      for (int c = 0; c < njobs; ++c) {
        const CentreJob<T>& j = jobs[c];
        const int ra = j.a.slot >= 0 ? codes[j.a.slot * 256 + t] : j.a.idx(p);
        const T* A = j.a.ptr + (int64_t)ra * j.chi;
        e += j.a.exps ? j.a.exps[ra] : 0;
        T s = Sc<T>::zero();
        if (!j.b.ptr) {
          s = A[0];
        } else {
          const int rb = j.b.slot >= 0 ? codes[j.b.slot * 256 + t] : j.b.idx(p);
          const T* B = j.b.ptr + (int64_t)rb * j.chi;
          e += j.b.exps ? j.b.exps[rb] : 0;
          int ea = 0, eb = 0;
          if (j.a.scale | j.b.scale) {
            typename Real<T>::t ma = 0, mb = 0;
            for (int k = l; k < j.chi; k += G) {
              ma = mag_max(ma, A[k]);
              mb = mag_max(mb, B[k]);
            }
#pragma unroll
            for (int o = G / 2; o; o >>= 1) {
              ma = mag_max(ma, __shfl_xor_sync(0xffffffffu, ma, o));
              mb = mag_max(mb, __shfl_xor_sync(0xffffffffu, mb, o));
            }
            ea = exponent_of(ma);
            eb = exponent_of(mb);
            e += ea + eb;
          }
          if constexpr (VEC > 1) {
            for (int k = l * VEC; k < j.chi; k += G * VEC) {
              const int4 xa = *reinterpret_cast<const int4*>(A + k), xb = *reinterpret_cast<const int4*>(B + k);
              const T* pa = reinterpret_cast<const T*>(&xa);
              const T* pb = reinterpret_cast<const T*>(&xb);
#pragma unroll
              for (int i = 0; i < VEC; ++i) {
                const T x = ea ? scale_pow2(pa[i], -ea) : pa[i], y = eb ? scale_pow2(pb[i], -eb) : pb[i];
                s = Sc<T>::fma(x, y, s);
              }
            }
          } else {
            for (int k = l; k < j.chi; k += G) {
              const T x = ea ? scale_pow2(A[k], -ea) : A[k], y = eb ? scale_pow2(B[k], -eb) : B[k];
              s = Sc<T>::fma(x, y, s);
            }
          }
#pragma unroll
          for (int o = G / 2; o; o >>= 1) s = s + shfl_x(s, o);
        }
        v = c == 0 ? s : v * s;
      }
      if (l == 0) {
        val[t] = v;
        vex[t] = e;
      }
    }
    __syncthreads();
    if (base + tid < Pc) write_out<T>(out, kind, p0 + base + tid, P, val[tid], vex[tid]);
  }
}

__device__ __forceinline__ void copy_async16(void* d, const void* s) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(d)), "l"(s));
}
__device__ __forceinline__ void copy_async4(void* d, const void* s) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(d)), "l"(s));
}

// bytes (a multiple of 4) of global memory to shared memory, by the whole block
__device__ __forceinline__ void copy_async_block(void* d, const void* s, int bytes) {
  const int n16 = (((uintptr_t)s | (uintptr_t)d) & 15) == 0 ? bytes / 16 : 0;
  for (int i = threadIdx.x; i < n16; i += blockDim.x) copy_async16((char*)d + 16 * i, (const char*)s + 16 * i);
  for (int i = n16 * 4 + threadIdx.x; i < bytes / 4; i += blockDim.x)
    copy_async4((char*)d + 4 * i, (const char*)s + 4 * i);
}

// The common case of k_centre -- one component, both sides tables, few digit
// runs -- with everything but the rows in kernel parameters and registers: a
// thread digitizes its point, then G lanes take each of the warp's points in
// turn.  k_centre spent 350 instructions per point on job records, digit runs
// and codes in memory.  At bond 2 the FP64 pipe (2 multiply-adds per point at
// 2 per clock per SM) and HBM (16 bytes per point) are about even.
constexpr int CENTRE_RUNS = 12;
template <class T>
struct PairParams {
  const double* X;
  void* out;
  int* err;
  int64_t P, p0;
  const T *A, *B;
  const int *ea, *eb;  // null: zero
  const int *pa, *pb;  // set on the device: the exponent of all rows of the side, INT_MIN if they differ (null: not known)
  int na, nb;          // rows
  int ncols, Pc, nruns, chi, sa, sb, kind, scale;  // sa, sb: code slots; scale: rows of a leaf tensor
  DigitRun runs[CENTRE_RUNS];
};
// SM: both tables are copied to shared memory first.  A gather of 32 different
// rows costs a cache line per lane in L1 (32 cycles), a few bank conflicts
// there.
// FEW: at most two runs, both bit fields (a side's digits are one block of a
// variable's): their fields stay in registers and the next point's coordinates
// are on their way while this one's rows are summed.  With the loop over run
// records, and each thread waiting for its coordinate, 10^7 points at bond 2
// took 104 us of k_centre_pair (256 instructions a point), now 63 (180), of
// which the two multiply-adds a point are 34.
template <class T, int G, int VEC, bool SM, bool FEW>
__global__ void __launch_bounds__(256) k_centre_pair(const __grid_constant__ PairParams<T> W) {
  extern __shared__ __align__(16) unsigned char pair_sh[];
  const int lane = threadIdx.x & 31, l = lane % G;
  const T* tabA = W.A;
  const T* tabB = W.B;
  if constexpr (SM) {
    const int na = W.na * W.chi, nb = W.nb * W.chi;
    T* sa = (T*)pair_sh;
    T* sb = sa + (na + VEC - 1) / VEC * VEC;
    copy_async_block(sa, W.A, na * (int)sizeof(T));
    copy_async_block(sb, W.B, nb * (int)sizeof(T));
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    tabA = sa;
    tabB = sb;
  }
  const int ca = W.ea && W.pa ? *W.pa : INT_MIN, cb = W.eb && W.pb ? *W.pb : INT_MIN;
  const int* xa_ = ca == INT_MIN ? W.ea : nullptr;
  const int* xb_ = cb == INT_MIN ? W.eb : nullptr;
  const int e0 = (ca == INT_MIN ? 0 : ca) + (cb == INT_MIN ? 0 : cb);
  constexpr int PG = 32 / G;  // points per pass
  // (unsigned: below 2^31 points, and a grid's step more stays below 2^32)
  const unsigned Pc = (unsigned)W.Pc, step = gridDim.x * blockDim.x;
  const unsigned base0 = blockIdx.x * blockDim.x + threadIdx.x - lane;
  const bool two = W.nruns > 1, own = two && W.runs[1].start;  // the second run's column is its own
  const int f0 = W.runs[0].first - 1, n0 = 32 - W.runs[0].n, w0 = W.runs[0].w, r0 = W.runs[0].rev;
  const int f1 = two ? W.runs[1].first - 1 : 0, n1 = two ? 32 - W.runs[1].n : 0, w1 = two ? W.runs[1].w : 0;
  const int r1 = two ? W.runs[1].rev : 0;
  const bool a0 = W.runs[0].slot == W.sa, a1 = two && W.runs[1].slot == W.sa;
  double x0 = 0.0, x1 = 0.0;
  auto fetch = [&](unsigned b) {
    const double* Xp = W.X + (int64_t)min(Pc - 1, b + lane) * W.ncols;  // the padding lanes repeat the last point
    x0 = Xp[W.runs[0].col];
    if (own) x1 = Xp[W.runs[1].col];
  };
  auto in_domain = [&](double& x) {
    const unsigned long long xb = (unsigned long long)__double_as_longlong(x);
    if (xb > 0x8000000000000000ull || (xb & 0x7FF0000000000000ull) == 0x7FF0000000000000ull) {
      raise_domain(W.err);
      x = 0.0;
    }
  };
  if (FEW && base0 < Pc) fetch(base0);
  for (unsigned base = base0; base < Pc; base += step) {
    const int p = (int)min(Pc - 1, base + lane);
    int c[2] = {0, 0};
    if constexpr (FEW) {
      double xa = x0, xb = x1;
      if (base + step < Pc) fetch(base + step);
      in_domain(xa);
      const unsigned long long u = unit_fraction(xa);
      unsigned long long v = u;
      if (own) {
        in_domain(xb);
        v = unit_fraction(xb);
      }
      const unsigned g0 = (unsigned)((u << f0) >> 32), g1 = (unsigned)((v << f1) >> 32);
      const int c0 = (int)(r0 ? __brev(g0) & (0xFFFFFFFFu >> n0) : g0 >> n0) * w0;
      const int c1 = (int)(r1 ? __brev(g1) & (0xFFFFFFFFu >> n1) : g1 >> n1) * w1;
      c[0] = (a0 ? c0 : 0) + (a1 ? c1 : 0);
      c[1] = (a0 ? 0 : c0) + (a1 ? 0 : c1);
    } else {
      double xr = 0.0;
      unsigned long long u = 0;
      for (int e = 0; e < W.nruns; ++e) {
        const DigitRun& d = W.runs[e];
        if (d.start) {
          xr = W.X[(int64_t)p * W.ncols + d.col];
          const unsigned long long xb = (unsigned long long)__double_as_longlong(xr);
          if (xb > 0x8000000000000000ull || (xb & 0x7FF0000000000000ull) == 0x7FF0000000000000ull) {
            raise_domain(W.err);
            xr = 0.0;
          }
          u = unit_fraction(xr);
        }
        int add;
        if (d.bits) {
          const unsigned f = (unsigned)((u << (d.first - 1)) >> 32);
          add = (int)(d.rev ? __brev(f) & (0xFFFFFFFFu >> (32 - d.n)) : f >> (32 - d.n)) * d.w;
        } else {
          int dig = 0;
          for (int v = d.base - 1; v >= 1; --v) {
            const double t = (double)v * d.invb;
            if (xr >= t) {
              dig = v;
              xr -= t;
              break;
            }
          }
          add = dig * d.w;
        }
        if (d.slot == W.sa) c[0] += add;
        else c[1] += add;
      }
    }
    T v = Sc<T>::zero();
    int ve = 0;
#pragma unroll
    for (int i = 0; i < G; ++i) {
      const int t = i * PG + lane / G;  // the point of this pass
      const int ra = G == 1 ? c[0] : __shfl_sync(0xffffffffu, c[0], t);
      const int rb = G == 1 ? c[1] : __shfl_sync(0xffffffffu, c[1], t);
      const T* A = SM ? tabA + ra * W.chi : tabA + (int64_t)ra * W.chi;
      const T* B = SM ? tabB + rb * W.chi : tabB + (int64_t)rb * W.chi;
      int e = e0 + (xa_ ? xa_[ra] : 0) + (xb_ ? xb_[rb] : 0), ea = 0, eb = 0;
      if (W.scale) {
        typename Real<T>::t ma = 0, mb = 0;
        for (int k = l; k < W.chi; k += G) {
          ma = mag_max(ma, A[k]);
          mb = mag_max(mb, B[k]);
        }
#pragma unroll
        for (int o = G / 2; o; o >>= 1) {
          ma = mag_max(ma, __shfl_xor_sync(0xffffffffu, ma, o));
          mb = mag_max(mb, __shfl_xor_sync(0xffffffffu, mb, o));
        }
        ea = exponent_of(ma);
        eb = exponent_of(mb);
        e += ea + eb;
      }
      T s = Sc<T>::zero();
      auto dot = [&](auto scaled) {
        for (int k = l * VEC; k < W.chi; k += G * VEC) {
          T xa[VEC], xb[VEC];
          if constexpr (VEC > 1) {
            *reinterpret_cast<int4*>(xa) = *reinterpret_cast<const int4*>(A + k);
            *reinterpret_cast<int4*>(xb) = *reinterpret_cast<const int4*>(B + k);
          } else {
            xa[0] = A[k];
            xb[0] = B[k];
          }
#pragma unroll
          for (int q = 0; q < VEC; ++q) {
            if constexpr (decltype(scaled)::value)
              s = Sc<T>::fma(ea ? scale_pow2(xa[q], -ea) : xa[q], eb ? scale_pow2(xb[q], -eb) : xb[q], s);
            else
              s = Sc<T>::fma(xa[q], xb[q], s);
          }
        }
      };
      if (W.scale) dot(std::true_type{});
      else dot(std::false_type{});
#pragma unroll
      for (int o = G / 2; o; o >>= 1) s = s + shfl_x(s, o);
      // hand the sum to the point's own lane
      if constexpr (G == 1) {
        v = s;
        ve = e;
      } else {
        const int src = ((lane - i * PG) * G) & 31;
        const T sv = shfl_i(s, src);
        const int se = __shfl_sync(0xffffffffu, e, src);
        if (lane / PG == i) {
          v = sv;
          ve = se;
        }
      }
    }
    if (base + lane < Pc) write_out<T>(W.out, W.kind, W.p0 + base + lane, W.P, v, ve);
  }
}

// --------------------------------------------------- small-bond walk ----
// Small bonds: a thread takes its point through every vertex that has no table
// in one launch, and no message goes through HBM.  The two sides of the centre
// are walked by two threads (half the chain each).  The schedule and, up to 64
// KB, the network's tensors are copied to shared memory asynchronously while
// the points are digitized; the tensors are read through strides, so no vertex
// needs a copy in another axis order.  Up to bond 8 the message of a step stays
// in registers for the next one when that reads it (a path never stores one);
// otherwise messages are in shared memory, [slot][entry][point].  For a few
// thousand points G lanes share a point: each makes CHI / G rows of a step and
// the message is put together by shuffles, because one warp's FP64 multiply-add
// takes 64 cycles of its scheduler and a chain of them on few warps leaves the
// other schedulers idle.
template <class T>
struct WalkStep {
  const T* B;       // tensor slices (vertex tensor, or one with an absorbed table)
  const int* gexp;  // exponent of a slice, null: zero
  const T* t1;      // first child's table, null: its message slot
  const T* t2;      // last child's
  const int* e1;    // the tables' exponents, null: zero
  const int* e2;
  int stage;        // element offset of B in the staged network tensors, -1: read in place
  int key;          // code slot of the slice, -1: slice 0
  int chi_a;
  int d1, d2;       // first and last child's bonds (1 when absent)
  int c1, c2;       // code slot (table) or message slot of the children; -1: none, -2: the previous step's registers
  int sg, sa, s1, s2;  // strides of slice, row, first and last child in B
  int out;          // message slot, -1: stays in registers
};
template <class T>
struct WalkSide {
  const T* tab;  // null: message slot `at`
  const int* exps;
  int at;        // code slot or message slot
  int chi;       // 0: absent (a vertex centre)
};
template <class T>
struct WalkParams {
  const double* X;
  const unsigned char* blob;  // runs, steps (side 0's, then side 1's), sides (two per component)
  const T* tensors;
  void* out;
  int* err;
  int64_t P, p0;
  int ncols, Pc, nruns, nslots, nsteps0, nsteps, ncomp, nmsg, nstage, kind;
};

template <class T>
__host__ __device__ inline size_t walk_blob(int nruns, int nsteps, int ncomp) {
  return (nruns * sizeof(DigitRun) + nsteps * sizeof(WalkStep<T>) + 2 * ncomp * sizeof(WalkSide<T>) + 15) / 16 * 16;
}
template <class T>
__host__ __device__ inline size_t walk_smem(int chi, int tp, int nstage, int nmsg, int nslots, int nruns, int nsteps,
                                            int ncomp) {
  return walk_blob<T>(nruns, nsteps, ncomp) + ((size_t)nstage * sizeof(T) + 15) / 16 * 16 +
         (size_t)nmsg * chi * tp * sizeof(T) + (size_t)(2 + nslots) * tp * 4;
}

template <class T, int CHI, int G>
__global__ void __launch_bounds__(256) k_walk(const __grid_constant__ WalkParams<T> W) {
  constexpr bool REG = CHI <= 8;  // the message also in registers (unrolled rows)
  constexpr int RL = CHI / G;     // rows per lane
  static_assert(REG || G == 1, "lanes share a point only with the message in registers");
  extern __shared__ __align__(16) unsigned char walk_sh[];
  const int tl = blockDim.x >> 1, tp = tl / G;  // threads and points per side
  const int side = threadIdx.x >= tl, t = (threadIdx.x - side * tl) / G, gl = threadIdx.x % G;
  const DigitRun* runs = (const DigitRun*)walk_sh;
  const WalkStep<T>* st = (const WalkStep<T>*)(runs + W.nruns);
  const WalkSide<T>* sd = (const WalkSide<T>*)(st + W.nsteps);
  const size_t nblob = walk_blob<T>(W.nruns, W.nsteps, W.ncomp);
  T* ten = (T*)(walk_sh + nblob);
  T* msg = (T*)(walk_sh + nblob + ((size_t)W.nstage * sizeof(T) + 15) / 16 * 16);
  int* sex = (int*)(msg + (size_t)W.nmsg * CHI * tp);  // [2][tp] exponents of the sides
  int* codes = sex + 2 * tp;                           // [nslots][tp]
  copy_async_block(walk_sh, W.blob, (int)nblob);
  asm volatile("cp.async.commit_group;" ::: "memory");
  copy_async_block(ten, W.tensors, W.nstage * (int)sizeof(T));
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 1;" ::: "memory");
  __syncthreads();
  auto M = [&](int slot, int k) -> T& { return msg[((size_t)slot * CHI + k) * tp + t]; };
  for (int base = blockIdx.x * tp; base < W.Pc; base += gridDim.x * tp) {
    const int p = base + t;
    if (side == 0 && gl == 0) {
      for (int s = 0; s < W.nslots; ++s) codes[s * tp + t] = 0;
      if (p < W.Pc) digit_codes(W.X + (int64_t)p * W.ncols, runs, W.nruns, codes + t, tp, 0, W.nslots, W.err);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    int ex_acc = 0;
    T cur[REG ? CHI : 1];
    const int i1 = side ? W.nsteps : W.nsteps0;
    for (int i = side ? W.nsteps0 : 0; i < i1; ++i) {
      const WalkStep<T>& s = st[i];
      const int g = s.key >= 0 ? codes[s.key * tp + t] : 0;
      const int d1 = s.d1, d2 = s.d2, chi_a = s.chi_a, sa = s.sa, s1 = s.s1, s2 = s.s2, c1 = s.c1, c2 = s.c2;
      const T* B = (s.stage >= 0 ? ten + s.stage : s.B) + (int64_t)g * s.sg;
      if (s.gexp) ex_acc += s.gexp[g];
      // the last child's row in registers; a table's row is scaled here, a
      // message was when it was made
      T ml[CHI];
      if (REG && c2 == -2) {
#pragma unroll
        for (int c = 0; c < CHI; ++c) ml[c] = cur[REG ? c : 0];
      } else if (s.t2) {
        const int r = codes[c2 * tp + t];
        const T* row = s.t2 + (int64_t)r * d2;
        typename Real<T>::t m = 0;
#pragma unroll
        for (int c = 0; c < CHI; ++c) {
          ml[c] = c < d2 ? row[c] : Sc<T>::zero();
          m = mag_max(m, ml[c]);
        }
        const int e = exponent_of(m);
        ex_acc += e + (s.e2 ? s.e2[r] : 0);
        if (e)
#pragma unroll
          for (int c = 0; c < CHI; ++c) ml[c] = scale_pow2(ml[c], -e);
      } else {
#pragma unroll
        for (int c = 0; c < CHI; ++c) ml[c] = c < d2 ? M(c2, c) : Sc<T>::zero();
      }
      const T* row1 = nullptr;
      int e1 = 0;
      if (s.t1) {
        const int r = codes[c1 * tp + t];
        row1 = s.t1 + (int64_t)r * d1;
        typename Real<T>::t m = 0;
        for (int b = 0; b < d1; ++b) m = mag_max(m, row1[b]);
        e1 = exponent_of(m);
        ex_acc += e1 + (s.e1 ? s.e1[r] : 0);
      }
      auto row = [&](int a) {
        const T* Ba = B + a * sa;
        T acc = Sc<T>::zero();
        if (c1 == -1) {
#pragma unroll
          for (int c = 0; c < CHI; ++c)
            if (c < d2) acc = Sc<T>::fma(Ba[c * s2], ml[c], acc);
        } else {
          for (int b = 0; b < d1; ++b) {
            T in = Sc<T>::zero();
#pragma unroll
            for (int c = 0; c < CHI; ++c)
              if (c < d2) in = Sc<T>::fma(Ba[b * s1 + c * s2], ml[c], in);
            const T x = row1 ? scale_pow2(row1[b], -e1) : M(c1, b);
            acc = Sc<T>::fma(x, in, acc);
          }
        }
        return acc;
      };
      typename Real<T>::t mx = 0;
      if constexpr (REG) {
        T mine[RL];
#pragma unroll
        for (int a = 0; a < RL; ++a) mine[a] = a * G + gl < chi_a ? row(a * G + gl) : Sc<T>::zero();
#pragma unroll
        for (int a = 0; a < CHI; ++a) {
          cur[a] = G == 1 ? mine[a / G] : shfl_i(mine[a / G], (threadIdx.x & 31) - gl + a % G);
          mx = mag_max(mx, cur[a]);
        }
        const int ex = exponent_of(mx);
        if (ex) {
          ex_acc += ex;
#pragma unroll
          for (int a = 0; a < CHI; ++a) cur[a] = scale_pow2(cur[a], -ex);
        }
        if (s.out >= 0) {
          if (gl == 0)
#pragma unroll
            for (int a = 0; a < CHI; ++a)
              if (a < chi_a) M(s.out, a) = cur[a];
          if (G > 1) __syncwarp();
        }
      } else {
        for (int a = 0; a < chi_a; ++a) {
          const T x = row(a);
          M(s.out, a) = x;
          mx = mag_max(mx, x);
        }
        const int ex = exponent_of(mx);
        ex_acc += ex;
        if (ex)
          for (int a = 0; a < chi_a; ++a) M(s.out, a) = scale_pow2(M(s.out, a), -ex);
      }
    }
    if (gl == 0) sex[side * tp + t] = ex_acc;
    __syncthreads();
    if (side == 0 && gl == 0 && p < W.Pc) {
      T v = Sc<T>::one();
      int e = sex[t] + sex[tp + t];
      for (int c = 0; c < W.ncomp; ++c) {
        const WalkSide<T>&A = sd[2 * c], &B = sd[2 * c + 1];
        const T* ra = nullptr;
        const T* rb = nullptr;
        if (A.tab) {
          const int r = codes[A.at * tp + t];
          ra = A.tab + (int64_t)r * A.chi;
          e += A.exps ? A.exps[r] : 0;
        }
        if (B.tab) {
          const int r = codes[B.at * tp + t];
          rb = B.tab + (int64_t)r * B.chi;
          e += B.exps ? B.exps[r] : 0;
        }
        T s = Sc<T>::zero();
        if (B.chi == 0) {
          s = ra ? ra[0] : M(A.at, 0);
        } else {
          typename Real<T>::t ma = 0, mb = 0;
          if (ra)
            for (int k = 0; k < A.chi; ++k) ma = mag_max(ma, ra[k]);
          if (rb)
            for (int k = 0; k < A.chi; ++k) mb = mag_max(mb, rb[k]);
          const int ea = exponent_of(ma), eb = exponent_of(mb);
          e += ea + eb;
          for (int k = 0; k < A.chi; ++k) {
            const T x = ra ? scale_pow2(ra[k], -ea) : M(A.at, k), y = rb ? scale_pow2(rb[k], -eb) : M(B.at, k);
            s = Sc<T>::fma(x, y, s);
          }
        }
        v = c == 0 ? s : v * s;
      }
      write_out<T>(W.out, W.kind, W.p0 + p, W.P, v, e);
    }
    __syncthreads();
  }
}

// Rows of a table scaled to a largest entry in [1/2, 1), the exponents kept.
template <class T>
struct NormJob {
  T* tab;
  int* exps;
  int rows, chi;
};
// (8 lanes per row; per: rows in flight, r0: the caller's row of the first pass)
template <class T>
__device__ __forceinline__ void norm_run(const NormJob<T>& j, int r0, int per) {
  const int l = threadIdx.x & 7;
  const int n = (j.rows + per - 1) / per;
  for (int i = 0; i < n; ++i) {
    const int r = i * per + r0;
    const bool ok = r < j.rows;
    T* row = j.tab + (int64_t)(ok ? r : 0) * j.chi;
    typename Real<T>::t m = 0;
    if (ok)
      for (int k = l; k < j.chi; k += 8) m = mag_max(m, row[k]);
    for (int o = 4; o; o >>= 1) m = mag_max(m, __shfl_xor_sync(0xffffffffu, m, o));
    const int ex = exponent_of(m);
    if (!ok || !ex) continue;
    for (int k = l; k < j.chi; k += 8) row[k] = scale_pow2(row[k], -ex);
    if (l == 0) j.exps[r] += ex;
  }
}
template <class T>
__global__ void k_norm_rows(const NormJob<T>* __restrict__ jobs) {
  norm_run<T>(jobs[blockIdx.y], (blockIdx.x * blockDim.x + threadIdx.x) / 8, gridDim.x * (blockDim.x >> 3));
}

// The first levels of the tables, where a launch costs more than its work: one
// block takes everything below one vertex in shared memory.  The tensors are
// copied there in one go (read through strides, so none needs its axes
// permuted), level follows level behind a block barrier, and only the top
// table goes out.  Each level would be a launch otherwise, and from global
// memory every one of them costs two or three L2 latencies (4 us, measured).
// A side of the centre leaves with its rows scaled; if the rows' exponents lie
// within range of their least, the powers of two above that one join the
// entries and *plain receives it (else INT_MIN): the centre then reads no
// exponent per point.  Entries only grow by it, so none becomes subnormal that
// was not, and their products stay below the type's limit.
struct HeadJob {
  int A, Aexp;    // rows: element offset, exponents' offset (-1: zero)
  int lda;        // row pitch
  int B, gexp;    // tensor slices, their exponents' offset (-1: zero)
  int out, oexp, ldo;
  int K, N, rows, rpg;
  int bg, n2, bn1, bn2, bk;  // B strides; column n = (n / n2, n % n2)
  int level;
};
template <class T>
struct HeadCopy {
  const T* src;
  int dst, n;
};
template <class T>
struct HeadBlock {
  T* tab;       // the top table in global memory
  int* exps;
  int copy0, copy1, job0, job1;
  int top, topexp, ld, rows, chi;  // the top table in shared memory
  int centre;   // a side of the centre: rows are scaled
  int plain;    // index of its word
};
template <class T, int KM>
__device__ __forceinline__ void head_item(const HeadJob& j, T* sh, int* ex, int q, int n0) {
  const int g = (int)((unsigned)q / (unsigned)j.rpg), ar = q - g * j.rpg;
  const T* A = sh + j.A + ar * j.lda;
  T a[KM];
  typename Real<T>::t m = 0;
#pragma unroll
  for (int k = 0; k < KM; ++k) {
    a[k] = k < j.K ? A[k] : Sc<T>::zero();
    m = mag_max(m, a[k]);
  }
  const int e = exponent_of(m);
  if (e)
#pragma unroll
    for (int k = 0; k < KM; ++k) a[k] = scale_pow2(a[k], -e);
  T* o = sh + j.out + q * j.ldo + n0;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int n = n0 + c;
    if (n >= j.N) break;
    const int n1 = j.n2 == j.N ? 0 : n / j.n2;
    const T* B = sh + j.B + g * j.bg + n1 * j.bn1 + (n - n1 * j.n2) * j.bn2;
    T s = Sc<T>::zero();
#pragma unroll
    for (int k = 0; k < KM; ++k)
      if (k < j.K) s = Sc<T>::fma(a[k], B[k * j.bk], s);
    o[c] = s;
  }
  if (n0 == 0) ex[j.oexp + q] = e + (j.Aexp >= 0 ? ex[j.Aexp + ar] : 0) + (j.gexp >= 0 ? ex[j.gexp + g] : 0);
}
template <class T, int KM>
__global__ void __launch_bounds__(256) k_head(const HeadBlock<T>* __restrict__ blocks,
                                              const HeadCopy<T>* __restrict__ copies,
                                              const HeadJob* __restrict__ gjobs, int nelem, int nexp, int njobs,
                                              int* __restrict__ plain, int range) {
  extern __shared__ __align__(16) unsigned char head_sh[];
  __shared__ int red[2];
  T* sh = (T*)head_sh;
  int* ex = (int*)(sh + nelem);
  HeadJob* jobs = (HeadJob*)(ex + nexp);
  const HeadBlock<T> h = blocks[blockIdx.x];
  const int nj = h.job1 - h.job0;
  const int lane = threadIdx.x & 31;
  for (int i = h.copy0 + (threadIdx.x >> 5); i < h.copy1; i += blockDim.x >> 5) {
    const HeadCopy<T> c = copies[i];
    for (int k = lane; k < c.n * (int)(sizeof(T) / 4); k += 32)
      copy_async4((int*)(sh + c.dst) + k, (const int*)c.src + k);
  }
  for (int i = threadIdx.x; i < nj * (int)(sizeof(HeadJob) / 4); i += blockDim.x)
    copy_async4((int*)jobs + i, (const int*)(gjobs + h.job0) + i);
  if (threadIdx.x == 0) red[0] = INT_MAX, red[1] = INT_MIN;
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  for (int i = 0; i < nj; ++i) {
    const HeadJob& j = jobs[i];
    if (i > 0 && j.level != jobs[i - 1].level) __syncthreads();
    // rows fastest: a warp's lanes read one column of B and rows a pitch apart
    const unsigned rows = j.rows, n = rows * ((j.N + 3) / 4);
    for (unsigned it = threadIdx.x; it < n; it += blockDim.x) {
      const unsigned c = it / rows;
      head_item<T, KM>(j, sh, ex, (int)(it - c * rows), (int)c * 4);
    }
  }
  __syncthreads();
  int shift = 0, least = 0;  // plain: the exponents above the least go into the entries
  if (h.centre) {
    int lo = INT_MAX, hi = INT_MIN;  // of the rows that are not zero
    for (int r = threadIdx.x; r < h.rows; r += blockDim.x) {
      T* row = sh + h.top + r * h.ld;
      typename Real<T>::t m = 0;
      for (int k = 0; k < h.chi; ++k) m = mag_max(m, row[k]);
      const int e = exponent_of(m);
      if (e)
        for (int k = 0; k < h.chi; ++k) row[k] = scale_pow2(row[k], -e);
      const int t = ex[h.topexp + r] += e;
      if (m != 0) lo = min(lo, t), hi = max(hi, t);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lane == 0) {
      atomicMin(&red[0], lo);
      atomicMax(&red[1], hi);
    }
    __syncthreads();
    least = red[0];
    shift = least <= red[1] && red[1] - least <= range;
    if (threadIdx.x == 0) plain[h.plain] = shift ? least : INT_MIN;
  }
  for (int i = threadIdx.x; i < h.rows * h.chi; i += blockDim.x) {
    const int r = i / h.chi;
    const T v = sh[h.top + r * h.ld + (i - r * h.chi)];
    h.tab[i] = shift ? scale_pow2(v, ex[h.topexp + r] - least) : v;
  }
  for (int r = threadIdx.x; r < h.rows; r += blockDim.x) h.exps[r] = shift ? least : ex[h.topexp + r];
}

}  // namespace tnfa

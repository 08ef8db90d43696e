// Device code of the row-gather contractions of batched evaluation: digit
// codes, the one-child contraction over gathered rows, permuted tensor
// copies, and the dot product at the centre.
#pragma once
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

// Adds every run to codes[slot * ld] for the slots [s0, s1).
__device__ __forceinline__ void digit_codes(const double* __restrict__ Xp, const DigitRun* runs, int nruns,
                                            int* codes, int ld, int s0, int s1, int* err) {
  double xr = 0.0;
  unsigned long long u = 0;
  for (int e = 0; e < nruns; ++e) {
    const DigitRun d = runs[e];
    if (d.start) {
      xr = Xp[d.col];
      const unsigned hi = (unsigned)((unsigned long long)__double_as_longlong(xr) >> 32);
      const bool neg = (hi >> 31) && xr != 0.0;
      if (neg || (hi & 0x7FF00000u) == 0x7FF00000u) {  // negative, infinite or NaN
        atomicOr(err, 1);
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
  int K, N, rows;
  int rpg;  // > 0: uniform groups
  const int* perm;  // null: identity
  const int* grp_off;
  const int* grp_cnt;
  const int* tile_start;
  int ngroups;
};

// A block: TM = 8 RM rows x TN = 32 CN columns, 8 warps of RM rows each (a
// warp without valid rows skips the products, so short groups cost their own
// rows only), a lane CN neighbouring columns; K in chunks of 32 through shared
// memory.  On the FP64 pipe (2 multiply-adds per clock per SM) any tile is
// compute bound and small ones spread over more SMs; FP32 takes 64 x 128
// (8 x 4 accumulators per thread: 12 shared-memory words per 32 FMAs).
template <class T, int RM, int CN>
__global__ void __launch_bounds__(256) k_rows_gemm(const RowJob<T> one, const RowJob<T>* __restrict__ jobs,
                                                   const int* __restrict__ first, int njobs) {
  constexpr int TM = 8 * RM, TN = 32 * CN, KC = 32;
  constexpr int LA = TM + (sizeof(T) == 4 ? 4 : 2), LB = TN + (sizeof(T) == 4 ? 4 : 2);
  __shared__ __align__(16) T As[KC * LA];
  __shared__ __align__(16) T Bs[KC * LB];
  __shared__ int arow[TM], item[TM], rex[TM];
  int b = blockIdx.x;
  RowJob<T> j = one;
  if (njobs > 0) {
    const int i = find_group(first, njobs, b);
    j = jobs[i];
    b -= first[i];
  }
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
  if (n0 == 0 && tid < nrows)
    j.out_exp[item[tid]] = rex[tid] + (j.Aexp ? j.Aexp[arow[tid]] : 0) + (j.gexp ? j.gexp[g] : 0);
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
__global__ void k_move(const MoveJob* __restrict__ jobs) {
  const MoveJob& j = jobs[blockIdx.y];
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < j.n; i += (int64_t)gridDim.x * blockDim.x) {
    int64_t q = i, s = 0;
    for (int d = j.nd - 1; d >= 0; --d) {
      const int64_t t = q / j.dim[d];
      s += (q - t * j.dim[d]) * j.str[d];
      q = t;
    }
    ((T*)j.dst)[i] = ((const T*)j.src)[s];
  }
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
    ((double*)out)[p] = scale_pow2(v, e);
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

// Rows of a table scaled to a largest entry in [1/2, 1), the exponents kept.
template <class T>
struct NormJob {
  T* tab;
  int* exps;
  int rows, chi;
};
template <class T>
__global__ void k_norm_rows(const NormJob<T>* __restrict__ jobs) {
  const NormJob<T> j = jobs[blockIdx.y];
  // 8 lanes per row
  const int l = threadIdx.x & 7;
  const int per = gridDim.x * (blockDim.x >> 3);
  const int n = (j.rows + per - 1) / per;
  for (int i = 0; i < n; ++i) {
    const int r = i * per + (blockIdx.x * blockDim.x + threadIdx.x) / 8;
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

}  // namespace tnfa

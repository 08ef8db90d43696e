// Device code of the vector-Jacobian product of batched evaluation: weights of
// the points, sums of point adjoints into table rows, and the adjoints of the
// row products that built the tables.
#pragma once
#include "rows.cuh"

namespace tnfa {

template <class T>
__device__ inline void atomic_add_T(T* a, T v);
template <>
__device__ inline void atomic_add_T<double>(double* a, double v) { atomicAdd(a, v); }
template <>
__device__ inline void atomic_add_T<float>(float* a, float v) { atomicAdd(a, v); }
template <>
__device__ inline void atomic_add_T<cplx>(cplx* a, cplx v) {
  atomicAdd(&a->re, v.re);
  atomicAdd(&a->im, v.im);
}
template <class T>
__device__ inline T from_real(double x) { return (T)x; }
template <>
__device__ inline cplx from_real<cplx>(double x) { return {x, 0.0}; }

// The common power of two of one chunk's weights (no point had one: 0).
__device__ __forceinline__ int common_exp(const int* S) { return *S < -(1 << 30) ? 0 : *S; }

// Per point and component: dout times the values of the other components
// (wv, with exponent we), and the largest exponent of any point's weight.
template <class T>
__global__ void k_adj_prep(const double* __restrict__ dout, int Pc, const CentreJob<T>* __restrict__ jobs, int ncomp,
                           T* __restrict__ wv, int* __restrict__ we, int64_t ld, int* __restrict__ S) {
  int top = INT_MIN;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < Pc; p += gridDim.x * blockDim.x) {
    const T d = from_real<T>(dout[p]);
    if (ncomp > 1)
      for (int c = 0; c < ncomp; ++c) {  // values of the components
        const CentreJob<T>& j = jobs[c];
        const int ra = j.a.idx(p);
        const T* A = j.a.ptr + (int64_t)ra * j.chi;
        int e = j.a.exps ? j.a.exps[ra] : 0;
        T v = Sc<T>::zero();
        if (j.b.ptr) {
          const int rb = j.b.idx(p);
          const T* B = j.b.ptr + (int64_t)rb * j.chi;
          e += j.b.exps ? j.b.exps[rb] : 0;
          typename Real<T>::t ma = 0, mb = 0;
          for (int k = 0; k < j.chi; ++k) {
            ma = mag_max(ma, A[k]);
            mb = mag_max(mb, B[k]);
          }
          const int ea = exponent_of(ma), eb = exponent_of(mb);
          for (int k = 0; k < j.chi; ++k) v = Sc<T>::fma(scale_pow2(A[k], -ea), scale_pow2(B[k], -eb), v);
          e += ea + eb;
        } else {
          v = A[0];
        }
        wv[c * ld + p] = v;
        we[c * ld + p] = e;
      }
    for (int c = 0; c < ncomp; ++c) {
      const CentreJob<T>& j = jobs[c];
      T v = d;
      int e = 0;
      if (ncomp > 1) {
        for (int o = 0; o < ncomp; ++o)
          if (o != c) {
            v = v * wv[o * ld + p];
            e += we[o * ld + p];
          }
      }
      // the products above read wv of the others: results go behind them
      wv[(ncomp + c) * ld + p] = v;
      we[(ncomp + c) * ld + p] = e;
      typename Real<T>::t m = mag_max((typename Real<T>::t)0, v);
      if (m != 0) {
        if (j.a.exps) e += j.a.exps[j.a.idx(p)];
        if (j.b.ptr && j.b.exps) e += j.b.exps[j.b.idx(p)];
        top = max(top, e + exponent_of(m));
      }
    }
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if ((threadIdx.x & 31) == 0 && top != INT_MIN) atomicMax(S, top);
}

// w[p] = wv * 2^(we + exponents of both rows - S): with it both sides' rows
// enter as stored.
template <class T>
__global__ void k_adj_weight(const T* __restrict__ wv, const int* __restrict__ we, int Pc, const CentreJob<T>* jobs,
                             int c, const int* __restrict__ S, T* __restrict__ w) {
  const CentreJob<T>& j = jobs[c];
  const int s = common_exp(S);
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < Pc; p += gridDim.x * blockDim.x) {
    int e = we[p] - s;
    if (j.a.exps) e += j.a.exps[j.a.idx(p)];
    if (j.b.ptr && j.b.exps) e += j.b.exps[j.b.idx(p)];
    w[p] = scale_pow2(wv[p], e);
  }
}

// Adjoint of a side that has a row per point: E[p] = wv * (other side's row).
template <class T>
__global__ void k_adj_seed(const T* __restrict__ wv, const int* __restrict__ we, int Pc, const CentreSide<T> o, int chi,
                           const int* __restrict__ S, T* __restrict__ E, int* __restrict__ Ee) {
  const int s = common_exp(S);
  const int64_t n = (int64_t)Pc * chi;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int p = (int)(i / chi), k = (int)(i - (int64_t)p * chi);
    if (!o.ptr) {  // a vertex centre
      E[i] = wv[p];
      Ee[p] = we[p] - s;
      continue;
    }
    const int r = o.idx(p);
    E[i] = wv[p] * o.ptr[(int64_t)r * chi + k];
    if (k == 0) Ee[p] = we[p] + (o.exps ? o.exps[r] : 0) - s;
  }
}

// dst[g] += sum over the points p of group g (the points that read table row
// g) of weight * src row.  weight: w[p], or 2^(we[p] + rexp[g]).  A warp takes
// up to 128 points of one group: its lanes are the columns, several points side
// by side when the row is short, and one atomic per column ends the run.
// Bound by the gather of the source rows from L2.
constexpr int SEG_TILE = 128;
template <class T>
__global__ void __launch_bounds__(256) k_segsum(const T* __restrict__ src, const RowIdx sidx, int chi,
                                                const T* __restrict__ w, const int* __restrict__ we,
                                                const int* __restrict__ rexp, const int* __restrict__ perm,
                                                const int* __restrict__ off, const int* __restrict__ cnt,
                                                const int* __restrict__ ts, int ng, T* __restrict__ dst) {
  const int lane = threadIdx.x & 31;
  const int b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (b >= ts[ng]) return;
  const int g = find_group(ts, ng, b);
  const int i0 = off[g] + (b - ts[g]) * SEG_TILE, n = min(SEG_TILE, off[g] + cnt[g] - i0);
  if (n <= 0) return;
  const int cw = chi >= 32 ? 32 : chi > 16 ? 32 : chi > 8 ? 16 : chi > 4 ? 8 : chi > 2 ? 4 : chi > 1 ? 2 : 1;
  const int pw = 32 / cw, pl = lane / cw, cl = lane % cw;
  const int ge = rexp ? rexp[g] : 0;
  for (int k0 = 0; k0 < chi; k0 += cw) {
    const int k = k0 + cl;
    T s = Sc<T>::zero();
#pragma unroll 4
    for (int i = pl; i < n; i += pw) {
      const int p = perm ? perm[i0 + i] : i0 + i;
      const T x = !src ? Sc<T>::one() : k < chi ? src[(int64_t)sidx(p) * chi + k] : Sc<T>::zero();
      if (w) s = Sc<T>::fma(w[p], x, s);
      else s = s + scale_pow2(x, we[p] + ge);
    }
    for (int o = cw; o < 32; o <<= 1) s = s + shfl_x(s, o);
    if (pl == 0 && k < chi) atomic_add_T<T>(dst + (int64_t)g * chi + k, s);
  }
}

// Adjoints of a table product out[(g, r)][n] = sum_k a[r][k] B[g][n][k] with
// a = A 2^-rex (the scaling of the row that the forward product took):
//   dB[g][n][k] += sum_r  bar[(g, r)][n] a[r][k]
//   dA[r][k]    += 2^-rex sum_(g, n) bar[(g, r)][n] B[g][n][k]
// One launch takes every product of a level; a block makes one 32 x 32 tile of
// either sum over a slice of its terms and adds it atomically, so that a sum
// over thousands of rows into a small tensor still fills the SMs.  A table also
// has the rows that no point reads, whose adjoint is zero: where they (or the
// tensor's slices behind them) are not finite the zeros are left out.
__device__ __forceinline__ bool not_finite(float x) { return (__float_as_uint(x) & 0x7F800000u) == 0x7F800000u; }
__device__ __forceinline__ bool not_finite(double x) { return ((unsigned)__double2hiint(x) & 0x7FF00000u) == 0x7FF00000u; }
__device__ __forceinline__ bool not_finite(cplx z) { return not_finite(z.re) || not_finite(z.im); }
__device__ __forceinline__ bool is_zero(float x) { return x == 0.f; }
__device__ __forceinline__ bool is_zero(double x) { return x == 0.0; }
__device__ __forceinline__ bool is_zero(cplx z) { return z.re == 0.0 && z.im == 0.0; }

template <class T>
struct BackJob {
  const T* A;
  const int* rex;
  const T* B;
  const T* bar;
  T* dB;
  T* dA;
  int K, N, rpg, ng;
  int sb, sa;   // slices of the two sums
  int nb;       // blocks of dB (the rest of the job's are dA's)
};
constexpr int BACK_T = 32, BACK_C = 16;
template <class T>
__global__ void __launch_bounds__(256) k_rows_back(const BackJob<T>* __restrict__ jobs, const int* __restrict__ first,
                                                   int njobs) {
  __shared__ T xs[BACK_C][BACK_T + 1], ys[BACK_C][BACK_T + 1];
  const int ji = find_group(first, njobs, blockIdx.x);
  const BackJob<T> j = jobs[ji];
  int b = blockIdx.x - first[ji];
  const int nk = (j.K + BACK_T - 1) / BACK_T;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  T acc[2][2] = {{Sc<T>::zero(), Sc<T>::zero()}, {Sc<T>::zero(), Sc<T>::zero()}};
  auto multiply = [&](bool guard) {  // guard: some y is not finite
    if (guard) {
      for (int z = 0; z < BACK_C; ++z)
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const T x = xs[z][ty + 16 * i];
            if (!is_zero(x)) acc[i][q] = Sc<T>::fma(x, ys[z][tx + 16 * q], acc[i][q]);
          }
      return;
    }
#pragma unroll
    for (int z = 0; z < BACK_C; ++z) {
      const T x0 = xs[z][ty], x1 = xs[z][ty + 16], y0 = ys[z][tx], y1 = ys[z][tx + 16];
      acc[0][0] = Sc<T>::fma(x0, y0, acc[0][0]);
      acc[0][1] = Sc<T>::fma(x0, y1, acc[0][1]);
      acc[1][0] = Sc<T>::fma(x1, y0, acc[1][0]);
      acc[1][1] = Sc<T>::fma(x1, y1, acc[1][1]);
    }
  };
  if (b < j.nb) {
    const int nn = (j.N + BACK_T - 1) / BACK_T;
    const int k0 = (b % nk) * BACK_T;
    b /= nk;
    const int n0 = (b % nn) * BACK_T;
    b /= nn;
    const int g = b % j.ng, sl = b / j.ng;
    const int per = (j.rpg + j.sb - 1) / j.sb, r0 = sl * per, r1 = min(j.rpg, r0 + per);
    for (int r = r0; r < r1; r += BACK_C) {
      bool bad = false;
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int z = (tid + 256 * i) >> 5, c = tid & 31;
        const bool in = r + z < r1;
        xs[z][c] = in && n0 + c < j.N ? j.bar[((int64_t)g * j.rpg + r + z) * j.N + n0 + c] : Sc<T>::zero();
        T y = Sc<T>::zero();
        if (in && k0 + c < j.K) {
          y = j.A[(int64_t)(r + z) * j.K + k0 + c];
          const int e = j.rex[r + z];
          if (e) y = scale_pow2(y, -e);
        }
        ys[z][c] = y;
        bad |= not_finite(y);
      }
      multiply(__syncthreads_or(bad));
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int n = n0 + ty + 16 * i, k = k0 + tx + 16 * q;
        if (n < j.N && k < j.K) atomic_add_T<T>(j.dB + ((int64_t)g * j.N + n) * j.K + k, acc[i][q]);
      }
    return;
  }
  b -= j.nb;
  const int k0 = (b % nk) * BACK_T;
  b /= nk;
  const int nr = (j.rpg + BACK_T - 1) / BACK_T;
  const int r0 = (b % nr) * BACK_T, sl = b / nr;
  const int64_t tot = (int64_t)j.ng * j.N;
  const int64_t per = (tot + j.sa - 1) / j.sa, z0 = sl * per, z1 = min(tot, z0 + per);
  for (int64_t zz = z0; zz < z1; zz += BACK_C) {
    bool bad = false;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = tid + 256 * i;
      {  // rows r, terms z: neighbouring terms are neighbouring entries of bar
        const int c = t >> 4, z = t & 15;
        const int64_t q = zz + z;
        T x = Sc<T>::zero();
        if (q < z1 && r0 + c < j.rpg) {
          const int64_t g = q / j.N;
          x = j.bar[(g * j.rpg + r0 + c) * j.N + (q - g * j.N)];
        }
        xs[z][c] = x;
      }
      const int z = t >> 5, c = t & 31;
      const T y = zz + z < z1 && k0 + c < j.K ? j.B[(zz + z) * j.K + k0 + c] : Sc<T>::zero();
      ys[z][c] = y;
      bad |= not_finite(y);
    }
    multiply(__syncthreads_or(bad));
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = r0 + ty + 16 * i;
    if (r >= j.rpg) continue;
    const int e = j.rex[r];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int k = k0 + tx + 16 * q;
      if (k < j.K) atomic_add_T<T>(j.dA + (int64_t)r * j.K + k, e ? scale_pow2(acc[i][q], -e) : acc[i][q]);
    }
  }
}

// User gradient += 2^S * adjoint tensors, back in the stored axis order
// (MoveJob: dst the adjoint tensor, src the stored one's place).
template <class T>
__global__ void k_adj_add(const MoveJob* __restrict__ jobs, const int* __restrict__ S) {
  const MoveJob& j = jobs[blockIdx.y];
  const int s = common_exp(S);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < j.n; i += (int64_t)gridDim.x * blockDim.x) {
    int64_t q = i, at = 0;
    for (int d = j.nd - 1; d >= 0; --d) {
      const int64_t t = q / j.dim[d];
      at += (q - t * j.dim[d]) * j.str[d];
      q = t;
    }
    T* o = (T*)j.src + at;
    *o = *o + scale_pow2(((const T*)j.dst)[i], s);
  }
}

}  // namespace tnfa

// Integration of a tree tensor network function over [0,1)^n.
//
// Reference: integrate (src/integration.jl:6-17) multiplies every vertex by
// ITensor(c, site_inds...) with c = 1/base (1 with take_sum) and contracts the
// network with belief propagation.  Here (tnfa_integrate): one HBM-streaming
// launch per level of the tree (k_integrate_level), leaves first, reads each
// tensor once and contracts it at the same time with the site weights and the
// children's messages; messages are kept in FP64 (or complex FP64) with a
// power-of-two exponent per vertex.
// site_reduced_net (the site-reduced network as a network) serves the
// operator and partial integrals.
#include <cmath>

#include "evaluate.cuh"

namespace tnfa {

struct ReduceJob {
  int64_t soff, doff, slice;
  int sd;
  double w;
};

// dst_v[i] = w_v * sum_s src_v[s * slice + i] for every vertex v (blockIdx.y).
template <class T>
__global__ void k_site_reduce(const T* __restrict__ src, T* __restrict__ dst,
                              const ReduceJob* __restrict__ jobs) {
  const ReduceJob jb = jobs[blockIdx.y];
  const T* s = src + jb.soff;
  T* d = dst + jb.doff;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < jb.slice;
       i += (int64_t)gridDim.x * blockDim.x) {
    T acc = Sc<T>::zero();
    for (int q = 0; q < jb.sd; ++q) acc += s[(int64_t)q * jb.slice + i];
    d[i] = acc * (T)jb.w;
  }
}
template <>
__global__ void k_site_reduce<cplx>(const cplx* __restrict__ src, cplx* __restrict__ dst,
                                    const ReduceJob* __restrict__ jobs) {
  const ReduceJob jb = jobs[blockIdx.y];
  const cplx* s = src + jb.soff;
  cplx* d = dst + jb.doff;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < jb.slice;
       i += (int64_t)gridDim.x * blockDim.x) {
    cplx acc{0.0, 0.0};
    for (int q = 0; q < jb.sd; ++q) acc += s[(int64_t)q * jb.slice + i];
    d[i] = cplx{acc.re * jb.w, acc.im * jb.w};
  }
}

// ----------------------------------------------------- tnfa_integrate ----
// A vertex's height is one more than its highest child's; the vertices of a
// height are a launch (several where they do not fit its parameters).  A leaf
// of at most kFoldSites site values costs less to sum again where its parent
// reads it than a launch does, so it has no height of its own.
//
// A block belongs to one vertex and its 8 warps take a task each: up to kb <= 32
// consecutive rows (s, a, k) with the same (s, a).  A warp issues the loads of its
// first rows, and only then the block waits for the launch before it
// (programmatic dependent launch: the next level's blocks start, and their
// tensors stream in, while this level's last tasks run).  The block brings the
// children's messages to shared memory, scaled by a power of two into [1/2, 1)
// and in the tensors' own type (so FP32 networks keep the FP32 pipe); a warp
// contracts its rows with the last child's message, each row weighted by the
// other children's entries, and adds the sum to its vertex's FP64 (complex
// FP64) message with one atomic that nothing waits for.  The exponents go to
// the host with the roots' messages.
//
// Row loads are 16-byte vectors (4 FP32, 2 FP64 or 1 complex value per lane)
// when the vertex's rows allow it; G = 2^lg lanes share a row (rows of few
// vectors leave no lane idle), NCH vectors a lane cover a row of up to
// 32 * NCH * VE entries and max(NCH, 4) loads are in flight per lane (twice as
// many and 24 instead of 32 warps per SM took 2-5 us longer a call).
//
// Bound by HBM at large bonds in FP32 and by the FP64 pipe in FP64 (one FMA per
// entry, 203 us of the 284 below: there the rows are summed with their weights
// before the last child's message comes in, once per task).  A call on
// the 60-vertex binary tree, against one persistent launch fed by bulk copies
// whose consumers waited for their children's flags task by task: bond 128
// (117 M entries) FP32 120 us (194), FP64 284 us (350); bond 48 FP32 50 us (129);
// path of 60 vertices, bond 256, FP64 284 us (1312), bond 6 208 us (425).
template <class T> struct IntAcc { using type = double; };
template <> struct IntAcc<cplx> { using type = cplx; };
__device__ inline void atomicAddAcc(double* a, double v) { atomicAdd(a, v); }
__device__ inline void atomicAddAcc(cplx* a, cplx v) {
  atomicAdd(&a->re, v.re);
  atomicAdd(&a->im, v.im);
}
__device__ inline double mulw(double x, double w) { return x * w; }
__device__ inline cplx mulw(cplx x, double w) { return cplx{x.re * w, x.im * w}; }
__device__ inline double to_acc(float x, double) { return (double)x; }
__device__ inline double to_acc(double x, double) { return x; }
__device__ inline cplx to_acc(cplx x, cplx) { return x; }
__device__ inline float to_dot(double x, float) { return (float)x; }
__device__ inline double to_dot(double x, double) { return x; }
__device__ inline cplx to_dot(cplx x, cplx) { return x; }
__device__ inline float ldcg_acc(const float* p) { return __ldcg(p); }
__device__ inline double ldcg_acc(const double* p) { return __ldcg(p); }
__device__ inline cplx ldcg_acc(const cplx* p) {
  const double2 v = __ldcg((const double2*)p);
  return {v.x, v.y};
}

template <class T> struct Vec;
template <> struct Vec<float> {
  static constexpr int VE = 4;
  __device__ static void load(const float* p, float* e) {
    const float4 v = __ldcs((const float4*)p);
    e[0] = v.x;
    e[1] = v.y;
    e[2] = v.z;
    e[3] = v.w;
  }
};
template <> struct Vec<double> {
  static constexpr int VE = 2;
  __device__ static void load(const double* p, double* e) {
    const double2 v = __ldcs((const double2*)p);
    e[0] = v.x;
    e[1] = v.y;
  }
};
template <> struct Vec<cplx> {
  static constexpr int VE = 1;
  __device__ static void load(const cplx* p, cplx* e) {
    const double2 v = __ldcs((const double2*)p);
    e[0] = cplx{v.x, v.y};
  }
};

constexpr int INT_MAXV = 24, INT_MAXCH = 56;  // of a launch: its parameters stay below 4 KB
constexpr int INT_WARPS = 8;
constexpr int kFoldSites = 8;
// blocks per SM: 64 registers a thread, 128 where a row's vectors need them
// (FP32 rows of 257 to 512 entries, NCH = 4, spill 24 bytes a thread at 64)
constexpr int int_blocks(size_t size, int nch) { return size == 16 || nch >= 8 ? 2 : 4; }
// messages of a vertex's children kept on chip: with the block's static
// reductions (4 bytes a child and warp) within the 48 KB of a plain launch
constexpr int INT_SMEM = 48 * 1024 - EVAL_MAXC * INT_WARPS * 4;
constexpr int INT_SMEM_LONG = 200 * 1024;  // where rows are long

struct IntChild {
  int64_t src;  // offset of its message, or of its tensor (sd > 0)
  double w;     // site weight of a leaf summed here
  int dim, sd, v;
};
struct IntVertex {
  int64_t off;     // tensor offset (elements)
  int64_t kouter;  // rows per (s, a): product of the children's dims but the last
  int64_t out;     // offset of its message
  double w;        // site weight: prod of 1 / leg dim (1 with take_sum)
  int b0, ntask;   // first block of the launch; tasks
  int nkb, kb;     // tasks per (s, a); rows per task
  int sd, chi_a, last;    // last: entries of the last child
  int nchild, ch0;        // its children in the launch's list
  short lg, vec;   // vec: rows are read as 16-byte vectors, 2: rows longer than the lanes hold
  short staged;    // the messages are in shared memory (2: without an unscaled copy)
  short tpw;       // tasks per warp
};

template <class T>
struct IntLevel {
  using A = typename IntAcc<T>::type;
  const T* tensors;
  A* msgs;    // accumulators (zeroed)
  int* exps;  // per vertex: exponent taken out of its message
  int nv;
  IntVertex v[INT_MAXV];
  IntChild ch[INT_MAXCH];
};

template <class T>
__device__ inline T shfl_t(T v, int src) {
  if constexpr (sizeof(T) == 16) {
    cplx z = *(cplx*)&v;
    z.re = __shfl_sync(0xffffffffu, z.re, src);
    z.im = __shfl_sync(0xffffffffu, z.im, src);
    return *(T*)&z;
  } else {
    return __shfl_sync(0xffffffffu, v, src);
  }
}

// High word of the larger magnitude: enough for the exponent.
__device__ inline unsigned hi_abs(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }
__device__ inline unsigned hi_abs(cplx z) { return max(hi_abs(z.re), hi_abs(z.im)); }
// Exponent taken out of a message whose largest high word is hw.
__device__ inline int msg_exponent(unsigned hw) {
  const int e = (int)(hw >> 20);
  return e == 0x7ff ? 0 : min(e - 1022, 1022);  // none where an entry is not finite
}

template <class T>
__device__ inline T warp_total(T v) {
  for (int o = 16; o; o >>= 1) {
    if constexpr (sizeof(T) == 16) {
      cplx z = *(cplx*)&v;
      z.re += __shfl_xor_sync(0xffffffffu, z.re, o);
      z.im += __shfl_xor_sync(0xffffffffu, z.im, o);
      v = *(T*)&z;
    } else {
      v = v + __shfl_xor_sync(0xffffffffu, v, o);
    }
  }
  return v;
}

// Rows longer than the lanes of the main path hold (over 1024 FP32, 512 FP64
// or 256 complex entries): a warp walks its row with 8 vectors per lane in
// flight, each summed on its own, and takes several tasks, because a message of
// that length costs its block about as long to stage as eight rows to read.  A
// path of 4 vertices, against the scalar loop of the unaligned rows and against
// one persistent launch: bond 4096 FP32 158 us (741, 480), bond 6000 FP64 356
// us (1233, 982).
template <class T, class Unscale, class Entry>
__device__ inline void long_rows(const IntLevel<T>& L, const IntVertex& iv, const IntChild* ch, const T* cm,
                                 const Unscale& unscale, const Entry& entry) {
  using A = typename IntAcc<T>::type;
  constexpr int VE = Vec<T>::VE, LU = 8;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nchild = iv.nchild, last = iv.last;
  const IntChild& cl = ch[nchild - 1];
  const double ul = unscale(nchild - 1);
  int olast = 0;
  for (int c = 0; c + 1 < nchild; ++c) olast += ch[c].dim;
  for (int i = 0; i < iv.tpw; ++i) {
    const int64_t t64 = ((int64_t)((int)blockIdx.x - iv.b0) * iv.tpw + i) * INT_WARPS + warp;
    if (t64 >= iv.ntask) return;
    const int t = (int)t64, sa = t / iv.nkb, a = sa % iv.chi_a;
    const int64_t k0 = (int64_t)(t - sa * iv.nkb) * iv.kb;
    const int nr = (int)min((int64_t)iv.kb, iv.kouter - k0);
    T w = Sc<T>::one();  // lane r: the weight of row r
    if (nchild > 1 && lane < nr) {
      int64_t kk = k0 + lane;
      int o = olast;
      for (int c = nchild - 2; c >= 0; --c) {
        const int d = ch[c].dim, j = c ? (int)(kk % d) : (int)kk;
        o -= d;
        w = w * (iv.staged ? cm[o + j] : to_dot(mulw(entry(ch[c], j), unscale(c)), T{}));
        if (c) kk /= d;
      }
    }
    T partial = Sc<T>::zero();
    for (int r = 0; r < nr; ++r) {
      const T* row = L.tensors + iv.off + ((int64_t)sa * iv.kouter + k0 + r) * last;
      T acc[LU];
#pragma unroll
      for (int u = 0; u < LU; ++u) acc[u] = Sc<T>::zero();
      for (int j0 = lane * VE; j0 < last; j0 += 32 * VE * LU) {
        T x[LU][VE];
#pragma unroll
        for (int u = 0; u < LU; ++u) {
          const int j = j0 + 32 * VE * u;
          if (j < last) Vec<T>::load(row + j, x[u]);
        }
#pragma unroll
        for (int u = 0; u < LU; ++u) {
          const int j = j0 + 32 * VE * u;
          if (j >= last) break;
#pragma unroll
          for (int e = 0; e < VE; ++e) {
            const T m = iv.staged ? cm[olast + j + e] : to_dot(mulw(entry(cl, j + e), ul), T{});
            acc[u] = Sc<T>::fma(x[u][e], m, acc[u]);
          }
        }
      }
#pragma unroll
      for (int u = 1; u < LU; ++u) acc[0] = acc[0] + acc[u];
      partial = Sc<T>::fma(shfl_t(w, r), acc[0], partial);
    }
    partial = warp_total(partial);
    if (lane == 0) atomicAddAcc(L.msgs + iv.out + a, mulw(to_acc(partial, A{}), iv.w));
  }
}

template <class T, int NCH>
__global__ void __launch_bounds__(32 * INT_WARPS, int_blocks(sizeof(T), NCH)) k_integrate_level(const __grid_constant__ IntLevel<T> L) {
  using A = typename IntAcc<T>::type;
  constexpr int VE = Vec<T>::VE, U = NCH >= 4 ? 1 : 4 / NCH;
  extern __shared__ __align__(16) unsigned char int_smem[];
  __shared__ unsigned red[EVAL_MAXC][INT_WARPS];
  asm volatile("griddepcontrol.launch_dependents;");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int vi = 0, hi = L.nv;
  while (hi - vi > 1) {
    const int mid = (vi + hi) >> 1;
    if (L.v[mid].b0 <= (int)blockIdx.x) vi = mid;
    else hi = mid;
  }
  const IntVertex& iv = L.v[vi];
  const int nchild = iv.nchild, last = iv.last, lg = iv.lg;
  if (nchild == 0) {
    // a leaf: msg[a] = w sum_s T[s, a]
    const T* base = L.tensors + iv.off;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int a = threadIdx.x; a < iv.chi_a; a += blockDim.x) {
      T acc = Sc<T>::zero();
      for (int s = 0; s < iv.sd; ++s) acc += base[(int64_t)s * iv.chi_a + a];
      L.msgs[iv.out + a] = mulw(to_acc(acc, A{}), iv.w);
    }
    return;
  }
  const IntChild* ch = L.ch + iv.ch0;
  const int t = ((int)blockIdx.x - iv.b0) * INT_WARPS + warp;
  const int sa = t / iv.nkb, a = sa % iv.chi_a;
  const int64_t k0 = (int64_t)(t - sa * iv.nkb) * iv.kb;
  const int nr = t < iv.ntask ? (int)min((int64_t)iv.kb, iv.kouter - k0) : 0;
  const T* rows = L.tensors + iv.off + ((int64_t)sa * iv.kouter + k0) * last;

  // the first rows: RPI of them per load, lane jl of row sub
  const int sub = lane >> lg, jl = lane & ((1 << lg) - 1), RPI = 32 >> lg;
  T x[U][NCH][VE];
  auto load = [&](int r0) {
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        const int j = (jl + (c << lg)) * VE, r = r0 + u * RPI + sub;
        if (r < nr && j < last) {
          Vec<T>::load(rows + (int64_t)r * last + j, x[u][c]);
        } else {
#pragma unroll
          for (int e = 0; e < VE; ++e) x[u][c][e] = Sc<T>::zero();
        }
      }
  };
  if (iv.vec == 1) load(0);
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // the children's messages
  auto entry = [&](const IntChild& c, int j) -> A {
    if (c.sd == 0) return ldcg_acc(L.msgs + c.src + j);
    const T* base = L.tensors + c.src + j;
    T acc = Sc<T>::zero();
    for (int s = 0; s < c.sd; ++s) acc += base[(int64_t)s * c.dim];
    return mulw(to_acc(acc, A{}), c.w);
  };
  A* const raw = (A*)int_smem;
  T* cm = (T*)int_smem;  // scaled in place where the types are the same
  if constexpr (sizeof(A) != sizeof(T)) {
    if (iv.staged) {
      int sum = 0;
      for (int c = 0; c < nchild; ++c) sum += ch[c].dim;
      if (iv.staged == 1) cm = (T*)(raw + sum);
    }
  }
  int at = 0;
  for (int c = 0; c < nchild; ++c) {
    unsigned hw = 0;
    for (int j = threadIdx.x; j < ch[c].dim; j += 32 * INT_WARPS) {
      const A e = entry(ch[c], j);
      if (iv.staged == 1) raw[at + j] = e;
      hw = max(hw, hi_abs(e));
    }
    hw = __reduce_max_sync(0xffffffffu, hw);
    if (lane == 0) red[c][warp] = hw;
    at += ch[c].dim;
  }
  __syncthreads();
  auto exponent = [&](int c) {
    unsigned hw = 0;
#pragma unroll
    for (int q = 0; q < INT_WARPS; ++q) hw = max(hw, red[c][q]);
    return msg_exponent(hw);
  };
  auto unscale = [&](int c) { return __hiloint2double((1023 - exponent(c)) << 20, 0); };
  if ((int)blockIdx.x == iv.b0 && (int)threadIdx.x < nchild) L.exps[ch[threadIdx.x].v] = exponent(threadIdx.x);
  if (iv.staged) {
    at = 0;
    for (int c = 0; c < nchild; ++c) {
      const double f = unscale(c);
      for (int j = threadIdx.x; j < ch[c].dim; j += 32 * INT_WARPS) 
        cm[at + j] = to_dot(mulw(iv.staged == 1 ? raw[at + j] : entry(ch[c], j), f), T{});
      at += ch[c].dim;
    }
    __syncthreads();
  }
  if constexpr (NCH == 8) {  // (the other forms are launched where every row fits)
    if (iv.vec == 2) {
      long_rows<T>(L, iv, ch, cm, unscale, entry);
      return;
    }
  }
  if (nr <= 0) return;
  // entry j of child c's scaled message (o: where its entries start)
  auto mval = [&](int c, int o, int j) -> T {
    return iv.staged ? cm[o + j] : to_dot(mulw(entry(ch[c], j), unscale(c)), T{});
  };
  int olast = 0;
  for (int c = 0; c + 1 < nchild; ++c) olast += ch[c].dim;
  // weight of row r: the product of the other children's entries
  T w32 = Sc<T>::one();
  if (nchild > 1 && lane < nr) {
    int64_t kk = k0 + lane;
    int o = olast;
    for (int c = nchild - 2; c >= 0; --c) {
      const int d = ch[c].dim;
      o -= d;
      w32 = w32 * mval(c, o, c ? (int)(kk % d) : (int)kk);
      if (c) kk /= d;
    }
  }
  T partial = Sc<T>::zero();
  if (iv.vec == 1) {
    auto lastval = [&](int c, int e) -> T {
      const int j = (jl + (c << lg)) * VE + e;
      return j < last ? cm[olast + j] : Sc<T>::zero();
    };
    auto row_weight = [&](int r) -> T {
      const T w = shfl_t(w32, r & 31);
      return r < nr ? w : Sc<T>::zero();
    };
    if constexpr (sizeof(T) == 4) {
      // sum_r w_r (row_r . m): one rounding of the weight per row, the U rows
      // of a load summed before they join the others
      T ml[NCH][VE];
#pragma unroll
      for (int c = 0; c < NCH; ++c)
#pragma unroll
        for (int e = 0; e < VE; ++e) ml[c][e] = lastval(c, e);
      for (int r0 = 0; r0 < nr; r0 += U * RPI) {
        T dot[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          dot[u] = Sc<T>::zero();
#pragma unroll
          for (int c = 0; c < NCH; ++c)
#pragma unroll
            for (int e = 0; e < VE; ++e) dot[u] = Sc<T>::fma(x[u][c][e], ml[c][e], dot[u]);
        }
        if (r0 + U * RPI < nr) load(r0 + U * RPI);
        T sum = Sc<T>::zero();
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int r = r0 + u * RPI + sub;
          const T w = row_weight(r);
          if (r < nr) sum = Sc<T>::fma(w, dot[u], sum);  // no 0 x Inf from the rows beyond
        }
        partial += sum;
      }
    } else {
      // (sum_r w_r row_r) . m: one FP64 FMA per entry and no second one per row
      T acc[NCH][VE];
#pragma unroll
      for (int c = 0; c < NCH; ++c)
#pragma unroll
        for (int e = 0; e < VE; ++e) acc[c][e] = Sc<T>::zero();
      for (int r0 = 0; r0 < nr; r0 += U * RPI) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const T w = row_weight(r0 + u * RPI + sub);
#pragma unroll
          for (int c = 0; c < NCH; ++c)
#pragma unroll
            for (int e = 0; e < VE; ++e) acc[c][e] = Sc<T>::fma(w, x[u][c][e], acc[c][e]);
        }
        if (r0 + U * RPI < nr) load(r0 + U * RPI);
      }
#pragma unroll
      for (int c = 0; c < NCH; ++c)
#pragma unroll
        for (int e = 0; e < VE; ++e)
          if ((jl + (c << lg)) * VE + e < last) partial = Sc<T>::fma(acc[c][e], lastval(c, e), partial);
    }
  } else {
    // rows that are not 16-byte aligned
    for (int r = 0; r < nr; ++r) {
      const T* row = rows + (int64_t)r * last;
      T dot = Sc<T>::zero();
      for (int j = lane; j < last; j += 32) dot = Sc<T>::fma(row[j], mval(nchild - 1, olast, j), dot);
      partial = Sc<T>::fma(shfl_t(w32, r), dot, partial);
    }
  }
  partial = warp_total(partial);
  if (lane == 0) atomicAddAcc(L.msgs + iv.out + a, mulw(to_acc(partial, A{}), iv.w));
}

// A network with the same bonds and no site legs: the site-reduced tensors.
tnfa_net* site_reduced_net(tnfa_ctx* ctx, const tnfa_net* net, int take_sum) {
  const Topo& T = net->topo;
  Topo R = T;
  R.nlegs.assign(T.V, 0);
  R.leg_dim.clear();
  R.leg_var.clear();
  R.leg_digit.clear();
  R.leg_kind.clear();
  R.finalize();
  tnfa_net* out = new_net(ctx, R, net->dtype);
  std::vector<ReduceJob> jobs(T.V);
  int64_t maxslice = 1;
  for (int v = 0; v < T.V; ++v) {
    double w = 1.0;
    if (!take_sum)
      for (int l = T.leg_off[v]; l < T.leg_off[v + 1]; ++l) w /= T.leg_dim[l];
    jobs[v] = {T.off[v], R.off[v], R.size(v), T.site_dim[v], w};
    maxslice = std::max<int64_t>(maxslice, R.size(v));
  }
  DBuf dj(ctx, jobs.size() * sizeof(ReduceJob));
  TNFA_CUDA(cudaMemcpyAsync(dj.p, jobs.data(), jobs.size() * sizeof(ReduceJob),
                            cudaMemcpyHostToDevice, ctx->stream));
  TNFA_CHECK(T.V <= 65535, TNFA_ERR_UNSUPPORTED, "more than 65535 vertices");
  dim3 grid(grid_for(maxslice, 256, std::max(1, 4 * ctx->sm_count)), T.V);
  KernelScope ks(ctx, "site_reduce", (double)T.n_elem,
                 (double)dtype_size(net->dtype) * (double)(T.n_elem + R.n_elem));
  if (net->dtype == TNFA_F64)
    k_site_reduce<double><<<grid, 256, 0, ctx->stream>>>((const double*)net->d, (double*)out->d,
                                                         dj.as<ReduceJob>());
  else if (net->dtype == TNFA_F32)
    k_site_reduce<float><<<grid, 256, 0, ctx->stream>>>((const float*)net->d, (float*)out->d,
                                                        dj.as<ReduceJob>());
  else
    k_site_reduce<cplx><<<grid, 256, 0, ctx->stream>>>((const cplx*)net->d, (cplx*)out->d,
                                                       dj.as<ReduceJob>());
  TNFA_LAUNCH_CHECK();
  return out;
}

template <class T>
void integrate_levels(tnfa_ctx* ctx, const tnfa_net* net, int take_sum, double* out) {
  using A = typename IntAcc<T>::type;
  constexpr int VE = Vec<T>::VE;
  const Topo& Tp = net->topo;
  const int V = Tp.V;
  const std::vector<int> roots = Tp.roots();
  const int nr = (int)roots.size();
  std::vector<char> is_root(V, 0), folded(V, 0);
  for (int r : roots) is_root[r] = 1;
  // heights, children before their parent (a parent's index is smaller)
  std::vector<int> height(V, 0);
  std::vector<double> weight(V, 1.0);
  int hmax = 0, maxlast = 1;
  for (int v = V - 1; v >= 0; --v) {
    const auto& cs = Tp.children[v];
    TNFA_CHECK((int)cs.size() <= EVAL_MAXC, TNFA_ERR_UNSUPPORTED, "vertex degree too high");
    folded[v] = cs.empty() && !is_root[v] && Tp.site_dim[v] <= kFoldSites;
    for (int c : cs)
      if (!folded[c]) height[v] = std::max(height[v], height[c] + 1);
    if (!cs.empty()) maxlast = std::max(maxlast, Tp.link[cs.back()]);
    if (!take_sum)
      for (int l = Tp.leg_off[v]; l < Tp.leg_off[v + 1]; ++l) weight[v] /= Tp.leg_dim[l];
    hmax = std::max(hmax, height[v]);
  }
  std::vector<std::vector<int>> levels(hmax + 1);
  for (int v = 0; v < V; ++v)
    if (!folded[v]) levels[height[v]].push_back(v);
  // messages: the roots' first, read back with the exponents before them
  std::vector<int64_t> mofs(V, 0);
  int64_t nm = 0;
  for (int r : roots) {
    mofs[r] = nm;
    nm += Tp.link[r];
  }
  const int64_t nroot = nm;
  for (int v = 0; v < V; ++v)
    if (!is_root[v] && !folded[v]) {
      mofs[v] = nm;
      nm += Tp.link[v];
    }
  const size_t o_msgs = ((size_t)V * sizeof(int) + 15) & ~(size_t)15;
  DBuf scratch(ctx, o_msgs + (size_t)nm * sizeof(A));
  unsigned char* sb = (unsigned char*)scratch.p;
  TNFA_CUDA(cudaMemsetAsync(sb, 0, o_msgs + (size_t)nm * sizeof(A), ctx->stream));
  // vectors per lane covering the longest row (longer rows, and rows that
  // are not 16-byte aligned, take the generic path)
  int nch = 1;
  while (nch < 8 && 32 * VE * nch < maxlast) nch *= 2;
  const int64_t slots = (int64_t)ctx->sm_count * INT_WARPS * int_blocks(sizeof(T), nch);
  {
    KernelScope ks(ctx, "integrate", 2.0 * (double)Tp.n_elem, (double)dtype_size(net->dtype) * Tp.n_elem);
    bool first = true;
    IntLevel<T> L;
    L.tensors = (const T*)net->d;
    L.msgs = (A*)(sb + o_msgs);
    L.exps = (int*)sb;
    for (const auto& lv : levels) {
      int64_t rows = 0;
      for (int v : lv) {
        int64_t r = 1;
        for (size_t c = 0; c + 1 < Tp.children[v].size(); ++c) r *= Tp.link[Tp.children[v][c]];
        if (!Tp.children[v].empty()) rows += r * Tp.site_dim[v] * Tp.link[v];
      }
      // Rows per task: the level in w full waves of the warps the GPU holds, w
      // the one with the least w (rows + about three loads of rows, a block's
      // start).  Powers of two left a second wave of a few blocks at the narrow
      // levels and tasks of 4 rows at the middle ones (60-vertex binary tree,
      // FP32: bond 128 133 -> 121 us, bond 48 106 -> 50 us).
      const int start = 3 * (nch >= 4 ? 1 : 4 / nch) * std::max(1, 32 * VE / std::max(1, maxlast));
      int kb = 32;
      int64_t least = -1;
      for (int w = 1; w <= 8; ++w) {
        const int64_t k = std::max<int64_t>(1, (rows + slots * w - 1) / (slots * w));
        if (k > 32) continue;
        const int64_t cost = w * (k + start);
        if (least < 0 || cost < least) {
          least = cost;
          kb = (int)k;
        }
        if (k == 1) break;
      }
      int nc = 0;
      int64_t blocks = 0;
      size_t smem = 0;
      L.nv = 0;
      auto launch = [&]() {
        if (L.nv == 0) return;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)blocks);
        cfg.blockDim = dim3(32 * INT_WARPS);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = ctx->stream;
        cudaLaunchAttribute pdl[1];
        pdl[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        pdl[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = pdl;
        cfg.numAttrs = first ? 0 : 1;  // the first launch follows the clearing
        first = false;
        if (smem > INT_SMEM)
          TNFA_CUDA(cudaFuncSetAttribute(k_integrate_level<T, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, INT_SMEM_LONG));
        switch (nch) {
          case 1: TNFA_CUDA(cudaLaunchKernelEx(&cfg, k_integrate_level<T, 1>, L)); break;
          case 2: TNFA_CUDA(cudaLaunchKernelEx(&cfg, k_integrate_level<T, 2>, L)); break;
          case 4: TNFA_CUDA(cudaLaunchKernelEx(&cfg, k_integrate_level<T, 4>, L)); break;
          default: TNFA_CUDA(cudaLaunchKernelEx(&cfg, k_integrate_level<T, 8>, L)); break;
        }
        L.nv = nc = 0;
        blocks = 0;
        smem = 0;
      };
      for (int v : lv) {
        const auto& cs = Tp.children[v];
        IntVertex iv{};
        iv.off = Tp.off[v];
        iv.out = mofs[v];
        iv.w = weight[v];
        iv.sd = Tp.site_dim[v];
        iv.chi_a = Tp.link[v];
        iv.nchild = (int)cs.size();
        int64_t kouter = 1, sum = 0, ntask = 1;
        for (size_t c = 0; c < cs.size(); ++c) {
          if (c + 1 < cs.size()) kouter *= Tp.link[cs[c]];
          sum += Tp.link[cs[c]];
        }
        iv.kouter = kouter;
        iv.last = cs.empty() ? 1 : Tp.link[cs.back()];
        iv.kb = iv.nkb = 1;
        if (!cs.empty()) {
          // the tasks of an (s, a) of even length, as many as stay within the wave
          int64_t nkb = std::max<int64_t>(1, kouter / kb);
          if ((kouter + nkb - 1) / nkb > 32) nkb = (kouter + 31) / 32;
          iv.kb = (int)((kouter + nkb - 1) / nkb);
          nkb = (kouter + iv.kb - 1) / iv.kb;
          ntask = (int64_t)iv.sd * iv.chi_a * nkb;
          TNFA_CHECK(ntask < (int64_t(1) << 31) - 64, TNFA_ERR_UNSUPPORTED, "integrate: vertex too large");
          iv.nkb = (int)nkb;
        }
        iv.ntask = (int)ntask;
        size_t need = (size_t)sum * (sizeof(A) + (sizeof(A) != sizeof(T) ? sizeof(T) : 0));
        iv.staged = need <= INT_SMEM;
        iv.vec = !cs.empty() && iv.off % VE == 0 && iv.last % VE == 0 && ((uintptr_t)net->d & 15) == 0;
        iv.tpw = 1;
        if (iv.vec && iv.last > 32 * VE * nch) {
          iv.vec = 2;
          if (!iv.staged && (size_t)sum * sizeof(T) <= INT_SMEM_LONG) {
            iv.staged = sizeof(A) == sizeof(T) ? 1 : 2;
            need = (size_t)sum * sizeof(T);
          }
          const int64_t wave = (int64_t)ctx->sm_count * int_blocks(sizeof(T), nch) * INT_WARPS;
          iv.tpw = (short)std::min<int64_t>(32, (ntask + wave - 1) / wave);
        } else if (!iv.staged) {
          iv.vec = 0;
        }
        iv.lg = 5;
        if (iv.vec == 1)
          while (iv.lg > 0 && (1 << (iv.lg - 1)) * VE >= iv.last) --iv.lg;
        const int64_t nb = (ntask + INT_WARPS * iv.tpw - 1) / (INT_WARPS * iv.tpw);
        if (L.nv == INT_MAXV || nc + iv.nchild > INT_MAXCH || blocks + nb > 0x7fffffff) launch();
        iv.b0 = (int)blocks;
        iv.ch0 = nc;
        blocks += nb;
        if (iv.staged) smem = std::max(smem, need);
        for (int c : cs) L.ch[nc++] = IntChild{folded[c] ? Tp.off[c] : mofs[c], weight[c], Tp.link[c],
                                               folded[c] ? Tp.site_dim[c] : 0, c};
        L.v[L.nv++] = iv;
      }
      launch();
    }
  }
  // one read-back: the exponents and the roots' messages
  std::vector<unsigned char> hb(o_msgs + (size_t)nroot * sizeof(A));
  TNFA_CUDA(cudaMemcpyAsync(hb.data(), sb, hb.size(), cudaMemcpyDeviceToHost, ctx->stream));
  TNFA_CUDA(cudaStreamSynchronize(ctx->stream));
  // product over the roots of the forest, exponents applied at the end
  double re = 1.0, im = 0.0;
  int e = 0;
  for (int v = 0; v < V; ++v) {
    int ex;
    std::memcpy(&ex, hb.data() + v * sizeof(int), sizeof(int));
    e += ex;
  }
  for (int i = 0; i < nr; ++i) {
    A val;
    std::memcpy(&val, hb.data() + o_msgs + mofs[roots[i]] * sizeof(A), sizeof(A));
    double vr, vi;
    if constexpr (sizeof(A) == 16) {
      const cplx z = *(const cplx*)&val;
      vr = z.re;
      vi = z.im;
    } else {
      vr = *(const double*)&val;
      vi = 0.0;
    }
    const double nr_ = re * vr - im * vi, ni = re * vi + im * vr;
    re = nr_;
    im = ni;
  }
  out[0] = std::ldexp(re, e);
  if (net->dtype == TNFA_C128) out[1] = std::ldexp(im, e);
}

}  // namespace tnfa

using namespace tnfa;

extern "C" int tnfa_integrate(tnfa_ctx* ctx, const tnfa_net* net, int take_sum, double* out) {
  TNFA_API_BEGIN(ctx);
  require_ctx(ctx);
  require_net(net, "integrate");
  TNFA_CHECK(out, TNFA_ERR_INVALID_ARGUMENT, "null out");
  const Topo& T = net->topo;
  for (int l = 0; l < T.leg_off[T.V]; ++l)
    TNFA_CHECK(T.leg_kind[l] != TNFA_LEG_OPERATOR, TNFA_ERR_INVALID_ARGUMENT,
               "integrate needs a function network, got an operator");
  if (net->dtype == TNFA_F64)
    integrate_levels<double>(ctx, net, take_sum, out);
  else if (net->dtype == TNFA_F32)
    integrate_levels<float>(ctx, net, take_sum, out);
  else
    integrate_levels<cplx>(ctx, net, take_sum, out);
  TNFA_API_END
}

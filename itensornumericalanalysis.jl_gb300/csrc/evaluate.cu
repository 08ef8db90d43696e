// Batched point evaluation of a tree tensor network function.
//
// Reference path (ITensorNumericalAnalysis.jl): evaluate
// (src/itensornetworkfunction.jl:96-112) = calculate_ind_values (digits by
// greedy subtraction, src/IndexMaps/abstractindexmap.jl:121-138) -> project
// (one-hot slice of every site leg, :84-94) -> scalar(tn; alg="bp") (exact on
// a tree).  It handles one point per call.
//
// Here all points of a chunk go through the tree vertex by vertex (children
// before parents):
//   1. k_digitize: coordinates -> site value s_v(p) of every vertex (u8).
//   2. per vertex: group the points by s_v (count / scan / scatter), so that a
//      tile of points shares one slice T_v[s].
//   3. per vertex: out[p, a] = sum_k A[p, k] T_v[s][a][k] with A the row-wise
//      Kronecker product of the children's messages.  Leaves are never
//      materialised: a parent reads the leaf slice T_leaf[s_leaf(p)] directly.
//      Each message row is rescaled by a power of two when it is read (exact)
//      and the exponent is carried per point, so deep trees neither underflow
//      nor overflow.
//   4. k_combine: product over the roots of the forest, times 2^exponent.
#include <algorithm>
#include <memory>
#include <type_traits>

#include "eval_tree.cuh"
#include "evaluate.cuh"
#include "rows.cuh"

namespace tnfa {

// ------------------------------------------------------- contraction ----
template <class T>
__device__ inline bool locate_tile(const VertexJob<T>& j, int tp, int b, int& row0, int& nrows,
                                   int& g) {
  const int ng = j.ngroups;
  if (b >= j.tile_start[ng]) return false;
  const int gg = find_group(j.tile_start, ng, b);
  g = gg;
  row0 = j.grp_off[gg] + (b - j.tile_start[gg]) * tp;
  nrows = min(tp, j.grp_off[gg] + j.grp_cnt[gg] - row0);
  return nrows > 0;
}

template <class T> struct Frexp;
template <> struct Frexp<double> {
  __device__ static int e(double m) {
    int ex = 0;
    frexp(m, &ex);
    return ex;
  }
};
template <> struct Frexp<float> {
  __device__ static int e(float m) {
    int ex = 0;
    frexpf(m, &ex);
    return ex;
  }
};

// Load the message rows of every child for the tile's points into shared
// memory (child c at rows + choff_c * tp, row-major tp x dim_c), rescale each
// row by 2^-e so that its largest entry lies in [0.5, 1), and accumulate the
// exponents of the tile's points into eacc.  The gather issues LU loads per
// thread before storing any, so that a tile's rows are in flight together
// rather than one load latency per element.
template <class T>
__device__ void load_children(const VertexJob<T>& j, const int* pts, int nrows, int tp, T* rows,
                              int* eacc) {
  constexpr int LU = 8;
  int off = 0;
  for (int c = 0; c < j.nchild; ++c) {
    const ChildSrc<T> s = j.ch[c];
    T* dst = rows + (int64_t)off * tp;
    const int n = tp * s.dim;
    for (int i0 = threadIdx.x; i0 < n; i0 += blockDim.x * LU) {
      T v[LU];
#pragma unroll
      for (int u = 0; u < LU; ++u) {
        const int idx = i0 + u * (int)blockDim.x;
        const int r = idx / s.dim, i = idx - r * s.dim;
        v[u] = Sc<T>::zero();
        if (idx < n && r < nrows) {
          v[u] = s.ptr[(int64_t)s.idx(pts[r]) * s.dim + i];
        }
      }
#pragma unroll
      for (int u = 0; u < LU; ++u) {
        const int idx = i0 + u * (int)blockDim.x;
        if (idx < n) dst[idx] = v[u];
      }
    }
    off += s.dim;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  off = 0;
  for (int c = 0; c < j.nchild; ++c) {
    const ChildSrc<T> s = j.ch[c];
    T* base = rows + (int64_t)off * tp;
    for (int r = warp; r < nrows; r += nw) {
      T* row = base + (int64_t)r * s.dim;
      decltype(Sc<T>::absmax(Sc<T>::zero())) m = 0;
      for (int i = lane; i < s.dim; i += 32) m = max(m, Sc<T>::absmax(row[i]));
      for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
      int ex = (m > 0) ? Frexp<decltype(m)>::e(m) : 0;
      if (ex != 0)
        for (int i = lane; i < s.dim; i += 32) row[i] = Sc<T>::scale2(row[i], -ex);
      if (lane == 0) atomicAdd(&eacc[r], ex + (s.exps ? s.exps[s.idx(pts[r])] : 0));
    }
    off += s.dim;
  }
  __syncthreads();
}

// A[r, k] for the tile: product of the children's row entries.
template <class T>
__device__ inline T kr_entry(const VertexJob<T>& j, const T* rows, int tp, int r, int k) {
  T a = Sc<T>::one();
  int off_end = 0;
  for (int c = 0; c < j.nchild; ++c) off_end += j.ch[c].dim;
  int off = off_end;
  for (int c = j.nchild - 1; c >= 0; --c) {
    int d = j.ch[c].dim;
    off -= d;
    int kc = k % d;
    k /= d;
    a = a * rows[(int64_t)off * tp + (int64_t)r * d + kc];
  }
  return a;
}

// General SIMT contraction: CTA tile = TP points x TA output columns, 256
// threads as (256 / (TA / 4)) row threads x (TA / 4) column threads, each
// with a (TP / row threads) x 4 register micro-tile; K streamed in chunks of
// 16.  TA follows the parent bond (32, 64 or 128) so that thin bonds do not
// pay for idle columns.
template <class T, int TP, int TA>
__global__ void __launch_bounds__(256) k_contract_gemm(const VertexJob<T> j) {
  constexpr int KC = 16, CT = TA / 4, RT = 256 / CT, RM = TP / RT;
  static_assert(RM >= 1 && RM * RT == TP, "tile rows must cover the row threads");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int row0, nrows, g;
  if (!locate_tile(j, TP, blockIdx.x, row0, nrows, g)) return;
  const int a0 = blockIdx.y * TA;
  int sumdim = 0;
  for (int c = 0; c < j.nchild; ++c) sumdim += j.ch[c].dim;
  T* rows = (T*)smem_raw;
  T* As = rows + (int64_t)sumdim * TP;  // [KC][TP]
  T* Bs = As + KC * TP;                 // [KC][TA]
  int* pts = (int*)(Bs + KC * TA);
  int* eacc = pts + TP;
  for (int r = threadIdx.x; r < TP; r += blockDim.x) {
    pts[r] = r < nrows ? (j.perm ? j.perm[row0 + r] : row0 + r) : 0;
    eacc[r] = 0;
  }
  __syncthreads();
  load_children(j, pts, nrows, TP, rows, eacc);

  const T* Bg = j.B + (int64_t)g * j.chi_a * j.K;
  const int tx = threadIdx.x % CT, ty = threadIdx.x / CT;
  T acc[RM][4];
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[i][q] = Sc<T>::zero();

  for (int k0 = 0; k0 < j.K; k0 += KC) {
    for (int idx = threadIdx.x; idx < KC * TP; idx += blockDim.x) {
      int kk = idx / TP, r = idx - kk * TP;
      int k = k0 + kk;
      As[idx] = (k < j.K && r < nrows) ? kr_entry(j, rows, TP, r, k) : Sc<T>::zero();
    }
    for (int idx = threadIdx.x; idx < KC * TA; idx += blockDim.x) {
      int a = idx / KC, kk = idx - a * KC;
      int k = k0 + kk, aa = a0 + a;
      Bs[kk * TA + a] = (k < j.K && aa < j.chi_a) ? Bg[(int64_t)aa * j.K + k] : Sc<T>::zero();
    }
    __syncthreads();
#pragma unroll 4
    for (int kk = 0; kk < KC; ++kk) {
      T av[RM], bv[4];
#pragma unroll
      for (int i = 0; i < RM; ++i) av[i] = As[kk * TP + ty * RM + i];
#pragma unroll
      for (int q = 0; q < 4; ++q) bv[q] = Bs[kk * TA + tx + CT * q];
#pragma unroll
      for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[i][q] = Sc<T>::fma(av[i], bv[q], acc[i][q]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    int r = ty * RM + i;
    if (r >= nrows) continue;
    int p = pts[r];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int a = a0 + tx + CT * q;
      if (a < j.chi_a) j.out[(int64_t)p * j.chi_a + a] = acc[i][q];
    }
  }
  if (blockIdx.y == 0)
    for (int r = threadIdx.x; r < nrows; r += blockDim.x)
      j.out_exp[pts[r]] = eacc[r] + (j.gexp ? j.gexp[g] : 0);
}

// Narrow outputs (chi_a <= 16): one warp per point, lanes split K, shuffle
// reduction.  Used at the roots (chi_a = 1) and on thin bonds.
template <class T, int NA>
__global__ void __launch_bounds__(256) k_contract_narrow(const VertexJob<T> j) {
  constexpr int TP = 8;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int row0, nrows, g;
  if (!locate_tile(j, TP, blockIdx.x, row0, nrows, g)) return;
  int sumdim = 0;
  for (int c = 0; c < j.nchild; ++c) sumdim += j.ch[c].dim;
  T* rows = (T*)smem_raw;
  int* pts = (int*)(rows + (int64_t)sumdim * TP);
  int* eacc = pts + TP;
  for (int r = threadIdx.x; r < TP; r += blockDim.x) {
    pts[r] = r < nrows ? (j.perm ? j.perm[row0 + r] : row0 + r) : 0;
    eacc[r] = 0;
  }
  __syncthreads();
  load_children(j, pts, nrows, TP, rows, eacc);
  const int lane = threadIdx.x & 31, r = threadIdx.x >> 5;
  if (r >= nrows) return;
  const T* Bg = j.B + (int64_t)g * j.chi_a * j.K;
  T acc[NA];
#pragma unroll
  for (int q = 0; q < NA; ++q) acc[q] = Sc<T>::zero();
  const int dl = j.nchild ? j.ch[j.nchild - 1].dim : 1;
  if (j.nchild >= 1 && j.nchild <= 2 && dl >= 16) {
    // lanes over the last child's entries, a loop over the other child's:
    // no index decoding in the loop
    const int offl = sumdim - dl;
    const int Ko = j.K / dl;
    const T* ml = rows + (int64_t)offl * TP + (int64_t)r * dl;
    const T* m0 = rows + (int64_t)r * (j.nchild == 2 ? j.ch[0].dim : 0);
    for (int ko = 0; ko < Ko; ++ko) {
      const T ao = j.nchild == 2 ? m0[ko] : Sc<T>::one();
      const T* Bk = Bg + (int64_t)ko * dl;
      for (int kl = lane; kl < dl; kl += 32) {
        const T a = ao * ml[kl];
#pragma unroll
        for (int q = 0; q < NA; ++q)
          acc[q] = Sc<T>::fma(a, q < j.chi_a ? Bk[(int64_t)q * j.K + kl] : Sc<T>::zero(), acc[q]);
      }
    }
  } else {
    for (int k = lane; k < j.K; k += 32) {
      T a = kr_entry(j, rows, TP, r, k);
#pragma unroll
      for (int q = 0; q < NA; ++q)
        acc[q] = Sc<T>::fma(a, q < j.chi_a ? Bg[(int64_t)q * j.K + k] : Sc<T>::zero(), acc[q]);
    }
  }
  int p = pts[r];
#pragma unroll
  for (int q = 0; q < NA; ++q) {
    if (q >= j.chi_a) continue;
    T v = acc[q];
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
    if (lane == 0) j.out[(int64_t)p * j.chi_a + q] = v;
  }
  if (lane == 0) j.out_exp[p] = eacc[r] + (j.gexp ? j.gexp[g] : 0);
}

// --------------------------------------------- fused small-bond path ----
// For networks whose bonds are all small (chi <= 16, or chi <= 32 on paths),
// one thread walks its point through the whole tree: digits from the digit
// program, then the vertices in post-order, each a chain of small
// matrix-vector products against the network's tensors held in shared
// memory, the messages in shared memory ([slot][entry][thread], conflict
// free), each message rescaled by a power of two with the exponent carried.
// One launch per chunk instead of about four per vertex, and no message
// traffic through HBM.
struct FusedStep {
  int off;       // element offset of the vertex tensor in the shared copy
  int vertex;
  int chi_a;     // parent bond (1 at a root)
  int nchild;    // 0, 1 or 2
  int d1, d2;    // child bonds (1 when absent)
  int in1, in2;  // message slots of the children
  int out;       // message slot of this vertex; -1 at a root
};
constexpr int FUSED_MAXV = 128;

template <class T, int CHI>
__global__ void __launch_bounds__(128) k_eval_fused(
    const double* __restrict__ X, int ncols, int Pc, const DigitRun* __restrict__ prog, int nprog,
    const FusedStep* __restrict__ steps, int nsteps, const T* __restrict__ tensors, int n_elem,
    int V, int nslots, size_t off_msg, size_t off_prog, size_t off_steps, void* out, int kind,
    int64_t P, int64_t p0, int* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // the tensors in shared memory when they fit (off_msg > 0), else read in
  // place (a few hundred KB at most: they stay in L1 / L2)
  const T* ts = off_msg ? (const T*)smem_raw : tensors;
  T* msg = (T*)(smem_raw + off_msg);
  DigitRun* pg = (DigitRun*)(smem_raw + off_prog);
  FusedStep* st = (FusedStep*)(smem_raw + off_steps);
  if (off_msg)
    for (int i = threadIdx.x; i < n_elem; i += blockDim.x) ((T*)smem_raw)[i] = tensors[i];
  for (int i = threadIdx.x; i < nprog; i += blockDim.x) pg[i] = prog[i];
  for (int i = threadIdx.x; i < nsteps; i += blockDim.x) st[i] = steps[i];
  __syncthreads();
  const int tpb = blockDim.x, tid = threadIdx.x;
  auto M = [&](int slot, int k) -> T& { return msg[((size_t)slot * CHI + k) * tpb + tid]; };
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < Pc; p += gridDim.x * blockDim.x) {
    int dg[FUSED_MAXV];
    for (int v = 0; v < V; ++v) dg[v] = 0;
    digit_codes(X + (int64_t)p * ncols, pg, nprog, dg, 1, 0, V, err);
    T val = Sc<T>::one();
    int ex_acc = 0;
    for (int i = 0; i < nsteps; ++i) {
      const FusedStep s = st[i];
      const int K = s.d1 * s.d2;
      const T* Tv = ts + s.off + (int64_t)dg[s.vertex] * s.chi_a * K;
      // the last child's message in registers; the first child's (two
      // children) read from its slot inside the loop, which the output slot
      // never aliases (it is taken before the children's slots are freed)
      const int dl = s.nchild == 2 ? s.d2 : s.d1;
      const int il = s.nchild == 2 ? s.in2 : s.in1;
      T ml[CHI];
#pragma unroll
      for (int c = 0; c < CHI; ++c) ml[c] = (s.nchild > 0 && c < dl) ? M(il, c) : Sc<T>::zero();
      decltype(Sc<T>::absmax(Sc<T>::zero())) mx = 0;
      T rv = Sc<T>::zero();
      for (int a = 0; a < s.chi_a; ++a) {
        const T* Ta = Tv + (int64_t)a * K;
        T acc = Sc<T>::zero();
        if (s.nchild == 0) {
          acc = Ta[0];
        } else if (s.nchild == 1) {
#pragma unroll
          for (int c = 0; c < CHI; ++c)
            if (c < dl) acc = Sc<T>::fma(Ta[c], ml[c], acc);
        } else {
          for (int b = 0; b < s.d1; ++b) {
            const T* Tb = Ta + b * dl;
            T in = Sc<T>::zero();
#pragma unroll
            for (int c = 0; c < CHI; ++c)
              if (c < dl) in = Sc<T>::fma(Tb[c], ml[c], in);
            acc = Sc<T>::fma(M(s.in1, b), in, acc);
          }
        }
        if (s.out < 0) {
          rv = acc;  // a root: its parent bond is 1
        } else {
          M(s.out, a) = acc;
          mx = max(mx, Sc<T>::absmax(acc));
        }
      }
      if (s.out < 0) {
        val = val * rv;
        continue;
      }
      const int ex = mx > 0 ? Frexp<decltype(mx)>::e(mx) : 0;
      ex_acc += ex;
      if (ex != 0)
        for (int a = 0; a < s.chi_a; ++a) M(s.out, a) = Sc<T>::scale2(M(s.out, a), -ex);
    }
    write_out<T>(out, kind, p0 + p, P, val, ex_acc);
  }
}

struct FusedPlan {
  bool ok = false;
  int chi = 0;  // CHI of the kernel
  int nslots = 0, tpb = 0;
  std::vector<FusedStep> steps;
  size_t off_msg = 0, off_prog = 0, off_steps = 0, smem = 0;
};

// Whether the fused kernel takes this network, and its schedule (post-order,
// message slots recycled as children are consumed) and shared-memory layout.
static FusedPlan make_fused_plan(const Topo& T, size_t tsize, size_t nprog, int64_t npoints) {
  FusedPlan F;
  const char* env = getenv("TNFA_EVAL_FUSED");
  if (env && *env == '0') return F;
  if (T.V > FUSED_MAXV) return F;
  int chimax = 1, maxch = 0;
  for (int v = 0; v < T.V; ++v) {
    chimax = std::max(chimax, T.link[v]);
    maxch = std::max(maxch, (int)T.children[v].size());
    if (T.site_dim[v] > 256) return F;
  }
  if (maxch > 2 || chimax > 32 || (chimax > 16 && maxch > 1)) return F;
  // a thread per point: above chi 8 a few thousand points leave the GPU
  // mostly idle, where the per-vertex kernels spread a point over a warp
  if (chimax > 8 && npoints < 32768) return F;
  if (T.n_elem * (int64_t)tsize > 4 * 1024 * 1024) return F;
  F.chi = chimax <= 2 ? 2 : chimax <= 4 ? 4 : chimax <= 8 ? 8 : chimax <= 16 ? 16 : 32;
  std::vector<int> slot(T.V, -1), free_slots;
  int n = 0;
  for (int r : T.roots()) {
    std::vector<std::pair<int, int>> stack{{r, 0}};
    while (!stack.empty()) {
      auto& [v, i] = stack.back();
      if (i < (int)T.children[v].size()) {
        const int c = T.children[v][i++];
        stack.push_back({c, 0});
        continue;
      }
      FusedStep s{};
      s.off = (int)T.off[v];
      s.vertex = v;
      s.chi_a = T.link[v];
      s.nchild = (int)T.children[v].size();
      s.d1 = s.nchild >= 1 ? T.link[T.children[v][0]] : 1;
      s.d2 = s.nchild >= 2 ? T.link[T.children[v][1]] : 1;
      s.in1 = s.nchild >= 1 ? slot[T.children[v][0]] : 0;
      s.in2 = s.nchild >= 2 ? slot[T.children[v][1]] : 0;
      // the output slot is taken before the children's are released, so it
      // never aliases a message the step still reads
      if (T.parent[v] >= 0) {
        if (free_slots.empty()) free_slots.push_back(n++);
        s.out = slot[v] = free_slots.back();
        free_slots.pop_back();
      } else {
        s.out = -1;
      }
      for (int c : T.children[v]) free_slots.push_back(slot[c]);
      F.steps.push_back(s);
      stack.pop_back();
    }
  }
  F.nslots = std::max(n, 1);
  auto al = [](size_t x) { return (x + 15) & ~(size_t)15; };
  // threads per block: as many as keep the messages within 64 KB, 32..128
  const size_t per_thread = (size_t)F.nslots * F.chi * tsize;
  F.tpb = (int)std::min<size_t>(128, std::max<size_t>(32, (64 * 1024 / per_thread) / 32 * 32));
  if ((size_t)F.tpb * per_thread > 64 * 1024) return F;
  const bool ts_smem = (size_t)T.n_elem * tsize <= 96 * 1024;
  F.off_msg = ts_smem ? al((size_t)T.n_elem * tsize) : 0;
  F.off_prog = al(F.off_msg + (size_t)F.tpb * per_thread);
  F.off_steps = al(F.off_prog + nprog * sizeof(DigitRun));
  F.smem = F.off_steps + F.steps.size() * sizeof(FusedStep);
  F.ok = F.smem <= 200 * 1024;
  return F;
}

template <class T>
static void launch_fused(tnfa_ctx* ctx, const FusedPlan& F, const FusedStep* dsteps, const T* tensors,
                         const Topo& Tp, const double* Xc, int ncols, int Pc,
                         const DigitRun* dprog, int nprog, void* o, int kind, int64_t Pout,
                         int64_t pofs, int* derr) {
  const int tpb = F.tpb;
  const unsigned grid = grid_for(Pc, tpb, ctx->sm_count * (2048 / tpb));
  double fl = 0;
  for (const auto& s : F.steps) fl += 2.0 * s.chi_a * s.d1 * s.d2;
  KernelScope ks(ctx, "eval_fused", fl * Pc, (double)Pc * (ncols * 8.0 + 8.0));
  auto go = [&](auto kern) {
    TNFA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F.smem));
    kern<<<grid, tpb, F.smem, ctx->stream>>>(Xc, ncols, Pc, dprog, nprog, dsteps, (int)F.steps.size(),
                                             tensors, (int)Tp.n_elem, Tp.V, F.nslots, F.off_msg,
                                             F.off_prog, F.off_steps, o, kind, Pout, pofs, derr);
  };
  switch (F.chi) {
    case 2: go(k_eval_fused<T, 2>); break;
    case 4: go(k_eval_fused<T, 4>); break;
    case 8: go(k_eval_fused<T, 8>); break;
    case 16: go(k_eval_fused<T, 16>); break;
    default: go(k_eval_fused<T, 32>); break;
  }
  TNFA_LAUNCH_CHECK();
}

// -------------------------------------------------------------- driver ----
struct EvalPlan {
  std::vector<int> order;        // vertices computed, children before parents
  std::vector<char> fused_leaf;  // non-root leaf read directly by its parent
  std::vector<int> slot;         // message slot of a computed non-root vertex
  int nslots = 0;
  std::vector<int> roots;
  int chimax = 1;
};

// A vertex's output slot is taken while its children still hold theirs, so
// that it never shares memory with the messages it reads: the contraction
// kernels write their output as they go (tiles split over columns, the
// sliced kernel's two phases) and the autotuner runs one contraction several
// times over the same inputs.
static EvalPlan make_plan(const Topo& T) {
  EvalPlan P;
  P.fused_leaf.assign(T.V, 0);
  P.slot.assign(T.V, -1);
  P.roots = T.roots();
  for (int v = 0; v < T.V; ++v)
    if (T.parent[v] >= 0 && T.children[v].empty()) P.fused_leaf[v] = 1;
  // Post-order DFS per root keeps the number of live messages near the depth.
  for (int r : P.roots) {
    std::vector<std::pair<int, int>> st{{r, 0}};
    while (!st.empty()) {
      auto& [v, i] = st.back();
      if (i < (int)T.children[v].size()) {
        int c = T.children[v][i++];
        st.push_back({c, 0});
      } else {
        if (!P.fused_leaf[v]) P.order.push_back(v);
        st.pop_back();
      }
    }
  }
  std::vector<int> free_slots;
  int n = 0;
  for (int v : P.order) {
    if (T.parent[v] >= 0) {
      if (free_slots.empty()) free_slots.push_back(n++);
      P.slot[v] = free_slots.back();
      free_slots.pop_back();
      P.chimax = std::max(P.chimax, T.link[v]);
    }
    for (int c : T.children[v])
      if (!P.fused_leaf[c]) free_slots.push_back(P.slot[c]);
  }
  P.nslots = n;
  return P;
}

// Tile of k_contract_gemm for a parent bond chi_a > 16 and children rows of
// sumdim entries: TP x TA with TA the smallest of 32 / 64 / 128 covering
// chi_a, and TP = 4096 / TA (a 4 x 4 micro-tile per thread) while the
// children rows of the tile fit in shared memory, else TP = 1024 / TA (one
// row per thread).
struct GemmTile {
  int tp, ta;
};
static GemmTile gemm_tile(int chi_a, int sumdim, size_t tsize) {
  const size_t row_bytes = (size_t)sumdim * tsize;
  const int ta = chi_a <= 32 ? 32 : chi_a <= 64 ? 64 : 128;
  const int tp = 4096 / ta;
  if (row_bytes * tp + (size_t)16 * (tp + ta) * tsize <= 160 * 1024) return {tp, ta};
  return {1024 / ta, ta};
}

// Tiles worth timing against each other for one shape: the rule's choice
// first, then a 4 x 4 micro-tile at each other column width that fits.
static std::vector<GemmTile> gemm_tile_candidates(int chi_a, int sumdim, size_t tsize) {
  std::vector<GemmTile> c{gemm_tile(chi_a, sumdim, tsize)};
  const size_t row_bytes = (size_t)sumdim * tsize;
  for (int ta : {32, 64, 128}) {
    const int tp = 4096 / ta;
    if (row_bytes * tp + (size_t)16 * (tp + ta) * tsize > 160 * 1024) continue;
    if (tp == c[0].tp && ta == c[0].ta) continue;
    c.push_back({tp, ta});
  }
  return c;
}

template <class T> struct FamilyName;
template <> struct FamilyName<double> { static constexpr const char* v = "contract_f64"; };
template <> struct FamilyName<float> { static constexpr const char* v = "contract_f32"; };
template <> struct FamilyName<cplx> { static constexpr const char* v = "contract_c128"; };

template <class T>
static void launch_contract(tnfa_ctx* ctx, const VertexJob<T>& j, int Pc,
                            const GemmTile* tile = nullptr) {
  int sumdim = 0;
  for (int c = 0; c < j.nchild; ++c) sumdim += j.ch[c].dim;
  KernelScope ks(ctx, FamilyName<T>::v, 2.0 * Pc * (double)j.K * j.chi_a,
                 (double)sizeof(T) * ((double)Pc * (sumdim + j.chi_a) +
                                      (double)j.site_dim * j.chi_a * j.K));
  if (j.chi_a <= 16) {
    constexpr int TP = 8;
    size_t sm = (size_t)sumdim * TP * sizeof(T) + 2 * TP * sizeof(int);
    TNFA_CHECK(sm <= 200 * 1024, TNFA_ERR_UNSUPPORTED, "children bonds too large for evaluation");
    if (sm > 48 * 1024)
      for (auto kern : {k_contract_narrow<T, 1>, k_contract_narrow<T, 4>, k_contract_narrow<T, 16>})
        TNFA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    unsigned gx = (unsigned)((Pc + TP - 1) / TP + j.ngroups);
    // accumulators per lane: as many as the parent bond, so that they stay in registers
    if (j.chi_a == 1) k_contract_narrow<T, 1><<<gx, 256, sm, ctx->stream>>>(j);
    else if (j.chi_a <= 4) k_contract_narrow<T, 4><<<gx, 256, sm, ctx->stream>>>(j);
    else k_contract_narrow<T, 16><<<gx, 256, sm, ctx->stream>>>(j);
  } else {
    const GemmTile t = tile ? *tile : gemm_tile(j.chi_a, sumdim, sizeof(T));
    const size_t sm = (size_t)sumdim * sizeof(T) * t.tp + (size_t)16 * (t.tp + t.ta) * sizeof(T) +
                      2 * t.tp * sizeof(int);
    TNFA_CHECK(sm <= 200 * 1024, TNFA_ERR_UNSUPPORTED, "children bonds too large for evaluation");
    dim3 grid((unsigned)((Pc + t.tp - 1) / t.tp + j.ngroups), (unsigned)((j.chi_a + t.ta - 1) / t.ta));
    auto go = [&](auto kern) {
      if (sm > 48 * 1024)
        TNFA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
      kern<<<grid, 256, sm, ctx->stream>>>(j);
    };
    if (t.ta == 32) t.tp == 128 ? go(k_contract_gemm<T, 128, 32>) : go(k_contract_gemm<T, 32, 32>);
    else if (t.ta == 64) t.tp == 64 ? go(k_contract_gemm<T, 64, 64>) : go(k_contract_gemm<T, 16, 64>);
    else t.tp == 32 ? go(k_contract_gemm<T, 32, 128>) : go(k_contract_gemm<T, 8, 128>);
  }
  TNFA_LAUNCH_CHECK();
}

static int contract_tile_rows(int chi_a, int sumdim, size_t tsize) {
  return chi_a <= 16 ? 8 : gemm_tile(chi_a, sumdim, tsize).tp;
}

// Digits of a network for the given variable list, in the order the digit map
// takes them (variable, part, digit).
struct DigitRef {
  int col, base, vertex, digit;
  int stride;   // weight of this leg inside the vertex's site value
  double invb;  // base^-digit, correctly rounded
  int start;    // first digit of a (variable, part)
};

static std::vector<DigitRef> make_digit_program(const Topo& T, int n_dims, const int32_t* dims,
                                                int* ncols_out) {
  bool has_imag = false;
  int L = T.leg_off[T.V];
  for (int l = 0; l < L; ++l) {
    TNFA_CHECK(T.leg_kind[l] != TNFA_LEG_OPERATOR, TNFA_ERR_INVALID_ARGUMENT,
               "evaluate needs a function network, got an operator");
    if (T.leg_kind[l] == TNFA_LEG_IMAG) has_imag = true;
  }
  const int ncols = has_imag ? 2 * n_dims : n_dims;
  *ncols_out = ncols;
  struct LegRef {
    int var, kind, digit, leg, vertex, stride;
  };
  std::vector<LegRef> refs;
  for (int v = 0; v < T.V; ++v) {
    int stride = 1;
    for (int l = T.leg_off[v + 1] - 1; l >= T.leg_off[v]; --l) {
      refs.push_back({T.leg_var[l], T.leg_kind[l], T.leg_digit[l], l, v, stride});
      stride *= T.leg_dim[l];
    }
  }
  std::sort(refs.begin(), refs.end(), [](const LegRef& a, const LegRef& b) {
    if (a.var != b.var) return a.var < b.var;
    if (a.kind != b.kind) return a.kind < b.kind;
    return a.digit < b.digit;
  });
  std::vector<DigitRef> prog;
  prog.reserve(refs.size());
  for (size_t i = 0; i < refs.size(); ++i) {
    const LegRef& r = refs[i];
    bool start = (i == 0 || refs[i - 1].var != r.var || refs[i - 1].kind != r.kind);
    int expect = start ? 1 : refs[i - 1].digit + 1;
    TNFA_CHECK(r.digit == expect, TNFA_ERR_TOPOLOGY,
               "digits of variable " + std::to_string(r.var) +
                   " are not 1..L (missing or repeated digit " + std::to_string(expect) + ")");
    int col = -1;
    for (int j = 0; j < n_dims; ++j)
      if (dims[j] == r.var) col = j;
    TNFA_CHECK(col >= 0, TNFA_ERR_INVALID_ARGUMENT,
               "variable " + std::to_string(r.var) + " has digits but is not listed in dims");
    int base = T.leg_dim[r.leg];
    TNFA_CHECK(base >= 2 && base <= 255, TNFA_ERR_UNSUPPORTED, "digit base outside 2..255");
    double bk = 1.0;
    for (int k = 0; k < r.digit; ++k) bk *= base;
    TNFA_CHECK(bk < 9007199254740992.0, TNFA_ERR_UNSUPPORTED, "base^digit above 2^53");
    DigitRef d;
    d.col = has_imag ? 2 * col + (r.kind == TNFA_LEG_IMAG ? 1 : 0) : col;
    d.base = base;
    d.vertex = r.vertex;
    d.digit = r.digit;
    d.stride = r.stride;
    d.invb = 1.0 / bk;
    d.start = start ? 1 : 0;
    prog.push_back(d);
  }
  return prog;
}

// The digits as runs that add to codes: the digit of vertex v counts
// mult[v] * stride in code slot[v].  A column in base 2 throughout becomes bit
// fields (neighbouring digits whose strides double or halve join one field).
static std::vector<DigitRun> make_runs(const std::vector<DigitRef>& prog, const std::vector<int>& slot,
                                       const std::vector<int>& mult) {
  std::vector<DigitRun> runs;
  for (size_t i = 0; i < prog.size();) {
    size_t e = i + 1;
    while (e < prog.size() && !prog[e].start) ++e;
    bool binary = true;
    for (size_t k = i; k < e; ++k) binary &= prog[k].base == 2;
    for (size_t k = i; k < e; ++k) {
      const DigitRef& d = prog[k];
      const int w = mult[d.vertex] * d.stride, s = slot[d.vertex];
      if (binary && k > i && runs.back().slot == s && runs.back().n < 31) {
        DigitRun& r = runs.back();
        if ((r.n == 1 || !r.rev) && (int64_t)w * 2 == r.w) {
          r.w = w;
          r.n += 1;
          continue;
        }
        if ((r.n == 1 || r.rev) && (int64_t)r.w << r.n == w) {
          r.rev = 1;
          r.n += 1;
          continue;
        }
      }
      DigitRun r{};
      r.col = d.col;
      r.slot = s;
      r.w = w;
      r.first = (short)d.digit;
      r.n = 1;
      r.base = (short)d.base;
      r.bits = binary;
      r.start = k == i;
      r.invb = d.invb;
      runs.push_back(r);
    }
    i = e;
  }
  return runs;
}

// The fused small-bond kernel keeps every vertex's site value by itself.
static std::vector<DigitRun> make_fused_runs(const Topo& T, const std::vector<DigitRef>& prog) {
  std::vector<int> slot(T.V), mult(T.V, 1);
  for (int v = 0; v < T.V; ++v) slot[v] = v;
  return make_runs(prog, slot, mult);
}

static size_t digitize_smem(int n, int block) { return (size_t)n * block * sizeof(int); }

// Codes of Pc points into C[slot][ldC].
static void launch_digitize(tnfa_ctx* ctx, const double* X, int ncols, int Pc, const DigitRun* runs,
                            int nruns, int nslots, int* C, int64_t ldC, int* err) {
  const int block = nslots <= 48 ? 256 : 64;
  const int per = block == 256 ? 48 : 192;
  for (int s0 = 0; s0 < nslots; s0 += per) {
    const int s1 = std::min(nslots, s0 + per);
    KernelScope ks(ctx, "digitize", 0.0, (double)Pc * (ncols * 8.0 + 4.0 * (s1 - s0)));
    k_digitize<<<grid_for(Pc, block, 8 * 152 * 8), block, digitize_smem(s1 - s0, block), ctx->stream>>>(
        X, ncols, Pc, runs, nruns, C, ldC, s0, s1, err);
    TNFA_LAUNCH_CHECK();
  }
}

// Groups Pc points by key (null: one group); meta as in group_meta_ints.
static const int* launch_group(tnfa_ctx* ctx, const int* key, int Pc, int ng, int tp, int* meta, int* perm) {
  KernelScope ks(ctx, "group", 0.0, key ? (double)Pc * 12.0 : 0.0);
  if (!key) {
    k_group_identity<<<1, 1, 0, ctx->stream>>>(meta, Pc, tp);
    TNFA_LAUNCH_CHECK();
    return nullptr;
  }
  TNFA_CUDA(cudaMemsetAsync(meta + ng, 0, ng * sizeof(int), ctx->stream));
  const size_t sm = ng <= GROUP_SMEM ? ng * sizeof(int) : 0;
  k_group_count<<<grid_for(Pc, 256, 4 * 152), 256, sm, ctx->stream>>>(key, Pc, ng, meta + ng);
  k_group_scan<<<1, 1024, 0, ctx->stream>>>(meta, ng, tp);
  const unsigned gs = (unsigned)((Pc + 256 * SCATTER_ITEMS - 1) / (256 * SCATTER_ITEMS));
  k_group_scatter<<<gs, 256, 2 * sm, ctx->stream>>>(key, Pc, ng, meta + 3 * ng + 1, perm);
  TNFA_LAUNCH_CHECK();
  return perm;
}
static void launch_retile(tnfa_ctx* ctx, bool keyed, int Pc, int ng, int tp, int* meta) {
  if (keyed) k_group_scan<<<1, 1024, 0, ctx->stream>>>(meta, ng, tp);
  else k_group_identity<<<1, 1, 0, ctx->stream>>>(meta, Pc, tp);
  TNFA_LAUNCH_CHECK();
}

// ------------------------------------------------- row-gather launches ----
// Tiles of k_rows_gemm by type, largest first.
template <class T> struct RowTiles;
template <> struct RowTiles<float> {
  static constexpr int n = 3;
  static constexpr int rm[3] = {8, 4, 2}, cn[3] = {4, 2, 1};
};
template <> struct RowTiles<double> {
  static constexpr int n = 3;
  static constexpr int rm[3] = {4, 2, 1}, cn[3] = {2, 1, 1};
};
template <> struct RowTiles<cplx> {
  static constexpr int n = 2;
  static constexpr int rm[2] = {2, 1}, cn[2] = {1, 1};
};

template <class T>
static int64_t row_blocks(const RowJob<T>& j, int tile) {
  const int tm = 8 * RowTiles<T>::rm[tile], tn = 32 * RowTiles<T>::cn[tile];
  const int64_t nbn = (j.N + tn - 1) / tn;
  if (j.rpg > 0) return (int64_t)(j.rows / j.rpg) * ((j.rpg + tm - 1) / tm) * nbn;
  return ((int64_t)(j.rows + tm - 1) / tm + j.ngroups) * nbn;
}

// The largest tile that still gives every SM two blocks, else the smallest:
// short tables are bound by the SMs they reach, not by the tile's reuse.
template <class T>
static int row_tile(tnfa_ctx* ctx, const std::vector<RowJob<T>>& jobs) {
  for (int t = 0; t + 1 < RowTiles<T>::n; ++t) {
    int64_t nb = 0;
    for (const auto& j : jobs) nb += row_blocks(j, t);
    if (nb >= 2 * ctx->sm_count) return t;
  }
  return RowTiles<T>::n - 1;
}

template <class T>
static void launch_rows(tnfa_ctx* ctx, int tile, int64_t blocks, const RowJob<T>& one,
                        const RowJob<T>* jobs, const int* first, int njobs) {
  TNFA_CHECK(blocks < (int64_t(1) << 31), TNFA_ERR_UNSUPPORTED, "contraction too large");
  auto go = [&](auto kern) { kern<<<(unsigned)blocks, 256, 0, ctx->stream>>>(one, jobs, first, njobs); };
  if constexpr (std::is_same<T, float>::value) {
    if (tile == 0) go(k_rows_gemm<T, 8, 4>);
    else if (tile == 1) go(k_rows_gemm<T, 4, 2>);
    else go(k_rows_gemm<T, 2, 1>);
  } else if constexpr (std::is_same<T, double>::value) {
    if (tile == 0) go(k_rows_gemm<T, 4, 2>);
    else if (tile == 1) go(k_rows_gemm<T, 2, 1>);
    else go(k_rows_gemm<T, 1, 1>);
  } else {
    if (tile == 0) go(k_rows_gemm<T, 2, 1>);
    else go(k_rows_gemm<T, 1, 1>);
  }
  TNFA_LAUNCH_CHECK();
}

// ------------------------------------------------------------- engine ----
// Scratch handed out in 256-byte pieces from one block (or counted, base null).
struct Carve {
  unsigned char* base = nullptr;
  size_t used = 0;
  template <class U> U* take(size_t n) {
    const size_t off = (used + 255) & ~(size_t)255;
    used = off + n * sizeof(U);
    return reinterpret_cast<U*>(base + off);
  }
};

// One evaluation call: the schedule of eval_tree.cuh laid out over scratch,
// then run.  Tables are built level by level (all row products of a level in
// one launch) once per call; the points follow in chunks: codes, the messages
// that have one row per point, the dot products at the centre.
template <class T>
class EvalEngine {
 public:
  EvalEngine(tnfa_ctx* ctx, const tnfa_net* net, const T* tensors, const std::vector<DigitRef>& prog,
             int ncols, int64_t P, bool use_tc, bool use_oz, size_t budget)
      : ctx_(ctx), net_(net), tensors_(tensors), topo_(net->topo), prog_(prog), ncols_(ncols), P_(P),
        use_tc_(use_tc), use_oz_(use_oz) {
    const int V = topo_.V;
    EvalTreeOptions o;
    o.points = (double)P;
    o.rule = use_tc ? CentreRule::ROOT : use_oz ? CentreRule::ROOT_EDGE : CentreRule::ANY_EDGE;
    o.absorb = !use_tc;
    if (use_tc || use_oz) {
      o.tensor_ok.assign(V, 0);
      for (int v = 0; v < V; ++v) {
        int cd[EVAL_MAXC];
        const auto& kids = topo_.children[v];
        if (kids.size() > (size_t)EVAL_MAXC) continue;
        bool aligned = true;  // leaf rows are read in place, 16 bytes at a time by the FP32 kernels
        for (size_t i = 0; i < kids.size(); ++i) {
          cd[i] = topo_.link[kids[i]];
          if (topo_.children[kids[i]].empty())
            aligned &= ((uintptr_t)(tensors + topo_.off[kids[i]]) & 15) == 0 && cd[i] % 4 == 0;
        }
        o.tensor_ok[v] = use_tc ? aligned && tc_vertex_eligible((int)kids.size(), cd, topo_.link[v])
                                : oz_vertex_eligible((int)kids.size(), cd, topo_.link[v]);
      }
    }
    // Tables take at most half the scratch: the row bound shrinks until they
    // fit.  Every digit code stays within 31 bits.
    double rows = std::min((double)P, 134217728.0);
    for (;;) {
      o.table_rows = rows;
      o.table_elems = std::min(1073741824.0, (double)(budget / 2) / sizeof(T));
      tree_ = EvalTreeBuilder(topo_, o).build();
      if (table_bytes() <= budget / 2 || o.rule == CentreRule::ROOT && rows < 1) break;
      rows = std::floor(rows / 4);
      if (rows < 1) {  // the stored order, nothing but points
        o.rule = CentreRule::ROOT;
        o.absorb = false;
      }
    }
    plan();
    per_point_ = (size_t)nmsg_ * (msg_chi_ * sizeof(T) + sizeof(int)) + (size_t)ncodes_ * 4 + (npp_ ? 4 : 0);
    const size_t tab = scratch(0);
    const size_t left = budget > tab ? budget - tab : 0;
    int64_t pc = per_point_ ? (int64_t)(left / per_point_) / 256 * 256 : int64_t(1) << 30;
    Pc_ = (int)std::min<int64_t>(P, std::max<int64_t>(256, std::min<int64_t>(pc, int64_t(1) << 30)));
  }

  int chunk() const { return Pc_; }
  void set_chunk(int pc) { Pc_ = pc; }
  size_t per_point() const { return per_point_; }
  // Bytes of scratch for chunks of pc points.
  size_t scratch(int64_t pc) {
    Carve c;
    lay_out(c, pc);
    return c.used + 256;
  }

  // Lays the call out over scratch at base (scratch(chunk()) bytes, 256-byte
  // aligned) and fills the host image of the job tables.
  void bind(void* base) {
    Carve c;
    c.base = (unsigned char*)base;
    lay_out(c, Pc_);
    fill_blob();
  }
  int* err_flag() const { return err_; }
  // The job tables and the cleared error flag go to the scratch (stream order).
  void upload() {
    h2d(ctx_, blob_, host_.data(), host_.size());
    clear_error();
  }
  void clear_error() { TNFA_CUDA(cudaMemsetAsync(err_, 0, 4, ctx_->stream)); }

  // Tables: permuted tensors, then every level.
  void tables() {
    if (!moves_.empty()) {
      int64_t n = 1;
      for (const auto& m : moves_) n = std::max(n, m.n);
      KernelScope ks(ctx_, "move", 0.0, 0.0);
      k_move<T><<<dim3(grid_for(n, 256, 1024), (unsigned)moves_.size()), 256, 0, ctx_->stream>>>(dmoves_);
      TNFA_LAUNCH_CHECK();
    }
    for (size_t l = 0; l < levels_.size(); ++l) {
      Level& L = levels_[l];
      if (!L.rows.empty()) {
        double fl = 0;
        std::string key = std::string("simt:") + FamilyName<T>::v + ":rows";
        for (const auto& j : L.rows) fl += 2.0 * (double)j.rows * j.N * j.K;
        const bool tuned = fl >= ctx_->autotune_min_work;
        if (tuned)
          for (const auto& j : L.rows)
            key += ":" + std::to_string(j.rows) + "x" + std::to_string(j.N) + "x" + std::to_string(j.K);
        const int rule = row_tile(ctx_, L.rows);
        auto go = [&](int i) {
          const int t = i == 0 ? rule : i <= rule ? i - 1 : i;
          KernelScope ks(ctx_, FamilyName<T>::v, fl, 0.0);
          launch_rows<T>(ctx_, t, L.first[t].back(), RowJob<T>{}, L.drows, L.dfirst[t], (int)L.rows.size());
        };
        if (tuned) tune(ctx_, key, RowTiles<T>::n, fl, go);
        else go(0);
      }
      for (int v : L.verts) contract_table(v);
    }
    if (!norms_.empty()) {
      int n = 1;
      for (const auto& m : norms_) n = std::max(n, m.rows);
      k_norm_rows<T><<<dim3(grid_for(n, 32, 1024), (unsigned)norms_.size()), 256, 0, ctx_->stream>>>(dnorms_);
      TNFA_LAUNCH_CHECK();
    }
  }

  // Points [p0, p0 + n) of the call, X the chunk's coordinates.
  void points(const double* X, int n, void* out, int kind, int64_t Pout, int64_t pofs) {
    if (ncodes_ > 0)
      launch_digitize(ctx_, X, ncols_, n, druns_, (int)runs_.size(), ncodes_, codes_, Pc_, err_);
    for (int v : tree_.order)
      if (!tree_.v[v].tabled) contract_points(v, n);
    centre(X, n, out, kind, Pout, pofs);
  }

 private:
  struct Level {
    std::vector<RowJob<T>> rows;
    std::vector<int> verts;  // table vertices of the multi-child kernels
    RowJob<T>* drows = nullptr;
    std::vector<int> first[3];
    int* dfirst[3] = {nullptr, nullptr, nullptr};
  };

  size_t table_bytes() const {
    double b = 0;
    for (int v = 0; v < topo_.V; ++v) {
      const EvalVertex& e = tree_.v[v];
      if (e.tabled && !e.leaf) b += (double)e.N * (e.chi * sizeof(T) + 4);
      if (e.absorb) b += absorbed_rows(v) * (e.W / tree_chi(e.kids.back(), v) * sizeof(T) + 4);
      if (e.moved) b += (double)topo_.size(v) * sizeof(T);
    }
    return (size_t)std::min(b, 1e18);
  }
  int tree_chi(int w, int) const { return tree_.v[w].chi; }
  double absorbed_rows(int v) const {
    return (double)topo_.site_dim[v] * (double)tree_.v[tree_.v[v].kids.back()].N;
  }

  // Codes, message slots and table levels of the schedule.
  void plan() {
    const int V = topo_.V;
    slot_.assign(V, -1);
    mult_.assign(V, 1);
    key_slot_.assign(V, -1);
    row_slot_.assign(V, -1);
    msg_.assign(V, -1);
    npp_ = 0;
    for (int v = 0; v < V; ++v) npp_ += !tree_.v[v].tabled;
    int n = 0;
    for (int v : tree_.order) {
      const EvalVertex& e = tree_.v[v];
      if (e.tabled) continue;
      const int ab = e.absorb ? e.kids.back() : -1;
      if (e.absorb || topo_.site_dim[v] > 1) {
        key_slot_[v] = slot_[v] = n++;
        mult_[v] = e.absorb ? (int)tree_.v[ab].N : 1;
        if (e.absorb) assign(ab, slot_[v], 1);
      } else {
        slot_[v] = -2;  // one site value, no digits
      }
      for (int w : e.kids)
        if (w != ab && tree_.v[w].tabled) assign(w, row_slot_[w] = n++, 1);
    }
    for (const auto& c : tree_.comps)
      for (int v : {c.a, c.b})
        if (v >= 0 && tree_.v[v].tabled) assign(v, row_slot_[v] = n++, 1);
    nslots_ = n;
    // all sides are tables: the centre kernel takes the digits itself, as long
    // as its shared memory holds them
    fused_ = npp_ == 0 && n <= 16 && prog_.size() <= 256;
    ncodes_ = fused_ ? 0 : n;
    runs_ = make_runs(prog_, slot_, mult_);
    // message slots (rows per point), reused once read; the output's is taken
    // before the kids' are given back, so it never shares memory with them
    std::vector<int> free_slots;
    nmsg_ = 0;
    msg_chi_ = 1;
    for (int v : tree_.order) {
      const EvalVertex& e = tree_.v[v];
      if (e.tabled) continue;
      if (free_slots.empty()) free_slots.push_back(nmsg_++);
      msg_[v] = free_slots.back();
      free_slots.pop_back();
      msg_chi_ = std::max(msg_chi_, e.chi);
      for (int w : e.kids)
        if (!tree_.v[w].tabled) free_slots.push_back(msg_[w]);
    }
    max_group_ = 1;
    for (int v = 0; v < V; ++v)
      if (!tree_.v[v].tabled)
        max_group_ = std::max<int64_t>(max_group_, tree_.v[v].absorb ? (int64_t)absorbed_rows(v) : topo_.site_dim[v]);
    // levels
    lvl_.assign(V, 0);
    lvl_m_.assign(V, 0);
    int top = 0;
    for (int v : tree_.order) {
      const EvalVertex& e = tree_.v[v];
      if (e.leaf) continue;
      int l = 0;
      for (size_t i = 0; i < e.kids.size(); ++i) {
        const bool ab = e.absorb && i + 1 == e.kids.size();
        if (ab) lvl_m_[v] = lvl_[e.kids[i]] + 1;
        l = std::max(l, ab ? lvl_m_[v] : tree_.v[e.kids[i]].tabled ? lvl_[e.kids[i]] : 0);
      }
      if (e.tabled) lvl_[v] = l + 1;
      top = std::max({top, lvl_m_[v], e.tabled ? lvl_[v] : 0});
    }
    levels_.assign(top + 1, Level{});
    for (int v : tree_.order) {
      const EvalVertex& e = tree_.v[v];
      if (e.leaf) continue;
      if (e.absorb) levels_[lvl_m_[v]].rows.emplace_back();
      if (!e.tabled) continue;
      if (row_form(v)) levels_[lvl_[v]].rows.emplace_back();
      else levels_[lvl_[v]].verts.push_back(v);
    }
  }
  // One kid besides the absorbed one: the row-gather kernel.
  bool row_form(int v) const {
    const EvalVertex& e = tree_.v[v];
    return !e.tensor && (int)e.kids.size() - (e.absorb ? 1 : 0) == 1;
  }
  // Digit codes of everything below v: v's site value first, then the absorbed
  // kid, then the others in order, the last one fastest.
  void assign(int v, int s, int64_t m) {
    const EvalVertex& e = tree_.v[v];
    const int nk = (int)e.kids.size() - (e.absorb ? 1 : 0);
    for (int i = nk - 1; i >= 0; --i) {
      assign(e.kids[i], s, m);
      m *= tree_.v[e.kids[i]].N;
    }
    if (e.absorb) {
      assign(e.kids.back(), s, m);
      m *= tree_.v[e.kids.back()].N;
    }
    slot_[v] = s;
    mult_[v] = (int)m;
  }

  void lay_out(Carve& c, int64_t pc) {
    const int V = topo_.V;
    err_ = c.take<int>(1);
    // the job tables (sizes known from the plan)
    druns_ = c.take<DigitRun>(runs_.size());
    blob_ = (unsigned char*)druns_;
    moves_.clear();
    int nmove = 0, nnorm = 0;
    for (int v = 0; v < V; ++v) nmove += needs_move(v);
    for (const auto& cc : tree_.comps)
      for (int v : {cc.a, cc.b}) nnorm += v >= 0 && tree_.v[v].tabled && !tree_.v[v].leaf;
    dmoves_ = c.take<MoveJob>(nmove);
    dnorms_ = c.take<NormJob<T>>(nnorm);
    dcentre_ = c.take<CentreJob<T>>(tree_.comps.size());
    for (auto& L : levels_) {
      L.drows = c.take<RowJob<T>>(L.rows.size());
      for (int t = 0; t < RowTiles<T>::n; ++t) L.dfirst[t] = c.take<int>(L.rows.size() + 1);
    }
    tmeta_.assign(V, nullptr);
    ttile_.assign(V, 0);
    for (const auto& L : levels_)
      for (int v : L.verts) tmeta_[v] = c.take<int>(group_meta_ints(table_groups(v)));
    blob_bytes_ = c.used - (size_t)(blob_ - c.base);
    // tensors and tables
    ten_.assign(V, nullptr);
    tab_.assign(V, nullptr);
    tabe_.assign(V, nullptr);
    abs_.assign(V, nullptr);
    abse_.assign(V, nullptr);
    for (int v = 0; v < V; ++v) {
      const EvalVertex& e = tree_.v[v];
      ten_[v] = needs_move(v) ? c.take<T>(topo_.size(v)) : const_cast<T*>(tensors_ + topo_.off[v]);
      if (e.leaf) {
        tab_[v] = ten_[v];
      } else if (e.tabled) {
        tab_[v] = c.take<T>((size_t)e.N * e.chi);
        tabe_[v] = c.take<int>(e.N);
      }
      if (e.absorb) {
        const int64_t r = (int64_t)absorbed_rows(v);
        abs_[v] = c.take<T>((size_t)(r * (int64_t)(e.W / tree_.v[e.kids.back()].chi)));
        abse_[v] = c.take<int>(r);
      }
    }
    // per point
    codes_ = c.take<int>((size_t)ncodes_ * pc);
    perm_ = c.take<int>(npp_ ? pc : 0);
    meta_ = c.take<int>(npp_ ? group_meta_ints((int)max_group_) : 0);
    mval_ = c.take<T>((size_t)nmsg_ * pc * msg_chi_);
    mexp_ = c.take<int>((size_t)nmsg_ * pc);
    ld_ = pc;
  }
  bool needs_move(int v) const { return tree_.v[v].moved; }
  int table_groups(int v) const {
    return tree_.v[v].absorb ? (int)absorbed_rows(v) : topo_.site_dim[v];
  }

  RowIdx table_row(int div, int64_t mod) const {
    RowIdx r;
    r.div = div;
    r.mod = (int)mod;
    return r;
  }

  void fill_blob() {
    host_.assign(blob_bytes_, 0);
    auto put = [&](const void* dev, const void* src, size_t n) {
      if (n) std::memcpy(host_.data() + ((const unsigned char*)dev - blob_), src, n);
    };
    put(druns_, runs_.data(), runs_.size() * sizeof(DigitRun));
    moves_.clear();
    norms_.clear();
    for (int v = 0; v < topo_.V; ++v) {
      const EvalVertex& e = tree_.v[v];
      if (!needs_move(v)) continue;
      std::vector<int> shape{topo_.site_dim[v], topo_.link[v]};
      for (int c : topo_.children[v]) shape.push_back(topo_.link[c]);
      TNFA_CHECK(shape.size() <= (size_t)MOVE_MAXD, TNFA_ERR_UNSUPPORTED, "vertex degree too high");
      std::vector<int64_t> str(shape.size(), 1);
      for (int i = (int)shape.size() - 2; i >= 0; --i) str[i] = str[i + 1] * shape[i + 1];
      MoveJob m{};
      m.src = tensors_ + topo_.off[v];
      m.dst = ten_[v];
      m.n = topo_.size(v);
      m.nd = (int)e.axes.size();
      for (int i = 0; i < m.nd; ++i) {
        m.dim[i] = shape[e.axes[i]];
        m.str[i] = str[e.axes[i]];
      }
      moves_.push_back(m);
    }
    put(dmoves_, moves_.data(), moves_.size() * sizeof(MoveJob));
    std::vector<CentreJob<T>> cj;
    for (const auto& c : tree_.comps) {
      CentreJob<T> j{};
      j.chi = tree_.v[c.a].chi;
      j.a = side(c.a);
      if (c.b >= 0) j.b = side(c.b);
      cj.push_back(j);
      for (int v : {c.a, c.b})
        if (v >= 0 && tree_.v[v].tabled && !tree_.v[v].leaf)
          norms_.push_back({tab_[v], tabe_[v], (int)tree_.v[v].N, tree_.v[v].chi});
    }
    put(dcentre_, cj.data(), cj.size() * sizeof(CentreJob<T>));
    put(dnorms_, norms_.data(), norms_.size() * sizeof(NormJob<T>));
    centre_chi_ = 1;
    centre_vec_ = true;
    constexpr int vec = 16 / sizeof(T);
    for (const auto& j : cj) {
      centre_chi_ = std::max(centre_chi_, j.chi);
      centre_vec_ &= j.chi % vec == 0 && ((uintptr_t)j.a.ptr & 15) == 0 && ((uintptr_t)j.b.ptr & 15) == 0;
    }
    for (auto& L : levels_) L.rows.clear();
    for (int v : tree_.order) {
      const EvalVertex& e = tree_.v[v];
      if (e.leaf) continue;
      if (e.absorb) {
        const int w = e.kids.back();
        const EvalVertex& k = tree_.v[w];
        RowJob<T> j{};
        j.A = tab_[w];
        j.Aexp = tabe_[w];
        j.aidx = table_row(1, k.N);
        j.B = ten_[v];
        j.out = abs_[v];
        j.out_exp = abse_[v];
        j.K = k.chi;
        j.N = (int)(e.W / k.chi);
        j.rpg = (int)k.N;
        j.rows = topo_.site_dim[v] * j.rpg;
        levels_[lvl_m_[v]].rows.push_back(j);
      }
      if (e.tabled && row_form(v)) {
        const int w = e.kids[0];
        const EvalVertex& k = tree_.v[w];
        RowJob<T> j{};
        j.A = tab_[w];
        j.Aexp = tabe_[w];
        j.aidx = table_row(1, k.N);
        j.B = e.absorb ? abs_[v] : ten_[v];
        j.gexp = e.absorb ? abse_[v] : nullptr;
        j.out = tab_[v];
        j.out_exp = tabe_[v];
        j.K = k.chi;
        j.N = e.chi;
        j.rpg = (int)k.N;
        j.rows = (int)e.N;
        levels_[lvl_[v]].rows.push_back(j);
      }
      if (tmeta_[v]) {  // uniform groups of a multi-child table
        const int ng = table_groups(v), m = (int)(e.N / ng);
        std::vector<int> g(group_meta_ints(ng));
        const int tp = ttile_[v] = table_tile_rows(v);
        for (int i = 0; i < ng; ++i) {
          g[i] = i * m;
          g[ng + i] = m;
          g[2 * ng + i] = i * ((m + tp - 1) / tp);
        }
        g[3 * ng] = ng * ((m + tp - 1) / tp);
        put(tmeta_[v], g.data(), g.size() * sizeof(int));
      }
    }
    for (auto& L : levels_) {
      put(L.drows, L.rows.data(), L.rows.size() * sizeof(RowJob<T>));
      for (int t = 0; t < RowTiles<T>::n; ++t) {
        L.first[t].assign(1, 0);
        int64_t b = 0;
        for (const auto& j : L.rows) {
          b += row_blocks(j, t);
          TNFA_CHECK(b < (int64_t(1) << 31), TNFA_ERR_UNSUPPORTED, "contraction too large");
          L.first[t].push_back((int)b);
        }
        put(L.dfirst[t], L.first[t].data(), L.first[t].size() * sizeof(int));
      }
    }
  }

  CentreSide<T> side(int v) const {
    const EvalVertex& e = tree_.v[v];
    CentreSide<T> s{};
    s.slot = -1;
    if (e.tabled) {
      s.ptr = tab_[v];
      s.exps = tabe_[v];
      if (fused_) s.slot = row_slot_[v];
      else s.idx.codes = codes_ + (int64_t)row_slot_[v] * ld_;
      s.scale = e.leaf;
    } else {
      s.ptr = mval_ + (int64_t)msg_[v] * ld_ * msg_chi_;
      s.exps = mexp_ + (int64_t)msg_[v] * ld_;
      s.scale = 1;
    }
    return s;
  }

  // The multi-child job of vertex v (table rows or points), without groups.
  VertexJob<T> vertex_job(int v) const {
    const EvalVertex& e = tree_.v[v];
    VertexJob<T> j{};
    const int nk = (int)e.kids.size() - (e.absorb ? 1 : 0);
    TNFA_CHECK(nk <= EVAL_MAXC, TNFA_ERR_UNSUPPORTED,
               "vertex degree above " + std::to_string(EVAL_MAXC) + " children");
    j.nchild = nk;
    int64_t K = 1;
    int div = 1;
    for (int i = nk - 1; i >= 0; --i) {
      const EvalVertex& k = tree_.v[e.kids[i]];
      ChildSrc<T>& s = j.ch[i];
      s.dim = k.chi;
      K *= k.chi;
      if (k.tabled) {
        s.ptr = tab_[e.kids[i]];
        s.exps = tabe_[e.kids[i]];
        if (e.tabled) {
          s.idx.div = div;
          s.idx.mod = (int)k.N;
          div *= (int)k.N;
        } else {
          s.idx.codes = codes_ + (int64_t)row_slot_[e.kids[i]] * ld_;
        }
      } else {
        s.ptr = mval_ + (int64_t)msg_[e.kids[i]] * ld_ * msg_chi_;
        s.exps = mexp_ + (int64_t)msg_[e.kids[i]] * ld_;
      }
    }
    TNFA_CHECK(K < (int64_t(1) << 31), TNFA_ERR_UNSUPPORTED, "contraction too large");
    j.K = (int)K;
    j.chi_a = e.chi;
    j.B = e.absorb ? abs_[v] : ten_[v];
    j.gexp = e.absorb ? abse_[v] : nullptr;
    j.site_dim = j.ngroups = e.absorb ? (int)absorbed_rows(v) : topo_.site_dim[v];
    if (e.tabled) {
      j.out = tab_[v];
      j.out_exp = tabe_[v];
      j.Pc = (int)e.N;
    } else {
      j.out = mval_ + (int64_t)msg_[v] * ld_ * msg_chi_;
      j.out_exp = mexp_ + (int64_t)msg_[v] * ld_;
    }
    return j;
  }
  int job_sumdim(int v) const {
    const EvalVertex& e = tree_.v[v];
    int s = 0;
    for (size_t i = 0; i + (e.absorb ? 1 : 0) < e.kids.size(); ++i) s += tree_.v[e.kids[i]].chi;
    return s;
  }
  std::vector<GemmTile> vertex_tiles(int v, std::string* key) const {
    const EvalVertex& e = tree_.v[v];
    if (e.tensor || e.chi <= 16) return {};
    *key = std::string("simt:") + FamilyName<T>::v + ":" + std::to_string(e.chi) + ":";
    const int nk = (int)e.kids.size() - (e.absorb ? 1 : 0);
    for (int i = 0; i < nk; ++i)
      *key += std::to_string(tree_.v[e.kids[i]].chi) + (i + 1 < nk ? "x" : "");
    return gemm_tile_candidates(e.chi, job_sumdim(v), sizeof(T));
  }
  int table_tile_rows(int v) const {
    if (tree_.v[v].tensor) return use_tc_ ? tc_tile_rows() : oz_tile_rows();
    std::string key;
    const auto cand = vertex_tiles(v, &key);
    if (cand.empty()) return contract_tile_rows(tree_.v[v].chi, job_sumdim(v), sizeof(T));
    const int kept = tuned_choice(ctx_, key);
    return cand[kept >= 0 ? kept : 0].tp;
  }

  // Runs a multi-child job whose groups are in meta with tile rows tp.
  void contract_vertex(int v, VertexJob<T>& j, int* meta, bool keyed, int tp) {
    const int ng = j.ngroups;
    j.grp_off = meta;
    j.grp_cnt = meta + ng;
    j.tile_start = meta + 2 * ng;
    if (tree_.v[v].tensor) {
      if constexpr (std::is_same<T, float>::value) {
        tc_contract_vertex(ctx_, net_, v, j, tp, err_);
        return;
      }
      if constexpr (std::is_same<T, double>::value) {
        oz_contract_vertex(ctx_, net_, v, j, tp, err_);
        return;
      }
    }
    std::string key;
    const auto cand = vertex_tiles(v, &key);
    if (cand.empty()) {
      launch_contract<T>(ctx_, j, j.Pc);
      return;
    }
    int cur = tp;
    tune(ctx_, key, (int)cand.size(), 2.0 * j.Pc * (double)j.K * j.chi_a, [&](int i) {
      if (cand[i].tp != cur) {  // tile table for this candidate's rows per tile
        launch_retile(ctx_, keyed, j.Pc, ng, cand[i].tp, meta);
        cur = cand[i].tp;
      }
      launch_contract<T>(ctx_, j, j.Pc, &cand[i]);
    });
  }

  void contract_table(int v) {
    VertexJob<T> j = vertex_job(v);
    contract_vertex(v, j, tmeta_[v], true, ttile_[v]);
  }

  RowJob<T> point_rows(int v, int n) const {
    const EvalVertex& e = tree_.v[v];
    const int w = e.kids[0];
    const EvalVertex& k = tree_.v[w];
    RowJob<T> j{};
    if (k.tabled) {
      j.A = tab_[w];
      j.Aexp = tabe_[w];
      j.aidx.codes = codes_ + (int64_t)row_slot_[w] * ld_;
    } else {
      j.A = mval_ + (int64_t)msg_[w] * ld_ * msg_chi_;
      j.Aexp = mexp_ + (int64_t)msg_[w] * ld_;
    }
    j.B = e.absorb ? abs_[v] : ten_[v];
    j.gexp = e.absorb ? abse_[v] : nullptr;
    j.out = mval_ + (int64_t)msg_[v] * ld_ * msg_chi_;
    j.out_exp = mexp_ + (int64_t)msg_[v] * ld_;
    j.K = k.chi;
    j.N = e.chi;
    j.rows = n;
    j.ngroups = e.absorb ? (int)absorbed_rows(v) : topo_.site_dim[v];
    j.grp_off = meta_;
    j.grp_cnt = meta_ + j.ngroups;
    j.tile_start = meta_ + 2 * j.ngroups;
    return j;
  }

  void contract_points(int v, int n) {
    const EvalVertex& e = tree_.v[v];
    const int* key = key_slot_[v] >= 0 ? codes_ + (int64_t)key_slot_[v] * ld_ : nullptr;
    if (!row_form(v)) {
      VertexJob<T> j = vertex_job(v);
      j.Pc = n;
      const int tp = table_tile_rows(v);
      j.perm = launch_group(ctx_, key, n, j.ngroups, tp, meta_, perm_);
      contract_vertex(v, j, meta_, key != nullptr, tp);
      return;
    }
    RowJob<T> j = point_rows(v, n);
    const double fl = 2.0 * n * (double)j.N * j.K;
    const int rule = group_tile(j);
    const std::string tkey = std::string("simt:") + FamilyName<T>::v + ":points:" + std::to_string(j.N) + "x" +
                             std::to_string(j.K) + ":" + std::to_string(j.ngroups > 1024 ? n / j.ngroups : 0);
    const int kept = tuned_choice(ctx_, tkey);
    auto tile_of = [&](int i) { return i == 0 ? rule : i <= rule ? i - 1 : i; };
    int cur = 8 * RowTiles<T>::rm[tile_of(kept >= 0 ? kept : 0)];
    j.perm = launch_group(ctx_, key, n, j.ngroups, cur, meta_, perm_);
    tune(ctx_, tkey, RowTiles<T>::n, fl, [&](int i) {
      const int t = tile_of(i), tp = 8 * RowTiles<T>::rm[t];
      if (tp != cur) {
        launch_retile(ctx_, key != nullptr, n, j.ngroups, tp, meta_);
        cur = tp;
      }
      KernelScope ks(ctx_, FamilyName<T>::v, fl, (double)sizeof(T) * n * (j.N + j.K));
      launch_rows<T>(ctx_, t, row_blocks(j, t), j, nullptr, nullptr, 0);
    });
  }
  int group_tile(const RowJob<T>& j) const { return row_tile<T>(ctx_, {j}); }

  void centre(const double* X, int n, void* out, int kind, int64_t Pout, int64_t pofs) {
    const int ns = fused_ ? nslots_ : 0;
    const size_t sm = 256 * (sizeof(T) + 4) + (size_t)ns * 1024 + (fused_ ? runs_.size() * sizeof(DigitRun) : 0);
    KernelScope ks(ctx_, "centre", 2.0 * n * centre_chi_, (double)n * (ncols_ * 8.0 + 8.0));
    const unsigned grid = grid_for(n, 256, ctx_->sm_count * 8);
    auto go = [&](auto kern) {
      kern<<<grid, 256, sm, ctx_->stream>>>(X, ncols_, n, druns_, (int)runs_.size(), ns, dcentre_,
                                           (int)tree_.comps.size(), out, kind, Pout, pofs, err_);
    };
    constexpr int vec = 16 / sizeof(T);
    if constexpr (vec > 1) {
      if (centre_vec_) {
        const int lanes = (centre_chi_ + vec - 1) / vec;
        if (lanes <= 1) go(k_centre<T, 1, vec>);
        else if (lanes <= 2) go(k_centre<T, 2, vec>);
        else if (lanes <= 4) go(k_centre<T, 4, vec>);
        else go(k_centre<T, 8, vec>);
        TNFA_LAUNCH_CHECK();
        return;
      }
    }
    if (centre_chi_ <= 2) go(k_centre<T, 1, 1>);
    else if (centre_chi_ <= 8) go(k_centre<T, 2, 1>);
    else go(k_centre<T, 8, 1>);
    TNFA_LAUNCH_CHECK();
  }

  tnfa_ctx* ctx_;
  const tnfa_net* net_;
  const T* tensors_;
  const Topo& topo_;
  const std::vector<DigitRef>& prog_;
  int ncols_;
  int64_t P_;
  bool use_tc_, use_oz_;
  EvalTree tree_;
  std::vector<int> ttile_;  // tile rows that the group table of a table vertex was made for
  std::vector<int> slot_, mult_, key_slot_, row_slot_, msg_, lvl_, lvl_m_;
  std::vector<DigitRun> runs_;
  std::vector<Level> levels_;
  int nslots_ = 0, ncodes_ = 0, nmsg_ = 0, msg_chi_ = 1, npp_ = 0, Pc_ = 0, centre_chi_ = 1;
  int64_t max_group_ = 1, ld_ = 0;
  bool fused_ = false, centre_vec_ = false;
  size_t per_point_ = 0, blob_bytes_ = 0;
  std::vector<unsigned char> host_;
  std::vector<MoveJob> moves_;
  std::vector<NormJob<T>> norms_;
  // scratch
  int* err_ = nullptr;
  unsigned char* blob_ = nullptr;
  DigitRun* druns_ = nullptr;
  MoveJob* dmoves_ = nullptr;
  NormJob<T>* dnorms_ = nullptr;
  CentreJob<T>* dcentre_ = nullptr;
  std::vector<int*> tmeta_, tabe_, abse_;
  std::vector<T*> ten_, tab_, abs_;
  int *codes_ = nullptr, *perm_ = nullptr, *meta_ = nullptr, *mexp_ = nullptr;
  T* mval_ = nullptr;
};

static size_t out_elem_size(int out_kind) {
  return out_kind == TNFA_OUT_F64 ? 8 : out_kind == TNFA_OUT_F32 ? 4 : out_kind == TNFA_OUT_F32_SCALED ? 8 : 16;
}

static void check_eval_error(tnfa_ctx* ctx, const int* derr) {
  int herr = 0;
  TNFA_CUDA(cudaMemcpyAsync(&herr, derr, 4, cudaMemcpyDeviceToHost, ctx->stream));
  TNFA_CUDA(cudaStreamSynchronize(ctx->stream));
  TNFA_CHECK((herr & 2) == 0, TNFA_ERR_TIMEOUT,
             "a tensor-core pipeline wait ran out of its iteration budget");
  TNFA_CHECK(herr == 0, TNFA_ERR_DOMAIN,
             "a coordinate is negative or not finite (the digit map needs x >= 0)");
}

template <class T>
static void evaluate_impl(tnfa_ctx* ctx, const tnfa_net* net, const T* tensors, const double* X,
                          int64_t P, int ncols, const std::vector<DigitRef>& prog, int xmem,
                          void* out, int out_kind, int out_mem, bool use_tc,
                          bool use_oz = false) {
  const size_t out_elem = out_elem_size(out_kind);
  const size_t staged = (xmem == TNFA_MEM_HOST ? ncols * 8 : 0) + (out_mem == TNFA_MEM_HOST ? out_elem : 0);
  // small bonds everywhere: the whole tree per thread in one launch
  const FusedPlan F = make_fused_plan(net->topo, sizeof(T), prog.size(), P);
  std::unique_ptr<EvalEngine<T>> E;
  std::vector<DigitRun> runs;
  int64_t Pcap;
  if (F.ok) {
    runs = make_fused_runs(net->topo, prog);
    Pcap = staged ? std::max<int64_t>(256, (int64_t)(ctx->eval_budget / staged) / 256 * 256) : int64_t(1) << 30;
  } else {
    E.reset(new EvalEngine<T>(ctx, net, tensors, prog, ncols, P, use_tc, use_oz, ctx->eval_budget));
    Pcap = E->chunk();
    if (staged) Pcap = std::min(Pcap, std::max<int64_t>(256, (int64_t)(ctx->eval_budget / staged) / 256 * 256));
  }
  Pcap = std::max<int64_t>(1, std::min<int64_t>({P, Pcap, int64_t(1) << 30}));
  DBuf dX(ctx, xmem == TNFA_MEM_HOST ? (size_t)Pcap * ncols * 8 : 0);
  DBuf dout(ctx, out_mem == TNFA_MEM_HOST ? (size_t)Pcap * out_elem : 0);
  DBuf derr(ctx, 4), arena, dprog, dsteps;
  int* err;
  if (F.ok) {
    dprog = DBuf(ctx, std::max<size_t>(runs.size(), 1) * sizeof(DigitRun));
    h2d(ctx, dprog.p, runs.data(), runs.size() * sizeof(DigitRun));
    dsteps = DBuf(ctx, F.steps.size() * sizeof(FusedStep));
    h2d(ctx, dsteps.p, F.steps.data(), F.steps.size() * sizeof(FusedStep));
    err = derr.as<int>();
    TNFA_CUDA(cudaMemsetAsync(err, 0, 4, ctx->stream));
  } else {
    E->set_chunk((int)Pcap);
    arena = DBuf(ctx, E->scratch(Pcap));
    E->bind(arena.p);
    E->upload();
    E->tables();
    err = E->err_flag();
  }
  for (int64_t p0 = 0; p0 < P; p0 += Pcap) {
    const int Pc = (int)std::min<int64_t>(Pcap, P - p0);
    const double* Xc = X + p0 * ncols;
    if (xmem == TNFA_MEM_HOST) {
      TNFA_CUDA(cudaMemcpyAsync(dX.p, Xc, (size_t)Pc * ncols * 8, cudaMemcpyHostToDevice, ctx->stream));
      Xc = dX.as<double>();
    }
    void* o = out_mem == TNFA_MEM_HOST ? dout.p : out;
    const int64_t Pout = out_mem == TNFA_MEM_HOST ? Pc : P, pofs = out_mem == TNFA_MEM_HOST ? 0 : p0;
    if (F.ok)
      launch_fused<T>(ctx, F, dsteps.as<FusedStep>(), tensors, net->topo, Xc, ncols, Pc,
                      dprog.as<DigitRun>(), (int)runs.size(), o, out_kind, Pout, pofs, err);
    else
      E->points(Xc, Pc, o, out_kind, Pout, pofs);
    if (out_mem == TNFA_MEM_HOST) {
      if (out_kind == TNFA_OUT_F32_SCALED) {
        TNFA_CUDA(cudaMemcpyAsync((float*)out + p0, dout.p, (size_t)Pc * 4, cudaMemcpyDeviceToHost,
                                  ctx->stream));
        TNFA_CUDA(cudaMemcpyAsync((int*)((float*)out + P) + p0, (float*)dout.p + Pc, (size_t)Pc * 4,
                                  cudaMemcpyDeviceToHost, ctx->stream));
      } else {
        TNFA_CUDA(cudaMemcpyAsync((char*)out + p0 * out_elem, dout.p, (size_t)Pc * out_elem,
                                  cudaMemcpyDeviceToHost, ctx->stream));
      }
    }
  }
  check_eval_error(ctx, err);
}

}  // namespace tnfa

using namespace tnfa;

extern "C" int tnfa_evaluate(tnfa_ctx* ctx, const tnfa_net* net, const double* X, int64_t n_points,
                             int32_t n_dims, const int32_t* dims, int x_memory, void* out,
                             int out_kind, int out_memory, int precision) {
  TNFA_API_BEGIN(ctx);
  require_ctx(ctx);
  require_net(net, "evaluate");
  TNFA_CHECK(n_points >= 0, TNFA_ERR_INVALID_ARGUMENT, "n_points < 0");
  if (n_points == 0) return TNFA_OK;
  TNFA_CHECK(X && out && (n_dims == 0 || dims), TNFA_ERR_INVALID_ARGUMENT, "null X, out or dims");
  TNFA_CHECK(n_dims >= 0 && n_dims <= 64, TNFA_ERR_INVALID_ARGUMENT, "n_dims out of range");
  TNFA_CHECK(x_memory == TNFA_MEM_HOST || x_memory == TNFA_MEM_DEVICE, TNFA_ERR_INVALID_ARGUMENT,
             "bad x_memory");
  TNFA_CHECK(out_memory == TNFA_MEM_HOST || out_memory == TNFA_MEM_DEVICE,
             TNFA_ERR_INVALID_ARGUMENT, "bad out_memory");
  for (int v = 0; v < net->topo.V; ++v)
    TNFA_CHECK(net->topo.site_dim[v] <= 256, TNFA_ERR_UNSUPPORTED, "site dimension above 256");
  int ncols = 0;
  std::vector<DigitRef> prog = make_digit_program(net->topo, n_dims, dims, &ncols);
  if (net->dtype == TNFA_C128) {
    TNFA_CHECK(out_kind == TNFA_OUT_C128, TNFA_ERR_DTYPE, "complex networks need TNFA_OUT_C128");
    TNFA_CHECK(precision == TNFA_PREC_F64, TNFA_ERR_UNSUPPORTED,
               "complex networks evaluate in TNFA_PREC_F64 only");
    evaluate_impl<cplx>(ctx, net, (const cplx*)net->d, X, n_points, ncols, prog, x_memory, out,
                        out_kind, out_memory, false);
  } else {
    TNFA_CHECK(out_kind == TNFA_OUT_F64 || out_kind == TNFA_OUT_F32 ||
                   out_kind == TNFA_OUT_F32_SCALED,
               TNFA_ERR_DTYPE, "real networks need a real output kind");
    if (precision == TNFA_PREC_F64) {
      TNFA_CHECK(net->dtype == TNFA_F64, TNFA_ERR_DTYPE, "TNFA_PREC_F64 needs an FP64 network");
      evaluate_impl<double>(ctx, net, (const double*)net->d, X, n_points, ncols, prog, x_memory,
                            out, out_kind, out_memory, false);
    } else if (precision == TNFA_PREC_MIXED) {
      // FP64 messages; two-child vertices of tensor-core shape take the
      // error-free sliced products, the rest the FP64 kernels
      oz_prepare_net(ctx, net);
      const double* t64 =
          net->dtype == TNFA_F64 ? (const double*)net->d : (const double*)net->d_f64;
      evaluate_impl<double>(ctx, net, t64, X, n_points, ncols, prog, x_memory, out, out_kind,
                            out_memory, false, true);
    } else if (precision == TNFA_PREC_F32 || precision == TNFA_PREC_MIXED_FAST) {
      const float* t32;
      if (net->dtype == TNFA_F32) {
        t32 = (const float*)net->d;
      } else {
        if (!net->d_f32) {
          net->d_f32 = dalloc(ctx, (size_t)net->topo.n_elem * 4);
          convert_f64_to_f32(ctx, (const double*)net->d, (float*)net->d_f32, net->topo.n_elem);
        }
        t32 = (const float*)net->d_f32;
      }
      if (precision == TNFA_PREC_MIXED_FAST) tc_prepare_net(ctx, net);
      evaluate_impl<float>(ctx, net, t32, X, n_points, ncols, prog, x_memory, out, out_kind,
                           out_memory, precision == TNFA_PREC_MIXED_FAST);
    } else {
      fail(TNFA_ERR_INVALID_ARGUMENT, "unknown precision");
    }
  }
  TNFA_API_END
}

// ------------------------------------------ evaluation without allocation ----
// tnfa_evaluate_noalloc: the same digitize / group / contract / combine
// kernels as tnfa_evaluate, with every scratch buffer carved out of one
// file-scope device array instead of the stream-ordered allocator.
#include <array>
#include <mutex>

namespace tnfa {
namespace {

constexpr size_t NOALLOC_BYTES = (size_t)32 << 20;  // 32 MiB, held by every device
__device__ __align__(256) unsigned char noalloc_scratch[NOALLOC_BYTES];

// Host code cannot use the array's name as a device address; this looks the
// address up once per device (with that device current) and caches it.
unsigned char* noalloc_base(int device) {
  static std::mutex mu;
  static std::vector<unsigned char*> addr;
  std::lock_guard<std::mutex> lock(mu);
  if ((int)addr.size() <= device) addr.resize(device + 1, nullptr);
  if (!addr[device]) {
    // the look-up needs `device` current; the caller's current device is
    // put back afterwards
    int prev = -1;
    TNFA_CUDA(cudaGetDevice(&prev));
    if (prev != device) TNFA_CUDA(cudaSetDevice(device));
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, noalloc_scratch);
    if (prev != device) TNFA_CUDA(cudaSetDevice(prev));
    TNFA_CUDA(e);
    addr[device] = (unsigned char*)p;
  }
  return addr[device];
}

// Scratch bytes by which a request is accepted: digit program, fused schedule,
// digits, permutation, group tables, error flag, message slots of every point
// and root values, in 256-byte pieces.  The calls that fit are part of the
// interface; the schedule itself works in chunks that fit (FixedRun).
template <class T>
size_t noalloc_bytes(const tnfa_net* net, int64_t P, size_t prog_entries) {
  const Topo& Tp = net->topo;
  const FusedPlan F = make_fused_plan(Tp, sizeof(T), prog_entries, P);
  const EvalPlan plan = make_plan(Tp);
  const size_t nroots = plan.roots.size();
  int maxsd = 1;
  for (int v = 0; v < Tp.V; ++v) maxsd = std::max(maxsd, Tp.site_dim[v]);
  std::array<size_t, 10> sizes{prog_entries * 32, 0, 0, 0, 0, 4, 0, 0, 0, 0};
  if (F.ok) {
    sizes[1] = F.steps.size() * sizeof(FusedStep);
  } else {
    sizes[2] = (size_t)Tp.V * P;
    sizes[3] = (size_t)P * 4;
    sizes[4] = group_meta_ints(maxsd) * 4;
    sizes[6] = (size_t)plan.nslots * P * plan.chimax * sizeof(T);
    sizes[7] = (size_t)plan.nslots * P * sizeof(int);
    sizes[8] = nroots * P * sizeof(T);
    sizes[9] = nroots * P * sizeof(int);
  }
  Carve dry;
  for (size_t s : sizes) dry.take<unsigned char>(s);
  return dry.used;
}

// An evaluation over scratch that the caller owns: stage() sends the job
// tables there, enqueue() runs the kernels (and nothing else, so that it can
// be captured).
template <class T>
class FixedRun {
 public:
  FixedRun(tnfa_ctx* ctx, const tnfa_net* net, const T* tensors, const std::vector<DigitRef>& prog, int ncols,
           int64_t P, size_t budget)
      : ctx_(ctx), net_(net), tensors_(tensors), ncols_(ncols), P_(P),
        F_(make_fused_plan(net->topo, sizeof(T), prog.size(), P)) {
    if (F_.ok) {
      runs_ = make_fused_runs(net->topo, prog);
      return;
    }
    E_.reset(new EvalEngine<T>(ctx, net, tensors, prog, ncols, P, false, false, budget));
    int pc = E_->chunk();
    while (pc > 1 && E_->scratch(pc) > budget) pc = std::max(1, pc / 2);
    E_->set_chunk(pc);
  }
  size_t bytes() {
    if (!F_.ok) return E_->scratch(E_->chunk());
    Carve c;
    lay_out(c);
    return c.used + 256;
  }
  void bind(void* base) {
    Carve c;
    c.base = (unsigned char*)base;
    if (F_.ok) lay_out(c);
    else E_->bind(base);
  }
  void stage() {
    if (F_.ok) {
      h2d(ctx_, dprog_, runs_.data(), runs_.size() * sizeof(DigitRun));
      h2d(ctx_, dsteps_, F_.steps.data(), F_.steps.size() * sizeof(FusedStep));
    } else {
      E_->upload();
    }
  }
  int* err_flag() const { return F_.ok ? err_ : E_->err_flag(); }
  void enqueue(const double* X, void* out, int out_kind) {
    TNFA_CUDA(cudaMemsetAsync(err_flag(), 0, 4, ctx_->stream));
    if (F_.ok) {
      launch_fused<T>(ctx_, F_, dsteps_, tensors_, net_->topo, X, ncols_, (int)P_, dprog_, (int)runs_.size(), out,
                      out_kind, P_, 0, err_);
      return;
    }
    E_->tables();
    for (int64_t p0 = 0; p0 < P_; p0 += E_->chunk())
      E_->points(X + p0 * ncols_, (int)std::min<int64_t>(E_->chunk(), P_ - p0), out, out_kind, P_, p0);
  }

 private:
  void lay_out(Carve& c) {
    dprog_ = c.take<DigitRun>(runs_.size());
    dsteps_ = c.take<FusedStep>(F_.steps.size());
    err_ = c.take<int>(1);
  }
  tnfa_ctx* ctx_;
  const tnfa_net* net_;
  const T* tensors_;
  int ncols_;
  int64_t P_;
  FusedPlan F_;
  std::vector<DigitRun> runs_;
  std::unique_ptr<EvalEngine<T>> E_;
  DigitRun* dprog_ = nullptr;
  FusedStep* dsteps_ = nullptr;
  int* err_ = nullptr;
};

template <class T>
void evaluate_noalloc_impl(tnfa_ctx* ctx, const tnfa_net* net, const T* tensors, const double* X, int64_t P,
                           int ncols, const std::vector<DigitRef>& prog, void* out, int out_kind) {
  const size_t need = noalloc_bytes<T>(net, P, prog.size());
  if (need > NOALLOC_BYTES) {
    const size_t per_point = (need - prog.size() * 32) / (size_t)std::max<int64_t>(P, 1) + 1;
    fail(TNFA_ERR_INVALID_ARGUMENT,
         "tnfa_evaluate_noalloc: " + std::to_string(P) + " points need " + std::to_string(need) +
             " bytes of scratch, above the fixed " + std::to_string(NOALLOC_BYTES) +
             "; this network allows about " + std::to_string(NOALLOC_BYTES / per_point) + " points per call");
  }
  FixedRun<T> run(ctx, net, tensors, prog, ncols, P, NOALLOC_BYTES);
  TNFA_CHECK(run.bytes() <= NOALLOC_BYTES, TNFA_ERR_INVALID_ARGUMENT, "scratch overflow");
  run.bind(noalloc_base(ctx->device));
  run.stage();
  run.enqueue(X, out, out_kind);
  check_eval_error(ctx, run.err_flag());
}

}  // namespace
}  // namespace tnfa

extern "C" int tnfa_evaluate_noalloc(tnfa_ctx* ctx, const tnfa_net* net, const double* X,
                                     int64_t n_points, int32_t n_dims, const int32_t* dims,
                                     void* out, int out_kind, int precision) {
  TNFA_API_BEGIN(ctx);
  require_ctx(ctx);
  require_net(net, "evaluate_noalloc");
  TNFA_CHECK(n_points >= 0, TNFA_ERR_INVALID_ARGUMENT, "n_points < 0");
  if (n_points == 0) return TNFA_OK;
  TNFA_CHECK(X && out && (n_dims == 0 || dims), TNFA_ERR_INVALID_ARGUMENT, "null X, out or dims");
  TNFA_CHECK(n_dims >= 0 && n_dims <= 64, TNFA_ERR_INVALID_ARGUMENT, "n_dims out of range");
  TNFA_CHECK(n_points < (int64_t(1) << 31), TNFA_ERR_INVALID_ARGUMENT, "too many points");
  for (int v = 0; v < net->topo.V; ++v)
    TNFA_CHECK(net->topo.site_dim[v] <= 256, TNFA_ERR_UNSUPPORTED, "site dimension above 256");
  int ncols = 0;
  std::vector<DigitRef> prog = make_digit_program(net->topo, n_dims, dims, &ncols);
  if (net->dtype == TNFA_C128) {
    TNFA_CHECK(out_kind == TNFA_OUT_C128 && precision == TNFA_PREC_F64, TNFA_ERR_DTYPE,
               "complex networks: TNFA_OUT_C128 and TNFA_PREC_F64");
    evaluate_noalloc_impl<cplx>(ctx, net, (const cplx*)net->d, X, n_points, ncols, prog, out,
                                out_kind);
  } else {
    TNFA_CHECK(out_kind == TNFA_OUT_F64 || out_kind == TNFA_OUT_F32 ||
                   out_kind == TNFA_OUT_F32_SCALED,
               TNFA_ERR_DTYPE, "real networks need a real output kind");
    if (precision == TNFA_PREC_F64 && net->dtype == TNFA_F64)
      evaluate_noalloc_impl<double>(ctx, net, (const double*)net->d, X, n_points, ncols, prog, out,
                                    out_kind);
    else if (precision == TNFA_PREC_F32 && net->dtype == TNFA_F32)
      evaluate_noalloc_impl<float>(ctx, net, (const float*)net->d, X, n_points, ncols, prog, out,
                                   out_kind);
    else
      fail(TNFA_ERR_UNSUPPORTED,
           "tnfa_evaluate_noalloc computes in the network's own type: TNFA_PREC_F64 on FP64 "
           "networks or TNFA_PREC_F32 on FP32 networks");
  }
  TNFA_API_END
}

// ------------------------------------------------ captured evaluation ----
// tnfa_eval_plan: the no-allocation kernel sequence for fixed device buffers
// (X, out) and a fixed point count, captured once into a CUDA graph over
// scratch the plan owns, then replayed with one graph launch per call.  For
// small batches evaluation is launch-bound (about four launches per vertex),
// and the replay removes the per-launch host cost.
struct tnfa_eval_plan {
  tnfa_ctx* ctx = nullptr;
  const tnfa_net* net = nullptr;
  void* scratch = nullptr;
  int* derr = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  int64_t n_points = 0;
};

namespace tnfa {
namespace {
void plan_free(tnfa_eval_plan* p) {
  if (!p) return;
  if (p->exec) cudaGraphExecDestroy(p->exec);
  if (p->graph) cudaGraphDestroy(p->graph);
  if (p->scratch) cudaFree(p->scratch);
  if (p->ctx) ctx_release(p->ctx);
  delete p;
}

template <class T>
void plan_build(tnfa_eval_plan* p, const T* tensors, const double* X, int ncols,
                const std::vector<DigitRef>& prog, void* out, int out_kind) {
  tnfa_ctx* ctx = p->ctx;
  FixedRun<T> run(ctx, p->net, tensors, prog, ncols, p->n_points, ctx->eval_budget);
  TNFA_CUDA(cudaMalloc(&p->scratch, run.bytes()));
  run.bind(p->scratch);
  p->derr = run.err_flag();
  // one eager run: validates the inputs, sets kernel attributes, stages the
  // job tables in the scratch (where the capture expects them)
  run.stage();
  run.enqueue(X, out, out_kind);
  check_eval_error(ctx, p->derr);
  TNFA_CUDA(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
  ctx->capturing = true;
  try {
    run.enqueue(X, out, out_kind);
  } catch (...) {
    ctx->capturing = false;
    cudaGraph_t g = nullptr;
    cudaStreamEndCapture(ctx->stream, &g);
    if (g) cudaGraphDestroy(g);
    cudaGetLastError();
    throw;
  }
  ctx->capturing = false;
  TNFA_CUDA(cudaStreamEndCapture(ctx->stream, &p->graph));
  TNFA_CUDA(cudaGraphInstantiate(&p->exec, p->graph, 0));
}
}  // namespace
}  // namespace tnfa

extern "C" int tnfa_eval_plan_create(tnfa_ctx* ctx, const tnfa_net* net, const double* X,
                                     int64_t n_points, int32_t n_dims, const int32_t* dims,
                                     void* out, int out_kind, int precision,
                                     tnfa_eval_plan** plan) {
  TNFA_API_BEGIN(ctx);
  require_ctx(ctx);
  require_net(net, "eval_plan_create");
  TNFA_CHECK(plan, TNFA_ERR_INVALID_ARGUMENT, "null plan");
  *plan = nullptr;
  TNFA_CHECK(n_points > 0 && n_points < (int64_t(1) << 31), TNFA_ERR_INVALID_ARGUMENT,
             "n_points must be in [1, 2^31)");
  TNFA_CHECK(X && out && (n_dims == 0 || dims), TNFA_ERR_INVALID_ARGUMENT, "null X, out or dims");
  TNFA_CHECK(n_dims >= 0 && n_dims <= 64, TNFA_ERR_INVALID_ARGUMENT, "n_dims out of range");
  for (int v = 0; v < net->topo.V; ++v)
    TNFA_CHECK(net->topo.site_dim[v] <= 256, TNFA_ERR_UNSUPPORTED, "site dimension above 256");
  int ncols = 0;
  std::vector<DigitRef> prog = make_digit_program(net->topo, n_dims, dims, &ncols);
  tnfa_eval_plan* p = new tnfa_eval_plan;
  p->ctx = ctx;
  ctx->refs += 1;
  p->net = net;
  p->n_points = n_points;
  try {
    if (net->dtype == TNFA_C128) {
      TNFA_CHECK(out_kind == TNFA_OUT_C128 && precision == TNFA_PREC_F64, TNFA_ERR_DTYPE,
                 "complex networks: TNFA_OUT_C128 and TNFA_PREC_F64");
      plan_build<cplx>(p, (const cplx*)net->d, X, ncols, prog, out, out_kind);
    } else {
      TNFA_CHECK(out_kind == TNFA_OUT_F64 || out_kind == TNFA_OUT_F32 ||
                     out_kind == TNFA_OUT_F32_SCALED,
                 TNFA_ERR_DTYPE, "real networks need a real output kind");
      if (precision == TNFA_PREC_F64 && net->dtype == TNFA_F64)
        plan_build<double>(p, (const double*)net->d, X, ncols, prog, out, out_kind);
      else if (precision == TNFA_PREC_F32 && net->dtype == TNFA_F32)
        plan_build<float>(p, (const float*)net->d, X, ncols, prog, out, out_kind);
      else
        fail(TNFA_ERR_UNSUPPORTED,
             "an evaluation plan computes in the network's own type: TNFA_PREC_F64 on FP64 "
             "networks or TNFA_PREC_F32 on FP32 networks");
    }
  } catch (...) {
    plan_free(p);
    throw;
  }
  *plan = p;
  TNFA_API_END
}

extern "C" int tnfa_eval_plan_launch(tnfa_ctx* ctx, tnfa_eval_plan* plan) {
  TNFA_API_BEGIN(ctx);
  require_ctx(ctx);
  TNFA_CHECK(plan && plan->exec && plan->ctx == ctx, TNFA_ERR_INVALID_ARGUMENT,
             "not a plan of this context");
  TNFA_CUDA(cudaGraphLaunch(plan->exec, ctx->stream));
  TNFA_API_END
}

extern "C" int tnfa_eval_plan_check(tnfa_ctx* ctx, tnfa_eval_plan* plan) {
  TNFA_API_BEGIN(ctx);
  require_ctx(ctx);
  TNFA_CHECK(plan && plan->derr && plan->ctx == ctx, TNFA_ERR_INVALID_ARGUMENT,
             "not a plan of this context");
  int herr = 0;
  TNFA_CUDA(cudaMemcpyAsync(&herr, plan->derr, 4, cudaMemcpyDeviceToHost, ctx->stream));
  TNFA_CUDA(cudaStreamSynchronize(ctx->stream));
  TNFA_CHECK(herr == 0, TNFA_ERR_DOMAIN,
             "a coordinate is negative or not finite (the digit map needs x >= 0)");
  TNFA_API_END
}

extern "C" int tnfa_eval_plan_destroy(tnfa_eval_plan* plan) {
  if (!plan) return TNFA_OK;
  cudaStreamSynchronize(plan->ctx->stream);
  tnfa::plan_free(plan);
  return TNFA_OK;
}

// ----------------------------------------------- vector-Jacobian product ----
// d/dT of sum_p dout_p f(x_p).  For vertex v with outside message E_v (the
// contraction of everything but v's subtree, as a vector over v's parent
// bond) and inside messages m_c of its children,
//   dT_v[s][a][c1..ck] += sum_{p: s_v(p) = s} dout_p E_v[p][a] prod_j m_cj[p][c_j].
// Inside messages come from the forward contraction (kept for every vertex);
// E of a child is the same contraction with that child's bond as the output
// (the vertex tensor with the child's axis moved first, E_v as one more input);
// the accumulation treats E_v as one more Kronecker factor and reduces over
// the points of each digit group (split over point tiles, atomics per tile).
#include "linalg.cuh"

namespace tnfa {
namespace {

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

// dT_v[g][k] += sum over the points p of site value g of scale_p * prod_c m_c[p][k_c]
// (k decoded as the mixed-radix tuple of the child entries, last child
// fastest).  Each CTA walks a contiguous run of tiles of tiles_per_cta point
// tiles, keeps its partial sums in registers and adds them to dT once per site
// value it met, so the atomics on the few thousand dT entries stay far from
// the point count.
template <class T, int TP, int KQ>
__global__ void __launch_bounds__(256) k_grad_acc(const VertexJob<T> j, T* __restrict__ dT,
                                                  int tiles_per_cta) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int sumdim = 0;
  for (int c = 0; c < j.nchild; ++c) sumdim += j.ch[c].dim;
  T* rows = (T*)smem_raw;
  T* scale = rows + (int64_t)sumdim * TP;
  int* pts = (int*)(scale + TP);
  int* eacc = pts + TP;
  // KQ entries k = blockIdx.y * 256 KQ + threadIdx.x + 256 q per thread, each
  // with its child row offsets decoded once
  int kq[KQ], off0[KQ], off1[KQ];
#pragma unroll
  for (int q = 0; q < KQ; ++q) {
    kq[q] = blockIdx.y * blockDim.x * KQ + threadIdx.x + blockDim.x * q;
    int kk = kq[q] < j.K ? kq[q] : 0;
    // the general product below decodes per point; two children (the common
    // case: the outside message and one child) keep both offsets here
    const int d1 = j.nchild > 1 ? j.ch[1].dim : 1;
    off0[q] = (kk / d1);
    off1[q] = j.ch[0].dim * TP + kk % d1;
  }
  const int ntiles = j.tile_start[j.ngroups];
  const int b0 = blockIdx.x * tiles_per_cta;
  const int b1 = min(ntiles, b0 + tiles_per_cta);
  T acc[KQ];
#pragma unroll
  for (int q = 0; q < KQ; ++q) acc[q] = Sc<T>::zero();
  int gcur = -1;
  for (int b = b0; b < b1; ++b) {
    int row0, nrows, g;
    if (!locate_tile(j, TP, b, row0, nrows, g)) continue;  // uniform over the CTA
    if (g != gcur) {
      if (gcur >= 0)
#pragma unroll
        for (int q = 0; q < KQ; ++q)
          if (kq[q] < j.K) atomic_add_T<T>(dT + (int64_t)gcur * j.K + kq[q], acc[q]);
#pragma unroll
      for (int q = 0; q < KQ; ++q) acc[q] = Sc<T>::zero();
      gcur = g;
    }
    __syncthreads();  // the previous tile's rows are no longer read
    for (int r = threadIdx.x; r < TP; r += blockDim.x) {
      pts[r] = r < nrows ? (j.perm ? j.perm[row0 + r] : row0 + r) : 0;
      eacc[r] = 0;
    }
    __syncthreads();
    load_children(j, pts, nrows, TP, rows, eacc);
    for (int r = threadIdx.x; r < nrows; r += blockDim.x) scale[r] = Sc<T>::scale2(Sc<T>::one(), eacc[r]);
    __syncthreads();
    if (j.nchild == 2) {
      const int d0 = j.ch[0].dim, d1 = j.ch[1].dim;
      for (int r = 0; r < nrows; ++r) {
        const T sc = scale[r];
        const T* r0 = rows + r * d0;
        const T* r1 = rows + r * d1;
#pragma unroll
        for (int q = 0; q < KQ; ++q) acc[q] = Sc<T>::fma(sc * r0[off0[q]], r1[off1[q]], acc[q]);
      }
    } else {
#pragma unroll
      for (int q = 0; q < KQ; ++q) {
        if (kq[q] >= j.K) continue;
        for (int r = 0; r < nrows; ++r) {
          T a = scale[r];
          int kk = kq[q], off = sumdim;
          for (int c = j.nchild - 1; c >= 0; --c) {
            const int d = j.ch[c].dim;
            off -= d;
            a = a * rows[off * TP + r * d + kk % d];
            kk /= d;
          }
          acc[q] = acc[q] + a;
        }
      }
    }
  }
  if (gcur >= 0)
#pragma unroll
    for (int q = 0; q < KQ; ++q)
      if (kq[q] < j.K) atomic_add_T<T>(dT + (int64_t)gcur * j.K + kq[q], acc[q]);
}

template <class T>
__global__ void k_vjp_seed(const double* __restrict__ dout, const T* __restrict__ rootv,
                           const int* __restrict__ roote, int nroots, int r, int Pc, T* __restrict__ E,
                           int* __restrict__ Eexp) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < Pc; p += gridDim.x * blockDim.x) {
    T v = Sc<T>::one();
    if constexpr (sizeof(T) == 16)
      v = T{dout[p], 0.0};
    else
      v = (T)dout[p];
    int e = 0;
    for (int q = 0; q < nroots; ++q) {
      if (q == r) continue;
      v = v * rootv[(int64_t)q * Pc + p];
      e += roote[(int64_t)q * Pc + p];
    }
    E[p] = v;
    Eexp[p] = e;
  }
}

// Group the points of a chunk by the site value of vertex v (fills the job's
// group fields; tp = tile rows of the kernel that will consume them).
template <class T>
void group_by_site(tnfa_ctx* ctx, VertexJob<T>& j, const int* key, int Pc, int ng, int tp, int* meta,
                   int* perm) {
  j.ngroups = ng;
  j.grp_off = meta;
  j.grp_cnt = meta + ng;
  j.tile_start = meta + 2 * ng;
  j.perm = launch_group(ctx, ng > 1 ? key : nullptr, Pc, ng, tp, meta, perm);
}

template <class T>
void vjp_impl(tnfa_ctx* ctx, const tnfa_net* net, const T* tensors, const double* X, int64_t P,
              int ncols, const std::vector<DigitRef>& prog, int xmem, const double* dout,
              int dout_mem, T* dT) {
  const Topo& Tp = net->topo;
  const int V = Tp.V;
  EvalPlan plan = make_plan(Tp);
  const int nroots = (int)plan.roots.size();
  std::vector<int> root_index(V, -1);
  for (int r = 0; r < nroots; ++r) root_index[plan.roots[r]] = r;
  size_t per_point = V * 4 + 4 + (xmem == TNFA_MEM_HOST ? ncols * 8 : 0) +
                     (dout_mem == TNFA_MEM_HOST ? 8 : 0) + nroots * (sizeof(T) + 4);
  for (int v = 0; v < V; ++v) per_point += 2 * ((size_t)Tp.link[v] * sizeof(T) + 4);
  int64_t Pc_max = (int64_t)(ctx->eval_budget / per_point);
  Pc_max = std::max<int64_t>(256, std::min<int64_t>(Pc_max, int64_t(1) << 30));
  const int Pcap = (int)std::max<int64_t>(std::min<int64_t>(P, (Pc_max / 256) * 256), 1);
  int maxsd = 1;
  for (int v = 0; v < V; ++v) maxsd = std::max(maxsd, Tp.site_dim[v]);
  const std::vector<DigitRun> runs = make_fused_runs(Tp, prog);
  DBuf dprog(ctx, std::max<size_t>(runs.size(), 1) * sizeof(DigitRun));
  h2d(ctx, dprog.p, runs.data(), runs.size() * sizeof(DigitRun));
  DBuf dS(ctx, (size_t)V * Pcap * 4), dperm(ctx, (size_t)Pcap * 4);
  DBuf dmeta(ctx, group_meta_ints(maxsd) * 4), derr(ctx, 4);
  TNFA_CUDA(cudaMemsetAsync(derr.p, 0, 4, ctx->stream));
  std::vector<DBuf> in(V), ine(V), E(V), Ee(V);
  for (int v = 0; v < V; ++v) {
    if (!plan.fused_leaf[v]) {
      in[v] = DBuf(ctx, (size_t)Pcap * Tp.link[v] * sizeof(T));
      ine[v] = DBuf(ctx, (size_t)Pcap * 4);
    }
    E[v] = DBuf(ctx, (size_t)Pcap * Tp.link[v] * sizeof(T));
    Ee[v] = DBuf(ctx, (size_t)Pcap * 4);
  }
  DBuf droot(ctx, (size_t)nroots * Pcap * sizeof(T)), droote(ctx, (size_t)nroots * Pcap * 4);
  DBuf dX(ctx, xmem == TNFA_MEM_HOST ? (size_t)Pcap * ncols * 8 : 0);
  DBuf ddout(ctx, dout_mem == TNFA_MEM_HOST ? (size_t)Pcap * 8 : 0);
  int* meta = dmeta.as<int>();
  auto inside_src = [&](int c) {
    ChildSrc<T> s{};
    s.dim = Tp.link[c];
    if (plan.fused_leaf[c]) {
      s.ptr = tensors + Tp.off[c];
      s.exps = nullptr;
      s.idx.codes = dS.as<int>() + (int64_t)c * Pcap;
    } else {
      s.ptr = in[c].as<T>();
      s.exps = ine[c].as<int>();
    }
    return s;
  };
  for (int64_t p0 = 0; p0 < P; p0 += Pcap) {
    const int Pc = (int)std::min<int64_t>(Pcap, P - p0);
    const double* Xc = X + p0 * ncols;
    if (xmem == TNFA_MEM_HOST) {
      TNFA_CUDA(cudaMemcpyAsync(dX.p, Xc, (size_t)Pc * ncols * 8, cudaMemcpyHostToDevice, ctx->stream));
      Xc = dX.as<double>();
    }
    const double* dc = dout + p0;
    if (dout_mem == TNFA_MEM_HOST) {
      TNFA_CUDA(cudaMemcpyAsync(ddout.p, dc, (size_t)Pc * 8, cudaMemcpyHostToDevice, ctx->stream));
      dc = ddout.as<double>();
    }
    launch_digitize(ctx, Xc, ncols, Pc, dprog.as<DigitRun>(), (int)runs.size(), V, dS.as<int>(), Pcap,
                    derr.as<int>());
    // forward: inside messages of every non-leaf vertex
    for (int v : plan.order) {
      VertexJob<T> j{};
      j.nchild = (int)Tp.children[v].size();
      TNFA_CHECK(j.nchild <= EVAL_MAXC, TNFA_ERR_UNSUPPORTED, "vertex degree too high");
      int64_t K = 1;
      int sumdim = 0;
      for (int i = 0; i < j.nchild; ++i) {
        j.ch[i] = inside_src(Tp.children[v][i]);
        K *= j.ch[i].dim;
        sumdim += j.ch[i].dim;
      }
      j.K = (int)K;
      j.chi_a = Tp.link[v];
      j.site_dim = Tp.site_dim[v];
      j.B = tensors + Tp.off[v];
      j.Pc = Pc;
      if (Tp.parent[v] < 0) {
        j.out = (T*)droot.p + (size_t)root_index[v] * Pcap;
        j.out_exp = droote.as<int>() + (size_t)root_index[v] * Pcap;
      } else {
        j.out = in[v].as<T>();
        j.out_exp = ine[v].as<int>();
      }
      group_by_site(ctx, j, dS.as<int>() + (int64_t)v * Pcap, Pc, j.site_dim,
                    contract_tile_rows(j.chi_a, sumdim, sizeof(T)), meta, dperm.as<int>());
      launch_contract<T>(ctx, j, Pc);
    }
    // seeds: E of a root = dout times the other roots' values
    for (int r = 0; r < nroots; ++r)
      k_vjp_seed<T><<<grid_for(Pc, 256, 4096), 256, 0, ctx->stream>>>(
          dc, (const T*)droot.p, droote.as<int>(), nroots, r, Pcap, E[plan.roots[r]].as<T>(),
          Ee[plan.roots[r]].as<int>());
    TNFA_LAUNCH_CHECK();
    // top-down: outside messages of every child
    for (int v = 0; v < V; ++v) {
      const auto& kids = Tp.children[v];
      std::vector<int> shp{Tp.site_dim[v], Tp.link[v]};
      for (int c : kids) shp.push_back(Tp.link[c]);
      for (size_t jx = 0; jx < kids.size(); ++jx) {
        const int c = kids[jx];
        // T_v with child c's axis moved to position 1: [s][c][parent][others]
        DBuf perm_t(ctx, (size_t)Tp.size(v) * sizeof(T));
        la::PermJob pj{};
        pj.src = tensors + Tp.off[v];
        pj.dst = perm_t.p;
        pj.nd = (int)shp.size();
        TNFA_CHECK(pj.nd <= la::MAXD, TNFA_ERR_UNSUPPORTED, "vertex degree too high");
        std::vector<int> order;
        order.push_back(0);
        order.push_back(2 + (int)jx);
        for (int a = 1; a < pj.nd; ++a)
          if (a != 2 + (int)jx) order.push_back(a);
        pj.n = Tp.size(v);
        for (int a = 0; a < pj.nd; ++a) {
          pj.shape[a] = shp[a];
          pj.perm[a] = order[a];
        }
        la::permute<T>(ctx, {pj});
        VertexJob<T> j{};
        j.nchild = 0;
        ChildSrc<T> e{};
        e.ptr = E[v].as<T>();
        e.exps = Ee[v].as<int>();
        e.dim = Tp.link[v];
        j.ch[j.nchild++] = e;
        int64_t K = e.dim;
        int sumdim = e.dim;
        for (size_t q = 0; q < kids.size(); ++q) {
          if (q == jx) continue;
          TNFA_CHECK(j.nchild < EVAL_MAXC, TNFA_ERR_UNSUPPORTED, "vertex degree too high");
          j.ch[j.nchild++] = inside_src(kids[q]);
          K *= Tp.link[kids[q]];
          sumdim += Tp.link[kids[q]];
        }
        j.K = (int)K;
        j.chi_a = Tp.link[c];
        j.site_dim = Tp.site_dim[v];
        j.B = perm_t.as<T>();
        j.Pc = Pc;
        j.out = E[c].as<T>();
        j.out_exp = Ee[c].as<int>();
        group_by_site(ctx, j, dS.as<int>() + (int64_t)v * Pcap, Pc, j.site_dim,
                      contract_tile_rows(j.chi_a, sumdim, sizeof(T)), meta, dperm.as<int>());
        launch_contract<T>(ctx, j, Pc);
      }
    }
    // accumulation: dT_v[s][(a, c...)] += sum_p E_v[p][a] prod m_c[p][c]
    for (int v = 0; v < V; ++v) {
      VertexJob<T> j{};
      ChildSrc<T> e{};
      e.ptr = E[v].as<T>();
      e.exps = Ee[v].as<int>();
      e.dim = Tp.link[v];
      j.ch[j.nchild++] = e;
      int64_t K = e.dim;
      int sumdim = e.dim;
      for (int c : Tp.children[v]) {
        TNFA_CHECK(j.nchild < EVAL_MAXC, TNFA_ERR_UNSUPPORTED, "vertex degree too high");
        j.ch[j.nchild++] = inside_src(c);
        K *= Tp.link[c];
        sumdim += Tp.link[c];
      }
      TNFA_CHECK(K < (int64_t(1) << 31), TNFA_ERR_UNSUPPORTED, "gradient block too large");
      j.K = (int)K;
      j.chi_a = 1;
      j.site_dim = Tp.site_dim[v];
      j.Pc = Pc;
      constexpr int TP = 64;
      group_by_site(ctx, j, dS.as<int>() + (int64_t)v * Pcap, Pc, j.site_dim, TP, meta,
                    dperm.as<int>());
      const size_t sm = (size_t)sumdim * TP * sizeof(T) + TP * sizeof(T) + 2 * TP * sizeof(int);
      TNFA_CHECK(sm <= 200 * 1024, TNFA_ERR_UNSUPPORTED, "bonds too large for the gradient kernel");
      constexpr int KQ = 4;
      auto kern = k_grad_acc<T, TP, KQ>;
      if (sm > 48 * 1024)
        TNFA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
      // one wave of resident CTAs, each over a run of consecutive tiles
      int occ = 0, nsm = 0, dev = 0;
      TNFA_CUDA(cudaGetDevice(&dev));
      TNFA_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
      TNFA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 256, sm));
      const int ntiles = (int)((Pc + TP - 1) / TP + j.ngroups);
      const int ky = (int)((K + 256 * KQ - 1) / (256 * KQ));
      const int want = std::max(1, std::max(occ, 1) * nsm / ky);
      const int per = std::max(1, (ntiles + want - 1) / want);
      dim3 grid((unsigned)((ntiles + per - 1) / per), (unsigned)ky);
      KernelScope ks(ctx, "grad_acc", 2.0 * Pc * (double)K, 0.0);
      kern<<<grid, 256, sm, ctx->stream>>>(j, dT + Tp.off[v], per);
      TNFA_LAUNCH_CHECK();
    }
  }
  int herr = 0;
  TNFA_CUDA(cudaMemcpyAsync(&herr, derr.p, 4, cudaMemcpyDeviceToHost, ctx->stream));
  TNFA_CUDA(cudaStreamSynchronize(ctx->stream));
  TNFA_CHECK(herr == 0, TNFA_ERR_DOMAIN,
             "a coordinate is negative or not finite (the digit map needs x >= 0)");
}

}  // namespace
}  // namespace tnfa

extern "C" int tnfa_evaluate_vjp(tnfa_ctx* ctx, const tnfa_net* net, const double* X,
                                 int64_t n_points, int32_t n_dims, const int32_t* dims,
                                 int x_memory, const double* dout, int dout_memory, void* dtensors,
                                 int dtensors_memory) {
  TNFA_API_BEGIN(ctx);
  require_ctx(ctx);
  require_net(net, "evaluate_vjp");
  TNFA_CHECK(n_points >= 0, TNFA_ERR_INVALID_ARGUMENT, "n_points < 0");
  if (n_points == 0) return TNFA_OK;
  TNFA_CHECK(X && dout && dtensors && (n_dims == 0 || dims), TNFA_ERR_INVALID_ARGUMENT,
             "null X, dout, dtensors or dims");
  for (int m : {x_memory, dout_memory, dtensors_memory})
    TNFA_CHECK(m == TNFA_MEM_HOST || m == TNFA_MEM_DEVICE, TNFA_ERR_INVALID_ARGUMENT, "bad memory kind");
  for (int v = 0; v < net->topo.V; ++v)
    TNFA_CHECK(net->topo.site_dim[v] <= 256, TNFA_ERR_UNSUPPORTED, "site dimension above 256");
  int ncols = 0;
  std::vector<DigitRef> prog = make_digit_program(net->topo, n_dims, dims, &ncols);
  const size_t es = dtype_size(net->dtype);
  const size_t bytes = (size_t)net->topo.n_elem * es;
  DBuf acc;
  void* dT = dtensors;
  if (dtensors_memory == TNFA_MEM_HOST) {
    acc = DBuf(ctx, bytes);
    TNFA_CUDA(cudaMemcpyAsync(acc.p, dtensors, bytes, cudaMemcpyHostToDevice, ctx->stream));
    dT = acc.p;
  }
  if (net->dtype == TNFA_F64)
    vjp_impl<double>(ctx, net, (const double*)net->d, X, n_points, ncols, prog, x_memory, dout,
                     dout_memory, (double*)dT);
  else if (net->dtype == TNFA_F32)
    vjp_impl<float>(ctx, net, (const float*)net->d, X, n_points, ncols, prog, x_memory, dout,
                    dout_memory, (float*)dT);
  else
    vjp_impl<cplx>(ctx, net, (const cplx*)net->d, X, n_points, ncols, prog, x_memory, dout,
                   dout_memory, (cplx*)dT);
  if (dtensors_memory == TNFA_MEM_HOST) {
    TNFA_CUDA(cudaMemcpyAsync(dtensors, acc.p, bytes, cudaMemcpyDeviceToHost, ctx->stream));
    TNFA_CUDA(cudaStreamSynchronize(ctx->stream));
  }
  TNFA_API_END
}

// Batched point evaluation of a tree tensor network function.
//
// Reference path (ITensorNumericalAnalysis.jl): evaluate
// (src/itensornetworkfunction.jl:96-112) = calculate_ind_values (digits by
// greedy subtraction, src/IndexMaps/abstractindexmap.jl:121-138) -> project
// (one-hot slice of every site leg, :84-94) -> scalar(tn; alg="bp") (exact on
// a tree).  It handles one point per call.
//
// Here a message is formed once for every combination of the digits below its
// edge where there are fewer combinations than points, and once per point
// elsewhere (the schedule: eval_tree.cuh; EvalEngine lays it out and runs it):
//   1. tables, level by level: row r of a vertex is its message for digit
//      combination r; the products of a level are one launch.
//   2. k_digitize: coordinates -> the codes (table rows, site values) that the
//      points read (in the kernels of 4 where those do it themselves).
//   3. vertices without a table, per chunk of points: group the points by site
//      value (count / scan / scatter), so that a tile of points shares one slice
//      T_v[s]; out[p, a] = sum_k A[p, k] T_v[s][a][k] with A the row-wise
//      Kronecker product of the children's messages, read from their tables by
//      code.  At small bonds one launch walks a point through all of them.
//   4. the centre, any one edge: f(p) = sum_c A[p, c] B[p, c] over the two
//      messages that meet there, times the other components' values.
// Each row is rescaled by a power of two when it is made or read (exact) and the
// exponent is carried per row, so deep trees neither underflow nor overflow.
#include <algorithm>
#include <memory>
#include <type_traits>

#include "eval_tree.cuh"
#include "adjoint.cuh"
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

// ------------------------------------------------- small-bond networks ----
// TNFA_EVAL_FUSED=0 turns the one-launch kernels off (the walk, and digits
// taken by the centre kernel).
static bool fused_allowed() {
  const char* env = getenv("TNFA_EVAL_FUSED");
  return !(env && *env == '0');
}
constexpr int FUSED_MAXV = 128;

// Networks whose points a thread can walk: every bond <= 16 (<= 32 on paths),
// at most two children per vertex, 64 KB of messages per 32 points.  A thread
// per point: above bond 8 a few thousand points leave the GPU mostly idle,
// where the per-vertex kernels spread a point over a warp.
static bool small_bonds(const Topo& T, size_t tsize, int64_t npoints) {
  if (!fused_allowed() || T.V > FUSED_MAXV) return false;
  int chimax = 1, maxch = 0;
  for (int v = 0; v < T.V; ++v) {
    chimax = std::max(chimax, T.link[v]);
    maxch = std::max(maxch, (int)T.children[v].size());
    if (T.site_dim[v] > 256) return false;
  }
  if (maxch > 2 || chimax > 32 || (chimax > 16 && maxch > 1)) return false;
  if (chimax > 8 && npoints < 32768) return false;
  return T.n_elem * (int64_t)tsize <= 4 * 1024 * 1024;
}

// -------------------------------------------------------------- driver ----
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

constexpr size_t CONTRACT_SMEM = 200 * 1024;

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
    TNFA_CHECK(sm <= CONTRACT_SMEM, TNFA_ERR_UNSUPPORTED, "children bonds too large for evaluation");
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
    TNFA_CHECK(sm <= CONTRACT_SMEM, TNFA_ERR_UNSUPPORTED, "children bonds too large for evaluation");
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

// Shared memory of launch_contract for one vertex.
static size_t contract_smem(int chi_a, int64_t sumdim, size_t tsize) {
  if (chi_a <= 16) return sumdim * 8 * tsize + 2 * 8 * sizeof(int);
  const GemmTile t = gemm_tile(chi_a, (int)sumdim, tsize);
  return sumdim * tsize * t.tp + (size_t)16 * (t.tp + t.ta) * tsize + 2 * t.tp * sizeof(int);
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

// Jobs with their first blocks (first has one entry more): in the launch's
// parameters when they fit, else from the device tables.
template <class T>
static RowPack<T> pack_rows(const std::vector<RowJob<T>>& jobs, const std::vector<int>& first, const RowJob<T>* djobs,
                            const int* dfirst) {
  RowPack<T> p{};
  p.total = (int)jobs.size();
  if (jobs.size() <= (size_t)ROW_PACK) {
    p.n = p.total;
    std::copy(jobs.begin(), jobs.end(), p.j);
    std::copy(first.begin(), first.end(), p.f);
  } else {
    p.jobs = djobs;
    p.first = dfirst;
  }
  return p;
}

template <class T>
static void launch_rows(tnfa_ctx* ctx, int tile, int64_t blocks, const RowPack<T>& pack) {
  TNFA_CHECK(blocks < (int64_t(1) << 31), TNFA_ERR_UNSUPPORTED, "contraction too large");
  auto go = [&](auto kern) { kern<<<(unsigned)blocks, 256, 0, ctx->stream>>>(pack); };
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

// Products of the thread-per-row kernel: fewer columns than a tile's 32 lanes.
template <class T>
static bool small_rows(const RowJob<T>& j) {
  return j.rpg > 0 && j.K <= 32 && j.N < 32 && (int64_t)j.rows * ((j.N + 3) / 4) < (int64_t(1) << 31);
}
template <class T>
static int64_t small_blocks(const RowJob<T>& j) {
  return ((int64_t)j.rows * ((j.N + 3) / 4) + 127) / 128;
}
template <class T>
static void launch_small_rows(tnfa_ctx* ctx, int64_t blocks, int kmax, const RowPack<T>& pack) {
  auto go = [&](auto kern) { kern<<<(unsigned)blocks, 128, 0, ctx->stream>>>(pack); };
  if (kmax <= 4) go(k_rows_small<T, 4>);
  else if (kmax <= 8) go(k_rows_small<T, 8>);
  else if (kmax <= 16) go(k_rows_small<T, 16>);
  else go(k_rows_small<T, 32>);
  TNFA_LAUNCH_CHECK();
}

// Multiply-adds per second by which the walk of a call is counted against the
// 20 us up to which no tables are laid out at all.  Its latency is in them: the
// rate of many points alone is higher (SmallCosts::point_madd).
template <class T> struct WalkRate;
template <> struct WalkRate<float> { static constexpr double v = 4e12; };
template <> struct WalkRate<double> { static constexpr double v = 3e11; };
template <> struct WalkRate<cplx> { static constexpr double v = 8e10; };

// Microseconds of a call beyond what every call costs, where the walk and tables
// are close: fitted to 1485 calls (paths, combs and binary trees of 12 to 30
// vertices, bonds 2 to 8, 500 to 128000 points), each by the walk and from
// tables; 8 % rms off in FP32 and FP64, 13 % in complex.  The walk: a vertex
// and a multiply-add of one point's chain, and of all points (work counted with
// bonds padded to 2, 4 or 8).  Tables: a level's launch, a table with launches
// of its own (two kids, neither absorbed), the permuted tensors, the head and
// one of its vertices, a multiply-add of the tables beyond it, the centre.
struct SmallCosts {
  double vertex, madd, point_vertex, point_madd;
  double level, table, move, head, head_vertex, table_madd, centre;
};
template <class T> struct SmallCost;
template <> struct SmallCost<double> {
  static constexpr SmallCosts v{0.98, 0.0085, 4.9e-6, 2.1e-6, 7.2, 10, 12, 14, 0.83, 7.0e-6, 31e-6};
};
template <> struct SmallCost<float> {
  static constexpr SmallCosts v{0.81, 0.0031, 3.6e-6, 0.33e-6, 5.9, 11, 12, 8.8, 1.0, 6.0e-6, 10e-6};
};
template <> struct SmallCost<cplx> {
  static constexpr SmallCosts v{1.0, 0.027, 23e-6, 4.7e-6, 10, 9.5, 14, 23, 0.35, 18e-6, 58e-6};
};

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
             int ncols, int64_t P, bool use_tc, bool use_oz, size_t budget, bool adjoint = false,
             double max_rows = 134217728.0)
      : ctx_(ctx), net_(net), tensors_(tensors), topo_(net->topo), prog_(prog), ncols_(ncols), P_(P),
        use_tc_(use_tc), use_oz_(use_oz), adjoint_(adjoint) {
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
    check_shapes(o.tensor_ok);
    // Tables (and their adjoints, of the same size) take at most half the
    // scratch: the row bound shrinks until they fit.  Every digit code stays
    // within 31 bits.
    const double copies = adjoint_ ? 2.0 : 1.0;
    double rows = std::min((double)P, max_rows);
    if (adjoint_) {  // every product of a table is a row product (see AdjointEngine)
      o.table_kids = 2;
      o.absorb_points = false;
    }
    small_ = !adjoint_ && !use_tc && !use_oz && small_bonds(topo_, sizeof(T), P);
    if (small_) {
      // Points that a thread walks cost one launch; a level of tables costs
      // another (about 3 us).  Up to about 20 us of walking there are no tables;
      // beyond, a table of half as many rows as points or less pays.
      double w = 0;
      bool path = true;
      int top = 1;
      for (int v = 0; v < V; ++v) {
        double x = topo_.link[v];
        for (int c : topo_.children[v]) x *= topo_.link[c];
        w += x;
        path &= topo_.children[v].size() <= (topo_.parent[v] < 0 ? 2u : 1u);
        top = std::max(top, topo_.link[v]);
      }
      bool walk = w * P <= 20e-6 * WalkRate<T>::v;
      // FP64 paths of bond 5 to 8: their tables are too large for k_head and
      // take a launch of 10 us for every two vertices beyond about ten, 6 V -
      // 39 us in all; the walk takes 1.4 us a vertex and up to 64 multiply-adds
      // per vertex and point at 5.4e11 a second.  Calls on 17 vertices, bond 7:
      // 15000 points 85 us walked, 94 from tables; 22000 points 114 and 94.
      if (std::is_same<T, double>::value && path && top > 4 && top <= 8)
        walk |= 64.0 * V * P <= (4.6e-6 * V - 39e-6) * 5.4e11;
      o.balance = true;
      rows = walk ? 0 : std::floor(rows / 2);
    }
    for (;;) {
      o.table_rows = rows;
      o.table_elems = std::min(1073741824.0, (double)(budget / 2) / sizeof(T));
      tree_ = EvalTreeBuilder(topo_, o).build();
      // The stored order fits (check_shapes).  (Never a gradient's case, whose
      // two-kid tables need absorption: its narrower bonds fit in any order.)
      if (!jobs_fit()) {
        o.rule = CentreRule::ROOT;
        o.absorb = false;
        tree_ = EvalTreeBuilder(topo_, o).build();
      }
      if (copies * table_bytes() <= budget / 2 || rows < 1) break;
      rows = std::floor(rows / 4);
      if (rows < 1 && !small_) {  // the stored order, nothing but points
        o.rule = CentreRule::ROOT;
        o.absorb = false;
      }
    }
    plan();
    if (small_ && rows > 0) {
      // Where the walk by itself is cheaper than these tables by more than the
      // second schedule (about 10 us) and the costs' error, it is taken after all.
      // Trees have many levels of small tables: 30-vertex binary tree, bond 2,
      // complex, 16000 points 184 us from tables, 92 so; bond 4, FP64, 8000 points
      // 161 and 94.  The same with bond 8, FP64: 113 from tables, 220 walked.
      const double error = sizeof(T) == 16 ? 1.2 : 1.1;
      if (error * walk_cost(true) + 12.0 <= table_cost()) {
        EvalTree kept = std::move(tree_);
        o.table_rows = 0;
        tree_ = EvalTreeBuilder(topo_, o).build();
        plan();
        if (!walk_) {  // (not in this order's shared memory)
          tree_ = std::move(kept);
          plan();
        }
      }
    }
    per_point_ = (size_t)nmsg_ * (msg_chi_ * sizeof(T) + sizeof(int)) + (size_t)ncodes_ * 4 + (npp_ ? 4 : 0);
    const size_t tab = scratch(0);
    const size_t left = budget > tab ? budget - tab : 0;
    int64_t pc = per_point_ ? (int64_t)(left / per_point_) / 256 * 256 : int64_t(1) << 30;
    Pc_ = (int)std::min<int64_t>(P, std::max<int64_t>(256, std::min<int64_t>(pc, int64_t(1) << 30)));
  }

  int chunk() const { return Pc_; }
  int64_t table_rows() const {  // of the longest table
    int64_t n = 0;
    for (const EvalVertex& e : tree_.v)
      if (e.tabled && !e.leaf) n = std::max(n, e.N);
    return n;
  }
  void set_chunk(int pc) { Pc_ = pc; }
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
  // The job tables go to the scratch (stream order).
  void upload() {
    h2d(ctx_, blob_, host_.data(), host_.size());
  }
  void clear_error() { TNFA_CUDA(cudaMemsetAsync(err_, 0, 4, ctx_->stream)); }
  void use_error(int* word) { err_ = word; }  // after bind: a synchronous call's own word

  // Tables: permuted tensors, then every level.
  void tables() {
    if (!moves_.empty()) {
      int64_t n = 1;
      for (const auto& m : moves_) n = std::max(n, m.n);
      KernelScope ks(ctx_, "move", 0.0, 0.0);
      k_move<T><<<dim3(grid_for(n, 256, 1024), (unsigned)moves_.size()), 256, 0, ctx_->stream>>>(dmoves_);
      TNFA_LAUNCH_CHECK();
    }
    if (!hgroups_.empty()) {
      KernelScope ks(ctx_, FamilyName<T>::v, 0.0, 0.0);
      const size_t sm = head_elems_ * sizeof(T) + head_exps_ * 4 + head_jobs_ * sizeof(HeadJob);
      auto go = [&](auto kern) {
        if (sm > 47 * 1024)  // (48 KB with the kernel's static words)
          TNFA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
        // range of a side's exponents: products of two sides stay far below the type's limit
        kern<<<(unsigned)hgroups_.size(), 256, sm, ctx_->stream>>>(dhblocks_, dhcopies_, dhjobs_, head_elems_,
                                                                    head_exps_, head_jobs_, plain_,
                                                                    sizeof(T) == 4 ? 40 : 400);
      };
      if (head_k_ <= 4) go(k_head<T, 4>);
      else if (head_k_ <= 8) go(k_head<T, 8>);
      else if (head_k_ <= 16) go(k_head<T, 16>);
      else go(k_head<T, 32>);
      TNFA_LAUNCH_CHECK();
    }
    for (size_t l = 0; l < levels_.size(); ++l) {
      Level& L = levels_[l];
      if (!L.small.empty()) {
        double fl = 0;
        int kmax = 1;
        for (const auto& j : L.small) {
          fl += 2.0 * (double)j.rows * j.N * j.K;
          kmax = std::max(kmax, j.K);
        }
        KernelScope ks(ctx_, FamilyName<T>::v, fl, 0.0);
        launch_small_rows<T>(ctx_, L.sfirst.back(), kmax, pack_rows(L.small, L.sfirst, L.dsmall, L.dsfirst));
      }
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
          launch_rows<T>(ctx_, t, L.first[t].back(), pack_rows(L.rows, L.first[t], L.drows, L.dfirst[t]));
        };
        if (tuned) tune(ctx_, key, RowTiles<T>::n, fl, go);
        else go(0);
      }
      if constexpr (std::is_same<T, double>::value) {
        // the sliced tensor-core tables of a level in one launch
        std::vector<std::pair<int, VertexJob<double>>> oz;
        for (int v : L.verts) {
          if (!tree_.v[v].tensor) continue;
          oz.push_back({v, vertex_job(v)});
          bind_groups(oz.back().second, tmeta_[v]);
        }
        if (!oz.empty()) oz_contract(ctx_, net_, oz, err_);
      }
      for (int v : L.verts)
        if (!std::is_same<T, double>::value || !tree_.v[v].tensor) contract_table(v);
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
    if (walk_) {
      walk(X, n, out, kind, Pout, pofs);
      return;
    }
    if (ncodes_ > 0)
      launch_digitize(ctx_, X, ncols_, n, druns_, (int)runs_.size(), ncodes_, codes_, Pc_, err_);
    for (int v : tree_.order)
      if (!tree_.v[v].tabled) contract_points(v, n);
    centre(X, n, out, kind, Pout, pofs);
  }

 protected:
  struct Level {
    std::vector<RowJob<T>> rows;
    std::vector<int> verts;  // table vertices of the multi-child kernels
    RowJob<T>* drows = nullptr;
    std::vector<RowJob<T>> small;  // of the thread-per-row kernel
    RowJob<T>* dsmall = nullptr;
    std::vector<int> sfirst;
    int* dsfirst = nullptr;
    int njobs = 0;
    std::vector<int> first[3];
    int* dfirst[3] = {nullptr, nullptr, nullptr};
  };

  // The networks that evaluation takes, whatever the schedule: those whose
  // contraction in the stored order the per-point kernels take.
  void check_shapes(const std::vector<char>& tensor_ok) const {
    for (int v = 0; v < topo_.V; ++v) {
      const auto& kids = topo_.children[v];
      if (topo_.parent[v] >= 0 && kids.empty()) continue;
      TNFA_CHECK(kids.size() <= (size_t)EVAL_MAXC, TNFA_ERR_UNSUPPORTED,
                 "vertex degree above " + std::to_string(EVAL_MAXC) + " children");
      int64_t K = 1, sum = 0;
      for (int c : kids) {
        K = std::min(K * topo_.link[c], int64_t(1) << 31);
        sum += topo_.link[c];
      }
      TNFA_CHECK(K < (int64_t(1) << 31), TNFA_ERR_UNSUPPORTED, "contraction too large");
      TNFA_CHECK((!tensor_ok.empty() && tensor_ok[v]) || contract_smem(topo_.link[v], sum, sizeof(T)) <= CONTRACT_SMEM,
                 TNFA_ERR_UNSUPPORTED, "children bonds too large for evaluation");
    }
  }
  // (in another orientation a vertex may have to take its parent's bond in)
  bool jobs_fit() const {
    for (int v = 0; v < topo_.V; ++v) {
      const EvalVertex& e = tree_.v[v];
      if (e.leaf || e.tensor || row_form(v)) continue;
      int64_t K = 1;
      for (size_t i = 0; i + (e.absorb ? 1 : 0) < e.kids.size(); ++i)
        K = std::min(K * tree_.v[e.kids[i]].chi, int64_t(1) << 31);
      if (K >= (int64_t(1) << 31) || contract_smem(e.chi, job_sumdim(v), sizeof(T)) > CONTRACT_SMEM) return false;
    }
    return true;
  }

  // Microseconds of walking all vertices, or those without a table (SmallCosts).
  double walk_cost(bool all) const {
    constexpr SmallCosts c = SmallCost<T>::v;
    double n = 0, w = 0;
    int top = 1;
    for (int v = 0; v < topo_.V; ++v) {
      top = std::max(top, topo_.link[v]);
      if (!all && tree_.v[v].tabled) continue;
      n += 1;
      w += tree_.v[v].W;
    }
    w *= (top <= 2 ? 2.0 : top <= 4 ? 4.0 : top <= 8 ? 8.0 : top) / top;
    return n * c.vertex + w * c.madd + P_ * (n * c.point_vertex + w * c.point_madd);
  }
  // Microseconds of the schedule as planned: its tables and its points.
  double table_cost() const {
    constexpr SmallCosts c = SmallCost<T>::v;
    double t = 0, n = 0;
    bool moves = false;
    for (const Level& L : levels_) {
      if (L.njobs > 0 || !L.verts.empty()) t += c.level;
      t += c.table * L.verts.size();
    }
    for (int v = 0; v < topo_.V; ++v) {
      const EvalVertex& e = tree_.v[v];
      moves |= needs_move(v);
      if (e.leaf) continue;
      if (!e.tabled) {
        n += 1;
      } else if (head_[v]) {
        t += c.head_vertex;
      } else {
        const double k = e.absorb ? e.W / tree_.v[e.kids.back()].chi : e.W;
        t += c.table_madd * (e.N * k + (e.absorb ? absorbed_rows(v) * e.W : 0.0));
      }
    }
    if (moves) t += c.move;
    if (!hgroups_.empty()) t += c.head;
    return t + (n > 0 ? walk_cost(false) : P_ * c.centre);
  }

  size_t table_bytes() const {
    double b = 0;
    for (int v = 0; v < topo_.V; ++v) {
      const EvalVertex& e = tree_.v[v];
      if (e.tabled && !e.leaf) b += (double)e.N * (e.chi * sizeof(T) + 4);
      if (e.absorb) b += absorbed_rows(v) * (e.W / tree_chi(e.kids.back(), v) * sizeof(T) + 4);
      if (e.moved) b += (double)topo_.size(v) * sizeof(T);  // (more than a walk needs)
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
    fused_ = !adjoint_ && fused_allowed() && npp_ == 0 && n <= 16 && prog_.size() <= 256;
    runs_ = make_runs(prog_, slot_, mult_);
    walk_ = small_ && npp_ > 0 && plan_walk();
    ncodes_ = fused_ || walk_ ? 0 : n;
    if (walk_) {
      nmsg_ = 0;
      msg_chi_ = max_group_ = 1;
      plan_levels();
      return;
    }
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
        if (!tree_.v[w].tabled && !adjoint_) free_slots.push_back(msg_[w]);
    }
    max_group_ = 1;
    for (int v = 0; v < V; ++v)
      if (!tree_.v[v].tabled)
        max_group_ = std::max<int64_t>(max_group_, tree_.v[v].absorb ? (int64_t)absorbed_rows(v) : topo_.site_dim[v]);
    plan_levels();
  }

  // The walk's schedule: steps of side 0, then side 1, message slots, and the
  // points per block that its shared memory allows.
  bool plan_walk() {
    const int V = topo_.V;
    std::vector<int> side(V, 0);
    for (const auto& c : tree_.comps)
      if (c.b >= 0) side[c.b] = 1;
    for (size_t i = tree_.order.size(); i-- > 0;) {
      const int v = tree_.order[i];
      for (int w : tree_.v[v].kids) side[w] = side[v];
    }
    wsteps_.clear();
    wchi_ = 1;
    nstage_ = 0;
    nsteps0_ = 0;
    int nmsg = 0;
    for (int sd = 0; sd < 2; ++sd) {
      std::vector<int> free_slots;
      for (int v : tree_.order) {
        const EvalVertex& e = tree_.v[v];
        if (e.tabled || side[v] != sd) continue;
        const int nk = (int)e.kids.size() - (e.absorb ? 1 : 0);
        if (nk > 2) return false;
        WalkVertex w;
        w.v = v;
        w.nk = nk;
        w.d1 = nk == 2 ? tree_.v[e.kids[0]].chi : 1;
        w.d2 = nk >= 1 ? tree_.v[e.kids[nk - 1]].chi : 1;
        wchi_ = std::max({wchi_, e.chi, w.d1, w.d2});
        if (free_slots.empty()) free_slots.push_back(nmsg++);
        msg_[v] = free_slots.back();
        free_slots.pop_back();
        for (int i = 0; i < nk; ++i)
          if (!tree_.v[e.kids[i]].tabled) free_slots.push_back(msg_[e.kids[i]]);
        wsteps_.push_back(w);
      }
      if (sd == 0) nsteps0_ = (int)wsteps_.size();
    }
    // the sides of a vertex centre and tables at the centre
    for (const auto& c : tree_.comps) wchi_ = std::max(wchi_, tree_.v[c.a].chi);
    if (wchi_ > 32) return false;
    wchi_ = wchi_ <= 2 ? 2 : wchi_ <= 4 ? 4 : wchi_ <= 8 ? 8 : wchi_ <= 16 ? 16 : 32;
    wmsg_ = nmsg;
    nstage_ = (size_t)topo_.n_elem * sizeof(T) <= 64 * 1024 ? (int)topo_.n_elem : 0;
    // points per block: spread over the SMs first, then as many as the shared
    // memory allows two blocks per SM with
    wtp_ = P_ <= 64 * 4 * ctx_->sm_count ? 32 : 128;
    while (wtp_ > 32 && walk_bytes() > 100 * 1024) wtp_ /= 2;
    // lanes per point: up to four while the points alone do not give every
    // second scheduler (four per SM) a warp.  Twice as many lanes cost more in
    // shuffles than their warps hide: 26 vertices, bond 6, FP64, 8000 points 104
    // us a call against 91, 19078 points 124 against 108
    wlanes_ = 1;
    if (wchi_ <= 8)
      while (wlanes_ < std::min(4, wchi_) && 2 * P_ * wlanes_ < 64 * 2 * (int64_t)ctx_->sm_count) wlanes_ *= 2;
    if (wlanes_ > 1) wtp_ = 32 / wlanes_ * (wlanes_ == 4 ? 2 : 1);
    return walk_bytes() <= 200 * 1024;
  }
  size_t walk_bytes() const {
    return walk_smem<T>(wchi_, wtp_, nstage_, wmsg_, nslots_, (int)runs_.size(), (int)wsteps_.size(),
                        (int)tree_.comps.size());
  }

  // Multiply-adds of one table product that a single block finishes in less
  // than a launch takes (an SM does 2 FP64 or 128 FP32 a clock), and the shared
  // memory of a block's tensors and tables.
  static constexpr double kHeadWork = sizeof(T) == 4 ? 65536 : sizeof(T) == 8 ? 6144 : 1536;
  static constexpr int kHeadK = 32;
  static constexpr int64_t kHeadBytes = 96 * 1024;
  int table_pitch(int chi) const { return chi | 1; }  // odd: rows start in different banks

  void plan_levels() {
    const int V = topo_.V;
    lvl_.assign(V, 0);
    lvl_m_.assign(V, 0);
    // head vertices: every product of the subtree is small
    head_.assign(V, 0);
    plain_of_.assign(V, -1);
    std::vector<int> reader(V, -1);
    std::vector<int64_t> bytes(V, 0);
    for (int v : tree_.order) {
      const EvalVertex& e = tree_.v[v];
      for (int w : e.kids) reader[w] = v;
      bytes[v] = topo_.size(v) * (int64_t)sizeof(T);
      if (adjoint_ || e.leaf || !e.tabled || !row_form(v)) continue;
      bool ok = e.kids.size() <= 2;
      for (int w : e.kids) {
        ok &= tree_.v[w].leaf || head_[w];
        bytes[v] += bytes[w];
      }
      const double row_k = tree_.v[e.kids[0]].chi;
      ok &= row_k <= kHeadK && (double)e.N * e.chi * row_k <= kHeadWork;
      bytes[v] += e.N * (table_pitch(e.chi) * (int64_t)sizeof(T) + 4) + sizeof(HeadJob);
      if (e.absorb) {
        const int64_t r = (int64_t)absorbed_rows(v), k = tree_.v[e.kids.back()].chi;
        ok &= k <= kHeadK && r * e.W <= kHeadWork;
        bytes[v] += r * ((int64_t)(e.W / k) * (int64_t)sizeof(T) + 4) + sizeof(HeadJob);
      }
      head_[v] = ok && bytes[v] <= kHeadBytes;
    }
    hgroups_.clear();
    nhead_copies_ = 0;
    for (int v : tree_.order) {
      if (!head_[v] || (reader[v] >= 0 && head_[reader[v]])) continue;
      std::vector<int> g, todo{v};
      while (!todo.empty()) {
        const int x = todo.back();
        todo.pop_back();
        g.push_back(x);
        for (int w : tree_.v[x].kids) {
          if (head_[w]) todo.push_back(w);
          else ++nhead_copies_;  // a leaf
        }
      }
      nhead_copies_ += (int)g.size();
      std::reverse(g.begin(), g.end());
      plain_of_[v] = (int)hgroups_.size();
      hgroups_.push_back(g);
    }
    int top = 0;
    nhead_jobs_ = 0;
    for (int v : tree_.order) {
      const EvalVertex& e = tree_.v[v];
      if (e.leaf) continue;
      // (levels inside the head order its jobs; to the launches it is level 0)
      auto lv = [&](int w) { return !head_[v] && head_[w] ? 0 : tree_.v[w].tabled ? lvl_[w] : 0; };
      int l = 0;
      for (size_t i = 0; i < e.kids.size(); ++i) {
        const bool ab = e.absorb && i + 1 == e.kids.size();
        if (ab) lvl_m_[v] = lv(e.kids[i]) + 1;
        l = std::max(l, ab ? lvl_m_[v] : lv(e.kids[i]));
      }
      if (e.tabled) lvl_[v] = l + 1;
      if (head_[v]) nhead_jobs_ += e.absorb ? 2 : 1;
      else top = std::max({top, lvl_m_[v], e.tabled ? lvl_[v] : 0});
    }
    levels_.assign(top + 1, Level{});
    for (int v : tree_.order) {
      const EvalVertex& e = tree_.v[v];
      if (e.leaf || head_[v]) continue;
      if (e.absorb) levels_[lvl_m_[v]].njobs += 1;
      if (!e.tabled) continue;
      if (row_form(v)) levels_[lvl_[v]].njobs += 1;
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
      for (int v : {cc.a, cc.b}) nnorm += !walk_ && !adjoint_ && v >= 0 && tree_.v[v].tabled && !tree_.v[v].leaf && !head_[v];
    dmoves_ = c.take<MoveJob>(nmove);
    dnorms_ = c.take<NormJob<T>>(nnorm);
    dcentre_ = c.take<CentreJob<T>>(tree_.comps.size());
    dwalk_ = c.take<unsigned char>(
        walk_ ? walk_blob<T>((int)runs_.size(), (int)wsteps_.size(), (int)tree_.comps.size()) : 0);
    dhblocks_ = c.take<HeadBlock<T>>(hgroups_.size());
    dhcopies_ = c.take<HeadCopy<T>>(nhead_copies_);
    dhjobs_ = c.take<HeadJob>(nhead_jobs_);
    for (auto& L : levels_) {
      L.drows = c.take<RowJob<T>>(L.njobs);
      L.dsmall = c.take<RowJob<T>>(L.njobs);
      L.dsfirst = c.take<int>(L.njobs + 1);
      for (int t = 0; t < RowTiles<T>::n; ++t) L.dfirst[t] = c.take<int>(L.njobs + 1);
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
    rex_.assign(V, nullptr);
    for (int v = 0; v < V; ++v) {
      const EvalVertex& e = tree_.v[v];
      ten_[v] = needs_move(v) ? c.take<T>(topo_.size(v)) : const_cast<T*>(tensors_ + topo_.off[v]);
      if (adjoint_ && e.tabled) rex_[v] = c.take<int>(e.N);
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
    plain_ = c.take<int>(hgroups_.size());
    // per point
    codes_ = c.take<int>((size_t)ncodes_ * pc);
    perm_ = c.take<int>(npp_ && !walk_ ? pc : 0);
    meta_ = c.take<int>(npp_ && !walk_ ? group_meta_ints((int)max_group_) : 0);
    mval_ = c.take<T>((size_t)nmsg_ * pc * msg_chi_);
    mexp_ = c.take<int>((size_t)nmsg_ * pc);
    ld_ = pc;
  }
  // (a walked vertex is read through strides; an absorbing one needs the kid last)
  bool needs_move(int v) const {
    const EvalVertex& e = tree_.v[v];
    return e.moved && !head_[v] && (e.absorb || !(walk_ && !e.tabled));
  }
  // Strides of the stored tensor of v in the order its axes are read.
  std::vector<int64_t> stored_strides(int v) const {
    std::vector<int64_t> str(2 + topo_.children[v].size(), 1), out;
    for (int i = (int)str.size() - 2; i >= 0; --i)
      str[i] = str[i + 1] * (i == 0 ? topo_.link[v] : topo_.link[topo_.children[v][i - 1]]);
    for (int a : tree_.v[v].axes) out.push_back(str[a]);
    return out;
  }
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
    for (int v = 0; v < topo_.V; ++v)
      if (needs_move(v)) moves_.push_back(move_job(v));
    put(dmoves_, moves_.data(), moves_.size() * sizeof(MoveJob));
    if (walk_) fill_walk(put);
    std::vector<CentreJob<T>> cj;
    for (const auto& c : tree_.comps) {
      if (walk_) break;
      CentreJob<T> j{};
      j.chi = tree_.v[c.a].chi;
      j.a = side(c.a);
      if (c.b >= 0) j.b = side(c.b);
      cj.push_back(j);
      for (int v : {c.a, c.b})
        if (!walk_ && !adjoint_ && v >= 0 && tree_.v[v].tabled && !tree_.v[v].leaf && !head_[v])
          norms_.push_back({tab_[v], tabe_[v], (int)tree_.v[v].N, tree_.v[v].chi});
    }
    put(dcentre_, cj.data(), cj.size() * sizeof(CentreJob<T>));
    put(dnorms_, norms_.data(), norms_.size() * sizeof(NormJob<T>));
    fill_head(put);
    centre_chi_ = 1;
    centre_vec_ = true;
    constexpr int vec = 16 / sizeof(T);
    for (const auto& j : cj) {
      centre_chi_ = std::max(centre_chi_, j.chi);
      centre_vec_ &= j.chi % vec == 0 && ((uintptr_t)j.a.ptr & 15) == 0 && ((uintptr_t)j.b.ptr & 15) == 0;
    }
    for (auto& L : levels_) {
      L.rows.clear();
      L.small.clear();
    }
    auto add = [&](Level& L, const RowJob<T>& j) { (small_rows(j) ? L.small : L.rows).push_back(j); };
    for (int v : tree_.order) {
      const EvalVertex& e = tree_.v[v];
      if (e.leaf) continue;
      if (head_[v]) continue;
      if (e.absorb) add(levels_[lvl_m_[v]], absorb_job(v));
      if (e.tabled && row_form(v)) add(levels_[lvl_[v]], table_job(v));
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
      put(L.dsmall, L.small.data(), L.small.size() * sizeof(RowJob<T>));
      L.sfirst.assign(1, 0);
      int64_t sb = 0;
      for (const auto& j : L.small) {
        sb += small_blocks(j);
        TNFA_CHECK(sb < (int64_t(1) << 31), TNFA_ERR_UNSUPPORTED, "contraction too large");
        L.sfirst.push_back((int)sb);
      }
      put(L.dsfirst, L.sfirst.data(), L.sfirst.size() * sizeof(int));
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

  template <class Put>
  void fill_walk(Put& put) {
    std::vector<WalkStep<T>> st;
    const bool reg = wchi_ <= 8;
    for (size_t at_ = 0; at_ < wsteps_.size(); ++at_) {
      const WalkVertex& w = wsteps_[at_];
      const EvalVertex& e = tree_.v[w.v];
      WalkStep<T> s{};
      s.B = e.absorb ? abs_[w.v] : ten_[w.v];
      s.gexp = e.absorb ? abse_[w.v] : nullptr;
      s.key = key_slot_[w.v];
      s.chi_a = e.chi;
      s.d1 = w.d1;
      s.d2 = w.d2;
      s.c1 = s.c2 = -1;
      for (int i = 0; i < w.nk; ++i) {
        const int k = e.kids[i];
        const bool last = i + 1 == w.nk, tab = tree_.v[k].tabled;
        (last ? s.t2 : s.t1) = tab ? tab_[k] : nullptr;
        (last ? s.e2 : s.e1) = tab ? tabe_[k] : nullptr;
        (last ? s.c2 : s.c1) = tab ? row_slot_[k] : msg_[k];
        // the previous step's message, still in registers
        if (reg && last && !tab && at_ != (size_t)nsteps0_ && at_ > 0 && wsteps_[at_ - 1].v == k) s.c2 = -2;
      }
      if (e.absorb || !e.moved) {
        s.s2 = 1;
        s.s1 = w.d2;
        s.sa = w.d1 * w.d2;
        s.sg = e.chi * s.sa;
      } else {  // the stored tensor's strides in the order read
        const std::vector<int64_t> str = stored_strides(w.v);
        // axes: sites, (a root's parent axis of dimension 1,) up, kids
        const int at = (int)str.size() - w.nk;
        s.sg = (int)str[0];
        s.sa = e.up >= 0 ? (int)str[at - 1] : 0;
        s.s1 = w.nk == 2 ? (int)str[at] : 0;
        s.s2 = w.nk >= 1 ? (int)str[at + w.nk - 1] : 0;
      }
      s.out = msg_[w.v];
      s.stage = nstage_ && !e.absorb && ten_[w.v] == tensors_ + topo_.off[w.v] ? (int)topo_.off[w.v] : -1;
      st.push_back(s);
    }
    // a message that only the next step reads, from registers, is not stored
    for (size_t i = 0; i + 1 < st.size(); ++i)
      if (st[i + 1].c2 == -2) st[i].out = -1;
    unsigned char* at = dwalk_;
    put(at, runs_.data(), runs_.size() * sizeof(DigitRun));
    at += runs_.size() * sizeof(DigitRun);
    put(at, st.data(), st.size() * sizeof(WalkStep<T>));
    at += st.size() * sizeof(WalkStep<T>);
    std::vector<WalkSide<T>> sd;
    for (const auto& c : tree_.comps)
      for (int v : {c.a, c.b}) {
        WalkSide<T> s{};
        if (v >= 0) {
          const EvalVertex& e = tree_.v[v];
          s.chi = e.chi;
          s.tab = e.tabled ? tab_[v] : nullptr;
          s.exps = e.tabled ? tabe_[v] : nullptr;
          s.at = e.tabled ? row_slot_[v] : msg_[v];
        }
        sd.push_back(s);
      }
    put(at, sd.data(), sd.size() * sizeof(WalkSide<T>));
  }

  void walk(const double* X, int n, void* out, int kind, int64_t Pout, int64_t pofs) {
    WalkParams<T> W{};
    W.X = X;
    W.blob = dwalk_;
    W.tensors = tensors_;
    W.out = out;
    W.err = err_;
    W.P = Pout;
    W.p0 = pofs;
    W.ncols = ncols_;
    W.Pc = n;
    W.nruns = (int)runs_.size();
    W.nslots = nslots_;
    W.nsteps0 = nsteps0_;
    W.nsteps = (int)wsteps_.size();
    W.ncomp = (int)tree_.comps.size();
    W.nmsg = wmsg_;
    W.nstage = nstage_;
    W.kind = kind;
    const size_t sm = walk_bytes();
    double fl = 0;
    for (const auto& w : wsteps_) fl += 2.0 * tree_.v[w.v].chi * w.d1 * w.d2;
    KernelScope ks(ctx_, "eval_fused", fl * n, (double)n * (ncols_ * 8.0 + 8.0));
    const int per_sm = std::max(1, std::min((int)(220 * 1024 / std::max<size_t>(sm, 1)), 1024 / (wtp_ * wlanes_)));
    const unsigned grid = grid_for(n, wtp_, ctx_->sm_count * per_sm);
    auto go = [&](auto kern) {
      if (sm > 48 * 1024)
        TNFA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
      kern<<<grid, 2 * wtp_ * wlanes_, sm, ctx_->stream>>>(W);
    };
    if (wchi_ == 2) wlanes_ == 1 ? go(k_walk<T, 2, 1>) : go(k_walk<T, 2, 2>);
    else if (wchi_ == 4) wlanes_ == 1 ? go(k_walk<T, 4, 1>) : wlanes_ == 2 ? go(k_walk<T, 4, 2>) : go(k_walk<T, 4, 4>);
    else if (wchi_ == 8) wlanes_ == 1 ? go(k_walk<T, 8, 1>) : wlanes_ == 2 ? go(k_walk<T, 8, 2>) : go(k_walk<T, 8, 4>);
    else if (wchi_ == 16) go(k_walk<T, 16, 1>);
    else go(k_walk<T, 32, 1>);
    TNFA_LAUNCH_CHECK();
  }

  MoveJob move_job(int v) const {
    const EvalVertex& e = tree_.v[v];
    std::vector<int> shape{topo_.site_dim[v], topo_.link[v]};
    for (int c : topo_.children[v]) shape.push_back(topo_.link[c]);
    TNFA_CHECK(shape.size() <= (size_t)MOVE_MAXD, TNFA_ERR_UNSUPPORTED, "vertex degree too high");
    const std::vector<int64_t> str = stored_strides(v);
    MoveJob m{};
    m.src = tensors_ + topo_.off[v];
    m.dst = ten_[v];
    m.n = topo_.size(v);
    m.nd = (int)e.axes.size();
    for (int i = 0; i < m.nd; ++i) {
      m.dim[i] = shape[e.axes[i]];
      m.str[i] = str[i];
    }
    return m;
  }
  // The absorption of the last kid's table into the tensor of v.
  RowJob<T> absorb_job(int v) const {
    const EvalVertex& e = tree_.v[v];
    const int w = e.kids.back();
    const EvalVertex& k = tree_.v[w];
    RowJob<T> j{};
    j.A = tab_[w];
    j.Aexp = tabe_[w];
    j.aidx = table_row(1, k.N);
    j.B = ten_[v];
    j.out = abs_[v];
    j.out_exp = abse_[v];
    j.rex = rex_[w];
    j.K = k.chi;
    j.N = (int)(e.W / k.chi);
    j.rpg = (int)k.N;
    j.rows = topo_.site_dim[v] * j.rpg;
    return j;
  }
  // The table of v from its one kid (besides the absorbed one).
  RowJob<T> table_job(int v) const {
    const EvalVertex& e = tree_.v[v];
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
    j.rex = rex_[w];
    j.K = k.chi;
    j.N = e.chi;
    j.rpg = (int)k.N;
    j.rows = (int)e.N;
    return j;
  }
  template <class Put>
  void fill_head(Put& put) {
    std::vector<HeadBlock<T>> hb;
    std::vector<HeadCopy<T>> cp;
    std::vector<HeadJob> jobs;
    head_k_ = 1;
    head_elems_ = head_exps_ = head_jobs_ = 0;
    for (const auto& g : hgroups_) {
      HeadBlock<T> h{};
      int at = 0, ea = 0;
      h.copy0 = (int)cp.size();
      h.job0 = (int)jobs.size();
      std::vector<int> ten(topo_.V, -1), tab(topo_.V, -1), te(topo_.V, -1);
      auto stage = [&](int v) {
        cp.push_back({tensors_ + topo_.off[v], at, (int)topo_.size(v)});
        ten[v] = at;
        at += (int)topo_.size(v);
      };
      for (int v : g) {
        stage(v);
        for (int w : tree_.v[v].kids)
          if (tree_.v[w].leaf) {
            stage(w);
            tab[w] = ten[w];
          }
      }
      for (int v : g) {
        const EvalVertex& e = tree_.v[v];
        const std::vector<int64_t> str = stored_strides(v);
        const int nk = (int)e.kids.size(), up = e.up >= 0 ? (int)str[str.size() - nk - 1] : 0;
        int mo = -1, me = -1;
        auto rows_of = [&](HeadJob& j, int w) {
          j.A = tab[w];
          j.Aexp = te[w];
          j.lda = tree_.v[w].leaf ? tree_.v[w].chi : table_pitch(tree_.v[w].chi);
          j.K = tree_.v[w].chi;
          j.rpg = (int)tree_.v[w].N;
        };
        if (e.absorb) {  // columns (up, the other kid)
          HeadJob j{};
          rows_of(j, e.kids[1]);
          j.B = ten[v];
          j.gexp = -1;
          j.bg = (int)str[0];
          j.n2 = tree_.v[e.kids[0]].chi;
          j.N = e.chi * j.n2;
          j.bn1 = up;
          j.bn2 = (int)str[str.size() - 2];
          j.bk = (int)str.back();
          j.rows = topo_.site_dim[v] * j.rpg;
          j.out = mo = at;
          j.ldo = j.N;
          j.oexp = me = ea;
          at += j.rows * j.N;
          ea += j.rows;
          j.level = lvl_m_[v];
          jobs.push_back(j);
        }
        HeadJob j{};
        rows_of(j, e.kids[0]);
        j.N = j.n2 = e.chi;
        j.B = e.absorb ? mo : ten[v];
        j.gexp = e.absorb ? me : -1;
        j.bk = e.absorb ? 1 : (int)str.back();
        j.bn2 = e.absorb ? j.K : up;
        j.bg = e.absorb ? j.N * j.K : (int)str[0];
        j.rows = (int)e.N;
        j.out = tab[v] = at;
        j.ldo = table_pitch(e.chi);
        j.oexp = te[v] = ea;
        at += j.rows * j.ldo;
        ea += j.rows;
        j.level = lvl_[v];
        jobs.push_back(j);
      }
      h.copy1 = (int)cp.size();
      h.job1 = (int)jobs.size();
      std::stable_sort(jobs.begin() + h.job0, jobs.end(),
                       [](const HeadJob& x, const HeadJob& y) { return x.level < y.level; });
      const int v = g.back();
      h.tab = tab_[v];
      h.exps = tabe_[v];
      h.top = tab[v];
      h.topexp = te[v];
      h.chi = tree_.v[v].chi;
      h.ld = table_pitch(h.chi);
      h.rows = (int)tree_.v[v].N;
      h.plain = (int)hb.size();
      for (const auto& c : tree_.comps) h.centre |= !walk_ && (c.a == v || c.b == v);
      hb.push_back(h);
      head_elems_ = std::max(head_elems_, at);
      head_exps_ = std::max(head_exps_, ea);
      head_jobs_ = std::max(head_jobs_, h.job1 - h.job0);
    }
    for (const auto& j : jobs) head_k_ = std::max(head_k_, j.K);
    head_elems_ += head_elems_ & 1;  // the exponents and jobs behind stay aligned
    put(dhblocks_, hb.data(), hb.size() * sizeof(HeadBlock<T>));
    put(dhcopies_, cp.data(), cp.size() * sizeof(HeadCopy<T>));
    put(dhjobs_, jobs.data(), jobs.size() * sizeof(HeadJob));
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
  static void bind_groups(VertexJob<T>& j, int* meta) {
    j.grp_off = meta;
    j.grp_cnt = meta + j.ngroups;
    j.tile_start = meta + 2 * j.ngroups;
  }
  void contract_vertex(int v, VertexJob<T>& j, int* meta, bool keyed, int tp) {
    const int ng = j.ngroups;
    bind_groups(j, meta);
    if (tree_.v[v].tensor) {
      if constexpr (std::is_same<T, float>::value) {
        tc_contract_vertex(ctx_, net_, v, j, tp, err_);
        return;
      }
      if constexpr (std::is_same<T, double>::value) {
        oz_contract(ctx_, net_, {{v, j}}, err_);
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
      launch_rows<T>(ctx_, t, row_blocks(j, t), pack_rows<T>({j}, {0, 0}, nullptr, nullptr));
    });
  }
  int group_tile(const RowJob<T>& j) const { return row_tile<T>(ctx_, {j}); }

  void centre_pair(const double* X, int n, void* out, int kind, int64_t Pout, int64_t pofs) {
    const int a = tree_.comps[0].a, b = tree_.comps[0].b;
    PairParams<T> W{};
    W.X = X;
    W.out = out;
    W.err = err_;
    W.P = Pout;
    W.p0 = pofs;
    W.A = tab_[a];
    W.B = tab_[b];
    W.ea = tabe_[a];
    W.eb = tabe_[b];
    W.ncols = ncols_;
    W.Pc = n;
    W.nruns = (int)runs_.size();
    W.chi = tree_.v[a].chi;
    W.sa = row_slot_[a];
    W.sb = row_slot_[b];
    W.kind = kind;
    W.scale = tree_.v[a].leaf || tree_.v[b].leaf;
    std::copy(runs_.begin(), runs_.end(), W.runs);
    KernelScope ks(ctx_, "eval_fused", 2.0 * n * W.chi, (double)n * (ncols_ * 8.0 + 8.0));
    W.na = (int)tree_.v[a].N;
    W.nb = (int)tree_.v[b].N;
    W.pa = plain_of_[a] >= 0 && !walk_ ? plain_ + plain_of_[a] : nullptr;
    W.pb = plain_of_[b] >= 0 && !walk_ ? plain_ + plain_of_[b] : nullptr;
    constexpr int vec = 16 / sizeof(T);
    // short rows gathered by many points: from shared memory, if 4 blocks of it
    // fit an SM and every copied row is read about 8 times or more
    const size_t sm = ((size_t)(W.na + W.nb) * W.chi + 2 * vec) * sizeof(T);
    const bool shared = W.chi * sizeof(T) <= 64 && sm <= 48 * 1024 &&
                        (double)n >= 8.0 * (W.na + W.nb) * ctx_->sm_count;
    const unsigned grid = grid_for(n, 256, ctx_->sm_count * (shared ? 4 : 8));
    bool few = W.nruns >= 1 && W.nruns <= 2;
    for (int i = 0; i < std::min(W.nruns, 2); ++i) few &= W.runs[i].bits != 0;
    auto run = [&](auto kern, size_t bytes) { kern<<<grid, 256, bytes, ctx_->stream>>>(W); };
    auto go = [&](auto g, auto v, auto may_share) {
      constexpr int GG = decltype(g)::value, VV = decltype(v)::value;
      if constexpr (decltype(may_share)::value) {
        if (shared) {
          few ? run(k_centre_pair<T, GG, VV, true, true>, sm) : run(k_centre_pair<T, GG, VV, true, false>, sm);
          return;
        }
      }
      few ? run(k_centre_pair<T, GG, VV, false, true>, 0) : run(k_centre_pair<T, GG, VV, false, false>, 0);
    };
    using std::integral_constant;
    if constexpr (vec > 1) {
      if (centre_vec_) {
        const int lanes = (W.chi + vec - 1) / vec;
        if (lanes <= 2) go(integral_constant<int, 1>{}, integral_constant<int, vec>{}, std::true_type{});
        else if (lanes <= 4) go(integral_constant<int, 4>{}, integral_constant<int, vec>{}, std::true_type{});
        else go(integral_constant<int, 8>{}, integral_constant<int, vec>{}, std::false_type{});
        TNFA_LAUNCH_CHECK();
        return;
      }
    }
    if (W.chi <= 4) go(integral_constant<int, 1>{}, integral_constant<int, 1>{}, std::true_type{});
    else if (W.chi <= 8) go(integral_constant<int, 4>{}, integral_constant<int, 1>{}, std::true_type{});
    else go(integral_constant<int, 8>{}, integral_constant<int, 1>{}, std::true_type{});
    TNFA_LAUNCH_CHECK();
  }

  void centre(const double* X, int n, void* out, int kind, int64_t Pout, int64_t pofs) {
    const int ns = fused_ ? nslots_ : 0;
    const size_t sm = 256 * (sizeof(T) + 4) + (size_t)ns * 1024 + (fused_ ? runs_.size() * sizeof(DigitRun) : 0);
    if (fused_ && tree_.comps.size() == 1 && tree_.comps[0].b >= 0 && runs_.size() <= (size_t)CENTRE_RUNS) {
      centre_pair(X, n, out, kind, Pout, pofs);
      return;
    }
    KernelScope ks(ctx_, fused_ ? "eval_fused" : "centre", 2.0 * n * centre_chi_, (double)n * (ncols_ * 8.0 + 8.0));
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
  bool use_tc_, use_oz_, adjoint_;
  EvalTree tree_;
  std::vector<int> ttile_;  // tile rows that the group table of a table vertex was made for
  std::vector<int> slot_, mult_, key_slot_, row_slot_, msg_, lvl_, lvl_m_;
  std::vector<DigitRun> runs_;
  std::vector<Level> levels_;
  int nslots_ = 0, ncodes_ = 0, nmsg_ = 0, msg_chi_ = 1, npp_ = 0, Pc_ = 0, centre_chi_ = 1;
  int64_t max_group_ = 1, ld_ = 0;
  bool fused_ = false, centre_vec_ = false, small_ = false, walk_ = false;
  struct WalkVertex {
    int v, nk, d1, d2;
  };
  std::vector<WalkVertex> wsteps_;
  int wchi_ = 1, wmsg_ = 0, wtp_ = 32, wlanes_ = 1, nstage_ = 0, nsteps0_ = 0;
  unsigned char* dwalk_ = nullptr;
  // head of the tables: groups of vertices by block
  std::vector<char> head_;
  std::vector<int> plain_of_;  // head block of its top vertex
  std::vector<std::vector<int>> hgroups_;
  int nhead_jobs_ = 0, nhead_copies_ = 0, head_k_ = 1, head_elems_ = 0, head_exps_ = 0, head_jobs_ = 0;
  int* plain_ = nullptr;  // per head block: the exponent that all its rows carry, or INT_MIN
  HeadBlock<T>* dhblocks_ = nullptr;
  HeadCopy<T>* dhcopies_ = nullptr;
  HeadJob* dhjobs_ = nullptr;
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
  std::vector<int*> tmeta_, tabe_, abse_, rex_;
  std::vector<T*> ten_, tab_, abs_;
  int *codes_ = nullptr, *perm_ = nullptr, *meta_ = nullptr, *mexp_ = nullptr;
  T* mval_ = nullptr;
};

static size_t out_elem_size(int out_kind) {
  return out_kind == TNFA_OUT_F64 ? 8 : out_kind == TNFA_OUT_F32 ? 4 : out_kind == TNFA_OUT_F32_SCALED ? 8 : 16;
}

static void check_error_word(int herr) {
  TNFA_CHECK((herr & 2) == 0, TNFA_ERR_TIMEOUT,
             "a tensor-core pipeline wait ran out of its iteration budget");
  TNFA_CHECK(herr == 0, TNFA_ERR_DOMAIN,
             "a coordinate is negative or not finite (the digit map needs x >= 0)");
}
static void check_eval_error(tnfa_ctx* ctx, const int* derr) {
  int herr = 0;
  TNFA_CUDA(cudaMemcpyAsync(&herr, derr, 4, cudaMemcpyDeviceToHost, ctx->stream));
  TNFA_CUDA(cudaStreamSynchronize(ctx->stream));
  check_error_word(herr);
}

template <class T>
static void evaluate_impl(tnfa_ctx* ctx, const tnfa_net* net, const T* tensors, const double* X,
                          int64_t P, int ncols, const std::vector<DigitRef>& prog, int xmem,
                          void* out, int out_kind, int out_mem, bool use_tc,
                          bool use_oz = false) {
  const size_t out_elem = out_elem_size(out_kind);
  const size_t staged = (xmem == TNFA_MEM_HOST ? ncols * 8 : 0) + (out_mem == TNFA_MEM_HOST ? out_elem : 0);
  EvalEngine<T> E(ctx, net, tensors, prog, ncols, P, use_tc, use_oz, ctx->eval_budget);
  int64_t Pcap = E.chunk();
  if (staged) Pcap = std::min(Pcap, std::max<int64_t>(256, (int64_t)(ctx->eval_budget / staged) / 256 * 256));
  Pcap = std::max<int64_t>(1, std::min(P, Pcap));
  DBuf dX(ctx, xmem == TNFA_MEM_HOST ? (size_t)Pcap * ncols * 8 : 0);
  DBuf dout(ctx, out_mem == TNFA_MEM_HOST ? (size_t)Pcap * out_elem : 0);
  E.set_chunk((int)Pcap);
  DBuf arena(ctx, E.scratch(Pcap));
  E.bind(arena.p);
  E.upload();
  int* const err = error_word(ctx);
  E.use_error(err);
  E.tables();
  for (int64_t p0 = 0; p0 < P; p0 += Pcap) {
    const int Pc = (int)std::min<int64_t>(Pcap, P - p0);
    const double* Xc = X + p0 * ncols;
    if (xmem == TNFA_MEM_HOST) {
      TNFA_CUDA(cudaMemcpyAsync(dX.p, Xc, (size_t)Pc * ncols * 8, cudaMemcpyHostToDevice, ctx->stream));
      Xc = dX.as<double>();
    }
    void* o = out_mem == TNFA_MEM_HOST ? dout.p : out;
    const int64_t Pout = out_mem == TNFA_MEM_HOST ? Pc : P, pofs = out_mem == TNFA_MEM_HOST ? 0 : p0;
    E.points(Xc, Pc, o, out_kind, Pout, pofs);
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
  TNFA_CUDA(cudaStreamSynchronize(ctx->stream));
  check_error_word(*(volatile int*)err);
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

// Scratch bytes by which a request is accepted: a limit of the interface, not
// what a call uses (it works in chunks that fit, FixedRun).  Requests are taken
// up to the point count whose digits, permutation, group tables, root values
// and messages, one row per point for every message alive at once in a
// depth-first contraction, fit the array.
template <class T>
size_t noalloc_bytes(const tnfa_net* net, int64_t P, size_t prog_entries) {
  const Topo& Tp = net->topo;
  int maxsd = 1, chimax = 1;
  for (int v = 0; v < Tp.V; ++v) maxsd = std::max(maxsd, Tp.site_dim[v]);
  // messages alive at once below and at every vertex (a leaf's is read in place)
  std::vector<int> alive(Tp.V, 0);
  size_t nroots = 0;
  int nslots = 0;
  for (int v = Tp.V - 1; v >= 0; --v) {  // children before parents
    const bool root = Tp.parent[v] < 0;
    nroots += root;
    int held = 0;
    for (int c : Tp.children[v]) {
      alive[v] = std::max(alive[v], held + alive[c]);
      held += !Tp.children[c].empty();
    }
    if (root) {
      nslots = std::max(nslots, alive[v]);
    } else if (!Tp.children[v].empty()) {
      alive[v] = std::max(alive[v], held + 1);
      chimax = std::max(chimax, Tp.link[v]);
    }
  }
  std::array<size_t, 10> sizes{prog_entries * 32, 0, 0, 0, 0, 4, 0, 0, 0, 0};
  if (small_bonds(Tp, sizeof(T), P)) {
    sizes[1] = (size_t)Tp.V * 36;
  } else {
    sizes[2] = (size_t)Tp.V * P;
    sizes[3] = (size_t)P * 4;
    sizes[4] = group_meta_ints(maxsd) * 4;
    sizes[6] = (size_t)nslots * P * chimax * sizeof(T);
    sizes[7] = (size_t)nslots * P * sizeof(int);
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
      : ncols_(ncols), P_(P), E_(ctx, net, tensors, prog, ncols, P, false, false, budget) {
    int pc = E_.chunk();
    while (pc > 1 && E_.scratch(pc) > budget) pc = std::max(1, pc / 2);
    E_.set_chunk(pc);
  }
  size_t bytes() { return E_.scratch(E_.chunk()); }
  void bind(void* base) { E_.bind(base); }
  void stage() { E_.upload(); }
  int* err_flag() const { return E_.err_flag(); }
  void enqueue(const double* X, void* out, int out_kind) {
    E_.clear_error();
    E_.tables();
    for (int64_t p0 = 0; p0 < P_; p0 += E_.chunk())
      E_.points(X + p0 * ncols_, (int)std::min<int64_t>(E_.chunk(), P_ - p0), out, out_kind, P_, p0);
  }

 private:
  int ncols_;
  int64_t P_;
  EvalEngine<T> E_;
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
namespace tnfa {
namespace {

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
size_t grad_acc_smem(int sumdim, int tp) {
  return (size_t)sumdim * tp * sizeof(T) + tp * sizeof(T) + 2 * tp * sizeof(int);
}

// dT += the job's sums (children: the outside message, then the kids).
template <class T, int TP, int KQ>
void launch_grad_acc(tnfa_ctx* ctx, const VertexJob<T>& j, int sumdim, int Pc, T* dT) {
  const size_t sm = grad_acc_smem<T>(sumdim, TP);
  auto kern = k_grad_acc<T, TP, KQ>;
  if (sm > 48 * 1024)
    TNFA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  // one wave of resident CTAs, each over a run of consecutive tiles
  int occ = 0;
  TNFA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 256, sm));
  const int ntiles = (int)((Pc + TP - 1) / TP + j.ngroups);
  const int ky = (int)((j.K + 256 * KQ - 1) / (256 * KQ));
  const int want = std::max(1, std::max(occ, 1) * ctx->sm_count / ky);
  const int per = std::max(1, (ntiles + want - 1) / want);
  dim3 grid((unsigned)((ntiles + per - 1) / per), (unsigned)ky);
  KernelScope ks(ctx, "grad_acc", 2.0 * Pc * (double)j.K, 0.0);
  kern<<<grid, 256, sm, ctx->stream>>>(j, dT, per);
  TNFA_LAUNCH_CHECK();
}

// d/dT of sum_p dout_p f(x_p), on the table schedule of the evaluation.  With
// the two rows A, B that meet at the centre for point p, the adjoint of a
// table's row is the sum of dout_p times the other side's row over the points
// that read it; from there the products that built the tables are run
// backwards, once per table row instead of once per point.  A vertex without a
// table has one adjoint row per point (E), the adjoint of its message: E of a
// kid is the same contraction with that kid's bond as the output (the tensor
// with the kid's axis moved first, E as one more input), and
//   dT_v[s][a][c1..ck] += sum_{p: s_v(p) = s} E_v[p][a] prod_j m_cj[p][c_j]
// (k_grad_acc).  All adjoints carry one common power of two per chunk, taken
// from the largest weight, so that networks of tiny values do not lose their
// FP32 gradients on the way.
template <class T>
class AdjointEngine : public EvalEngine<T> {
  using Base = EvalEngine<T>;
  using Base::abs_;
  using Base::abse_;
  using Base::codes_;
  using Base::ctx_;
  using Base::dcentre_;
  using Base::druns_;
  using Base::err_;
  using Base::key_slot_;
  using Base::ld_;
  using Base::lvl_;
  using Base::lvl_m_;
  using Base::mexp_;
  using Base::meta_;
  using Base::msg_;
  using Base::msg_chi_;
  using Base::mval_;
  using Base::ncodes_;
  using Base::ncols_;
  using Base::nmsg_;
  using Base::Pc_;
  using Base::perm_;
  using Base::rex_;
  using Base::row_slot_;
  using Base::runs_;
  using Base::tab_;
  using Base::tabe_;
  using Base::ten_;
  using Base::topo_;
  using Base::tree_;

 public:
  AdjointEngine(tnfa_ctx* ctx, const tnfa_net* net, const T* tensors, const std::vector<DigitRef>& prog, int ncols,
                int64_t P, size_t budget, double max_rows)
      : Base(ctx, net, tensors, prog, ncols, P, false, false, budget, true, max_rows) {
    const int V = topo_.V;
    has_e_.assign(V, 0);
    for (int v = 0; v < V; ++v)
      if (!tree_.v[v].tabled)
        for (int w : tree_.v[v].kids) has_e_[w] = 1;
    for (const EvalTree::Comp& c : tree_.comps) {
      if (!tree_.v[c.a].tabled) has_e_[c.a] = 1;
      if (c.b >= 0 && !tree_.v[c.b].tabled) has_e_[c.b] = 1;
    }
    const size_t fixed = this->scratch(0) + adjoint_scratch(0);
    const size_t per = (this->scratch(1 << 12) + adjoint_scratch(1 << 12) - fixed) / (1 << 12) + 1;
    const size_t left = budget > fixed ? budget - fixed : 0;
    const int64_t pc = std::max<int64_t>(256, std::min<int64_t>((int64_t)(left / per) / 256 * 256, int64_t(1) << 30));
    Pc_ = (int)std::min<int64_t>(P, pc);
  }
  size_t bytes() { return this->scratch(Pc_) + adjoint_scratch(Pc_); }
  void bind_all(void* base, T* dT) {
    const size_t own = (this->scratch(Pc_) + 255) / 256 * 256;
    this->bind(base);
    Carve c;
    c.base = (unsigned char*)base + own;
    lay_out_adjoint(c, Pc_);
    fill_adjoint(dT);
  }
  void upload_all() {
    this->upload();
    h2d(ctx_, blob_, host_.data(), host_.size());
    for (const auto& m : tmoves_) max_move_ = std::max(max_move_, m.n);
    if (!tmoves_.empty()) {
      k_move<T><<<dim3(grid_for(max_move_, 256, 1024), (unsigned)tmoves_.size()), 256, 0, ctx_->stream>>>(dtmoves_);
      TNFA_LAUNCH_CHECK();
    }
  }

  // Adds the gradient of the chunk's n points.
  void chunk_gradient(const double* X, int n, const double* dout) {
    cudaStream_t st = ctx_->stream;
    if (ncodes_ > 0) launch_digitize(ctx_, X, ncols_, n, druns_, (int)runs_.size(), ncodes_, codes_, ld_, err_);
    for (int v : tree_.order)
      if (!tree_.v[v].tabled) this->contract_points(v, n);
    TNFA_CUDA(cudaMemsetAsync(zero_, 0, zero_bytes_, st));
    TNFA_CUDA(cudaMemsetAsync(S_, 0x80, sizeof(int), st));
    const int nc = (int)tree_.comps.size();
    const unsigned grid = grid_for(n, 256, ctx_->sm_count * 8);
    {
      KernelScope ks(ctx_, "adjoint", 0.0, 0.0);
      k_adj_prep<T><<<grid, 256, 0, st>>>(dout, n, dcentre_, nc, wv_, we_, ld_, S_);
      TNFA_LAUNCH_CHECK();
    }
    for (int c = 0; c < nc; ++c) {
      const T* wv = wv_ + (int64_t)(nc + c) * ld_;
      const int* we = we_ + (int64_t)(nc + c) * ld_;
      const int a = tree_.comps[c].a, b = tree_.comps[c].b;
      if (tree_.v[a].tabled || (b >= 0 && tree_.v[b].tabled)) {
        KernelScope ks(ctx_, "adjoint", 0.0, 0.0);
        k_adj_weight<T><<<grid, 256, 0, st>>>(wv, we, n, dcentre_, c, S_, w_);
        TNFA_LAUNCH_CHECK();
      }
      for (int sd = 0; sd < (b >= 0 ? 2 : 1); ++sd) {
        const int v = sd ? b : a, o = sd ? a : b;
        CentreSide<T> other{};
        if (o >= 0) other = this->side(o);
        if (tree_.v[v].tabled) {
          segsum(v, n, other.ptr, other.idx, w_, nullptr);
        } else {
          KernelScope ks(ctx_, "adjoint", 0.0, 0.0);
          const int chi = tree_.v[v].chi;
          k_adj_seed<T><<<grid_for((int64_t)n * chi, 256, ctx_->sm_count * 16), 256, 0, st>>>(
              wv, we, n, other, chi, S_, ev_[v], ee_[v]);
          TNFA_LAUNCH_CHECK();
        }
      }
    }
    for (size_t i = tree_.order.size(); i-- > 0;)
      if (!tree_.v[tree_.order[i]].tabled) points_back(tree_.order[i], n);
    for (size_t l = levels_.size(); l-- > 0;) {
      const BackLevel& L = levels_[l];
      if (L.jobs.empty()) continue;
      KernelScope ks(ctx_, "adjoint_rows", 0.0, 0.0);
      k_rows_back<T><<<(unsigned)L.first.back(), 256, 0, st>>>(L.djobs, L.dfirst, (int)L.jobs.size());
      TNFA_LAUNCH_CHECK();
    }
    k_adj_add<T><<<dim3(grid_for(max_add_, 256, 256), (unsigned)topo_.V), 256, 0, st>>>(dadds_, S_);
    TNFA_LAUNCH_CHECK();
  }

 private:
  struct BackLevel {
    std::vector<BackJob<T>> jobs;
    std::vector<int> first;
    BackJob<T>* djobs = nullptr;
    int* dfirst = nullptr;
    int njobs = 0;
  };

  size_t adjoint_scratch(int64_t pc) {
    Carve c;
    lay_out_adjoint(c, pc);
    return c.used + 512;
  }

  void lay_out_adjoint(Carve& c, int64_t pc) {
    const int V = topo_.V;
    // job tables
    blob_ = (unsigned char*)c.take<MoveJob>(V);
    dadds_ = (MoveJob*)blob_;
    int nt = 0;
    for (int v = 0; v < V; ++v)
      if (!tree_.v[v].tabled) nt += (int)tree_.v[v].kids.size();
    dtmoves_ = c.take<MoveJob>(nt);
    int top = 0;
    for (int v = 0; v < V; ++v)
      if (!tree_.v[v].leaf) top = std::max({top, lvl_m_[v], lvl_[v]});
    levels_.assign(top + 1, BackLevel{});
    for (int v : tree_.order) {
      const EvalVertex& e = tree_.v[v];
      if (e.leaf || !e.tabled) continue;
      levels_[lvl_[v]].njobs += 1;
      if (e.absorb) levels_[lvl_m_[v]].njobs += 1;
    }
    for (auto& L : levels_) {
      L.djobs = c.take<BackJob<T>>(L.njobs);
      L.dfirst = c.take<int>(L.njobs + 1);
    }
    blob_bytes_ = c.used - (size_t)(blob_ - c.base);
    // adjoints that start at zero
    dten_.assign(V, nullptr);
    bar_.assign(V, nullptr);
    dabs_.assign(V, nullptr);
    S_ = c.take<int>(1);
    zero_ = c.take<unsigned char>(1);
    for (int v = 0; v < V; ++v) {
      const EvalVertex& e = tree_.v[v];
      dten_[v] = c.take<T>(topo_.size(v));
      if (e.leaf) bar_[v] = dten_[v];
      else if (e.tabled) bar_[v] = c.take<T>((size_t)e.N * e.chi);
      if (e.absorb)
        dabs_[v] = c.take<T>((size_t)this->absorbed_rows(v) * (size_t)(e.W / tree_.v[e.kids.back()].chi));
    }
    zero_bytes_ = c.used - (size_t)(zero_ - c.base);
    // tensors with a kid's axis first
    tk_.assign(V, nullptr);
    for (int v = 0; v < V; ++v)
      if (!tree_.v[v].tabled)
        for (int w : tree_.v[v].kids) tk_[w] = c.take<T>(topo_.size(v));
    // per point
    const size_t nc = tree_.comps.size();
    wv_ = c.take<T>(2 * nc * pc);
    we_ = c.take<int>(2 * nc * pc);
    w_ = c.take<T>(pc);
    sperm_ = c.take<int>(pc);
    int64_t ng = 1;
    for (int v = 0; v < V; ++v)
      if (tree_.v[v].tabled && row_slot_[v] >= 0) ng = std::max(ng, tree_.v[v].N);
    smeta_ = c.take<int>(group_meta_ints((int)ng));
    ev_.assign(V, nullptr);
    ee_.assign(V, nullptr);
    for (int v = 0; v < V; ++v)
      if (has_e_[v]) {
        ev_[v] = c.take<T>((size_t)pc * tree_.v[v].chi);
        ee_[v] = c.take<int>(pc);
      }
  }

  BackJob<T> back_job(const RowJob<T>& f, int kid, const T* bar, T* dB) const {
    BackJob<T> j{};
    j.A = f.A;
    j.rex = rex_[kid];
    j.B = f.B;
    j.bar = bar;
    j.dB = dB;
    j.dA = bar_[kid];
    j.K = f.K;
    j.N = f.N;
    j.rpg = f.rpg;
    j.ng = f.rows / f.rpg;
    const int nk = (j.K + BACK_T - 1) / BACK_T, nn = (j.N + BACK_T - 1) / BACK_T;
    j.sb = std::max(1, std::min(256, j.rpg / 128));
    j.sa = (int)std::max<int64_t>(1, std::min<int64_t>(256, (int64_t)j.ng * j.N / 256));
    j.nb = nk * nn * j.ng * j.sb;
    return j;
  }
  static int64_t back_blocks(const BackJob<T>& j) {
    return (int64_t)j.nb + (int64_t)((j.K + BACK_T - 1) / BACK_T) * ((j.rpg + BACK_T - 1) / BACK_T) * j.sa;
  }

  void fill_adjoint(T* dT) {
    host_.assign(blob_bytes_, 0);
    auto put = [&](const void* dev, const void* src, size_t n) {
      if (n) std::memcpy(host_.data() + ((const unsigned char*)dev - blob_), src, n);
    };
    std::vector<MoveJob> adds;
    tmoves_.clear();
    max_add_ = max_move_ = 1;
    for (int v = 0; v < topo_.V; ++v) {
      MoveJob m = this->move_job(v);
      m.src = dT + topo_.off[v];
      m.dst = dten_[v];
      adds.push_back(m);
      max_add_ = std::max(max_add_, m.n);
      const EvalVertex& e = tree_.v[v];
      if (e.tabled) continue;
      for (size_t i = 0; i < e.kids.size(); ++i) {  // sites, kid, up, the other kids
        MoveJob t = this->move_job(v);
        t.dst = tk_[e.kids[i]];
        const int nk = (int)e.kids.size(), at = t.nd - nk + (int)i, up = t.nd - nk - 1;
        const int dim = t.dim[at];
        const int64_t str = t.str[at];
        for (int d = at; d > up; --d) {
          t.dim[d] = t.dim[d - 1];
          t.str[d] = t.str[d - 1];
        }
        t.dim[up] = dim;
        t.str[up] = str;
        tmoves_.push_back(t);
      }
    }
    put(dadds_, adds.data(), adds.size() * sizeof(MoveJob));
    put(dtmoves_, tmoves_.data(), tmoves_.size() * sizeof(MoveJob));
    for (int v : tree_.order) {
      const EvalVertex& e = tree_.v[v];
      if (e.leaf || !e.tabled) continue;
      levels_[lvl_[v]].jobs.push_back(
          back_job(this->table_job(v), e.kids[0], bar_[v], e.absorb ? dabs_[v] : dten_[v]));
      if (e.absorb) levels_[lvl_m_[v]].jobs.push_back(back_job(this->absorb_job(v), e.kids.back(), dabs_[v], dten_[v]));
    }
    for (auto& L : levels_) {
      L.first.assign(1, 0);
      int64_t b = 0;
      for (const auto& j : L.jobs) {
        b += back_blocks(j);
        TNFA_CHECK(b < (int64_t(1) << 31), TNFA_ERR_UNSUPPORTED, "gradient block too large");
        L.first.push_back((int)b);
      }
      put(L.djobs, L.jobs.data(), L.jobs.size() * sizeof(BackJob<T>));
      put(L.dfirst, L.first.data(), L.first.size() * sizeof(int));
    }
  }

  // bar[row] += point adjoints (weight w, or E's own exponents) of the table of v.
  void segsum(int v, int n, const T* src, const RowIdx& sidx, const T* w, const int* we) {
    const EvalVertex& e = tree_.v[v];
    const int ng = (int)e.N;
    const int* key = codes_ + (int64_t)row_slot_[v] * ld_;
    const int* perm = launch_group(ctx_, ng > 1 ? key : nullptr, n, ng, SEG_TILE, smeta_, sperm_);
    KernelScope ks(ctx_, "adjoint_sum", 2.0 * n * e.chi, (double)n * e.chi * sizeof(T));
    const int64_t tiles = (n + SEG_TILE - 1) / SEG_TILE + ng;
    k_segsum<T><<<(unsigned)((tiles + 7) / 8), 256, 0, ctx_->stream>>>(
        src, sidx, e.chi, w, we, w ? nullptr : tabe_[v], perm, smeta_, smeta_ + ng, smeta_ + 2 * ng, ng, bar_[v]);
    TNFA_LAUNCH_CHECK();
  }

  ChildSrc<T> kid_src(int w) const {
    ChildSrc<T> s{};
    s.dim = tree_.v[w].chi;
    if (tree_.v[w].tabled) {
      s.ptr = tab_[w];
      s.exps = tabe_[w];
      s.idx.codes = codes_ + (int64_t)row_slot_[w] * ld_;
    } else {
      s.ptr = mval_ + (int64_t)msg_[w] * ld_ * msg_chi_;
      s.exps = mexp_ + (int64_t)msg_[w] * ld_;
    }
    return s;
  }

  // From E of v: E of its kids, the gradient of its tensor, and the rows of
  // the kids' tables.
  void points_back(int v, int n) {
    const EvalVertex& e = tree_.v[v];
    const int ng = topo_.site_dim[v];
    const int* key = key_slot_[v] >= 0 ? codes_ + (int64_t)key_slot_[v] * ld_ : nullptr;
    ChildSrc<T> E{};
    E.ptr = ev_[v];
    E.exps = ee_[v];
    E.dim = e.chi;
    bool grouped = false;
    const int* perm = nullptr;
    auto group = [&](VertexJob<T>& j, int tp) {
      if (!grouped) perm = launch_group(ctx_, key, n, ng, tp, meta_, perm_);
      else launch_retile(ctx_, key != nullptr, n, ng, tp, meta_);
      grouped = true;
      j.perm = perm;
      j.ngroups = ng;
      j.grp_off = meta_;
      j.grp_cnt = meta_ + ng;
      j.tile_start = meta_ + 2 * ng;
      j.site_dim = ng;
      j.Pc = n;
    };
    for (int w : e.kids) {
      VertexJob<T> j{};
      j.ch[j.nchild++] = E;
      int64_t K = e.chi;
      int sumdim = e.chi;
      for (int o : e.kids)
        if (o != w) {
          TNFA_CHECK(j.nchild < EVAL_MAXC, TNFA_ERR_UNSUPPORTED, "vertex degree too high");
          j.ch[j.nchild++] = kid_src(o);
          K *= tree_.v[o].chi;
          sumdim += tree_.v[o].chi;
        }
      j.K = (int)K;
      j.chi_a = tree_.v[w].chi;
      j.B = tk_[w];
      j.out = ev_[w];
      j.out_exp = ee_[w];
      group(j, contract_tile_rows(j.chi_a, sumdim, sizeof(T)));
      launch_contract<T>(ctx_, j, n);
    }
    VertexJob<T> j{};
    j.ch[j.nchild++] = E;
    int64_t K = e.chi;
    int sumdim = e.chi;
    for (int w : e.kids) {
      TNFA_CHECK(j.nchild < EVAL_MAXC, TNFA_ERR_UNSUPPORTED, "vertex degree too high");
      j.ch[j.nchild++] = kid_src(w);
      K *= tree_.v[w].chi;
      sumdim += tree_.v[w].chi;
    }
    j.K = (int)K;
    j.chi_a = 1;
    constexpr int TP = 64, KQ = 4;
    group(j, TP);
    launch_grad_acc<T, TP, KQ>(ctx_, j, sumdim, n, dten_[v]);
    for (int w : e.kids)
      if (tree_.v[w].tabled) segsum(w, n, ev_[w], RowIdx{}, nullptr, ee_[w]);
  }

  std::vector<char> has_e_;
  std::vector<BackLevel> levels_;
  std::vector<unsigned char> host_;
  std::vector<MoveJob> tmoves_;
  int64_t max_add_ = 1, max_move_ = 1;
  size_t blob_bytes_ = 0, zero_bytes_ = 0;
  unsigned char *blob_ = nullptr, *zero_ = nullptr;
  MoveJob *dadds_ = nullptr, *dtmoves_ = nullptr;
  std::vector<T*> dten_, bar_, dabs_, tk_, ev_;
  std::vector<int*> ee_;
  T *wv_ = nullptr, *w_ = nullptr;
  int *we_ = nullptr, *S_ = nullptr, *sperm_ = nullptr, *smeta_ = nullptr;
};

template <class T>
void vjp_impl(tnfa_ctx* ctx, const tnfa_net* net, const T* tensors, const double* X, int64_t P,
              int ncols, const std::vector<DigitRef>& prog, int xmem, const double* dout,
              int dout_mem, T* dT) {
  const Topo& Tp = net->topo;
  // shapes the per-point kernels take (whether or not this call runs them)
  for (int v = 0; v < Tp.V; ++v) {
    TNFA_CHECK(Tp.children[v].size() < (size_t)EVAL_MAXC, TNFA_ERR_UNSUPPORTED, "vertex degree too high");
    int64_t K = Tp.link[v], sumdim = Tp.link[v];
    for (int c : Tp.children[v]) {
      K *= Tp.link[c];
      sumdim += Tp.link[c];
    }
    TNFA_CHECK(K < (int64_t(1) << 31), TNFA_ERR_UNSUPPORTED, "gradient block too large");
    TNFA_CHECK(grad_acc_smem<T>((int)sumdim, 64) <= 200 * 1024, TNFA_ERR_UNSUPPORTED,
               "bonds too large for the gradient kernel");
  }
  const size_t staged = (xmem == TNFA_MEM_HOST ? ncols * 8 : 0) + (dout_mem == TNFA_MEM_HOST ? 8 : 0);
  // The tables run backwards once per chunk: no table may be longer than one.
  // (A path of 48 vertices, bond 46, FP64, 4 x 10^6 points: 120 chunks behind
  // tables of 2 x 10^6 rows took 13.4 s, the points alone 6.0.)
  double rows = 134217728.0;
  std::unique_ptr<AdjointEngine<T>> engine;
  for (;;) {
    engine.reset(new AdjointEngine<T>(ctx, net, tensors, prog, ncols, P, ctx->eval_budget, rows));
    if (engine->chunk() >= P || engine->table_rows() <= engine->chunk()) break;
    rows = engine->chunk();
  }
  AdjointEngine<T>& E = *engine;
  int64_t Pcap = E.chunk();
  if (staged) Pcap = std::min(Pcap, std::max<int64_t>(256, (int64_t)(ctx->eval_budget / staged) / 256 * 256));
  E.set_chunk((int)Pcap);
  DBuf dX(ctx, xmem == TNFA_MEM_HOST ? (size_t)Pcap * ncols * 8 : 0);
  DBuf ddout(ctx, dout_mem == TNFA_MEM_HOST ? (size_t)Pcap * 8 : 0);
  DBuf arena(ctx, E.bytes() + 512);
  E.bind_all(arena.p, dT);
  E.upload_all();
  int* const err = error_word(ctx);
  E.use_error(err);
  E.tables();
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
    E.chunk_gradient(Xc, Pc, dc);
  }
  TNFA_CUDA(cudaStreamSynchronize(ctx->stream));
  check_error_word(*(volatile int*)err);
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

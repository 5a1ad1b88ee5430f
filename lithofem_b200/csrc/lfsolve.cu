// liblfsolve.so -- multifrontal sparse LU for the assembled LithoFEM systems
// on B200 (sm_100a), in place of the reference's cuDSS solver
// (solver/cudss_solver.inc:79-309).  C ABI: include/lfsolve.h.
//
// Pipeline
//   analyze (host): nested dissection of the mesh by element bisection (a
//     subdomain's elements are split at the median centroid coordinate
//     along the axis that gives the smallest separator; the separator is the
//     set of still unnumbered DOFs that elements of both halves touch), the
//     postorder elimination tree, every front's index list (its pivots, then
//     the ancestor DOFs its subtree touches) and the maps below;
//   factor (device): depth by depth from the deepest level, the fronts of a
//     level are written from their children's Schur complements, receive their
//     original entries (CSR position -> front offset map) and are partially
//     factored, in groups of similar shape: P F11 = L11 U11 with partial pivoting among
//     the front's pivot rows, all fronts of the level together in own kernels
//     (lfsolve_lu.cuh), U12 = L11^-1 P F12 and L21 = F21 U11^-1 in leaves of
//     64 pivots with matrix products between them (lfsolve_trsm.cuh), F22 -=
//     L21 U12 (library gemm; complex64 on TF32 tensor cores in split form);
//     the L and U blocks are copied to the factor store;
//   solve (device): forward and backward sweeps over the tree, each front's
//     right-hand side gathered from the global vector and its children's
//     update vectors (no atomics), the triangles in steps of 256 pivots
//     (lfsolve_sweeps.cuh); A^T is solved with the same factors (U^T forward,
//     L^T backward, inverse pivots last);
//   refine: FP64 residual on the complex128 CSR, corrections from the
//     factors, per right-hand-side column.
#include <cublas_v2.h>
#include <cuComplex.h>
#include <cuda_runtime.h>
#include <cusolverDn.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <complex>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <numeric>
#include <string>
#include <thread>
#include <vector>

#include "../../include/lfsolve.h"

namespace {

thread_local std::string g_err;

int fail(int code, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  std::vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_err = buf;
  return code;
}

#define LS_CUDA(call)                                                                   \
  do {                                                                                  \
    cudaError_t e_ = (call);                                                            \
    if (e_ != cudaSuccess) {                                                            \
      std::printf("lfsolve: CUDA error '%s' at %s:%d\n", cudaGetErrorString(e_),        \
                  __FILE__, __LINE__);                                                  \
      std::fflush(stdout);                                                              \
      return fail(LFSOLVE_ERR_CUDA, "CUDA error '%s' at %s:%d", cudaGetErrorString(e_), \
                  __FILE__, __LINE__);                                                  \
    }                                                                                   \
  } while (0)

#define LS_BLAS(call)                                                                     \
  do {                                                                                    \
    const int s_ = (int)(call);                                                           \
    if (s_ != 0)                                                                          \
      return fail(LFSOLVE_ERR_CUDA, "library status %d at %s:%d", s_, __FILE__, __LINE__); \
  } while (0)

constexpr long long ALIGN = 32;  // front / factor block alignment (entries)
inline long long align_up(long long x) { return (x + ALIGN - 1) / ALIGN * ALIGN; }
// pivot blocks and leading dimensions of the fronts are padded to this many
// entries, so that F11, F12, F21 and F22 all start on 128-byte boundaries
// (256 for complex128) with row strides of whole 128-byte lines
constexpr int FPAD = 16;
inline int pad_up(int x) { return (x + FPAD - 1) / FPAD * FPAD; }

constexpr int MAX_NRHS_PASS = 2;  // right-hand sides per solve pass
constexpr int SWEEP_BLOCKS = 1184;  // blocks of a sweep phase that fill the GPU (8 a SM)
constexpr int LANES = 8;          // streams (and library handles) for the fronts
// What a group of cnt fronts padded to kp pivots and rp update rows is taken to
// cost, in seconds: per leaf of 64 pivots its launches, and its flops and its
// entries at the rates of mid-sized fronts.  Fronts share a group where that
// is the cheaper (group_fronts).  With whole depths as one group where padding
// grew them by less than a quarter, or from 128 fronts on, and a front a group
// else, and so: 298 and 278 ms (complex64, 524k-row line grating), 60.3 and
// 57.9 ms (complex128, 111k-row hole), 4.2 and 3.3 ms (6k-row slab).
constexpr double GROUP_LEAF_S = 20e-6, GROUP_FLOPS = 6e13, GROUP_ENTRIES = 1.5e11;
constexpr int GROUP_SHAPES = 64;  // shapes of a depth that are told apart, at most
// pivot rows left, squared, times fronts from which the next panel is factored
// beside a step's update (never, from 3e6, 1e6, 3e5 on: 279.6, 266.1, 265.7,
// 266.3 ms in complex64 on a 524k-row line grating; 57.7, 57.3, 56.8, 56.5 ms
// in complex128 on a 111k-row hole)
constexpr double LU_AHEAD_MIN = 1e6;
// complex64 fronts whose Schur update F22 -= L21 U12 has at least this many
// complex multiply-adds use three TF32 tensor-core GEMMs on split operands
constexpr double TF32X3_MIN_MACS = 2e9;
// Pivots one product of the large TF32 terms runs through.  The tensor cores cut
// every partial sum off towards zero, so that the error grows with the depth, and
// every further piece reads and writes the result once more.  Unrefined errors
// (solution, transposed solution, their residuals; 271k-row line grating) over
// those of FP32 substitution with F22's product in split form and one piece, and
// the time of a factorization (524k-row one):
//   512 everywhere       1.19  1.38  0.73  2.50    235 ms
//   256 everywhere       0.91  1.09  0.67  2.67    246 ms
//   128 everywhere       0.63  0.74  0.60  2.00    276 ms
//   256 large, 64 else   0.43  0.68  0.59  1.03    262 ms
//   64 everywhere        0.42  0.68  0.57  0.94    341 ms
//   FP32 products        0.34  0.61  0.59  1.35    413 ms
// Large are the fronts that are split by themselves (TF32X3_MIN_MACS); the others,
// many to a group, lose most where their pivots go in one piece.
constexpr int TF32_PIVOTS = 64, TF32_PIVOTS_LARGE = 256;
// memory the split operands of fronts in flight may take
constexpr size_t SPLIT_BYTES = (size_t)6 << 30;

// ---------------------------------------------------------------------------
// analysis (host)
// ---------------------------------------------------------------------------
struct Node {
  int parent = -1, nchild = 0, child[2] = {-1, -1};
  int depth = 0;
  int p0 = 0, k = 0, m = 0;   // pivots [p0, p0 + k) of the new numbering; k + r rows
  std::vector<int> R;         // update rows: new indices, ascending
  long long arena_off = 0;    // front offset in its depth's arena (entries)
  long long fac_off = 0;      // factor block offset: P (m x k) then U12 (k x r)
  long long r_off = 0;        // offset of its update rows' original indices
  long long rel_off = 0;      // offset of its rows' positions in the parent front
  long long vec_off = 0;      // solve vector block offset (rows)
  int el0 = 0, el1 = 0;       // element range (leaves)
  int ld = 0;                 // leading dimension of its front in the arena
  int roff = 0;               // front row of its first update row (its group's
                              // padded pivot count)
};

// host array of n values left uninitialised (filled by the caller), the
// assembly map's hundreds of MB not zeroed first
template <typename T>
struct HostBuf {
  std::unique_ptr<T[]> p;
  size_t n = 0;
  void resize(size_t m) { p.reset(m ? new T[m] : nullptr); n = m; }
  T *data() { return p.get(); }
  const T *data() const { return p.get(); }
  T &operator[](size_t i) { return p[i]; }
  const T &operator[](size_t i) const { return p[i]; }
  size_t size() const { return n; }
  bool empty() const { return n == 0; }
};

// cnt fronts of a depth taken together on a uniform padded layout: kp pivot
// rows (dummy identity pivots after the real ones), rp update rows (zero rows
// after the real ones), one every `stride` entries of the arena from `off` on
struct FrontGroup { int cnt, kp, rp; long long off, stride; };

// largest rows, pivots and update rows of a depth's fronts
struct SolveShape { int m = 0, k = 0, r = 0; };

struct Plan {
  int n = 0, n_ess = 0, nn = 0;       // rows, essential rows, numbered rows
  long long nnz = 0;
  std::vector<Node> nodes;            // preorder ids
  std::vector<int> post;              // postorder
  std::vector<int> perm, iperm;       // new -> original, original -> new (-1: essential)
  std::vector<int> node_of;           // new index -> node
  std::vector<std::vector<int>> by_depth;
  std::vector<SolveShape> shape;      // per depth
  std::vector<long long> arena_size;  // per depth (entries)
  long long factor_entries = 0, vec_rows = 0;
  std::vector<int> r_orig;            // update rows (original indices), node blocks
  std::vector<int> rel;               // rows of each child in its parent front
  std::vector<std::vector<FrontGroup>> groups;  // per depth
  std::vector<int> ess;
  // assembly map per depth: CSR position -> arena offset
  std::vector<HostBuf<int>> asm_src;        // every entry is written: no zero fill
  std::vector<HostBuf<long long>> asm_dst;
  HostBuf<int> tpos;                  // CSR position of the transposed entry
  double flops = 0.0;
  int max_front = 0, max_k = 0, max_depth = 0;
  long long peak_front_entries = 0;
};

// Nested dissection by element bisection.  Returns the nodes in preorder.
void bisect(int n, int ne, int nd, const int *edof, const double *cen,
            const std::vector<char> &is_ess, int leaf, Plan &P, std::vector<int> &owner,
            std::vector<int> &elems) {
  elems.resize(ne);
  std::iota(elems.begin(), elems.end(), 0);
  owner.assign(n, -1);
  std::vector<int> markL(n, -1), markR(n, -1);
  int stamp = 0;
  struct Item { int a, b, parent, depth, slot; };
  std::vector<Item> stack{{0, ne, -1, 0, 0}};
  std::vector<int> trial, best;
  while (!stack.empty()) {
    const Item it = stack.back();
    stack.pop_back();
    const int id = (int)P.nodes.size();
    P.nodes.emplace_back();
    Node &nd_ = P.nodes.back();
    nd_.parent = it.parent;
    nd_.depth = it.depth;
    nd_.el0 = it.a;
    nd_.el1 = it.b;
    if (it.parent >= 0) {
      Node &par = P.nodes[it.parent];
      par.child[it.slot] = id;
      par.nchild = std::max(par.nchild, it.slot + 1);
    }
    const int cnt = it.b - it.a;
    if (cnt <= leaf) {  // leaf: every unnumbered DOF of its elements
      for (int e = it.a; e < it.b; ++e)
        for (int q = 0; q < nd; ++q) {
          const int d = edof[(size_t)elems[e] * nd + q];
          if (owner[d] < 0 && !is_ess[d]) owner[d] = id;
        }
      continue;
    }
    const int mid = it.a + cnt / 2;
    long long best_sep = -1;
    for (int ax = 0; ax < 3; ++ax) {
      trial.assign(elems.begin() + it.a, elems.begin() + it.b);
      std::nth_element(trial.begin(), trial.begin() + (mid - it.a), trial.end(),
                       [&](int x, int y) {
                         const double cx = cen[(size_t)x * 3 + ax], cy = cen[(size_t)y * 3 + ax];
                         return cx < cy || (cx == cy && x < y);
                       });
      ++stamp;
      for (int t = 0; t < mid - it.a; ++t)
        for (int q = 0; q < nd; ++q) markL[edof[(size_t)trial[t] * nd + q]] = stamp;
      long long sep = 0;
      for (int t = mid - it.a; t < cnt; ++t)
        for (int q = 0; q < nd; ++q) {
          const int d = edof[(size_t)trial[t] * nd + q];
          if (markL[d] == stamp && markR[d] != stamp && owner[d] < 0 && !is_ess[d]) {
            markR[d] = stamp;
            ++sep;
          }
        }
      if (best_sep < 0 || sep < best_sep) {
        best_sep = sep;
        best.swap(trial);
      }
    }
    std::copy(best.begin(), best.end(), elems.begin() + it.a);
    ++stamp;
    for (int e = it.a; e < mid; ++e)
      for (int q = 0; q < nd; ++q) markL[edof[(size_t)elems[e] * nd + q]] = stamp;
    for (int e = mid; e < it.b; ++e)
      for (int q = 0; q < nd; ++q) {
        const int d = edof[(size_t)elems[e] * nd + q];
        if (markL[d] == stamp && owner[d] < 0 && !is_ess[d]) owner[d] = id;
      }
    stack.push_back({mid, it.b, id, it.depth + 1, 1});
    stack.push_back({it.a, mid, id, it.depth + 1, 0});
  }
}

// f(item, worker) for every item of [0, n) on the host threads, items handed
// out one at a time (the fronts' work varies by orders of magnitude)
template <typename F>
void parallel_items(int n, F f) {
  int T = (int)std::min(32u, std::max(1u, std::thread::hardware_concurrency()));
  T = std::max(1, std::min(T, n));
  std::atomic<int> next{0};
  auto run = [&](int w) {
    for (int i = next++; i < n; i = next++) f(i, w);
  };
  if (T == 1) { run(0); return; }
  std::vector<std::thread> th;
  for (int w = 0; w < T; ++w) th.emplace_back(run, w);
  for (auto &t : th) t.join();
}
inline int host_workers(int n) {
  return std::max(1, std::min((int)std::min(32u, std::max(1u, std::thread::hardware_concurrency())), n));
}

// The fronts of one depth in groups that are factored together (FrontGroup):
// fronts of the same padded shape, and then, pair by pair, the groups whose
// union costs less than the two.  all: from so many fronts on one group, else
// a front a group (0: by cost).
std::vector<std::vector<int>> group_fronts(const Plan &P, const std::vector<int> &fronts, int all) {
  std::vector<std::vector<int>> out;
  if (all) {
    if ((int)fronts.size() >= all) return {fronts};
    for (int s : fronts) out.push_back({s});
    return out;
  }
  struct Shape { int k = 0, r = 0; std::vector<int> ids; };
  std::vector<Shape> G;
  for (int grain = FPAD;; grain *= 2) {
    std::map<std::pair<int, int>, Shape> by;
    for (int s : fronts) {
      const int k = P.nodes[s].k, r = P.nodes[s].m - k;
      Shape &Z = by[{(k + grain - 1) / grain, (r + grain - 1) / grain}];
      Z.k = std::max(Z.k, k);
      Z.r = std::max(Z.r, r);
      Z.ids.push_back(s);
    }
    if ((int)by.size() > GROUP_SHAPES) continue;
    for (auto &kv : by) G.push_back(std::move(kv.second));
    break;
  }
  auto cost = [](double k, double r, double cnt) {
    return GROUP_LEAF_S * (1.0 + std::ceil(k / 64)) +
           cnt * (8.0 * (k * k * k / 3.0 + k * k * r + k * r * r) / GROUP_FLOPS +
                  (k + r) * (k + r) / GROUP_ENTRIES);
  };
  auto gain = [&](const Shape &a, const Shape &b) {
    const double na = a.ids.size(), nb = b.ids.size();
    return cost(a.k, a.r, na) + cost(b.k, b.r, nb) -
           cost(std::max(a.k, b.k), std::max(a.r, b.r), na + nb);
  };
  while (G.size() > 1) {
    double best = 0.0;
    size_t bi = 0, bj = 0;
    for (size_t i = 0; i < G.size(); ++i)
      for (size_t j = i + 1; j < G.size(); ++j) {
        const double g = gain(G[i], G[j]);
        if (g > best) { best = g; bi = i; bj = j; }
      }
    if (best <= 0.0) break;
    G[bi].k = std::max(G[bi].k, G[bj].k);
    G[bi].r = std::max(G[bi].r, G[bj].r);
    G[bi].ids.insert(G[bi].ids.end(), G[bj].ids.begin(), G[bj].ids.end());
    G.erase(G.begin() + bj);
  }
  for (Shape &Z : G) out.push_back(std::move(Z.ids));
  return out;
}


int build_plan(int n, const int *I, const int *J, long long nnz, int ne, int nd,
               const int *edof, const double *cen, const int *ess, int n_ess, int leaf,
               Plan &P) {
  P = Plan();
  P.n = n;
  P.nnz = nnz;
  std::vector<char> is_ess(n, 0);
  for (int i = 0; i < n_ess; ++i) {
    if (ess[i] < 0 || ess[i] >= n) return fail(LFSOLVE_ERR_ARG, "essential row %d out of range", ess[i]);
    is_ess[ess[i]] = 1;
  }
  for (int i = 0; i < n; ++i)
    if (is_ess[i]) P.ess.push_back(i);
  P.n_ess = (int)P.ess.size();
  for (long long t = 0; t < (long long)ne * nd; ++t)
    if (edof[t] < 0 || edof[t] >= n) return fail(LFSOLVE_ERR_ARG, "element DOF %d out of range", edof[t]);
  // LFSOLVE_PROFILE set: host seconds of the analysis phases printed
  const bool prof = std::getenv("LFSOLVE_PROFILE") != nullptr;
  auto tick = std::chrono::steady_clock::now();
  auto phase = [&](const char *what) {
    if (!prof) return;
    const auto now = std::chrono::steady_clock::now();
    std::printf("lfsolve analysis: %-28s %8.3f s\n", what,
                std::chrono::duration<double>(now - tick).count());
    std::fflush(stdout);
    tick = now;
  };
  std::vector<int> owner, elems;
  bisect(n, ne, nd, edof, cen, is_ess, leaf, P, owner, elems);
  phase("nested dissection");
  for (int i = 0; i < n; ++i)
    if (!is_ess[i] && owner[i] < 0)
      return fail(LFSOLVE_ERR_ARG, "row %d is touched by no element", i);
  const int ns = (int)P.nodes.size();
  // postorder (children before parents)
  P.post.reserve(ns);
  {
    std::vector<std::pair<int, int>> st{{0, 0}};
    while (!st.empty()) {
      auto &[u, i] = st.back();
      if (i < P.nodes[u].nchild) {
        const int c = P.nodes[u].child[i++];
        st.push_back({c, 0});
      } else {
        P.post.push_back(u);
        st.pop_back();
      }
    }
  }
  // pivots of each node (ascending original index) and the new numbering
  std::vector<std::vector<int>> piv(ns);
  for (int i = 0; i < n; ++i)
    if (owner[i] >= 0) piv[owner[i]].push_back(i);
  P.perm.clear();
  P.iperm.assign(n, -1);
  P.node_of.clear();
  for (int s : P.post) {
    Node &N = P.nodes[s];
    N.p0 = (int)P.perm.size();
    N.k = (int)piv[s].size();
    for (int i : piv[s]) {
      P.iperm[i] = (int)P.perm.size();
      P.perm.push_back(i);
      P.node_of.push_back(s);
    }
  }
  P.nn = (int)P.perm.size();
  // update rows, bottom-up
  for (int s : P.post) {
    Node &N = P.nodes[s];
    std::vector<int> R;
    if (N.nchild == 0) {
      for (int e = N.el0; e < N.el1; ++e)
        for (int q = 0; q < nd; ++q) {
          const int d = edof[(size_t)elems[e] * nd + q];
          const int v = P.iperm[d];
          if (v >= N.p0 + N.k) R.push_back(v);
        }
    } else {
      for (int c = 0; c < N.nchild; ++c)
        for (int v : P.nodes[N.child[c]].R)
          if (v >= N.p0 + N.k) R.push_back(v);
    }
    std::sort(R.begin(), R.end());
    R.erase(std::unique(R.begin(), R.end()), R.end());
    N.R.swap(R);
    N.m = N.k + (int)N.R.size();
    P.max_front = std::max(P.max_front, N.m);
    P.max_k = std::max(P.max_k, N.k);
    P.max_depth = std::max(P.max_depth, N.depth);
    const double k = N.k, r = (double)N.R.size();
    P.flops += 8.0 * (k * k * k / 3.0 + k * k * r + k * r * r);
  }
  phase("numbering, update rows");
  // layouts
  P.by_depth.assign(P.max_depth + 1, {});
  for (int s : P.post) P.by_depth[P.nodes[s].depth].push_back(s);
  P.arena_size.assign(P.max_depth + 1, 0);
  P.groups.assign(P.max_depth + 1, {});
  // LFSOLVE_BATCH_MIN: depths of so many fronts as one group, others a front a group
  const char *batch_env = std::getenv("LFSOLVE_BATCH_MIN");
  for (int d = 0; d <= P.max_depth; ++d) {
    const int all = batch_env ? std::max(1, std::atoi(batch_env)) : 0;
    for (const std::vector<int> &ids : group_fronts(P, P.by_depth[d], all)) {
      FrontGroup G{(int)ids.size(), 0, 0, P.arena_size[d], 0};
      int r = 0;
      for (int s : ids) {
        G.kp = std::max(G.kp, pad_up(P.nodes[s].k));
        r = std::max(r, P.nodes[s].m - P.nodes[s].k);
      }
      G.rp = pad_up(r);
      const long long ld = G.kp + G.rp;
      G.stride = align_up(ld * ld);
      for (int s : ids) {
        Node &N = P.nodes[s];
        N.arena_off = P.arena_size[d];
        N.ld = (int)ld;
        N.roff = G.kp;
        P.arena_size[d] += G.stride;
      }
      P.groups[d].push_back(G);
    }
  }
  long long fac = 0, roff = 0, vec = 0;
  P.shape.assign(P.max_depth + 1, {});
  for (int d = 0; d <= P.max_depth; ++d)
    for (int s : P.by_depth[d]) {
      Node &N = P.nodes[s];
      SolveShape &Z = P.shape[d];
      Z.m = std::max(Z.m, N.m);
      Z.k = std::max(Z.k, N.k);
      Z.r = std::max(Z.r, N.m - N.k);
      N.fac_off = fac;
      const long long r = (long long)N.R.size();
      fac += align_up((long long)N.m * N.k + (long long)N.k * r);
      N.r_off = roff;
      roff += r;
      N.vec_off = vec;
      vec += N.m;
    }
  P.factor_entries = fac;
  P.vec_rows = vec;
  if (vec >= (1LL << 31)) return fail(LFSOLVE_ERR_ARG, "the fronts' rows exceed 2^31");
  // the workspace a factorization holds: the largest even and the largest odd depth
  long long half[2] = {0, 0};
  for (int d = 0; d <= P.max_depth; ++d) half[d & 1] = std::max(half[d & 1], P.arena_size[d]);
  P.peak_front_entries = half[0] + half[1];
  P.r_orig.resize(roff);
  for (int s = 0; s < ns; ++s) {
    const Node &N = P.nodes[s];
    for (size_t t = 0; t < N.R.size(); ++t) P.r_orig[N.r_off + t] = P.perm[N.R[t]];
  }
  // each child's update rows located in its parent's front
  std::vector<int> loc(P.nn, -1);
  P.rel.assign(roff, 0);
  for (int s = 0; s < ns; ++s) {
    const Node &N = P.nodes[s];
    if (N.nchild == 0) continue;
    for (int t = 0; t < N.k; ++t) loc[N.p0 + t] = t;
    for (size_t t = 0; t < N.R.size(); ++t) loc[N.R[t]] = N.k + (int)t;
    for (int c = 0; c < N.nchild; ++c) {
      Node &C = P.nodes[N.child[c]];
      C.rel_off = C.r_off;
      for (size_t t = 0; t < C.R.size(); ++t) {
        const int l = loc[C.R[t]];
        if (l < 0) return fail(LFSOLVE_ERR_ARG, "internal: child row missing from its parent front");
        P.rel[C.r_off + t] = l;
      }
    }
    for (int t = 0; t < N.k; ++t) loc[N.p0 + t] = -1;
    for (int v : N.R) loc[v] = -1;
  }
  phase("layouts, child row maps");
  // transposed positions: entry (i, j) -> the position of (j, i), by binary
  // search in row j (columns sorted); the structure must be symmetric
  P.tpos.resize(nnz);  // every entry written below (or the call fails)
  {
    std::atomic<long long> bad{-1};
    constexpr int ROWS = 4096;  // rows an item
    parallel_items((n + ROWS - 1) / ROWS, [&](int it, int) {
      for (int i = it * ROWS; i < std::min(n, (it + 1) * ROWS); ++i)
        for (long long p = I[i]; p < I[i + 1]; ++p) {
          const int j = J[p];
          const int *b = J + I[j], *e = J + I[j + 1];
          const int *f = std::lower_bound(b, e, i);
          if (f == e || *f != i) {
            long long expect = -1;
            bad.compare_exchange_strong(expect, (long long)i << 32 | (unsigned)j);
            return;
          }
          P.tpos[p] = (int)(f - J);
        }
    });
    if (bad >= 0)
      return fail(LFSOLVE_ERR_ARG, "the CSR structure is not symmetric (row %d, column %d)",
                  (int)(bad >> 32), (int)(bad & 0xffffffff));
  }
  phase("transposed positions");
  // assembly map: every entry (i, j) with i eliminated at front s and j not
  // eliminated before it goes to its front position (and the transposed
  // entry, when j is an update row); per depth, fronts in index order, each
  // front's entries in row order.  A counting pass sizes every front's
  // slice, then the fronts fill their slices on the host threads.
  P.asm_src.clear();
  P.asm_src.resize(P.max_depth + 1);
  P.asm_dst.clear();
  P.asm_dst.resize(P.max_depth + 1);
  {
    const int W = host_workers(ns);
    std::vector<std::vector<int>> wloc(W, std::vector<int>(P.nn, -1));
    std::vector<long long> cnt(ns, 0), off(ns, 0);
    parallel_items(ns, [&](int s, int) {
      const Node &N = P.nodes[s];
      long long c = 0;
      for (int t = 0; t < N.k; ++t) {
        const int i = P.perm[N.p0 + t];
        for (long long p = I[i]; p < I[i + 1]; ++p) {
          const int vj = P.iperm[J[p]];
          if (vj < N.p0) continue;  // essential, or eliminated further down
          c += vj >= N.p0 + N.k ? 2 : 1;
        }
      }
      cnt[s] = c;
    });
    std::vector<long long> total(P.max_depth + 1, 0);
    for (int s = 0; s < ns; ++s) {
      off[s] = total[P.nodes[s].depth];
      total[P.nodes[s].depth] += cnt[s];
    }
    for (int d = 0; d <= P.max_depth; ++d) {
      P.asm_src[d].resize(total[d]);
      P.asm_dst[d].resize(total[d]);
    }
    std::atomic<int> outside{0};
    parallel_items(ns, [&](int s, int w) {
      const Node &N = P.nodes[s];
      std::vector<int> &lc = wloc[w];
      for (int t = 0; t < N.k; ++t) lc[N.p0 + t] = t;
      for (size_t t = 0; t < N.R.size(); ++t) lc[N.R[t]] = N.roff + (int)t;
      int *src = P.asm_src[N.depth].data() + off[s];
      long long *dst = P.asm_dst[N.depth].data() + off[s];
      long long q = 0;
      for (int t = 0; t < N.k; ++t) {
        const int i = P.perm[N.p0 + t];
        const long long li = t;
        for (long long p = I[i]; p < I[i + 1]; ++p) {
          const int vj = P.iperm[J[p]];
          if (vj < N.p0) continue;
          const long long lj = lc[vj];
          if (lj < 0) { outside = 1; continue; }
          src[q] = (int)p;
          dst[q++] = N.arena_off + li + lj * N.ld;
          if (vj >= N.p0 + N.k) {
            src[q] = P.tpos[p];
            dst[q++] = N.arena_off + lj + li * N.ld;
          }
        }
      }
      for (int t = 0; t < N.k; ++t) lc[N.p0 + t] = -1;
      for (int v : N.R) lc[v] = -1;
    });
    if (outside) return fail(LFSOLVE_ERR_ARG, "internal: coupling outside the front");
  }
  phase("assembly map");
  return LFSOLVE_OK;
}

// ---------------------------------------------------------------------------
// device helpers
// ---------------------------------------------------------------------------
template <typename T> struct CT;
template <> struct CT<cuComplex> {
  using R = float;
  __host__ __device__ static cuComplex mk(double a, double b) { return make_cuComplex((float)a, (float)b); }
};
template <> struct CT<cuDoubleComplex> {
  using R = double;
  __host__ __device__ static cuDoubleComplex mk(double a, double b) { return make_cuDoubleComplex(a, b); }
};
__device__ __forceinline__ cuComplex cmul(cuComplex a, cuComplex b) { return cuCmulf(a, b); }
__device__ __forceinline__ cuDoubleComplex cmul(cuDoubleComplex a, cuDoubleComplex b) { return cuCmul(a, b); }
__device__ __forceinline__ cuComplex csub(cuComplex a, cuComplex b) { return cuCsubf(a, b); }
__device__ __forceinline__ cuDoubleComplex csub(cuDoubleComplex a, cuDoubleComplex b) { return cuCsub(a, b); }
__device__ __forceinline__ cuComplex cadd(cuComplex a, cuComplex b) { return cuCaddf(a, b); }
__device__ __forceinline__ cuDoubleComplex cadd(cuDoubleComplex a, cuDoubleComplex b) { return cuCadd(a, b); }
template <typename T> __device__ __forceinline__ T czero() { return CT<T>::mk(0.0, 0.0); }
// a - b c
template <typename T> __device__ __forceinline__ T cfms(T a, T b, T c) {
  a.x = fma(-b.x, c.x, a.x); a.x = fma(b.y, c.y, a.x);
  a.y = fma(-b.x, c.y, a.y); a.y = fma(-b.y, c.x, a.y);
  return a;
}

struct StripItem { int node, col0; };
struct NodeDev {  // per-node data the kernels read
  long long arena_off, fac_off, r_off, vec_off;
  int parent, k, m, p0, depth, ld, roff;
};

// original entries into the fronts of one depth (each position once)
template <typename T>
__global__ void k_assemble(long long cnt, const int *__restrict__ src,
                           const long long *__restrict__ dst, const double2 *__restrict__ vals,
                           T *__restrict__ arena) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < cnt;
       t += (long long)gridDim.x * blockDim.x) {
    const double2 v = __ldg(vals + src[t]);
    T *d = arena + dst[t];
    *d = cadd(*d, CT<T>::mk(v.x, v.y));
  }
}

// Every entry of a depth's fronts, from the children's update blocks: item =
// (front, first of a strip of 32 columns of its padded layout).  The entry of
// rows a and b is the sum over the children that have both (src: the child's
// vector row of a front's row, -1: none), the diagonal of a dummy pivot is one,
// all else zero.  A thread keeps its row's places in the children over the
// strip.  Bound: HBM; each entry is written once and each child entry read
// once.  (Zeroed, then added to by a launch a child: 22.6 ms of a factorization
// of a 524k-row line grating in complex64, 11.7 ms so.)
constexpr int BUILD_T = 256, BUILD_C = 32;
template <typename T>
__global__ void __launch_bounds__(BUILD_T)
k_build_fronts(const StripItem *__restrict__ items, const NodeDev *__restrict__ nodes,
               const int *__restrict__ child, const int2 *__restrict__ src,
               const T *__restrict__ child_arena, T *__restrict__ arena) {
  __shared__ int col[2][BUILD_C];   // the strip's columns in the children, -1: none
  const StripItem it = items[blockIdx.x];
  const NodeDev N = nodes[it.node];
  const int c[2] = {child[2 * it.node], child[2 * it.node + 1]};
  const T *U[2] = {nullptr, nullptr};   // the children's F22
  int ld[2] = {0, 0}, base[2] = {0, 0};
#pragma unroll
  for (int q = 0; q < 2; ++q)
    if (c[q] >= 0) {
      const NodeDev C = nodes[c[q]];
      U[q] = child_arena + C.arena_off + C.roff + (long long)C.roff * C.ld;
      ld[q] = C.ld;
      base[q] = (int)C.vec_off + C.k;
    }
  // a row of the padded layout in the children (update rows of each)
  auto places = [&](int i, int (&p)[2]) {
    const int v = i < N.k ? i : i >= N.roff && i - N.roff < N.m - N.k ? N.k + i - N.roff : -1;
    const int2 s = v < 0 ? make_int2(-1, -1) : src[N.vec_off + v];
    p[0] = s.x < 0 ? -1 : s.x - base[0];
    p[1] = s.y < 0 ? -1 : s.y - base[1];
  };
  const int nc = min(BUILD_C, N.ld - it.col0);
  if (threadIdx.x < nc) {
    int p[2];
    places(it.col0 + threadIdx.x, p);
    col[0][threadIdx.x] = p[0];
    col[1][threadIdx.x] = p[1];
  }
  __syncthreads();
  T *F = arena + N.arena_off + (long long)it.col0 * N.ld;
  for (int i = threadIdx.x; i < N.ld; i += BUILD_T) {
    int p[2];
    places(i, p);
    const int one = i >= N.k && i < N.roff ? i - it.col0 : -1;
#pragma unroll 4
    for (int j = 0; j < nc; ++j) {
      const int a = col[0][j], b = col[1][j];
      T v = CT<T>::mk(j == one ? 1.0 : 0.0, 0.0);
      if (p[0] >= 0 && a >= 0) v = U[0][p[0] + (long long)a * ld[0]];
      if (p[1] >= 0 && b >= 0) v = cadd(v, U[1][p[1] + (long long)b * ld[1]]);
      F[i + (long long)j * N.ld] = v;
    }
  }
}

// copy the L and U blocks of the factored fronts to the factor store:
// P = F[:, 0:k] (m x k) then U12 = F[0:k, k:m] (k x r); item = (node, col0).  A
// warp a column, eight loads in flight: a block a column left most threads of
// small fronts idle (149 us over a 6k-row slab's fronts, 92 us so).  Bound: HBM.
template <typename T>
__global__ void k_copy_out(const StripItem *__restrict__ items, const NodeDev *__restrict__ nodes,
                           const T *__restrict__ arena, T *__restrict__ fac) {
  const StripItem it = items[blockIdx.x];
  const NodeDev N = nodes[it.node];
  const int lane = threadIdx.x & 31, gap = N.roff - N.k;   // dummy pivots
  const T *F = arena + N.arena_off;
  T *Pf = fac + N.fac_off;
  T *U12 = Pf + (long long)N.m * N.k;
  const int c1 = min(it.col0 + 32, N.m);
  for (int c = it.col0 + (threadIdx.x >> 5); c < c1; c += (int)blockDim.x >> 5) {
    // compact column c: a pivot column (< k) or update column c - k, which
    // sits at front column roff + c - k
    const bool piv = c < N.k;
    const T *__restrict__ Fc = F + (long long)(piv ? c : c + gap) * N.ld;
    T *__restrict__ dst = piv ? Pf + (long long)c * N.m : U12 + (long long)(c - N.k) * N.k;
    const int n = piv ? N.m : N.k;
#pragma unroll 8
    for (int a = lane; a < n; a += 32) dst[a] = Fc[a < N.k ? a : a + gap];
  }
}

// the row interchanges of a front's pivot block (ipiv, 1-based, applied in
// order) on ncol columns of ld-strided storage: a thread per column
template <typename T>
__global__ void k_swap_cols(int k, int ncol, const int *__restrict__ ipiv, T *__restrict__ A,
                            int ld) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncol) return;
  T *col = A + (long long)c * ld;
  for (int i = 0; i < k; ++i) {
    const int p = ipiv[i] - 1;
    if (p != i) {
      const T t = col[i];
      col[i] = col[p];
      col[p] = t;
    }
  }
}

// y = A x (or A^T x through the transposed positions) in FP64, a warp per
// row; one column
__global__ void k_spmv(int n, const int *__restrict__ I, const int *__restrict__ J,
                       const double2 *__restrict__ vals, const int *__restrict__ tpos,
                       const double2 *__restrict__ x, double2 *__restrict__ y) {
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n) return;
  double ar = 0.0, ai = 0.0;
  for (int p = I[row] + lane; p < I[row + 1]; p += 32) {
    const double2 a = vals[tpos ? tpos[p] : p];
    const double2 xv = x[J[p]];
    ar = fma(a.x, xv.x, ar); ar = fma(-a.y, xv.y, ar);
    ai = fma(a.x, xv.y, ai); ai = fma(a.y, xv.x, ai);
  }
  for (int o = 16; o; o >>= 1) {
    ar += __shfl_xor_sync(0xffffffffu, ar, o);
    ai += __shfl_xor_sync(0xffffffffu, ai, o);
  }
  if (lane == 0) y[row] = make_double2(ar, ai);
}

// ---------------------------------------------------------------------------
// solve kernels
// ---------------------------------------------------------------------------
#include "lfsolve_lu.cuh"
#include "lfsolve_sweeps.cuh"
#include "lfsolve_trsm.cuh"

// Pivot order of a front from the library's sequential row swaps (ipiv,
// 1-based, applied to the identity), so that the swapped vector is v[perm[i]]
// at row i; the swaps in shared memory up to PERM_CAP pivots (global beyond)
constexpr int PERM_CAP = 12288;
__device__ void perm_from_ipiv(int k, const int *__restrict__ pv, int *__restrict__ dst,
                               int *__restrict__ sp) {
  int *w = k <= PERM_CAP ? sp : dst;
  for (int i = threadIdx.x; i < k; i += blockDim.x) w[i] = i;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int q = 0; q < k; ++q) {
      const int p = pv[q] - 1;
      if (p != q && p >= 0 && p < k) {
        const int t = w[q];
        w[q] = w[p];
        w[p] = t;
      }
    }
  __syncthreads();
  if (k <= PERM_CAP)
    for (int i = threadIdx.x; i < k; i += blockDim.x) dst[i] = sp[i];
}
// one front's permutation (k pivots at pv) into perm
__global__ void k_ipiv_to_perm_one(int k, const int *__restrict__ pv, int *__restrict__ perm) {
  __shared__ int sp[PERM_CAP];
  perm_from_ipiv(k, pv, perm, sp);
}
// pivots that k_perm_f12 can stage
template <typename T>
constexpr int perm_smem_max() { return (int)(160 * 1024 / sizeof(T)); }

// x[ess] = b[ess]
template <typename T>
__global__ void k_ess_copy(int ne, const int *__restrict__ ess, const T *__restrict__ b, int ldb,
                           T *__restrict__ x, int ldx, int nrhs) {
  for (int c = 0; c < nrhs; ++c)
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < ne; a += gridDim.x * blockDim.x)
      x[(long long)c * ldx + ess[a]] = b[(long long)c * ldb + ess[a]];
}

// conversions: out = (T)(in * scale[c]);  acc += scale[c] * (double)d
template <typename T>
__global__ void k_to_prec(long long n, int ncol, const double2 *__restrict__ in,
                          const double *__restrict__ scale, T *__restrict__ out) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n * ncol;
       t += (long long)gridDim.x * blockDim.x) {
    const double s = scale ? scale[t / n] : 1.0;
    out[t] = CT<T>::mk(in[t].x * s, in[t].y * s);
  }
}
template <typename T>
__global__ void k_from_prec(long long n, int ncol, const T *__restrict__ d,
                            const double *__restrict__ scale, double2 *__restrict__ acc,
                            int accumulate) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n * ncol;
       t += (long long)gridDim.x * blockDim.x) {
    const double s = scale ? scale[t / n] : 1.0;
    const double2 v = make_double2((double)d[t].x * s, (double)d[t].y * s);
    acc[t] = accumulate ? make_double2(acc[t].x + v.x, acc[t].y + v.y) : v;
  }
}

// FP64 residual r = b - A x (or A^T x through the transposed positions), a
// warp per row, and per column partial sums of |r|^2, |b|^2, max |r|
__global__ void k_resid(int n, int ncol, const int *__restrict__ I, const int *__restrict__ J,
                        const double2 *__restrict__ vals, const int *__restrict__ tpos,
                        const double2 *__restrict__ x, const double2 *__restrict__ b,
                        double2 *__restrict__ r, double *__restrict__ part) {
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int c = blockIdx.y;
  double rn = 0.0, bn = 0.0, rmax = 0.0;
  if (row < n) {
    const double2 *xc = x + (long long)c * n;
    double ar = 0.0, ai = 0.0;
    for (int p = I[row] + lane; p < I[row + 1]; p += 32) {
      const double2 a = vals[tpos ? tpos[p] : p];
      const double2 xv = xc[J[p]];
      ar = fma(a.x, xv.x, ar); ar = fma(-a.y, xv.y, ar);
      ai = fma(a.x, xv.y, ai); ai = fma(a.y, xv.x, ai);
    }
    for (int o = 16; o; o >>= 1) {
      ar += __shfl_xor_sync(0xffffffffu, ar, o);
      ai += __shfl_xor_sync(0xffffffffu, ai, o);
    }
    if (lane == 0) {
      const double2 bv = b[(long long)c * n + row];
      const double dr = bv.x - ar, di = bv.y - ai;
      r[(long long)c * n + row] = make_double2(dr, di);
      rn = dr * dr + di * di;
      bn = bv.x * bv.x + bv.y * bv.y;
      rmax = fmax(fabs(dr), fabs(di));
    }
  }
  __shared__ double red[3][32];
  const int w = threadIdx.x >> 5;
  if (lane == 0) { red[0][w] = rn; red[1][w] = bn; red[2][w] = rmax; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a0 = 0.0, a1 = 0.0, a2 = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) {
      a0 += red[0][q]; a1 += red[1][q]; a2 = fmax(a2, red[2][q]);
    }
    double *pp = part + 3 * ((long long)c * gridDim.x + blockIdx.x);
    pp[0] = a0; pp[1] = a1; pp[2] = a2;
  }
}
__global__ void k_resid_sum(int nblk, int ncol, const double *__restrict__ part,
                            double *__restrict__ out) {
  const int c = blockIdx.x;
  double a0 = 0.0, a1 = 0.0, a2 = 0.0;
  for (int i = threadIdx.x; i < nblk; i += blockDim.x) {
    const double *pp = part + 3 * ((long long)c * nblk + i);
    a0 += pp[0]; a1 += pp[1]; a2 = fmax(a2, pp[2]);
  }
  __shared__ double red[3][32];
  for (int o = 16; o; o >>= 1) {
    a0 += __shfl_xor_sync(0xffffffffu, a0, o);
    a1 += __shfl_xor_sync(0xffffffffu, a1, o);
    a2 = fmax(a2, __shfl_xor_sync(0xffffffffu, a2, o));
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) { red[0][w] = a0; red[1][w] = a1; red[2][w] = a2; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) {
      s0 += red[0][q]; s1 += red[1][q]; s2 = fmax(s2, red[2][q]);
    }
    out[3 * c] = s0; out[3 * c + 1] = s1; out[3 * c + 2] = s2;
  }
}

// ---------------------------------------------------------------------------
// library dispatch by precision
// ---------------------------------------------------------------------------
inline cusolverStatus_t getrf_buf(cusolverDnHandle_t h, int m, int n, cuComplex *A, int lda, int *lw) {
  return cusolverDnCgetrf_bufferSize(h, m, n, A, lda, lw);
}
inline cusolverStatus_t getrf_buf(cusolverDnHandle_t h, int m, int n, cuDoubleComplex *A, int lda, int *lw) {
  return cusolverDnZgetrf_bufferSize(h, m, n, A, lda, lw);
}
inline cusolverStatus_t getrf(cusolverDnHandle_t h, int m, int n, cuComplex *A, int lda, cuComplex *w, int *ip, int *info) {
  return cusolverDnCgetrf(h, m, n, A, lda, w, ip, info);
}
inline cusolverStatus_t getrf(cusolverDnHandle_t h, int m, int n, cuDoubleComplex *A, int lda, cuDoubleComplex *w, int *ip, int *info) {
  return cusolverDnZgetrf(h, m, n, A, lda, w, ip, info);
}
inline cublasStatus_t gemm_sb(cublasHandle_t h, int m, int n, int k, const cuComplex *al,
                              const cuComplex *A, int lda, long long sa, const cuComplex *B, int ldb,
                              long long sb, const cuComplex *be, cuComplex *C, int ldc, long long sc,
                              int b) {
  return cublasCgemmStridedBatched(h, CUBLAS_OP_N, CUBLAS_OP_N, m, n, k, al, A, lda, sa, B, ldb,
                                   sb, be, C, ldc, sc, b);
}
inline cublasStatus_t gemm_sb(cublasHandle_t h, int m, int n, int k, const cuDoubleComplex *al,
                              const cuDoubleComplex *A, int lda, long long sa,
                              const cuDoubleComplex *B, int ldb, long long sb,
                              const cuDoubleComplex *be, cuDoubleComplex *C, int ldc, long long sc,
                              int b) {
  return cublasZgemmStridedBatched(h, CUBLAS_OP_N, CUBLAS_OP_N, m, n, k, al, A, lda, sa, B, ldb,
                                   sb, be, C, ldc, sc, b);
}

}  // namespace

// ---------------------------------------------------------------------------
// solver object
// ---------------------------------------------------------------------------
struct lfsolve {
  int dev = 0;
  cudaStream_t stream = nullptr;
  bool analyzed = false, uploaded = false;
  Plan P;
  lfsolve_stats st{};
  // device copies of the plan
  NodeDev *d_nodes = nullptr;
  int *d_child = nullptr, *d_perm = nullptr, *d_rorig = nullptr,
      *d_ess = nullptr, *d_tpos = nullptr;
  std::vector<int *> d_asm_src;
  std::vector<long long *> d_asm_dst;
  std::vector<StripItem *> d_bf, d_co;    // per depth: strips to build, to copy out
  std::vector<int> n_bf, n_co;
  std::vector<int *> d_all;               // per depth: its fronts
  LuSwaps *d_swaps = nullptr;             // interchanges of two steps (n_swaps: max fronts of a depth)
  size_t n_swaps = 0;
  int *d_src = nullptr;                   // children's vector rows per vector row
  DiagItem *d_diag = nullptr;             // 32 x 32 diagonal blocks of the fronts
  std::vector<int> diag_at;               // per depth: its first entry (and the end)
  // factors
  int prec = -1;
  void *d_fac = nullptr;
  int *d_info = nullptr;
  int *d_pperm = nullptr;  // per-front pivot permutations
  int lu_cluster[2] = {0, 0};  // largest panel cluster the device takes, per precision
  // lanes
  cudaStream_t lane[LANES] = {};
  cublasHandle_t blas[LANES] = {};
  cusolverDnHandle_t sol[LANES] = {};
  void *work[LANES] = {};
  size_t work_bytes[LANES] = {};
  cudaEvent_t ev_main = nullptr, ev_lane[LANES] = {};
  // panels factored beside the update before them (lu_depth)
  cudaStream_t ahead = nullptr;
  cudaEvent_t ev_rest = nullptr;
  // front workspace, kept between factorizations: the fronts of the even and
  // of the odd depths (a depth reads its children's from the other one), and
  // the split operands of the fronts in flight
  void *d_arena[2] = {nullptr, nullptr}, *d_split = nullptr;
  size_t arena_bytes[2] = {0, 0}, split_bytes = 0;
  int *lpiv[LANES] = {};  // pivots of a front's padded pivot block
  int lpiv_n[LANES] = {};
  cublasHandle_t blas_main = nullptr;
  // solve scratch
  void *d_V = nullptr, *d_Y = nullptr, *d_bw = nullptr, *d_part_y = nullptr;
  size_t V_bytes = 0, Y_bytes = 0, bw_bytes = 0, part_y_bytes = 0;
  double2 *d_r = nullptr, *d_x64 = nullptr;
  size_t r_bytes = 0;
  double *d_part = nullptr, *d_scale = nullptr;
  size_t part_bytes = 0, scale_bytes = 0;
  cudaEvent_t t0 = nullptr, t1 = nullptr;
};

namespace {

template <typename T>
int upload(T **dst, const HostBuf<T> &v, cudaStream_t st) {
  *dst = nullptr;
  if (v.empty()) return LFSOLVE_OK;
  LS_CUDA(cudaMalloc((void **)dst, v.size() * sizeof(T)));
  LS_CUDA(cudaMemcpyAsync(*dst, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st));
  return LFSOLVE_OK;
}
template <typename T>
int upload(T **dst, const std::vector<T> &v, cudaStream_t st) {
  *dst = nullptr;
  if (v.empty()) return LFSOLVE_OK;
  LS_CUDA(cudaMalloc((void **)dst, v.size() * sizeof(T)));
  LS_CUDA(cudaMemcpyAsync(*dst, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st));
  return LFSOLVE_OK;
}

template <typename T> void drop(T *&p) {
  if (p) cudaFree(p);
  p = nullptr;
}

void free_factors(lfsolve *s) {
  drop(s->d_fac);
  s->prec = -1;
}

// the factors, and everything on the device that was sized for a plan
void free_plan(lfsolve *s) {
  free_factors(s);
  s->uploaded = false;
  drop(s->d_nodes);
  for (int **p : {&s->d_child, &s->d_perm, &s->d_rorig, &s->d_ess, &s->d_tpos, &s->d_src, &s->d_info,
                  &s->d_pperm})
    drop(*p);
  drop(s->d_diag);
  drop(s->d_swaps);
  for (auto &p : s->d_asm_src) drop(p);
  for (auto &p : s->d_asm_dst) drop(p);
  for (auto &p : s->d_bf) drop(p);
  for (auto &p : s->d_co) drop(p);
  for (auto &p : s->d_all) drop(p);
}

int ensure_uploaded(lfsolve *s) {
  if (s->uploaded) return LFSOLVE_OK;
  free_plan(s);   // what an upload that failed midway left
  Plan &P = s->P;
  const int ns = (int)P.nodes.size();
  std::vector<NodeDev> nd(ns);
  std::vector<int> child(2 * ns, -1);
  for (int i = 0; i < ns; ++i) {
    const Node &N = P.nodes[i];
    nd[i] = {N.arena_off, N.fac_off, N.r_off, N.vec_off, N.parent, N.k, N.m, N.p0, N.depth,
             N.ld, N.roff};
    child[2 * i] = N.child[0];
    child[2 * i + 1] = N.nchild > 1 ? N.child[1] : -1;
  }
  cudaStream_t st = s->stream;
  int rc;
  if ((rc = upload(&s->d_nodes, nd, st))) return rc;
  if ((rc = upload(&s->d_child, child, st))) return rc;
  if ((rc = upload(&s->d_perm, P.perm, st))) return rc;
  if ((rc = upload(&s->d_rorig, P.r_orig, st))) return rc;
  if ((rc = upload(&s->d_ess, P.ess, st))) return rc;
  if ((rc = upload(&s->d_tpos, P.tpos, st))) return rc;
  // per vector row: the child rows that the forward sweep adds to it
  std::vector<int> src(2 * (size_t)P.vec_rows, -1);
  for (int i = 0; i < ns; ++i) {
    const Node &N = P.nodes[i];
    for (int q = 0; q < N.nchild; ++q) {
      const Node &C = P.nodes[N.child[q]];
      for (int t = 0; t < C.m - C.k; ++t)
        src[2 * (size_t)(N.vec_off + P.rel[C.r_off + t]) + q] = (int)(C.vec_off + C.k + t);
    }
  }
  std::vector<DiagItem> diag;
  s->diag_at.assign(1, 0);
  for (const auto &fronts : P.by_depth) {
    for (int i : fronts)
      for (int j0 = 0; j0 < P.nodes[i].k; j0 += 32) diag.push_back({i, j0});
    s->diag_at.push_back((int)diag.size());
  }
  if ((rc = upload(&s->d_src, src, st))) return rc;
  if ((rc = upload(&s->d_diag, diag, st))) return rc;
  const int D = P.max_depth + 1;
  s->d_asm_src.assign(D, nullptr);
  s->d_asm_dst.assign(D, nullptr);
  s->d_bf.assign(D, nullptr);
  s->n_bf.assign(D, 0);
  s->d_co.assign(D, nullptr);
  s->n_co.assign(D, 0);
  s->d_all.assign(D, nullptr);
  size_t maxb = 1;
  for (int d = 0; d < D; ++d) maxb = std::max(maxb, P.by_depth[d].size());
  s->n_swaps = maxb;
  LS_CUDA(cudaMalloc((void **)&s->d_swaps, sizeof(LuSwaps) * 2 * maxb));
  for (int d = 0; d < D; ++d) {
    if ((rc = upload(&s->d_asm_src[d], P.asm_src[d], st))) return rc;
    if ((rc = upload(&s->d_asm_dst[d], P.asm_dst[d], st))) return rc;
    std::vector<StripItem> bf, co;
    for (int id : P.by_depth[d]) {
      const Node &N = P.nodes[id];
      for (int c0 = 0; c0 < N.ld; c0 += BUILD_C) bf.push_back({id, c0});
      for (int c0 = 0; c0 < N.m; c0 += 32) co.push_back({id, c0});
    }
    if ((rc = upload(&s->d_bf[d], bf, st))) return rc;
    s->n_bf[d] = (int)bf.size();
    if ((rc = upload(&s->d_co[d], co, st))) return rc;
    s->n_co[d] = (int)co.size();
    if ((rc = upload(&s->d_all[d], P.by_depth[d], st))) return rc;
  }
  LS_CUDA(cudaStreamSynchronize(st));
  s->uploaded = true;
  return LFSOLVE_OK;
}

template <typename T>
cudaLaunchConfig_t lu_panel_config(int fronts, int csize, int threads, cudaStream_t st,
                                   cudaLaunchAttribute *attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(fronts * csize));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = (size_t)threads * LU_NB * sizeof(T);
  cfg.stream = st;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = (unsigned)csize;
  attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// the largest power-of-two cluster of full panel blocks that fits the device
template <typename T> int lu_clusters(int *out) {
  LS_CUDA(cudaFuncSetAttribute(k_lu_panel<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  LS_CUDA(cudaFuncSetAttribute(k_lu_panel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)(LU_ROWS<T> * LU_NB * sizeof(T))));
  *out = 1;
  for (int c = 2; c <= LU_MAX_CLUSTER; c *= 2) {
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = lu_panel_config<T>(1, c, LU_ROWS<T>, nullptr, &attr);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_lu_panel<T>, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();  // this size is not on offer
      break;
    }
    *out = c;
  }
  return LFSOLVE_OK;
}

int ensure_lanes(lfsolve *s) {
  if (s->blas_main) return LFSOLVE_OK;
  LS_BLAS(cublasCreate(&s->blas_main));
  LS_BLAS(cublasSetStream(s->blas_main, s->stream));
  // the column permutations stage up to 160 kB of pivot rows
  LS_CUDA(cudaFuncSetAttribute(k_perm_f12<cuComplex>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024));
  LS_CUDA(cudaFuncSetAttribute(k_perm_f12<cuDoubleComplex>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024));
  int rc;
  if ((rc = lu_clusters<cuComplex>(&s->lu_cluster[LFSOLVE_C64]))) return rc;
  if ((rc = lu_clusters<cuDoubleComplex>(&s->lu_cluster[LFSOLVE_C128]))) return rc;
  LS_CUDA(cudaFuncSetAttribute(k_leaf<cuComplex>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)sizeof(LeafSmem<cuComplex>)));
  LS_CUDA(cudaFuncSetAttribute(k_leaf<cuDoubleComplex>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)sizeof(LeafSmem<cuDoubleComplex>)));
  for (auto kern : {k_sweep_tri<1, 0, 0>, k_sweep_tri<1, 0, 1>, k_sweep_tri<1, 1, 0>,
                    k_sweep_tri<1, 1, 1>, k_sweep_tri<2, 0, 0>, k_sweep_tri<2, 0, 1>,
                    k_sweep_tri<2, 1, 0>, k_sweep_tri<2, 1, 1>})
    LS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TRI_SMEM));
  for (int l = 0; l < LANES; ++l) {
    LS_CUDA(cudaStreamCreateWithFlags(&s->lane[l], cudaStreamNonBlocking));
    LS_BLAS(cublasCreate(&s->blas[l]));
    LS_BLAS(cublasSetStream(s->blas[l], s->lane[l]));
    LS_BLAS(cusolverDnCreate(&s->sol[l]));
    LS_BLAS(cusolverDnSetStream(s->sol[l], s->lane[l]));
    LS_CUDA(cudaEventCreateWithFlags(&s->ev_lane[l], cudaEventDisableTiming));
  }
  LS_CUDA(cudaEventCreateWithFlags(&s->ev_main, cudaEventDisableTiming));
  LS_CUDA(cudaEventCreateWithFlags(&s->ev_rest, cudaEventDisableTiming));
  int least = 0, greatest = 0;
  LS_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
  LS_CUDA(cudaStreamCreateWithPriority(&s->ahead, cudaStreamNonBlocking, greatest));
  LS_CUDA(cudaEventCreate(&s->t0));
  LS_CUDA(cudaEventCreate(&s->t1));
  return LFSOLVE_OK;
}

// main stream -> every lane, and back
int fork_lanes(lfsolve *s) {
  LS_CUDA(cudaEventRecord(s->ev_main, s->stream));
  for (int l = 0; l < LANES; ++l) LS_CUDA(cudaStreamWaitEvent(s->lane[l], s->ev_main, 0));
  return LFSOLVE_OK;
}
int join_lanes(lfsolve *s) {
  for (int l = 0; l < LANES; ++l) {
    LS_CUDA(cudaEventRecord(s->ev_lane[l], s->lane[l]));
    LS_CUDA(cudaStreamWaitEvent(s->stream, s->ev_lane[l], 0));
  }
  return LFSOLVE_OK;
}

int chunks(int n) { return n > 0 ? (n + SW_CHUNK - 1) / SW_CHUNK : 0; }

int grid_for(long long n, int threads) {
  return (int)std::max<long long>(1, std::min<long long>((n + threads - 1) / threads, 148LL * 16));
}

// fronts from this many complex multiply-adds of Schur update on
// (LFSOLVE_TF32X3_MIN overrides TF32X3_MIN_MACS)
double tf32x3_min() {
  const char *e = std::getenv("LFSOLVE_TF32X3_MIN");
  return e ? std::atof(e) : TF32X3_MIN_MACS;
}

// the 3xTF32 path: complex64 only, off with LFSOLVE_TF32X3=0
template <typename T> bool use_tf32x3(lfsolve *) { return false; }
template <> bool use_tf32x3<cuComplex>(lfsolve *) {
  const char *e = std::getenv("LFSOLVE_TF32X3");
  return !(e && e[0] == '0');
}

// C -= A B of every front of a group over the k pivots from p0: in the front's
// own precision, or from split operands (rows from i0 of a left operand As,
// columns from j0 of a right operand Bs) as two real TF32 products with FP32
// accumulation
template <typename T>
int group_product(cublasHandle_t h, const Group<T> &G, int m, int n, int p0, int k, const T *A,
                  const T *B, T *C, const Operand &As, int i0, const Operand &Bs, int j0) {
  if (As.p) {
    const float mone = -1.f, one = 1.f;
    // nk pivots from q0; per = 4 or 2 columns a pivot
    auto product = [&](int per, const float *a, const float *b, int q0, int nk) {
      return cublasGemmStridedBatchedEx(
          h, CUBLAS_OP_N, CUBLAS_OP_N, 2 * m, n, per * nk, &mone,
          a + 2 * i0 + (long long)per * q0 * As.ld, CUDA_R_32F, (int)As.ld, per * As.n,
          b + per * (q0 + (long long)j0 * G.kk), CUDA_R_32F, per * G.kk, per * Bs.n, &one, C,
          CUDA_R_32F, 2 * G.ld, 2 * G.S, G.cnt, CUBLAS_COMPUTE_32F_FAST_TF32, CUBLAS_GEMM_DEFAULT);
    };
    LS_BLAS(product(4, As.both(0), Bs.both(0), p0, k));
    const int piece = (double)G.r * G.r * G.kk >= TF32X3_MIN_MACS ? TF32_PIVOTS_LARGE : TF32_PIVOTS;
    for (int q0 = p0; q0 < p0 + k; q0 += piece)
      LS_BLAS(product(2, As.hi(G.cnt, 0), Bs.hi(G.cnt, 0), q0, std::min(piece, p0 + k - q0)));
    return LFSOLVE_OK;
  }
  const T mone = CT<T>::mk(-1.0, 0.0), one = CT<T>::mk(1.0, 0.0);
  LS_BLAS(gemm_sb(h, m, n, k, &mone, A, G.ld, G.S, B, G.ld, G.S, &one, C, G.ld, G.S, G.cnt));
  return LFSOLVE_OK;
}

// floats of split operands a front needs
inline size_t split_floats(int kk, int r) {
  return (size_t)18 * kk * ((size_t)kk + r);
}

// U12, L21 and F22 -= L21 U12 of a group; buf: its products on TF32 tensor
// cores with the split operands there (cnt x split_floats), null: in T
template <typename T>
int group_update(cudaStream_t st, cublasHandle_t h, Group<T> G, float *buf) {
  const int nl = (G.kk + LEAF - 1) / LEAF, ld = G.ld;
  if (buf) {
    float *at = buf;
    auto operand = [&](long long ld, long long n) {
      const Operand o{at, ld, n};
      at += 6 * n * G.cnt;
      return o;
    };
    G.AF = operand(2LL * G.kk, 2LL * G.kk * G.kk);
    G.BF = operand(0, (long long)G.kk * G.kk);
    G.AL = operand(2LL * G.r, 2LL * G.r * G.kk);
    G.BU = operand(0, (long long)G.kk * G.r);
    if (nl > 1) {
      k_split_f11<T><<<dim3((unsigned)(nl - 1), (unsigned)(nl - 1), (unsigned)G.cnt), SPLIT_T, 0, st>>>(G);
      LS_CUDA(cudaGetLastError());
    }
  }
  T *F = G.F;
  int rc;
  for (int i = 1; i <= nl; ++i) {
    k_leaf<T><<<dim3((unsigned)((G.r + LEAF_C<T> - 1) / LEAF_C<T>), (unsigned)G.cnt, 2), LEAF_T,
                sizeof(LeafSmem<T>), st>>>(G, (i - 1) * LEAF);
    LS_CUDA(cudaGetLastError());
    if (i == nl) break;
    const int t = i & -i, p0 = (i - t) * LEAF, pk = t * LEAF, q0 = i * LEAF;
    const int qn = std::min(G.kk, std::min(nl, i + t) * LEAF) - q0;
    if ((rc = group_product<T>(h, G, qn, G.r, p0, pk, F + q0 + (long long)p0 * ld,
                               F + p0 + (long long)G.kk * ld, F + q0 + (long long)G.kk * ld, G.AF, q0,
                               G.BU, 0)) ||
        (rc = group_product<T>(h, G, G.r, qn, p0, pk, F + G.kk + (long long)p0 * ld,
                               F + p0 + (long long)q0 * ld, F + G.kk + (long long)q0 * ld, G.AL, 0,
                               G.BF, q0)))
      return rc;
  }
  return group_product<T>(h, G, G.r, G.r, 0, G.kk, F + G.kk, F + (long long)G.kk * ld,
                          F + G.kk + (long long)G.kk * ld, G.AL, 0, G.BU, 0);
}

// which fronts go through split operands
template <typename T> bool front_split(lfsolve *s, double r, double kk, double cnt) {
  return use_tf32x3<T>(s) && r * r * kk * cnt >= tf32x3_min();
}
// how a depth's groups are taken: on so many lanes, with so many floats of
// split operands each, a group as many fronts at once as those hold
struct DepthPlan { int lanes = 1; size_t floats = 0; };
template <typename T> DepthPlan depth_plan(lfsolve *s, int d) {
  DepthPlan Q;
  size_t largest = 0;
  std::vector<std::pair<size_t, size_t>> split;  // floats a front, fronts
  int busy = 0;
  for (const FrontGroup &G : s->P.groups[d]) {
    if (G.kp == 0 || G.rp == 0) continue;
    ++busy;
    if (!front_split<T>(s, G.rp, G.kp, G.cnt)) continue;
    split.push_back({split_floats(G.kp, G.rp), (size_t)G.cnt});
    largest = std::max(largest, split.back().first);
  }
  Q.lanes = std::max(1, std::min(busy, LANES));
  if (!largest) return Q;
  Q.lanes = (int)std::max<size_t>(1, std::min<size_t>(Q.lanes, SPLIT_BYTES / (4 * largest)));
  const size_t cap = std::max(largest, SPLIT_BYTES / 4 / Q.lanes);
  for (auto &g : split) Q.floats = std::max(Q.floats, g.first * std::min(g.second, cap / g.first));
  return Q;
}

int ensure_bytes(void **p, size_t *have, size_t need) {
  if (*have >= need) return LFSOLVE_OK;
  if (*p) LS_CUDA(cudaFree(*p));
  *p = nullptr;
  *have = 0;
  LS_CUDA(cudaMalloc(p, need));
  *have = need;
  return LFSOLVE_OK;
}

// P F11 = L11 U11 of every front of depth d with at most cap pivots, the pivot
// order applied to F12 too
template <typename T>
int lu_depth(lfsolve *s, int d, T *arena, int cap) {
  Plan &P = s->P;
  cudaStream_t st = s->stream;
  const int cnt = (int)P.by_depth[d].size();
  int kmax = 0, rmax = 0;
  for (int id : P.by_depth[d]) {
    const Node &N = P.nodes[id];
    if (N.k > cap) continue;
    kmax = std::max(kmax, N.k);
    rmax = std::max(rmax, N.m - N.k);
  }
  const int *list = s->d_all[d];
  auto strips = [&](cudaStream_t on, int which, int j0) -> int {
    const int rows = kmax - j0;
    const int n = (which == LU_NEXT ? LU_NB : kmax + LU_STRIP<T> - 1) / LU_STRIP<T>;
    // rows of the update split where the strips alone leave SMs idle
    const int groups = (rows - LU_NB + LU_STRIP_T - 1) / LU_STRIP_T;
    const bool split = groups > 1 && (which == LU_NEXT ||
                                      (long long)cnt * ((rows - 1) / LU_STRIP<T>) < 2 * 148);
    for (int f0 = 0; f0 < cnt; f0 += 65535) {
      const dim3 g((unsigned)n, (unsigned)std::min(65535, cnt - f0));
      const int *li = list + f0;
      const LuSwaps *sw = s->d_swaps + (j0 / LU_NB & 1) * s->n_swaps + f0;
      if (!split) {
        k_lu_strip<T, 0><<<g, LU_STRIP_T, 0, on>>>(li, s->d_nodes, arena, j0, cap, sw, which);
      } else {
        k_lu_strip<T, 1><<<g, LU_STRIP_T, 0, on>>>(li, s->d_nodes, arena, j0, cap, sw, which);
        k_lu_strip<T, 2><<<dim3(g.x, g.y, (unsigned)groups), LU_STRIP_T, 0, on>>>(
            li, s->d_nodes, arena, j0, cap, sw, which);
      }
      LS_CUDA(cudaGetLastError());
    }
    return LFSOLVE_OK;
  };
  // While a step's update is large, the next panel is factored beside it: its
  // columns are updated first, on a stream of their own, and the panel (few
  // blocks, a chain of exchanges) goes before the rest's blocks by priority.
  // The step then takes the longer of the two instead of their sum.
  bool ahead = false;
  int rc;
  for (int j0 = 0; j0 < kmax; j0 += LU_NB) {
    const int rows = kmax - j0;
    const bool was = ahead;
    ahead = (double)cnt * rows * rows >= LU_AHEAD_MIN;  // rows shrink: on at first, then off
    if (ahead != was) {  // the panel's stream waits for what came before, or the other way round
      LS_CUDA(cudaEventRecord(s->ev_main, was ? s->ahead : st));
      LS_CUDA(cudaStreamWaitEvent(was ? st : s->ahead, s->ev_main, 0));
    }
    int csize = 1;
    // the fewest blocks that hold the rows: smaller blocks in larger clusters
    // cost more in cluster barriers than they save in issue slots (4,200 pivots
    // in complex64: 17.7 ms with 640 rows a block, 18.4 with 320, 19.3 with 160)
    while (csize * LU_ROWS<T> < rows) csize *= 2;
    const int threads = ((rows + csize - 1) / csize + 31) / 32 * 32;
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg =
        lu_panel_config<T>(cnt, csize, threads, ahead ? s->ahead : st, &attr);
    // two sets of interchanges: a step's strips read theirs while the next panel writes
    LS_CUDA(cudaLaunchKernelEx(&cfg, k_lu_panel<T>, list, (const NodeDev *)s->d_nodes, arena, j0,
                               csize, cap, s->d_swaps + (j0 / LU_NB & 1) * s->n_swaps, s->d_pperm,
                               s->d_info));
    if (kmax <= LU_NB) break;
    if (!ahead) {
      if ((rc = strips(st, LU_ALL, j0))) return rc;
      continue;
    }
    LS_CUDA(cudaEventRecord(s->ev_main, s->ahead));
    // the next panel's columns carry the rest of the step before
    if (was) LS_CUDA(cudaStreamWaitEvent(s->ahead, s->ev_rest, 0));
    if ((rc = strips(s->ahead, LU_NEXT, j0))) return rc;
    LS_CUDA(cudaStreamWaitEvent(st, s->ev_main, 0));
    if ((rc = strips(st, LU_REST, j0))) return rc;
    LS_CUDA(cudaEventRecord(s->ev_rest, st));
  }
  if (ahead) {
    LS_CUDA(cudaEventRecord(s->ev_main, s->ahead));
    LS_CUDA(cudaStreamWaitEvent(st, s->ev_main, 0));
  }
  if (kmax > 1 && rmax > 0) {
    const size_t per = (size_t)kmax * sizeof(T);
    const int warps = (int)std::max<size_t>(1, std::min<size_t>(8, 48 * 1024 / per));
    for (int f0 = 0; f0 < cnt; f0 += 65535) {
      k_perm_f12<T><<<dim3((unsigned)((rmax + warps - 1) / warps),
                           (unsigned)std::min(65535, cnt - f0)), warps * 32, per * warps, st>>>(
          list + f0, s->d_nodes, arena, cap, s->d_pperm, kmax);
      LS_CUDA(cudaGetLastError());
    }
  }
  return LFSOLVE_OK;
}

// The same for the fronts of depth d with more than cap pivots: the library's
// getrf on the padded pivot block, its swaps on F12, spread over the lanes
template <typename T>
int lu_library(lfsolve *s, int d, T *arena, int cap) {
  Plan &P = s->P;
  cudaStream_t st = s->stream;
  int lw_max = 0, kk_max = 0;
  for (int id : P.by_depth[d]) {
    const Node &N = P.nodes[id];
    if (N.k <= cap) continue;
    int lw = 0;
    LS_BLAS(getrf_buf(s->sol[0], N.roff, N.roff, arena + N.arena_off, N.ld, &lw));
    lw_max = std::max(lw_max, lw);
    kk_max = std::max(kk_max, N.roff);
  }
  if (kk_max == 0) return LFSOLVE_OK;
  for (int l = 0; l < LANES; ++l) {
    if (s->work_bytes[l] < (size_t)lw_max * sizeof(T)) {
      LS_CUDA(cudaStreamSynchronize(st));
      if (s->work[l]) LS_CUDA(cudaFree(s->work[l]));
      s->work_bytes[l] = (size_t)lw_max * sizeof(T);
      LS_CUDA(cudaMalloc(&s->work[l], s->work_bytes[l]));
    }
    if (s->lpiv_n[l] < kk_max) {
      LS_CUDA(cudaStreamSynchronize(st));
      if (s->lpiv[l]) LS_CUDA(cudaFree(s->lpiv[l]));
      s->lpiv_n[l] = kk_max;
      LS_CUDA(cudaMalloc((void **)&s->lpiv[l], sizeof(int) * kk_max));
    }
  }
  int rc = fork_lanes(s), li = 0;
  if (rc) return rc;
  for (int id : P.by_depth[d]) {
    const Node &N = P.nodes[id];
    if (N.k <= cap) continue;
    const int l = li++ % LANES, k = N.k, r = N.m - N.k, kk = N.roff;
    T *F = arena + N.arena_off;
    LS_BLAS(getrf(s->sol[l], kk, kk, F, N.ld, static_cast<T *>(s->work[l]), s->lpiv[l],
                  s->d_info + id));
    if (r > 0)
      k_swap_cols<T><<<(r + 127) / 128, 128, 0, s->lane[l]>>>(k, r, s->lpiv[l],
                                                              F + (long long)kk * N.ld, N.ld);
    k_ipiv_to_perm_one<<<1, 256, 0, s->lane[l]>>>(k, s->lpiv[l], s->d_pperm + N.p0);
    LS_CUDA(cudaGetLastError());
  }
  return join_lanes(s);
}

template <typename T>
int factor_impl(lfsolve *s, const double2 *vals) {
  Plan &P = s->P;
  cudaStream_t st = s->stream;
  const int D = P.max_depth + 1;
  // LFSOLVE_PROFILE set: per-depth device times printed after the call
  const bool prof = std::getenv("LFSOLVE_PROFILE") != nullptr;
  std::vector<cudaEvent_t> evs;
  if (prof) {
    evs.resize(2 * D);
    for (auto &e : evs) LS_CUDA(cudaEventCreate(&e));
  }
  T *fac = static_cast<T *>(s->d_fac);
  std::vector<DepthPlan> plan(D);
  size_t need[2] = {256, 256}, floats = 0;
  for (int d = 0; d < D; ++d) {
    plan[d] = depth_plan<T>(s, d);
    need[d & 1] = std::max(need[d & 1], (size_t)P.arena_size[d] * sizeof(T));
    floats = std::max(floats, plan[d].floats * plan[d].lanes);
  }
  int rc;
  for (int i = 0; i < 2; ++i)
    if ((rc = ensure_bytes(&s->d_arena[i], &s->arena_bytes[i], need[i]))) return rc;
  if (floats && (rc = ensure_bytes(&s->d_split, &s->split_bytes, floats * sizeof(float)))) return rc;
  float *split_buf = static_cast<float *>(s->d_split);
  std::vector<T *> arena(D);
  for (int d = 0; d < D; ++d) arena[d] = static_cast<T *>(s->d_arena[d & 1]);
  // pivot blocks beyond the panel kernel's rows go through the library
  // (LFSOLVE_LU_MAX lowers the bound)
  int lu_cap = std::min(LU_ROWS<T> * s->lu_cluster[s->prec], perm_smem_max<T>());
  if (const char *e = std::getenv("LFSOLVE_LU_MAX")) lu_cap = std::min(lu_cap, std::max(0, std::atoi(e)));
  for (int d = D - 1; d >= 0; --d) {
    if (prof) LS_CUDA(cudaEventRecord(evs[2 * d], st));
    const int cnt = (int)P.by_depth[d].size();
    if (s->n_bf[d] > 0) {
      k_build_fronts<T><<<s->n_bf[d], BUILD_T, 0, st>>>(s->d_bf[d], s->d_nodes, s->d_child,
                                                        reinterpret_cast<const int2 *>(s->d_src),
                                                        d + 1 < D ? arena[d + 1] : nullptr, arena[d]);
      LS_CUDA(cudaGetLastError());
    }
    const long long na = (long long)P.asm_src[d].size();
    if (na > 0) {
      k_assemble<T><<<grid_for(na, 256), 256, 0, st>>>(na, s->d_asm_src[d], s->d_asm_dst[d], vals,
                                                       arena[d]);
      LS_CUDA(cudaGetLastError());
    }
    if ((rc = lu_depth<T>(s, d, arena[d], lu_cap)) || (rc = lu_library<T>(s, d, arena[d], lu_cap))) return rc;
    // the update blocks and the sweeps read U's diagonal blocks divided by their pivots
    const int ni = s->diag_at[d + 1] - s->diag_at[d];
    if (ni > 0) {
      k_diag_scale<T><<<(ni + DIAG_WARPS - 1) / DIAG_WARPS, DIAG_WARPS * 32, 0, st>>>(
          ni, s->d_diag + s->diag_at[d], s->d_nodes, arena[d]);
      LS_CUDA(cudaGetLastError());
    }
    const DepthPlan &Q = plan[d];
    // the groups with most work first, spread over the lanes
    std::vector<FrontGroup> order;
    for (const FrontGroup &G : P.groups[d])
      if (G.kp > 0 && G.rp > 0) order.push_back(G);
    auto work = [](const FrontGroup &G) { return (double)G.cnt * G.kp * G.rp * (G.kp + G.rp); };
    std::sort(order.begin(), order.end(),
              [&](const FrontGroup &a, const FrontGroup &b) { return work(a) > work(b); });
    const bool fork = Q.lanes > 1;
    if (fork && (rc = fork_lanes(s))) return rc;
    int li = 0;
    for (const FrontGroup &g : order) {
      const int l = li++ % Q.lanes;
      const bool split = front_split<T>(s, g.rp, g.kp, g.cnt);
      const int step = split ? (int)std::min<size_t>(32768, Q.floats / split_floats(g.kp, g.rp)) : 32768;
      for (int f0 = 0; f0 < g.cnt; f0 += step) {
        const Group<T> G{arena[d] + g.off + f0 * g.stride, g.stride, std::min(step, g.cnt - f0), g.kp,
                         g.rp, g.kp + g.rp, {}, {}, {}, {}};
        if ((rc = group_update<T>(fork ? s->lane[l] : st, fork ? s->blas[l] : s->blas_main, G,
                                  split ? split_buf + l * Q.floats : nullptr)))
          return rc;
      }
    }
    if (fork && (rc = join_lanes(s))) return rc;
    if (s->n_co[d] > 0) {
      k_copy_out<T><<<s->n_co[d], 256, 0, st>>>(s->d_co[d], s->d_nodes, arena[d], fac);
      LS_CUDA(cudaGetLastError());
    }
    if (prof) LS_CUDA(cudaEventRecord(evs[2 * d + 1], st));
  }
  if (prof) {
    LS_CUDA(cudaStreamSynchronize(st));
    for (int d = D - 1; d >= 0; --d) {
      float ms = 0.f;
      LS_CUDA(cudaEventElapsedTime(&ms, evs[2 * d], evs[2 * d + 1]));
      double fl = 0.0;
      int mmax = 0;
      for (int id : P.by_depth[d]) {
        const Node &N = P.nodes[id];
        const double k = N.k, r = N.m - N.k;
        fl += 8.0 * (k * k * k / 3.0 + k * k * r + k * r * r);
        mmax = std::max(mmax, N.m);
      }
      std::printf("lfsolve profile: depth %2d fronts %5zu max m %5d  %8.2f ms  %7.2f TFLOP/s\n", d,
                  P.by_depth[d].size(), mmax, ms, fl / (ms * 1e-3) / 1e12);
    }
    std::fflush(stdout);
    for (auto &e : evs) cudaEventDestroy(e);
  }
  return LFSOLVE_OK;
}

// one launch that may start while the launch before it is still running
template <typename T>
int sweep_launch(void (*kern)(Sweep<T>, int), const Sweep<T> &S, dim3 grid, size_t smem, int j0,
                 cudaStream_t st) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(SW_T);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  LS_CUDA(cudaLaunchKernelEx(&cfg, kern, S, j0));
  return LFSOLVE_OK;
}

// Depths of at most so many fronts are bound by the latency of a step's two
// phases and take the kernels that hold their factors on chip; with more, HBM
// is the bound, and blocks that stream them with more of their kind on an SM
// are the faster (524k-row line grating, held and streamed, forward + backward:
// 1 front 0.32 and 0.64 ms, 4 fronts 0.62 and 0.75, 16 fronts 0.39 and 0.42,
// 32 fronts 0.51 and 0.53, 64 fronts 0.48 and 0.48, 256 fronts 0.33 and 0.31).
constexpr int HELD_FRONTS = 32;

// one launch of a phase over the fronts of a depth (fewer than 1,024,
// front_per_block), at most nch chunks each in nz parts
template <typename T, int NR, int TRANS, int PH>
int sweep_phase(const Sweep<T> &S, int nch, int fronts, int j0, cudaStream_t st, int nz = 1) {
  if (nch <= 0) return LFSOLVE_OK;
  constexpr bool FWD = PH == PH_FWD_A || PH == PH_FWD_B;
  const dim3 grid((unsigned)nch, (unsigned)fronts, (unsigned)nz);
  void (*kern)(Sweep<T>, int) = k_sweep<T, NR, TRANS, PH>;
  size_t smem = 0;
  if constexpr (sizeof(T) == 8) {
    if constexpr (PH == PH_FWD_A || PH == PH_BWD_A)
      if (fronts <= HELD_FRONTS) kern = k_sweep_tri<NR, TRANS, !FWD>, smem = TRI_SMEM;
    if constexpr (PH == PH_FWD_B || PH == PH_BWD_B)
      if (fronts <= HELD_FRONTS) kern = k_sweep_apply<NR, TRANS, !FWD>;
  }
  return sweep_launch<T>(kern, S, grid, smem, j0, st);
}

// A block per front walks through its phases where that fills the GPU evenly
// (three blocks a SM) or the fronts are so small that launches would dominate;
// else a launch per phase.  512 fronts are between the two (more than one wave);
// a sweep pair of one column in complex64, so and by phases: 0.089 and 0.097 ms
// with at most 282 rows, 0.124 and 0.124 with 360, 0.366 and 0.369 with 633,
// 0.565 and 0.557 with 861; of two columns 0.102 and 0.109, 0.139 and 0.143,
// 0.409 and 0.391, 0.622 and 0.575.
bool front_per_block(size_t fronts, int max_m) {
  return fronts >= 1024 || (fronts >= 512 && max_m <= 512) || max_m <= 160;
}

// Parts that a depth's first backward product takes its update rows in: where the
// pivot chunks alone are too few blocks (or rows) to keep HBM busy, at least 256
// rows each; 1: no partial sums
int sweep_parts(const SolveShape &Z, int fronts) {
  if (Z.k == 0 || Z.r == 0 || front_per_block(fronts, Z.m)) return 1;
  return std::max(1, std::min(std::min(SW_PARTS, Z.r / 256), SWEEP_BLOCKS / (chunks(Z.k) * fronts)));
}

// one pass of NR columns: b (n x NR, ld n, precision T, original numbering)
// -> x (same layout)
template <typename T, int NR, int TRANS>
int solve_pass(lfsolve *s, const T *b, T *x) {
  Plan &P = s->P;
  cudaStream_t st = s->stream;
  const int D = P.max_depth + 1, n = P.n;
  Sweep<T> S{s->d_nodes, nullptr, static_cast<const T *>(s->d_fac), s->d_perm, s->d_pperm,
             s->d_rorig, s->d_src, static_cast<T *>(s->d_V), static_cast<T *>(s->d_Y),
             P.vec_rows, P.nn, n, b, x, static_cast<T *>(s->d_part_y)};
  // LFSOLVE_PROFILE set: per-depth device times of both sweeps
  const bool prof = std::getenv("LFSOLVE_PROFILE") != nullptr;
  std::vector<cudaEvent_t> evs;
  if (prof) {
    evs.resize(4 * D);
    for (auto &e : evs) LS_CUDA(cudaEventCreate(&e));
  }
  int rc;
  // forward, deepest level first
  for (int d = D - 1; d >= 0; --d) {
    if (prof) LS_CUDA(cudaEventRecord(evs[4 * d], st));
    const int cnt = (int)P.by_depth[d].size();
    const SolveShape &Z = P.shape[d];
    S.list = s->d_all[d];
    if (front_per_block(cnt, Z.m)) {
      k_sweep_fwd_front<T, NR, TRANS><<<cnt, SW_T, 0, st>>>(S);
      LS_CUDA(cudaGetLastError());
    } else {
      if ((rc = sweep_phase<T, NR, TRANS, PH_GATHER>(S, (Z.m + SW_T - 1) / SW_T, cnt, 0, st))) return rc;
      for (int j0 = 0; j0 < Z.k; j0 += SB) {
        const int below = TRANS ? Z.k - j0 - SB : std::max(Z.m - j0 - SB, Z.r);
        if ((rc = sweep_phase<T, NR, TRANS, PH_FWD_A>(S, 1, cnt, j0, st))) return rc;
        if ((rc = sweep_phase<T, NR, TRANS, PH_FWD_B>(S, chunks(below), cnt, j0, st))) return rc;
      }
      if (TRANS && (rc = sweep_phase<T, NR, TRANS, PH_FWD_U>(S, chunks(Z.r), cnt, 0, st))) return rc;
    }
    if (prof) LS_CUDA(cudaEventRecord(evs[4 * d + 1], st));
  }
  // essential rows
  if (P.n_ess > 0) {
    k_ess_copy<T><<<grid_for(P.n_ess, 256), 256, 0, st>>>(P.n_ess, s->d_ess, b, n, x, n, NR);
    LS_CUDA(cudaGetLastError());
  }
  // backward, root first
  for (int d = 0; d < D; ++d) {
    if (prof) LS_CUDA(cudaEventRecord(evs[4 * d + 2], st));
    const int cnt = (int)P.by_depth[d].size();
    const SolveShape &Z = P.shape[d];
    S.list = s->d_all[d];
    if (front_per_block(cnt, Z.m)) {
      k_sweep_bwd_front<T, NR, TRANS><<<cnt, SW_T, 0, st>>>(S);
      LS_CUDA(cudaGetLastError());
    } else if (Z.k > 0) {
      if (Z.r > 0) {
        const int nz = sweep_parts(Z, cnt);
        if ((rc = sweep_phase<T, NR, TRANS, PH_BWD_R>(S, chunks(Z.k), cnt, 0, st, nz))) return rc;
        if (nz > 1 && (rc = sweep_phase<T, NR, TRANS, PH_BWD_S>(S, (Z.k + SW_T - 1) / SW_T, cnt, nz, st)))
          return rc;
      }
      for (int j0 = (Z.k - 1) / SB * SB; j0 >= 0; j0 -= SB) {
        if ((rc = sweep_phase<T, NR, TRANS, PH_BWD_A>(S, 1, cnt, j0, st))) return rc;
        if ((rc = sweep_phase<T, NR, TRANS, PH_BWD_B>(S, chunks(j0), cnt, j0, st))) return rc;
      }
    }
    if (prof) LS_CUDA(cudaEventRecord(evs[4 * d + 3], st));
  }
  if (prof) {
    LS_CUDA(cudaStreamSynchronize(st));
    for (int d = D - 1; d >= 0; --d) {
      float f = 0.f, w = 0.f;
      LS_CUDA(cudaEventElapsedTime(&f, evs[4 * d], evs[4 * d + 1]));
      LS_CUDA(cudaEventElapsedTime(&w, evs[4 * d + 2], evs[4 * d + 3]));
      std::printf("lfsolve solve profile (%s, %d rhs): depth %2d fronts %5zu  "
                  "forward %7.3f ms  backward %7.3f ms\n", TRANS ? "A^T" : "A", NR, d,
                  P.by_depth[d].size(), f, w);
    }
    std::fflush(stdout);
    for (auto &e : evs) cudaEventDestroy(e);
  }
  return LFSOLVE_OK;
}
template <typename T>
int solve_pass(lfsolve *s, int nr, const T *b, T *x, int trans) {
  if (nr == 1) return trans ? solve_pass<T, 1, 1>(s, b, x) : solve_pass<T, 1, 0>(s, b, x);
  return trans ? solve_pass<T, 2, 1>(s, b, x) : solve_pass<T, 2, 0>(s, b, x);
}

int ensure_solve_scratch(lfsolve *s, size_t es) {
  Plan &P = s->P;
  const size_t V = (size_t)P.vec_rows * MAX_NRHS_PASS * es;
  const size_t Y = (size_t)std::max(1, P.nn) * MAX_NRHS_PASS * es;
  const size_t bw = (size_t)P.n * 2 * MAX_NRHS_PASS * es;  // b and x in the factor precision
  int rc, parts = 1;
  for (int d = 0; d <= P.max_depth; ++d)
    parts = std::max(parts, sweep_parts(P.shape[d], (int)P.by_depth[d].size()));
  if ((rc = ensure_bytes(&s->d_V, &s->V_bytes, V)) || (rc = ensure_bytes(&s->d_Y, &s->Y_bytes, Y)) ||
      (rc = ensure_bytes(&s->d_part_y, &s->part_y_bytes, parts > 1 ? Y * parts : 0)) ||
      (rc = ensure_bytes(&s->d_bw, &s->bw_bytes, bw)))
    return rc;
  return LFSOLVE_OK;
}

// complex128 in / out, any nrhs, optional per-column scale of the input
// (the output is scaled back): x = A_f^-1 (b * s) / s, accumulate: x += ...
template <typename T>
int solve_any(lfsolve *s, int nrhs, const double2 *b, double2 *x, int trans,
              const double *d_scale, int accumulate) {
  int rc = ensure_solve_scratch(s, sizeof(T));
  if (rc) return rc;
  const int n = s->P.n;
  T *bw = static_cast<T *>(s->d_bw);
  T *xw = bw + (size_t)n * MAX_NRHS_PASS;
  cudaStream_t st = s->stream;
  for (int c0 = 0; c0 < nrhs; c0 += MAX_NRHS_PASS) {
    const int nr = std::min(MAX_NRHS_PASS, nrhs - c0);
    k_to_prec<T><<<grid_for((long long)n * nr, 256), 256, 0, st>>>(
        n, nr, b + (size_t)c0 * n, d_scale ? d_scale + c0 : nullptr, bw);
    LS_CUDA(cudaGetLastError());
    if ((rc = solve_pass<T>(s, nr, bw, xw, trans))) return rc;
    if (d_scale) {
      // the scale was applied to b; undo it on x: pass 1 / scale
      k_from_prec<T><<<grid_for((long long)n * nr, 256), 256, 0, st>>>(
          n, nr, xw, d_scale + nrhs + c0, x + (size_t)c0 * n, accumulate);
    } else {
      k_from_prec<T><<<grid_for((long long)n * nr, 256), 256, 0, st>>>(
          n, nr, xw, nullptr, x + (size_t)c0 * n, accumulate);
    }
    LS_CUDA(cudaGetLastError());
  }
  return LFSOLVE_OK;
}

int solve_dispatch(lfsolve *s, int nrhs, const double2 *b, double2 *x, int trans,
                   const double *d_scale, int accumulate) {
  return s->prec == LFSOLVE_C64 ? solve_any<cuComplex>(s, nrhs, b, x, trans, d_scale, accumulate)
                                : solve_any<cuDoubleComplex>(s, nrhs, b, x, trans, d_scale, accumulate);
}

// GMRES-IR for one column: restarted GMRES(m) on A x = b in FP64 (complex128
// vectors, modified Gram-Schmidt Arnoldi, complex Givens rotations), right
// preconditioned by the factors (M^-1 v: one triangular solve of the
// factorization's precision), from the current x.  The Krylov basis, the
// Hessenberg solve and the update x += M^-1 (V y) follow the standard
// algorithm (Saad and Schultz 1986; with a low-precision preconditioner,
// Carson and Higham's GMRES-based iterative refinement, 2017-2018).  *iters
// counts the Arnoldi steps; *rel is the final true relative residual.
int gmres_column(lfsolve *s, const int *d_I, const int *d_J, const double2 *vals, const int *tp,
                 const double2 *b, double2 *x, int trans, double tol, int max_steps, int m,
                 double *rel, int *iters) {
  using cd = std::complex<double>;
  const int n = s->P.n;
  cudaStream_t st = s->stream;
  int rc = ensure_lanes(s);
  if (rc) return rc;
  cublasHandle_t hb = s->blas_main;
  LS_BLAS(cublasSetPointerMode(hb, CUBLAS_POINTER_MODE_HOST));
  double2 *V = nullptr, *z = nullptr, *w = nullptr;
  LS_CUDA(cudaMalloc((void **)&V, sizeof(double2) * (size_t)n * (m + 1)));
  LS_CUDA(cudaMalloc((void **)&z, sizeof(double2) * (size_t)n));
  LS_CUDA(cudaMalloc((void **)&w, sizeof(double2) * (size_t)n));
  struct Free {
    void *a, *b, *c;
    ~Free() { cudaFree(a); cudaFree(b); cudaFree(c); }
  } guard{V, z, w};
  auto spmv = [&](const double2 *in, double2 *out) -> int {
    k_spmv<<<(n + 7) / 8, 256, 0, st>>>(n, d_I, d_J, vals, tp, in, out);
    LS_CUDA(cudaGetLastError());
    return LFSOLVE_OK;
  };
  auto zc = [](cuDoubleComplex v) { return cd(v.x, v.y); };
  auto cz = [](cd v) { return make_cuDoubleComplex(v.real(), v.imag()); };
  double bn = 0.0;
  LS_BLAS(cublasDznrm2(hb, n, reinterpret_cast<const cuDoubleComplex *>(b), 1, &bn));
  if (bn == 0.0) bn = 1.0;
  std::vector<cd> H((size_t)(m + 1) * m), g(m + 1), sn(m), y(m);
  std::vector<double> cs(m);
  int steps = 0;
  *rel = 1.0;
  while (true) {
    // r = b - A x into V[0]
    if ((rc = spmv(x, w))) return rc;
    LS_CUDA(cudaMemcpyAsync(V, b, sizeof(double2) * n, cudaMemcpyDeviceToDevice, st));
    const cuDoubleComplex mone = make_cuDoubleComplex(-1.0, 0.0);
    auto *V0 = reinterpret_cast<cuDoubleComplex *>(V);
    LS_BLAS(cublasZaxpy(hb, n, &mone, reinterpret_cast<const cuDoubleComplex *>(w), 1, V0, 1));
    double beta = 0.0;
    LS_BLAS(cublasDznrm2(hb, n, V0, 1, &beta));
    *rel = beta / bn;
    if (*rel <= tol || steps >= max_steps || beta == 0.0) break;
    const double ib = 1.0 / beta;
    LS_BLAS(cublasZdscal(hb, n, &ib, V0, 1));
    std::fill(g.begin(), g.end(), cd(0.0));
    g[0] = beta;
    int k = 0;
    for (; k < m && steps < max_steps; ++k) {
      auto *Vk = reinterpret_cast<cuDoubleComplex *>(V + (size_t)k * n);
      // w = A M^-1 v_k
      if ((rc = solve_dispatch(s, 1, reinterpret_cast<const double2 *>(Vk), z, trans, nullptr, 0)))
        return rc;
      if ((rc = spmv(z, w))) return rc;
      auto *W = reinterpret_cast<cuDoubleComplex *>(w);
      for (int i = 0; i <= k; ++i) {
        auto *Vi = reinterpret_cast<cuDoubleComplex *>(V + (size_t)i * n);
        cuDoubleComplex hij;
        LS_BLAS(cublasZdotc(hb, n, Vi, 1, W, 1, &hij));
        H[(size_t)i * m + k] = zc(hij);
        const cuDoubleComplex neg = make_cuDoubleComplex(-hij.x, -hij.y);
        LS_BLAS(cublasZaxpy(hb, n, &neg, Vi, 1, W, 1));
      }
      double hn = 0.0;
      LS_BLAS(cublasDznrm2(hb, n, W, 1, &hn));
      H[(size_t)(k + 1) * m + k] = hn;
      if (hn > 0.0) {
        const double ih = 1.0 / hn;
        LS_CUDA(cudaMemcpyAsync(V + (size_t)(k + 1) * n, w, sizeof(double2) * n,
                                cudaMemcpyDeviceToDevice, st));
        LS_BLAS(cublasZdscal(hb, n, &ih,
                             reinterpret_cast<cuDoubleComplex *>(V + (size_t)(k + 1) * n), 1));
      }
      // earlier rotations on column k, then the one that zeroes H[k+1][k]
      for (int i = 0; i < k; ++i) {
        const cd a = H[(size_t)i * m + k], c = H[(size_t)(i + 1) * m + k];
        H[(size_t)i * m + k] = cs[i] * a + sn[i] * c;
        H[(size_t)(i + 1) * m + k] = -std::conj(sn[i]) * a + cs[i] * c;
      }
      const cd a = H[(size_t)k * m + k];
      const double bb = hn, r = std::hypot(std::abs(a), bb);
      if (std::abs(a) == 0.0) {
        cs[k] = 0.0;
        sn[k] = 1.0;
        H[(size_t)k * m + k] = bb;
      } else {
        const cd ph = a / std::abs(a);
        cs[k] = std::abs(a) / r;
        sn[k] = ph * bb / r;
        H[(size_t)k * m + k] = ph * r;
      }
      H[(size_t)(k + 1) * m + k] = 0.0;
      g[k + 1] = -std::conj(sn[k]) * g[k];
      g[k] = cs[k] * g[k];
      ++steps;
      if (std::abs(g[k + 1]) / bn <= 0.5 * tol || hn == 0.0) {
        ++k;
        break;
      }
    }
    // y = H^-1 g (upper triangular k x k), u = V y, x += M^-1 u
    for (int i = k - 1; i >= 0; --i) {
      cd t = g[i];
      for (int j = i + 1; j < k; ++j) t -= H[(size_t)i * m + j] * y[j];
      y[i] = t / H[(size_t)i * m + i];
    }
    LS_CUDA(cudaMemsetAsync(w, 0, sizeof(double2) * n, st));
    for (int i = 0; i < k; ++i) {
      const cuDoubleComplex yi = cz(y[i]);
      LS_BLAS(cublasZaxpy(hb, n, &yi, reinterpret_cast<const cuDoubleComplex *>(V + (size_t)i * n),
                          1, reinterpret_cast<cuDoubleComplex *>(w), 1));
    }
    if ((rc = solve_dispatch(s, 1, w, x, trans, nullptr, 1))) return rc;
  }
  *iters = steps;
  LS_CUDA(cudaStreamSynchronize(st));
  return LFSOLVE_OK;
}

void free_workspace(lfsolve *s) {
  for (int i = 0; i < 2; ++i) {
    if (s->d_arena[i]) cudaFree(s->d_arena[i]);
    s->d_arena[i] = nullptr;
    s->arena_bytes[i] = 0;
  }
  if (s->d_split) cudaFree(s->d_split);
  s->d_split = nullptr;
  s->split_bytes = 0;
}

}  // namespace

extern "C" {

const char *lfsolve_last_error(void) { return g_err.c_str(); }

int lfsolve_create(int gpu_id, lfsolve **out) {
  g_err.clear();
  if (!out) return fail(LFSOLVE_ERR_ARG, "NULL output pointer");
  *out = nullptr;
  lfsolve *s = new lfsolve();
  s->dev = gpu_id;
  *out = s;
  return LFSOLVE_OK;
}

int lfsolve_set_stream(lfsolve *s, void *stream) {
  if (!s) return fail(LFSOLVE_ERR_ARG, "NULL solver");
  s->stream = (cudaStream_t)stream;
  if (s->blas_main) LS_BLAS(cublasSetStream(s->blas_main, s->stream));
  return LFSOLVE_OK;
}

int lfsolve_analyze(lfsolve *s, int n, const int *I, const int *J, long long nnz, int ne, int nd,
                    const int *elem_dof, const double *centroid, const int *ess, int n_ess,
                    int leaf_elements) {
  g_err.clear();
  if (!s || !I || !J || !elem_dof || !centroid || (n_ess > 0 && !ess))
    return fail(LFSOLVE_ERR_ARG, "NULL argument");
  if (n <= 0 || ne <= 0 || nd <= 0 || nnz <= 0 || n_ess < 0)
    return fail(LFSOLVE_ERR_ARG, "sizes must be positive");
  if (nnz >= (1LL << 31)) return fail(LFSOLVE_ERR_ARG, "nnz beyond the int32 CSR contract");
  if (I[0] != 0 || I[n] != nnz) return fail(LFSOLVE_ERR_ARG, "row pointer does not span nnz");
  const auto t0 = std::chrono::steady_clock::now();
  const int leaf = leaf_elements > 0 ? leaf_elements : 32;
  // the device tables, the factors and the buffers sized by the plan go with it
  if (s->blas_main) {
    LS_CUDA(cudaSetDevice(s->dev));
    free_plan(s);
  }
  s->analyzed = false;   // until the plan stands
  const int rc = build_plan(n, I, J, nnz, ne, nd, elem_dof, centroid, ess, n_ess, leaf, s->P);
  if (rc) return rc;
  const auto t1 = std::chrono::steady_clock::now();
  s->analyzed = true;
  lfsolve_stats &st = s->st;
  st = lfsolve_stats{};
  st.n = n;
  st.n_ess = s->P.n_ess;
  st.n_fronts = (int)s->P.nodes.size();
  st.depth = s->P.max_depth + 1;
  st.max_front = s->P.max_front;
  st.max_pivots = s->P.max_k;
  st.factor_entries = s->P.factor_entries;
  st.factor_flops = s->P.flops;
  st.peak_front_entries = s->P.peak_front_entries;
  st.analyze_s = std::chrono::duration<double>(t1 - t0).count();
  return LFSOLVE_OK;
}

int lfsolve_get_ordering(lfsolve *s, int *perm, int *node_of) {
  if (!s || !s->analyzed) return fail(LFSOLVE_ERR_STATE, "lfsolve_analyze has not run");
  if (perm) std::copy(s->P.perm.begin(), s->P.perm.end(), perm);
  if (node_of) std::copy(s->P.node_of.begin(), s->P.node_of.end(), node_of);
  return LFSOLVE_OK;
}

int lfsolve_get_fronts(lfsolve *s, int *parent, int *depth, int *k, int *m) {
  if (!s || !s->analyzed) return fail(LFSOLVE_ERR_STATE, "lfsolve_analyze has not run");
  const std::vector<Node> &nodes = s->P.nodes;
  for (size_t i = 0; i < nodes.size(); ++i) {
    if (parent) parent[i] = nodes[i].parent;
    if (depth) depth[i] = nodes[i].depth;
    if (k) k[i] = nodes[i].k;
    if (m) m[i] = nodes[i].m;
  }
  return LFSOLVE_OK;
}

int lfsolve_get_stats(lfsolve *s, lfsolve_stats *out) {
  if (!s || !out) return fail(LFSOLVE_ERR_ARG, "NULL argument");
  *out = s->st;
  return LFSOLVE_OK;
}

int lfsolve_factor(lfsolve *s, const void *d_vals, int prec) {
  g_err.clear();
  if (!s || !d_vals) return fail(LFSOLVE_ERR_ARG, "NULL argument");
  if (!s->analyzed) return fail(LFSOLVE_ERR_STATE, "lfsolve_analyze has not run");
  if (prec != LFSOLVE_C64 && prec != LFSOLVE_C128) return fail(LFSOLVE_ERR_ARG, "unknown precision %d", prec);
  LS_CUDA(cudaSetDevice(s->dev));
  int rc = ensure_lanes(s);
  if (rc) return rc;
  if ((rc = ensure_uploaded(s))) return rc;
  const size_t es = prec == LFSOLVE_C64 ? sizeof(cuComplex) : sizeof(cuDoubleComplex);
  if (s->prec != prec) {
    free_factors(s);
    LS_CUDA(cudaMalloc(&s->d_fac, std::max<size_t>((size_t)s->P.factor_entries * es, 256)));
    s->prec = prec;
  }
  if (!s->d_pperm) LS_CUDA(cudaMalloc((void **)&s->d_pperm, sizeof(int) * std::max(1, s->P.nn)));
  if (!s->d_info) LS_CUDA(cudaMalloc((void **)&s->d_info, sizeof(int) * s->P.nodes.size()));
  LS_CUDA(cudaMemsetAsync(s->d_info, 0, sizeof(int) * s->P.nodes.size(), s->stream));
  LS_CUDA(cudaEventRecord(s->t0, s->stream));
  rc = prec == LFSOLVE_C64 ? factor_impl<cuComplex>(s, static_cast<const double2 *>(d_vals))
                           : factor_impl<cuDoubleComplex>(s, static_cast<const double2 *>(d_vals));
  if (rc) return rc;
  LS_CUDA(cudaEventRecord(s->t1, s->stream));
  LS_CUDA(cudaStreamSynchronize(s->stream));
  LS_CUDA(cudaEventElapsedTime(&s->st.factor_ms, s->t0, s->t1));
  std::vector<int> info(s->P.nodes.size());
  LS_CUDA(cudaMemcpy(info.data(), s->d_info, sizeof(int) * info.size(), cudaMemcpyDeviceToHost));
  for (size_t i = 0; i < info.size(); ++i)
    if (info[i] != 0)
      return fail(LFSOLVE_ERR_SINGULAR, "front %zu: zero pivot at position %d of %d", i, info[i],
                  s->P.nodes[i].k);
  return LFSOLVE_OK;
}

int lfsolve_solve(lfsolve *s, int nrhs, const void *d_b, void *d_x, int transpose) {
  g_err.clear();
  if (!s || !d_b || !d_x || nrhs <= 0) return fail(LFSOLVE_ERR_ARG, "bad arguments");
  if (!s->d_fac) return fail(LFSOLVE_ERR_STATE, "lfsolve_factor has not run");
  LS_CUDA(cudaSetDevice(s->dev));
  LS_CUDA(cudaEventRecord(s->t0, s->stream));
  int rc = solve_dispatch(s, nrhs, static_cast<const double2 *>(d_b), static_cast<double2 *>(d_x),
                          transpose != 0, nullptr, 0);
  if (rc) return rc;
  LS_CUDA(cudaEventRecord(s->t1, s->stream));
  LS_CUDA(cudaStreamSynchronize(s->stream));
  LS_CUDA(cudaEventElapsedTime(&s->st.solve_ms, s->t0, s->t1));
  return LFSOLVE_OK;
}

int lfsolve_solve_refined(lfsolve *s, const int *d_I, const int *d_J, const void *d_vals,
                          int nrhs, const void *d_b, void *d_x, int transpose, double tol,
                          int max_iter, double *rel_out, int *iters_out) {
  g_err.clear();
  if (!s || !d_I || !d_J || !d_vals || !d_b || !d_x || nrhs <= 0)
    return fail(LFSOLVE_ERR_ARG, "bad arguments");
  if (!s->d_fac) return fail(LFSOLVE_ERR_STATE, "lfsolve_factor has not run");
  if (d_b == d_x) return fail(LFSOLVE_ERR_ARG, "the refined solve needs x and b apart");
  LS_CUDA(cudaSetDevice(s->dev));
  const int n = s->P.n;
  cudaStream_t st = s->stream;
  const size_t rb = (size_t)n * nrhs * sizeof(double2);
  int rc;
  if ((rc = ensure_bytes((void **)&s->d_r, &s->r_bytes, rb))) return rc;
  const int wpb = 8;
  const int nblk = (n + wpb - 1) / wpb;
  const size_t pb = (size_t)3 * nblk * nrhs * sizeof(double) + (size_t)3 * nrhs * sizeof(double);
  if ((rc = ensure_bytes((void **)&s->d_part, &s->part_bytes, pb)) ||
      (rc = ensure_bytes((void **)&s->d_scale, &s->scale_bytes, sizeof(double) * 2 * nrhs)))
    return rc;
  double *sums = s->d_part + (size_t)3 * nblk * nrhs;
  const double2 *b = static_cast<const double2 *>(d_b);
  double2 *x = static_cast<double2 *>(d_x);
  const int *tp = transpose ? s->d_tpos : nullptr;
  std::vector<double> h(3 * nrhs), sc(2 * nrhs);
  auto residual = [&](double *worst) -> int {
    k_resid<<<dim3(nblk, nrhs), wpb * 32, 0, st>>>(n, nrhs, d_I, d_J,
                                                   static_cast<const double2 *>(d_vals), tp, x, b,
                                                   s->d_r, s->d_part);
    LS_CUDA(cudaGetLastError());
    k_resid_sum<<<nrhs, 1024, 0, st>>>(nblk, nrhs, s->d_part, sums);
    LS_CUDA(cudaGetLastError());
    LS_CUDA(cudaMemcpyAsync(h.data(), sums, sizeof(double) * 3 * nrhs, cudaMemcpyDeviceToHost, st));
    LS_CUDA(cudaStreamSynchronize(st));
    *worst = 0.0;
    for (int c = 0; c < nrhs; ++c) {
      const double rel = h[3 * c + 1] > 0 ? std::sqrt(h[3 * c] / h[3 * c + 1]) : std::sqrt(h[3 * c]);
      if (rel_out) rel_out[c] = rel;
      *worst = std::max(*worst, rel);
      // the correction's right-hand side is scaled to a unit max entry
      const double mx = h[3 * c + 2] > 0 ? h[3 * c + 2] : 1.0;
      sc[c] = 1.0 / mx;
      sc[nrhs + c] = mx;
    }
    return LFSOLVE_OK;
  };
  LS_CUDA(cudaEventRecord(s->t0, st));
  if ((rc = solve_dispatch(s, nrhs, b, x, transpose != 0, nullptr, 0))) return rc;
  double worst = 0.0;
  int it = 0, steps = 0;
  if ((rc = residual(&worst))) return rc;
  // classical refinement while it contracts; when a correction reduces the
  // worst residual by less than half (or LFSOLVE_GMRES=1 asks for it from
  // the start), GMRES-IR takes over, column by column, with up to
  // 10 max_iter Arnoldi steps (LFSOLVE_GMRES=0: never)
  const char *ge = std::getenv("LFSOLVE_GMRES");
  bool gmres = ge && ge[0] == '1';
  const bool no_gmres = ge && ge[0] == '0';  // classical refinement only
  // (comparisons written so that a NaN residual counts as not converged)
  while (!gmres && !(worst <= tol) && it < max_iter) {
    LS_CUDA(cudaMemcpyAsync(s->d_scale, sc.data(), sizeof(double) * 2 * nrhs, cudaMemcpyHostToDevice, st));
    if ((rc = solve_dispatch(s, nrhs, s->d_r, x, transpose != 0, s->d_scale, 1))) return rc;
    ++it;
    const double prev = worst;
    if ((rc = residual(&worst))) return rc;
    if (!(worst <= tol) && !(worst <= 0.5 * prev) && !no_gmres) gmres = true;
  }
  if (gmres && !(worst <= tol)) {
    // a diverged refinement leaves x worse than zero: start from x = 0
    if (!(worst < 1.0)) LS_CUDA(cudaMemsetAsync(x, 0, sizeof(double2) * (size_t)n * nrhs, st));
    for (int c = 0; c < nrhs; ++c) {
      double rel = 0.0;
      int k = 0;
      if ((rc = gmres_column(s, d_I, d_J, static_cast<const double2 *>(d_vals), tp,
                             b + (size_t)c * n, x + (size_t)c * n, transpose != 0, tol,
                             10 * std::max(1, max_iter), 30, &rel, &k)))
        return rc;
      steps += k;
    }
    if ((rc = residual(&worst))) return rc;
  }
  it += steps;
  LS_CUDA(cudaEventRecord(s->t1, st));
  LS_CUDA(cudaStreamSynchronize(st));
  LS_CUDA(cudaEventElapsedTime(&s->st.solve_ms, s->t0, s->t1));
  s->st.refine_iters = it;
  s->st.refine_rel = worst;
  if (iters_out) *iters_out = it;
  if (!(worst <= tol))
    return fail(LFSOLVE_ERR_NOCONV,
                "refinement stopped at relative residual %.3e after %d corrections / GMRES steps",
                worst, it);
  return LFSOLVE_OK;
}

int lfsolve_release_factors(lfsolve *s) {
  if (!s) return fail(LFSOLVE_ERR_ARG, "NULL solver");
  cudaSetDevice(s->dev);
  free_factors(s);
  free_workspace(s);
  return LFSOLVE_OK;
}

void lfsolve_destroy(lfsolve *s) {
  if (!s) return;
  cudaSetDevice(s->dev);
  if (s->stream) cudaStreamSynchronize(s->stream);
  free_plan(s);
  free_workspace(s);
  void *bufs[] = {s->d_V, s->d_Y, s->d_part_y, s->d_bw, s->d_r, s->d_part, s->d_scale};
  for (void *p : bufs)
    if (p) cudaFree(p);
  for (int l = 0; l < LANES; ++l) {
    if (s->work[l]) cudaFree(s->work[l]);
    if (s->lpiv[l]) cudaFree(s->lpiv[l]);
    if (s->blas[l]) cublasDestroy(s->blas[l]);
    if (s->sol[l]) cusolverDnDestroy(s->sol[l]);
    if (s->lane[l]) cudaStreamDestroy(s->lane[l]);
    if (s->ev_lane[l]) cudaEventDestroy(s->ev_lane[l]);
  }
  if (s->blas_main) cublasDestroy(s->blas_main);
  if (s->ev_main) cudaEventDestroy(s->ev_main);
  if (s->ev_rest) cudaEventDestroy(s->ev_rest);
  if (s->ahead) cudaStreamDestroy(s->ahead);
  if (s->t0) cudaEventDestroy(s->t0);
  if (s->t1) cudaEventDestroy(s->t1);
  delete s;
}

}  // extern "C"

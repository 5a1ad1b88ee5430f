// LU factorization of the fronts' pivot blocks, included by lfsolve.cu inside
// its namespace.  All fronts of a depth advance together, 32 columns a step:
//
//   k_lu_panel   P [A_jj; A_below] = [L_jj; L_below] U_jj with partial
//                pivoting among the pivot rows left, a cluster of blocks per
//                front, a thread per row with its 32 entries in registers;
//   k_lu_strip   the step's interchanges on every other column of the pivot
//                block, U_j = L_jj^-1 A_j to the right and the rank-32 update
//                of what is below, a block per strip of columns.
//
// A column of the panel costs one reduction and one broadcast over the rows.
// Rows never move while the panel is factored: each thread tracks the place
// its row goes to and stores it there at the end.  Bound: the panel by the
// latency of those two exchanges, the strips by FP32 / FP64 FMA issue.
#include <cooperative_groups.h>

constexpr int LU_NB = 32;                  // columns of a step
// rows a panel block takes (a thread each; 65,536 registers a SM)
template <typename T> constexpr int LU_ROWS = sizeof(T) == 8 ? 640 : 320;
constexpr int LU_MAX_CLUSTER = 16;         // above 8: non-portable, asked for
template <typename T> constexpr int LU_STRIP = sizeof(T) == 8 ? 32 : 16;  // columns of a strip
constexpr int LU_STRIP_T = 256;            // threads of a strip block

// a step's interchanges: pivot j0 + i takes row src[i]; the row that was at
// j0 + i goes to dst[i]
struct LuSwaps { int src[LU_NB], dst[LU_NB]; };

// ordered key of |re| + |im| (NaN above infinity), and its largest over a warp
template <typename T> struct LuKeyOf { using type = unsigned; };
template <> struct LuKeyOf<cuDoubleComplex> { using type = unsigned long long; };
template <typename T> using LuKey = typename LuKeyOf<T>::type;
__device__ __forceinline__ unsigned lu_key(cuComplex v) {
  return __float_as_uint(fabsf(v.x) + fabsf(v.y));
}
__device__ __forceinline__ unsigned long long lu_key(cuDoubleComplex v) {
  return (unsigned long long)__double_as_longlong(fabs(v.x) + fabs(v.y));
}
__device__ __forceinline__ unsigned lu_max(unsigned k) { return __reduce_max_sync(0xffffffffu, k); }
__device__ __forceinline__ unsigned long long lu_max(unsigned long long k) {
  const unsigned hi = lu_max((unsigned)(k >> 32));
  const unsigned lo = lu_max((unsigned)(k >> 32) == hi ? (unsigned)k : 0u);
  return (unsigned long long)hi << 32 | lo;
}

// 1 / v, scaled by |re| + |im| so that neither square over- nor underflows, and a
// Newton step r += r (1 - v r): every multiplier of a column and every solution
// entry of a row carries this error (its root mean square over random pivots is
// 0.9 units without the step)
template <typename T> __device__ __forceinline__ T lu_rcp(T v) {
  const auto s = 1 / (fabs(v.x) + fabs(v.y));
  const auto x = v.x * s, y = v.y * s;
  const auto d = s / (x * x + y * y);
  T r;
  r.x = x * d;
  r.y = -y * d;
  const auto p = v.x * r.y;
  const auto ex = fma(v.y, r.y, fma(-v.x, r.x, decltype(p)(1)));
  const auto ey = -(fma(v.y, r.x, p) + fma(v.x, r.y, -p));
  T o;
  o.x = fma(-r.y, ey, fma(r.x, ex, r.x));
  o.y = fma(r.x, ey, fma(r.y, ex, r.y));
  return o;
}

// a candidate row: its reciprocal pivot, then its entries from the column on
template <typename T> struct __align__(16) LuCand { T rp, unused, row[LU_NB]; };
template <typename T> struct LuSmem {
  // per warp (one block) or per rank (a cluster)
  LuCand<T> cand[2][LU_ROWS<T> / 32 > LU_MAX_CLUSTER ? LU_ROWS<T> / 32 : LU_MAX_CLUSTER];
  LuKey<T> key[2][32];                         // per warp
  int tid[2][32], place[2][32];
  LuKey<T> ckey[2][LU_MAX_CLUSTER];            // per cluster rank
  int cplace[2][LU_MAX_CLUSTER];
};

// two complex64 entries, or one complex128, a load
__device__ __forceinline__ void lu_load2(const cuComplex *p, cuComplex &a, cuComplex &b) {
  const float4 v = *reinterpret_cast<const float4 *>(p);
  a = make_cuComplex(v.x, v.y);
  b = make_cuComplex(v.z, v.w);
}
__device__ __forceinline__ void lu_load2(const cuDoubleComplex *p, cuDoubleComplex &a,
                                         cuDoubleComplex &b) {
  a = p[0];
  b = p[1];
}

// What one thread carries through the panel.
template <typename T> struct LuRow {
  T a[LU_NB];      // its entries from the current column on
  int place;       // where the row goes
  bool active;     // not a pivot yet
};

// Columns [jb, je), at most W left at jb.  The current column is always a[0]:
// each step's update shifts the row by one, so that the loop body is one piece
// of code (fully unrolled, the instructions of 32 columns no longer fit the
// instruction cache: 3.1 us a column).  done[j]: the finished entry.
template <typename T, int W>
__device__ __forceinline__ void lu_columns(LuSmem<T> &sm, LuRow<T> &R, T *done, int jb, int je,
                                           int j0, int csize, int rank, int &bad) {
  namespace cg = cooperative_groups;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
#pragma unroll 1
  for (int j = jb; j < je; ++j) {
    const int b = j & 1;
    // the block's largest entry of the column (ties: the lowest thread); every
    // row works out its reciprocal while the reduction is under way
    const LuKey<T> key = R.active ? lu_key(R.a[0]) : 0;
    const LuKey<T> best = lu_max(key);
    const unsigned at = __ballot_sync(0xffffffffu, R.active && key == best);
    const T rp = lu_rcp(R.a[0]);
    auto put = [&](LuCand<T> &C) {
      C.rp = rp;
#pragma unroll
      for (int c = 0; c < W; ++c) C.row[c] = R.a[c];
    };
    const bool lead = at && lane == __ffs(at) - 1;   // the warp's candidate
    if (lead) {
      sm.place[b][w] = R.place;
      if (csize == 1) put(sm.cand[b][w]);
    }
    if (lane == 0) {
      sm.key[b][w] = best;
      sm.tid[b][w] = at ? w * 32 + __ffs(at) - 1 : -1;
    }
    __syncthreads();
    const int wt = lane < nw ? sm.tid[b][lane] : -1;
    const LuKey<T> wk = wt >= 0 ? sm.key[b][lane] : 0;
    const LuKey<T> top = lu_max(wk);
    const unsigned from = __ballot_sync(0xffffffffu, wt >= 0 && wk == top);
    int src = __ffs(from) - 1;                       // the winning warp, -1: no row left here
    const int win = src >= 0 ? sm.tid[b][src] : -1;
    int pl = src >= 0 ? sm.place[b][src] : -1;
    bool here = true;
    if (csize > 1) {
      // the block's row to every block of the cluster
      cg::cluster_group cl = cg::this_cluster();
      if (win < 0) {
        if (tid < csize) cl.map_shared_rank(&sm, tid)->cplace[b][rank] = -1;
      } else if (w == win >> 5) {
        // staged in the block's own slot, then pushed a lane per entry
        if (tid == win) put(sm.cand[b][rank]);
        __syncwarp();
        const T v = sm.cand[b][rank].row[lane];
        const T v0 = sm.cand[b][rank].rp;
        for (int r = 0; r < csize; ++r) {
          LuSmem<T> *o = cl.map_shared_rank(&sm, r);
          if (r != rank && lane < W) o->cand[b][rank].row[lane] = v;
          if (lane == 0) {
            if (r != rank) o->cand[b][rank].rp = v0;
            o->ckey[b][rank] = top;
            o->cplace[b][rank] = pl;
          }
        }
      }
      cl.sync();
      // the best of the blocks' rows (one is left as long as j < je)
      const int cp = lane < csize ? sm.cplace[b][lane] : -1;
      const LuKey<T> ck = cp >= 0 ? sm.ckey[b][lane] : 0;
      const LuKey<T> ct = lu_max(ck);
      src = __ffs(__ballot_sync(0xffffffffu, cp >= 0 && ck == ct)) - 1;
      pl = sm.cplace[b][src];
      here = src == rank;
    }
    const LuCand<T> &C = sm.cand[b][src];
    T p0, p1;
    lu_load2(C.row, p0, p1);
    const bool zero = p0.x == 0 && p0.y == 0;
    if (R.place == j0 + j) R.place = pl;  // the row that makes room
    T l = czero<T>();
    if (here && tid == win) {
      R.place = j0 + j;
      R.active = false;
    } else if (R.active && !zero) {
      l = cmul(R.a[0], C.rp);
      R.a[0] = l;
    }
    if (zero && bad == 0) bad = j0 + j + 1;  // a zero column: nothing to eliminate
    done[(size_t)j * blockDim.x] = R.a[0];
    R.a[0] = cfms(R.a[1], l, p1);
#pragma unroll
    for (int c = 2; c < W; c += 2) {
      lu_load2(C.row + c, p0, p1);
      R.a[c - 1] = cfms(R.a[c], l, p0);
      if (c + 1 < W) R.a[c] = cfms(R.a[c + 1], l, p1);
    }
  }
}

// block rank r of a front's cluster holds rows j0 + r blockDim + t; dynamic
// shared memory: LU_NB entries a thread
template <typename T>
__global__ void __launch_bounds__(LU_ROWS<T>, 1)
k_lu_panel(const int *__restrict__ list, const NodeDev *__restrict__ nodes, T *arena, int j0,
           int csize, int cap, LuSwaps *__restrict__ swaps, int *__restrict__ pperm,
           int *__restrict__ info) {
  extern __shared__ __align__(16) unsigned char lu_raw[];
  __shared__ LuSmem<T> sm;
  const int f = blockIdx.x / csize, rank = blockIdx.x % csize;
  const int id = list[f];
  const NodeDev N = nodes[id];
  const int k = N.k, nb = min(LU_NB, k - j0);
  if (nb <= 0 || k > cap) return;  // the whole cluster
  // a block's shared memory is another block's to write only once it runs: every
  // block reports here, and waits for the others behind its loads
  if (csize > 1) cooperative_groups::this_cluster().barrier_arrive();
  const int tid = threadIdx.x;
  const int row = j0 + rank * (int)blockDim.x + tid;
  const bool mine = row < k;
  T *A = arena + N.arena_off + (long long)j0 * N.ld;
  T *done = reinterpret_cast<T *>(lu_raw) + tid;
  LuRow<T> R;
#pragma unroll
  for (int c = 0; c < LU_NB; ++c)
    R.a[c] = mine && c < nb ? A[row + (long long)c * N.ld] : czero<T>();
  // the pivot order so far moves with the rows: pivot p is original row pperm[p]
  const int orig = !mine ? 0 : j0 == 0 ? row : pperm[N.p0 + row];
  R.place = row;
  R.active = mine;
  int bad = 0;
  if (csize > 1) cooperative_groups::this_cluster().barrier_wait();
  lu_columns<T, 32>(sm, R, done, 0, min(nb, 12), j0, csize, rank, bad);
  lu_columns<T, 20>(sm, R, done, 12, min(nb, 22), j0, csize, rank, bad);
  lu_columns<T, 10>(sm, R, done, 22, nb, j0, csize, rank, bad);
  if (mine) {
    for (int c = 0; c < nb; ++c) A[R.place + (long long)c * N.ld] = done[(size_t)c * blockDim.x];
    if (R.place < j0 + nb) swaps[f].src[R.place - j0] = row;
    if (row < j0 + nb) swaps[f].dst[row - j0] = R.place;
    pperm[N.p0 + R.place] = orig;
  }
  if (bad && rank == 0 && tid == 0 && info[id] == 0) info[id] = bad;
  if (csize > 1) cooperative_groups::this_cluster().sync();  // no block leaves while others push to it
}

// strips of the columns outside the panel, front blockIdx.y: all of them, the
// next panel's, or all but those (lu_depth).
enum { LU_ALL, LU_NEXT, LU_REST };
// PART 0: a whole strip; where fronts x strips leave SMs idle, PART 1 does the
// exchange and U_j, and PART 2 the update with the rows split over blockIdx.z
// (a 2,528-pivot front alone: 118 us a step in one part, its first step).
template <typename T, int PART>
__global__ void __launch_bounds__(LU_STRIP_T, 2)
k_lu_strip(const int *__restrict__ list, const NodeDev *__restrict__ nodes, T *arena, int j0,
           int cap, const LuSwaps *__restrict__ swaps, int which) {
  constexpr int SC = LU_STRIP<T>, CW = SC / 2;
  __shared__ __align__(16) T X[LU_NB][SC];     // the pivot rows of the strip, then U_j
  __shared__ T L[LU_NB][LU_NB + 1];            // L_jj
  __shared__ LuSwaps sw;
  const int f = blockIdx.y, id = list[f];
  const NodeDev N = nodes[id];
  const int k = N.k, nb = min(LU_NB, k - j0), ld = N.ld;
  const int first = j0 / SC, strip = blockIdx.x;
  const int q0 = SC * (which == LU_NEXT ? first + strip
                       : which == LU_REST && strip >= first ? strip + LU_NB / SC : strip);
  if (nb <= 0 || k > cap || q0 >= k - nb) return;
  const bool right = q0 >= j0;                 // j0 is a multiple of the strip width
  if (PART == 2 && !right) return;
  const int c0 = right ? q0 + nb : q0, nc = min(SC, (right ? k : j0) - c0);
  const int tid = threadIdx.x;
  T *A = arena + N.arena_off + (long long)c0 * ld;
  const T *P = arena + N.arena_off + (long long)j0 * ld;
  if (PART == 2) {
    for (int t = tid; t < LU_NB * SC; t += LU_STRIP_T) {
      const int i = t % LU_NB, c = t / LU_NB;
      X[i][c] = c < nc ? A[j0 + i + (long long)c * ld] : czero<T>();
    }
    __syncthreads();
  } else {
    if (tid < nb) {
      sw.src[tid] = swaps[f].src[tid];
      sw.dst[tid] = swaps[f].dst[tid];
    }
    __syncthreads();
    // every load of the exchange in flight before the first store (a column's
    // rows belong to one warp)
    constexpr int IT = LU_NB * SC / LU_STRIP_T, CS = LU_STRIP_T / LU_NB;
    const int i = tid % LU_NB, ci = tid / LU_NB;
    T old[IT], nw[IT];
#pragma unroll
    for (int u = 0; u < IT; ++u) {
      const int c = ci + u * CS;
      const bool in = i < nb && c < nc;
      old[u] = in ? A[j0 + i + (long long)c * ld] : czero<T>();
      nw[u] = in ? A[sw.src[i] + (long long)c * ld] : czero<T>();
    }
    if (right)
#pragma unroll
      for (int c = ci; c < LU_NB; c += CS)  // right strips: nb = LU_NB
        L[i][c] = i > c ? P[j0 + i + (long long)c * ld] : czero<T>();
    __syncwarp();
#pragma unroll
    for (int u = 0; u < IT; ++u) {
      const int c = ci + u * CS;
      X[i][c] = nw[u];
      if (i >= nb || c >= nc) continue;
      if (sw.dst[i] >= j0 + nb) A[sw.dst[i] + (long long)c * ld] = old[u];
      if (!right) A[j0 + i + (long long)c * ld] = nw[u];
    }
    if (!right) return;
    __syncthreads();
    {  // U_j = L_jj^-1 X: a lane per row, the strip's columns dealt to the warps
      const int lane = tid & 31, w = tid >> 5;
      constexpr int NW = LU_STRIP_T / 32;
      for (int c = w; c < SC; c += 2 * NW) {
        const int d = c + NW;  // two columns at once
        T x = X[lane][c], y = X[lane][d];
#pragma unroll 4
        for (int l = 0; l < LU_NB - 1; ++l) {
          T u, v;
          u.x = __shfl_sync(0xffffffffu, x.x, l); u.y = __shfl_sync(0xffffffffu, x.y, l);
          v.x = __shfl_sync(0xffffffffu, y.x, l); v.y = __shfl_sync(0xffffffffu, y.y, l);
          const T e = L[lane][l];             // zero on and above the diagonal
          x = cfms(x, e, u);
          y = cfms(y, e, v);
        }
        __syncwarp();
        X[lane][c] = x;
        X[lane][d] = y;
        if (c < nc) A[j0 + lane + (long long)c * ld] = x;
        if (d < nc) A[j0 + lane + (long long)d * ld] = y;
      }
    }
    __syncthreads();
    if (PART == 1) return;
  }
  // A_below -= L_below U_j: a thread per row, half the strip at a time in
  // registers, its sums and its entries of A, eight columns of L ahead.  The 32
  // terms are summed by themselves and A takes their sum: one rounding of A a
  // step, as in a matrix product (residuals of a dense 5,153-pivot front in
  // complex64: 1.7e-6 with A as the accumulator, 3.6e-7 so; its factorization
  // 20.9 and 21.3 ms.  With the whole strip's sums at once the registers do not
  // hold A too, and its loads come last: 249 instead of 235 ms for a 524k-row
  // line grating)
  for (int r = j0 + LU_NB + (PART == 2 ? blockIdx.z * LU_STRIP_T : 0) + tid; r < k;
       r += LU_STRIP_T * (PART == 2 ? gridDim.z : 1)) {
    T *Ar = A + r;
#pragma unroll 1
    for (int cb = 0; cb < nc; cb += CW, Ar += (long long)CW * ld) {
      T acc[CW], old[CW], v[8], nx[8];
#pragma unroll
      for (int l = 0; l < 8; ++l) nx[l] = P[r + (long long)l * ld];
#pragma unroll
      for (int c = 0; c < CW; ++c) old[c] = cb + c < nc ? Ar[(long long)c * ld] : czero<T>();
#pragma unroll
      for (int c = 0; c < CW; ++c) acc[c] = czero<T>();
#pragma unroll 1
      for (int l0 = 0; l0 < LU_NB; l0 += 8) {
#pragma unroll
        for (int l = 0; l < 8; ++l) v[l] = nx[l];
        if (l0 + 8 < LU_NB)
#pragma unroll
          for (int l = 0; l < 8; ++l) nx[l] = P[r + (long long)(l0 + 8 + l) * ld];
#pragma unroll
        for (int l = 0; l < 8; ++l)
#pragma unroll
          for (int c = 0; c < CW; c += 2) {
            T u0, u1;
            lu_load2(&X[l0 + l][cb + c], u0, u1);
            acc[c] = cfms(acc[c], v[l], u0);
            acc[c + 1] = cfms(acc[c + 1], v[l], u1);
          }
      }
#pragma unroll
      for (int c = 0; c < CW; ++c)
        if (cb + c < nc) Ar[(long long)c * ld] = cadd(old[c], acc[c]);
    }
  }
}

// the pivot order on the update columns F12 of every front of a depth: a warp
// per column, the pivot rows staged in shared memory (k entries a warp)
template <typename T>
__global__ void k_perm_f12(const int *__restrict__ list, const NodeDev *__restrict__ nodes, T *arena,
                           int cap, const int *__restrict__ pperm, int stage) {
  extern __shared__ __align__(16) unsigned char pf_raw[];
  const NodeDev N = nodes[list[blockIdx.y]];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int c = blockIdx.x * (blockDim.x >> 5) + w;
  if (c >= N.m - N.k || N.k > cap) return;
  T *sv = reinterpret_cast<T *>(pf_raw) + (size_t)w * stage;
  T *col = arena + N.arena_off + (long long)(N.roff + c) * N.ld;
  for (int i = lane; i < N.k; i += 32) sv[i] = col[i];
  __syncwarp();
  for (int i = lane; i < N.k; i += 32) col[i] = sv[pperm[N.p0 + i]];
}

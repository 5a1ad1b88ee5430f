// Triangular sweeps of the multifrontal solve, included by lfsolve.cu inside
// its namespace (after NodeDev and the complex helpers).
//
// A front's factors are P (m x k: L11\U11, then L21) and U12 (k x r).  A
// substitution with L11 or U11 is a serial chain of k pivots.  Here it is cut
// into steps of SB pivots: one block solves a step's SB x SB triangle
// (diag_solve), then as many blocks as there are rows apply its columns.
// Inside the triangle a warp substitutes through a link of 32 pivots by itself
// (unit_solve), a lane a pivot, and hands the results to the others.  The rows
// of U's 32 x 32 diagonal blocks are kept divided by their pivots, and the
// pivots as their reciprocals (k_diag_scale, once per factorization, in place),
// so that a link is a unit triangle in all four sweeps: no division and no
// multiplication in its chain.  (Inverses of the blocks in their place are a
// product without a chain, 4.8 instead of 5.4 ms for two columns on a 524k-row
// line grating in complex64 and 2.7 instead of 2.9 ms in complex128 on a
// 111k-row hole, but not backward stable: triangles of -1 leave residuals 10^5
// times those of substitution.)
//
// Bound: every factor entry is read once a sweep pair from HBM; on the
// smallest systems the launches.
//
// Vectors: node s owns V[vec_off .. vec_off + m) per right-hand-side column
// (columns VR apart); Y[p0 .. p0 + k) (columns nn apart) holds its
// intermediate pivot values.
//
// Step of a front, pivots J = [j0, j1):
//   forward,  A:    Y_J = L_JJ^-1 V_J;      V_rest -= P_rest,J Y_J
//   forward,  A^T:  Y_J = U_JJ^-T V_J;      V_(>J) -= P_J,(>J)^T Y_J; after
//                   the last step V_R -= U12^T Y
//   backward, A:    Y -= U12 x_R; then from the last step: V_J = U_JJ^-1 Y_J,
//                   Y_(<J) -= P_(<J),J V_J
//   backward, A^T:  Y -= L21^T x_R; then V_J = L_JJ^-T Y_J,
//                   Y_(<J) -= P_J,(<J)^T V_J
constexpr int SB = 256;        // pivots of a step
constexpr int SW_T = 256;      // threads of a sweep block (one per pivot of a step)
constexpr int SW_W = SW_T / 32;
constexpr int SW_TILE = 256;   // vector entries staged at a time
constexpr int SW_CHUNK = 32;   // rows (or columns of the transposed product) a block forms at once
static_assert(SB == SW_T, "diag_solve takes a pivot a thread");

template <typename T> __device__ __forceinline__ void cfma(T &a, T x, T y) {
  a.x = fma(x.x, y.x, a.x); a.x = fma(-x.y, y.y, a.x);
  a.y = fma(x.x, y.y, a.y); a.y = fma(x.y, y.x, a.y);
}

template <typename T> struct Sweep {
  const NodeDev *nodes;
  const int *list;          // the fronts of the depth
  const T *fac;
  const int *perm, *pperm;  // elimination order; pivot permutation of every front
  const int *rorig;         // update rows in the original numbering
  const int *src;           // per vector row: the two children's rows that add to it (-1: none)
  T *V, *Y;
  long long VR;
  int nn, n;
  const T *b;               // right-hand side (n a column, original numbering)
  T *x;                     // solution
  T *part;                  // partial sums of the backward sweep's first product
};
constexpr int SW_PARTS = 8;   // at most so many a pivot

template <typename T, int NR> struct SweepSmem {
  T in[SW_TILE * NR];
  T red[SW_W * SW_CHUNK * NR];
};

// acc[q] += sum over c = c0, c0 + step, ... < c1 of A[row, c] in[c], A at the
// lane's row; 128 bytes a lane in flight
template <typename T, int NR>
__device__ __forceinline__ void row_dot(const T *__restrict__ Ar, long long ld, int c0, int c1, int step,
                                        const T *in, T (&acc)[NR]) {
  constexpr int U = 128 / sizeof(T);
  int c = c0;
  for (; c + (U - 1) * step < c1; c += U * step) {
    T a[U];
#pragma unroll
    for (int u = 0; u < U; ++u) a[u] = Ar[(c + u * step) * ld];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int q = 0; q < NR; ++q) cfma(acc[q], a[u], in[(c + u * step) * NR + q]);
  }
#pragma unroll 4
  for (; c < c1; c += step) {
    const T a = Ar[c * ld];
#pragma unroll
    for (int q = 0; q < NR; ++q) cfma(acc[q], a, in[c * NR + q]);
  }
}

// out[q] (threads 0..31: row r0 + lane) = sum over c < nc of A[row, c] in(c, q),
// the warps taking every SW_W-th column; reduced in warp order
template <typename T, int NR, class In>
__device__ __forceinline__ void tile_rows(const T *__restrict__ A, int ld, int r0, int nr, int nc,
                                          In in, SweepSmem<T, NR> &sm, T (&out)[NR]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int row = r0 + lane;
  const T *Ar = A + min(row, nr - 1);
  T acc[NR];
#pragma unroll
  for (int q = 0; q < NR; ++q) acc[q] = czero<T>();
  for (int t0 = 0; t0 < nc; t0 += SW_TILE) {
    const int tn = min(SW_TILE, nc - t0);
    __syncthreads();
    for (int t = threadIdx.x; t < tn * NR; t += SW_T) sm.in[t] = in(t0 + t / NR, t % NR);
    __syncthreads();
    row_dot<T, NR>(Ar + (long long)t0 * ld, ld, w, tn, SW_W, sm.in, acc);
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NR; ++q) sm.red[(w * SW_CHUNK + lane) * NR + q] = acc[q];
  __syncthreads();
  if (w == 0)
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      T s = sm.red[lane * NR + q];
#pragma unroll
      for (int v = 1; v < SW_W; ++v) s = cadd(s, sm.red[(v * SW_CHUNK + lane) * NR + q]);
      out[q] = s;
    }
}

// The same for all nr rows of A, a warp per 32 rows and no reduction, where
// there are enough of them (else the warps split the columns): store(row, out)
template <typename T, int NR, class In, class F>
__device__ __forceinline__ void all_rows(const T *__restrict__ A, int ld, int nr, int nc, In in,
                                         SweepSmem<T, NR> &sm, F store) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nch = (nr + SW_CHUNK - 1) / SW_CHUNK;
  if (nch < 6) {
    for (int ch = 0; ch < nch; ++ch) {
      T o[NR];
      tile_rows<T, NR>(A, ld, ch * SW_CHUNK, nr, nc, in, sm, o);
      const int i = ch * SW_CHUNK + threadIdx.x;
      if (threadIdx.x < 32 && i < nr) store(i, o);
    }
    return;
  }
  for (int c0 = 0; c0 < nch; c0 += SW_W) {
    const int row = (c0 + w) * SW_CHUNK + lane;
    const T *Ar = A + min(row, nr - 1);
    T acc[NR];
#pragma unroll
    for (int q = 0; q < NR; ++q) acc[q] = czero<T>();
    for (int t0 = 0; t0 < nc; t0 += SW_TILE) {
      const int tn = min(SW_TILE, nc - t0);
      if (c0 == 0 || nc > SW_TILE) {
        __syncthreads();
        for (int t = threadIdx.x; t < tn * NR; t += SW_T) sm.in[t] = in(t0 + t / NR, t % NR);
        __syncthreads();
      }
      if (c0 + w < nch) row_dot<T, NR>(Ar + (long long)t0 * ld, ld, 0, tn, 1, sm.in, acc);
    }
    if (row < nr) store(row, acc);
  }
}

// out[u][q] (every lane of warp w: column c0 + w + SW_W u) = sum over rows i < nr
// of A[i, column] in(i, q): lanes along the contiguous rows, four columns a
// warp with their loads in flight together
template <typename T, int NR, class In>
__device__ __forceinline__ void tile_cols(const T *__restrict__ A, int ld, int nr, int c0, int nc,
                                          In in, SweepSmem<T, NR> &sm,
                                          T (&out)[SW_CHUNK / SW_W][NR]) {
  constexpr int NC = SW_CHUNK / SW_W;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const T *Ac[NC];
#pragma unroll
  for (int u = 0; u < NC; ++u) {
    Ac[u] = A + (long long)min(c0 + w + SW_W * u, nc - 1) * ld;
#pragma unroll
    for (int q = 0; q < NR; ++q) out[u][q] = czero<T>();
  }
  for (int t0 = 0; t0 < nr; t0 += SW_TILE) {
    const int tn = min(SW_TILE, nr - t0);
    __syncthreads();
    for (int t = threadIdx.x; t < tn * NR; t += SW_T) sm.in[t] = in(t0 + t / NR, t % NR);
    __syncthreads();
#pragma unroll 2
    for (int i = lane; i < tn; i += 32) {
      T a[NC];
#pragma unroll
      for (int u = 0; u < NC; ++u) a[u] = Ac[u][t0 + i];
#pragma unroll
      for (int u = 0; u < NC; ++u)
#pragma unroll
        for (int q = 0; q < NR; ++q) cfma(out[u][q], a[u], sm.in[i * NR + q]);
    }
  }
#pragma unroll
  for (int u = 0; u < NC; ++u)
#pragma unroll
    for (int q = 0; q < NR; ++q)
      for (int o = 16; o; o >>= 1) {
        out[u][q].x += __shfl_xor_sync(0xffffffffu, out[u][q].x, o);
        out[u][q].y += __shfl_xor_sync(0xffffffffu, out[u][q].y, o);
      }
}

// f(column, out[q]) for the chunk's columns below nc, one lane each
template <typename T, int NR, class F>
__device__ __forceinline__ void each_col(T (&out)[SW_CHUNK / SW_W][NR], int c0, int nc, F f) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int u = 0; u < SW_CHUNK / SW_W; ++u) {
    const int col = c0 + w + SW_W * u;
    if (lane == u && col < nc) f(col, out[u]);
  }
}

// A unit triangle of 32 pivots across the warp, pivots h H .. h H + H - 1 of
// them: a[i] = the lane's entry of pivot h H + i (zero but for the pivots before
// the lane's in the order of substitution), v = the lane's entry, in place.  W
// pivots a round: every lane takes their entries, works through their W x W
// corner by itself and subtracts all W, so that a round waits for one shuffle.
template <typename T> constexpr int UNIT_W = sizeof(T) == 8 ? 4 : 2;
template <typename T, int NR, int BWD, int H>
__device__ __forceinline__ void unit_solve(const T (&a)[H], int h, T (&v)[NR]) {
  constexpr int W = UNIT_W<T>;
  auto from = [](T x, int p) {
    x.x = __shfl_sync(0xffffffffu, x.x, p);
    x.y = __shfl_sync(0xffffffffu, x.y, p);
    return x;
  };
#pragma unroll
  for (int g = 0; g < H; g += W) {
    T x[W][NR];
    auto at = [&](int j) { return BWD ? H - 1 - g - j : g + j; };   // the round's pivot j
#pragma unroll
    for (int j = 0; j < W; ++j)
#pragma unroll
      for (int q = 0; q < NR; ++q) x[j][q] = from(v[q], h * H + at(j));
#pragma unroll
    for (int j = 1; j < W; ++j)
#pragma unroll
      for (int i = 0; i < j; ++i) {
        const T c = from(a[at(i)], h * H + at(j));
#pragma unroll
        for (int q = 0; q < NR; ++q) x[j][q] = cfms(x[j][q], c, x[i][q]);
      }
#pragma unroll
    for (int j = 0; j < W; ++j)
#pragma unroll
      for (int q = 0; q < NR; ++q) v[q] = cfms(v[q], a[at(j)], x[j][q]);
  }
}

// The triangle of one step, v[q] = this thread's pivot of the step (thread t:
// pivot t < nb), in place: forward with L (TRANS = 0) or U^T, backward with U
// or L^T.  A thread keeps its own entry in a register and reads its row (for
// the transposed triangles its column) of D a link of 32 entries at a time:
// AHEAD a whole link before it is used (a block alone on its SM), else 16
// entries at once (several blocks a SM, fewer registers).  The warp of a link
// substitutes through it (unit_solve) and hands its 32 results to the others.
template <typename T, int NR, int TRANS, int BWD, bool AHEAD>
__device__ __forceinline__ void diag_solve(const T *__restrict__ D, int ld, int nb, T (&v)[NR],
                                           T *ys) {
  constexpr int H = AHEAD ? 32 : 16;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int links = (nb + 31) / 32;
  T a[H], nx[AHEAD ? 32 : 1];
  constexpr bool UNIT = TRANS == BWD;   // L; U's pivots come as reciprocals
  const T rd = !UNIT && t < nb ? D[t + (long long)t * ld] : CT<T>::mk(1.0, 0.0);
  auto load = [&](int s, int l0, T *dst) {
    // entries a link needs: its own warp's triangle, later warps' updates
    const bool need = t < nb && (BWD ? w <= s : w >= s);
#pragma unroll
    for (int i = 0; i < H; ++i) {
      const int l = l0 + i, o = 32 * s + l;
      const bool on = w != s || (BWD ? l > lane : l < lane);
      dst[i] = need && on && o < nb ? D[TRANS ? o + (long long)t * ld : t + (long long)o * ld]
                                    : czero<T>();
    }
  };
  if (AHEAD) load(BWD ? links - 1 : 0, 0, nx);
  for (int u = 0; u < links; ++u) {
    const int s = BWD ? links - 1 - u : u;
    if (AHEAD) {
#pragma unroll
      for (int l = 0; l < H; ++l) a[l] = nx[AHEAD ? l : 0];
      if (u + 1 < links) load(BWD ? s - 1 : s + 1, 0, nx);
    } else {
      load(s, BWD && w == s ? 32 - H : 0, a);
    }
    T *y = ys + (u & 1) * 32 * NR;
    if (w == s) {
      if (!UNIT && BWD)
#pragma unroll
        for (int q = 0; q < NR; ++q) v[q] = cmul(v[q], rd);
#pragma unroll
      for (int i = 0; i < 32 / H; ++i) {
        const int h = BWD ? 32 / H - 1 - i : i;
        if (i > 0) load(s, h * H, a);
        unit_solve<T, NR, BWD, H>(a, h, v);
      }
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        if (!UNIT && !BWD) v[q] = cmul(v[q], rd);
        y[lane * NR + q] = v[q];
      }
    }
    __syncthreads();
    if (BWD ? w < s : w > s) {
      T o[NR];
#pragma unroll
      for (int q = 0; q < NR; ++q) o[q] = czero<T>();
#pragma unroll
      for (int h = 0; h < 32 / H; ++h) {
        if (h > 0) load(s, h * H, a);
#pragma unroll
        for (int i = 0; i < H; ++i)
#pragma unroll
          for (int q = 0; q < NR; ++q) cfma(o[q], a[i], y[(h * H + i) * NR + q]);
      }
#pragma unroll
      for (int q = 0; q < NR; ++q) v[q] = csub(v[q], o[q]);
    }
  }
  __syncthreads();
}

__device__ __forceinline__ int chunks_of(int n) { return (n + SW_CHUNK - 1) / SW_CHUNK; }

// One front's part of each phase: `ch` = chunk, and the number of chunks.
template <typename T, int NR, int TRANS, bool AHEAD> struct Front {
  const Sweep<T> &S;
  const NodeDev N;
  SweepSmem<T, NR> &sm;
  const T *P, *U12;
  T *V, *Y;
  int m, k, r;
  __device__ Front(const Sweep<T> &S_, int id, SweepSmem<T, NR> &sm_)
      : S(S_), N(S_.nodes[id]), sm(sm_), m(N.m), k(N.k), r(N.m - N.k) {
    P = S.fac + N.fac_off;
    U12 = P + (long long)m * k;
    V = S.V + N.vec_off;
    Y = S.Y + N.p0;
  }
  // rows [a0, m) step da of the front's right-hand side: its pivots' entries
  // (in pivot order for A) plus the children's update rows
  __device__ void gather(int a0, int da) {
    for (int a = a0; a < m; a += da) {
      const int v = a >= k ? a : TRANS ? a : S.pperm[N.p0 + a];
      const int2 c = reinterpret_cast<const int2 *>(S.src)[N.vec_off + v];
      const int g = a < k ? S.perm[N.p0 + v] : -1;
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        T s = g >= 0 ? S.b[(long long)q * S.n + g] : czero<T>();
        if (c.x >= 0) s = cadd(s, S.V[c.x + q * S.VR]);
        if (c.y >= 0) s = cadd(s, S.V[c.y + q * S.VR]);
        V[a + q * S.VR] = s;
      }
    }
  }
  __device__ void fwd_a(int j0) {
    const int nb = min(SB, k - j0), i = threadIdx.x;
    T v[NR];
#pragma unroll
    for (int q = 0; q < NR; ++q) v[q] = i < nb ? V[j0 + i + q * S.VR] : czero<T>();
    diag_solve<T, NR, TRANS, 0, AHEAD>(P + j0 + (long long)j0 * m, m, nb, v, sm.in);
    if (i < nb)
#pragma unroll
      for (int q = 0; q < NR; ++q) Y[j0 + i + (long long)q * S.nn] = v[q];
  }
  __device__ int fwd_b_chunks(int j0) const {
    return chunks_of((TRANS ? k : m) - min(k, j0 + SB));
  }
  __device__ void fwd_b(int j0, int ch) {
    const int nb = min(SB, k - j0), j1 = j0 + nb;
    auto in = [&](int t, int q) { return Y[j0 + t + (long long)q * S.nn]; };
    if (TRANS) {
      T o[SW_CHUNK / SW_W][NR];
      tile_cols<T, NR>(P + j0 + (long long)j1 * m, m, nb, ch * SW_CHUNK, k - j1, in, sm, o);
      each_col<T, NR>(o, ch * SW_CHUNK, k - j1, [&](int c, T (&v)[NR]) {
#pragma unroll
        for (int q = 0; q < NR; ++q) V[j1 + c + q * S.VR] = csub(V[j1 + c + q * S.VR], v[q]);
      });
    } else {
      T o[NR];
      tile_rows<T, NR>(P + j1 + (long long)j0 * m, m, ch * SW_CHUNK, m - j1, nb, in, sm, o);
      const int i = j1 + ch * SW_CHUNK + threadIdx.x;
      if (threadIdx.x < 32 && i < m)
#pragma unroll
        for (int q = 0; q < NR; ++q) V[i + q * S.VR] = csub(V[i + q * S.VR], o[q]);
    }
  }
  __device__ void fwd_b_all(int j0) {
    if (TRANS) {
      for (int c = 0; c < fwd_b_chunks(j0); ++c) fwd_b(j0, c);
      return;
    }
    const int nb = min(SB, k - j0), j1 = j0 + nb;
    all_rows<T, NR>(P + j1 + (long long)j0 * m, m, m - j1, nb,
                    [&](int t, int q) { return Y[j0 + t + (long long)q * S.nn]; }, sm,
                    [&](int i, T (&o)[NR]) {
#pragma unroll
                      for (int q = 0; q < NR; ++q) {
                        T &v = V[j1 + i + q * S.VR];
                        v = csub(v, o[q]);
                      }
                    });
  }
  __device__ int fwd_u_chunks() const { return TRANS ? chunks_of(r) : 0; }
  __device__ void fwd_u(int ch) {
    T o[SW_CHUNK / SW_W][NR];
    tile_cols<T, NR>(U12, k, k, ch * SW_CHUNK, r,
                               [&](int t, int q) { return Y[t + (long long)q * S.nn]; }, sm, o);
    each_col<T, NR>(o, ch * SW_CHUNK, r, [&](int c, T (&v)[NR]) {
#pragma unroll
      for (int q = 0; q < NR; ++q) V[k + c + q * S.VR] = csub(V[k + c + q * S.VR], v[q]);
    });
  }
  // Y -= U12 x_R (L21^T x_R): part z of nz of the update rows; one part
  // subtracts, several leave their sums in S.part for bwd_s
  __device__ int bwd_r_chunks() const { return r > 0 ? chunks_of(k) : 0; }
  __device__ void bwd_r(int ch, int z, int nz) {
    const int per = (r + nz - 1) / nz, t0 = min(r, z * per), rn = min(r, t0 + per) - t0;
    const int *ro = S.rorig + N.r_off + t0;
    auto in = [&](int t, int q) { return S.x[(long long)q * S.n + ro[t]]; };
    auto put = [&](int i, T (&o)[NR]) {
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        T &y = Y[i + (long long)q * S.nn];
        if (nz == 1) y = csub(y, o[q]);
        else S.part[((long long)z * NR + q) * S.nn + N.p0 + i] = o[q];
      }
    };
    if (TRANS) {
      T o[SW_CHUNK / SW_W][NR];
      tile_cols<T, NR>(P + k + t0, m, rn, ch * SW_CHUNK, k, in, sm, o);
      each_col<T, NR>(o, ch * SW_CHUNK, k, put);
    } else {
      T o[NR];
      tile_rows<T, NR>(U12 + (long long)t0 * k, k, ch * SW_CHUNK, k, rn, in, sm, o);
      const int i = ch * SW_CHUNK + threadIdx.x;
      if (threadIdx.x < 32 && i < k) put(i, o);
    }
  }
  __device__ void bwd_r_all() {
    if (r == 0) return;
    if (TRANS) {
      for (int c = 0; c < bwd_r_chunks(); ++c) bwd_r(c, 0, 1);
      return;
    }
    const int *ro = S.rorig + N.r_off;
    all_rows<T, NR>(U12, k, k, r, [&](int t, int q) { return S.x[(long long)q * S.n + ro[t]]; }, sm,
                    [&](int i, T (&o)[NR]) {
#pragma unroll
                      for (int q = 0; q < NR; ++q) {
                        T &y = Y[i + (long long)q * S.nn];
                        y = csub(y, o[q]);
                      }
                    });
  }
  __device__ void bwd_s(int i, int nz) {
    if (i >= k || r == 0) return;
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      T &y = Y[i + (long long)q * S.nn];
      T v = y;
      for (int z = 0; z < nz; ++z) v = csub(v, S.part[((long long)z * NR + q) * S.nn + N.p0 + i]);
      y = v;
    }
  }
  __device__ void bwd_a(int j0) {
    const int nb = min(SB, k - j0), i = threadIdx.x;
    T v[NR];
#pragma unroll
    for (int q = 0; q < NR; ++q) v[q] = i < nb ? Y[j0 + i + (long long)q * S.nn] : czero<T>();
    diag_solve<T, NR, TRANS, 1, AHEAD>(P + j0 + (long long)j0 * m, m, nb, v, sm.in);
    if (i >= nb) return;
    // the pivots' solution: for the front's own products, and to x
    const int g = S.perm[N.p0 + (TRANS ? S.pperm[N.p0 + j0 + i] : j0 + i)];
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      V[j0 + i + q * S.VR] = v[q];
      S.x[(long long)q * S.n + g] = v[q];
    }
  }
  __device__ int bwd_b_chunks(int j0) const { return chunks_of(j0); }
  __device__ void bwd_b(int j0, int ch) {
    const int nb = min(SB, k - j0);
    auto in = [&](int t, int q) { return V[j0 + t + q * S.VR]; };
    if (TRANS) {
      T o[SW_CHUNK / SW_W][NR];
      tile_cols<T, NR>(P + j0, m, nb, ch * SW_CHUNK, j0, in, sm, o);
      each_col<T, NR>(o, ch * SW_CHUNK, j0, [&](int c, T (&v)[NR]) {
#pragma unroll
        for (int q = 0; q < NR; ++q) {
          T &y = Y[c + (long long)q * S.nn];
          y = csub(y, v[q]);
        }
      });
    } else {
      T o[NR];
      tile_rows<T, NR>(P + (long long)j0 * m, m, ch * SW_CHUNK, j0, nb, in, sm, o);
      const int i = ch * SW_CHUNK + threadIdx.x;
      if (threadIdx.x < 32 && i < j0)
#pragma unroll
        for (int q = 0; q < NR; ++q) {
          T &y = Y[i + (long long)q * S.nn];
          y = csub(y, o[q]);
        }
    }
  }
  __device__ void bwd_b_all(int j0) {
    if (TRANS) {
      for (int c = 0; c < bwd_b_chunks(j0); ++c) bwd_b(j0, c);
      return;
    }
    const int nb = min(SB, k - j0);
    if (j0 == 0) return;
    all_rows<T, NR>(P + (long long)j0 * m, m, j0, nb,
                    [&](int t, int q) { return V[j0 + t + q * S.VR]; }, sm,
                    [&](int i, T (&o)[NR]) {
#pragma unroll
                      for (int q = 0; q < NR; ++q) {
                        T &y = Y[i + (long long)q * S.nn];
                        y = csub(y, o[q]);
                      }
                    });
  }
  // lines of the matrix a phase's block will read, asked for from HBM while
  // the phase before is still under way
  __device__ void ahead(const T *A, int ld, int rows, int cols) {
    for (int c = threadIdx.x; c < cols; c += SW_T)
      for (int b = 0; b < rows * (int)sizeof(T); b += 128)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char *>(A + (long long)c * ld) + b));
  }
};

// Depths of many fronts (or of small ones): a block per front walks through
// all its phases, one launch a depth and sweep.
template <typename T, int NR, int TRANS>
__global__ void __launch_bounds__(SW_T, sizeof(T) == 8 ? 3 : 2) k_sweep_fwd_front(const Sweep<T> S) {
  __shared__ SweepSmem<T, NR> sm;
  Front<T, NR, TRANS, false> F(S, S.list[blockIdx.x], sm);
  F.gather(threadIdx.x, SW_T);
  __syncthreads();
  for (int j0 = 0; j0 < F.k; j0 += SB) {
    F.fwd_a(j0);
    __syncthreads();
    F.fwd_b_all(j0);
    __syncthreads();
  }
  for (int c = 0; c < F.fwd_u_chunks(); ++c) F.fwd_u(c);
}
template <typename T, int NR, int TRANS>
__global__ void __launch_bounds__(SW_T, sizeof(T) == 8 ? 3 : 2) k_sweep_bwd_front(const Sweep<T> S) {
  __shared__ SweepSmem<T, NR> sm;
  Front<T, NR, TRANS, false> F(S, S.list[blockIdx.x], sm);
  F.bwd_r_all();
  __syncthreads();
  for (int j0 = (F.k - 1) / SB * SB; j0 >= 0 && F.k > 0; j0 -= SB) {
    F.bwd_a(j0);
    __syncthreads();
    F.bwd_b_all(j0);
    __syncthreads();
  }
}

// Depths of few large fronts: a launch per phase, a block per (chunk, front).
// The launches overlap (programmatic dependent launch): a block asks for its
// part of the factors, which no phase writes, and only then waits for the
// phase before.
enum { PH_GATHER, PH_FWD_A, PH_FWD_B, PH_FWD_U, PH_BWD_R, PH_BWD_S, PH_BWD_A, PH_BWD_B };
template <typename T, int NR, int TRANS, int PH>
__global__ void __launch_bounds__(SW_T) k_sweep(const Sweep<T> S, int j0) {
  __shared__ SweepSmem<T, NR> sm;
  cudaTriggerProgrammaticLaunchCompletion();
  Front<T, NR, TRANS, sizeof(T) == 8> F(S, S.list[blockIdx.y], sm);
  const int ch = blockIdx.x, r0 = ch * SW_CHUNK;
  const int nb = min(SB, F.k - j0), j1 = j0 + nb;
  const bool on = PH == PH_GATHER || PH == PH_BWD_S ? true
                  : j0 >= F.k                       ? false
                  : PH == PH_FWD_B                  ? ch < F.fwd_b_chunks(j0)
                  : PH == PH_FWD_U                  ? ch < F.fwd_u_chunks()
                  : PH == PH_BWD_R                  ? ch < F.bwd_r_chunks()
                  : PH == PH_BWD_B                  ? ch < F.bwd_b_chunks(j0)
                                                    : true;
  if (on) {
    if (PH == PH_FWD_A || PH == PH_BWD_A) {
      // the triangle: the lower (L) or upper (U) half of each of its columns
      const bool lower = (TRANS != 0) == (PH == PH_BWD_A);
      for (int c = threadIdx.x; c < nb; c += SW_T) {
        const T *D = F.P + j0 + (long long)(j0 + c) * F.m;
        for (int i = lower ? c & ~15 : 0; i < (lower ? nb : c + 1); i += 128 / (int)sizeof(T))
          asm volatile("prefetch.global.L2 [%0];" ::"l"(D + i));
      }
    }
    const int n0 = min(SW_CHUNK, (TRANS ? (PH == PH_FWD_U ? F.r : PH == PH_FWD_B ? F.k - j1 : j0)
                                        : (PH == PH_FWD_B ? F.m - j1 : j0)) - r0);
    if (PH == PH_FWD_B) {
      if (TRANS) F.ahead(F.P + j0 + (long long)(j1 + r0) * F.m, F.m, nb, n0);
      else F.ahead(F.P + j1 + r0 + (long long)j0 * F.m, F.m, n0, nb);
    }
    if (PH == PH_BWD_B) {
      if (TRANS) F.ahead(F.P + j0 + (long long)r0 * F.m, F.m, nb, n0);
      else F.ahead(F.P + r0 + (long long)j0 * F.m, F.m, n0, nb);
    }
  }
  cudaGridDependencySynchronize();
  if (PH == PH_GATHER) F.gather(ch * SW_T + threadIdx.x, gridDim.x * SW_T);
  if (PH == PH_BWD_S) F.bwd_s(ch * SW_T + threadIdx.x, j0);  // j0: the number of parts
  if (!on) return;
  if (PH == PH_FWD_A) F.fwd_a(j0);
  if (PH == PH_FWD_B) F.fwd_b(j0, ch);
  if (PH == PH_FWD_U) F.fwd_u(ch);
  if (PH == PH_BWD_R) F.bwd_r(ch, blockIdx.z, gridDim.z);
  if (PH == PH_BWD_A) F.bwd_a(j0);
  if (PH == PH_BWD_B) F.bwd_b(j0, ch);
}

// The same for the two phases of a step of few fronts in complex64, where a
// block can hold its part of the factors: all of it is on chip before the phase before is
// waited for, and what is left is arithmetic and the vectors' latency.
//
// k_sweep_tri: a step's triangle, a block a front.  The 28 off-diagonal 32 x 32
// blocks in shared memory (224 kB of the 227 an SM has), every warp's own
// triangle in its registers.  Warp s substitutes through it, and hands its 32
// results to the warps after it over a barrier of its own, so that no warp waits
// for one that is behind it.  The results lie where the warp's last used block was.
// Sweep pair of a 524k-row line grating's root front (17 steps, triangle and
// columns): 0.64 ms with the links loaded a link ahead and a block-wide barrier
// each, 0.32 ms so.
constexpr int TRI_TILE = 32 * 32;
constexpr size_t TRI_SMEM = (size_t)(28 * TRI_TILE + 64) * sizeof(cuComplex);
__device__ __forceinline__ int tri_tile(int a, int b) {
  const int hi = max(a, b), lo = min(a, b);
  return (hi * (hi - 1) / 2 + lo) * TRI_TILE;
}
__device__ __forceinline__ void tri_copy(cuComplex *dst, const cuComplex *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
template <int NR, int TRANS, int BWD>
__global__ void __launch_bounds__(SW_T, 1) k_sweep_tri(const Sweep<cuComplex> S, int j0) {
  using T = cuComplex;
  extern __shared__ __align__(16) unsigned char tri_raw[];
  T *tiles = reinterpret_cast<T *>(tri_raw);
  cudaTriggerProgrammaticLaunchCompletion();
  const NodeDev N = S.nodes[S.list[blockIdx.y]];
  const int k = N.k, m = N.m, t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int nb = min(SB, k - j0), links = (nb + 31) / 32;
  const bool on = nb > 0;
  const T *D = S.fac + N.fac_off + j0 + (long long)j0 * m;
  constexpr bool UNIT = TRANS == BWD;   // L; U's pivots come as reciprocals
  T own[32], rd = CT<T>::mk(1.0, 0.0);
  if (on) {
    // block (w2, s2): rows (TRANS: columns) of warp w2 against link s2, four of
    // its lines a warp; lanes along the contiguous rows of D, so that transposed
    // blocks are swizzled
    T *dst = tiles;
    for (int hi = 1; hi < links; ++hi)
      for (int lo = 0; lo < hi; ++lo, dst += TRI_TILE) {
        const int w2 = BWD ? lo : hi, s2 = BWD ? hi : lo;
        // row and column of D of this lane's entry of line w
        const int row = 32 * (TRANS ? s2 : w2) + lane, col = 32 * (TRANS ? w2 : s2) + w;
        const T *src = D + row + (long long)col * m;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int i = w + 8 * u;
          T *to = dst + (TRANS ? lane * 32 + (i ^ lane) : i * 32 + lane);
          if (row < nb && col + 8 * u < nb) tri_copy(to, src + (long long)(8 * u) * m);
          else *to = czero<T>();
        }
      }
#pragma unroll
    for (int l = 0; l < 32; ++l) {
      const int o = 32 * w + l;
      const bool in = BWD ? l > lane : l < lane;
      own[l] = in && t < nb && o < nb ? D[TRANS ? o + (long long)t * m : t + (long long)o * m] : czero<T>();
    }
    if (!UNIT && t < nb) rd = D[t + (long long)t * m];
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
  }
  cudaGridDependencySynchronize();
  if (!on || w >= links) return;
  T v[NR];
#pragma unroll
  for (int q = 0; q < NR; ++q)
    v[q] = t >= nb ? czero<T>()
           : BWD   ? S.Y[N.p0 + j0 + t + (long long)q * S.nn]
                   : S.V[N.vec_off + j0 + t + q * S.VR];
  // the results of link s: 32 NR entries
  auto slot = [&](int s) {
    const int first = BWD ? links - 1 : 0;
    return s == first ? tiles + 28 * TRI_TILE : tiles + tri_tile(s, BWD ? s + 1 : s - 1);
  };
  const int before = BWD ? links - 1 - w : w;   // links this warp takes results from
  for (int u = 0; u < before; ++u) {
    const int s = BWD ? links - 1 - u : u;
    asm volatile("bar.sync %0, %1;" ::"r"(1 + s), "r"(32 * (links - u)) : "memory");
    const T *y = slot(s), *c = tiles + tri_tile(w, s);
    T o[NR];
#pragma unroll
    for (int q = 0; q < NR; ++q) o[q] = czero<T>();
#pragma unroll
    for (int l = 0; l < 32; ++l) {
      const T a = c[l * 32 + (TRANS ? lane ^ l : lane)];
#pragma unroll
      for (int q = 0; q < NR; ++q) cfma(o[q], a, y[l * NR + q]);
    }
#pragma unroll
    for (int q = 0; q < NR; ++q) v[q] = csub(v[q], o[q]);
  }
  {
    T *y = slot(w);
    if (!UNIT && BWD)
#pragma unroll
      for (int q = 0; q < NR; ++q) v[q] = cmul(v[q], rd);
    unit_solve<T, NR, BWD, 32>(own, 0, v);
    __syncwarp();   // every lane has read the slot as a block
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      if (!UNIT && !BWD) v[q] = cmul(v[q], rd);
      y[lane * NR + q] = v[q];
    }
    if (before + 1 < links)
      asm volatile("bar.arrive %0, %1;" ::"r"(1 + w), "r"(32 * (links - before)) : "memory");
  }
  if (t >= nb) return;
  if (!BWD) {
#pragma unroll
    for (int q = 0; q < NR; ++q) S.Y[N.p0 + j0 + t + (long long)q * S.nn] = v[q];
    return;
  }
  const int g = S.perm[N.p0 + (TRANS ? S.pperm[N.p0 + j0 + t] : j0 + t)];
#pragma unroll
  for (int q = 0; q < NR; ++q) {
    S.V[N.vec_off + j0 + t + q * S.VR] = v[q];
    S.x[(long long)q * S.n + g] = v[q];
  }
}

// k_sweep_apply: a step's columns on SW_CHUNK rows (A^T: columns) outside its
// triangle, 32 entries a thread in registers
template <int NR, int TRANS, int BWD>
__global__ void __launch_bounds__(SW_T) k_sweep_apply(const Sweep<cuComplex> S, int j0) {
  using T = cuComplex;
  __shared__ SweepSmem<T, NR> sm;
  cudaTriggerProgrammaticLaunchCompletion();
  const NodeDev N = S.nodes[S.list[blockIdx.y]];
  const int k = N.k, m = N.m, t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int nb = min(SB, k - j0), j1 = j0 + nb;
  // the rows (columns) of the pivot block's step it applies to: [r0, r1)
  const int r0 = (BWD ? 0 : j1) + (int)blockIdx.x * SW_CHUNK, r1 = BWD ? j0 : TRANS ? k : m;
  const bool on = nb > 0 && r0 < r1;
  const T *P = S.fac + N.fac_off;
  T a[32];
  if (on) {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      // rows: column w + 8 i of the step; columns: column w + 8 (i / 8) of the
      // chunk, rows lane + 32 (i % 8) of the step
      const int o = TRANS ? lane + 32 * (i & 7) : w + SW_W * i;
      const int r = min(r0 + (TRANS ? w + SW_W * (i >> 3) : lane), r1 - 1);
      a[i] = o < nb ? P[TRANS ? j0 + o + (long long)r * m : r + (long long)(j0 + o) * m] : czero<T>();
    }
  }
  cudaGridDependencySynchronize();
  if (!on) return;
  T *const out = BWD ? S.Y + N.p0 : S.V + N.vec_off;
  const long long so = BWD ? S.nn : S.VR;
  // the entry this thread writes, and the step's vector
  const int mine = r0 + (TRANS ? w + SW_W * lane : t);
  const bool writes = (TRANS ? lane < SW_CHUNK / SW_W : t < SW_CHUNK) && mine < r1;
  T old[NR];
#pragma unroll
  for (int q = 0; q < NR; ++q) {
    old[q] = writes ? out[mine + q * so] : czero<T>();
    sm.in[t * NR + q] = t >= nb ? czero<T>()
                        : BWD   ? S.V[N.vec_off + j0 + t + q * S.VR]
                                : S.Y[N.p0 + j0 + t + (long long)q * S.nn];
  }
  __syncthreads();
  if (TRANS) {
    T acc[4][NR];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        acc[u][q] = czero<T>();
#pragma unroll
        for (int i = 0; i < 8; ++i) cfma(acc[u][q], a[8 * u + i], sm.in[(lane + 32 * i) * NR + q]);
        for (int x = 16; x; x >>= 1) {
          acc[u][q].x += __shfl_xor_sync(0xffffffffu, acc[u][q].x, x);
          acc[u][q].y += __shfl_xor_sync(0xffffffffu, acc[u][q].y, x);
        }
      }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (lane == u && writes)
#pragma unroll
        for (int q = 0; q < NR; ++q) out[mine + q * so] = csub(old[q], acc[u][q]);
  } else {
    T acc[NR];
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      acc[q] = czero<T>();
#pragma unroll
      for (int i = 0; i < 32; ++i) cfma(acc[q], a[i], sm.in[(w + SW_W * i) * NR + q]);
      sm.red[(w * SW_CHUNK + lane) * NR + q] = acc[q];
    }
    __syncthreads();
    if (writes)
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        T v = sm.red[lane * NR + q];
#pragma unroll
        for (int u = 1; u < SW_W; ++u) v = cadd(v, sm.red[(u * SW_CHUNK + lane) * NR + q]);
        out[mine + q * so] = csub(old[q], v);
      }
  }
}

// The 32 x 32 blocks on the diagonals of U11 of a depth's fronts, in place: rows
// divided by their pivots, the pivots as reciprocals; a warp per (front, block),
// a lane a row.
constexpr int DIAG_WARPS = 4;
struct DiagItem { int node, j0; };
template <typename T>
__global__ void __launch_bounds__(DIAG_WARPS * 32)
k_diag_scale(int cnt, const DiagItem *__restrict__ items, const NodeDev *__restrict__ nodes,
             T *arena) {
  const int lane = threadIdx.x & 31, i0 = blockIdx.x * DIAG_WARPS + (threadIdx.x >> 5);
  if (i0 >= cnt) return;
  const DiagItem it = items[i0];
  const NodeDev N = nodes[it.node];
  const int n = min(32, N.k - it.j0);
  if (lane >= n) return;
  T *D = arena + N.arena_off + it.j0 + (long long)it.j0 * N.ld + lane;
  const T rd = lu_rcp(D[(long long)lane * N.ld]);
#pragma unroll 8
  for (int c = 0; c < n; ++c) {
    T &d = D[(long long)c * N.ld];
    if (c >= lane) d = c == lane ? rd : cmul(d, rd);
  }
}

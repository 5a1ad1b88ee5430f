// Triangular solves of the update blocks, included by lfsolve.cu inside its
// namespace after lfsolve_sweeps.cuh: U12 = L11^-1 P F12 and L21 = F21 U11^-1
// of a group of fronts of the same (padded) shape.
//
// The pivots are taken in leaves of 64.  A leaf's triangle is applied here by
// substitution, eight pivots at a time (leaf_triangle; U's 32 x 32 diagonal
// blocks come as unit triangles and reciprocal pivots, k_diag_scale), and what a
// solved range of leaves contributes to the next one is
// a matrix product, binary: after leaf i, with 2^t the power of two in i, the
// last 2^t leaves update the next 2^t.  So all but k x 64 of the work is in
// products at least 64 deep, half of it in products of half the pivots.
//
// In complex64 those products run on TF32 tensor cores in split form (below);
// the leaf kernel writes its results in that form as it stores them, so that
// the Schur update reads the same operands.
//
// Error-compensated TF32 operands of a complex64 product L U (real
// formulation): the complex product is the real product of A (2 rows x 2
// columns of L; column 2 j is column j of L read as (re, im) float pairs,
// column 2 j + 1 that of i L) and B (U read as (re, im) pairs), and the real
// result read as floats is the complex result.  Every float x is split as hi =
// its TF32 rounding (cvt.rna.tf32.f32, 10 mantissa bits) and lo = x - hi, and
// hi hi' + hi lo' + lo hi' carries the product to about 2^-22 relative.  Per
// leaf of kb pivots A holds [hi | lo] (4 kb columns) and B [lo ; hi] (4 kb
// rows), so that one real product over any range of leaves gives the two small
// terms; hi is stored once more by itself for the large one.  The two stay
// apart because the tensor cores truncate as they accumulate: all three terms
// in one product of depth 6 k left residuals twice as large (1.7e-3 against
// 0.9e-3 unrefined on a 111k-row contact hole).
constexpr int LEAF = 64;
constexpr int LEAF_T = 128;
constexpr int SPLIT_T = 256;
// columns of F12 (rows of F21) a block takes: three (complex128: two) blocks a SM
template <typename T> constexpr int LEAF_C = sizeof(T) == 8 ? 64 : 32;

// a group of cnt fronts: front f at F + f S, kk pivot rows (dummies included),
// r update rows (padding included), leading dimension ld; split operands (null
// where the products run in T): AF of L11, BF of U11, AL of L21, BU of U12,
// each the cnt fronts' [hi | lo] parts, then their hi parts
struct Operand {
  float *p;           // null: none
  long long ld, n;    // leading dimension of a left operand (of a right one: 4 kk and 2 kk); entries
  __host__ __device__ float *both(int f) const { return p + f * 4 * n; }
  __host__ __device__ float *hi(int cnt, int f) const { return p + (cnt * 4 + f * 2LL) * n; }
};
template <typename T> struct Group {
  T *F;
  long long S;
  int cnt, kk, r, ld;
  Operand AF, BF, AL, BU;
};

__device__ __forceinline__ float tf32_round(float x) {
  unsigned u;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(u) : "f"(x));
  return __uint_as_float(u);
}
__device__ __forceinline__ void tf32_split(cuComplex v, float2 &h, float2 &l) {
  h = make_float2(tf32_round(v.x), tf32_round(v.y));
  l = make_float2(v.x - h.x, v.y - h.y);
}
// entry (row i, pivot l of a leaf of kb pivots starting at pivot p0) of a left operand
__device__ __forceinline__ void put_left(const Operand &A, int cnt, int f, int p0, int kb, int i, int l,
                                         cuComplex v) {
  float2 h, e;
  tf32_split(v, h, e);
  float *c = A.both(f) + (4LL * p0 + 2 * l) * A.ld + 2 * i;
  *reinterpret_cast<float2 *>(c) = h;
  *reinterpret_cast<float2 *>(c + A.ld) = make_float2(-h.y, h.x);
  c += 2LL * kb * A.ld;
  *reinterpret_cast<float2 *>(c) = e;
  *reinterpret_cast<float2 *>(c + A.ld) = make_float2(-e.y, e.x);
  c = A.hi(cnt, f) + 2LL * (p0 + l) * A.ld + 2 * i;
  *reinterpret_cast<float2 *>(c) = h;
  *reinterpret_cast<float2 *>(c + A.ld) = make_float2(-h.y, h.x);
}
// entry (pivot l, column c) of a right operand
__device__ __forceinline__ void put_right(const Operand &B, int cnt, int f, int kk, int p0, int kb,
                                          int l, long long c, cuComplex v) {
  float2 h, e;
  tf32_split(v, h, e);
  float *r = B.both(f) + 4LL * p0 + 2 * l + c * 4 * kk;
  *reinterpret_cast<float2 *>(r) = e;
  *reinterpret_cast<float2 *>(r + 2 * kb) = h;
  *reinterpret_cast<float2 *>(B.hi(cnt, f) + 2LL * (p0 + l) + c * 2 * kk) = h;
}
__device__ __forceinline__ void put_left(const Operand &, int, int, int, int, int, int, cuDoubleComplex) {}
__device__ __forceinline__ void put_right(const Operand &, int, int, int, int, int, int, long long,
                                          cuDoubleComplex) {}

// split operands of L11 (below its leaves) and U11 (right of them): block =
// (leaf, 64 rows or columns further on), front blockIdx.z
template <typename T>
__global__ void __launch_bounds__(SPLIT_T) k_split_f11(const Group<T> G) {
  const int p0 = blockIdx.x * LEAF, q0 = (blockIdx.x + 1 + blockIdx.y) * LEAF;
  if (q0 >= G.kk) return;
  const int qn = min(LEAF, G.kk - q0);  // a leaf with others after it is full
  const T *F = G.F + blockIdx.z * G.S;
  const int f = blockIdx.z;
  for (int t = threadIdx.x; t < LEAF * LEAF; t += SPLIT_T) {
    const int i = t % LEAF, l = t / LEAF;
    if (i < qn)
      put_left(G.AF, G.cnt, f, p0, LEAF, q0 + i, l, F[q0 + i + (long long)(p0 + l) * G.ld]);
    if (l < qn)
      put_right(G.BF, G.cnt, f, G.kk, p0, LEAF, i, q0 + l, F[p0 + i + (long long)(q0 + l) * G.ld]);
  }
}

template <typename T> struct LeafSmem {
  T D[LEAF][LEAF + 1];          // the leaf's triangle, zero beyond
  T X[LEAF][LEAF_C<T> + 1];     // pivots x columns (left) or pivots x rows (right)
};

// rows [o0 + 8 q0, o0 + 32) of X -= sum over l in [l0, l0 + n) of coef(o, l) X[l],
// the sums formed by themselves, a thread per 4 pivots x LEAF_C / 16 columns
template <typename T, class C>
__device__ __forceinline__ void leaf_update(LeafSmem<T> &sm, int o0, int q0, int l0, int n, C coef) {
  constexpr int NB = LEAF_C<T> / 16;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  T acc[4][NB];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < NB; ++b) acc[a][b] = czero<T>();
#pragma unroll 2
  for (int l = l0; l < l0 + n; ++l) {
    T d[4], x[NB];
#pragma unroll
    for (int a = q0; a < 4; ++a) d[a] = coef(o0 + ty + 8 * a, l);
#pragma unroll
    for (int b = 0; b < NB; ++b) x[b] = sm.X[l][tx + 16 * b];
#pragma unroll
    for (int a = q0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < NB; ++b) acc[a][b] = cfms(acc[a][b], d[a], x[b]);
  }
#pragma unroll
  for (int a = q0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      T &x = sm.X[o0 + ty + 8 * a][tx + 16 * b];
      x = cadd(x, acc[a][b]);
    }
  __syncthreads();
}

// A unit triangle of 32 pivots from o0 on: eight pivots of a column by a thread,
// then their part of the rows left.  SCALE: the results times the reciprocal
// pivots at the end, eight rows at a time by the threads without a column.
template <typename T, bool SCALE, class C>
__device__ __forceinline__ void leaf_triangle(LeafSmem<T> &sm, int o0, C coef) {
  constexpr int NC = LEAF_C<T>;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int l0 = o0 + 8 * q;
    if (threadIdx.x < NC) {
      T x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = sm.X[l0 + i][threadIdx.x];
#pragma unroll
      for (int i = 0; i < 7; ++i)
#pragma unroll
        for (int j = i + 1; j < 8; ++j) x[j] = cfms(x[j], coef(l0 + j, l0 + i), x[i]);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        sm.X[l0 + i][threadIdx.x] = SCALE && q == 3 ? cmul(x[i], sm.D[l0 + i][l0 + i]) : x[i];
    } else if (SCALE && q > 0) {
      for (int t = threadIdx.x - NC; t < 8 * NC; t += LEAF_T - NC) {
        const int l = l0 - 8 + t / NC;
        sm.X[l][t % NC] = cmul(sm.X[l][t % NC], sm.D[l][l]);
      }
    }
    __syncthreads();
    if (q < 3) leaf_update<T>(sm, o0, q + 1, l0, 8, coef);
  }
}

template <typename T, bool LEFT>
__device__ __forceinline__ void leaf_side(const Group<T> &G, int p0, LeafSmem<T> &sm) {
  constexpr int NC = LEAF_C<T>, B = 64 / sizeof(T);   // loads of a thread in flight
  const int kb = min(LEAF, G.kk - p0), c0 = blockIdx.x * NC, nc = min(NC, G.r - c0);
  T *F = G.F + blockIdx.y * G.S;
  const T *D = F + p0 + (long long)p0 * G.ld;
  // F12 rows p0 .., columns c0 ..; F21 rows c0 .., columns p0 ..
  T *X = LEFT ? F + p0 + (long long)(G.kk + c0) * G.ld : F + G.kk + c0 + (long long)p0 * G.ld;
  for (int t0 = threadIdx.x; t0 < LEAF * LEAF; t0 += B * LEAF_T) {
    T v[B];
#pragma unroll
    for (int u = 0; u < B; ++u) {
      const int t = t0 + u * LEAF_T, i = t % LEAF, l = t / LEAF;   // i along a column of memory
      v[u] = i < kb && l < kb && (LEFT ? i > l : i <= l) ? D[i + (long long)l * G.ld] : czero<T>();
    }
#pragma unroll
    for (int u = 0; u < B; ++u) {
      const int t = t0 + u * LEAF_T, i = t % LEAF, l = t / LEAF;
      sm.D[i][l] = v[u];
    }
  }
  constexpr int XI = LEFT ? LEAF : NC;   // entries along a column of memory
  for (int t0 = threadIdx.x; t0 < LEAF * NC; t0 += B * LEAF_T) {
    T v[B];
#pragma unroll
    for (int u = 0; u < B; ++u) {
      const int t = t0 + u * LEAF_T, i = t % XI, l = t / XI;
      v[u] = (LEFT ? i < kb && l < nc : l < kb && i < nc) ? X[i + (long long)l * G.ld] : czero<T>();
    }
#pragma unroll
    for (int u = 0; u < B; ++u) {
      const int t = t0 + u * LEAF_T, i = t % XI, l = t / XI;
      if (LEFT) sm.X[i][l] = v[u];
      else sm.X[l][i] = v[u];
    }
  }
  __syncthreads();
  // X = L^-1 X by halves: X_0 = L_00^-1 X_0; X_1 = L_11^-1 (X_1 - L_10 X_0);
  // for F21 the same with the transposed coefficients of U
  auto coef = [&](int o, int l) { return LEFT ? sm.D[o][l] : sm.D[l][o]; };
#pragma unroll 1
  for (int o0 = 0; o0 < kb; o0 += 32) {
    if (o0) leaf_update<T>(sm, 32, 0, 0, 32, coef);
    leaf_triangle<T, !LEFT>(sm, o0, coef);
  }
#pragma unroll 4
  for (int t = threadIdx.x; t < LEAF * NC; t += LEAF_T) {
    const int i = t % XI, l = t / XI;
    if (LEFT) {
      if (i >= kb || l >= nc) continue;
      const T v = sm.X[i][l];
      X[i + (long long)l * G.ld] = v;
      if (G.BU.p) put_right(G.BU, G.cnt, blockIdx.y, G.kk, p0, kb, i, c0 + l, v);
    } else {
      if (l >= kb || i >= nc) continue;
      const T v = sm.X[l][i];
      X[i + (long long)l * G.ld] = v;
      if (G.AL.p) put_left(G.AL, G.cnt, blockIdx.y, p0, kb, c0 + i, l, v);
    }
  }
}

// One leaf (pivots p0 .. p0 + kb) of every front of the group: F12
// (blockIdx.z = 0) and F21 in one launch, LEAF_C columns (rows) a block.
// Bound: FP32 (FP64) FMA issue and the stores of the split operands, about
// equal.  The substitution takes what products with the inverses of the 32 x 32
// blocks took (a factorization 235.3 and 234.6 ms in complex64 on a 524k-row line
// grating, 52.1 and 51.6 ms in complex128 on a 111k-row hole).
template <typename T>
__global__ void __launch_bounds__(LEAF_T, sizeof(T) == 8 ? 3 : 2) k_leaf(const Group<T> G, int p0) {
  extern __shared__ __align__(16) unsigned char leaf_raw[];
  LeafSmem<T> &sm = *reinterpret_cast<LeafSmem<T> *>(leaf_raw);
  if (blockIdx.z == 0) leaf_side<T, true>(G, p0, sm);
  else leaf_side<T, false>(G, p0, sm);
}

// The element loop y = (lapf K + massf M) x, by sibling families.
//
// A family is one parent octant with those of its 8 children that are
// leaves.  Its elements only ever refer to the 27 points of the 3x3x3
// lattice that the children's vertices form: a vertex that does not hang is
// a lattice point, and a hanging one refers to the parent's corner, the
// lattice corner of its child.  So a family is the unit of work of one
// thread: gather its lattice once, apply its elements in registers, add the
// lattice out once.  An octree has (E - 1) / 7 internal octants, so a family
// holds 7.4 elements on the workloads' meshes and touches 18 mesh nodes:
// 2.5 gathers and adds per element against 8 for an element-wise loop.
//
// Hanging points: an edge midpoint of the parent that hangs takes the mean of
// its edge's two corners, a face centre that hangs the mean of two opposite
// edge midpoints of its face (which then hang too), and the results at
// hanging points are passed back by the transpose.  That is the P^T S P of
// the reference's 18 element types, so the elements themselves are all the
// plain trilinear one, and no stencil table is read.
//
// Elements in floating point (cube_rows): the entries of the trilinear K are 0
// for vertices an odd number of steps apart but for the opposite one, and its rows
// sum to 0, so K x needs the differences within a vertex's class (the vertices an
// even number of steps away) and to its opposite only; M adds the classes' sums.
// 44 operations per element where a dense stencil takes 64 multiply-adds.  Every
// row is made of its own entries times x, as with the stencil, so a row among
// small values keeps its accuracy beside large ones; and of differences, so that
// smooth fields, on which the stencil's terms cancel, keep theirs.
//
// Elements in fixed point: K and M are tensor products, diagonal in a basis of
// sums and differences.  For the assembled 2x2x2 family, per axis
//   M = 1/4 s s^T + 1/3 o o^T + 1/12 q q^T,  A = 1/4 o o^T + 1/4 q q^T
// with s = (1,2,1), o = (1,0,-1), q = (1,-2,1); for one element
//   M = 1/2 s s^T + 1/6 d d^T,  A = 1/2 d d^T,  s = (1,1), d = (1,-1).
// So a complete family (3 of 4) costs 27 lines each way (4 and 5 operations a
// line, all coefficients 1 or 2) and 27 multiplications, which are what counts
// there; one with subdivided children is applied element by element.
//
// On 1.1e7 elements of a Gaussian cloud (GB300) FP32 takes 105 us and FP64
// vectors 344 us; what bounds them stands at the kernels.  An element-wise loop
// over dense stencils, 8 gathers and 8 atomics per element, took 348 and 1,820
// us.  128 families per patch: 64 and 256 measured 152 / 150 us where 128 took
// 143 (FP32); a patch of 256 leaves too few blocks on small meshes.
//
// Patches: FAM consecutive families (in element order) make a patch, one
// thread block's work at a time.  fam[(p * 4 + w) * FAM + t] is word w of the
// patch's family t: 27 x 16 bits, the patch-local number of the node at each
// lattice point (0: no node there), then 16 bits level and 8 bits mask of the
// children that are leaves, then 18 bits of hanging points.  Complete families
// come first, so that most warps hold one kind.  pinfo[p] = {offset of the
// patch's nodes in prun (64 bits), their number, unused}; prun holds the nodes,
// number 1 first, with two flags.
#pragma once

#include "dg_prims.cuh"

namespace dg {

constexpr int FAM = 128;                // families per patch, threads per block
constexpr int FAM_MAX_RUN = 27 * FAM;  // most nodes a patch can touch
constexpr uint32_t PRUN_COMPLETE = 1u << 31;  // no other patch touches the node: its sum is stored, not added
constexpr uint32_t PRUN_BDY = 1u << 30;       // the node lies on the domain boundary
constexpr uint32_t PRUN_NODE = PRUN_BDY - 1;

// lattice point of child c's vertex k
__host__ __device__ constexpr int lat_vertex(int c, int k) {
  return ((c & 1) + (k & 1)) + 3 * ((c >> 1 & 1) + (k >> 1 & 1)) + 9 * ((c >> 2 & 1) + (k >> 2 & 1));
}
// lattice point of the parent's corner k
__host__ __device__ constexpr int lat_corner(int k) { return 2 * (k & 1) + 6 * (k >> 1 & 1) + 18 * (k >> 2 & 1); }

// the 18 lattice points that can hang: edge midpoints (i = 0..11, along axis
// i / 4) with the two corners of their edge, face centres (i = 12..17, normal
// to axis (i - 12) / 2) with two opposite edge midpoints of their face
__host__ __device__ constexpr int lat_stride(int ax) { return ax % 3 == 0 ? 1 : ax % 3 == 1 ? 3 : 9; }
__host__ __device__ constexpr int hang_pos(int i) {
  return i < 12 ? lat_stride(i / 4) + 2 * (i & 1) * lat_stride(i / 4 + 1) + 2 * (i >> 1 & 1) * lat_stride(i / 4 + 2)
                : 2 * (i & 1) * lat_stride((i - 12) / 2) + lat_stride((i - 12) / 2 + 1) + lat_stride((i - 12) / 2 + 2);
}
__host__ __device__ constexpr int hang_step(int i) {
  return i < 12 ? lat_stride(i / 4) : lat_stride((i - 12) / 2 + 1);
}
__host__ __device__ constexpr int hang_a(int i) { return hang_pos(i) - hang_step(i); }
__host__ __device__ constexpr int hang_b(int i) { return hang_pos(i) + hang_step(i); }
__host__ __device__ constexpr int hang_bit(int pos) {
  for (int i = 0; i < 18; i++)
    if (hang_pos(i) == pos) return i;
  return -1;
}

// Diagonal of the operator in the sum / difference basis, per level: entry
// dfam(o, q) for a family mode with o factors o and q factors q, entry
// DCHILD + p for an element mode with p factors d.  Rows are padded so that
// neighbouring levels fall in different shared-memory banks.
constexpr int DTAB_CHILD = 10, DTAB_STRIDE = 15, DTAB_LEVELS = 31;
constexpr int DTAB_ENTRIES = DTAB_LEVELS * DTAB_STRIDE;
__host__ __device__ constexpr int dfam(int o, int q) { return o == 0 ? q : o == 1 ? 4 + q : o == 2 ? 7 + q : 9; }

// 2^-l exactly, from the exponent bits (0 <= l <= 30)
__device__ __forceinline__ float exp2_neg(float, unsigned l) { return __int_as_float((int)(127u - l) << 23); }
__device__ __forceinline__ double exp2_neg(double, unsigned l) {
  return __longlong_as_double((long long)(1023u - l) << 52);
}
__device__ __forceinline__ bool is_finite(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }
__device__ __forceinline__ bool is_finite(double v) {
  return ((uint32_t)__double2hiint(v) & 0x7ff00000u) != 0x7ff00000u;
}

// The trilinear element's operator lap K + mass M (scaled by h / 2 and h^3 / 8).
// With r one vertex of i's class, e = x - r within it, E the sum of those, D = x of
// i's opposite - x_i, and T the sum over the other class: row i is
//   within e_i + across D_i + cls E + other (T + 11/4 r).
template <typename T>
struct __align__(16) Cube {
  T within, across, cls, other;
};
template <typename T>
__device__ __forceinline__ Cube<T> cube_of(T lap, T mass) {
  return Cube<T>{lap * (T)(2.0 / 3.0) + mass * (T)(1.0 / 9.0), -lap * (T)(1.0 / 6.0) - mass * (T)(1.0 / 9.0),
                 -lap * (T)(1.0 / 6.0) + mass * (T)(2.0 / 27.0), mass * (T)(4.0 / 27.0)};
}
// the rows of one element, add(k, row) for vertex k; classes {0, 3, 5, 6} and
// their opposites {7, 4, 2, 1}
template <typename T, typename X, typename Add>
__device__ __forceinline__ void cube_rows(const Cube<T> &s, X &&x, Add &&add) {
  T e[2][4], c[2], sum[2];
#pragma unroll
  for (int p = 0; p < 2; p++) {
    const int o = 7 * p;
    const T r = x(o);
    e[p][1] = x(3 ^ o) - r;
    e[p][2] = x(5 ^ o) - r;
    e[p][3] = x(6 ^ o) - r;
    const T all = e[p][1] + e[p][2] + e[p][3];
    sum[p] = (T)4 * r + all;
    c[p] = s.cls * all + s.other * (T)2.75 * r;
  }
  c[0] += s.other * sum[1];
  c[1] += s.other * sum[0];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int k = j == 0 ? 0 : j == 1 ? 3 : j == 2 ? 5 : 6;
    const T d = s.across * (x(k ^ 7) - x(k));
    add(k, j == 0 ? d + c[0] : s.within * e[0][j] + (d + c[0]));
    add(k ^ 7, j == 0 ? c[1] - d : s.within * e[1][j] + (c[1] - d));
  }
}
// ... per level
template <typename T>
__global__ void k_cube_table(Cube<T> *__restrict__ out, double lapf, double massf) {
  const int l = threadIdx.x;
  if (l >= DTAB_LEVELS) return;
  const double h = ldexp(1.0, -l);
  const Cube<double> c = cube_of<double>(lapf * h * 0.5, massf * h * h * h * 0.125);
  out[l] = Cube<T>{(T)c.within, (T)c.across, (T)c.cls, (T)c.other};
}

// entry i of the table of modes, lap and mass scaled likewise
__device__ __forceinline__ double dtab_entry(int i, double lap, double mass) {
  double m[3], a[3];  // mode weights of the three axes
  if (i < DTAB_CHILD) {
    const int o = i < 4 ? 0 : i < 7 ? 1 : i < 9 ? 2 : 3;
    const int q = i - (i < 4 ? 0 : i < 7 ? 4 : i < 9 ? 7 : 9);
    for (int k = 0; k < 3; k++) {
      m[k] = k < o ? 1.0 / 3.0 : k < o + q ? 1.0 / 12.0 : 0.25;
      a[k] = k < o + q ? 0.25 : 0.0;
    }
  } else {
    for (int k = 0; k < 3; k++) {
      m[k] = k < i - DTAB_CHILD ? 1.0 / 6.0 : 0.5;
      a[k] = k < i - DTAB_CHILD ? 0.5 : 0.0;
    }
  }
  return lap * (a[0] * m[1] * m[2] + m[0] * a[1] * m[2] + m[0] * m[1] * a[2]) + mass * (m[0] * m[1] * m[2]);
}

// The table of modes for 64-bit fixed point, a row per level: entry i times
// 2^(63 - k), split into its upper bits and its 30 lowest, with 2^k the power
// of two not below the level's |lap| + |mass| (so that |entry| <= 2^(k - 3));
// k in the row's last place, FIX_NONE where it leaves the range that the element
// loop's exponents have room for.
constexpr int FIX_K = DTAB_STRIDE - 1, FIX_K_MAX = 400, FIX_NONE = 0x7fffffff;
static_assert(DTAB_CHILD + 4 <= FIX_K, "a place for the exponent");
static __global__ void k_fix_table(int2 *__restrict__ out, double lapf, double massf) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= DTAB_ENTRIES) return;
  const double h = ldexp(1.0, -(i / DTAB_STRIDE)), lap = lapf * h * 0.5, mass = massf * h * h * h * 0.125;
  const double most = fabs(lap) + fabs(mass);
  int k = 0;
  if (most > 0.0 && frexp(most, &k) == 0.5) k--;
  const bool ok = is_finite(most) && k >= -FIX_K_MAX && k <= FIX_K_MAX && (most > 0.0 || (lapf == 0.0 && massf == 0.0));
  const int q = i % DTAB_STRIDE;
  int2 e = make_int2(0, 0);
  if (q == FIX_K) e.x = ok ? k : FIX_NONE;
  else if (ok) {
    const long long f = __double2ll_rn(ldexp(dtab_entry(q, lap, mass), 63 - k));
    e = make_int2((int)(f & ((1 << 30) - 1)), (int)(f >> 30));
  }
  out[i] = e;
}

// arithmetic of one lattice value: FP32, FP64 or 64-bit fixed point
template <typename V>
struct LatOps {
  static __device__ __forceinline__ V half_add(V v, V half_of) { return v + (V)0.5 * half_of; }
  static __device__ __forceinline__ V mean(V a, V b) { return (V)0.5 * a + (V)0.5 * b; }  // no overflow
};
template <>
struct LatOps<long long> {
  static __device__ __forceinline__ long long half_add(long long v, long long half_of) { return v + (half_of >> 1); }
  static __device__ __forceinline__ long long mean(long long a, long long b) { return (a + b) >> 1; }
};

// values at hanging points from the points they depend on
template <typename V>
__device__ __forceinline__ void lat_interpolate(V (&u)[27], uint32_t hang) {
#pragma unroll
  for (int i = 0; i < 18; i++)
    if (hang >> i & 1u) u[hang_pos(i)] = LatOps<V>::mean(u[hang_a(i)], u[hang_b(i)]);
}
// the transpose: results at hanging points passed back (faces first)
template <typename V>
__device__ __forceinline__ void lat_distribute(V (&v)[27], uint32_t hang) {
#pragma unroll
  for (int i = 17; i >= 0; i--)
    if (hang >> i & 1u) {
      v[hang_a(i)] = LatOps<V>::half_add(v[hang_a(i)], v[hang_pos(i)]);
      v[hang_b(i)] = LatOps<V>::half_add(v[hang_b(i)], v[hang_pos(i)]);
    }
}

// any family in floating point, v = sum over its elements of S u; coef(c): child
// c's operator.  A child that is not there gets no value, and a value that is not
// finite reaches the rows of its elements only.
__host__ __device__ constexpr bool odd_vertex(int k) { return ((k ^ k >> 1 ^ k >> 2) & 1) != 0; }
template <typename T, typename Coef>
__device__ __forceinline__ void lat_cubes(const T (&u)[27], T (&v)[27], uint32_t mask, Coef &&coef) {
#pragma unroll
  for (int i = 0; i < 27; i++) v[i] = (T)0;
#pragma unroll
  for (int c = 0; c < 8; c++)
    if (mask >> c & 1u)
      cube_rows<T>(coef(c), [&](int k) { return u[lat_vertex(c, k)]; }, [&](int k, T row) { v[lat_vertex(c, k)] += row; });
}

// a complete family: to the sum / difference basis and back, in place
__device__ __forceinline__ void lat_forward(long long (&u)[27]) {
#pragma unroll
  for (int ax = 0; ax < 3; ax++) {
    const int st = ax == 0 ? 1 : ax == 1 ? 3 : 9;
#pragma unroll
    for (int n = 0; n < 9; n++) {
      const int i = ax == 0 ? 3 * n : ax == 1 ? n % 3 + 9 * (n / 3) : n;
      const long long e = u[i] + u[i + 2 * st], o = u[i] - u[i + 2 * st], b = u[i + st];
      u[i] = e + 2 * b;
      u[i + st] = o;
      u[i + 2 * st] = e - 2 * b;
    }
  }
}
__device__ __forceinline__ void lat_backward(long long (&u)[27]) {
#pragma unroll
  for (int ax = 0; ax < 3; ax++) {
    const int st = ax == 0 ? 1 : ax == 1 ? 3 : 9;
#pragma unroll
    for (int n = 0; n < 9; n++) {
      const int i = ax == 0 ? 3 * n : ax == 1 ? n % 3 + 9 * (n / 3) : n;
      const long long t = u[i] + u[i + 2 * st], r = u[i] - u[i + 2 * st], o = u[i + st];
      u[i] = t + o;
      u[i + st] = r + r;
      u[i + 2 * st] = t - o;
    }
  }
}
// the modes times their table entries; mul(t, i): t times entry i
template <typename Mul>
__device__ __forceinline__ void lat_scale(long long (&u)[27], Mul &&mul) {
#pragma unroll
  for (int i = 0; i < 27; i++) {
    const int x = i % 3, y = i / 3 % 3, z = i / 9;
    u[i] = mul(u[i], dfam((x == 1) + (y == 1) + (z == 1), (x == 2) + (y == 2) + (z == 2)));
  }
}

// any family, v = sum over its elements of S u, element by element in the
// basis of one element, the sums and differences of shared edges and faces
// formed once: 148 operations in, 64 multiplications, 185 out for 8 elements
// (333 for each on its own: 512).  mul(t, p): t times the entry for p factors d.
// A child that is not there gets no value.
template <typename Mul>
__device__ __forceinline__ void lat_elements(const long long (&u)[27], long long (&v)[27], uint32_t mask, Mul &&mul) {
  typedef long long V;
#pragma unroll
  for (int cx = 0; cx < 2; cx++) {
    V a[2][9], sum_x[2][9];  // [factor along x][y + 3 z]
#pragma unroll
    for (int i = 0; i < 9; i++) {
      a[0][i] = u[3 * i + cx] + u[3 * i + cx + 1];
      a[1][i] = u[3 * i + cx] - u[3 * i + cx + 1];
    }
#pragma unroll
    for (int cy = 0; cy < 2; cy++) {
      V b[4][3], sum_y[4][3];  // [factors along x, y][z]
#pragma unroll
      for (int z = 0; z < 3; z++)
#pragma unroll
        for (int m = 0; m < 2; m++) {
          b[m][z] = a[m][3 * z + cy] + a[m][3 * z + cy + 1];
          b[m + 2][z] = a[m][3 * z + cy] - a[m][3 * z + cy + 1];
        }
#pragma unroll
      for (int cz = 0; cz < 2; cz++) {
        const int c = cx + 2 * cy + 4 * cz;
        const bool there = mask >> c & 1u;
#pragma unroll
        for (int m = 0; m < 4; m++) {
          const int p = (m & 1) + (m >> 1);
          V s = mul(b[m][cz] + b[m][cz + 1], p), d = mul(b[m][cz] - b[m][cz + 1], p + 1);
          s = there ? s : (V)0;
          d = there ? d : (V)0;
          sum_y[m][cz] = cz == 0 ? s + d : sum_y[m][cz] + (s + d);
          sum_y[m][cz + 1] = s - d;
        }
      }
#pragma unroll
      for (int z = 0; z < 3; z++)
#pragma unroll
        for (int m = 0; m < 2; m++) {
          const V s = sum_y[m][z], d = sum_y[m + 2][z];
          sum_x[m][3 * z + cy] = cy == 0 ? s + d : sum_x[m][3 * z + cy] + (s + d);
          sum_x[m][3 * z + cy + 1] = s - d;
        }
    }
#pragma unroll
    for (int i = 0; i < 9; i++) {
      const V s = sum_x[0][i], d = sum_x[1][i];
      v[3 * i + cx] = cx == 0 ? s + d : v[3 * i + cx] + (s + d);
      v[3 * i + cx + 1] = s - d;
    }
  }
}

// the 16-bit number i of a family's four words
__device__ __forceinline__ uint32_t fam_u16(const uint4 (&w)[4], int i) {
  const uint4 q = w[i >> 3];
  const uint32_t word = (i >> 1 & 3) == 0 ? q.x : (i >> 1 & 3) == 1 ? q.y : (i >> 1 & 3) == 2 ? q.z : q.w;
  return (i & 1) ? word >> 16 : word & 0xffffu;
}
__device__ __forceinline__ uint32_t fam_level(const uint4 (&w)[4]) { return fam_u16(w, 27) & 31u; }
__device__ __forceinline__ uint32_t fam_mask(const uint4 (&w)[4]) { return fam_u16(w, 28) & 255u; }
__device__ __forceinline__ uint32_t fam_hang(const uint4 (&w)[4]) {
  return fam_u16(w, 29) | fam_u16(w, 30) << 16;
}

// Family f in floating point: its lattice from xs, its elements in registers,
// its lattice added into ys with shared-memory atomics.  COEF: element e's
// factors are coef[2e] (Laplacian) and coef[2e + 1] (mass) instead of the
// table's; fchild[8 f + c] gives e.  Differences and sums of the values may pass
// the end of the range where the rows do not: where the results are not all
// finite, nothing is added and the caller tries again with values scaled down (by a
// power of two below 1).
template <typename T, bool COEF>
__device__ __forceinline__ bool family_floating(const uint4 (&w)[4], size_t f, const T *xs, T *ys, const Cube<T> *tab,
                                                const double *__restrict__ coef,
                                                const uint32_t *__restrict__ fchild, T scale = (T)1) {
  const uint32_t hang = fam_hang(w);
  T u[27], v[27];
#pragma unroll
  for (int i = 0; i < 27; i++) u[i] = xs[fam_u16(w, i)] * scale;
  lat_interpolate(u, hang);
  Cube<T> s;
  if constexpr (!COEF) s = tab[fam_level(w)];
  lat_cubes(u, v, fam_mask(w), [&](int c) {
    if constexpr (COEF) {
      const size_t e = fchild[8 * f + c];
      const T h = exp2_neg((T)0, fam_level(w));
      s = cube_of<T>((T)coef[2 * e] * h * (T)0.5, (T)coef[2 * e + 1] * h * h * h * (T)0.125);
    }
    return s;
  });
  lat_distribute(v, hang);
  if (scale == (T)1) {
    T all = (T)0;
#pragma unroll
    for (int i = 0; i < 27; i++) all += v[i];
    if (!is_finite(all)) return false;
  }
  const T back = (T)1 / scale;
#pragma unroll
  for (int i = 0; i < 27; i++) {
    const uint32_t n = fam_u16(w, i);
    if (n) atomicAdd(&ys[n], v[i] * back);
  }
  return true;
}
// ... out of line, fw: the family's words
template <typename T, bool COEF>
__device__ __noinline__ void family_scaled(const uint4 *__restrict__ fw, size_t f, const T *xs, T *ys,
                                           const Cube<T> *tab, const double *__restrict__ coef,
                                           const uint32_t *__restrict__ fchild) {
  uint4 w[4];
#pragma unroll
  for (int q = 0; q < 4; q++) w[q] = fw[q * FAM];
  family_floating<T, COEF>(w, f, xs, ys, tab, coef, fchild, (T)0.0625);
}

// FP32: one block per patch, grid-strided, the next patch's x on its way while
// this one is applied.  Per patch, two barriers:
//   1. wait for x of this patch's nodes (and the words of the next one's), then
//      start copying the next one's x into the other buffer (cp.async; boundary
//      columns of the Dirichlet form are filled with zeros);
//   2. thread t = family t: its lattice from xs, its elements in registers,
//      its lattice added into ys with shared-memory atomics;
//   3. each node's sum stored (nodes of this patch alone) or added to y, and ys
//      left zero; the first 8 words per thread are loaded before the barrier.
// DIR, the Dirichlet form: boundary rows are the identity (y = x), boundary
// columns are dropped.
//
// 1.1e7 elements: 105 us; with the elements in the basis of sums and differences
// 109 us, and in that form with x gathered after each barrier 142 us (warps waited
// 6.6 of 15.2 cycles per instruction for it), with the copies but the words of step
// 3 loaded in step 3 118 us.  With sums of the classes in place of differences 96
// us, but on 9e7 elements a CG with this operator, which takes 7 iterations to
// 1e-8, then stops gaining at 1e-5.  The shared-memory and load/store
// pipe is two thirds busy; DRAM traffic alone would take 34.  Blocks per SM
// (registers, shared memory): 3, 4, 5, 6 took 165, 135, 121, 118 us; 12 words
// ahead 112, 4 words 115.
__device__ __forceinline__ void async_word(void *dst, const void *src, bool zero) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(zero ? 0 : 4)
               : "memory");
}
__device__ __forceinline__ void async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ size_t run_base(uint4 info) { return (size_t)info.x | (size_t)info.y << 32; }

template <bool DIR>
__global__ void __launch_bounds__(FAM, 6)
    k_family_matvec(const uint4 *__restrict__ fam, const uint32_t *__restrict__ prun, const uint4 *__restrict__ pinfo,
                    size_t n_fam, size_t n_patch, int max_run, const Cube<float> *__restrict__ tab,
                    const float *__restrict__ x, float *__restrict__ y) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float *xs = reinterpret_cast<float *>(smem_raw);  // two buffers
  float *ys = xs + 2 * (max_run + 1);
  uint32_t *ids = reinterpret_cast<uint32_t *>(ys + (max_run + 1));  // words of the next patch (a thread reads its own)
  Cube<float> *st = reinterpret_cast<Cube<float> *>(ids + (max_run + 1));
  const int tid = threadIdx.x;
  const uint4 none = make_uint4(0, 0, 0, 0);
  if (tid < DTAB_LEVELS) st[tid] = tab[tid];
  for (int i = tid; i <= max_run; i += FAM) ys[i] = 0.f;
  if (tid == 0) xs[0] = xs[max_run + 1] = 0.f;
  auto copy_ids = [&](uint4 info) {
    const uint32_t *src = prun + run_base(info);
    for (int u = tid; u < (int)info.z; u += FAM) async_word(ids + u, src + u, false);
  };
  auto copy_x = [&](uint4 info, int par) {
    float *dst = xs + par * (max_run + 1) + 1;
    for (int u = tid; u < (int)info.z; u += FAM) {
      const uint32_t r = ids[u];
      async_word(dst + u, x + (r & PRUN_NODE), DIR && (r & PRUN_BDY));
    }
  };
  uint4 w[4];
  auto load_w = [&](size_t p) {
#pragma unroll
    for (int q = 0; q < 4; q++) w[q] = p * FAM + tid < n_fam ? fam[(p * 4 + q) * FAM + tid] : none;
  };
  const size_t G = gridDim.x;
  size_t p = blockIdx.x;
  uint4 info = p < n_patch ? pinfo[p] : none, next = p + G < n_patch ? pinfo[p + G] : none;
  copy_ids(info);
  async_wait();
  copy_x(info, 0);
  copy_ids(next);
  load_w(p);
  for (int par = 0; p < n_patch; p += G, par ^= 1) {
    const uint4 after = p + 2 * G < n_patch ? pinfo[p + 2 * G] : none;
    async_wait();
    __syncthreads();  // x of this patch is there, ys is zero, the other buffer is free
    copy_x(next, par ^ 1);
    copy_ids(after);
    if (p * FAM + tid < n_fam &&
        !family_floating<float, false>(w, 0, xs + par * (max_run + 1), ys, st, nullptr, nullptr))
      family_scaled<float, false>(fam + p * 4 * FAM + tid, 0, xs + par * (max_run + 1), ys, st, nullptr, nullptr);
    const uint32_t *run = prun + run_base(info);
    const int nr = (int)info.z;
    constexpr int AHEAD = 8;
    uint32_t r0[AHEAD];
#pragma unroll
    for (int k = 0; k < AHEAD; k++) r0[k] = tid + k * FAM < nr ? run[tid + k * FAM] : 0u;
    load_w(p + G);
    __syncthreads();
    auto put = [&](int u, uint32_t r) {
      const uint32_t g = r & PRUN_NODE;
      const float v = ys[u + 1];
      ys[u + 1] = 0.f;
      if (DIR && (r & PRUN_BDY)) y[g] = x[g];
      else if (r & PRUN_COMPLETE) y[g] = v;
      else atomicAdd(&y[g], v);
    };
#pragma unroll
    for (int k = 0; k < AHEAD; k++)
      if (tid + k * FAM < nr) put(tid + k * FAM, r0[k]);
#pragma unroll 2
    for (int u = tid + AHEAD * FAM; u < nr; u += FAM) put(u, run[u]);
    info = next;
    next = after;
  }
}

inline size_t family_smem(int max_run) { return 16 * (size_t)(max_run + 1) + DTAB_LEVELS * sizeof(Cube<float>); }

// Elements with factors of their own (FP32 and FP64): as above without the
// copies ahead.
template <typename T>
__global__ void __launch_bounds__(FAM, sizeof(T) == 4 ? 6 : 3)
    k_family_coef(const uint4 *__restrict__ fam, const uint32_t *__restrict__ prun, const uint4 *__restrict__ pinfo,
                  size_t n_fam, size_t n_patch, int max_run, const T *__restrict__ x, T *__restrict__ y,
                  const double *__restrict__ coef, const uint32_t *__restrict__ fchild) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *xs = reinterpret_cast<T *>(smem_raw);
  T *ys = xs + (max_run + 1);
  const int tid = threadIdx.x;
  if (tid == 0) xs[0] = (T)0;
  for (size_t p = blockIdx.x; p < n_patch; p += gridDim.x) {
    const bool have = p * FAM + tid < n_fam;
    const uint4 info = pinfo[p];
    const size_t base = run_base(info);
    const int nr = (int)info.z;
    uint4 w[4];
#pragma unroll
    for (int q = 0; q < 4; q++) w[q] = have ? fam[(p * 4 + q) * FAM + tid] : make_uint4(0, 0, 0, 0);
    __syncthreads();  // the previous patch is done with xs and ys
#pragma unroll 4
    for (int u = tid; u < nr; u += FAM) {
      xs[u + 1] = x[prun[base + u] & PRUN_NODE];
      ys[u + 1] = (T)0;
    }
    __syncthreads();
    if (have && !family_floating<T, true>(w, p * FAM + tid, xs, ys, nullptr, coef, fchild))
      family_scaled<T, true>(fam + p * 4 * FAM + tid, p * FAM + tid, xs, ys, nullptr, coef, fchild);
    __syncthreads();
#pragma unroll 4
    for (int u = tid; u < nr; u += FAM) {
      const uint32_t r = prun[base + u], g = r & PRUN_NODE;
      if (r & PRUN_COMPLETE) y[g] = ys[u + 1];
      else atomicAdd(&y[g], ys[u + 1]);
    }
  }
}

template <typename T>
inline size_t family_coef_smem(int max_run) {
  return 2 * (size_t)(max_run + 1) * sizeof(T);
}

// ---- FP64 vectors ----
// GB300 issues FP64 at 2 multiply-adds per clock per SM, and an element loop in
// FP64 is bound by that: 1,270 us on 1.1e7 elements.  In the sum / difference
// basis the operator is additions and one factor per mode, so integers do all
// of it, in 64-bit fixed point with an exponent per family:
//   - x of the patch's nodes is kept as mantissa and exponent in one word; a
//     family shifts its 27 values to its largest exponent: |u| < 2^55, cut
//     below the last place (values within a factor of 4 are exact);
//   - modes, |t| < 2^61, times table entries of 2^63 scale, rounded: results
//     in units of 2^(k - 3) u.  A child's row sums |entries| to at most
//     4/3 (|lap| + |mass|), a family's lattice point to 8 of them, so |v| <
//     2^(55 + 3.42 + 3): sums in between may wrap, the results do not;
//   - a node's sum is kept in half the unit of the coarsest of the families that
//     touch it: at most 43 times 2^(55 + 2) < 2^63 (4 of 8 octants around it
//     refined, all their edges and faces hanging).  That unit is found by one
//     more round of shared-memory atomics where the patch's families differ by
//     more than FIX_EVEN binary places (without the rule 394 -> 357 us); the sum
//     becomes FP64 once per node.
// Errors in a family's result are a few units, 2^-57 of its largest value
// times the level's |lap| + |mass|.  Measured against extended precision (norm;
// 1.6e5 elements; dense FP64 stencils in brackets): uniform random x 8.9e-17
// (1.4e-16), products of sines 3.9e-16 (3.0e-15), a Gaussian 8.3e-16 (7.0e-15),
// one node 1.4e-17 (2.2e-17).
// Values far below their family's largest do not keep their own last places, so
// families in which that would show leave the fixed form: each row of a child has
// a part of the size of its class (the vertices an even number of steps away,
// itself among them), so where the largest value of every class of every child
// lies within 2^-4 of the family's, a row is off by at most 2^-44 of the sum of
// its terms' magnitudes, and mostly by less than FP64 is.  A family with a class
// below that (1 in 1e4 where x is random) is applied in FP64 and added to y
// directly (families_alone).  Classes that hold boundary nodes of the Dirichlet
// form alone have no rows; they occur at the domain's corners in every solve.
// The limit: at 2^-4, 2^-3, 2^-2 344, 360, 446 us on 1.1e7 elements, 9.2, 9.9, 11.9
// ms for an FP64 solve of 5e5 points (9.2 without a limit).
// Patches with more than FIX_ALONE such families, values that are not finite or not
// within 2^-509 .. 2^511, or factors beyond 2^+-400, take floating point, all of
// them.  1.1e7 elements in us with at most 8, 16, 32, 128 alone: x over 16 decades
// 1,585, 1,580, 1,583, 2,992; 1 in 100 nodes 1e12 times larger 1,580, 1,377, 841, 783;
// 1 in 1,000 546, 494, 491, 489; zero on one side 462, 396, 372, 372.
// What bounds it: 344 us on 1.1e7 elements (DRAM traffic alone 50): 3,600
// instructions per 32 families at 1.5 per clock per SM; warps wait for the
// gathers (3.0 of 10.5 cycles per instruction), barriers (1.6) and
// instructions (1.5: the code is long, so loops over nodes unroll no further
// than they must: by 4 and 1 350 us, 4 and 4 359, 8 and 8 405, before the limit was looked at).  Copying the next
// patch's x ahead gains 3% here and loses as much on half as many elements.  Blocks per
// SM: at 3, 4, 5, 6 451, 387, 411, 480 us.  Small meshes are bound by latency
// (2e4 elements 16 us).
// x as one word: its 53-bit mantissa, signed, above a 10-bit exponent (0: zero; 1:
// no value's)
constexpr int FIX_EXP = 10, FIX_BIAS = 511;
constexpr long long FIX_EDGE = 1;  // a boundary column of the Dirichlet form
constexpr uint32_t FIX_EVEN = 2;
constexpr int FIX_ALONE = 32;  // most families of a patch that go alone
constexpr uint32_t FIX_EMASK = (1u << FIX_EXP) - 1;

__device__ __forceinline__ long long fix_pack(double v, bool &outside) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  if (!(b << 1)) return 0;
  const int e = ((int)(b >> 52) & 0x7ff) - FIX_BIAS;
  outside = outside || e < 2 || e > (int)FIX_EMASK;
  const long long m = (long long)((b & 0xfffffffffffffull) | 1ull << 52);
  return (long long)((unsigned long long)((long long)b < 0 ? -m : m) << FIX_EXP) | (e & (int)FIX_EMASK);
}

// t times the table entry d, over 2^60: |t| < 2^61, |d| <= 2^60.  The product
// of the two low parts is replaced by its mean
__device__ __forceinline__ long long fix_mul(long long t, int2 d) {
  const int th = (int)(t >> 30), tl = (int)t & ((1 << 30) - 1);
  const long long mid = (long long)th * d.x + ((long long)tl * d.y + ((1 << 29) + (d.x >> 1)));
  return (long long)th * d.y + (mid >> 30);
}

// t / 2^n rounded down, also for n > 63
__device__ __forceinline__ long long fix_shr(long long t, uint32_t n) {
  long long r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(t), "r"(n));
  return r;
}

// adds v to a 64-bit sum in shared memory, as two words and a carry: the
// 64-bit atomic is a loop there (382 -> 357 us on 1.1e7 elements; plain adds
// would take 355)
__device__ __forceinline__ void fix_add(long long *at, long long v) {
  uint32_t *w = reinterpret_cast<uint32_t *>(at);
  const uint32_t lo = (uint32_t)v, old = atomicAdd(w, lo);
  atomicAdd(w + 1, (uint32_t)(v >> 32) + (old + lo < lo ? 1u : 0u));
}

// f * 2^-s as FP64, rounded (a normal number)
__device__ __forceinline__ double fix_to_double(long long f, int s) {
  const unsigned long long a = f < 0 ? 0ull - (unsigned long long)f : (unsigned long long)f;
  if (!a) return 0.0;
  const int lz = __clzll((long long)a);
  const int e = 1023 + 63 - lz - s;  // biased exponent before rounding
  // 53 bits with the leading one, which adds 1 to the exponent field
  const unsigned long long m = lz <= 10 ? (a + (1ull << (10 - lz))) >> (11 - lz) : a << (lz - 11);
  return __longlong_as_double((long long)((((unsigned long long)(e - 1)) << 52) + m) |
                              (f < 0 ? (long long)(1ull << 63) : 0ll));
}

// a family of a patch that takes floating point (out of line, it is rare)
__device__ __noinline__ bool family_fp64(const uint4 *__restrict__ fw, const double *xs, double *ys,
                                         const Cube<double> *__restrict__ tab, double scale) {
  uint4 w[4];
#pragma unroll
  for (int q = 0; q < 4; q++) w[q] = fw[q * FAM];
  return family_floating<double, false>(w, 0, xs, ys, tab, nullptr, nullptr, scale);
}

// The families of a patch that go alone (a bit each), in FP64 from x and onto y, a
// pair of warps for each: thread = child and vertex.  One thread per family took
// 17 us: a warp issues an FP64 operation every 64 clocks, however few lanes.  A
// vertex hangs where the family has no node at its lattice point.
template <bool DIR>
__device__ __noinline__ void families_alone(const uint4 *__restrict__ fam, const uint32_t *alone,
                                            const uint32_t *__restrict__ run, const double *x, double *y,
                                            const Cube<double> *__restrict__ tab) {
  const int k = threadIdx.x & 7, c = threadIdx.x >> 3 & 7, d = k ^ c, low = d & -d;
  int turn = 0;
  for (int w = 0; w < FAM / 32; w++)
    for (uint32_t m = alone[w]; m; m &= m - 1, turn++) {
      if ((turn & 1) != (int)(threadIdx.x >> 6)) continue;
      const uint4 *fw = fam + 32 * w + __ffs((int)m) - 1;
      auto u16 = [&](int i) -> uint32_t { return reinterpret_cast<const uint16_t *>(fw + (i >> 3) * FAM)[i & 7]; };
      const bool there = u16(28) >> c & 1u;
      const uint32_t own = u16(lat_vertex(c, k));
      const int cnt = own ? 1 : __popc(d) == 1 ? 2 : 4;  // nodes that the vertex takes the mean of
      const double share = cnt == 1 ? 1.0 : cnt == 2 ? 0.5 : 0.25;
      uint32_t r[4];
      double u = 0.0;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int s = j == 0 ? 0 : j == 1 ? low : j == 2 ? d ^ low : d;
        const uint32_t n = !there || j >= cnt ? 0u : own ? own : u16(lat_corner(c ^ s));
        r[j] = n ? run[n - 1] : PRUN_NODE;  // PRUN_NODE: no row
        if (n && !(DIR && (r[j] & PRUN_BDY))) u += x[r[j] & PRUN_NODE] * share;
        else r[j] = PRUN_NODE;
      }
      const Cube<double> s = tab[u16(27) & 31u];
      // cube_rows with r = x_i: e_i = 0
      const double e = __shfl_xor_sync(0xffffffffu, u, 3) - u + (__shfl_xor_sync(0xffffffffu, u, 5) - u) +
                       (__shfl_xor_sync(0xffffffffu, u, 6) - u);
      const double across = __shfl_xor_sync(0xffffffffu, u, 7) - u;
      const double sum = __shfl_xor_sync(0xffffffffu, 4.0 * u + e, 7);
      const double v = (s.across * across + (s.cls * e + s.other * (sum + 2.75 * u))) * share;
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (r[j] != PRUN_NODE) atomicAdd(&y[r[j] & PRUN_NODE], v);
    }
}

// the upper words' magnitudes of the family's values, united over each class of
// each child: the least of them (children that are not there left out) ...
constexpr uint32_t FIX_SMALL = 1u << 18;  // 2^-4 of a family's largest, which is 2^54 or more
__device__ __forceinline__ uint32_t fix_least(const long long (&u)[27], uint32_t mask) {
  uint32_t m[27], least = 0xffffffffu;
#pragma unroll
  for (int i = 0; i < 27; i++) m[i] = (uint32_t)abs((int)(u[i] >> 32));
#pragma unroll
  for (int c = 0; c < 8; c++) {
    uint32_t o[2];
    o[0] = o[1] = (mask >> c & 1u) ? 0u : 0xffffffffu;
#pragma unroll
    for (int k = 0; k < 8; k++) o[odd_vertex(k)] |= m[lat_vertex(c, k)];
    least = min(least, min(o[0], o[1]));
  }
  return least;
}
// ... and whether one below the limit has a node that is not a boundary column
// (fw: the family's words, xs: the patch's packed values)
__device__ __forceinline__ bool fix_rows(const long long (&u)[27], uint32_t mask, const uint4 *__restrict__ fw,
                                         const long long *xs) {
  uint32_t small = 0;  // bit 2 c the even class of child c, 2 c + 1 the odd one
#pragma unroll
  for (int c = 0; c < 8; c++) {
    uint32_t o[2] = {0, 0};
#pragma unroll
    for (int k = 0; k < 8; k++) o[odd_vertex(k)] |= (uint32_t)abs((int)(u[lat_vertex(c, k)] >> 32));
    if (mask >> c & 1u) small |= (o[0] < FIX_SMALL ? 1u << (2 * c) : 0u) | (o[1] < FIX_SMALL ? 2u << (2 * c) : 0u);
  }
#pragma unroll 1
  for (; small; small &= small - 1) {
    const int b = __ffs((int)small) - 1;
#pragma unroll 1
    for (int k = 0; k < 8; k++) {
      if (odd_vertex(k) != (b & 1)) continue;
      const int i = lat_vertex(b >> 1, k);
      const uint32_t n = reinterpret_cast<const uint16_t *>(fw + (i >> 3) * FAM)[i & 7];
      if (!n || xs[n] != FIX_EDGE) return true;
    }
  }
  return false;
}

template <bool DIR>
__global__ void __launch_bounds__(FAM, 4)
    k_family_matvec_fix(const uint4 *__restrict__ fam, const uint32_t *__restrict__ prun,
                        const uint4 *__restrict__ pinfo, size_t n_fam, size_t n_patch, int max_run,
                        const int2 *__restrict__ ftab, const Cube<double> *__restrict__ tab,
                        const double *__restrict__ x, double *__restrict__ y) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  long long *xs = reinterpret_cast<long long *>(smem_raw);
  long long *ys = xs + (max_run + 1);
  int2 *ft = reinterpret_cast<int2 *>(ys + (max_run + 1));
  uint32_t *unit = reinterpret_cast<uint32_t *>(ft + DTAB_ENTRIES);
  __shared__ uint32_t s_q[2];           // most and least unit of the patch's families
  __shared__ uint32_t s_alone[FAM / 32];  // families that go alone
  const int tid = threadIdx.x;
  for (int i = tid; i < DTAB_ENTRIES; i += FAM) ft[i] = ftab[i];
  if (tid == 0) xs[0] = 0;
  for (size_t p = blockIdx.x; p < n_patch; p += gridDim.x) {
    const bool have = p * FAM + tid < n_fam;
    const uint4 info = pinfo[p];
    const size_t base = run_base(info);
    const int nr = (int)info.z;
    uint4 w[4];
#pragma unroll
    for (int q = 0; q < 4; q++) w[q] = have ? fam[(p * 4 + q) * FAM + tid] : make_uint4(0, 0, 0, 0);
    __syncthreads();  // the previous patch is done with xs, ys and the units
    if (tid < 2) s_q[tid] = tid ? 0xffffffffu : 0u;
    bool plain = false;  // no fixed point
#pragma unroll 4
    for (int u = tid; u < nr; u += FAM) {
      const uint32_t r = prun[base + u];
      xs[u + 1] = (DIR && (r & PRUN_BDY)) ? FIX_EDGE : fix_pack(x[r & PRUN_NODE], plain);
      ys[u + 1] = 0;
      unit[u + 1] = 0;
    }
    __syncthreads();
    const uint32_t mask = fam_mask(w), hang = fam_hang(w), level = fam_level(w);
    const int k = ft[level * DTAB_STRIDE + FIX_K].x;
    long long u[27];
    uint32_t emax = 0;
    if (have) {
#pragma unroll
      for (int i = 0; i < 27; i++) {
        u[i] = xs[fam_u16(w, i)];
        emax = max(emax, (uint32_t)u[i] & FIX_EMASK);
      }
      plain = plain || k == FIX_NONE;
    }
    bool alone = false;
    if (emax > 1) {
#pragma unroll
      for (int i = 0; i < 27; i++) {
        const uint32_t e = (uint32_t)u[i] & FIX_EMASK;
        u[i] = fix_shr(u[i] & ~(long long)FIX_EMASK, FIX_EXP - 2 + emax - e);
      }
      lat_interpolate(u, hang);
      if (fix_least(u, mask) < FIX_SMALL) alone = !DIR || fix_rows(u, mask, fam + p * 4 * FAM + tid, xs);
    }
    const bool fixed = emax > 1 && !alone;
    const uint32_t q = fixed ? emax + (uint32_t)k + 1024u : 0u;
    const uint32_t hi = __reduce_max_sync(0xffffffffu, q), lo = __reduce_min_sync(0xffffffffu, q ? q : 0xffffffffu);
    const uint32_t uneven = __ballot_sync(0xffffffffu, alone);
    if ((tid & 31) == 0) {
      atomicMax(&s_q[0], hi);
      atomicMin(&s_q[1], lo);
      s_alone[tid >> 5] = uneven;
    }
    if (fixed) {
      const int2 *d = ft + level * DTAB_STRIDE;
      if (__all_sync(__activemask(), mask == 255u)) {
        lat_forward(u);
        lat_scale(u, [&](long long t, int i) { return fix_mul(t, d[i]); });
        lat_backward(u);
      } else {
        long long v[27];
        lat_elements(u, v, mask, [&](long long t, int i) { return fix_mul(t, d[DTAB_CHILD + i]); });
#pragma unroll
        for (int i = 0; i < 27; i++) u[i] = v[i];
      }
      lat_distribute(u, hang);
    }
    plain = __syncthreads_or(plain);
    static_assert(FAM == 128, "four words of families");
    const int apart = __popc(s_alone[0]) + __popc(s_alone[1]) + __popc(s_alone[2]) + __popc(s_alone[3]);
    plain = plain || apart > FIX_ALONE;
    const uint32_t qmax = s_q[0], qmin = s_q[1];
    const bool even = qmax - qmin <= FIX_EVEN;
    if (!plain) {
      if (!even) {
        if (fixed)
#pragma unroll
          for (int i = 0; i < 27; i++) {
            const uint32_t n = fam_u16(w, i);
            if (n) atomicMax(&unit[n], q);
          }
        __syncthreads();
      }
      if (fixed)
#pragma unroll
        for (int i = 0; i < 27; i++) {
          const uint32_t n = fam_u16(w, i);
          if (n) fix_add(&ys[n], fix_shr(u[i], (even ? qmax : unit[n]) + 1 - q));
        }
    } else {
      double *xd = reinterpret_cast<double *>(xs);
      for (int u = tid; u < nr; u += FAM) {
        const uint32_t r = prun[base + u];
        xd[u + 1] = (DIR && (r & PRUN_BDY)) ? 0.0 : x[r & PRUN_NODE];
      }
      __syncthreads();
      double *yd = reinterpret_cast<double *>(ys);
      if (have && !family_fp64(fam + p * 4 * FAM + tid, xd, yd, tab, 1.0))
        family_fp64(fam + p * 4 * FAM + tid, xd, yd, tab, 0.0625);
    }
    __syncthreads();
    const bool store = plain || apart == 0;
#pragma unroll 1
    for (int u = tid; u < nr; u += FAM) {
      const uint32_t r = prun[base + u], g = r & PRUN_NODE;
      const double v = plain ? __longlong_as_double(ys[u + 1])
                             : fix_to_double(ys[u + 1], 1024 + 1079 - FIX_BIAS - (int)(even ? qmax : unit[u + 1]));
      if (DIR && (r & PRUN_BDY)) y[g] = x[g];
      else if ((r & PRUN_COMPLETE) && store) y[g] = v;
      else atomicAdd(&y[g], v);
    }
    if (!store) families_alone<DIR>(fam + p * 4 * FAM, s_alone, prun + base, x, y, tab);
  }
}

inline size_t family_fix_smem(int max_run) { return ((size_t)max_run + 1) * 20 + DTAB_ENTRIES * sizeof(int2); }

// ---- small meshes: one thread per element, straight from the node lists.
// Vertices are numbered from the child's own corner, r = k ^ c, in which all
// children are alike: hanging vertices are r = 1, 2, 4 (mean of 0 and r) and 3,
// 5, 6 (mean of 0, r and its two edges).
//
// The rule: a patch takes 10 us in FP32 and 16 us in FP64 from its first load to
// its last store, however few there are; this chain (node numbers, values, some
// 70 operations, global atomic adds) is shorter until the atomics, and in FP64
// the operations, fill the chip.  Patches / elements in us: FP32 10.1 / 6.5 at
// 7.1e3 elements, 10.4 / 8.6 at 3.7e4, 10.1 / 9.5 at 5.4e4; FP64 15.3 / 10.8 at
// 7.1e3, 16 / 12.4 at 2.0e4.
template <typename T>
constexpr size_t elem_wise_max = sizeof(T) == 4 ? 90000 : 32000;

template <typename T, bool DIR>
__global__ void __launch_bounds__(128)
    k_elem_matvec(const uint32_t *__restrict__ meta, const uint32_t *__restrict__ conn, size_t E,
                  const uint8_t *__restrict__ bdy, T lapf, T massf, const T *__restrict__ x, T *__restrict__ y) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= E) return;
  const uint32_t me = meta[e], c = me >> 8 & 7u, hm = me >> 16 & 255u;
  uint32_t id[8];
#pragma unroll
  for (int r = 0; r < 8; r++) id[r] = conn[(size_t)(r ^ c) * E + e];
  T u[8];
  uint32_t edge = 0;  // vertices on the domain boundary
#pragma unroll
  for (int r = 0; r < 8; r++) {
    u[r] = x[id[r]];
    if (DIR && bdy[id[r]]) edge |= 1u << r;
  }
  T own[8];
#pragma unroll
  for (int r = 0; r < 8; r++) {
    own[r] = u[r];
    if (DIR && (edge >> r & 1u)) u[r] = (T)0;
  }
  uint32_t hang = 0;
#pragma unroll
  for (int r = 1; r < 7; r++) hang |= (hm >> (r ^ c) & 1u) << r;
  T v[8];
#pragma unroll
  for (int r = 0; r < 8; r++) {
    v[r] = u[r];
    const int a = r == 3 || r == 5 ? 1 : 2, b = r ^ a;
    if (hang >> r & 1u) {
      if (r == 1 || r == 2 || r == 4) v[r] = (T)0.5 * u[0] + (T)0.5 * u[r];
      else v[r] = ((T)0.25 * u[0] + (T)0.25 * u[r]) + ((T)0.25 * u[a] + (T)0.25 * u[b]);
    }
  }
  const T h = exp2_neg((T)0, me & 31u);
  const Cube<T> s = cube_of<T>(lapf * h * (T)0.5, massf * h * h * h * (T)0.125);
  T w[8], all = (T)0;
  cube_rows<T>(s, [&](int r) { return v[r]; }, [&](int r, T row) {
    w[r] = row;
    all += row;
  });
  if (!is_finite(all))  // as family_floating
    cube_rows<T>(s, [&](int r) { return (T)0.0625 * v[r]; }, [&](int r, T row) { w[r] = (T)16 * row; });
#pragma unroll
  for (int r = 0; r < 8; r++) v[r] = w[r];
#pragma unroll
  for (int r = 1; r < 7; r++) {
    const int a = r == 3 || r == 5 ? 1 : 2, b = r ^ a;
    if (hang >> r & 1u) {
      if (r == 1 || r == 2 || r == 4) {
        w[r] -= (T)0.5 * v[r];
        w[0] += (T)0.5 * v[r];
      } else {
        w[r] -= (T)0.75 * v[r];
        w[0] += (T)0.25 * v[r];
        w[a] += (T)0.25 * v[r];
        w[b] += (T)0.25 * v[r];
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 8; r++) {
    if (DIR && (edge >> r & 1u)) y[id[r]] = own[r];
    else atomicAdd(&y[id[r]], w[r]);
  }
}

}  // namespace dg

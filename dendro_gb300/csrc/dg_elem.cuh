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
// Elements: K and M are tensor products, diagonal in a basis of sums and
// differences.  For the assembled 2x2x2 family, per axis
//   M = 1/4 s s^T + 1/3 o o^T + 1/12 q q^T,  A = 1/4 o o^T + 1/4 q q^T
// with s = (1,2,1), o = (1,0,-1), q = (1,-2,1); for one element
//   M = 1/2 s s^T + 1/6 d d^T,  A = 1/2 d d^T,  s = (1,1), d = (1,-1).
// So a complete family (3 of 4) costs 27 lines each way (4 and 5 operations a
// line, all coefficients 1 or 2) and 27 multiplications: 262 operations for 8
// elements, where 8 dense 8x8 stencils cost 512 multiply-adds.  A family with
// subdivided children is applied element by element: 397 operations.
//
// What bounds it (1.1e7 elements of a Gaussian cloud, GB300): FP32 143 us,
// instruction issue and the latency of the gathers (DRAM traffic alone would
// take 34 us; without the shared-memory atomics 116 us, without the x gather
// 124 us); FP64 1,270 us, the FP64 pipe, which issues 2 operations per clock
// per SM; fixed point 293 us, integer issue.  An element-wise loop over dense
// stencils, 8 gathers and 8 atomics per element, took 348, 1,820 and 873 us
// (the last in double-single arithmetic).  128 families per patch: 64 and 256
// measured 152 / 150 us in FP32 and 1,296 / 1,481 us in FP64; a patch of 256
// leaves too few blocks on small meshes.
//
// Patches: FAM consecutive families (in element order) make a patch, one
// thread block's work at a time.  fam[(p * 4 + w) * FAM + t] is word w of the
// patch's family t: 27 x 16 bits, the patch-local number of the node at each
// lattice point (0: no node there), then 16 bits level and 8 bits mask of the
// children that are leaves, then 18 bits of hanging points.  Complete families
// come first, so that most warps hold one kind.  pinfo[p] = {offset of the
// patch's nodes in prun (64 bits), their number, the level of its coarsest
// element}; prun holds the nodes, number 1 first, with two flags.
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

// entry i of the table: lap and mass already scaled by h / 2 and h^3 / 8
template <typename T>
__device__ __forceinline__ T dtab_entry(int i, T lap, T mass) {
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
  return lap * (T)(a[0] * m[1] * m[2] + m[0] * a[1] * m[2] + m[0] * m[1] * a[2]) + mass * (T)(m[0] * m[1] * m[2]);
}

template <typename T>
__global__ void k_dtab(T *__restrict__ out, double lapf, double massf) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= DTAB_ENTRIES) return;
  const double h = ldexp(1.0, -(i / DTAB_STRIDE));
  const int q = i % DTAB_STRIDE;
  out[i] = q < DTAB_CHILD + 4 ? (T)dtab_entry<double>(q, lapf * h * 0.5, massf * h * h * h * 0.125) : (T)0;
}

// The table entries of K + M as fractions: entry i is
// (alpha fix_lap(i) + beta fix_mass(i)) / (27 * 2^fix_shift(i)) with
// alpha = h / 2, beta = h^3 / 8
__host__ __device__ constexpr int fix_weight(int i, bool lap) {
  int m[3] = {}, a[3] = {};  // mode weights times 12 (a family's) or 6 (an element's)
  if (i < DTAB_CHILD) {
    const int o = i < 4 ? 0 : i < 7 ? 1 : i < 9 ? 2 : 3;
    const int q = i - (i < 4 ? 0 : i < 7 ? 4 : i < 9 ? 7 : 9);
    for (int k = 0; k < 3; k++) {
      m[k] = k < o ? 4 : k < o + q ? 1 : 3;
      a[k] = k < o + q ? 3 : 0;
    }
  } else {
    for (int k = 0; k < 3; k++) {
      m[k] = k < i - DTAB_CHILD ? 1 : 3;
      a[k] = k < i - DTAB_CHILD ? 3 : 0;
    }
  }
  return lap ? a[0] * m[1] * m[2] + m[0] * a[1] * m[2] + m[0] * m[1] * a[2] : m[0] * m[1] * m[2];
}
__host__ __device__ constexpr int fix_shift(int i) { return i < DTAB_CHILD ? 6 : 3; }

// arithmetic of one lattice value: FP32, FP64 or 64-bit fixed point
template <typename V>
struct LatOps {
  static __device__ __forceinline__ V add_twice(V a, V b) { return a + (V)2 * b; }
  static __device__ __forceinline__ V sub_twice(V a, V b) { return a - (V)2 * b; }
  static __device__ __forceinline__ V half_add(V v, V half_of) { return v + (V)0.5 * half_of; }
  static __device__ __forceinline__ V mean(V a, V b) { return (V)0.5 * (a + b); }
};
template <>
struct LatOps<long long> {
  static __device__ __forceinline__ long long add_twice(long long a, long long b) { return a + 2 * b; }
  static __device__ __forceinline__ long long sub_twice(long long a, long long b) { return a - 2 * b; }
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

// a complete family: to the sum / difference basis and back, in place
template <typename V>
__device__ __forceinline__ void lat_forward(V (&u)[27]) {
#pragma unroll
  for (int ax = 0; ax < 3; ax++) {
    const int st = ax == 0 ? 1 : ax == 1 ? 3 : 9;
#pragma unroll
    for (int n = 0; n < 9; n++) {
      const int i = ax == 0 ? 3 * n : ax == 1 ? n % 3 + 9 * (n / 3) : n;
      const V e = u[i] + u[i + 2 * st], o = u[i] - u[i + 2 * st], b = u[i + st];
      u[i] = LatOps<V>::add_twice(e, b);
      u[i + st] = o;
      u[i + 2 * st] = LatOps<V>::sub_twice(e, b);
    }
  }
}
template <typename V>
__device__ __forceinline__ void lat_backward(V (&u)[27]) {
#pragma unroll
  for (int ax = 0; ax < 3; ax++) {
    const int st = ax == 0 ? 1 : ax == 1 ? 3 : 9;
#pragma unroll
    for (int n = 0; n < 9; n++) {
      const int i = ax == 0 ? 3 * n : ax == 1 ? n % 3 + 9 * (n / 3) : n;
      const V t = u[i] + u[i + 2 * st], r = u[i] - u[i + 2 * st], o = u[i + st];
      u[i] = t + o;
      u[i + st] = r + r;
      u[i + 2 * st] = t - o;
    }
  }
}
// the modes times their table entries; mul(t, i): t times entry i
template <typename V, typename Mul>
__device__ __forceinline__ void lat_scale(V (&u)[27], Mul &&mul) {
#pragma unroll
  for (int i = 0; i < 27; i++) {
    const int x = i % 3, y = i / 3 % 3, z = i / 9;
    u[i] = mul(u[i], dfam((x == 1) + (y == 1) + (z == 1), (x == 2) + (y == 2) + (z == 2)));
  }
}

// any family, v = sum over its elements of S u, element by element in the
// basis of one element, the sums and differences of shared edges and faces
// formed once: 148 operations in, 64 multiplications, 185 out for 8 elements
// (333 for each on its own: 512).  begin(c) before child c; mul(t, p): t times
// its entry for p factors d.  A child that is not there gets no value.
template <typename V, typename Begin, typename Mul>
__device__ __forceinline__ void lat_elements(const V (&u)[27], V (&v)[27], uint32_t mask, Begin &&begin, Mul &&mul) {
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
        begin(c);
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

// One block per patch, grid-strided, three barriers per patch:
//   1. x of the patch's nodes into xs (node ids read coalesced), ys = 0;
//   2. thread t = family t: its lattice from xs, its elements in registers,
//      its lattice added into ys with shared-memory atomics;
//   3. each node's sum stored (nodes of this patch alone) or added to y.
// DIR, the Dirichlet form: boundary rows are the identity (y = x), boundary
// columns are dropped.  COEF: element e's factors are coef[2e] (Laplacian)
// and coef[2e + 1] (mass) instead of the table's; fchild[8 f + c] gives e.
// A family whose values are not all finite takes the element path, so that a
// non-finite x reaches exactly the rows of the elements that hold it.
// Blocks per SM (registers): FP32 at 4 to 8 blocks 158, 152, 143, 145, 151 us on
// 1.1e7 elements; FP64 at 2, 3, 4 blocks 1,350, 1,279, 1,267 us (4 spills).
template <typename T, bool DIR, bool COEF>
__global__ void __launch_bounds__(FAM, sizeof(T) == 4 ? 6 : 3)
    k_family_matvec(const uint4 *__restrict__ fam, const uint32_t *__restrict__ prun, const uint4 *__restrict__ pinfo,
                    size_t n_fam, size_t n_patch, int max_run, const T *__restrict__ dtab, const T *__restrict__ x,
                    T *__restrict__ y, const double *__restrict__ coef, const uint32_t *__restrict__ fchild) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *xs = reinterpret_cast<T *>(smem_raw);
  T *ys = xs + (max_run + 1);
  T *dt = ys + (max_run + 1);
  const int tid = threadIdx.x;
  if (!COEF)
    for (int i = tid; i < DTAB_ENTRIES; i += FAM) dt[i] = dtab[i];
  if (tid == 0) xs[0] = (T)0;
  for (size_t p = blockIdx.x; p < n_patch; p += gridDim.x) {
    const bool have = p * FAM + tid < n_fam;
    const uint4 info = pinfo[p];
    const size_t base = (size_t)info.x | (size_t)info.y << 32;
    const int nr = (int)info.z;
    uint4 w[4];
#pragma unroll
    for (int q = 0; q < 4; q++) w[q] = have ? fam[(p * 4 + q) * FAM + tid] : make_uint4(0, 0, 0, 0);
    __syncthreads();  // the previous patch is done with xs and ys
#pragma unroll 4
    for (int u = tid; u < nr; u += FAM) {
      const uint32_t r = prun[base + u];
      xs[u + 1] = (DIR && (r & PRUN_BDY)) ? (T)0 : x[r & PRUN_NODE];
      ys[u + 1] = (T)0;
    }
    __syncthreads();
    if (have) {
      const uint32_t mask = fam_mask(w), hang = fam_hang(w);
      T u[27];
      auto gather = [&]() {
#pragma unroll
        for (int i = 0; i < 27; i++) u[i] = xs[fam_u16(w, i)];
        lat_interpolate(u, hang);
      };
      gather();
      bool regather = false;
      // a warp takes one path: both cost more than the dearer one
      bool whole = !COEF && __all_sync(__activemask(), mask == 255u);
      if (whole) {
        lat_forward(u);
        regather = !is_finite(u[0]);  // the weighted sum of all 27
        whole = !regather;
      }
      if (whole) {
        const T *d = dt + fam_level(w) * DTAB_STRIDE;
        lat_scale(u, [&](T t, int i) { return t * d[i]; });
        lat_backward(u);
      } else {
        if (regather) gather();
        T v[27], d[4];
        if constexpr (!COEF) {
#pragma unroll
          for (int k = 0; k < 4; k++) d[k] = dt[fam_level(w) * DTAB_STRIDE + DTAB_CHILD + k];
        }
        lat_elements(
            u, v, mask,
            [&](int c) {
              if constexpr (COEF) {
                const size_t e = fchild[8 * (p * FAM + tid) + c];  // 0 where there is none
                const T h = exp2_neg((T)0, fam_level(w));
                const T lf = (T)coef[2 * e] * h * (T)0.5, mf = (T)coef[2 * e + 1] * h * h * h * (T)0.125;
#pragma unroll
                for (int k = 0; k < 4; k++) d[k] = dtab_entry(DTAB_CHILD + k, lf, mf);
              }
            },
            [&](T t, int q) { return t * d[q]; });
#pragma unroll
        for (int i = 0; i < 27; i++) u[i] = v[i];
      }
      lat_distribute(u, hang);
#pragma unroll
      for (int i = 0; i < 27; i++) {
        const uint32_t n = fam_u16(w, i);
        if (n) atomicAdd(&ys[n], u[i]);
      }
    }
    __syncthreads();
#pragma unroll 4
    for (int u = tid; u < nr; u += FAM) {
      const uint32_t r = prun[base + u], g = r & PRUN_NODE;
      if (DIR && (r & PRUN_BDY)) y[g] = x[g];
      else if (r & PRUN_COMPLETE) y[g] = ys[u + 1];
      else atomicAdd(&y[g], ys[u + 1]);
    }
  }
}

template <typename T>
inline size_t family_smem(int max_run) {
  return (2 * (size_t)(max_run + 1) + DTAB_ENTRIES) * sizeof(T);
}

// ---- fixed-point form for FP64 vectors: the CG operator (K + M, Dirichlet)
// of the FP32-V-cycle solve.  GB300 issues FP64 at 2 multiply-adds per clock
// per SM, and the FP64 loop is bound by that.  In the sum / difference basis
// the operator is additions and one factor per mode, a small integer over
// 27 * 2^k times powers of two of the level, so integers do all of it: each
// patch takes its x as 51-bit fixed point relative to the patch's largest
// entry, the sums and differences are exact, a mode's product is exact before
// its shift, and the node sums are integer atomic adds; 1/27 is applied to
// each node's sum.  With |x| < 2^51 a mode's product stays below 2^62
// (1728 + 144 times |x| at the most) and a node's sum too (at most 75 alpha
// times 27 |x|).  The rounding of x is 2^-52 of the patch's largest entry and
// that of the modes smaller.  Conversions are integer operations as well, so
// the loop issues one FP64 multiplication per node and the global adds.
// Against FP64 on uniform random x the result is off by 1.4e-16 of its norm
// (1.4e-15 for the FP32-pair arithmetic it replaces).  Blocks per SM: at 3, 4, 5,
// 6 blocks 367, 319, 293, 293 us on 1.1e7 elements.

// x * 2^s rounded to an integer (|x| * 2^s < 2^51)
__device__ __forceinline__ long long double_to_fix(unsigned long long bits, int s) {
  const int e = (int)(bits >> 52) & 0x7ff;
  unsigned long long m = bits & 0xfffffffffffffull;
  if (e) m |= 1ull << 52;
  const int sh = (e ? e : 1) - 1075 + s;
  unsigned long long r;
  if (sh >= 0) r = m << sh;
  else if (sh > -55) r = (m + (1ull << (-sh - 1))) >> -sh;
  else r = 0;
  return (bits >> 63) ? -(long long)r : (long long)r;
}

// f * 2^-s as FP64, rounded
__device__ __forceinline__ double fix_to_double(long long f, int s) {
  const unsigned long long a = f < 0 ? 0ull - (unsigned long long)f : (unsigned long long)f;
  if (!a) return 0.0;
  const int lz = __clzll((long long)a);
  const int e = 1023 + 63 - lz - s;  // biased exponent before rounding
  if (e < 1 || e > 2045) return ldexp((double)f, -s);
  // 53 bits with the leading one, which adds 1 to the exponent field
  const unsigned long long m = lz <= 10 ? (a + (1ull << (10 - lz))) >> (11 - lz) : a << (lz - 11);
  return __longlong_as_double((long long)((((unsigned long long)(e - 1)) << 52) + m) |
                              (f < 0 ? (long long)(1ull << 63) : 0ll));
}

template <bool DIR>
__global__ void __launch_bounds__(FAM, 5)
    k_family_matvec_fix(const uint4 *__restrict__ fam, const uint32_t *__restrict__ prun,
                        const uint4 *__restrict__ pinfo, size_t n_fam, size_t n_patch, int max_run,
                        const double *__restrict__ x, double *__restrict__ y) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  long long *xs = reinterpret_cast<long long *>(smem_raw);
  long long *ys = xs + (max_run + 1);
  __shared__ uint32_t s_emax[2];  // largest biased exponent of the patch's x, by patch parity
  const int tid = threadIdx.x;
  if (tid < 2) s_emax[tid] = 0;
  if (tid == 0) xs[0] = 0;
  int par = 0;
  for (size_t p = blockIdx.x; p < n_patch; p += gridDim.x, par ^= 1) {
    const bool have = p * FAM + tid < n_fam;
    const uint4 info = pinfo[p];
    const size_t base = (size_t)info.x | (size_t)info.y << 32;
    const int nr = (int)info.z;
    uint4 w[4];
#pragma unroll
    for (int q = 0; q < 4; q++) w[q] = have ? fam[(p * 4 + q) * FAM + tid] : make_uint4(0, 0, 0, 0);
    __syncthreads();  // the previous patch is done with xs, ys and its exponent
    uint32_t emax = 0;
#pragma unroll 4
    for (int u = tid; u < nr; u += FAM) {
      const uint32_t r = prun[base + u];
      const long long b = (DIR && (r & PRUN_BDY)) ? 0ll : __double_as_longlong(x[r & PRUN_NODE]);
      xs[u + 1] = b;
      ys[u + 1] = 0;
      emax = max(emax, (uint32_t)((unsigned long long)b >> 52) & 0x7ffu);
    }
    emax = __reduce_max_sync(0xffffffffu, emax);
    if ((tid & 31) == 0) atomicMax(&s_emax[par], emax);
    __syncthreads();
    emax = s_emax[par];
    if (tid == 0) s_emax[par ^ 1] = 0;  // for the next patch
    const bool finite = emax < 0x7ffu;
    const int s = 1073 - (int)(emax ? emax : 1u);  // |x| * 2^s < 2^51
    for (int u = tid; u < nr; u += FAM) xs[u + 1] = double_to_fix((unsigned long long)xs[u + 1], s);
    __syncthreads();
    if (have) {
      const uint32_t mask = fam_mask(w), hang = fam_hang(w);
      // in units of alpha / 27 of the patch's coarsest level
      const int finer = (int)fam_level(w) - (int)info.w, mass = 2 * (int)fam_level(w) + 2;
      long long u[27];
#pragma unroll
      for (int i = 0; i < 27; i++) u[i] = xs[fam_u16(w, i)];
      lat_interpolate(u, hang);
      auto mul = [&](long long t, int i) {
        return (t * fix_weight(i, true) + (t >> mass) * fix_weight(i, false)) >> (finer + fix_shift(i));
      };
      if (__all_sync(__activemask(), mask == 255u)) {
        lat_forward(u);
        lat_scale(u, mul);
        lat_backward(u);
      } else {
        long long v[27];
        lat_elements(u, v, mask, [](int) {}, [&](long long t, int q) { return mul(t, DTAB_CHILD + q); });
#pragma unroll
        for (int i = 0; i < 27; i++) u[i] = v[i];
      }
      lat_distribute(u, hang);
#pragma unroll
      for (int i = 0; i < 27; i++) {
        const uint32_t n = fam_u16(w, i);
        if (n) atomicAdd(reinterpret_cast<unsigned long long *>(&ys[n]), (unsigned long long)u[i]);
      }
    }
    __syncthreads();
    const int sy = s + (int)info.w + 1;
#pragma unroll 4
    for (int u = tid; u < nr; u += FAM) {
      const uint32_t r = prun[base + u], g = r & PRUN_NODE;
      // a patch with a non-finite x: all its rows are NaN
      const double v = finite ? fix_to_double(ys[u + 1], sy) * (1.0 / 27.0) : __longlong_as_double(0x7ff8000000000000ll);
      if (DIR && (r & PRUN_BDY)) y[g] = x[g];
      else if (r & PRUN_COMPLETE) y[g] = v;
      else atomicAdd(&y[g], v);
    }
  }
}

}  // namespace dg

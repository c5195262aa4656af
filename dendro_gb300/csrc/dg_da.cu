// Octree mesh build (ot::DA at one rank: src/oda/oda.cpp:250 ->
// DA_FactoryPart1..3, src/oda/private/odaFactory.cpp, odaBuildNlist.cpp)
// and the Laplacian + mass element loop (examples/src/backend/odaJac.C).
//
// Hanging vertices.  Element e at level l is child c of parent P (level
// l-1).  Only the vertices c^r with r in {1,2,4} (midpoints of P's edges
// through corner c) and r in {3,5,6} (centres of P's faces through corner
// c) can hang.  Such a vertex hangs when one of P's same-size neighbours
// that share that face or edge is an unrefined leaf (2:1 balance bounds the
// neighbour to level l-1).  A hanging vertex k refers to P's vertex k, which
// is always a mesh node; the element type (one of 18 per child number,
// include/oda/cnumEtypes.h) selects the stencil that folds the hanging
// interpolation into the element matrix.
//
// Nodes.  Every node is the anchor of exactly one octant of the reference's
// DA octant set (elements plus the positive-boundary pseudo-octants of
// octFunctions.cpp:681-770).  Here element e owns its anchor (when it does
// not hang) and its vertices on the positive domain boundary, so the node
// set is numbered by one scan over elements; the owner of any vertex is the
// leaf that contains it after clamping boundary coordinates inward.
#include "dg_da.cuh"
#include "dg_elem.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <vector>

namespace dg {

// ------------------------------------------------------------------------
// element-type and stencil tables (host)
// ------------------------------------------------------------------------
// The 18 hanging configurations in the reference's type order
// (include/oda/odaUtils.tcc:14-120), as vertex sets relative to the child's
// own corner: relative vertex r = 1, 2, 4 are the edge midpoints, 3, 5, 6 the
// face centres.  Bit r of each entry marks relative vertex r as hanging.
static const uint8_t kCanonRel[18] = {0x00, 0x04, 0x02, 0x06, 0x10, 0x14, 0x12, 0x16, 0x0e,
                                      0x1e, 0x54, 0x56, 0x5e, 0x32, 0x36, 0x3e, 0x76, 0x7e};
// Each child number's table is the canonical one with its axes permuted:
// the relative axis bit that canonical x, y, z map to.
static const uint8_t kAxisPerm[8][3] = {{1, 2, 4}, {2, 1, 4}, {2, 1, 4}, {1, 2, 4},
                                        {1, 4, 2}, {2, 4, 1}, {2, 4, 1}, {1, 4, 2}};

void gen_etype_masks(uint8_t masks[8 * 18]) {
  for (int c = 0; c < 8; c++)
    for (int t = 0; t < 18; t++) {
      uint8_t m = 0;
      for (int r = 0; r < 8; r++) {
        if (!(kCanonRel[t] >> r & 1)) continue;
        int pr = ((r & 1) ? kAxisPerm[c][0] : 0) | ((r & 2) ? kAxisPerm[c][1] : 0) | ((r & 4) ? kAxisPerm[c][2] : 0);
        m |= (uint8_t)(1u << (pr ^ c));
      }
      masks[c * 18 + t] = m;
    }
}

// S[c][t] = P^T K P on the reference element [-1,1]^3 with trilinear shape
// functions; K = stiffness (Laplacian) or mass; P maps the 8 referenced
// values to the child's vertex values (a hanging vertex is the average of
// the parent corners spanning its edge or face).
void gen_stencils(double *lap, double *mass) {
  const double m1[2][2] = {{2.0 / 3.0, 1.0 / 3.0}, {1.0 / 3.0, 2.0 / 3.0}};
  const double a1[2][2] = {{0.5, -0.5}, {-0.5, 0.5}};
  double K[8][8], M[8][8];
  for (int i = 0; i < 8; i++)
    for (int j = 0; j < 8; j++) {
      int ix = i & 1, iy = i >> 1 & 1, iz = i >> 2 & 1, jx = j & 1, jy = j >> 1 & 1, jz = j >> 2 & 1;
      K[i][j] = a1[ix][jx] * m1[iy][jy] * m1[iz][jz] + m1[ix][jx] * a1[iy][jy] * m1[iz][jz] +
                m1[ix][jx] * m1[iy][jy] * a1[iz][jz];
      M[i][j] = m1[ix][jx] * m1[iy][jy] * m1[iz][jz];
    }
  uint8_t masks[8 * 18];
  gen_etype_masks(masks);
  for (int c = 0; c < 8; c++)
    for (int t = 0; t < 18; t++) {
      double P[8][8];
      std::memset(P, 0, sizeof(P));
      uint8_t hm = masks[c * 18 + t];
      for (int k = 0; k < 8; k++) {
        if (!(hm >> k & 1)) {
          P[k][k] = 1.0;
          continue;
        }
        int d = k ^ c, cnt = 0;
        for (int s = 0; s < 8; s++) cnt += ((s & d) == s);
        for (int s = 0; s < 8; s++)
          if ((s & d) == s) P[k][c ^ s] += 1.0 / cnt;
      }
      for (int i = 0; i < 8; i++)
        for (int j = 0; j < 8; j++) {
          double sl = 0.0, sm = 0.0;
          for (int a = 0; a < 8; a++)
            for (int b = 0; b < 8; b++) {
              double w = P[a][i] * P[b][j];
              if (w != 0.0) {
                sl += w * K[a][b];
                sm += w * M[a][b];
              }
            }
          size_t o = (((size_t)c * 18 + t) * 8 + i) * 8 + j;
          lap[o] = sl;
          mass[o] = sm;
        }
    }
}


void ensure_stencils(Context &ctx) {
  if (ctx.d_sten64) return;
  std::vector<double> lap(8 * 18 * 64), mass(8 * 18 * 64);
  gen_stencils(lap.data(), mass.data());
  std::vector<double> s64(STEN_ENTRIES);
  std::vector<float> s32(STEN_ENTRIES);
  for (int ct = 0; ct < 8 * 18; ct++)
    for (int q = 0; q < 64; q++) {
      s64[ct * 128 + q] = lap[ct * 64 + q];
      s64[ct * 128 + 64 + q] = mass[ct * 64 + q];
    }
  for (int i = 0; i < STEN_ENTRIES; i++) s32[i] = (float)s64[i];
  uint8_t masks[8 * 18], etype_of[8 * 256];
  gen_etype_masks(masks);
  std::memset(etype_of, 0xff, sizeof(etype_of));
  for (int c = 0; c < 8; c++)
    for (int t = 0; t < 18; t++) etype_of[c * 256 + masks[c * 18 + t]] = (uint8_t)t;
  double *d64 = nullptr;
  float *d32 = nullptr;
  uint8_t *det = nullptr, *dem = nullptr;
  DG_CUDA(cudaMalloc((void **)&d64, STEN_ENTRIES * sizeof(double)));
  DG_CUDA(cudaMalloc((void **)&d32, STEN_ENTRIES * sizeof(float)));
  DG_CUDA(cudaMalloc((void **)&det, sizeof(etype_of)));
  DG_CUDA(cudaMalloc((void **)&dem, sizeof(masks)));
  DG_CUDA(cudaMemcpy(d64, s64.data(), STEN_ENTRIES * sizeof(double), cudaMemcpyHostToDevice));
  DG_CUDA(cudaMemcpy(d32, s32.data(), STEN_ENTRIES * sizeof(float), cudaMemcpyHostToDevice));
  DG_CUDA(cudaMemcpy(det, etype_of, sizeof(etype_of), cudaMemcpyHostToDevice));
  DG_CUDA(cudaMemcpy(dem, masks, sizeof(masks), cudaMemcpyHostToDevice));
  ctx.d_sten64 = d64;
  ctx.d_sten32 = d32;
  ctx.d_etype_of = det;
  ctx.d_etype_mask = dem;
}

// ------------------------------------------------------------------------
// mesh build
// ------------------------------------------------------------------------
// Anchor -> element map: no two octants of a linear octree share an anchor,
// so "the element anchored at p" is one look-up.  Open addressing with
// linear probing over a power-of-two table of element indices (at most half
// full); a slot's anchor is read back from the keys.
constexpr uint32_t AH_EMPTY = 0xffffffffu;

__device__ __forceinline__ uint64_t anchor_hash(Key128 a) {
  uint64_t x = a.lo ^ (a.hi * 0x9e3779b97f4a7c15ull);
  x ^= x >> 31;
  x *= 0xbf58476d1ce4e5b9ull;
  x ^= x >> 29;
  return x;
}

__global__ void k_anchor_insert(const Key128 *__restrict__ keys, size_t n, uint32_t *__restrict__ tab, uint64_t mask) {
  size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  uint64_t h = anchor_hash(tag_anchor(keys[e])) & mask;
  for (uint64_t probe = 0; probe <= mask; probe++) {
    if (atomicCAS(&tab[h], AH_EMPTY, (uint32_t)e) == AH_EMPTY) return;
    h = (h + 1) & mask;
  }
}

// element anchored at `pos` (a bare anchor), or AH_EMPTY
__device__ __forceinline__ uint32_t anchor_find(const Key128 *__restrict__ keys, const uint32_t *__restrict__ tab,
                                                uint64_t mask, Key128 pos) {
  uint64_t h = anchor_hash(pos) & mask;
  for (uint64_t probe = 0; probe <= mask; probe++) {
    const uint32_t e = tab[h];
    if (e == AH_EMPTY) return AH_EMPTY;
    if (key_eq(tag_anchor(keys[e]), pos)) return e;
    h = (h + 1) & mask;
  }
  return AH_EMPTY;
}

__device__ __forceinline__ bool is_leaf_at(const Key128 *__restrict__ keys, const uint32_t *__restrict__ tab,
                                           uint64_t mask, int64_t x, int64_t y, int64_t z, unsigned lev, int64_t dom) {
  if (x < 0 || y < 0 || z < 0 || x >= dom || y >= dom || z >= dom) return false;
  const uint32_t j = anchor_find(keys, tab, mask, morton3((uint32_t)x, (uint32_t)y, (uint32_t)z));
  return j != AH_EMPTY && tag_level(keys[j]) == lev;
}

__global__ void k_mesh_elems(const Key128 *__restrict__ keys, size_t n, const uint32_t *__restrict__ tab,
                             uint64_t mask, unsigned D, const uint8_t *__restrict__ etype_of,
                             uint32_t *__restrict__ meta, uint32_t *__restrict__ cnt, uint32_t *flags) {
  size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const Key128 ke = keys[e];
  const unsigned l = tag_level(ke);
  uint32_t ux, uy, uz;
  demorton3(tag_anchor(ke), ux, uy, uz);
  const int64_t dom = (int64_t)1 << D, h = (int64_t)1 << (D - l);
  const int64_t x = ux, y = uy, z = uz;
  int c = 0;
  if (l > 0) c = (int)(((x >> (D - l)) & 1) | (((y >> (D - l)) & 1) << 1) | (((z >> (D - l)) & 1) << 2));
  unsigned hm = 0;
  if (l > 1) {
    const int64_t H = 2 * h;
    const int64_t P[3] = {x - ((c & 1) ? h : 0), y - ((c & 2) ? h : 0), z - ((c & 4) ? h : 0)};
    const int64_t d[3] = {(c & 1) ? H : -H, (c & 2) ? H : -H, (c & 4) ? H : -H};
    // neighbours of P towards the child's exterior: leaf[s] for s in 1..7
    bool leaf[8];
    leaf[0] = false;
#pragma unroll
    for (int s = 1; s < 8; s++) {
      if (s == 7) {
        leaf[s] = false;  // the corner neighbour hangs no vertex of e
        continue;
      }
      leaf[s] = is_leaf_at(keys, tab, mask, P[0] + ((s & 1) ? d[0] : 0), P[1] + ((s & 2) ? d[1] : 0),
                           P[2] + ((s & 4) ? d[2] : 0), l - 1, dom);
    }
#pragma unroll
    for (int r = 1; r < 7; r++) {
      const int others = 7 & ~r;
      bool hang = false;
#pragma unroll
      for (int s = 1; s < 7; s++)
        if ((s & others) == s && leaf[s]) hang = true;
      if (hang) hm |= 1u << (c ^ r);
    }
  }
  unsigned et = etype_of[c * 256 + hm];
  if (et == 0xffu) {
    atomicOr(flags, DGF_NOT_BALANCED);
    et = 0;
  }
  meta[e] = l | ((unsigned)c << 8) | (hm << 16) | (et << 24);
  const unsigned bdy = ((x + h == dom) ? 1u : 0u) | ((y + h == dom) ? 2u : 0u) | ((z + h == dom) ? 4u : 0u);
  unsigned owned = 0;
#pragma unroll
  for (int k = 0; k < 8; k++)
    if ((k & bdy) == (unsigned)k && !(hm >> k & 1)) owned++;
  cnt[e] = owned;
}

__global__ void k_mesh_conn(const Key128 *__restrict__ keys, size_t n, const uint32_t *__restrict__ tab,
                            uint64_t mask, unsigned D, const uint32_t *__restrict__ meta,
                            const uint64_t *__restrict__ base, uint32_t *__restrict__ conn, uint32_t *__restrict__ nx,
                            uint32_t *__restrict__ ny, uint32_t *__restrict__ nz, size_t n_node, uint32_t *flags) {
  size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const Key128 ke = keys[e];
  const uint32_t me = meta[e];
  const unsigned l = me & 255u, c = (me >> 8) & 7u, hm = (me >> 16) & 255u;
  uint32_t ux, uy, uz;
  demorton3(tag_anchor(ke), ux, uy, uz);
  const int64_t dom = (int64_t)1 << D, h = (int64_t)1 << (D - l);
  const int64_t x = ux, y = uy, z = uz;
  const int64_t px = x - ((c & 1) ? h : 0), py = y - ((c & 2) ? h : 0), pz = z - ((c & 4) ? h : 0);
  // owned nodes: coordinates
  {
    const unsigned bdy = ((x + h == dom) ? 1u : 0u) | ((y + h == dom) ? 2u : 0u) | ((z + h == dom) ? 4u : 0u);
    uint64_t id = base[e];
    for (int k = 0; k < 8; k++) {
      if ((k & bdy) != (unsigned)k || (hm >> k & 1)) continue;
      if (id < n_node) {
        nx[id] = (uint32_t)(x + ((k & 1) ? h : 0));
        ny[id] = (uint32_t)(y + ((k & 2) ? h : 0));
        nz[id] = (uint32_t)(z + ((k & 4) ? h : 0));
      }
      id++;
    }
  }
#pragma unroll 1
  for (int k = 0; k < 8; k++) {
    int64_t v[3];
    if (hm >> k & 1) {
      v[0] = px + ((k & 1) ? 2 * h : 0);
      v[1] = py + ((k & 2) ? 2 * h : 0);
      v[2] = pz + ((k & 4) ? 2 * h : 0);
    } else {
      v[0] = x + ((k & 1) ? h : 0);
      v[1] = y + ((k & 2) ? h : 0);
      v[2] = z + ((k & 4) ? h : 0);
    }
    unsigned kb = 0;
    int64_t cl[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      if (v[a] == dom) {
        kb |= 1u << a;
        cl[a] = dom - 1;
      } else {
        cl[a] = v[a];
      }
    }
    // the owner is the element anchored at the vertex; on the positive domain
    // boundary, the leaf containing the vertex clamped inward (a search)
    size_t o;
    bool found = true;
    if (k == 0 && !(hm & 1u)) {
      o = e;  // a vertex 0 that does not hang is the element's own anchor
    } else if (kb == 0) {
      const uint32_t f = anchor_find(keys, tab, mask, morton3((uint32_t)cl[0], (uint32_t)cl[1], (uint32_t)cl[2]));
      found = f != AH_EMPTY;
      o = found ? f : 0;
    } else {
      o = find_leaf_from(keys, n, morton3((uint32_t)cl[0], (uint32_t)cl[1], (uint32_t)cl[2]), e);
    }
    const Key128 ko = keys[o];
    const unsigned lo_ = tag_level(ko);
    const int64_t ho = (int64_t)1 << (D - lo_);
    // the owner's anchor: the vertex itself when it was found by its anchor
    // (no decode needed), else decoded from the owner's key
    int64_t oc[3] = {v[0], v[1], v[2]};
    bool ok = found;
    if (kb != 0) {
      uint32_t ox, oy, oz;
      demorton3(tag_anchor(ko), ox, oy, oz);
      oc[0] = ox;
      oc[1] = oy;
      oc[2] = oz;
#pragma unroll
      for (int a = 0; a < 3; a++) ok = ok && ((kb >> a & 1) ? (oc[a] + ho == dom) : (oc[a] == v[a]));
    }
    const unsigned bo = ((oc[0] + ho == dom) ? 1u : 0u) | ((oc[1] + ho == dom) ? 2u : 0u) | ((oc[2] + ho == dom) ? 4u : 0u);
    const unsigned hmo = (meta[o] >> 16) & 255u;
    ok = ok && ((kb & bo) == kb) && !(hmo >> kb & 1);
    unsigned rank = 0;
    for (unsigned q = 0; q < kb; q++)
      if ((q & bo) == q && !(hmo >> q & 1)) rank++;
    uint64_t id = base[o] + rank;
    if (!ok || id >= n_node) {
      atomicOr(flags, DGF_NOT_BALANCED);
      id = 0;
    }
    conn[(size_t)k * n + e] = (uint32_t)id;
  }
}

// ------------------------------------------------------------------------
// element loop tables: families of siblings, their lattices, and the nodes
// of each patch of families (layout: dg_elem.cuh)
// ------------------------------------------------------------------------
// a family's first element: the lowest child of its parent that is a leaf
// (children before e: e - 1 in the usual case, else look-ups)
__global__ void k_family_heads(const Key128 *__restrict__ keys, size_t n, const uint32_t *__restrict__ tab,
                               uint64_t mask, unsigned D, uint32_t *__restrict__ head) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const Key128 ke = keys[e];
  const unsigned l = tag_level(ke);
  bool first = true;
  if (l > 0) {
    const Key128 a = tag_anchor(ke);
    const unsigned sh = 3 * (D - l);
    const unsigned c = (unsigned)(key_shr(a, sh).lo & 7u);
    if (c > 0 && e > 0) {
      const Key128 kp = keys[e - 1];
      first = !(tag_level(kp) == l && key_eq(key_shr(tag_anchor(kp), sh + 3), key_shr(a, sh + 3)));
      if (first) {
        for (unsigned q = 0; q < c && first; q++) {
          const uint32_t j =
              anchor_find(keys, tab, mask, key_xor(a, key_shl(Key128{(uint64_t)(q ^ c), 0}, sh)));
          first = !(j != AH_EMPTY && tag_level(keys[j]) == l);
        }
      }
    }
  }
  head[e] = first ? 1u : 0u;
}

__global__ void k_family_list(const uint32_t *__restrict__ head, const uint32_t *__restrict__ pos, size_t n,
                              uint32_t *__restrict__ first) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < n && head[e]) first[pos[e]] = (uint32_t)e;
}

// One block per patch.  Thread t finds family t's children (the element after
// a child is its next sibling, or a look-up tells); complete families move to
// the front; then thread t builds lattice t from the elements' node ids and
// the nodes are numbered through a shared-memory hash table.  The nodes are
// numbered in claim order, for the element loop's shared-memory banks (number
// mod 32; shared FP32 atomic adds at random banks cost about four times those
// at distinct banks, measured 13.7 against 3.3 cycles per warp instruction on
// an SM): the nodes that a warp claims at one lattice point take consecutive
// numbers, so they fall on distinct banks when that warp touches them
// together.  Patches append their nodes to one list (any order).
constexpr int PF_HT = 4096;  // hash slots, more than FAM_MAX_RUN
constexpr uint32_t PF_EMPTY = 0xffffffffu;
static_assert(FAM_MAX_RUN < PF_HT, "a patch's nodes must fit the hash table");

struct PatchFamSmem {
  uint32_t hkey[PF_HT];          // node of each hash slot
  uint32_t node[FAM_MAX_RUN];    // node of each number
  uint16_t num[PF_HT];           // number of each hash slot
  uint32_t child[8][FAM];        // elements of the reordered families
  uint32_t cmask[FAM];
  uint32_t minlev;
  int counter;
  unsigned long long base;
};

__global__ void __launch_bounds__(FAM)
    k_patch_families(const Key128 *__restrict__ keys, size_t n, const uint32_t *__restrict__ tab, uint64_t tmask,
                     unsigned D, const uint32_t *__restrict__ first, size_t n_fam, const uint32_t *__restrict__ meta,
                     const uint32_t *__restrict__ conn, uint4 *__restrict__ fam, uint4 *__restrict__ pinfo,
                     uint32_t *__restrict__ fchild, uint32_t *__restrict__ run_node,
                     uint32_t *__restrict__ node_patches, unsigned long long *__restrict__ n_run,
                     uint32_t *__restrict__ max_run) {
  extern __shared__ __align__(16) unsigned char pf_raw[];
  PatchFamSmem &S = *reinterpret_cast<PatchFamSmem *>(pf_raw);
  const int t = threadIdx.x, lane = t & 31;
  const size_t p = blockIdx.x, f = p * FAM + t;
  const bool have = f < n_fam;
  for (int i = t; i < PF_HT; i += FAM) S.hkey[i] = PF_EMPTY;
  if (t == 0) {
    S.counter = 0;
    S.minlev = 31;
  }
  // 1. the family's children
  uint32_t el[8], mask = 0;
#pragma unroll
  for (int c = 0; c < 8; c++) el[c] = 0;
  if (have) {
    const uint32_t e0 = first[f];
    const Key128 a = tag_anchor(keys[e0]);
    const unsigned l = tag_level(keys[e0]);
    if (l == 0) {
      el[0] = e0;
      mask = 1;
    } else {
      const unsigned sh = 3 * (D - l);
      const unsigned c0 = (unsigned)(key_shr(a, sh).lo & 7u);
      const Key128 par = key_shr(a, sh + 3);
      uint32_t prev = e0;
#pragma unroll
      for (unsigned c = 0; c < 8; c++) {
        if (c < c0) continue;
        uint32_t e = c == c0 ? e0 : prev + 1;
        bool ok = c == c0;
        if (!ok && e < n) {
          const Key128 k = keys[e];
          const Key128 s = key_shr(tag_anchor(k), sh);
          ok = tag_level(k) == l && (unsigned)(s.lo & 7u) == c && key_eq(key_shr(s, 3), par);
        }
        if (!ok) {
          e = anchor_find(keys, tab, tmask, key_xor(a, key_shl(Key128{(uint64_t)(c ^ c0), 0}, sh)));
          ok = e != AH_EMPTY && tag_level(keys[e]) == l;
        }
        if (ok) {
          el[c] = e;
          mask |= 1u << c;
          prev = e;
        }
      }
    }
  }
  // 2. complete families first
  int n_whole;
  const int whole = have && mask == 255u ? 1 : 0;
  const int before = block_excl_scan<int, FAM>(whole, n_whole);
  const int at = whole ? before : n_whole + (t - before);
  S.cmask[at] = mask;
#pragma unroll
  for (int c = 0; c < 8; c++) S.child[c][at] = el[c];
  __syncthreads();
  mask = S.cmask[t];
#pragma unroll
  for (int c = 0; c < 8; c++) el[c] = S.child[c][t];
  // 3. the lattice: node ids and hanging points
  uint32_t lat[27], hang = 0, lev = 0;
#pragma unroll
  for (int i = 0; i < 27; i++) lat[i] = PF_EMPTY;
#pragma unroll
  for (int c = 0; c < 8; c++) {
    if (!(mask >> c & 1u)) continue;
    const uint32_t me = meta[el[c]];
    lev = me & 255u;
    const uint32_t hm = me >> 16 & 255u;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int bit = hang_bit(lat_vertex(c, k));
      if (bit >= 0 && (hm >> k & 1u)) {
        hang |= 1u << (bit & 31);
        if (lat[lat_corner(k)] == PF_EMPTY) lat[lat_corner(k)] = conn[(size_t)k * n + el[c]];
      } else if (lat[lat_vertex(c, k)] == PF_EMPTY) {
        lat[lat_vertex(c, k)] = conn[(size_t)k * n + el[c]];
      }
    }
  }
  if (mask) atomicMin(&S.minlev, lev);
  if (have) {
    uint4 *fc = reinterpret_cast<uint4 *>(fchild + 8 * f);
    fc[0] = make_uint4(el[0], el[1], el[2], el[3]);
    fc[1] = make_uint4(el[4], el[5], el[6], el[7]);
  }
  // 4. number the nodes
  uint16_t slot[27];
#pragma unroll
  for (int i = 0; i < 27; i++) {
    const uint32_t g = lat[i];
    uint32_t h = (g * 2654435761u) >> (32 - 12);  // PF_HT = 2^12
    bool won = false;
    if (g != PF_EMPTY) {
      for (int probe = 0; probe < PF_HT; probe++) {
        const uint32_t cur = atomicCAS(&S.hkey[h], PF_EMPTY, g);
        won = cur == PF_EMPTY;
        if (won || cur == g) break;
        h = (h + 1) & (PF_HT - 1);
      }
    }
    slot[i] = (uint16_t)h;
    const unsigned claims = __ballot_sync(0xffffffffu, won);
    if (claims) {
      const int leader = __ffs(claims) - 1;
      int at0 = 0;
      if (lane == leader) at0 = atomicAdd(&S.counter, __popc(claims));
      at0 = __shfl_sync(0xffffffffu, at0, leader);
      if (won) {
        const int u = at0 + __popc(claims & ((1u << lane) - 1u));
        S.num[h] = (uint16_t)(u + 1);
        S.node[u] = g;
      }
    }
  }
  __syncthreads();
  const int nr = S.counter;
  if (t == 0) {
    S.base = atomicAdd(n_run, (unsigned long long)nr);
    atomicMax(max_run, (uint32_t)nr);
    pinfo[p] = make_uint4((uint32_t)S.base, (uint32_t)(S.base >> 32), (uint32_t)nr, S.minlev);
  }
  uint32_t w[16];
#pragma unroll
  for (int i = 0; i < 16; i++) w[i] = 0;
#pragma unroll
  for (int i = 0; i < 27; i++)
    if (lat[i] != PF_EMPTY) w[i >> 1] |= (uint32_t)S.num[slot[i]] << (i & 1 ? 16 : 0);
  w[13] |= lev << 16;
  w[14] = mask | (hang & 0xffffu) << 16;
  w[15] = hang >> 16;
#pragma unroll
  for (int q = 0; q < 4; q++)
    fam[(p * 4 + q) * FAM + t] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
  __syncthreads();
  for (int u = t; u < nr; u += FAM) {
    const uint32_t g = S.node[u];
    run_node[S.base + u] = g;
    atomicAdd(&node_patches[g], 1u);
  }
}

// the run words: node, "no other patch touches it", "on the domain boundary"
__global__ void k_run_flags(const uint32_t *__restrict__ run_node, size_t n_run,
                            const uint32_t *__restrict__ node_patches, const uint32_t *__restrict__ node_xyz, size_t V,
                            uint32_t dom, uint32_t *__restrict__ prun) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_run) return;
  const uint32_t g = run_node[i];
  const uint32_t x = node_xyz[g], y = node_xyz[V + g], z = node_xyz[2 * V + g];
  const bool bdy = x == 0 || y == 0 || z == 0 || x == dom || y == dom || z == dom;
  prun[i] = g | (node_patches[g] == 1u ? PRUN_COMPLETE : 0u) | (bdy ? PRUN_BDY : 0u);
}

// conn from the family tables: child c's vertex k is its lattice point, or
// the parent's corner k where that point hangs
__global__ void __launch_bounds__(FAM) k_conn_from_families(const uint4 *__restrict__ fam,
                                                            const uint4 *__restrict__ pinfo,
                                                            const uint32_t *__restrict__ prun,
                                                            const uint32_t *__restrict__ fchild, size_t n_fam,
                                                            size_t E, uint32_t *__restrict__ conn) {
  const size_t p = blockIdx.x;
  const int t = threadIdx.x;
  if (p * FAM + t >= n_fam) return;
  const uint4 info = pinfo[p];
  const uint32_t *run = prun + ((size_t)info.x | (size_t)info.y << 32);
  uint4 w[4];
#pragma unroll
  for (int q = 0; q < 4; q++) w[q] = fam[(p * 4 + q) * FAM + t];
  const uint32_t mask = fam_mask(w), hang = fam_hang(w);
#pragma unroll
  for (int c = 0; c < 8; c++) {
    if (!(mask >> c & 1u)) continue;
    const size_t e = fchild[8 * (p * FAM + t) + c];
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int bit = hang_bit(lat_vertex(c, k));
      const bool h = bit >= 0 && (hang >> (bit & 31) & 1u);
      const uint32_t u = h ? fam_u16(w, lat_corner(k)) : fam_u16(w, lat_vertex(c, k));
      conn[(size_t)k * E + e] = run[u - 1] & PRUN_NODE;
    }
  }
}

const uint32_t *mesh_conn(Context &ctx, const Mesh &m, DBuf<uint32_t> &tmp) {
  if (!m.compressed) return m.conn;
  tmp.alloc(8 * m.n_elem, ctx.stream);
  ProfScope _prof(ctx, "da_conn_decode", (double)m.n_elem * 32 + (double)m.n_fam * 96 + (double)m.n_run * 4);
  k_conn_from_families<<<(unsigned)m.n_patch, FAM, 0, ctx.stream>>>(m.fam, m.pinfo, m.prun, m.fchild, m.n_fam,
                                                                    m.n_elem, tmp.get());
  DG_LAUNCH_CHECK();
  return tmp.get();
}

size_t mesh_bytes(const Mesh &m) {
  size_t b = m.n_elem * 4 + m.n_node * 12;  // meta, node coordinates
  if (m.conn) b += 8 * m.n_elem * 4;
  b += m.n_patch * (4 * FAM + 1) * sizeof(uint4) + m.n_run * 4 + m.n_fam * 32;  // family tables
  return b;
}

static void mesh_families(Context &ctx, Mesh &m, const Key128 *keys, const uint32_t *atab, uint64_t amask) {
  cudaStream_t s = ctx.stream;
  const size_t n = m.n_elem;
  if (m.n_node >= (size_t)PRUN_BDY) fail(DG_ERR_INVALID_ARG, "DA: too many nodes for the element loop tables");
  DBuf<uint32_t> head(n, s), pos(n, s);
  {
    ProfScope _prof(ctx, "da_family_heads", (double)n * 20);
    k_family_heads<<<grid_for(n, 256), 256, 0, s>>>(keys, n, atab, amask, m.max_depth, head.get());
    DG_LAUNCH_CHECK();
  }
  uint32_t *d_total = reinterpret_cast<uint32_t *>(ctx.d_scratch);
  exclusive_scan<uint32_t, uint32_t>(head.get(), pos.get(), n, d_total, s);
  const size_t nf = read_scalar(ctx, d_total);
  const size_t np = (nf + FAM - 1) / FAM;
  DBuf<uint32_t> first(nf, s), fchild(8 * nf, s), run_node(27 * nf, s), npatch(m.n_node, s);
  {
    ProfScope _prof(ctx, "da_family_list", (double)n * 8 + (double)nf * 4);
    k_family_list<<<grid_for(n, 256), 256, 0, s>>>(head.get(), pos.get(), n, first.get());
    DG_LAUNCH_CHECK();
  }
  head.release();
  pos.release();
  DBuf<uint4> fam(np * 4 * FAM, s), pinfo(np, s);
  DG_CUDA(cudaMemsetAsync(npatch.get(), 0, m.n_node * sizeof(uint32_t), s));
  unsigned long long *d_run = ctx.d_scratch;  // {nodes of all patches, most of one}
  DG_CUDA(cudaMemsetAsync(d_run, 0, 2 * sizeof(unsigned long long), s));
  {
    ProfScope _prof(ctx, "da_patch_families", (double)n * (16 + 4 + 32) + (double)nf * 100);
    ensure_smem_attr(ctx, k_patch_families, (int)sizeof(PatchFamSmem));
    k_patch_families<<<(unsigned)np, FAM, sizeof(PatchFamSmem), s>>>(
        keys, n, atab, amask, m.max_depth, first.get(), nf, m.meta, m.conn, fam.get(), pinfo.get(), fchild.get(),
        run_node.get(), npatch.get(), d_run, reinterpret_cast<uint32_t *>(d_run + 1));
    DG_LAUNCH_CHECK();
  }
  DG_CUDA(cudaMemcpyAsync(ctx.h_scratch, d_run, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
  DG_CUDA(cudaStreamSynchronize(s));
  const size_t nruns = (size_t)ctx.h_scratch[0];
  m.max_run = (int)(uint32_t)ctx.h_scratch[1];
  DBuf<uint32_t> prun(nruns ? nruns : 1, s);
  {
    ProfScope _prof(ctx, "da_run_flags", (double)nruns * 24);
    k_run_flags<<<grid_for(nruns, 256), 256, 0, s>>>(run_node.get(), nruns, npatch.get(), m.node_xyz, m.n_node,
                                                     1u << m.max_depth, prun.get());
    DG_LAUNCH_CHECK();
  }
  m.n_fam = nf;
  m.n_patch = np;
  m.n_run = nruns;
  m.fam = fam.release_ptr();
  m.pinfo = pinfo.release_ptr();
  m.prun = prun.release_ptr();
  m.fchild = fchild.release_ptr();
}

void mesh_build(Context &ctx, const Octree &bal, Mesh &m, bool compress) {
  cudaStream_t s = ctx.stream;
  const size_t n = bal.n;
  const unsigned D = bal.max_depth;
  if (n == 0) fail(DG_ERR_INVALID_ARG, "DA: empty octree");
  if (n >= 0xffffffffull / 8) fail(DG_ERR_INVALID_ARG, "DA: too many elements");
  ensure_stencils(ctx);
  m.max_depth = D;
  m.n_elem = n;
  DBuf<uint32_t> meta(n, s), cnt(n, s);
  // anchor -> element map, at most half full
  size_t cap = 1;
  while (cap < 2 * n) cap <<= 1;
  DBuf<uint32_t> atab(cap, s);
  const uint64_t amask = cap - 1;
  DG_CUDA(cudaMemsetAsync(atab.get(), 0xff, cap * sizeof(uint32_t), s));
  {
    ProfScope _prof(ctx, "da_anchor_map", (double)n * 16 + (double)cap * 4);
    k_anchor_insert<<<grid_for(n, 256), 256, 0, s>>>(bal.keys, n, atab.get(), amask);
    DG_LAUNCH_CHECK();
  }
  DG_CUDA(cudaMemsetAsync(ctx.d_flags, 0, sizeof(uint32_t), s));
  {
    ProfScope _prof(ctx, "da_elems", (double)n * 24);
    k_mesh_elems<<<grid_for(n, 256), 256, 0, s>>>(bal.keys, n, atab.get(), amask, D, ctx.d_etype_of, meta.get(),
                                                 cnt.get(), ctx.d_flags);
  DG_LAUNCH_CHECK();
    }
  DBuf<uint64_t> base(n, s);
  uint64_t *d_total = reinterpret_cast<uint64_t *>(ctx.d_scratch);
  exclusive_scan<uint32_t, uint64_t>(cnt.get(), base.get(), n, d_total, s);
  size_t nn = (size_t)read_scalar(ctx, d_total);
  check_device_flags(ctx, "DA");
  if (nn >= 0xffffffffull) fail(DG_ERR_INVALID_ARG, "DA: too many nodes");
  cnt.release();
  DBuf<uint32_t> conn(8 * n, s), nxyz(3 * (nn ? nn : 1), s);
  {
    ProfScope _prof(ctx, "da_conn", (double)n * 56);
    k_mesh_conn<<<grid_for(n, 256), 256, 0, s>>>(bal.keys, n, atab.get(), amask, D, meta.get(), base.get(), conn.get(),
                                                nxyz.get(),
                                               nxyz.get() + nn, nxyz.get() + 2 * nn, nn, ctx.d_flags);
  DG_LAUNCH_CHECK();
    }
  check_device_flags(ctx, "DA");
  m.n_node = nn;
  m.meta = meta.release_ptr();
  m.conn = conn.release_ptr();
  m.node_xyz = nxyz.release_ptr();
  m.compressed = compress;
  mesh_families(ctx, m, bal.keys, atab.get(), amask);
  if (compress) {  // the element loop needs only the family tables
    cudaFreeAsync(m.conn, s);
    m.conn = nullptr;
  }
}

void mesh_free(Context &ctx, Mesh &m) {
  if (m.meta) cudaFreeAsync(m.meta, ctx.stream);
  if (m.conn) cudaFreeAsync(m.conn, ctx.stream);
  if (m.node_xyz) cudaFreeAsync(m.node_xyz, ctx.stream);
  if (m.fam) cudaFreeAsync(m.fam, ctx.stream);
  if (m.pinfo) cudaFreeAsync(m.pinfo, ctx.stream);
  if (m.prun) cudaFreeAsync(m.prun, ctx.stream);
  if (m.fchild) cudaFreeAsync(m.fchild, ctx.stream);
  m = Mesh();
}

// ------------------------------------------------------------------------
// element loop
// ------------------------------------------------------------------------
// the diagonal table of the element loop for these factors (kept on the
// context until a call with others)
template <typename T>
static const T *diag_table(Context &ctx, double lap_fac, double mass_fac) {
  const bool dbl = std::is_same<T, double>::value;
  Context::DiagTable &t = dbl ? ctx.dtab64 : ctx.dtab32;
  if (!t.p) DG_CUDA(cudaMalloc(&t.p, DTAB_ENTRIES * sizeof(T)));
  if (!t.ok || t.lap != lap_fac || t.mass != mass_fac) {
    k_dtab<T><<<(DTAB_ENTRIES + 127) / 128, 128, 0, ctx.stream>>>(static_cast<T *>(t.p), lap_fac, mass_fac);
    DG_LAUNCH_CHECK();
    t.lap = lap_fac;
    t.mass = mass_fac;
    t.ok = true;
  }
  return static_cast<const T *>(t.p);
}

// blocks of a grid-strided patch kernel
template <typename F>
static unsigned patch_grid(Context &ctx, F *kernel, size_t smem, size_t n_patch) {
  ensure_smem_attr(ctx, kernel, 227 * 1024 - 1024);
  int per_sm = 1;
  DG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, FAM, smem));
  return (unsigned)std::min<size_t>(n_patch, (size_t)std::max(per_sm, 1) * ctx.num_sms);
}

template <typename T, bool DIR>
void launch_family_matvec(Context &ctx, const Mesh &m, const T *x, T *y, double lap_fac, double mass_fac,
                          const char *name, double bytes) {
  const size_t smem = family_smem<T>(m.max_run);
  const unsigned grid = patch_grid(ctx, k_family_matvec<T, DIR, false>, smem, m.n_patch);
  const T *dtab = diag_table<T>(ctx, lap_fac, mass_fac);
  ProfScope _prof(ctx, name, bytes);
  k_family_matvec<T, DIR, false><<<grid, FAM, smem, ctx.stream>>>(m.fam, m.prun, m.pinfo, m.n_fam, m.n_patch,
                                                                  m.max_run, dtab, x, y, nullptr, nullptr);
  DG_LAUNCH_CHECK();
}
template void launch_family_matvec<float, true>(Context &, const Mesh &, const float *, float *, double, double,
                                                const char *, double);
template void launch_family_matvec<double, true>(Context &, const Mesh &, const double *, double *, double, double,
                                                 const char *, double);

void launch_family_matvec_fix(Context &ctx, const Mesh &m, const double *x, double *y, const char *name,
                              double bytes) {
  const size_t smem = 2 * ((size_t)m.max_run + 1) * sizeof(long long);
  const unsigned grid = patch_grid(ctx, k_family_matvec_fix<true>, smem, m.n_patch);
  ProfScope _prof(ctx, name, bytes);
  k_family_matvec_fix<true><<<grid, FAM, smem, ctx.stream>>>(m.fam, m.prun, m.pinfo, m.n_fam, m.n_patch, m.max_run,
                                                             x, y);
  DG_LAUNCH_CHECK();
}

template <typename T>
void mesh_matvec(Context &ctx, const Mesh &m, const T *x, T *y, double lap_fac, double mass_fac) {
  DG_CUDA(cudaMemsetAsync(y, 0, m.n_node * sizeof(T), ctx.stream));
  launch_family_matvec<T, false>(ctx, m, x, y, lap_fac, mass_fac, sizeof(T) == 4 ? "matvec_fp32" : "matvec_fp64",
                                 (double)m.n_elem * 36 + (double)m.n_node * 3 * sizeof(T));
}
template void mesh_matvec<float>(Context &, const Mesh &, const float *, float *, double, double);
template void mesh_matvec<double>(Context &, const Mesh &, const double *, double *, double, double);

template <typename T>
void mesh_matvec_coef(Context &ctx, const Mesh &m, const double *coef, const T *x, T *y) {
  DG_CUDA(cudaMemsetAsync(y, 0, m.n_node * sizeof(T), ctx.stream));
  const size_t smem = family_smem<T>(m.max_run);
  const unsigned grid = patch_grid(ctx, k_family_matvec<T, false, true>, smem, m.n_patch);
  ProfScope _prof(ctx, sizeof(T) == 4 ? "matvec_coef_fp32" : "matvec_coef_fp64",
                  (double)m.n_elem * (36 + 16 + 2) + (double)m.n_node * 3 * sizeof(T));
  k_family_matvec<T, false, true><<<grid, FAM, smem, ctx.stream>>>(m.fam, m.prun, m.pinfo, m.n_fam, m.n_patch,
                                                                   m.max_run, nullptr, x, y, coef, m.fchild);
  DG_LAUNCH_CHECK();
}
template void mesh_matvec_coef<float>(Context &, const Mesh &, const double *, const float *, float *);
template void mesh_matvec_coef<double>(Context &, const Mesh &, const double *, const double *, double *);

// diagonal entries per element, added atomically (a node's sum is over the
// elements that hold it)
__global__ void k_mesh_diag(const uint32_t *__restrict__ meta, const uint32_t *__restrict__ conn, size_t E,
                            const double *__restrict__ sten, const double *__restrict__ coef, double lap_fac,
                            double mass_fac, double *__restrict__ diag) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= E) return;
  const uint32_t me = meta[e];
  const unsigned l = me & 255u, c = (me >> 8) & 7u, t = me >> 24;
  const double h = 1.0 / (double)(1ull << l);
  const double lf = coef ? coef[2 * e] : lap_fac, mf = coef ? coef[2 * e + 1] : mass_fac;
  const double f1 = lf * h / 2.0, f2 = mf * h * h * h / 8.0;
  const double *S = sten + (c * 18 + t) * 128;
#pragma unroll
  for (int k = 0; k < 8; k++) atomicAdd(&diag[conn[(size_t)k * E + e]], f1 * S[9 * k] + f2 * S[64 + 9 * k]);
}

void mesh_diagonal(Context &ctx, const Mesh &m, const double *coef, double lap_fac, double mass_fac, double *diag) {
  ensure_stencils(ctx);
  cudaStream_t s = ctx.stream;
  DG_CUDA(cudaMemsetAsync(diag, 0, m.n_node * sizeof(double), s));
  if (!m.n_elem) return;
  DBuf<uint32_t> tmp;
  const uint32_t *conn = mesh_conn(ctx, m, tmp);
  ProfScope _prof(ctx, "mesh_diagonal", (double)m.n_elem * (4 + 32 + (coef ? 16 : 0)) + (double)m.n_node * 8);
  k_mesh_diag<<<grid_for(m.n_elem, 256), 256, 0, s>>>(m.meta, conn, m.n_elem, ctx.d_sten64, coef, lap_fac, mass_fac,
                                                       diag);
  DG_LAUNCH_CHECK();
}

}  // namespace dg

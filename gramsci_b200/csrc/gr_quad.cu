// 4PCF 4-clique counting: replaces query_4pcf_all2 (src/gramsci.F90:662-825),
// whose per-root triple loop performs three find_dist binary searches per
// candidate triple, and the -tetra counter query_graph_tetrahedron
// (:548-660).
//
// Every 4-clique is enumerated exactly once, from its smallest label p.  A
// warp takes roots from a work counter and stages R+(p) in shared memory
// (catalogue id, flags, weight, row start and length of every neighbour)
// with a per-root hash table (label offset -> row position).  For each a in
// R+(p) it builds X = R+(a) ∩ R+(p) beyond a's position, as a compacted list
// and a bitmask over R+(p)'s positions; then the work items (b, d) for b in X
// and d in R+(b) are flattened over the lanes (warp OR-reduction owners, as
// in the triangle kernel), d is looked up in the hash table and tested in
// the bitmask, and hits (cliques p < a < b < d) are queued and binned 32 at
// a time with all their data in shared memory.  A clique contributes, for
// every vertex r that is a root in the reference (not a buffer point, row
// length > 3), with the other three vertices taken in catalogue-id order
// (k1 < k2 < k3 of the reference), if the perimeter r-k1-k2-k3-r is
// canonical (bintable entry > 0), to N2 / N3 at (cfg, bin(r,k2), bin(k1,k3))
// and to the six disconnected pair terms.
//
// A second kernel (quad4g_kernel, the geometric mode) finds the edges among
// the members of R+(p) with the graph's own membership test on their
// positions instead of probing the members' rows; it is used whenever the
// rows fit (up to 256 members).
#include <algorithm>
#include <type_traits>

#include "gr_kernels.cuh"

namespace gr {

namespace {

constexpr int kQuadMaxWarps = 16;   // weighted / adjoint kernels (up to 128 registers)
constexpr int kQuadMaxWarpsU = 24;  // unweighted kernels (up to 85 registers)
#ifndef GR_QUADG_WEIGHTED_WARPS
#define GR_QUADG_WEIGHTED_WARPS 24
#endif
// Weighted geometric kernel: 24 warps (at most 85 registers, a few bytes
// spilled).  (The high limb of a sum in the low limb's line instead of a line of
// its own made the kernel 2% slower.)
constexpr int kQuadGWarpsW = GR_QUADG_WEIGHTED_WARPS;
// Geometric adjoint kernel: 24 warps too (13 warps: 5.5 against 3.2 ms).
constexpr int kQuadGWarpsA = 24;
constexpr size_t kQuadSmemLimit = 227 * 1024;
constexpr int kQQueue = 96;         // hit queue entries per warp (< 32 left + 64 pushed)
constexpr int kQMaxOffset = 1 << 22;  // hash entries: (label offset << 10) | position
constexpr uint8_t kFlagDeg4 = 4;    // staged flag: full row length > 3 (a reference root)
// The longest rows (a root's cost grows with the cube of its row length) are
// handed out as several work items each, every item staging the root in full
// and taking its share of the member pairs (geometric kernel) or of the first
// members (hash kernel): a heavy root on one warp otherwise ends the launch
// alone.  A row of 32 is one unit of work; longer ones take about as many
// parts as they have units, by the classes below, where the launch's warps
// outnumber the rows to split (in catalogues with more such rows than warps
// the shares would only repeat the staging).
constexpr int kSplitClasses = 5;
__host__ __device__ constexpr int split_row(int j) {
  return j == 0 ? 128 : (j == 1 ? 96 : (j == 2 ? 64 : (j == 3 ? 48 : 32)));
}
__host__ __device__ constexpr int split_parts(int j) {
  return j == 0 ? 64 : (j == 1 ? 32 : (j == 2 ? 16 : (j == 3 ? 4 : 2)));
}

// A window of slots (places in QuadParams::order): all rows, or, when some of
// a block's warps take the long ones (QuadParams::long_warps), those of at
// least kShortRow members (phase 0) or the others (phase 1); end[j]: slots
// before which rows of split class j end, relative to start.
constexpr int kShortRow = 64;
struct QuadWindow {
  int start, stop, end[kSplitClasses];
};
__device__ __forceinline__ QuadWindow quad_window(const QuadParams& Q, int n, int phase,
                                                  bool split = true) {
  QuadWindow W;
  W.start = 0;
  W.stop = n;
#pragma unroll
  for (int j = 0; j < kSplitClasses; ++j) W.end[j] = 0;
  if (!Q.order || !Q.above) return W;
  // above[b]: the number of rows with at least b members
  if (Q.long_warps > 0) {
    const int nlong = Q.above[kShortRow];
    if (phase == 0)
      W.stop = nlong;
    else
      W.start = nlong;
  }
  if (!split) return W;
  const int limit = (int)gridDim.x * (int)(blockDim.x >> 5);
#pragma unroll
  for (int j = 0; j < kSplitClasses; ++j)
    if (split_row(j) < Q.nclass)
      W.end[j] = max(0, min(min(Q.above[split_row(j)], W.stop) - W.start, limit));
  return W;
}
// The root, part and number of parts of work item `item`; false past the
// last root.
__device__ __forceinline__ bool quad_item(const QuadParams& Q, const QuadWindow& W, int item,
                                          int& p, int& part, int& nparts) {
  int slot = 0, first = 0;  // first slot of the class, and its first item
  part = 0;
  nparts = 1;
  bool done = false;
#pragma unroll
  for (int j = 0; j < kSplitClasses; ++j) {
    const int rows = W.end[j] - slot, items = rows * split_parts(j);
    if (!done && item < first + items) {
      const int i = (item - first) / split_parts(j);
      part = item - first - i * split_parts(j);
      nparts = split_parts(j);
      slot += i;
      done = true;
    }
    if (!done) {
      slot = W.end[j];
      first += items;
    }
  }
  if (!done) slot += item - first;
  slot += W.start;
  if (slot >= W.stop) return false;
  p = Q.order ? Q.order[slot] : slot;
  return true;
}

__host__ __device__ inline size_t qalign8(size_t x) { return (x + 7) & ~(size_t)7; }

__host__ __device__ inline int qhash_lg_max(int cap) {
  int lg = 6;
  while ((1 << lg) < 4 * cap) ++lg;
  return lg;
}

struct QuadLayout {
  size_t off_rank, off_cnt, off_warp, warp_bytes, total;
  // per-warp sub-offsets
  size_t o_rs, o_w, o_mo, o_g, o_col, o_len, o_xm, o_hkey, o_q, o_xy, o_xz, o_bits;
};

// ncounts: block-private 32-bit counters in shared memory (0: none);
// adj: per-neighbour 128-bit gradient accumulators (adjoint mode)
__host__ __device__ inline QuadLayout quad_layout(int nbins, int cap, int nwarps, int ncounts,
                                                  bool adj = false) {
  QuadLayout L;
  size_t o = 0;
  L.off_rank = o;
  o = qalign8(o + sizeof(int) * 4 * (size_t)(nbins + 2));
  L.off_cnt = o;
  o = qalign8(o + sizeof(unsigned int) * (size_t)ncounts);
  L.off_warp = o;
  size_t w = 0;
  L.o_rs = w;   w += (size_t)cap * 8;   // row start of each neighbour
  L.o_w = w;    w += (size_t)cap * 8;   // weight
  L.o_mo = w;   w += (size_t)cap * 8;   // (catalogue id << 32) | flags << 24 | meta(p, a)
  L.o_g = w;    w += adj ? (size_t)cap * 16 : 0;  // 128-bit gradient of each neighbour
  L.o_col = w;  w += (size_t)cap * 4;   // label
  L.o_len = w;  w += (size_t)cap * 4;   // row length
  L.o_xm = w;   w += (size_t)cap * 4;   // X entry z: meta(a, b)
  L.o_hkey = w; w += (size_t)(1u << qhash_lg_max(cap)) * 4;
  L.o_q = w;    w += (size_t)kQQueue * 8;
  L.o_xy = w;   w += (size_t)cap * 2;   // X entry z: position of b in R+(p)
  L.o_xz = w;   w += (size_t)cap * 2;   // position y: X entry (when its bit is set)
  L.o_bits = w; w += (size_t)((cap + 31) / 32) * 4;
  L.warp_bytes = qalign8(w);
  L.total = o + L.warp_bytes * nwarps;
  return L;
}

struct QuadCtx {
  const int* F;  // 4 x (nbins+2)
  int nbins, ncfg, nbin, tetra;
  unsigned long long *cnt, *dcnt;
  unsigned int *scnt, *sdcnt;  // block-private 32-bit counts in shared memory, or null
  unsigned long long *fix, *dfix;  // fixed-point (lo, hi) sums, hi at +5*nbin / +dhi
  int dhi;                          // disc entries on the device (hi offset in dfix)
  int split;                        // 1: sums as split limbs (fix_red), 0: carries (fix_add)
  int counts;                       // 0: weighted sums only, no integer counts
  double fscale;  // scale of the 4-point products
  double dscale;  // scale of the pair products of the disconnected terms
  const double* cot;  // adjoint: a line of cotangents per histogram index (quad_cot_lines)
};

// Logical entry i of a global fixed-point array: one entry per kFixStride
// 8-byte words, so that every entry has a 128-byte line of its own.  The
// hottest bins are neighbours in the dense order; packed 16 to a line they
// were served by a few L2 slices, and the weighted 4PCF kernel's time then
// depended on where the arrays happened to lie (measured 5.4 to 6.9 ms for
// the same launch as the arrays were moved in steps of 4 KB).
__device__ __forceinline__ unsigned long long* qfx(unsigned long long* a, int i) {
  return a + (size_t)i * kFixStride;
}

// one weighted update of a global fixed-point sum
__device__ __forceinline__ void qfix(const QuadCtx& X, unsigned long long* lo, unsigned long long* hi,
                                     double x, double scale) {
  if (X.split)
    fix_red(lo, hi, x, scale);
  else
    fix_add(lo, hi, x, scale);
}

template <bool SHC>
__device__ __forceinline__ void qcount(const QuadCtx& X, int k) {
  if (SHC) atomicAdd(&X.scnt[k], 1u);
  else if (X.counts) atomicAdd(&X.cnt[k], 1ull);
}
template <bool SHC>
__device__ __forceinline__ void qdcount(const QuadCtx& X, int k) {
  if (SHC) atomicAdd(&X.sdcnt[k], 1u);
  else if (X.counts) atomicAdd(&X.dcnt[k], 1ull);
}

// The four vertices of a clique: flags (with kFlagDeg4), catalogue ids and
// weights.
struct QVerts {
  uint8_t fl[4];
  int og[4];
  double w[4];
};

// Disconnected term t (t = 1..6 of gramsci.F90:754-818, here 0..5): the
// role whose randomness gates it and the two roles of its pair product
// (roles: 0 = root, 1..3 = the other vertices in catalogue-id order).  The
// -tetra terms (:591-646) use the same gate with the 3-product (gate, pu, pv).
// Written as functions of a loop index that is unrolled, so every use folds
// to a constant and no table is indexed at run time.
__host__ __device__ constexpr int term_gate(int t) { return t < 2 ? 3 : (t == 2 ? 1 : 0); }
__host__ __device__ constexpr int term_pu(int t) { return t < 3 ? 0 : (t == 3 ? 1 : 3); }
__host__ __device__ constexpr int term_pv(int t) { return t < 3 ? t + 1 : (t == 5 ? 1 : 2); }

// index (0..5) of the clique edge between vertices u != v: (0,1) (0,2) (0,3)
// (1,2) (1,3) (2,3)
__device__ __forceinline__ int qedge(int u, int v) {
  const int a = min(u, v), b = max(u, v);
  return a * (7 - a) / 2 - 1 + b - a;
}
// radial bin of edge (u, v) from the six bins packed a byte each
__device__ __forceinline__ int qbin(unsigned long long packed, int u, int v) {
  return (int)((packed >> (8 * qedge(u, v))) & 0xffull);
}
__device__ __forceinline__ double qsel(int i, const QVerts& V) {
  return i == 0 ? V.w[0] : (i == 1 ? V.w[1] : (i == 2 ? V.w[2] : V.w[3]));
}

// The three vertices other than root r, ordered by catalogue id (the
// reference's id-sorted row): a three-element sorting network on registers.
template <int R>
__device__ __forceinline__ void others_by_id(const QVerts& V, int& u0, int& u1, int& u2) {
  constexpr int O0 = R == 0 ? 1 : 0, O1 = R <= 1 ? 2 : 1, O2 = R <= 2 ? 3 : 2;
  int g0 = V.og[O0], g1 = V.og[O1], g2 = V.og[O2];
  u0 = O0;
  u1 = O1;
  u2 = O2;
  int t;
  if (g0 > g1) { t = g0; g0 = g1; g1 = t; t = u0; u0 = u1; u1 = t; }
  if (g1 > g2) { t = g1; g1 = g2; g2 = t; t = u1; u1 = u2; u2 = t; }
  if (g0 > g1) { t = g0; g0 = g1; g1 = t; t = u0; u0 = u1; u1 = t; }
}

// query_graph_tetrahedron: a 4-clique with all six edges in bin b counts from
// each non-buffer vertex (no row-length condition).
template <bool WEIGHTED, bool SHC, int R>
__device__ __forceinline__ int tetra_root(const QuadCtx& X, const QVerts& V, int b, unsigned rndm,
                                          int nr) {
  if (V.fl[R] & FLAG_BUFFER) return 0;
  int u0, u1, u2;
  others_by_id<R>(V, u0, u1, u2);
  const int role[4] = {R, u0, u1, u2};
  const int nb = X.nbins;
  qcount<SHC>(X, (b - 1) + nb * nr);
  if (WEIGHTED)
    qfix(X, qfx(X.fix, (b - 1) + nb * nr), qfx(X.fix, (b - 1) + nb * (nr + 5)),
            ((V.w[R] * qsel(u0, V)) * qsel(u1, V)) * qsel(u2, V), X.fscale);
#pragma unroll
  for (int tt = 0; tt < 6; ++tt) {
    if (!((rndm >> role[term_gate(tt)]) & 1u)) continue;
    const int ua = role[term_gate(tt)], ub = role[term_pu(tt)], uc = role[term_pv(tt)];
    const int nr3 = (int)((rndm >> ua) & 1u) + (int)((rndm >> ub) & 1u) + (int)((rndm >> uc) & 1u);
    const int kt = (b - 1) + nb * tt;
    const double qv = WEIGHTED ? (qsel(ua, V) * qsel(ub, V)) * qsel(uc, V) : 0.0;
    // discR (all three random) equals category 3 and is copied on the host
    qdcount<SHC>(X, kt + nb * 6 * nr3);
    if (WEIGHTED) qfix(X, qfx(X.dfix, kt + nb * 6 * nr3), qfx(X.dfix, kt + nb * 6 * nr3 + X.dhi), qv, X.dscale);
  }
  return 1;
}

template <bool WEIGHTED, bool SHC>
__device__ __forceinline__ int tetra_contrib(const QuadCtx& X, const QVerts& V, const uint32_t m[6]) {
  const int b = meta_bin(m[0]);
#pragma unroll
  for (int k = 1; k < 6; ++k)
    if (meta_bin(m[k]) != b) return 0;
  unsigned rndm = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) rndm |= (unsigned)(V.fl[k] & FLAG_RANDOM) << k;
  const int nr = __popc(rndm);
  return tetra_root<WEIGHTED, SHC, 0>(X, V, b, rndm, nr) + tetra_root<WEIGHTED, SHC, 1>(X, V, b, rndm, nr) +
         tetra_root<WEIGHTED, SHC, 2>(X, V, b, rndm, nr) + tetra_root<WEIGHTED, SHC, 3>(X, V, b, rndm, nr);
}

// Root R of a 4-clique for query_4pcf_all2: the histogram index of its
// contribution, (cfg, bin(r,k2), bin(k1,k3)) with k1 < k2 < k3 the other
// vertices in catalogue-id order (returned in u0..u2), or -1 when R is no
// root (buffer point, row length <= 3) or its perimeter is not canonical.
template <int R>
__device__ __forceinline__ int quad_root_index(const QuadCtx& X, const QVerts& V,
                                               unsigned long long packed, int& u0, int& u1,
                                               int& u2) {
  if (V.fl[R] & FLAG_BUFFER) return -1;
  if (!(V.fl[R] & kFlagDeg4)) return -1;
  others_by_id<R>(V, u0, u1, u2);
  const int b1 = qbin(packed, R, u0), b2 = qbin(packed, u0, u1), b3 = qbin(packed, u1, u2),
            b4 = qbin(packed, R, u2);
  if (!(b1 <= b2 && b2 <= b3 && b3 <= b4)) return -1;
  const int nb2 = X.nbins + 2;
  const int cfg = 1 + (X.F[b1] - X.F[1]) + (X.F[nb2 + b2] - X.F[nb2 + b1]) +
                  (X.F[2 * nb2 + b3] - X.F[2 * nb2 + b2]) + (X.F[3 * nb2 + b4] - X.F[3 * nb2 + b3]);
  const int d1 = qbin(packed, R, u1), d2 = qbin(packed, u0, u2);
  return (cfg - 1) + X.ncfg * ((d1 - 1) + X.nbins * (d2 - 1));
}

// N2 / N3 and the six disconnected terms of root R.  Unit weights: one
// count at (histogram index, randomness of the four roles) instead, the
// pattern histogram from which quad_expand_patterns forms the N2 / N3 and
// disconnected-term counts (which roles are random decides the category of
// each and which terms are gated in).
template <bool WEIGHTED, bool SHC, int R>
__device__ __forceinline__ int quad_root(const QuadCtx& X, const QVerts& V, unsigned long long packed,
                                         unsigned rndm, int nr) {
  int u0, u1, u2;
  const int kk = quad_root_index<R>(X, V, packed, u0, u1, u2);
  if (kk < 0) return 0;
  if constexpr (!WEIGHTED) {
    const unsigned pat = ((rndm >> R) & 1u) | (((rndm >> u0) & 1u) << 1) |
                         (((rndm >> u1) & 1u) << 2) | (((rndm >> u2) & 1u) << 3);
    qcount<SHC>(X, kk + X.nbin * (int)pat);
    return 1;
  }
  qcount<SHC>(X, kk + X.nbin * nr);
  if (WEIGHTED)
    qfix(X, qfx(X.fix, kk + X.nbin * nr), qfx(X.fix, kk + X.nbin * (nr + 5)),
            ((V.w[R] * qsel(u0, V)) * qsel(u1, V)) * qsel(u2, V), X.fscale);
  const int role[4] = {R, u0, u1, u2};
#pragma unroll
  for (int tt = 0; tt < 6; ++tt) {
    if (!((rndm >> role[term_gate(tt)]) & 1u)) continue;
    const int u = role[term_pu(tt)], vv = role[term_pv(tt)];
    const int npr = (int)((rndm >> u) & 1u) + (int)((rndm >> vv) & 1u);
    const int kt = kk + X.nbin * tt;
    const double q = WEIGHTED ? qsel(u, V) * qsel(vv, V) : 0.0;
    // discR (both random) equals category 2 and is copied on the host
    qdcount<SHC>(X, kt + X.nbin * 6 * npr);
    if (WEIGHTED)
      qfix(X, qfx(X.dfix, kt + X.nbin * 6 * npr), qfx(X.dfix, kt + X.nbin * 6 * npr + X.dhi), q, X.dscale);
  }
  return 1;
}

// m: bins of (0,1) (0,2) (0,3) (1,2) (1,3) (2,3) for vertices 0 = p, 1 = a,
// 2 = b, 3 = d.
template <bool WEIGHTED, bool SHC>
__device__ __forceinline__ int quad_contrib(const QuadCtx& X, const QVerts& V, const uint32_t m[6]) {
  unsigned long long packed = 0;
#pragma unroll
  for (int e = 0; e < 6; ++e) packed |= (unsigned long long)meta_bin(m[e]) << (8 * e);
  unsigned rndm = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) rndm |= (unsigned)(V.fl[k] & FLAG_RANDOM) << k;
  const int nr = __popc(rndm);
  return quad_root<WEIGHTED, SHC, 0>(X, V, packed, rndm, nr) + quad_root<WEIGHTED, SHC, 1>(X, V, packed, rndm, nr) +
         quad_root<WEIGHTED, SHC, 2>(X, V, packed, rndm, nr) + quad_root<WEIGHTED, SHC, 3>(X, V, packed, rndm, nr);
}

// Vertex indices 0..3 in ascending catalogue id, two bits each (the
// register sorting network the flattened drain and the gradient use).
__device__ __forceinline__ unsigned id_order(const QVerts& V) {
  int g0 = V.og[0], g1 = V.og[1], g2 = V.og[2], g3 = V.og[3];
  unsigned a0 = 0, a1 = 1, a2 = 2, a3 = 3;
  auto cx = [](int& ga, int& gb, unsigned& ia, unsigned& ib) {
    if (ga > gb) {
      const int t = ga; ga = gb; gb = t;
      const unsigned u = ia; ia = ib; ib = u;
    }
  };
  cx(g0, g1, a0, a1);
  cx(g2, g3, a2, a3);
  cx(g0, g2, a0, a2);
  cx(g1, g3, a1, a3);
  cx(g1, g2, a1, a2);
  return a0 | (a1 << 2) | (a2 << 4) | (a3 << 6);
}

// Gradient of one root's cotangent-weighted sums with respect to the weights
// of its four roles (0 = root, 1..3 = the other vertices in catalogue-id
// order; rb: whether each is a random): the sums are multilinear, so the
// 4-product contributes its cotangent times the product of the other three
// weights, a pair term its cotangent times the partner's weight.  Both
// 4-clique kernels round these four numbers to the fixed point, so their
// gradients are identical.
__device__ __forceinline__ void quad_root_grad(const QuadCtx& X, int kr, const unsigned rb[4],
                                               const double w[4], double g[4]) {
  const double* c = X.cot + (size_t)kr * kCotLine;
  const double c4 = __ldg(c + (rb[0] && rb[1] && rb[2] && rb[3] ? 1 : 0));
  double D[6];
#pragma unroll
  for (int tt = 0; tt < 6; ++tt) {
    D[tt] = 0.0;
    if (rb[term_gate(tt)]) D[tt] = __ldg(c + (rb[term_pu(tt)] && rb[term_pv(tt)] ? 8 : 2) + tt);
  }
  // terms: 0 (0,1) 1 (0,2) 2 (0,3) 3 (1,2) 4 (3,2) 5 (3,1)
  g[0] = c4 * (w[1] * w[2] * w[3]) + D[0] * w[1] + D[1] * w[2] + D[2] * w[3];
  g[1] = c4 * (w[0] * w[2] * w[3]) + D[0] * w[0] + D[3] * w[2] + D[5] * w[3];
  g[2] = c4 * (w[0] * w[1] * w[3]) + D[1] * w[0] + D[3] * w[1] + D[4] * w[3];
  g[3] = c4 * (w[0] * w[1] * w[2]) + D[2] * w[0] + D[5] * w[1] + D[4] * w[2];
}

// The weight gradient of one clique (vertices as in quad_contrib) from each
// of its valid roots: vertex 0's to racc, the others' to the accumulators at
// positions ya, yb, yd.  The roots are a loop that is not unrolled (unrolled,
// the code overflowed the instruction cache).  Returns the number of roots.
__device__ __forceinline__ int quad_grad_c(const QuadCtx& X, const QVerts& V, const uint32_t m[6],
                                           double gscale, Fix128& racc, unsigned* s_grad, int gcap,
                                           int ya, int yb, int yd) {
  unsigned long long packed = 0;
#pragma unroll
  for (int e = 0; e < 6; ++e) packed |= (unsigned long long)meta_bin(m[e]) << (8 * e);
  unsigned rndm = 0, flw = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    rndm |= (unsigned)(V.fl[k] & FLAG_RANDOM) << k;
    flw |= (unsigned)V.fl[k] << (8 * k);
  }
  const unsigned perm = id_order(V);
  int n = 0;
#pragma unroll 1
  for (int R = 0; R < 4; ++R) {
    const unsigned fr = flw >> (8 * R);
    if ((fr & FLAG_BUFFER) || !(fr & kFlagDeg4)) continue;
    int pos = 0;
#pragma unroll
    for (int i = 1; i < 4; ++i)
      if ((int)((perm >> (2 * i)) & 3u) == R) pos = i;
    const unsigned lowm = (1u << (2 * pos)) - 1u;
    const unsigned oth = (perm & lowm) | ((perm >> (2 * pos + 2)) << (2 * pos));
    const int u0 = (int)(oth & 3u), u1 = (int)((oth >> 2) & 3u), u2 = (int)((oth >> 4) & 3u);
    const int b1 = qbin(packed, R, u0), b2 = qbin(packed, u0, u1), b3 = qbin(packed, u1, u2),
              b4 = qbin(packed, R, u2);
    if (!(b1 <= b2 && b2 <= b3 && b3 <= b4)) continue;
    const int nb2 = X.nbins + 2;
    const int cfg = 1 + (X.F[b1] - X.F[1]) + (X.F[nb2 + b2] - X.F[nb2 + b1]) +
                    (X.F[2 * nb2 + b3] - X.F[2 * nb2 + b2]) + (X.F[3 * nb2 + b4] - X.F[3 * nb2 + b3]);
    const int d1 = qbin(packed, R, u1), d2 = qbin(packed, u0, u2);
    const int kk = (cfg - 1) + X.ncfg * ((d1 - 1) + X.nbins * (d2 - 1));
    ++n;
    const int v[4] = {R, u0, u1, u2};
    unsigned rb[4];
    double w[4], g[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      rb[j] = (rndm >> v[j]) & 1u;
      w[j] = qsel(v[j], V);
    }
    quad_root_grad(X, kk, rb, w, g);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (v[j] == 0)
        fix_acc(racc, g[j], gscale);
      else
        smem_fix_add(s_grad + (v[j] == 1 ? ya : (v[j] == 2 ? yb : yd)), gcap,
                     __double2ll_rn(g[j] * gscale));
    }
  }
  return n;
}

__device__ __forceinline__ uint32_t qfib_slot(uint32_t off, int lg) {
  return (off * 2654435769u) >> (32 - lg);
}

// Block-level context shared by the 4-clique kernels: rank tables in shared
// memory, output pointers, block-private counters (SHC), cotangents (ADJ).
template <bool SHC, bool ADJ>
__device__ __forceinline__ void quad_setup(QuadCtx& X, const QuadParams& Q, unsigned char* rank_smem,
                                           unsigned char* cnt_smem, unsigned long long* g_cnt,
                                           unsigned long long* g_fix, unsigned long long* d_cnt,
                                           unsigned long long* d_fix, int nh, int nd,
                                           double fscale, double dscale, const double* cot) {
  int* s_F = reinterpret_cast<int*>(rank_smem);
  const int nb2 = Q.nbins + 2;
  for (int k = threadIdx.x; k < 4 * nb2; k += blockDim.x) s_F[k] = Q.rank.F[k / nb2][k % nb2];
  __syncthreads();
  X.F = s_F;
  X.nbins = Q.nbins;
  X.ncfg = Q.ncfg;
  X.nbin = Q.tetra ? Q.nbins : Q.ncfg * Q.nbins * Q.nbins;
  X.tetra = Q.tetra;
  X.cnt = g_cnt;
  X.dcnt = d_cnt;
  X.fix = g_fix;
  X.dfix = d_fix;
  X.dhi = nd;
  X.split = Q.split;
  X.counts = Q.counts;
  X.scnt = nullptr;
  X.sdcnt = nullptr;
  if (SHC) {
    unsigned int* sc = reinterpret_cast<unsigned int*>(cnt_smem);
    for (int k = threadIdx.x; k < nh + nd; k += blockDim.x) sc[k] = 0u;
    __syncthreads();
    X.scnt = sc;
    X.sdcnt = sc + nh;
  }
  X.fscale = fscale;
  X.dscale = dscale;
  X.cot = cot;
}

// Weighted 4PCF contributions of the warp's cliques, flattened: every lane
// first evaluates the four roots of its clique (act: the lane holds one)
// without branching -- root validity, histogram index and the other three
// vertices in catalogue-id order -- then the warp takes the valid (clique,
// root) pairs 32 at a time, every lane updating one root's N2 / N3 sum and
// its gated pair terms.  The compact per-clique loops diverge (a quarter of
// the lanes active on average); here every lane is busy in both stages.
// The pairs are ordered by root index, then lane: one ballot per root index
// gives each pair's lane with no search, and the vertex weights are read
// from the staged weights (s_w at the positions packed 10 bits each in vpos
// for vertices 1..3; vertex 0 is the warp's root, weight wp).  Products and
// histogram indices are those of quad_root.
// Returns this lane's number of rooted contributions.
template <bool SHC>
__device__ __forceinline__ int quad_contrib_flat(const QuadCtx& X, const QVerts& V,
                                                 const uint32_t m[6], bool act, unsigned vpos,
                                                 const double* s_w, double wp) {
  const int lane = threadIdx.x & 31;
  unsigned long long packed = 0;
#pragma unroll
  for (int e = 0; e < 6; ++e) packed |= (unsigned long long)meta_bin(m[e]) << (8 * e);
  unsigned rndm = 0, flw = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    rndm |= (unsigned)(V.fl[k] & FLAG_RANDOM) << k;
    flw |= (unsigned)V.fl[k] << (8 * k);
  }
  const unsigned perm = id_order(V);
  // stage 1: the four roots of this lane's clique
  unsigned vm = 0, rpk = 0;
  int kk[4];
#pragma unroll
  for (int R = 0; R < 4; ++R) {
    kk[R] = 0;
    const unsigned fr = flw >> (8 * R);
    int pos = 0;
#pragma unroll
    for (int i = 1; i < 4; ++i)
      if ((int)((perm >> (2 * i)) & 3u) == R) pos = i;
    const unsigned lowm = (1u << (2 * pos)) - 1u;
    const unsigned oth = (perm & lowm) | ((perm >> (2 * pos + 2)) << (2 * pos));
    const int u0 = (int)(oth & 3u), u1 = (int)((oth >> 2) & 3u), u2 = (int)((oth >> 4) & 3u);
    const int b1 = qbin(packed, R, u0), b2 = qbin(packed, u0, u1), b3 = qbin(packed, u1, u2),
              b4 = qbin(packed, R, u2);
    const bool ok = act && !(fr & FLAG_BUFFER) && (fr & kFlagDeg4) && b1 <= b2 && b2 <= b3 &&
                    b3 <= b4;
    if (ok) {
      const int nb2 = X.nbins + 2;
      const int cfg = 1 + (X.F[b1] - X.F[1]) + (X.F[nb2 + b2] - X.F[nb2 + b1]) +
                      (X.F[2 * nb2 + b3] - X.F[2 * nb2 + b2]) +
                      (X.F[3 * nb2 + b4] - X.F[3 * nb2 + b3]);
      const int d1 = qbin(packed, R, u1), d2 = qbin(packed, u0, u2);
      kk[R] = (cfg - 1) + X.ncfg * ((d1 - 1) + X.nbins * (d2 - 1));
      vm |= 1u << R;
    }
    rpk |= ((unsigned)R | ((unsigned)u0 << 2) | ((unsigned)u1 << 4) | ((unsigned)u2 << 6)) << (8 * R);
  }
  // stage 2: pairs (root index R, lane) in that order
  unsigned mr[4];
  int c0, c1, c2, total;
#pragma unroll
  for (int R = 0; R < 4; ++R) mr[R] = __ballot_sync(0xffffffffu, (vm >> R) & 1u);
  c0 = __popc(mr[0]);
  c1 = c0 + __popc(mr[1]);
  c2 = c1 + __popc(mr[2]);
  total = c2 + __popc(mr[3]);
  for (int i0 = 0; i0 < total; i0 += 32) {
    const int i = i0 + lane;
    const int R = i < c0 ? 0 : (i < c1 ? 1 : (i < c2 ? 2 : 3));
    const int base = R == 0 ? 0 : (R == 1 ? c0 : (R == 2 ? c1 : c2));
    const unsigned mR = R == 0 ? mr[0] : (R == 1 ? mr[1] : (R == 2 ? mr[2] : mr[3]));
    const int o = i < total ? (int)__fns(mR, 0, i - base + 1) : 0;
    // every lane takes part in each shuffle; the select comes after
    const unsigned orp = __shfl_sync(0xffffffffu, rpk, o);
    const unsigned ornd = __shfl_sync(0xffffffffu, rndm, o);
    const unsigned opos = __shfl_sync(0xffffffffu, vpos, o);
    const int k0 = __shfl_sync(0xffffffffu, kk[0], o), k1 = __shfl_sync(0xffffffffu, kk[1], o),
              k2 = __shfl_sync(0xffffffffu, kk[2], o), k3 = __shfl_sync(0xffffffffu, kk[3], o);
    if (i >= total) continue;
    const int kr = R == 0 ? k0 : (R == 1 ? k1 : (R == 2 ? k2 : k3));
    const int onr = __popc(ornd);
    const unsigned rp = (orp >> (8 * R)) & 0xffu;
    const int u0 = (int)((rp >> 2) & 3u), u1 = (int)((rp >> 4) & 3u), u2 = (int)((rp >> 6) & 3u);
    const double w1 = s_w[opos & 0x3ffu], w2 = s_w[(opos >> 10) & 0x3ffu],
                 w3 = s_w[(opos >> 20) & 0x3ffu];
    auto wsel = [&](int v) { return v == 0 ? wp : (v == 1 ? w1 : (v == 2 ? w2 : w3)); };
    qcount<SHC>(X, kr + X.nbin * onr);
    qfix(X, qfx(X.fix, kr + X.nbin * onr), qfx(X.fix, kr + X.nbin * (onr + 5)),
         ((wsel(R) * wsel(u0)) * wsel(u1)) * wsel(u2), X.fscale);
#pragma unroll
    for (int tt = 0; tt < 6; ++tt) {
      const int ga = (int)((rp >> (2 * term_gate(tt))) & 3u);
      if (!((ornd >> ga) & 1u)) continue;
      const int u = (int)((rp >> (2 * term_pu(tt))) & 3u), vv = (int)((rp >> (2 * term_pv(tt))) & 3u);
      const int npr = (int)((ornd >> u) & 1u) + (int)((ornd >> vv) & 1u);
      const int kt = kr + X.nbin * tt;
      qdcount<SHC>(X, kt + X.nbin * 6 * npr);
      qfix(X, qfx(X.dfix, kt + X.nbin * 6 * npr), qfx(X.dfix, kt + X.nbin * 6 * npr + X.dhi),
           wsel(u) * wsel(vv), X.dscale);
    }
  }
  return __popc(vm);
}

// One 4-clique (p, a, b, d) = vertices 0..3 with edge metas m: its
// contributions to the histograms, or (ADJ) its weight gradient: the root's
// to racc, those of a, b, d to the per-neighbour accumulators at positions
// ya, yb, yd.  Returns the number of rooted contributions.
template <bool WEIGHTED, bool SHC, bool ADJ, bool COMPACT, bool TETRA>
__device__ __forceinline__ int quad_emit(const QuadCtx& X, const QVerts& V, const uint32_t m[6],
                                         double gscale, Fix128& racc, unsigned* s_grad, int gcap,
                                         int ya, int yb, int yd) {
  if constexpr (ADJ) {
    return quad_grad_c(X, V, m, gscale, racc, s_grad, gcap, ya, yb, yd);
  } else if constexpr (TETRA) {
    return tetra_contrib<WEIGHTED, SHC>(X, V, m);
  } else {
    static_assert(!(WEIGHTED && COMPACT), "weighted 4PCF sums take the flattened drain");
    return quad_contrib<WEIGHTED, SHC>(X, V, m);
  }
}

// SHC: integer counts in block-private 32-bit shared-memory counters,
// added to the global histograms at the end of the block.
// ADJ: instead of the histograms, the weight gradient (g_lo / g_hi, label
// order, scale gscale) of sum(c2 N2) + sum(c3 N3) + sum(cN discN) +
// sum(cR discR), cot = [c2 | c3 | cN | cR].
// COMPACT: the weighted 4PCF sums through the flattened drain
// (quad_contrib_flat) instead of the unrolled per-clique quad_contrib.
// TETRA: the -tetra counts (query_graph_tetrahedron) instead of the 4PCF;
// a template argument so that each kernel holds the code of one form only.
template <bool WEIGHTED, bool SHC, bool ADJ, bool COMPACT, bool TETRA>
__global__ void __launch_bounds__((WEIGHTED || ADJ ? kQuadMaxWarps : kQuadMaxWarpsU) * 32) quad4_kernel(
    DevCatalog C, CSRView G, QuadParams Q, unsigned long long* __restrict__ g_cnt,
    unsigned long long* __restrict__ g_fix, unsigned long long* __restrict__ d_cnt,
    unsigned long long* __restrict__ d_fix, int nh, int nd, double fscale, double dscale,
    unsigned long long* __restrict__ stats, int* __restrict__ work,
    const double* __restrict__ cot, double gscale, unsigned long long* __restrict__ g_lo,
    unsigned long long* __restrict__ g_hi) {
  constexpr bool LW = WEIGHTED || ADJ;  // weights staged
  extern __shared__ __align__(16) unsigned char smem[];
  const QuadLayout L = quad_layout(Q.nbins, Q.cap, blockDim.x >> 5, SHC ? nh + nd : 0, ADJ);
  QuadCtx X;
  quad_setup<SHC, ADJ>(X, Q, smem + L.off_rank, smem + L.off_cnt, g_cnt, g_fix, d_cnt, d_fix, nh,
                       nd, fscale, dscale, cot);

  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  unsigned char* wb = smem + L.off_warp + L.warp_bytes * (threadIdx.x >> 5);
  long long* s_rs = reinterpret_cast<long long*>(wb + L.o_rs);
  double* s_w = reinterpret_cast<double*>(wb + L.o_w);
  unsigned long long* s_mo = reinterpret_cast<unsigned long long*>(wb + L.o_mo);
  int* s_col = reinterpret_cast<int*>(wb + L.o_col);
  int* s_len = reinterpret_cast<int*>(wb + L.o_len);
  uint32_t* s_xm = reinterpret_cast<uint32_t*>(wb + L.o_xm);
  uint32_t* s_hkey = reinterpret_cast<uint32_t*>(wb + L.o_hkey);
  unsigned long long* s_q = reinterpret_cast<unsigned long long*>(wb + L.o_q);
  uint16_t* s_xy = reinterpret_cast<uint16_t*>(wb + L.o_xy);
  uint16_t* s_xz = reinterpret_cast<uint16_t*>(wb + L.o_xz);
  uint32_t* s_bits = reinterpret_cast<uint32_t*>(wb + L.o_bits);
  unsigned* s_grad = reinterpret_cast<unsigned*>(wb + L.o_g);  // four words per neighbour, cap apart
  const int cap = Q.cap;
  const int lg_max = qhash_lg_max(cap);
  unsigned long long quads = 0, rooted = 0, probes = 0;

  // position of label c in R+(p) via the hash table, or -1
  auto lookup = [&](int c, int p, int lg, bool live) -> int {
    const int off = c - p;
    live = live && off > 0 && off < kQMaxOffset;
    const int hs = 1 << lg;
    uint32_t h = qfib_slot((uint32_t)off, lg);
    uint32_t e = live ? s_hkey[h] : 0u;
    bool hit = live && (e >> 10) == (uint32_t)off;
    bool open = live && !hit && e != 0u;
    for (int it = 1; it < hs && __any_sync(0xffffffffu, open); ++it) {
      if (open) {
        h = (h + 1) & (uint32_t)(hs - 1);
        e = s_hkey[h];
        hit = (e >> 10) == (uint32_t)off;
        open = !hit && e != 0u;
      }
    }
    return hit ? (int)(e & 0x3ffu) : -1;
  };

  const QuadWindow win = quad_window(Q, C.n, 1);
  for (;;) {
    int item = 0;
    if (lane == 0) item = atomicAdd(work, 1);
    item = __shfl_sync(0xffffffffu, item, 0);
    int p, part, nparts;
    if (!quad_item(Q, win, item, p, part, nparts)) break;
    const int64_t b0 = G.start[p];
    const int k = G.len[p];
    if (k < 3 && Q.order) break;  // longest rows first: every later root is as short
    if (k < 3 || k > cap) continue;  // rows longer than cap are rejected on the host
    if (rec_col(G.rec[b0 + k - 1]) - p >= kQMaxOffset) {
      if (lane == 0) atomicMax(&stats[3], 1ull);  // reported to the host
      continue;
    }
    const uint8_t fp = C.flags[p] | (G.deg_full[p] > 3 ? kFlagDeg4 : 0);
    const int op = C.orig[p];
    const double wp = LW ? C.w[p] : 0.0;
    Fix128 racc = {0ull, 0ull};  // adjoint: gradient of the root, per lane
    int lg = 6;
    while (lg < lg_max && (1 << lg) < 8 * k) ++lg;
    const int hs = 1 << lg;
    __syncwarp();
    for (int h = lane; h < hs; h += 32) s_hkey[h] = 0u;
    __syncwarp();
    for (int xb = 0; xb < k; xb += 32) {
      const int x = xb + lane;
      if (x < k) {
        const unsigned long long r = G.rec[b0 + x];
        const int a = rec_col(r);
        s_col[x] = a;
        s_rs[x] = G.start[a];
        s_len[x] = G.len[a];
        const uint8_t fa = C.flags[a] | (G.deg_full[a] > 3 ? kFlagDeg4 : 0);
        s_mo[x] = ((unsigned long long)(uint32_t)C.orig[a] << 32) |
                  (rec_meta(r) | ((uint32_t)fa << 24));
        if (LW) s_w[x] = C.w[a];
        if (ADJ) {
          s_grad[x] = s_grad[Q.cap + x] = s_grad[2 * Q.cap + x] = s_grad[3 * Q.cap + x] = 0u;
        }
        const uint32_t off = (uint32_t)(a - p);
        const uint32_t key = (off << 10) | (uint32_t)x;
        uint32_t h = qfib_slot(off, lg);
        for (int t = 0; t < hs; ++t) {
          if (atomicCAS(&s_hkey[h], 0u, key) == 0u) break;
          h = (h + 1) & (uint32_t)(hs - 1);
        }
      }
    }
    __syncwarp();
    const int nwords = (k + 31) >> 5;
    for (int x = part; x < k - 2; x += nparts) {  // a split root: every nparts-th a
      // X = R+(a) ∩ R+(p) beyond position x, listed in label order and
      // marked in the bitmask
      for (int wd = lane; wd < nwords; wd += 32) s_bits[wd] = 0u;
      __syncwarp();
      const int64_t ra = s_rs[x];
      const int ka = s_len[x];
      if (lane == 0) probes += (unsigned long long)ka;
      int nx = 0;
      for (int j0 = 0; j0 < ka; j0 += 32) {
        const int j = j0 + lane;
        unsigned long long rr = 0;
        if (j < ka) rr = G.rec[ra + j];
        const int y = lookup(rec_col(rr), p, lg, j < ka);
        const bool found = y > x;
        const unsigned msk = __ballot_sync(0xffffffffu, found);
        if (found) {
          const int z = nx + __popc(msk & lt);
          s_xy[z] = (uint16_t)y;
          s_xm[z] = rec_meta(rr);
          s_xz[y] = (uint16_t)z;
          atomicOr(&s_bits[y >> 5], 1u << (y & 31));
        }
        nx += __popc(msk);
      }
      __syncwarp();
      if (nx < 2) continue;
      const unsigned long long mpa_w = s_mo[x];
      int qn = 0;
      // one queued clique: (p, a = row x, b = X entry z, d = row y_d), one
      // per lane (act: the lane holds entry e).  The weighted 4PCF bins the
      // warp's cliques together (quad_contrib_flat), so every lane takes
      // part; a lane without a clique reads nothing and holds zero bins
      // (no valid root).  Every other mode bins one clique per lane.
      auto drain_one = [&](int e, bool act) {
        constexpr bool FLAT = WEIGHTED && COMPACT && !ADJ && !TETRA;
        if (!act && !FLAT) return;
        QVerts V;
        uint32_t m[6] = {0u, 0u, 0u, 0u, 0u, 0u};
        int yb = 0, yd = 0;
        V.fl[0] = V.fl[1] = V.fl[2] = V.fl[3] = 0;
        V.og[0] = V.og[1] = V.og[2] = V.og[3] = 0;
        V.w[0] = V.w[1] = V.w[2] = V.w[3] = 0.0;
        if (act) {
          const unsigned long long qe = s_q[e];
          const int z = (int)(qe & 0x3ffu);
          yd = (int)((qe >> 10) & 0x3ffu);
          const uint32_t mbd = (uint32_t)(qe >> 32);
          yb = s_xy[z];
          const unsigned long long mpb_w = s_mo[yb], mpd_w = s_mo[yd];
          V.fl[0] = fp;
          V.fl[1] = (uint8_t)((uint32_t)mpa_w >> 24);
          V.fl[2] = (uint8_t)((uint32_t)mpb_w >> 24);
          V.fl[3] = (uint8_t)((uint32_t)mpd_w >> 24);
          V.og[0] = op;
          V.og[1] = (int)(mpa_w >> 32);
          V.og[2] = (int)(mpb_w >> 32);
          V.og[3] = (int)(mpd_w >> 32);
          V.w[0] = wp;
          V.w[1] = LW ? s_w[x] : 0.0;
          V.w[2] = LW ? s_w[yb] : 0.0;
          V.w[3] = LW ? s_w[yd] : 0.0;
          // m: (p,a) (p,b) (p,d) (a,b) (a,d) (b,d)
          m[0] = (uint32_t)mpa_w & 0xffffffu;
          m[1] = (uint32_t)mpb_w & 0xffffffu;
          m[2] = (uint32_t)mpd_w & 0xffffffu;
          m[3] = s_xm[z];
          m[4] = s_xm[s_xz[yd]];
          m[5] = mbd;
        }
        int nroot;
        if constexpr (FLAT)
          nroot = quad_contrib_flat<SHC>(X, V, m, act,
                                         (unsigned)x | ((unsigned)yb << 10) | ((unsigned)yd << 20),
                                         s_w, wp);
        else
          nroot = quad_emit<WEIGHTED, SHC, ADJ, COMPACT, TETRA>(X, V, m, gscale, racc, s_grad, Q.cap,
                                                                x, yb, yd);
        quads += nroot > 0;
        rooted += nroot;
      };
      // Work items (b = X[z], d in R+(b)): X entries in batches of 32, the
      // rows of a batch flattened over the lanes in windows of 32 items.
      // One loop over the windows, with a last pass (fin) that drains the
      // cliques still queued, so that the long binning code has one call
      // site (the X data of this a are replaced next).
      int zb = 0, tot = 0, t0 = 0, nrows = 0, incl = 0, excl = 0, cz = 0, done = 0;
      long long crs = 0;
      bool fin = false;
      for (;;) {
        while (!fin && t0 >= tot) {
          if (zb >= nx) {
            fin = true;
            break;
          }
          // the next batch of X entries with their rows
          const int z = zb + lane;
          int len = 0;
          long long rs = 0;
          if (z < nx) {
            const int yb = s_xy[z];
            len = s_len[yb];
            rs = s_rs[yb];
          }
          const unsigned nz = __ballot_sync(0xffffffffu, len > 0);
          nrows = __popc(nz);
          const int src = lane < nrows ? (int)__fns(nz, 0, lane + 1) : 0;
          // every lane takes part in each shuffle; the select comes after
          const int slen = __shfl_sync(0xffffffffu, len, src);
          const int clen = lane < nrows ? slen : 0;
          crs = __shfl_sync(0xffffffffu, rs, src);
          cz = zb + src;
          incl = clen;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int yv = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += yv;
          }
          tot = __shfl_sync(0xffffffffu, incl, 31);
          excl = incl - clen;
          if (lane == 0) probes += (unsigned long long)tot;
          done = 0;  // compacted rows that ended before the window
          t0 = 0;
          zb += 32;
        }
        if (!fin) {
          const int last = incl - 1 - t0;
          const unsigned bit = (lane < nrows && last >= 0 && last < 32) ? (1u << last) : 0u;
          const unsigned ends = __reduce_or_sync(0xffffffffu, bit);
          const int j = (done + __popc(ends & lt)) & 31;
          done += __popc(ends);
          const long long ors = __shfl_sync(0xffffffffu, crs, j);
          const int oex = __shfl_sync(0xffffffffu, excl, j);
          const int oz = __shfl_sync(0xffffffffu, cz, j);
          const int t = t0 + lane;
          unsigned long long rr = 0;
          if (t < tot) rr = G.rec[ors + (t - oex)];
          const int yd = lookup(rec_col(rr), p, lg, t < tot);
          const bool hit = yd >= 0 && ((s_bits[yd >> 5] >> (yd & 31)) & 1u);
          const unsigned m = __ballot_sync(0xffffffffu, hit);
          if (hit) {
            const int pos = qn + __popc(m & lt);
            s_q[pos] = ((unsigned long long)rec_meta(rr) << 32) | (uint32_t)(oz | (yd << 10));
          }
          qn += __popc(m);
          t0 += 32;
        }
        if (qn >= 32 || (fin && qn > 0)) {
          const int nq = min(qn, 32);
          __syncwarp();
          drain_one(qn - nq + lane, lane < nq);
          qn -= nq;
          __syncwarp();
        }
        if (fin && qn == 0) break;
      }
      __syncwarp();
    }
    if (ADJ) {
      // flush the gradients of this root and of its neighbours
      for (int x = lane; x < k; x += 32) {
        unsigned long long lo, hi;
        hist_fix_value(reinterpret_cast<const unsigned long long*>(s_grad), Q.cap, x, lo, hi);
        if (lo | hi) fix_merge(&g_lo[s_col[x]], &g_hi[s_col[x]], lo, hi);
      }
      racc = fix_warp_sum(racc);
      if (lane == 0 && (racc.lo | racc.hi)) fix_merge(&g_lo[p], &g_hi[p], racc.lo, racc.hi);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    quads += __shfl_xor_sync(0xffffffffu, quads, o);
    rooted += __shfl_xor_sync(0xffffffffu, rooted, o);
    probes += __shfl_xor_sync(0xffffffffu, probes, o);
  }
  if (lane == 0) {
    if (quads) atomicAdd(&stats[0], quads);
    if (rooted) atomicAdd(&stats[1], rooted);
    if (probes) atomicAdd(&stats[2], probes);
  }
  if (SHC) {
    __syncthreads();
    for (int k = threadIdx.x; k < nh + nd; k += blockDim.x) {
      const unsigned int v = X.scnt[k];
      if (v) atomicAdd(k < nh ? &X.cnt[k] : &X.dcnt[k - nh], (unsigned long long)v);
    }
  }
}

// Geometric mode.  The edges among the members of R+(p) are exactly the
// pairs that pass the graph's membership test, so the warp tests the
// k(k-1)/2 pairs of R+(p) once (closed-form inversion of the triangular pair
// index over the lanes) and records them as one adjacency bitmask row per
// member (bits of the later members).  The 4-cliques p < a < b < d are then
// the set bits d of row(a) AND row(b) for every edge (a, b): the edges are
// queued 32 at a time, each lane ANDs its two rows word by word and emits one
// clique per set bit into the clique queue, which is drained 32 at a time.  No
// row other than R+(p) is read; the tests are k(k-1)/2 per root instead of the
// sum over R+(p) of the members' row lengths.  Rows up to 256 members (8-bit
// positions).
//
// What a clique adds depends on its six radial bins, on the catalogue-id order
// of its vertices and on their flags.  Three things are therefore done once
// per row instead of once per clique: the members are sorted by catalogue id,
// so that only the root's place among the three members of a clique is open
// (three comparisons with its rank in the row, and at most three exchanges
// bring the bins into id order); the bins of all pairs are kept from the
// membership test (rows up to kMatCap members; else computed again); and
// the perimeter's rank and canonical order come from two tables over pairs of
// bins.  Each of the four roots is then a fixed formula of the ordered bins.
// Sorting ids, comparing perimeters and summing rank differences for every
// root of every clique took 1,600 warp instructions per 32 cliques, four fifths
// of the unit-weight kernel; it takes 420 now, with as much again for the
// enumeration.  4PCF workload (120,000 points, 42M cliques, rows up to 120):
// unit weights 2.70 -> 1.41 ms, issue-bound; weighted sums 4.2 -> 2.9 ms, bound
// by the L1 traffic of the reductions (71%); adjoint 7.2 -> 3.2 ms.
//
// Unit weights: one count per valid root (see quad_root).  Weighted sums and
// the adjoint take the valid (clique, root) pairs of the warp 32 at a time,
// every lane one root, whose role order makes all of its terms fixed formulas
// again.
constexpr int kQEdgeQueue = 64;  // edge queue entries per warp (< 32 left + 32 pushed)
constexpr int kMatCap = 128;
constexpr int kNoPerimeter = 1 << 29;  // table entry of two bins out of order

struct QuadGLayout {
  size_t off_rank, off_tab, off_cnt, off_warp;
};
// One warp's area for rows of up to cap members.
struct QuadGWarp {
  size_t pos, w, g, col, code, tb, adj, bin, q, eq, bytes;
};

// pairs whose bins a warp can keep
__host__ __device__ inline int quad_bins(int cap) {
  const int c = cap < kMatCap ? cap : kMatCap;
  return c * (c - 1) / 2;
}

// tetra: its six bins are equal, so there are no tables of perimeters (up to
// 129 KB, which would leave room for few warps) and no kept bins
__host__ __device__ inline QuadGLayout quadg_layout(int nbins, int ncounts, bool tetra) {
  QuadGLayout L;
  size_t o = 0;
  L.off_rank = o;
  o = qalign8(o + sizeof(int) * 4 * (size_t)(nbins + 2));
  L.off_tab = o;
  if (!tetra) o = qalign8(o + sizeof(int) * 2 * (size_t)nbins * nbins);
  L.off_cnt = o;
  o = o + sizeof(unsigned int) * (size_t)ncounts;
  L.off_warp = (o + 15) & ~(size_t)15;
  return L;
}

__host__ __device__ inline QuadGWarp quadg_warp(int cap, bool adj, bool lw, bool tetra) {
  QuadGWarp W;
  const size_t nwd = (size_t)(cap + 31) / 32;
  size_t w = 0;
  W.pos = w;  w += (size_t)cap * 16;              // float4 position of each member
  W.tb = w;   w += (size_t)cap * 4;               // catalogue id, then pair index base
  W.w = w;    w += lw ? ((size_t)cap + 1) * 8 : 0;  // weight, and the root's
  W.g = w;    w += adj ? (size_t)cap * 16 : 0;    // 128-bit gradient of each neighbour
  W.col = w;  w += (size_t)cap * 4;               // label
  W.code = w; w += (size_t)cap * 4;               // bin of (p, a) from 0 | random << 8 | root << 9
  W.adj = w;  w += (size_t)cap * nwd * 4;         // adjacency rows
  W.q = w;    w += (size_t)kQQueue * 4;           // cliques: a | b << 8 | d << 16 | bin(a,b) << 24
  W.eq = w;   w += (size_t)kQEdgeQueue * 4;       // edges: a | b << 8
  W.bin = w;  w += tetra ? 0 : (size_t)quad_bins(cap);  // bins of the pairs
  W.bytes = (w + 15) & ~(size_t)15;
  return W;
}

template <bool WEIGHTED, bool SHC, bool ADJ, bool TETRA>
__global__ void __launch_bounds__((ADJ ? kQuadGWarpsA : (WEIGHTED ? kQuadGWarpsW : kQuadMaxWarpsU)) * 32)
    quad4g_kernel(
    DevCatalog C, CSRView G, QuadParams Q, unsigned long long* __restrict__ g_cnt,
    unsigned long long* __restrict__ g_fix, unsigned long long* __restrict__ d_cnt,
    unsigned long long* __restrict__ d_fix, int nh, int nd, double fscale, double dscale,
    unsigned long long* __restrict__ stats, int* __restrict__ work,
    const double* __restrict__ cot, double gscale, unsigned long long* __restrict__ g_lo,
    unsigned long long* __restrict__ g_hi) {
  constexpr bool LW = WEIGHTED || ADJ;
  extern __shared__ __align__(16) unsigned char smem[];
  const QuadGLayout L = quadg_layout(Q.nbins, SHC ? nh + nd : 0, TETRA);
  QuadCtx X;
  quad_setup<SHC, ADJ>(X, Q, smem + L.off_rank, smem + L.off_cnt, g_cnt, g_fix, d_cnt, d_fix, nh,
                       nd, fscale, dscale, cot);
  const PairParams& P = Q.P;
  const int nb = Q.nbins;
  // rank - 1 of the perimeter b1 <= b2 <= b3 <= b4 is s_t12[b1, b2] +
  // s_t34[b3, b4] (bins from 0)
  int* const s_t12 = reinterpret_cast<int*>(smem + L.off_tab);
  int* const s_t34 = s_t12 + nb * nb;
  for (int k = TETRA ? nb * nb : threadIdx.x; k < nb * nb; k += blockDim.x) {
    const int i = k / nb + 1, j = k % nb + 1, n2 = nb + 2;
    const int* F = X.F;
    s_t12[k] = i <= j ? (F[i] - F[1]) + (F[n2 + j] - F[n2 + i]) - F[2 * n2 + j] : kNoPerimeter;
    s_t34[k] = i <= j ? F[2 * n2 + i] + (F[3 * n2 + j] - F[3 * n2 + i]) : kNoPerimeter;
  }
  __syncthreads();

  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  // the first long_warps warps hold rows of up to cap members, the others of
  // up to short_cap
  const int wid = threadIdx.x >> 5;
  const bool big = wid < Q.long_warps;
  const int cap = big || Q.long_warps == 0 ? Q.cap : Q.short_cap;
  const QuadGWarp A = quadg_warp(cap, ADJ, LW, TETRA);
  unsigned char* wb = smem + L.off_warp;
  if (big || Q.long_warps == 0)
    wb += A.bytes * wid;
  else
    wb += quadg_warp(Q.cap, ADJ, LW, TETRA).bytes * Q.long_warps + A.bytes * (wid - Q.long_warps);
  float4* const s_pos = reinterpret_cast<float4*>(wb + A.pos);
  double* const s_w = reinterpret_cast<double*>(wb + A.w);
  unsigned* const s_grad = reinterpret_cast<unsigned*>(wb + A.g);  // four words per neighbour, cap apart
  int* const s_col = reinterpret_cast<int*>(wb + A.col);
  int* const s_code = reinterpret_cast<int*>(wb + A.code);
  int* const s_tb = reinterpret_cast<int*>(wb + A.tb);
  uint32_t* const s_adj = reinterpret_cast<uint32_t*>(wb + A.adj);
  uint32_t* const s_q = reinterpret_cast<uint32_t*>(wb + A.q);
  uint32_t* const s_eq = reinterpret_cast<uint32_t*>(wb + A.eq);
  uint8_t* const s_bin = wb + A.bin;
  const int slot = cap;  // position of the root beside the members' (its weight is staged there)
  unsigned long long quads = 0, rooted = 0, probes = 0;
  const float guard = P.f32 ? P.tguard : INFINITY;
  // edge test and radial bin (from 0) of members x, y (see bin_pair_f32)
  auto pair_bin = [&](int x, int y, int& b0) -> bool {
    const float4 px = s_pos[x], py = s_pos[y];
    const float dx = py.x - px.x, dy = py.y - px.y, dz = py.z - px.z;
    const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    const float t = fmaf(d2 * rsqrt_approx(d2), P.f_inv_dr, P.f_t0);
    const float tr = __fadd_rn(t, 12582912.0f);
    const float tn = __fadd_rn(tr, -12582912.0f);
    b0 = __float_as_int(tr) - 0x4B400000 - (t < tn ? 1 : 0);
    bool in = (unsigned)b0 < (unsigned)nb;
    if (!(fabsf(t - tn) >= guard)) {
      int b = 1;
      in = d2 < P.rmax2_hi && d2 > P.rmin2_lo &&
           edge_radial_f64(C.posd[s_col[x]], C.posd[s_col[y]], P, b);
      b0 = b - 1;
    }
    return in;
  };

  int phase = big ? 0 : 1;  // long rows first, then the others (work[1], work[0])
  // -tetra with three bins or more: staging and testing a row is nearly all of
  // its work, which shares would repeat (40,000 points, rows up to 256, 20 bins
  // 5.0 ms with shares, 0.9 without; one bin, where every edge stays, 14 and 21)
  const bool split = !TETRA || nb <= 2;
  QuadWindow win = quad_window(Q, C.n, phase, split);
  for (;;) {
    int item = 0;
    if (lane == 0) item = atomicAdd(work + (1 - phase), 1);
    item = __shfl_sync(0xffffffffu, item, 0);
    int p, part, nparts;
    if (!quad_item(Q, win, item, p, part, nparts)) {
      if (phase == 1) break;
      phase = 1;
      win = quad_window(Q, C.n, 1, split);
      continue;
    }
    const int64_t b0 = G.start[p];
    const int k = G.len[p];
    if (k < 3 && Q.order) break;  // longest rows first: every later root is as short
    if (k < 3 || k > cap) continue;  // rows longer than cap are rejected on the host
    // a vertex is a root unless it is a buffer point or (not -tetra) its full
    // row is too short
    auto root_bit = [&](int v, uint8_t f) {
      return !(f & FLAG_BUFFER) && (TETRA || G.deg_full[v] > 3) ? 1u : 0u;
    };
    const uint8_t fp = C.flags[p];
    const unsigned prnd = fp & FLAG_RANDOM, proot = root_bit(p, fp);
    const int op = C.orig[p];
    Fix128 racc = {0ull, 0ull};
    const int nwk = (k + 31) >> 5;  // adjacency words per row for this root
    __syncwarp();
    // the members sorted by catalogue id
    int below = 0;
    const int k4 = (k + 3) & ~3;
    for (int x = lane; x < k4; x += 32) {
      const int id = x < k ? C.orig[rec_col(G.rec[b0 + x])] : 0x7fffffff;
      s_tb[x] = id;
      below += id < op ? 1 : 0;
    }
    const int rank_p = (int)__reduce_add_sync(0xffffffffu, (unsigned)below);
    for (int i = lane; i < k * nwk; i += 32) s_adj[i] = 0u;
    __syncwarp();
    for (int x = lane; x < k; x += 32) {
      const int id = s_tb[x];
      int at = 0;
      for (int j = 0; j < k4; j += 4) {
        const int4 v = *reinterpret_cast<const int4*>(&s_tb[j]);
        at += (v.x < id ? 1 : 0) + (v.y < id ? 1 : 0) + (v.z < id ? 1 : 0) + (v.w < id ? 1 : 0);
      }
      const unsigned long long r = G.rec[b0 + x];
      const int a = rec_col(r);
      const uint8_t fa = C.flags[a];
      s_col[at] = a;
      s_pos[at] = C.pos4[a];
      s_code[at] = (meta_bin(rec_meta(r)) - 1) | ((fa & FLAG_RANDOM) << 8) | (int)(root_bit(a, fa) << 9);
      if (LW) s_w[at] = C.w[a];
      if (ADJ) {
        s_grad[at] = s_grad[cap + at] = s_grad[2 * cap + at] = s_grad[3 * cap + at] = 0u;
      }
    }
    if (LW && lane == 0) s_w[slot] = C.w[p];
    __syncwarp();
    // pass 1: adjacency among the members of R+(p), and their bins
    const int npair = k * (k - 1) / 2;
    const int k2m1 = 2 * k - 1;
    const bool mat = !TETRA && npair <= quad_bins(cap);  // their bins are kept
    // index of the pair (x, y) is s_tb[x] + y
    for (int x = lane; x < k; x += 32) s_tb[x] = x * (k2m1 - x) / 2 - x - 1;
    if (lane == 0 && part == 0) probes += (unsigned long long)npair;  // once per root
    auto pair_of = [&](int t, int& x, int& y) {
      // x: the largest row with x (2k - 1 - x) / 2 <= t pairs before it
      // (exact for every k up to kPairRowExact)
      x = pair_row_biased(k2m1, t);
      y = t - (int)((unsigned)(x * (k2m1 - x)) >> 1) + x + 1;
    };
    for (int t = lane; t < npair; t += 32) {
      int x, y, bin;
      pair_of(t, x, y);
      // -tetra: an edge in another bin than both of its ends' to the root is in
      // no clique that counts (120,000 points, rows up to 120, weighted: 4 bins
      // 1.6 -> 0.45 ms, 127 bins 1.3 -> 0.3; rows of 200: 4.4 -> 0.4)
      if (pair_bin(x, y, bin) &&
          (!TETRA || (bin == (s_code[x] & 0xff) && bin == (s_code[y] & 0xff)))) {
        atomicOr(&s_adj[x * nwk + (y >> 5)], 1u << (y & 31));
        if (mat) s_bin[t] = (uint8_t)bin;
      }
    }
    __syncwarp();
    int qn = 0, en = 0;
    // one queued clique: (p, members x < y < z), one per lane (act: the lane
    // holds entry e; every lane takes part, one without a clique has no root)
    auto drain_one = [&](int e, bool act) {
      const uint32_t qe = act ? s_q[e] : 0u;
      const int x = (int)(qe & 0xffu), y = (int)((qe >> 8) & 0xffu), z = (int)((qe >> 16) & 0xffu);
      const int cx = s_code[x], cy = s_code[y], cz = s_code[z];
      if constexpr (TETRA) {
        // only cliques with all edges in one bin are queued: each of the four
        // vertices that can be a root is one
        if (!act) return;
        QVerts V;
        auto flags = [](int code) {
          return (uint8_t)(((code >> 8) & 1 ? FLAG_RANDOM : 0) | ((code >> 9) & 1 ? 0 : FLAG_BUFFER));
        };
        V.fl[0] = fp;
        V.fl[1] = flags(cx);
        V.fl[2] = flags(cy);
        V.fl[3] = flags(cz);
        V.og[0] = 2 * rank_p;  // places in id order
        V.og[1] = 2 * x + 1;
        V.og[2] = 2 * y + 1;
        V.og[3] = 2 * z + 1;
        V.w[0] = LW ? s_w[slot] : 0.0;
        V.w[1] = LW ? s_w[x] : 0.0;
        V.w[2] = LW ? s_w[y] : 0.0;
        V.w[3] = LW ? s_w[z] : 0.0;
        const uint32_t b = pack_meta((cx & 0xff) + 1, 1, 1), m[6] = {b, b, b, b, b, b};
        const int nroot = tetra_contrib<WEIGHTED, SHC>(X, V, m);
        quads += nroot > 0 ? 1 : 0;
        rooted += (unsigned)nroot;
        return;
      }
      int bxz = 0, byz = 0;
      if (act) {
        if (mat) {
          bxz = s_bin[s_tb[x] + z];
          byz = s_bin[s_tb[y] + z];
        } else {
          pair_bin(x, z, bxz);
          pair_bin(y, z, byz);
        }
      }
      // bins b_ij between the i-th and j-th vertex in catalogue-id order: the
      // root first, then moved behind the members of smaller id
      int b01 = cx & 0xff, b02 = cy & 0xff, b03 = cz & 0xff, b12 = (int)(qe >> 24), b13 = bxz, b23 = byz;
      auto swap_if = [](bool c, int& u, int& v) {
        const int t = c ? v : u;
        v = c ? u : v;
        u = t;
      };
      const bool r1 = x < rank_p, r2 = y < rank_p, r3 = z < rank_p;  // r3 implies r2 implies r1
      swap_if(r1, b02, b12);
      swap_if(r1, b03, b13);
      swap_if(r2, b01, b02);
      swap_if(r2, b13, b23);
      swap_if(r3, b02, b03);
      swap_if(r3, b12, b13);
      const int r = (r1 ? 1 : 0) + (r2 ? 1 : 0) + (r3 ? 1 : 0);
      // one bit per vertex in that order: randoms, and possible roots
      auto insert = [&](unsigned three, unsigned own) {
        const unsigned low = (1u << r) - 1u;
        return (three & low) | (own << r) | ((three & ~low) << 1);
      };
      const unsigned rnd = insert((unsigned)(((cx >> 8) & 1) | ((cy >> 7) & 2) | ((cz >> 6) & 4)), prnd);
      unsigned vm = insert((unsigned)(((cx >> 9) & 1) | ((cy >> 8) & 2) | ((cz >> 7) & 4)), proot);
      if (!act) vm = 0u;
      // histogram index of each root, or none when its perimeter is not
      // canonical
      int kk[4] = {0, 0, 0, 0};
      auto root = [&](int i, int b1, int b2, int b3, int b4, int d1, int d2) {
        const int cfg = s_t12[b1 * nb + b2] + s_t34[b3 * nb + b4];
        if (!((unsigned)cfg < (1u << 28) && b2 <= b3)) vm &= ~(1u << i);
        kk[i] = cfg + X.ncfg * (d1 + nb * d2);
      };
      root(0, b01, b12, b23, b03, b02, b13);
      root(1, b01, b02, b23, b13, b12, b03);
      root(2, b02, b01, b13, b23, b12, b03);
      root(3, b03, b01, b12, b23, b13, b02);
      quads += vm ? 1 : 0;
      rooted += (unsigned)__popc(vm);
      if constexpr (!LW) {
        // the pattern of root i: its randomness, then that of the others
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const unsigned low = (1u << i) - 1u;
          const unsigned pat = ((rnd >> i) & 1u) | ((rnd & low) << 1) | (rnd & ~(2u * low + 1u));
          if ((vm >> i) & 1u) qcount<SHC>(X, kk[i] + X.nbin * (int)pat);
        }
      } else {
        // the warp's valid roots, ordered by vertex, then lane
        const unsigned three = (unsigned)(x | (y << 8) | (z << 16));
        const unsigned lowb = r == 0 ? 0u : (0xffffffu >> (24 - 8 * r));
        // the root's byte is empty: its place is kept beside the random bits,
        // which leaves all 256 positions to members
        const unsigned vpos = (three & lowb) | (r == 3 ? 0u : (three & ~lowb) << 8);
        const unsigned vrnd = rnd | ((unsigned)r << 4);
        unsigned mr[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) mr[i] = __ballot_sync(0xffffffffu, (vm >> i) & 1u);
        const int c0 = __popc(mr[0]), c1 = c0 + __popc(mr[1]), c2 = c1 + __popc(mr[2]),
                  total = c2 + __popc(mr[3]);
        for (int i0 = 0; i0 < total; i0 += 32) {
          const int i = i0 + lane;
          const int R = i < c0 ? 0 : (i < c1 ? 1 : (i < c2 ? 2 : 3));
          const int base = R == 0 ? 0 : (R == 1 ? c0 : (R == 2 ? c1 : c2));
          const unsigned mR = R == 0 ? mr[0] : (R == 1 ? mr[1] : (R == 2 ? mr[2] : mr[3]));
          const int o = i < total ? (int)__fns(mR, 0, i - base + 1) : 0;
          // every lane takes part in each shuffle; the select comes after
          const unsigned ornd = __shfl_sync(0xffffffffu, vrnd, o);
          const unsigned opos = __shfl_sync(0xffffffffu, vpos, o);
          const int q0 = __shfl_sync(0xffffffffu, kk[0], o), q1 = __shfl_sync(0xffffffffu, kk[1], o),
                    q2 = __shfl_sync(0xffffffffu, kk[2], o), q3 = __shfl_sync(0xffffffffu, kk[3], o);
          if (i >= total) continue;
          const int kr = R == 0 ? q0 : (R == 1 ? q1 : (R == 2 ? q2 : q3));
          // roles: the root, then the other three in id order
          const int v[4] = {R, R == 0 ? 1 : 0, R <= 1 ? 2 : 1, R <= 2 ? 3 : 2};
          int pos[4];
          unsigned rb[4];
          double w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            pos[j] = v[j] == (int)(ornd >> 4) ? slot : (int)((opos >> (8 * v[j])) & 0xffu);
            rb[j] = (ornd >> v[j]) & 1u;
            w[j] = LW ? s_w[pos[j]] : 0.0;
          }
          const int onr = (int)(rb[0] + rb[1] + rb[2] + rb[3]);
          if constexpr (ADJ) {
            double g[4];
            quad_root_grad(X, kr, rb, w, g);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              if (pos[j] == slot)
                fix_acc(racc, g[j], gscale);
              else
                smem_fix_add(s_grad + pos[j], cap, __double2ll_rn(g[j] * gscale));
            }
          } else {
            qcount<SHC>(X, kr + X.nbin * onr);
            qfix(X, qfx(X.fix, kr + X.nbin * onr), qfx(X.fix, kr + X.nbin * (onr + 5)),
                 ((w[0] * w[1]) * w[2]) * w[3], X.fscale);
#pragma unroll
            for (int tt = 0; tt < 6; ++tt) {
              if (!rb[term_gate(tt)]) continue;
              const int u = term_pu(tt), vv = term_pv(tt);
              const int kt = kr + X.nbin * tt + X.nbin * 6 * (int)(rb[u] + rb[vv]);
              qdcount<SHC>(X, kt);
              qfix(X, qfx(X.dfix, kt), qfx(X.dfix, kt + X.dhi), w[u] * w[vv], X.dscale);
            }
          }
        }
      }
    };
    // the cliques of up to 32 queued edges (entry e, or none when e < 0);
    // every lane takes part.  fin: also drain the cliques still queued.
    // (One call site each for this and drain_one: their code is long.)
    auto run_edges = [&](int e, bool fin) {
      const bool live = e >= 0;
      int x = 0, y = 0, bxy = 0, cw = 0;
      unsigned cm = 0u;
      if (live) {
        const uint32_t ent = s_eq[e];
        x = (int)(ent & 0xffu);
        y = (int)((ent >> 8) & 0xffu);
        cw = y >> 5;
        cm = s_adj[x * nwk + cw] & s_adj[y * nwk + cw];
        if (mat)
          bxy = s_bin[s_tb[x] + y];
        else if (!TETRA)
          pair_bin(x, y, bxy);
      }
      for (;;) {
        if (live)
          while (cm == 0u && cw + 1 < nwk) {
            ++cw;
            cm = s_adj[x * nwk + cw] & s_adj[y * nwk + cw];
          }
        const bool has = live && cm != 0u;
        const unsigned hm = __ballot_sync(0xffffffffu, has);
        if (has) {
          const int z = cw * 32 + __ffs(cm) - 1;
          cm &= cm - 1u;
          s_q[qn + __popc(hm & lt)] = (uint32_t)(x | (y << 8) | (z << 16)) | ((uint32_t)bxy << 24);
        }
        qn += __popc(hm);
        if (qn >= 32 || (fin && hm == 0u && qn > 0)) {
          const int nq = min(qn, 32);
          __syncwarp();
          drain_one(qn - nq + lane, lane < nq);
          qn -= nq;
          __syncwarp();
        }
        if (hm == 0u && (!fin || qn == 0)) break;
      }
    };
    // pass 2: the edges in pair order, 32 at a time, then what is queued
    // (a split root: every nparts-th chunk of 32 pairs)
    for (int t0 = 0;; t0 += 32) {
      if (t0 < npair && ((t0 >> 5) % nparts) == part) {
        const int t = t0 + lane;
        bool edge = false;
        int x = 0, y = 0;
        if (t < npair) {
          pair_of(t, x, y);
          edge = (s_adj[x * nwk + (y >> 5)] >> (y & 31)) & 1u;
        }
        const unsigned em = __ballot_sync(0xffffffffu, edge);
        if (edge) s_eq[en + __popc(em & lt)] = (uint32_t)(x | (y << 8));
        en += __popc(em);
      }
      const bool last = t0 + 32 >= npair;
      if (en >= 32 || last) {
        const int ne = min(en, 32);
        const bool fin = last && en == ne;
        __syncwarp();
        run_edges(lane < ne ? en - ne + lane : -1, fin);
        en -= ne;
        __syncwarp();
        if (fin) break;
      }
    }
    if (ADJ) {
      for (int x = lane; x < k; x += 32) {
        unsigned long long lo, hi;
        hist_fix_value(reinterpret_cast<const unsigned long long*>(s_grad), cap, x, lo, hi);
        if (lo | hi) fix_merge(&g_lo[s_col[x]], &g_hi[s_col[x]], lo, hi);
      }
      racc = fix_warp_sum(racc);
      if (lane == 0 && (racc.lo | racc.hi)) fix_merge(&g_lo[p], &g_hi[p], racc.lo, racc.hi);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    quads += __shfl_xor_sync(0xffffffffu, quads, o);
    rooted += __shfl_xor_sync(0xffffffffu, rooted, o);
    probes += __shfl_xor_sync(0xffffffffu, probes, o);
  }
  if (lane == 0) {
    if (quads) atomicAdd(&stats[0], quads);
    if (rooted) atomicAdd(&stats[1], rooted);
    if (probes) atomicAdd(&stats[2], probes);
  }
  if (SHC) {
    __syncthreads();
    for (int k = threadIdx.x; k < nh + nd; k += blockDim.x) {
      const unsigned int v = X.scnt[k];
      if (v) atomicAdd(k < nh ? &X.cnt[k] : &X.dcnt[k - nh], (unsigned long long)v);
    }
  }
}

// Warps per block: as many as fit in shared memory (at most maxw).
int quad4_warps(int nbins, int cap, int ncounts, bool adj = false, int maxw = kQuadMaxWarps) {
  int nw = maxw;
  while (nw > 1 && quad_layout(nbins, cap, nw, ncounts, adj).total > kQuadSmemLimit) nw -= 1;
  return nw;
}

}  // namespace

// Block shape of the geometric kernel: rows beyond kShortRow members go to the
// first few warps of each block, with the capacity they need, and the others
// hold short rows only, which leaves room for 24 warps beside the pair bins.
// (4PCF workload, rows up to 120, unit weights: one capacity for all, 13
// warps, 1.97 ms; the long rows, 9% of the work, in a launch of their own
// 1.46 ms; this way 1.41 ms, and at a tenth of the size 0.21, 0.36 and 0.22.)  Catalogues whose
// average row is half of kShortRow or more take one capacity.
constexpr int kLongWarps = 4;
static QuadParams quadg_shape(const QuadParams& Q0, int ncounts, bool adj, bool lw, int maxw, int& nw,
                              size_t& smem) {
  QuadParams Q = Q0;
  const size_t fixed = quadg_layout(Q.nbins, ncounts, Q.tetra != 0).off_warp;
  const size_t big = quadg_warp(Q.cap, adj, lw, Q.tetra != 0).bytes;
  Q.long_warps = 0;
  Q.short_cap = kShortRow;
  if (Q.cap > kShortRow && Q.order && Q.above && Q.nclass > kShortRow && 2 * Q.mean_row < kShortRow) {
    const size_t small = quadg_warp(kShortRow, adj, lw, Q.tetra != 0).bytes;
    nw = maxw;
    while (nw > kLongWarps && fixed + kLongWarps * big + (nw - kLongWarps) * small > kQuadSmemLimit) --nw;
    smem = fixed + kLongWarps * big + (nw - kLongWarps) * small;
    if (nw >= 3 * kLongWarps) {
      Q.long_warps = kLongWarps;
      return Q;
    }
  }
  nw = maxw;
  while (nw > 1 && fixed + nw * big > kQuadSmemLimit) --nw;
  smem = fixed + nw * big;
  return Q;
}

// Launch of either 4-clique kernel: grid of resident blocks, dynamic roots.
template <typename K>
static void launch_quad_grid(K kfn, int nw, size_t smem, int n, int* work, cudaStream_t s,
                             const DevCatalog& C, const CSRView& G, const QuadParams& Q,
                             unsigned long long* g_cnt, unsigned long long* g_fix,
                             unsigned long long* d_cnt, unsigned long long* d_fix, int nh, int nd,
                             double fscale, double dscale, unsigned long long* stats,
                             const double* cot, double gscale, unsigned long long* g_lo,
                             unsigned long long* g_hi) {
  if (smem > kQuadSmemLimit) throw Error{-2, "4PCF: per-warp shared memory exceeds the SM limit"};
  GR_CUDA_TRY(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  GR_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, nw * 32, smem));
  if (per_sm < 1) per_sm = 1;
  int64_t blocks = (int64_t)per_sm * sm_count();
  const int64_t need = ((int64_t)n + nw - 1) / nw;
  if (blocks > need) blocks = need;
  if (blocks < 1) blocks = 1;
  GR_CUDA_TRY(cudaMemsetAsync(work, 0, 2 * sizeof(int), s));
  kfn<<<(unsigned)blocks, nw * 32, smem, s>>>(C, G, Q, g_cnt, g_fix, d_cnt, d_fix, nh, nd, fscale,
                                              dscale, stats, work, cot, gscale, g_lo, g_hi);
  GR_CHECK_LAUNCH();
}

bool launch_quad4(const DevCatalog& C, const CSRView& G, const QuadParams& Q, bool weighted,
                  unsigned long long* g_cnt, unsigned long long* g_fix, unsigned long long* d_cnt,
                  unsigned long long* d_fix, int nh, int nd, double fscale, double dscale,
                  bool shared_counts, unsigned long long* stats, int* work, cudaStream_t s) {
  if (C.n <= 0) return false;
  const int ncnt = nh + nd;
  int nw = 0;
  size_t smem = 0;
  QuadParams S = Q;
  auto go = [&](auto kfn) {
    launch_quad_grid(kfn, nw, smem, C.n, work, s, C, G, S, g_cnt, g_fix, d_cnt, d_fix, nh, nd,
                     fscale, dscale, stats, nullptr, 1.0, nullptr, nullptr);
  };
  // integer counts in block-private counters when they leave room for at
  // least 8 warps (weighted sums without counts need none)
  if (weighted && !Q.counts) shared_counts = false;
  if (Q.geo) {
    const int maxw = weighted ? kQuadGWarpsW : kQuadMaxWarpsU;
    if (shared_counts) {
      S = quadg_shape(Q, ncnt, false, weighted, maxw, nw, smem);
      if (nw < 8) shared_counts = false;
    }
    if (!shared_counts) S = quadg_shape(Q, 0, false, weighted, maxw, nw, smem);
    auto pick = [&](auto tetra_t) {
      constexpr bool TT = decltype(tetra_t)::value;
      if (weighted && shared_counts) go(quad4g_kernel<true, true, false, TT>);
      else if (weighted) go(quad4g_kernel<true, false, false, TT>);
      else if (shared_counts) go(quad4g_kernel<false, true, false, TT>);
      else go(quad4g_kernel<false, false, false, TT>);
    };
    Q.tetra ? pick(std::true_type{}) : pick(std::false_type{});
    return shared_counts;
  }
  S.long_warps = 0;
  if (quad4_warps(Q.nbins, Q.cap, ncnt) < 8) shared_counts = false;
  const int nc = shared_counts ? ncnt : 0;
  nw = quad4_warps(Q.nbins, Q.cap, nc, false, weighted ? kQuadMaxWarps : kQuadMaxWarpsU);
  smem = quad_layout(Q.nbins, Q.cap, nw, nc).total;
  // weighted: the compact contribution code (the unrolled form of its long
  // fixed-point updates overflows the instruction cache); unweighted: unrolled
  auto pick = [&](auto tetra_t) {
    constexpr bool TT = decltype(tetra_t)::value;
    if (weighted && shared_counts) go(quad4_kernel<true, true, false, true, TT>);
    else if (weighted) go(quad4_kernel<true, false, false, true, TT>);
    else if (shared_counts) go(quad4_kernel<false, true, false, false, TT>);
    else go(quad4_kernel<false, false, false, false, TT>);
  };
  Q.tetra ? pick(std::true_type{}) : pick(std::false_type{});
  return shared_counts;
}

void launch_adj4(const DevCatalog& C, const CSRView& G, const QuadParams& Q, const double* cot,
                 double gscale, unsigned long long* g_lo, unsigned long long* g_hi,
                 unsigned long long* stats, int* work, cudaStream_t s) {
  if (C.n <= 0) return;
  int nw = 0;
  size_t smem = 0;
  QuadParams S = Q;
  auto go = [&](auto kfn) {
    launch_quad_grid(kfn, nw, smem, C.n, work, s, C, G, S, nullptr, nullptr, nullptr, nullptr, 0, 0,
                     1.0, 1.0, stats, cot, gscale, g_lo, g_hi);
  };
  if (Q.geo) {
    S = quadg_shape(Q, 0, true, true, kQuadGWarpsA, nw, smem);
    go(quad4g_kernel<false, false, true, false>);
  } else {
    S.long_warps = 0;
    nw = quad4_warps(Q.nbins, Q.cap, 0, true);
    smem = quad_layout(Q.nbins, Q.cap, nw, 0, true).total;
    go(quad4_kernel<false, false, true, true, false>);
  }
}

void quad_expand_patterns(const unsigned long long* H, int nbin, unsigned long long* hc,
                          unsigned long long* dc) {
  std::fill(hc, hc + (size_t)nbin * 5, 0ull);
  std::fill(dc, dc + (size_t)nbin * 6 * 3, 0ull);
  for (int pat = 0; pat < kQuadPatterns; ++pat) {
    const int nr = __builtin_popcount((unsigned)pat);
    for (int k = 0; k < nbin; ++k) {
      const unsigned long long v = H[k + (size_t)nbin * pat];
      if (!v) continue;
      hc[k + (size_t)nbin * nr] += v;
      for (int tt = 0; tt < 6; ++tt) {
        if (!((pat >> term_gate(tt)) & 1)) continue;
        const int npr = ((pat >> term_pu(tt)) & 1) + ((pat >> term_pv(tt)) & 1);
        dc[k + (size_t)nbin * tt + (size_t)nbin * 6 * npr] += v;
      }
    }
  }
}

void quad_cot_lines(const double* cot2, const double* cot3, const double* cotN,
                    const double* cotR, int nbin, double* out) {
  for (int k = 0; k < nbin; ++k) {
    double* c = out + (size_t)k * kCotLine;
    c[0] = cot2[k];
    c[1] = cot2[k] + (cot3 ? cot3[k] : 0.0);
    for (int tt = 0; tt < 6; ++tt) {
      const size_t kt = k + (size_t)nbin * tt;
      c[2 + tt] = cotN ? cotN[kt] : 0.0;
      c[8 + tt] = c[2 + tt] + (cotR ? cotR[kt] : 0.0);
    }
    c[14] = c[15] = 0.0;
  }
}

}  // namespace gr

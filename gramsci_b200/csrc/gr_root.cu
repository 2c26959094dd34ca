// 3PCF triangle counting from the cell index: replaces query_graph_3pcf_all
// (src/gramsci.F90:463-510) together with the neighbour graph it reads
// (create_graph, :288-348).
//
// A warp takes a root point, collects its neighbours with larger labels from
// the cells around it into shared memory (position, bins of the edge to the
// root, weight) and tests every pair of them: the pair is the third edge of a
// triangle exactly when its separation lies in (rmin, rmax).  No graph is
// built and no row of another point is read.  Each triangle is found once,
// from its smallest label, and adds to the histogram of every non-buffer
// vertex.  Without mu bins these share one bin: the triangle is one update,
// made on the spot, that counts as often as it has non-buffer vertices.  With
// mu bins (MU) each vertex has its own bin, from the cosines of its two
// edges: hits go to a queue and are binned 32 at a time with every lane busy.
// (Collecting whole neighbourhoods instead, one update per rooted triangle
// without the third edge's cosine, tests four times the pairs: 1.36 ms against
// 0.72 ms on 400,000 points with 5 mu bins.)
//
// Short rows are taken up to kGroup roots of a cell at a time: the
// candidates are loaded once and tested against each root, the members of all
// rows are binned together, and one queue takes the hits of all of them.
// With a row of 14 members for 32 lanes each of these steps would run half
// empty for a single root.
//
// Pairs without mu bins: lane i holds neighbour x = i (32 at a time) in
// registers and meets neighbour y = x + j (mod k) in step j = 1 .. k/2, so
// every unordered pair comes up exactly once, y is read from consecutive
// shared words, and no pair index is inverted.  The last x's of a row, fewer than 32, share the warp:
// groups of lanes hold the same x's and take every G-th step.
//
// ADJ: the weight gradient, every sum of it an integer.  Without mu bins the
// pair's coefficient times the weight of y is summed in the lane that holds x,
// times the weight of x in y's shared accumulator (each y belongs to one lane
// per step, so plain reads and writes do, a warp barrier between steps), both
// in signed 64-bit fixed point with room for the row's weights and no more
// (T.rscale in the cotangents' table, for a full row of the largest weight, and
// a power of two in the row's weights); a row's sums, times the root's weight,
// go to the 128-bit fixed-point totals once.  With mu bins the queued hits add
// to signed 64-bit fixed-point sums per neighbour (the scale leaves room for
// 1024 terms).  The root's own sum has 128 bits.  Rounding of an entry without
// mu bins, rms in units of 2^-53 of the sum of its terms' sizes, lognormal and
// equal weights: rows of 14 members 0.21 and 0.22, of 170 0.03 and 0.03, of 600
// 0.13 and 0.35 (positive cotangents 0.6).  FP64 sums in their place: 0.22 and
// 0.21, 0.05 and 0.10, 0.12 and 0.96 (12: equal terms round alike); terms
// rounded at the totals' scale, as the hash-probe kernel does: 67 and 13, 3.4
// and 5.0, 0.6 and 3.6 (2.6).  The integers cost 76.8 -> 78.5 ms on 600,000
// points with rows of 170.
//
// Rows longer than a warp's capacity are listed and taken by a second launch
// (LONG) with one block per root and the row in global memory; its adjoint
// meets every ordered pair, so that only x's are summed.
//
// Bound by instruction issue (72% of the slots at 24 warps per SM, registers
// the limit; DRAM idle): about 100 warp instructions per 32 pairs without mu
// bins, half of which are triangles.  Against the graph build and the triangle
// kernel over its rows: 600,000 points with rows of 170, gradient and sums
// 153 -> 79 ms; 160,000 points with rows of 14, 346 -> 222 us; 400,000 points
// with 5 mu bins and rows of 14, 800 -> 720 us, of which collecting the rows
// takes 250, the pair tests 180 and the binning of the triangles 290.
#include <algorithm>

#include "gr_kernels.cuh"

namespace gr {

namespace {

constexpr int kRootWarps = 24;  // at most; 85 registers
constexpr int kLongWarps = 4;  // many small blocks: one collects its row while others count
constexpr size_t kSmemLimit = 227 * 1024;
constexpr int kCfgTableBins = 16;  // nbins up to which the configuration table is used

// Code of a row member, one byte each, in its position's fourth component:
// radial bin of its edge to the root (times nbins with a configuration
// table), mu bins of that edge seen from the root and from the member, flags.
__device__ __forceinline__ int code_byte(int code, int b) { return (code >> (8 * b)) & 0xff; }
__device__ __forceinline__ bool code_random(int code) { return code & (FLAG_RANDOM << 24); }
__device__ __forceinline__ bool code_buffer(int code) { return code & (FLAG_BUFFER << 24); }

constexpr int kGroup = 4;       // roots taken together, at most
constexpr int kRootQueue = 64;  // hits of a warp: fewer than 32 left and 32 pushed

// A root of the group.
struct GroupRoot {
  float4 pos;   // with its flags (pos4_flags)
  double w;
  int p, id;
};

struct RowPtrs {
  float4* pos;
  double* w;
  unsigned long long* g;  // ADJ: 64-bit fixed-point gradient (not MU: over the root's weight)
  int* q;     // labels
  int* id;    // catalogue ids (MU with an asymmetric normal table)
};

struct RootLayout {
  size_t off_cnt, off_lim, off_cot, off_fsc, off_norm, off_rank, off_cfg, off_warp;
  size_t o_w, o_g, o_q, o_id, o_seg, o_rng, o_hit, o_root, warp_bytes, total;
};

__host__ __device__ inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Entries of a root's candidate list: half the capacity for each of a group
// (a root with more is taken alone, with the lists of all).
__host__ __device__ inline int seg_cap(int cap, int group) { return group > 1 ? cap / 2 : cap; }

// cap 0: no rows in shared memory (LONG), one set of small tables per block.
__host__ __device__ inline RootLayout root_layout(int nh, int nmu, int nbins, int cap, bool shist,
                                                  bool weighted, bool counts, int nwarps, bool adj,
                                                  bool mu, bool ids, int group) {
  RootLayout L;
  size_t o = 0;
  L.off_cnt = o;
  if (shist && counts) o += (size_t)nh * 8;
  L.off_lim = o;
  if (shist && weighted) o += (size_t)nh * 16;
  L.off_cot = o;
  if (adj) o += (size_t)nh / 4 * 2 * 8;  // cot2, cot2 - cot3
  L.off_fsc = o;
  o += 4 * 8;
  L.off_norm = o;
  o = align_up(o + (size_t)nmu * nmu, 8);
  L.off_rank = o;
  o = align_up(o + sizeof(int) * 3 * (size_t)(nbins + 2), 8);
  L.off_cfg = o;
  if (nbins <= kCfgTableBins) o += sizeof(uint16_t) * (size_t)nbins * nbins * nbins;
  o = align_up(o, 16);
  L.off_warp = o;
  size_t w = (size_t)cap * 16;
  L.o_w = w;   if (weighted || adj) w += (size_t)cap * 8;
  L.o_g = w;   if (adj) w += (size_t)cap * 8;
  L.o_q = w;   w += (size_t)cap * 4;
  L.o_id = w;  if (ids) w += (size_t)cap * 4;
  L.o_seg = w; w += (size_t)group * seg_cap(cap, group) * 4;
  L.o_rng = w; w += 16 * sizeof(int);
  L.o_hit = w; if (mu && cap > 0) w += kRootQueue * sizeof(uint32_t);
  w = align_up(w, 16);
  L.o_root = w; w += kGroup * sizeof(GroupRoot);
  L.warp_bytes = align_up(w, 16);
  L.total = o + L.warp_bytes * (cap > 0 ? nwarps : 1);
  return L;
}

// x (any finite double below 2^94 in size) as a signed 128-bit integer,
// rounded once.
__device__ __forceinline__ Fix128 fix_from_double(double x) {
  const long long h = __double2ll_rd(x * 0x1p-32);
  const double rest = fma((double)h, -0x1p32, x);  // exact, in [0, 2^32]
  Fix128 v;
  v.lo = (unsigned long long)h << 32;
  v.hi = (unsigned long long)(h >> 32);
  const unsigned long long r = (unsigned long long)__double2ll_rn(rest);
  v.lo += r;
  v.hi += v.lo < r ? 1ull : 0ull;
  return v;
}

// 2^e, and the number of bits that n - 1 takes (n > 0: the least e with 2^e >= n).
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((1023 + e) << 20, 0); }
__device__ __forceinline__ int bits_of(int n) { return 32 - __clz(max(n, 1) - 1); }

__device__ __forceinline__ void fix_plus(Fix128& a, const Fix128& b) {
  a.lo += b.lo;
  a.hi += b.hi + (a.lo < b.lo ? 1ull : 0ull);
}

// Where integer counts go.
enum : int {
  kNoCounts = 0,
  kWithSums = 1,    // shared or global memory like the sums (SHIST)
  kCountsApart = 2  // global memory, the sums in shared memory
};

template <bool MU, bool WEIGHTED, int CMODE, bool SHIST, bool ADJ, bool BUF, bool LONG>
__global__ void __launch_bounds__(LONG ? kLongWarps * 32 : kRootWarps * 32, LONG ? 5 : 1)
    root3_kernel(DevCatalog C, RootParams T, unsigned long long* __restrict__ g_cnt,
                 unsigned long long* __restrict__ g_lim, unsigned long long* __restrict__ stats,
                 int* __restrict__ work, int* __restrict__ long_list, RootLong R,
                 const double* __restrict__ cot2, const double* __restrict__ cot3, double gscale,
                 unsigned long long* __restrict__ g_lo, unsigned long long* __restrict__ g_hi) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr bool W = WEIGHTED || ADJ;
  constexpr bool COUNTS = CMODE != kNoCounts, SCOUNTS = SHIST && CMODE == kWithSums;
  constexpr bool ROWSUM = ADJ && (!MU || LONG);  // sums over the root's weight, at T.rscale
  const PairParams& P = T.P;
  const int nb = T.nbins, ncfg = T.ncfg;
  const int nbin = ncfg * T.nmu, nh = nbin * 4;
  const bool ids = MU && T.asym;
  const RootLayout L = root_layout(nh, T.nmu, nb, LONG ? 0 : T.cap, SHIST, WEIGHTED, SCOUNTS,
                                   blockDim.x >> 5, ADJ, MU, ids, LONG ? 1 : T.group);
  unsigned long long* const s_cnt =
      SCOUNTS ? reinterpret_cast<unsigned long long*>(smem + L.off_cnt) : g_cnt;
  unsigned long long* const s_lim =
      SHIST ? reinterpret_cast<unsigned long long*>(smem + L.off_lim) : g_lim;
  double* const s_cot = reinterpret_cast<double*>(smem + L.off_cot);
  double* const s_fsc = reinterpret_cast<double*>(smem + L.off_fsc);
  uint8_t* const s_norm = smem + L.off_norm;
  int* const s_F = reinterpret_cast<int*>(smem + L.off_rank);
  uint16_t* const s_cfg = reinterpret_cast<uint16_t*>(smem + L.off_cfg);
  const int nb2 = nb + 2;
  const bool table = nb <= kCfgTableBins;
  // configuration of three radial bins from 0 (symmetric bin table,
  // gramsci.F90:1459-1474; -equi: the bin of three equal ones)
  auto rank3 = [&](int a, int b, int c) -> unsigned {
    if (T.equi) return (unsigned)a;  // three equal ones, tested before
    sort3i(a, b, c);
    ++a;
    ++b;
    ++c;
    return (unsigned)((s_F[a] - s_F[1]) + (s_F[nb2 + b] - s_F[nb2 + a]) +
                      (s_F[2 * nb2 + c] - s_F[2 * nb2 + b]));
  };
  if (threadIdx.x < 4) s_fsc[threadIdx.x] = T.fscale[threadIdx.x];
  if (ADJ)
    for (int k = threadIdx.x; k < nbin; k += blockDim.x) {
      // without mu bins and buffer points a triangle counts three times
      const double f = (!MU && !BUF ? 3.0 : 1.0) * (ROWSUM ? T.rscale : 1.0);
      s_cot[k] = f * cot2[k];
      s_cot[nbin + k] = f * (cot3 ? cot2[k] - cot3[k] : cot2[k]);
    }
  if (SHIST)
    for (int k = threadIdx.x; k < nh; k += blockDim.x) {
      if (SCOUNTS) s_cnt[k] = 0ull;
      if (WEIGHTED) {
        s_lim[k] = 0ull;
        s_lim[nh + k] = 0ull;
      }
    }
  for (int k = threadIdx.x; k < T.nmu * T.nmu; k += blockDim.x) s_norm[k] = T.rsd ? T.normal[k] - 1 : 0;
  for (int k = threadIdx.x; k < 3 * nb2; k += blockDim.x) s_F[k] = T.rank.F[k / nb2][k % nb2];
  __syncthreads();
  if (table)
    for (int k = threadIdx.x; k < nb * nb * nb; k += blockDim.x)
      s_cfg[k] = (uint16_t)rank3(k % nb, (k / nb) % nb, k / (nb * nb));
  __syncthreads();

  const int lane = threadIdx.x & 31;
  const int wid = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  unsigned char* const wb = smem + L.off_warp + (LONG ? 0 : L.warp_bytes * wid);
  int* const s_rng = reinterpret_cast<int*>(wb + L.o_rng);  // candidate ranges: begin, prefix
  // queued hits: x | y << 12 | root << 24
  uint32_t* const s_hit = reinterpret_cast<uint32_t*>(wb + L.o_hit);
  int* const s_seg = reinterpret_cast<int*>(wb + L.o_seg);            // candidate lists
  GroupRoot* const s_root = reinterpret_cast<GroupRoot*>(wb + L.o_root);
  RowPtrs row;
  if (LONG) {
    const size_t at = (size_t)blockIdx.x * R.cap;
    row = RowPtrs{R.pos + at, R.w + at, nullptr, R.q + at, R.id + at};
  } else {
    row = RowPtrs{reinterpret_cast<float4*>(wb), reinterpret_cast<double*>(wb + L.o_w),
                  reinterpret_cast<unsigned long long*>(wb + L.o_g), reinterpret_cast<int*>(wb + L.o_q),
                  reinterpret_cast<int*>(wb + L.o_id)};
  }

  unsigned long long tris = 0, rooted = 0, probes = 0, edges = 0, cands = 0, rechecks = 0;

  // Ranges of the candidates of the roots p, p + 1, ... of one cell (labels
  // above p) into s_rng, their total returned.  Those of the last cell are
  // kept (lane k < 5 holds the k-th).
  constexpr int NR = 5;
  int last_cell = -1, beg = 0, end = 0;
  auto ranges = [&](int p, int cell) -> int {
    if (cell != last_cell) {
      last_cell = cell;
      GridParams g;
      const int* cs;
      int lkey;
      cell_grid(C, cell, g, cs, lkey);
      const int yz = lkey / g.nx, cx = lkey - yz * g.nx;
      if (lane < NR) forward_slot<1>(lane, p + 1, cx, cx, yz, g, cs, beg, end);
    }
    if (lane == 0) beg = p + 1;
    const int len = max(end - beg, 0);
    int incl = len;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    __syncwarp();
    if (lane < NR) {
      s_rng[lane] = beg;
      s_rng[8 + lane] = incl - len;
    }
    __syncwarp();
    return __shfl_sync(0xffffffffu, incl, NR - 1);
  };
  // Label of candidate f; kr walks along with increasing f.
  auto candidate = [&](int f, int& kr) -> int {
    while (kr + 1 < NR && f >= s_rng[8 + kr + 1]) ++kr;
    return s_rng[kr] + (f - s_rng[8 + kr]);
  };
  auto in_band = [&](const float4& a, const float4& c) -> bool {
    const float dx = c.x - a.x, dy = c.y - a.y, dz = c.z - a.z;
    const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    return d2 < P.rmax2_hi && d2 > P.rmin2_lo;
  };
  // Bins of the edge root - member, packed with the member's flags; -1: no edge.
  auto edge_code = [&](int p, const float4& pr, int q, const float4& c) -> int {
    int b0 = 0, m0 = 0, st = P.f32 ? bin_pair_f32(pr, c, P, b0, m0) : 2;
    int mrev = P.nmu - 1 - m0;
    if (st == 2) {
      int b = 1, mf = 1, mr = 1;
      rechecks++;
      st = edge_f64(C.posd[p], C.posd[q], P, b, mf, mr) ? 1 : 0;
      b0 = b - 1;
      m0 = mf - 1;
      mrev = mr - 1;
    }
    if (st != 1) return -1;
    return (table ? b0 * nb : b0) | (m0 << 8) | (mrev << 16) |
           (pos4_random(c) ? FLAG_RANDOM << 24 : 0) | (pos4_buffer(c) ? FLAG_BUFFER << 24 : 0);
  };
  auto put_member = [&](int at, int q, float4 c, int code) {
    c.w = __int_as_float(code);
    row.pos[at] = c;
    row.q[at] = q;
    if (W) row.w[at] = C.w[q];
    if (ids) row.id[at] = C.orig[q];
    if (ADJ && !LONG) row.g[at] = 0ull;
  };

  // rooted triangles (BUF: else three each) and triangles of this lane
  unsigned nroot = 0, ntri = 0;

  // MU: the triangle of root R and members x, y (its edge x-y is known to
  // exist).  Histograms, or the sum over its non-buffer vertices of their
  // bins' cotangents (ADJ), returned.
  auto triangle = [&](const GroupRoot& R, int x, int y) -> double {
    const float4 px = row.pos[x], py = row.pos[y];
    const int cx = __float_as_int(px.w), cy = __float_as_int(py.w);
    int st = 2, b0 = 0, mx = 0, my = 0;  // edge x-y: radial bin, mu bin from x and from y
    if (P.f32) st = bin_pair_f32(px, py, P, b0, mx);
    my = P.nmu - 1 - mx;
    if (st == 2) {
      int b = 1, mf = 1, mr = 1;
      edge_f64(C.posd[row.q[x]], C.posd[row.q[y]], P, b, mf, mr);
      b0 = b - 1;
      mx = mf - 1;
      my = mr - 1;
    }
    const int xr = code_byte(cx, 0), yr = code_byte(cy, 0);
    if (T.equi && !(xr == yr && b0 * (table ? nb : 1) == xr)) return 0.0;
    const unsigned cfg = table ? s_cfg[xr * nb + yr + b0] : rank3(xr, yr, b0);
    // find_normal bin of each vertex, its two edges in catalogue-id order
    const int nmu = T.nmu;
    const int xf = code_byte(cx, 1), xv = code_byte(cx, 2);
    const int yf = code_byte(cy, 1), yv = code_byte(cy, 2);
    int i0 = xf + nmu * yf, i1 = xv + nmu * mx, i2 = yv + nmu * my;
    if (ids) {
      const int ix = row.id[x], iy = row.id[y];
      if (ix > iy) i0 = yf + nmu * xf;    // root: x, y
      if (R.id > iy) i1 = mx + nmu * xv;  // x: root, y
      if (R.id > ix) i2 = my + nmu * yv;  // y: root, x
    }
    const int m0 = s_norm[i0], m1 = s_norm[i1], m2 = s_norm[i2];
    const int nr = (pos4_random(R.pos) ? 1 : 0) + (code_random(cx) ? 1 : 0) + (code_random(cy) ? 1 : 0);
    const bool c0 = !BUF || !pos4_buffer(R.pos), c1 = !BUF || !code_buffer(cx),
               c2 = !BUF || !code_buffer(cy);
    if (BUF) nroot += (c0 ? 1u : 0u) + (c1 ? 1u : 0u) + (c2 ? 1u : 0u);
    ntri += (!BUF || c0 || c1 || c2) ? 1u : 0u;
    if (ADJ) {
      const double* t = s_cot + cfg + (nr == 3 ? nbin : 0);
      double cf = 0.0;
      if (c0) cf += t[ncfg * m0];
      if (c1) cf += t[ncfg * m1];
      if (c2) cf += t[ncfg * m2];
      return cf;
    }
    long long v = 0;
    if (WEIGHTED) v = __double2ll_rn(R.w * row.w[x] * row.w[y] * s_fsc[nr]);
    const int e = (int)cfg + nbin * nr;
    auto add = [&](int m, int n, bool count, bool sum) {
      if (COUNTS && count) hist_count_add<SCOUNTS>(s_cnt, nh, e + ncfg * m, (unsigned)n);
      if (WEIGHTED && sum) hist_fix_add<SHIST>(s_lim, nh, e + ncfg * m, v * n);
    };
    constexpr bool GCOUNTS = COUNTS && !SCOUNTS, GSUMS = WEIGHTED && !SHIST;
    if (SHIST) {
      // vertices in the same bin are not merged first: with 32 lanes some lane
      // needs each of the three updates
      if (c0) add(m0, 1, !GCOUNTS, true);
      if (c1) add(m1, 1, !GCOUNTS, true);
      if (c2) add(m2, 1, !GCOUNTS, true);
    }
    if (GCOUNTS || GSUMS) {
      // in global memory every lane's update counts, so vertices in the same
      // bin are merged
      int n0 = c0 ? 1 : 0, n1 = c1 ? 1 : 0, n2 = c2 ? 1 : 0;
      if (n1 && m1 == m0) {
        n1 += n0;
        n0 = 0;
      }
      if (n2 && m2 == m1) {
        n2 += n1;
        n1 = 0;
      }
      if (n2 && m2 == m0) {
        n2 += n0;
        n0 = 0;
      }
      if (n0) add(m0, n0, GCOUNTS, GSUMS);
      if (n1) add(m1, n1, GCOUNTS, GSUMS);
      if (n2) add(m2, n2, GCOUNTS, GSUMS);
    }
    return 0.0;
  };

  // MU: one queued hit.
  // this lane's part of the current root's gradient, times 2^shift (MU: 2^10)
  Fix128 gp = {0ull, 0ull};
  auto drain = [&](int e) {
    const uint32_t h = s_hit[e];
    const int x = (int)(h & 0xfffu), y = (int)((h >> 12) & 0xfffu);
    const GroupRoot& R = s_root[h >> 24];
    const double cf = triangle(R, x, y);
    if (ADJ && cf != 0.0) {
      const double wx = row.w[x], wy = row.w[y];
      fix_acc(gp, cf * (wx * wy), 1024.0 * gscale);  // a single term, without the room for 1024
      smem_add_s64(&row.g[x], __double2ll_rn(cf * (R.w * wy) * gscale));
      smem_add_s64(&row.g[y], __double2ll_rn(cf * (R.w * wx) * gscale));
    }
  };
  int qn = 0;  // queued hits

  // Every pair of the k members from `off` on, the row of root ri of the group
  // (LONG: of the x's of this warp); `last`: nothing stays queued.
  auto pairs = [&](int ri, int off, int k, bool last) {
    constexpr bool ORDERED = ADJ && LONG;      // every ordered pair, x's summed only
    constexpr bool QUEUE = MU && !LONG;
    constexpr bool ONE = ADJ && !MU && !LONG;  // plain updates of y: one lane per y
    const GroupRoot& R = s_root[ri];
    const float4* const pos = row.pos + off;
    const double* const rw = row.w + off;
    long long* const rg = reinterpret_cast<long long*>(row.g) + off;
    const double wp = W ? R.w : 0.0;
    int shift = ROWSUM ? 0 : 10;  // of the root's sum, and of the row's weights
    if (ROWSUM && !LONG) {
      // the sum of the weights' sizes, in units of 2^-20 of the largest
      unsigned sum = 0;
      for (int x = lane; x < k; x += 32)
        sum += min(__double2uint_ru(fabs(rw[x]) * T.winv), (1u << 20) + 1u);
      sum = __reduce_add_sync(0xffffffffu, sum);
      shift = min(32, max(0, 20 + bits_of(T.cap) - bits_of((int)sum)));
      for (int x = lane; x < k; x += 32) row.w[off + x] *= pow2(shift);
      __syncwarp();
    }
    // of the row's sums in units of the totals
    const double rinv = ROWSUM ? gscale / T.rscale * pow2(-shift) : 0.0;
    // Whether the pair x, y is an edge, and (not MU: binned later) its radial
    // bin from 0; no branch but the rare one into FP64, which lanes without a
    // pair (on = false) must not take.  The bounds send every pair there when
    // the FP32 path is off.
    const float in_hi = P.f32 ? P.rmax2_lo : -1.0f;
    const float guard = P.f32 ? P.tguard : INFINITY;
    auto edge = [&](const float4& px, const float4& py, int x, int y, bool on, int& b0) -> bool {
      const float dx = py.x - px.x, dy = py.y - px.y, dz = py.z - px.z;
      const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
      bool hit, exact;
      if (MU) {
        hit = d2 < in_hi && d2 > P.rmin2_hi;
        exact = !hit && d2 < P.rmax2_hi && d2 > P.rmin2_lo;
      } else {
        // radial part of bin_pair_f32
        const float t = fmaf(d2 * rsqrt_approx(d2), P.f_inv_dr, P.f_t0);
        const float tr = __fadd_rn(t, 12582912.0f);
        const float tn = __fadd_rn(tr, -12582912.0f);
        b0 = __float_as_int(tr) - 0x4B400000 - (t < tn ? 1 : 0);
        hit = (unsigned)b0 < (unsigned)nb;
        exact = !(fabsf(t - tn) >= guard);
      }
      if (exact && on) {
        int b = 1;
        hit = d2 < P.rmax2_hi && d2 > P.rmin2_lo &&
              edge_radial_f64(C.posd[row.q[off + x]], C.posd[row.q[off + y]], P, b);
        b0 = b - 1;
      }
      return hit && on;
    };
    if (QUEUE) {
      // all pairs in row-major order over the lanes (closed-form inversion of
      // the triangular pair index); at least one step, without pairs if need
      // be, for what is queued
      const int npair = k * (k - 1) / 2, k2m1 = 2 * k - 1;
      for (int t0 = 0;; t0 += 32) {
        const bool on = t0 + lane < npair;
        const int t = on ? t0 + lane : 0;
        int x = pair_row_biased(k2m1, t);
        if (k > kPairRowExact) {
          x = max(0, min(x, k - 2));
          if ((x + 1) * (k2m1 - x - 1) / 2 <= t) ++x;
          if (x * (k2m1 - x) / 2 > t) --x;
        }
        const int y = on ? t - (int)((unsigned)(x * (k2m1 - x)) >> 1) + x + 1 : 0;
        x = on ? x : 0;
        int b0;
        const bool hit = edge(pos[x], pos[y], x, y, on, b0);
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (hit)
          s_hit[qn + __popc(m & lt)] =
              (uint32_t)((off + x) | ((off + y) << 12)) | ((uint32_t)ri << 24);
        qn += __popc(m);
        // 32 hits, and what is left after the last row's last pairs
        const bool end = t0 + 32 >= npair, fin = (ADJ || last) && end;
        while (qn >= 32 || (fin && qn > 0)) {
          const int nq = min(qn, 32);
          __syncwarp();
          qn -= nq;
          if (lane < nq) drain(qn + lane);
          __syncwarp();
        }
        if (end) break;
      }
    } else {
      const bool rran = pos4_random(R.pos), rbuf = BUF && pos4_buffer(R.pos);
      const int nw = LONG ? (int)(blockDim.x >> 5) : 1;
      const int jmax = ORDERED ? k - 1 : k >> 1;
      for (int base = LONG ? 32 * wid : 0; base < k; base += 32 * nw) {
        const int r = min(32, k - base);
        // groups of lanes that share the warp's x's (the quotients' fractions
        // are at least 1/64 from 0 and 1)
        const float inv = __fdividef(1.0f, (float)r);
        const int G = ONE ? 1 : (int)(32.5f * inv);
        const int grp = (int)(((float)lane + 0.5f) * inv);
        const bool act = grp < G;
        const int x = act ? base + lane - grp * r : base;
        const float4 px = pos[x];
        const int cx = __float_as_int(px.w);
        const int xr = code_byte(cx, 0);
        const int xrow = table ? xr * nb : xr;
        const bool xran = code_random(cx);
        const double wx = W ? rw[x] : 0.0;
        const int nr0 = (rran ? 1 : 0) + (xran ? 1 : 0);
        const double wpx0 = WEIGHTED && !MU ? wp * wx * s_fsc[nr0] : 0.0;
        const double wpx1 = WEIGHTED && !MU ? wp * wx * s_fsc[nr0 + 1] : 0.0;
        const int xbase = ADJ ? (rran && xran ? nbin : 0) : nbin * nr0;
        const int xn = BUF ? (rbuf ? 0 : 1) + (code_buffer(cx) ? 0 : 1) : 2;
        long long gx = 0;
        for (int j0 = 1; j0 <= jmax; j0 += G) {
          const int j = j0 + grp;
          const bool on = act && j <= jmax && (ORDERED || 2 * j != k || x < j);
          int y = on ? x + j : 0;
          if (y >= k) y -= k;
          const float4 py = pos[y];
          int b0 = 0;
          bool hit = edge(px, py, x, y, on, b0);
          const int cy = __float_as_int(py.w);
          const int yr = code_byte(cy, 0);
          if (!MU && T.equi) hit = hit && xr == yr && b0 * (table ? nb : 1) == xr;
          if (hit) {
            // an ordered pair's triangle counts from its smaller member
            const unsigned root0 = nroot, tri0 = ntri;
            if (MU) {
              const double cf = triangle(R, off + x, off + y);
              if (ADJ) gx += __double2ll_rn(cf * rw[y]);
            } else {
              int e = (int)(table ? s_cfg[xrow + yr + b0] : rank3(xrow, yr, b0));
              const bool yran = code_random(cy);
              const int n = BUF ? xn + (code_buffer(cy) ? 0 : 1) : 3;
              if (BUF) nroot += (unsigned)n;
              ntri += !BUF || n > 0 ? 1u : 0u;
              if (ADJ) {
                // the cotangents hold the factor 3 of a catalogue without buffers
                double cf = s_cot[e + (yran ? xbase : 0)];
                if (BUF) cf *= (double)n;
                gx += __double2ll_rn(cf * rw[y]);
                if (!ORDERED) rg[y] += __double2ll_rn(cf * wx);
              } else {
                e += xbase + (yran ? nbin : 0);
                if (COUNTS) hist_count_add<SCOUNTS>(s_cnt, nh, e, (unsigned)n);
                if (WEIGHTED)
                  hist_fix_add<SHIST>(s_lim, nh, e,
                                      __double2ll_rn((yran ? wpx1 : wpx0) * rw[y]) * n);
              }
            }
            if (ORDERED && y < x) {
              nroot = root0;
              ntri = tri0;
            }
          }
          if (ONE) __syncwarp();
        }
        if (ORDERED) {
          // all of x's sum; every ordered pair was met, so the root's is half
          for (int g2 = 1; g2 < G; ++g2) {
            const long long o = __shfl_sync(0xffffffffu, gx, min(31, lane - grp * r + g2 * r));
            if (grp == 0) gx += o;
          }
          if (act && grp == 0) {
            const double sx = __ll2double_rn(gx) * rinv;
            fix_plus(gp, fix_from_double(0.5 * wx * sx));
            const int qx = row.q[off + x];
            const Fix128 v = fix_from_double(sx * wp);
            if (v.lo | v.hi) fix_merge(&g_lo[qx], &g_hi[qx], v.lo, v.hi);
          }
        } else if (ONE) {
          if (act) {
            rg[x] += gx;
            fix_plus(gp, fix_from_double(wx * (__ll2double_rn(gx) * rinv)));
          }
          __syncwarp();
        }
      }
    }
    if (ADJ && !LONG) {
      // the row's gradients
      for (int x = off + lane; x < off + k; x += 32) {
        const int q = row.q[x];
        Fix128 v;
        if (MU) {
          v.lo = row.g[x];
          v.hi = (long long)v.lo < 0 ? ~0ull : 0ull;
        } else {
          v = fix_from_double(__ll2double_rn((long long)row.g[x]) * rinv * wp);
        }
        if (v.lo | v.hi) fix_merge(&g_lo[q], &g_hi[q], v.lo, v.hi);
      }
    }
    if (ADJ) {
      Fix128 v = fix_warp_sum(gp);
      if (shift > 0) {  // to the totals' scale, rounded
        fix_plus(v, Fix128{1ull << (shift - 1), 0ull});
        v.lo = (v.lo >> shift) | (v.hi << (64 - shift));
        v.hi = (unsigned long long)((long long)v.hi >> shift);
      }
      if (lane == 0 && (v.lo | v.hi)) fix_merge(&g_lo[R.p], &g_hi[R.p], v.lo, v.hi);
      gp = Fix128{0ull, 0ull};
    }
    if (BUF) rooted += nroot;
    tris += ntri;
    nroot = ntri = 0;
    if (lane == 0 && k > 0 && (!LONG || wid == 0)) {
      edges += (unsigned long long)k;
      probes += (unsigned long long)k * (unsigned)(k - 1) / 2;
    }
  };

  if (LONG) {
    __shared__ int s_item, s_k;
    for (;;) {
      __syncthreads();
      if (threadIdx.x == 0) s_item = atomicAdd(work, 1);
      __syncthreads();
      if (s_item >= R.n) break;
      const int p = long_list[s_item];
      if (wid == 0) {
        // the first warp collects the row
        const float4 pr = C.pos4[p];
        if (lane == 0) s_root[0] = GroupRoot{pr, W ? C.w[p] : 0.0, p, ids ? C.orig[p] : 0};
        const int total = ranges(p, C.cell_key[p]);
        if (lane == 0) cands += (unsigned long long)total;
        int k = 0, kr = 0;
        for (int f0 = 0; f0 < total; f0 += 32) {
          const int f = f0 + lane;
          int q = 0, code = -1;
          float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
          if (f < total) {
            q = candidate(f, kr);
            c = C.pos4[q];
            if (in_band(pr, c)) code = edge_code(p, pr, q, c);
          }
          const unsigned m = __ballot_sync(0xffffffffu, code >= 0);
          const int at = k + __popc(m & lt);
          if (code >= 0 && at < R.cap) put_member(at, q, c, code);
          k += __popc(m);
        }
        if (lane == 0) {
          if (k > R.cap) {  // the host reports it
            atomicExch(&stats[7], 1ull);
            k = 0;
          }
          s_k = k;
        }
      }
      __syncthreads();
      pairs(0, 0, s_k, true);
    }
  } else {
    const int group = T.group, seg = seg_cap(T.cap, group);
    for (;;) {
      int p = 0;
      if (lane == 0) p = atomicAdd(work, T.chunk);
      p = __shfl_sync(0xffffffffu, p, 0);
      if (p >= C.n) break;
      const int end_root = min(p + T.chunk, C.n);
      bool alone = false;  // the next root's list exceeds a group's
      while (p < end_root) {
        // the next roots of one cell, at most `group`
        const int cell = C.cell_key[p];
        const int mine = min(p + lane, end_root - 1);
        const unsigned same =
            __ballot_sync(0xffffffffu, p + lane < end_root && C.cell_key[mine] == cell);
        int ng = alone ? 1 : min(group, __popc(same));
        __syncwarp();
        if (lane < ng)
          s_root[lane] = GroupRoot{C.pos4[p + lane], W ? C.w[p + lane] : 0.0, p + lane,
                                   ids ? C.orig[p + lane] : 0};
        const int total = ranges(p, cell);
        // candidates inside the outer bounds of the guard band, a list per root
        const int lim = alone ? group * seg : seg;
        int n0 = 0, n1 = 0, n2 = 0, n3 = 0, kr = 0;
        float4 r[kGroup];
#pragma unroll
        for (int i = 0; i < kGroup; ++i) r[i] = s_root[i < ng ? i : 0].pos;
        for (int f0 = 0; f0 < total; f0 += 32) {
          const int f = f0 + lane;
          int q = -1;  // no candidate
          float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
          if (f < total) {
            q = candidate(f, kr);
            c = C.pos4[q];
          }
          auto test = [&](int i, int& n) {
            const bool in = q > p + i && in_band(r[i], c);
            const unsigned m = __ballot_sync(0xffffffffu, in);
            const int at = n + __popc(m & lt);
            if (in && at < lim) s_seg[i * seg + at] = q;
            n += __popc(m);
          };
          test(0, n0);
          if (ng > 1) test(1, n1);
          if (ng > 2) test(2, n2);
          if (ng > 3) test(3, n3);
        }
        __syncwarp();
        if (n0 > min(lim, T.cap)) {
          if (!alone && n0 <= T.cap) {
            alone = true;  // again, with room for its list
            continue;
          }
          // beyond a warp's capacity: listed for the second launch
          if (lane == 0) {
            long_list[(int)atomicAdd(&stats[6], 1ull)] = p;
            atomicMax(&stats[8], (unsigned long long)n0);
          }
          alone = false;
          ++p;
          continue;
        }
        alone = false;
        // the roots whose members fit together
        if (n1 > seg || n0 + n1 > T.cap) ng = min(ng, 1);
        if (n2 > seg || n0 + n1 + n2 > T.cap) ng = min(ng, 2);
        if (n3 > seg || n0 + n1 + n2 + n3 > T.cap) ng = min(ng, 3);
        if (ng < 2) n1 = 0;
        if (ng < 3) n2 = 0;
        if (ng < 4) n3 = 0;
        const int o1 = n0, o2 = o1 + n1, o3 = o2 + n2, n = o3 + n3;
        // their bins; pairs that are no edges after all are dropped
        int k = 0, k0 = 0, k1 = 0, k2 = 0;  // members so far, of all and of the first roots
        for (int e0 = 0; e0 < n; e0 += 32) {
          const int e = e0 + lane;
          const int i = (e >= o1 ? 1 : 0) + (e >= o2 ? 1 : 0) + (e >= o3 ? 1 : 0);
          int q = 0, code = -1;
          float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
          if (e < n) {
            const int o = i == 0 ? 0 : (i == 1 ? o1 : (i == 2 ? o2 : o3));
            q = s_seg[i * seg + (e - o)];
            c = C.pos4[q];
            code = edge_code(p + i, s_root[i].pos, q, c);
          }
          const unsigned m = __ballot_sync(0xffffffffu, code >= 0);
          if (code >= 0) put_member(k + __popc(m & lt), q, c, code);
          // lanes of root i, from lane o_i - e0 on
          auto below = [&](int o) {
            return o <= e0 ? 0u : (o >= e0 + 32 ? 0xffffffffu : (1u << (o - e0)) - 1u);
          };
          k0 += __popc(m & below(o1));
          k1 += __popc(m & below(o2));
          k2 += __popc(m & below(o3));
          k += __popc(m);
        }
        __syncwarp();
        // k0, k1, k2: ends of the first three rows
        if (lane == 0) cands += (unsigned long long)total * ng - (unsigned)(ng * (ng - 1) / 2);
        // one call site: four copies of the pair and binning code ran 1.8
        // times slower (instruction fetch)
#pragma unroll 1
        for (int i = 0; i < ng; ++i) {
          const int o = i == 0 ? 0 : (i == 1 ? k0 : (i == 2 ? k1 : k2));
          const int o2 = i + 1 == ng ? k : (i == 0 ? k0 : (i == 1 ? k1 : k2));
          pairs(i, o, o2 - o, i + 1 == ng);
        }
        __syncwarp();
        p += ng;
      }
    }
  }
  if (!BUF) rooted = 3 * tris;
  unsigned long long sums[6] = {tris, rooted, probes, edges, cands, rechecks};
#pragma unroll
  for (int t = 0; t < 6; ++t) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sums[t] += __shfl_xor_sync(0xffffffffu, sums[t], o);
    if (lane == 0 && sums[t]) atomicAdd(&stats[t], sums[t]);
  }
  if (SHIST) {
    __syncthreads();
    for (int k = threadIdx.x; k < nh; k += blockDim.x) {
      if (SCOUNTS) {
        const unsigned long long v = hist_count_value(s_cnt, nh, k);
        if (v) atomicAdd(&g_cnt[k], v);
      }
      if (WEIGHTED) {
        unsigned long long lo, hi;
        hist_fix_value(s_lim, nh, k, lo, hi);
        if (lo | hi) fix_merge(&g_lim[k], &g_lim[nh + k], lo, hi);
      }
    }
  }
}

bool root_shist(int nh, bool weighted, bool counts) {
  return (size_t)nh * 8 * ((counts ? 1 : 0) + (weighted ? 2 : 0)) <= kMaxHistSmem;
}

// Warps of a block: as many as fit with rows of the wanted capacity, at
// least kMinWarps (the capacity is then what is left).
constexpr int kMinWarps = 12;
void root_shape(const RootParams& T, bool weighted, bool counts, bool shist, bool adj, int& nw,
                int& cap, size_t& smem) {
  const int nh = T.ncfg * T.nmu * 4;
  const bool mu = T.rsd != 0, ids = mu && T.asym;
  auto bytes = [&](int w, int c) {
    return root_layout(nh, T.nmu, T.nbins, c, shist, weighted, counts, w, adj, mu, ids, T.group).total;
  };
  nw = kRootWarps;
  cap = T.cap;
  while (nw > kMinWarps && bytes(nw, cap) > kSmemLimit) --nw;
  while (cap > 32 && bytes(nw, cap) > kSmemLimit) cap -= 32;
  while (nw > 1 && bytes(nw, cap) > kSmemLimit) --nw;
  smem = bytes(nw, cap);
  if (smem > kSmemLimit) throw Error{-2, "3PCF: per-warp shared memory exceeds the SM limit"};
}

struct RootArgs {
  unsigned long long *g_cnt, *g_lim;
  const double *cot2, *cot3;
  double gscale;
  unsigned long long *g_lo, *g_hi;
};

template <bool MU, bool BUF, bool LONG>
void launch_root(const DevCatalog& C, RootParams T, bool weighted, bool counts, bool adj,
                 const RootArgs& A, unsigned long long* stats, int* work, int* long_list,
                 const RootLong& R, cudaStream_t s) {
  const int nh = T.ncfg * T.nmu * 4;
  // all histograms in shared memory, else the sums alone: adding to counts in
  // global memory returns nothing to wait for
  const bool all = !adj && root_shist(nh, weighted, counts);
  const bool shist = all || (!adj && weighted && root_shist(nh, true, false));
  const bool scounts = counts && all;
  const bool ids = T.rsd && T.asym;
  int nw = kLongWarps;
  size_t smem = 0;
  int64_t blocks = 0;
  if (LONG) {
    smem = root_layout(nh, T.nmu, T.nbins, 0, shist, weighted && !adj, scounts, nw, adj, T.rsd != 0, ids, 1)
               .total;
    blocks = R.blocks;
  } else {
    if (weighted && !adj && !shist) {
      // sums in global memory: a warp waits for each update's old value, and
      // neighbours of a dense spot grabbed together end the launch alone (SMs
      // busy 61% of the time with four per grab).  With vertices of one bin
      // merged: 160,000 points, 1,540 configurations by 8 mu bins 0.61 -> 0.51
      // ms.
      T.chunk = std::max(1, std::min(T.chunk, (int)(C.n / ((int64_t)sm_count() * kRootWarps * 32))));
      T.group = std::min(T.group, T.chunk);
    }
    root_shape(T, weighted && !adj, scounts, shist, adj, nw, T.cap, smem);
    blocks = sm_count();
    const int64_t per = (int64_t)nw * T.chunk;
    const int64_t need = ((int64_t)C.n + per - 1) / per;
    if (blocks > need) blocks = need;
  }
  // room for as many terms as a row has members, below 2^63
  const int most = LONG ? R.cap : T.cap;
  int lg = 0;
  while (lg < 31 && ((int64_t)1 << lg) < most) ++lg;
  T.rscale = std::ldexp(T.rscale, 3 - lg);
  GR_CUDA_TRY(cudaMemsetAsync(work, 0, sizeof(int), s));
  auto go = [&](auto kfn) {
    GR_CUDA_TRY(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kfn<<<(unsigned)blocks, nw * 32, smem, s>>>(C, T, A.g_cnt, A.g_lim, stats, work, long_list, R,
                                                A.cot2, A.cot3, A.gscale, A.g_lo, A.g_hi);
  };
  if (adj) {
    go(root3_kernel<MU, false, kNoCounts, false, true, BUF, LONG>);
  } else if (weighted && counts) {
    if (all) go(root3_kernel<MU, true, kWithSums, true, false, BUF, LONG>);
    else if (shist) go(root3_kernel<MU, true, kCountsApart, true, false, BUF, LONG>);
    else go(root3_kernel<MU, true, kWithSums, false, false, BUF, LONG>);
  } else if (weighted) {
    if (shist) go(root3_kernel<MU, true, kNoCounts, true, false, BUF, LONG>);
    else go(root3_kernel<MU, true, kNoCounts, false, false, BUF, LONG>);
  } else {
    if (shist) go(root3_kernel<MU, false, kWithSums, true, false, BUF, LONG>);
    else go(root3_kernel<MU, false, kWithSums, false, false, BUF, LONG>);
  }
  GR_CHECK_LAUNCH();
}

void launch_either(const DevCatalog& C, const RootParams& T, bool weighted, bool counts, bool adj,
                   const RootArgs& A, unsigned long long* stats, int* work, int* long_list,
                   const RootLong* R, cudaStream_t s) {
  if (C.n <= 0) return;
  const RootLong none{};
  auto go = [&](auto f) { f(C, T, weighted, counts, adj, A, stats, work, long_list, R ? *R : none, s); };
  if (R) {
    if (T.rsd) go(launch_root<true, true, true>);
    else go(launch_root<false, true, true>);
  } else if (C.has_buffer) {
    if (T.rsd) go(launch_root<true, true, false>);
    else go(launch_root<false, true, false>);
  } else {
    if (T.rsd) go(launch_root<true, false, false>);
    else go(launch_root<false, false, false>);
  }
}

}  // namespace

void root3_plan(RootParams& T, int64_t n, double volume, double rmax) {
  const double ball = 4.18879020478639 * rmax * rmax * rmax;
  const double mean = 0.5 * (volume > 0.0 ? (double)n * std::min(1.0, ball / volume) : (double)n);
  T.group = mean <= 24.0 ? 4 : (mean <= 48.0 ? 2 : 1);
  // at most 1024: the adjoint's 64-bit sums
  const double all = T.group * mean;
  T.cap = std::min((int)std::min(all + 8.0 * std::sqrt(all) + 64.0, 1024.0) / 32 * 32 + 32, 1024);
  // a few groups per grab where the roots are many, for the cell's ranges
  const int64_t warps = (int64_t)sm_count() * kRootWarps;
  const int64_t per = n / (warps * 8);
  T.chunk = (int)std::min<int64_t>(4, std::max<int64_t>(1, per));
  if (T.chunk < T.group) T.group = T.chunk;
}

void launch_root3(const DevCatalog& C, const RootParams& T, bool weighted, bool counts,
                  unsigned long long* g_cnt, unsigned long long* g_lim, unsigned long long* stats,
                  int* work, int* long_list, const RootLong* R, cudaStream_t s) {
  const RootArgs A{g_cnt, g_lim, nullptr, nullptr, 0.0, nullptr, nullptr};
  launch_either(C, T, weighted, counts || !weighted, false, A, stats, work, long_list, R, s);
}

void launch_root3_adj(const DevCatalog& C, const RootParams& T, const double* cot2,
                      const double* cot3, double gscale, unsigned long long* g_lo,
                      unsigned long long* g_hi, unsigned long long* stats, int* work,
                      int* long_list, const RootLong* R, cudaStream_t s) {
  const RootArgs A{nullptr, nullptr, cot2, cot3, gscale, g_lo, g_hi};
  launch_either(C, T, false, false, true, A, stats, work, long_list, R, s);
}

}  // namespace gr

// Tile pair sweep for dense cells: the 2PCF pair binning of gr_pair.cu
// (create_graph + query_graph_2pcf, src/gramsci.F90:288-379) reorganised for
// cells holding tens to hundreds of points.
//
// A warp takes a cell from the work counter; its lanes hold 32 of the
// cell's points as roots.  The forward candidates (labels above the roots in
// the half stencil) are staged 32 at a time in the warp's own shared-memory
// tile, as separate x / y / z arrays, and every lane tests all 32 against its
// root with packed FP32x2 arithmetic (two candidates per instruction, four
// per 128-bit shared load) on the squared separation, without a square root,
// against the outer bounds of the guard band.  Each lane records its hits in
// a 32-bit mask (pairs of two buffer points are masked out); after the tile
// the masks are compacted into a per-warp queue and the hits are binned 32 at
// a time with every lane busy: FP32 with the guard band (bin_pair_f32), FP64
// inside it.  No block barrier is taken.
//
// On grids of cells at least rmax/2 wide (GridParams::sub = 2) the stencil
// is two cells on every axis: 15.6 rmax^3 of candidate volume per root
// against 27 rmax^3 with cells at least rmax wide, for the same 4.2 rmax^3
// of neighbour volume.
//
// One histogram update per pair.  A pair adds to the bin of each end that is
// a root; when both are, the second bin is the mirror of the first (mu bin
// nmu + 1 - m, categories of the two ends exchanged) and takes the same
// product, so the sweep records such pairs once, in a first table, and every
// flush adds the table to the result and, mirrored, once more.  Pairs with
// one buffer end go to a second table, seen from the root, which is added
// once.  (A pair decided in FP64 whose two mu bins do not mirror, a cosine on
// a bin edge to the last bit, is added to the result directly.)  Where both
// tables do not fit, pairs update the second one, twice.
//
// Tables are private to each warp in shared memory when they fit (32-bit
// counts, flushed to the global 64-bit counts before any could overflow, and
// 128-bit fixed-point sums for weighted catalogues), else the result is
// updated with global atomics.  With per-region output (batched regions) each
// region has its own histogram: a warp flushes its tables into the region of
// its cell whenever that region changes.
//
// The FP64 form (precision mode 1) stages the candidates' FP64 positions and
// tests membership with the reference arithmetic; every hit is binned by the
// exact FP64 predicate.  It is also what logarithmic bins take when the FP32
// form's guard would be wide (rmin below a few hundred units of the last place
// of the coordinates).  Logarithmic bins in FP32: 240,000 weighted points, 10
// children per parent, 12 bins, sweep 119 -> 89 us (an FP64 square root and
// log10 per pair before).
//
// Bound by instruction issue (about 80% of the slots, DRAM idle).  The binning
// of a hit took 183 warp instructions per 32 pairs with two updates, two
// divisions, clamps and per-byte flags, three quarters of the kernel; it takes
// 102 now.  Chunks that cross cells fill the lanes (a cell of 40 points gave
// one full chunk and one of 8), and candidates outside the chunk's box, a
// third of the stencil, are not tested.  12M points in 125 regions, 8.0e9
// pairs, 10 mu bins: 84.0 -> 53.7 ms; with one copy each without the binning,
// without the hit queue and without the tests, 24, 14 and 8 ms.
#include "gr_kernels.cuh"

#include <type_traits>

namespace gr {

namespace {

constexpr int kTileWarps = 8;
constexpr int kTileThreads = kTileWarps * 32;
// Resident blocks per SM the register allocation is sized for: 3 (at most 85
// registers, up to 48 bytes spilled); 4 for the adjoint on cells of rmax/2 (64
// registers, 20 bytes spilled), where the two are level: 3M weighted points
// with their gradient, 20.4 ms at 4 and 20.3 ms at 3.  The forward sweep at 4:
// 59.8 -> 66.1 ms on 12M points in 125 regions, 20.4 -> 21.4 on the 3M.
#ifndef GR_TILE_MIN_BLOCKS
#define GR_TILE_MIN_BLOCKS 3
#endif
constexpr int kTileQueue = 32 * 32;  // one tile's hits at most

// Shared memory of one warp: the accepted candidates (structure of arrays;
// two tiles of 32 in turn, one filled while the other is swept), the chunk's
// roots and the hit queue.  F32 false: FP64 positions.  W: weights.
template <bool F32, bool W, bool ADJ>
struct TileWarp {
  typename std::conditional<F32, float, double>::type x[64], y[64], z[64];
  float4 root[32];       // position and code of the chunk's roots
  int q[64], code[64];   // labels and codes of the candidates
  double wq[W ? 64 : 1], wr[W ? 32 : 1];  // weights of candidates and roots
  uint16_t queue[kTileQueue];
  int rb[16], rpre[16];  // candidate ranges of the current chunk: begin, prefix
  // adjoint: signed 64-bit fixed-point gradient partials of the chunk's
  // roots and of the tile's candidates (at most 32 terms each before they
  // are merged into the 128-bit totals after every tile)
  unsigned long long groot[ADJ ? 32 : 1], gcand[ADJ ? 32 : 1];
};

// Weight adjoint arguments (ADJ mode): coefficients (pair_coef_table) and
// the 128-bit gradient totals in label order.
struct TileAdj {
  const double* coef;
  double gscale;
  unsigned long long* g_lo;
  unsigned long long* g_hi;
};
// A warp's minimum and maximum of v over its lanes (v not NaN).
__device__ __forceinline__ int order_bits(float v) {
  const int i = __float_as_int(v);
  return i ^ ((i >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float warp_min(float v) {
  const int i = __reduce_min_sync(0xffffffffu, order_bits(v));
  return __int_as_float(i ^ ((i >> 31) & 0x7fffffff));
}
__device__ __forceinline__ float warp_max(float v) {
  const int i = __reduce_max_sync(0xffffffffu, order_bits(v));
  return __int_as_float(i ^ ((i >> 31) & 0x7fffffff));
}

enum : int { kTileF64 = 0, kTileF32 = 1, kTileF32Log = 2 };
// Tables of a launch (see the head of this file).
enum : int {
  kTabMirror = 0,  // first table only (no buffer points)
  kTabBoth = 1,    // both tables
  kTabRooted = 2   // second table only, one update per root
};

// MODE: kTileF64, or FP32 membership tests and binning with the guard band,
// on linear or logarithmic bins.
// WHIST: tables private to each warp in shared memory, of kind `tab` (else
// the result in global memory, one update per root).
// SUB: 1 (cells >= rmax, 5 ranges) or 2 (cells >= rmax/2, 13 ranges).
// PERREG: one histogram per region (C.cell_region), region r's counts at
// g_cnt + r*nh and fixed-point words at g_fix + 2*r*nh.
// ADJ: the 2PCF weight adjoint instead of histograms: each edge adds
// coef * w_q to dL/dw_p and coef * w_p to dL/dw_q (pair_coef).
template <int MODE, bool WEIGHTED, bool WHIST, int SUB, bool PERREG, bool ADJ>
__global__ void __launch_bounds__(kTileThreads, (ADJ && SUB == 2) ? 4 : GR_TILE_MIN_BLOCKS)
    pair2_tile_kernel(DevCatalog C, PairParams P, unsigned long long* __restrict__ g_cnt,
                      unsigned long long* __restrict__ g_fix, double fscale,
                      unsigned long long* __restrict__ stats, int* __restrict__ work, int tab,
                      int parts, TileAdj A) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr bool F32 = MODE != kTileF64;
  typedef TileWarp<F32, WEIGHTED || ADJ, ADJ> Tile;
  __shared__ __align__(16) Tile s_tw[kTileWarps];
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  Tile& T = s_tw[wib];
  const int nbm = P.nbins * P.nmu;
  const int nh = nbm * 4;
  const bool rooted = !WHIST || tab == kTabRooted;
  // per-warp tables: counts (32-bit), then fixed-point words
  const int nt = tab == kTabBoth ? 2 * nh : nh;
  const size_t wstride = WHIST ? (size_t)nt * (WEIGHTED ? 20 : 4) : 0;
  unsigned int* w_cnt = reinterpret_cast<unsigned int*>(smem + wstride * wib);
  unsigned long long* w_fix =
      reinterpret_cast<unsigned long long*>(smem + wstride * wib + (size_t)nt * 4);
  if (WHIST) {
    for (int k = lane; k < nt; k += 32) {
      w_cnt[k] = 0u;
      if (WEIGHTED) {
        w_fix[k] = 0ull;
        w_fix[nt + k] = 0ull;
      }
    }
  }
  if (ADJ) {
    T.groot[lane] = 0ull;
    T.gcand[lane] = 0ull;
  }
  __syncwarp();
  const int ncell = (int)C.grid.ncell;
  constexpr int NR = SUB == 2 ? 13 : 5;
  unsigned long long rechecks = 0, cands = 0, pairs = 0;
  unsigned int pending = 0;  // edges drained since the last flush (warp-uniform)
  int region = 0;            // region whose histogram the warp holds (PERREG)
  unsigned long long* o_cnt = g_cnt;
  unsigned long long* o_fix = g_fix;

  // A point's code.  Tables: the part of a pair's entry that the point
  // contributes, its sign bit a buffer root (the pair is then seen from the
  // candidate).  One update per root, adjoint: its flags.
  auto flag_code = [&](const float4& c) -> int {
    return (pos4_random(c) ? FLAG_RANDOM : 0) | (pos4_buffer(c) ? FLAG_BUFFER : 0);
  };
  auto root_code = [&](const float4& c) -> int {
    if (ADJ || rooted) return flag_code(c);
    const int r = pos4_random(c) ? 1 : 0;
    return pos4_buffer(c) ? (int)(0x80000000u | (unsigned)(nbm * r + (nt - nh))) : 2 * nbm * r;
  };
  auto cand_code = [&](const float4& c) -> int {
    if (ADJ || rooted) return flag_code(c);
    return (pos4_random(c) ? nbm : 0) + (pos4_buffer(c) ? nt - nh : 0);
  };

  auto flush = [&]() {
    if (!WHIST) return;
    __syncwarp();
    for (int k = lane; k < nt; k += 32) {
      const unsigned v = w_cnt[k];
      unsigned long long vlo = 0, vhi = 0;
      if (WEIGHTED) hist_fix_value(w_fix, nt, k, vlo, vhi);
      if (v == 0u && (vlo | vhi) == 0ull) continue;
      w_cnt[k] = 0u;
      if (WEIGHTED) {
        unsigned* w = reinterpret_cast<unsigned*>(w_fix);
        w[k] = w[nt + k] = w[2 * nt + k] = w[3 * nt + k] = 0u;
      }
      const int e = k < nh ? k : k - nh;
      atomicAdd(&o_cnt[e], (unsigned long long)v);
      if (WEIGHTED) fix_merge(&o_fix[e], &o_fix[nh + e], vlo, vhi);
      if (!rooted) pairs += v;
      if (!rooted && k < nh) {
        // from the other end: mirrored mu bin, categories exchanged
        const int cat = e / nbm, bm = e - cat * nbm;
        const int m = bm / P.nbins, b = bm - m * P.nbins;
        const int e2 = b + P.nbins * (P.nmu - 1 - m) + nbm * ((cat >> 1) | ((cat & 1) << 1));
        atomicAdd(&o_cnt[e2], (unsigned long long)v);
        if (WEIGHTED) fix_merge(&o_fix[e2], &o_fix[nh + e2], vlo, vhi);
      }
    }
    __syncwarp();
  };
  // a pair's entry of one end, added to the warp's second table (WHIST) or to
  // the result
  auto add_rooted = [&](int k, long long v, bool whist) {
    if (whist) {
      atomicAdd(&w_cnt[k], 1u);
      if (WEIGHTED) hist_fix_add<true>(w_fix, nt, k, v);
    } else {
      atomicAdd(&o_cnt[k], 1ull);
      if (WEIGHTED) fix_add_int(&o_fix[k], &o_fix[nh + k], v);
    }
  };

  for (;;) {
    int item = 0;
    if (lane == 0) item = atomicAdd(work, 1);
    item = __shfl_sync(0xffffffffu, item, 0);
    const int cell = parts == 1 ? item : item / parts;
    if (cell >= ncell) break;
    const int part = item - cell * parts;
    const int cb = C.cell_start[cell], ce = C.cell_start[cell + 1];
    if (cb == ce) continue;
    if (PERREG) {
      const int r = C.cell_region[cell];
      if (r != region) {
        flush();
        region = r;
        o_cnt = g_cnt + (size_t)r * nh;
        o_fix = g_fix + (size_t)r * 2 * nh;
      }
    }
    GridParams g;
    const int* cs;
    int lkey;
    cell_grid(C, cell, g, cs, lkey);
    const int cx = lkey % g.nx;
    const int row = lkey - cx;  // first cell of the x-row
    const int row_beg = cs[row], row_end = cs[row + g.nx];
    for (int c0 = row_beg + ((cb - row_beg + 31) & ~31); c0 < ce; c0 += 32) {
      const int cend = min(c0 + 32, row_end);
      // the chunk's candidate ranges, starting just after its first root
      const int cx1 = C.cell_key[cend - 1] - (cell - lkey) - row;
      int rbeg = 0, rend = 0;
      if (lane < NR) forward_slot<SUB>(lane, c0 + 1, cx, cx1, row / g.nx, g, cs, rbeg, rend);
      int len = lane < NR ? rend - rbeg : 0;
      int incl = len;
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      const int total = __shfl_sync(0xffffffffu, incl, NR - 1);
      // this item's share of them, a multiple of 32
      const int share = parts == 1 ? total : ((total + parts - 1) / parts + 31) & ~31;
      int f0 = part * share;
      const int f1 = min(total, f0 + share);
      if (f0 >= f1) continue;
      if (lane < NR) {
        T.rb[lane] = rbeg;
        T.rpre[lane] = incl - len;
      }
      const int p = c0 + lane;
      const bool act = p < cend;
      float4 pi = C.pos4[act ? p : c0];  // idle lanes: the first root again
      double4 pd = make_double4(0.0, 0.0, 0.0, 0.0);
      if (!F32 && act) pd = C.posd[p];
      const bool pbuf = pos4_buffer(pi);
      T.root[lane] = make_float4(pi.x, pi.y, pi.z, __int_as_float(root_code(pi)));
      if (act && (WEIGHTED || ADJ)) T.wr[lane] = C.w[p];
      // the roots' bounding box; candidates farther than rmax from it (with
      // the guard band) and, when every root is a buffer point, buffer
      // candidates are not staged
      const float blx = warp_min(pi.x), bhx = warp_max(pi.x), bly = warp_min(pi.y),
                  bhy = warp_max(pi.y), blz = warp_min(pi.z), bhz = warp_max(pi.z);
      const bool all_buf = __all_sync(0xffffffffu, pbuf);
      const float2 npx = make_float2(-pi.x, -pi.x), npy = make_float2(-pi.y, -pi.y),
                   npz = make_float2(-pi.z, -pi.z);
      const float hi = P.rmax2_hi, lo = P.rmin2_lo;
      // one compare per candidate: |d2 - mid| < half, the sum started at
      // -mid; widened by far more than the roundings (a few 2^-24 of
      // rmax2_hi), it accepts every d2 in (lo, hi); the few pairs just
      // outside the band that it also accepts are rejected by the binning
      const float midv = 0.5f * (hi + lo);
      const float halfv = __int_as_float(__float_as_int(0.5f * (hi - lo) + 1e-6f * fabsf(hi)) + 4);
      const float2 nmid2 = make_float2(-midv, -midv);
      __syncwarp();
      int kr = 0;             // range of this lane's next candidate
      int nacc = 0, done = 0; // candidates staged and swept (warp-uniform)
      for (;;) {
        if (nacc - done < 32 && f0 < f1) {
          // test candidates f0 + lane against the box and stage the rest
          const int f = f0 + lane;
          f0 += 32;
          bool keep = false, qbuf = false;
          int q = 0;
          float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
          if (f < f1) {
            while (kr + 1 < NR && f >= T.rpre[kr + 1]) ++kr;
            q = T.rb[kr] + (f - T.rpre[kr]);
            c = C.pos4[q];
            qbuf = pos4_buffer(c);
            const float ex = fmaxf(fmaxf(blx - c.x, c.x - bhx), 0.f);
            const float ey = fmaxf(fmaxf(bly - c.y, c.y - bhy), 0.f);
            const float ez = fmaxf(fmaxf(blz - c.z, c.z - bhz), 0.f);
            keep = fmaf(ez, ez, fmaf(ey, ey, ex * ex)) <= hi && !(all_buf && qbuf);
          }
          const unsigned kept = __ballot_sync(0xffffffffu, keep);
          const int at = (nacc + __popc(kept & lt)) & 63;
          if (keep) {
            if (F32) {
              T.x[at] = c.x;
              T.y[at] = c.y;
              T.z[at] = c.z;
            } else {
              const double4 cd = C.posd[q];
              T.x[at] = cd.x;
              T.y[at] = cd.y;
              T.z[at] = cd.z;
            }
            T.q[at] = q;
            T.code[at] = cand_code(c);
            if (WEIGHTED || ADJ) T.wq[at] = C.w[q];
          }
          nacc += __popc(kept);
          if (nacc - done < 32 && f0 < f1) continue;
        }
        const int tn = min(32, nacc - done);
        if (tn <= 0) break;
        const int tb = done & 63;  // first slot of the tile
        const bool first = part == 0 && done == 0;
        done += 32;
        if (lane >= tn) T.x[tb + lane] = NAN;  // never a hit
        __syncwarp();
        // buffer points among the tile's candidates
        const int code = T.code[tb + lane];
        const unsigned bufs = __ballot_sync(
            0xffffffffu, lane < tn && ((ADJ || rooted) ? (code & FLAG_BUFFER) != 0 : code >= nh));
        unsigned m = 0u;
        if (act) {
          if constexpr (F32) {
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              const float4 vx = *reinterpret_cast<const float4*>(&T.x[tb + j]);
              const float4 vy = *reinterpret_cast<const float4*>(&T.y[tb + j]);
              const float4 vz = *reinterpret_cast<const float4*>(&T.z[tb + j]);
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const float2 dx = __fadd2_rn(h ? make_float2(vx.z, vx.w) : make_float2(vx.x, vx.y), npx);
                const float2 dy = __fadd2_rn(h ? make_float2(vy.z, vy.w) : make_float2(vy.x, vy.y), npy);
                const float2 dz = __fadd2_rn(h ? make_float2(vz.z, vz.w) : make_float2(vz.x, vz.y), npz);
                const float2 dm = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, nmid2)));
                if (fabsf(dm.x) < halfv) m |= 1u << (j + 2 * h);
                if (fabsf(dm.y) < halfv) m |= 2u << (j + 2 * h);
              }
            }
          } else {
            // the reference's squared separation, separate roundings
#pragma unroll 8
            for (int j = 0; j < 32; ++j) {
              const double dx = __dsub_rn(T.x[tb + j], pd.x);
              const double dy = __dsub_rn(T.y[tb + j], pd.y);
              const double dz = __dsub_rn(T.z[tb + j], pd.z);
              double sd = __dmul_rn(dx, dx);
              sd = __dadd_rn(sd, __dmul_rn(dy, dy));
              sd = __dadd_rn(sd, __dmul_rn(dz, dz));
              if (sd <= P.rmax2 && !(P.rmin > 0.0 && sd <= P.rmin2)) m |= 1u << j;
            }
          }
          // the first candidates are the chunk's own labels c0 + 1, c0 + 2,
          // ..., none of them left out (inside the box, and not all buffer
          // points); those up to this lane's root come before it
          if (first && !all_buf) m &= 0xffffffffu << lane;
          if (pbuf) m &= ~bufs;
          cands += (unsigned long long)tn;
        }
        // compact the hits into the warp's queue, then bin them
        const int cnt = __popc(m);
        int ex = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, ex, o);
          if (lane >= o) ex += v;
        }
        const int tot = __shfl_sync(0xffffffffu, ex, 31);
        int pos = ex - cnt;
        while (m) {
          const int j = __ffs(m) - 1;
          T.queue[pos++] = (uint16_t)((lane << 5) | j);
          m &= m - 1u;
        }
        __syncwarp();
        for (int e0 = 0; e0 < tot; e0 += 32) {
          if (e0 + lane < tot) {
            const int ent = T.queue[e0 + lane];
            const int r = ent >> 5, jt = ent & 31, j = tb + jt;
            const float4 a = T.root[r];
            const int cr = __float_as_int(a.w), cq = T.code[j];
            int st = 2, b0 = 0, m0 = 0;
            if constexpr (F32)
              st = bin_pair_f32<MODE == kTileF32Log>(a, make_float4(T.x[j], T.y[j], T.z[j], 0.f), P, b0, m0);
            bool mirrored = true;
            int mrev = 0;  // mu bin from the candidate when it does not mirror m0
            if (st == 2) {
              if (F32) rechecks++;
              int bin, mf, mr;
              st = edge_f64(C.posd[c0 + r], C.posd[T.q[j]], P, bin, mf, mr) ? 1 : 0;
              if (st == 1) {
                b0 = bin - 1;
                m0 = mf - 1;
                mrev = mr - 1;
                mirrored = mrev == P.nmu - 1 - m0;
              }
            }
            if (st == 1 && ADJ) {
              const int rr = cr & cq & FLAG_RANDOM;
              const bool bp = cr & FLAG_BUFFER, bq = cq & FLAG_BUFFER;
              if (mirrored) mrev = P.nmu - 1 - m0;
              double cf;
              if (mirrored || bp || bq) {
                cf = A.coef[b0 + P.nbins * (bp ? mrev : m0) + nbm * (2 * (bp || bq) + rr)];
              } else {
                cf = A.coef[b0 + P.nbins * m0 + nbm * (2 + rr)] +
                     A.coef[b0 + P.nbins * mrev + nbm * (2 + rr)];
              }
              pairs++;
              if (cf != 0.0) {
                smem_add_s64(&T.groot[r], __double2ll_rn(cf * T.wq[j] * A.gscale));
                smem_add_s64(&T.gcand[jt], __double2ll_rn(cf * T.wr[r] * A.gscale));
              }
            } else if (st == 1) {
              const long long v = WEIGHTED ? __double2ll_rn(T.wr[r] * T.wq[j] * fscale) : 0ll;
              if (!rooted && mirrored) {
                const int bp = (int)((unsigned)cr >> 31);
                const int k = b0 + P.nbins * (bp ? P.nmu - 1 - m0 : m0) + (cr & 0x7fffffff) + (cq << bp);
                atomicAdd(&w_cnt[k], 1u);
                if (WEIGHTED) hist_fix_add<true>(w_fix, nt, k, v);
              } else {
                const uint8_t fp = C.flags[c0 + r], fq = C.flags[T.q[j]];
                const int rp = fp & FLAG_RANDOM, rq = fq & FLAG_RANDOM;
                if (mirrored) mrev = P.nmu - 1 - m0;
                if (!(fp & FLAG_BUFFER))
                  add_rooted(b0 + P.nbins * m0 + nbm * (2 * rp + rq), v, WHIST && rooted);
                if (!(fq & FLAG_BUFFER))
                  add_rooted(b0 + P.nbins * mrev + nbm * (2 * rq + rp), v, WHIST && rooted);
                pairs++;
              }
            }
          }
        }
        if (ADJ) {
          // merge the tile's gradient partials into the 128-bit totals
          __syncwarp();
          const long long vc = (long long)T.gcand[lane];
          const int ql = T.q[tb + lane];
          if (vc != 0) fix_add_int(&A.g_lo[ql], &A.g_hi[ql], vc);
          T.gcand[lane] = 0ull;
          const long long vr = (long long)T.groot[lane];
          if (vr != 0) fix_add_int(&A.g_lo[c0 + lane], &A.g_hi[c0 + lane], vr);
          T.groot[lane] = 0ull;
        }
        // a 32-bit count grows by at most 2 per binned pair
        pending += (unsigned)tot;
        if (pending > (1u << 30)) {
          flush();
          pending = 0u;
        }
        __syncwarp();
      }
    }
  }
  flush();
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    rechecks += __shfl_xor_sync(0xffffffffu, rechecks, o);
    pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
    cands += __shfl_xor_sync(0xffffffffu, cands, o);
  }
  if (lane == 0) {
    if (rechecks) atomicAdd(&stats[0], rechecks);
    if (cands) atomicAdd(&stats[1], cands);
    if (pairs) atomicAdd(&stats[2], pairs);
  }
}

}  // namespace

// Work items per cell: the candidates of each chunk are shared out over
// `parts` warps, up to 8, each with its own setup of the chunk.  Two reasons.
// Chunks too few for the resident warps (3,500 points at 10 per cell: 21 us
// with 8 parts, 31 us with one); and chunks so costly, with hundreds of
// candidates for every part, that the last ones leave warps idle at the end
// (300,000 points at 24 per rmax/2 cell: 3.5 ms forward and backward with 8,
// 4.1 ms with one).  Otherwise the setup only costs: 70,000 points at 9 per
// cell, 52 us with one part and 59 us with 4; 350,000 in mocks of 7,000, 153
// us with one and 235 us with 4.
static int tile_parts(const DevCatalog& C, int64_t blocks) {
  const int64_t warps = blocks * kTileWarps;
  const double per_cell = (double)C.n / (double)std::max<int64_t>(1, C.grid.ncell);
  const int64_t chunks = (int64_t)C.n / 32 + 1;
  // candidates of a chunk: the half stencil's cells, about twice as many for
  // a chunk that spans several sparse cells
  const double cands = per_cell * (C.grid.sub == 2 ? 63.0 : 14.0) * (per_cell < 16.0 ? 2.5 : 1.2);
  int64_t parts = 1;
  if (2 * chunks < warps) parts = warps / chunks;
  if (chunks < 16 * warps) parts = std::max(parts, (int64_t)(cands / 256.0));
  return (int)std::min<int64_t>(8, std::max<int64_t>(1, parts));
}

void launch_pair2_tile(const DevCatalog& C, const PairParams& P, bool weighted,
                       unsigned long long* g_cnt, unsigned long long* g_fix, double fscale,
                       unsigned long long* stats, int* work, cudaStream_t s, bool per_region) {
  if (C.n <= 0) return;
  if (per_region && !C.cell_region) throw Error{-1, "per-region output needs a region layout"};
  // one table's bytes over the warps of a block; both tables when the
  // catalogue has buffer points and they fit
  size_t smem = (size_t)P.nbins * P.nmu * 4 * (weighted ? 20 : 4) * kTileWarps;
  const bool whist = smem <= kMaxTileHistSmem;
  int tab = C.has_buffer ? (2 * smem <= kMaxTileHistSmem ? kTabBoth : kTabRooted) : kTabMirror;
  if (!whist) tab = kTabRooted;
  smem = whist ? (tab == kTabBoth ? 2 * smem : smem) : 0;
  GR_CUDA_TRY(cudaMemsetAsync(work, 0, sizeof(int), s));
  const int sub = C.grid.sub == 2 ? 2 : 1;
#define GR_TILE_LAUNCH(F, W, H, S)                                                           \
  do {                                                                                        \
    auto k = per_region ? pair2_tile_kernel<F, W, H, S, true, false>                         \
                        : pair2_tile_kernel<F, W, H, S, false, false>;                        \
    GR_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,         \
                                     (int)smem));                                             \
    int per_sm = 1;                                                                           \
    GR_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kTileThreads, smem)); \
    int64_t blocks = (int64_t)std::max(1, per_sm) * sm_count();                               \
    const int parts = tile_parts(C, blocks);                                                  \
    const int64_t need = (C.grid.ncell * parts + kTileWarps - 1) / kTileWarps;                \
    if (blocks > need) blocks = std::max<int64_t>(1, need);                                   \
    k<<<(unsigned)blocks, kTileThreads, smem, s>>>(C, P, g_cnt, g_fix, fscale, stats, work,   \
                                                   tab, parts, TileAdj{});                    \
  } while (0)
#define GR_TILE_S(F, W, H)                                                                   \
  do {                                                                                        \
    if (sub == 2) GR_TILE_LAUNCH(F, W, H, 2); else GR_TILE_LAUNCH(F, W, H, 1);                \
  } while (0)
#define GR_TILE_H(F, W)                                                                      \
  do {                                                                                        \
    if (whist) GR_TILE_S(F, W, true); else GR_TILE_S(F, W, false);                            \
  } while (0)
  if (P.f32) {
    if (weighted) GR_TILE_H(kTileF32, true); else GR_TILE_H(kTileF32, false);
  } else if (P.logbins == 2) {
    if (weighted) GR_TILE_H(kTileF32Log, true); else GR_TILE_H(kTileF32Log, false);
  } else {
    if (weighted) GR_TILE_H(kTileF64, true); else GR_TILE_H(kTileF64, false);
  }
#undef GR_TILE_H
#undef GR_TILE_S
#undef GR_TILE_LAUNCH
  GR_CHECK_LAUNCH();
}

void pair_coef_table(const double* cot2, const double* cot3, int nbins, int nmu, double* coef) {
  const int nbm = nbins * nmu;
  for (int m = 0; m < nmu; ++m)
    for (int b = 0; b < nbins; ++b) {
      const int k = b + nbins * m, k2 = b + nbins * (nmu - 1 - m);
      coef[k] = cot2[k] + cot2[k2];
      coef[nbm + k] = (cot2[k] + cot3[k]) + (cot2[k2] + cot3[k2]);
      coef[2 * nbm + k] = cot2[k];
      coef[3 * nbm + k] = cot2[k] + cot3[k];
    }
}

void launch_adj2_tile(const DevCatalog& C, const PairParams& P, const double* coef,
                      double gscale, unsigned long long* g_lo,
                      unsigned long long* g_hi, unsigned long long* stats, int* work,
                      cudaStream_t s) {
  if (C.n <= 0) return;
  GR_CUDA_TRY(cudaMemsetAsync(work, 0, sizeof(int), s));
  const TileAdj A{coef, gscale, g_lo, g_hi};
  const int sub = C.grid.sub == 2 ? 2 : 1;
#define GR_ADJT_LAUNCH(F, S)                                                                  \
  do {                                                                                        \
    auto k = pair2_tile_kernel<F, true, false, S, false, true>;                               \
    int per_sm = 1;                                                                           \
    GR_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kTileThreads, 0));  \
    int64_t blocks = (int64_t)std::max(1, per_sm) * sm_count();                               \
    const int parts = tile_parts(C, blocks);                                                  \
    const int64_t need = (C.grid.ncell * parts + kTileWarps - 1) / kTileWarps;                \
    if (blocks > need) blocks = std::max<int64_t>(1, need);                                   \
    k<<<(unsigned)blocks, kTileThreads, 0, s>>>(C, P, nullptr, nullptr, 1.0, stats, work,     \
                                                0, parts, A);                                 \
  } while (0)
  if (P.f32) {
    if (sub == 2) GR_ADJT_LAUNCH(kTileF32, 2); else GR_ADJT_LAUNCH(kTileF32, 1);
  } else if (P.logbins == 2) {
    if (sub == 2) GR_ADJT_LAUNCH(kTileF32Log, 2); else GR_ADJT_LAUNCH(kTileF32Log, 1);
  } else {
    if (sub == 2) GR_ADJT_LAUNCH(kTileF64, 2); else GR_ADJT_LAUNCH(kTileF64, 1);
  }
#undef GR_ADJT_LAUNCH
  GR_CHECK_LAUNCH();
}

}  // namespace gr

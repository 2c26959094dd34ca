// Sorted-cell index on the device: replaces the kd-tree of the reference
// (src/kdtree2.F90:611-1012) as the structure behind the fixed-radius
// queries.  Points are bucketed into a uniform grid whose cells are at least
// rmax wide, counting-sorted by cell key, and re-laid out in cell order as
// float4 (FP32 fast path) and double4 (FP64 guard band, weight) arrays.
#include "gr_index.cuh"

#include <atomic>
#include <cstring>

namespace gr {

namespace {

// Order-preserving map of doubles onto unsigned 64-bit ints, so that min/max
// reductions can use integer atomics.
__device__ __forceinline__ unsigned long long dbl_key(double v) {
  unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}

constexpr int kScanBlock = 384;  // a multiple of 3 and of the warp
constexpr int kScanUnroll = 4;   // loads in flight per thread

__device__ __forceinline__ unsigned long long shfl_down_u64(unsigned long long v, int o) {
  return __shfl_down_sync(0xffffffffu, v, o);
}

// One pass over a new catalogue: its bounding box, the largest weights,
// whether all weights of a class are equal, whether anything is not finite;
// with COPY the arrays also move to the context's own.  Coordinates are read
// as one flat array: the block size is a multiple of 3, so a thread always
// meets the same axis.  Every block leaves its partial result in part[word *
// gridDim.x + block]; the last block to arrive combines them and writes the
// result to pinned host memory, so no buffer is initialised and nothing is
// copied back.  Bound by the launch and the last block's wait at 4,000
// points, by DRAM above a few million.  In place of three copies, the upload
// of initial values, a weight pass and three read-backs here, and of three box
// passes and a host wait or a speculated grid in the count that follows.  With
// results_kernel in place of its read-backs, setting 3,500 points and counting
// them took 128 us before and 88 us after, 70,000 points 175 and 125 us.
template <bool COPY>
__global__ void __launch_bounds__(kScanBlock)
catalog_scan_kernel(const double* __restrict__ xyz, const double* __restrict__ w,
                    const int* __restrict__ buffer, int64_t n_data, int64_t n,
                    double* __restrict__ xyz_out, double* __restrict__ w_out,
                    int* __restrict__ buffer_out, unsigned long long* __restrict__ part,
                    unsigned int* __restrict__ arrived, CatalogScan* __restrict__ out) {
  constexpr int kWarps = kScanBlock / 32;
  __shared__ unsigned long long s_mn[kWarps][3], s_mx[kWarps][3], s_w[kWarps][2];
  __shared__ unsigned int s_flags, s_last;
  if (threadIdx.x == 0) s_flags = 0u;
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t tid = blockIdx.x * (int64_t)kScanBlock + threadIdx.x;
  const int64_t step = (int64_t)gridDim.x * kScanBlock;
  unsigned long long mn = ~0ull, mx = 0ull, mg = 0ull, mr = 0ull;
  unsigned int flags = 0u;
  for (int64_t i0 = tid; i0 < 3 * n; i0 += kScanUnroll * step) {
    double v[kScanUnroll];
#pragma unroll
    for (int u = 0; u < kScanUnroll; ++u) {
      const int64_t i = i0 + u * step;
      v[u] = xyz[i < 3 * n ? i : i0];
    }
#pragma unroll
    for (int u = 0; u < kScanUnroll; ++u) {
      const int64_t i = i0 + u * step;
      const unsigned long long k = dbl_key(v[u]);
      mn = k < mn ? k : mn;
      mx = k > mx ? k : mx;
      if (!isfinite(v[u])) flags |= kScanCoordBad;
      if (COPY && i < 3 * n) xyz_out[i] = v[u];
    }
  }
  const double refg = n_data > 0 ? w[0] : 0.0;
  const double refr = n > n_data ? w[n_data] : 0.0;
  for (int64_t i0 = tid; i0 < n; i0 += kScanUnroll * step) {
    double v[kScanUnroll];
#pragma unroll
    for (int u = 0; u < kScanUnroll; ++u) {
      const int64_t i = i0 + u * step;
      v[u] = w[i < n ? i : i0];
    }
#pragma unroll
    for (int u = 0; u < kScanUnroll; ++u) {
      const int64_t i = i0 + u * step;
      if (i >= n) break;
      if (!isfinite(v[u])) flags |= kScanWeightBad;
      if (__double_as_longlong(v[u]) != __double_as_longlong(i < n_data ? refg : refr))
        flags |= kScanWeightsDiffer;
      const unsigned long long a = (unsigned long long)__double_as_longlong(fabs(v[u]));
      if (i < n_data) mg = a > mg ? a : mg;
      else mr = a > mr ? a : mr;
      if (COPY) w_out[i] = v[u];
    }
  }
  if (COPY && buffer)
    for (int64_t i = tid; i < n; i += step) buffer_out[i] = buffer[i];

  // lanes l, l + 3, l + 6, ... share an axis: after these steps lanes 0..2
  // hold the warp's results (a lane past the end returns the reader's value)
#pragma unroll
  for (int o = 24; o >= 3; o >>= 1) {
    const unsigned long long a = shfl_down_u64(mn, o), b = shfl_down_u64(mx, o);
    mn = a < mn ? a : mn;
    mx = b > mx ? b : mx;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long a = shfl_down_u64(mg, o), b = shfl_down_u64(mr, o);
    mg = a > mg ? a : mg;
    mr = b > mr ? b : mr;
  }
  if (lane < 3) {
    const int axis = (2 * wid + lane) % 3;  // (32 wid + lane) mod 3
    s_mn[wid][axis] = mn;
    s_mx[wid][axis] = mx;
  }
  if (lane == 0) {
    s_w[wid][0] = mg;
    s_w[wid][1] = mr;
  }
  if (flags) atomicOr(&s_flags, flags);
  __syncthreads();
  if (threadIdx.x < kCatalogScanWords) {
    const int t = threadIdx.x;
    unsigned long long v = t == 8 ? s_flags : (t < 3 ? ~0ull : 0ull);
    if (t < 8)
      for (int k = 0; k < kWarps; ++k) {
        const unsigned long long u = t < 3 ? s_mn[k][t] : (t < 6 ? s_mx[k][t - 3] : s_w[k][t - 6]);
        v = t < 3 ? (u < v ? u : v) : (u > v ? u : v);
      }
    part[(int64_t)t * gridDim.x + blockIdx.x] = v;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(arrived, 1u) == gridDim.x - 1 ? 1u : 0u;
  __syncthreads();
  if (!s_last) return;
  // the last block: warp k combines word k
  __threadfence();
  if (wid < kCatalogScanWords) {
    unsigned long long v = wid < 3 ? ~0ull : 0ull;
    for (int b = lane; b < (int)gridDim.x; b += 32) {
      const unsigned long long u = __ldcg(&part[(int64_t)wid * gridDim.x + b]);
      v = wid < 3 ? (u < v ? u : v) : (wid == 8 ? (u | v) : (u > v ? u : v));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long u = __shfl_xor_sync(0xffffffffu, v, o);
      v = wid < 3 ? (u < v ? u : v) : (wid == 8 ? (u | v) : (u > v ? u : v));
    }
    if (lane == 0) out->word[wid] = v;
  }
  if (threadIdx.x == 0) {
    out->w0[0] = refg;
    out->w0[1] = refr;
    *arrived = 0u;  // for the next launch
  }
}

__device__ __forceinline__ int cell_coord(double v, double lo, double inv_cs, int nc) {
  int c = (int)floor((v - lo) * inv_cs);
  return c < 0 ? 0 : (c >= nc ? nc - 1 : c);
}

__global__ void cell_assign_kernel(const double* __restrict__ xyz, int64_t n, GridGeom g,
                                   int* __restrict__ key, int* __restrict__ slot,
                                   int* __restrict__ count) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int cx = cell_coord(xyz[3 * i + 0], g.lo[0], g.inv_cs[0], g.nc[0]);
    int cy = cell_coord(xyz[3 * i + 1], g.lo[1], g.inv_cs[1], g.nc[1]);
    int cz = cell_coord(xyz[3 * i + 2], g.lo[2], g.inv_cs[2], g.nc[2]);
    int k = (cz * g.nc[1] + cy) * g.nc[0] + cx;
    key[i] = k;
    slot[i] = atomicAdd(&count[k], 1);
  }
}

// Place every point at start[key] + (rank of its original index among the
// points of its cell).  The rank makes the layout deterministic: within a
// cell, points keep their catalogue order.
__global__ void cell_scatter_kernel(int64_t n, const int* __restrict__ key,
                                    const int* __restrict__ slot, const int64_t* __restrict__ start,
                                    int* __restrict__ tmp_perm) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    tmp_perm[start[key[i]] + slot[i]] = (int)i;
}

// Point i of the catalogue, in cell c, at place p of the layout.
__device__ __forceinline__ void put_point(int64_t p, int i, int c, const double* __restrict__ xyz,
                                          const double* __restrict__ w,
                                          const int* __restrict__ buffer, int64_t n_data,
                                          float4* __restrict__ pos4, double4* __restrict__ posd,
                                          double* __restrict__ wl, int* __restrict__ orig,
                                          uint8_t* __restrict__ flags, int* __restrict__ cell_key) {
  const double x = xyz[3 * (int64_t)i + 0], y = xyz[3 * (int64_t)i + 1],
               z = xyz[3 * (int64_t)i + 2];
  const double wi = w[i];
  uint8_t f = (i >= n_data) ? FLAG_RANDOM : 0;
  if (buffer && buffer[i] == 1) f |= FLAG_BUFFER;
  pos4[p] = make_float4(__double2float_rn(x), __double2float_rn(y), __double2float_rn(z),
                        pos4_flags(f));
  posd[p] = make_double4(x, y, z, wi);
  wl[p] = wi;
  orig[p] = i;
  flags[p] = f;
  cell_key[p] = c;
}

// Buffers from cudaMalloc start 256-byte aligned; each is zeroed with 16-byte
// stores for its body and 4-byte stores for a tail (sizes are multiples of 4).
__device__ __forceinline__ void zero_list(const ZeroList& z, size_t tid, size_t nthr) {
  for (int k = 0; k < z.n; ++k) {
    const size_t nv = z.bytes[k] / 16;
    uint4* v = reinterpret_cast<uint4*>(z.p[k]);
    for (size_t i = tid; i < nv; i += nthr) v[i] = make_uint4(0u, 0u, 0u, 0u);
    const size_t tail = (z.bytes[k] - nv * 16) / 4;
    uint32_t* t = reinterpret_cast<uint32_t*>(reinterpret_cast<unsigned char*>(z.p[k]) + nv * 16);
    if (tid < tail) t[tid] = 0u;
  }
}

// One warp per cell: rank each member by its catalogue index (O(c^2/32)),
// so that within a cell points keep their catalogue order, and write the
// member's data at its place in the cell-ordered layout (the scattered
// reads of the catalogue happen here, once per point).
__global__ void cell_order_gather_kernel(int64_t ncell, const int64_t* __restrict__ start,
                                         const int* __restrict__ tmp_perm,
                                         const double* __restrict__ xyz,
                                         const double* __restrict__ w,
                                         const int* __restrict__ buffer, int64_t n_data,
                                         float4* __restrict__ pos4, double4* __restrict__ posd,
                                         double* __restrict__ wl, int* __restrict__ orig,
                                         uint8_t* __restrict__ flags, int* __restrict__ cell_key) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t c = warp; c < ncell; c += nwarps) {
    const int64_t b = start[c], e = start[c + 1];
    const int cnt = (int)(e - b);
    for (int k = lane; k < cnt; k += 32) {
      const int i = tmp_perm[b + k];
      int r = 0;
      for (int j = 0; j < cnt; ++j) r += tmp_perm[b + j] < i;
      const int64_t p = b + r;
      put_point(p, i, (int)c, xyz, w, buffer, n_data, pos4, posd, wl, orig, flags, cell_key);
    }
  }
}

inline double key_to_dbl(unsigned long long k) {
  unsigned long long b = (k & 0x8000000000000000ull) ? (k & 0x7fffffffffffffffull) : ~k;
  double v;
  std::memcpy(&v, &b, 8);
  return v;
}

// blocks for n items, at most `waves` blocks per SM
int blocks_for(int64_t n, int threads, int waves = 16) {
  const int64_t cap = (int64_t)waves * sm_count();
  int64_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > cap) b = cap;
  return (int)b;
}

}  // namespace

namespace {

// Grids of catalogues up to this size are built by one launch whose blocks
// each sort the whole catalogue in shared memory and write their share of the
// layout; above it the passes over all SMs are faster.
constexpr int64_t kSmallIndex = 16384;
constexpr size_t kSmallIndexSmem = 200 << 10;
constexpr int kSmallThreads = 1024;
constexpr int kSmallShare = 256;  // points whose layout one block writes

size_t small_index_smem(int64_t n, int64_t ncell) {
  return sizeof(int) * (size_t)(ncell + 1) + (sizeof(int) + sizeof(uint16_t)) * (size_t)n;
}

// Counting sort of the whole catalogue by cell in every block, then the
// block's share of the layout: same order as the kernels above (cells, then
// catalogue order within a cell).  Launch latency is what bounds such a
// catalogue: the separate passes (clear, keys, scan, scatter, order) take
// 3.5 us each whatever they do.  Index phase 22 -> 10 us at 1,000 points,
// 22 -> 12 at 3,500, 27 -> 17 at 14,000; the work repeated in every block and
// the 16-bit places bound the rule at 16,384.
__global__ void __launch_bounds__(kSmallThreads)
index_small_kernel(const double* __restrict__ xyz, const double* __restrict__ w,
                   const int* __restrict__ buffer, int n, int n_data, GridGeom g, int ncell,
                   ZeroList z, float4* __restrict__ pos4, double4* __restrict__ posd,
                   double* __restrict__ wl, int* __restrict__ orig, uint8_t* __restrict__ flags,
                   int* __restrict__ cell_key, int* __restrict__ cell_start) {
  extern __shared__ int s_count[];                             // ncell + 1
  int* s_key = s_count + ncell + 1;                            // n
  uint16_t* s_perm = reinterpret_cast<uint16_t*>(s_key + n);   // n
  __shared__ int s_warp[32];
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  zero_list(z, blockIdx.x * (size_t)kSmallThreads + t, (size_t)gridDim.x * kSmallThreads);
  for (int k = t; k <= ncell; k += kSmallThreads) s_count[k] = 0;
  __syncthreads();
#pragma unroll 4
  for (int i = t; i < n; i += kSmallThreads) {
    const int cx = cell_coord(xyz[3 * i + 0], g.lo[0], g.inv_cs[0], g.nc[0]);
    const int cy = cell_coord(xyz[3 * i + 1], g.lo[1], g.inv_cs[1], g.nc[1]);
    const int cz = cell_coord(xyz[3 * i + 2], g.lo[2], g.inv_cs[2], g.nc[2]);
    const int k = (cz * g.nc[1] + cy) * g.nc[0] + cx;
    s_key[i] = k;
    atomicAdd(&s_count[k], 1);
  }
  __syncthreads();
  // exclusive scan; an odd number of cells per thread keeps the banks apart
  const int per = ((ncell + kSmallThreads) / kSmallThreads) | 1;
  const int k0 = min(t * per, ncell), k1 = min(k0 + per, ncell);
  int sum = 0;
  for (int k = k0; k < k1; ++k) sum += s_count[k];
  int x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[wid] = x;
  __syncthreads();
  if (wid == 0) {
    int y = s_warp[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, y, o);
      if (lane >= o) y += v;
    }
    s_warp[lane] = y;
  }
  __syncthreads();
  int ex = x - sum + (wid > 0 ? s_warp[wid - 1] : 0);
  for (int k = k0; k < k1; ++k) {
    const int c = s_count[k];
    s_count[k] = ex;
    ex += c;
  }
  __syncthreads();
  for (int k = blockIdx.x * kSmallThreads + t; k <= ncell; k += gridDim.x * kSmallThreads)
    cell_start[k] = k < ncell ? s_count[k] : n;
  __syncthreads();
  // cursors: s_count[k] ends as the end of cell k
  for (int i = t; i < n; i += kSmallThreads)
    s_perm[atomicAdd(&s_count[s_key[i]], 1)] = (uint16_t)i;
  __syncthreads();
  // the share is one of catalogue points, not of places: the order that the
  // cursors left within a cell differs from block to block
  const int i = blockIdx.x * kSmallShare + t;
  if (t < kSmallShare && i < n) {
    const int k = s_key[i];
    const int b = k > 0 ? s_count[k - 1] : 0, e = s_count[k];
    int r = 0;
    for (int j = b; j < e; ++j) r += s_perm[j] < i;
    put_point(b + r, i, k, xyz, w, buffer, n_data, pos4, posd, wl, orig, flags, cell_key);
  }
}

// The box of a scan as doubles.
CatalogBox box_of_scan(const CatalogScan& h, int64_t n) {
  CatalogBox b{};
  if (n <= 0) return b;
  for (int d = 0; d < 3; ++d) {
    b.lo[d] = key_to_dbl(h.word[d]);
    b.hi[d] = key_to_dbl(h.word[3 + d]);
    b.coord_max = std::max(b.coord_max, std::max(std::fabs(b.lo[d]), std::fabs(b.hi[d])));
  }
  b.finite = (h.word[8] & kScanCoordBad) == 0;
  return b;
}

}  // namespace

void scan_catalog(const double* xyz, const double* w, const int* buffer, int64_t n_data, int64_t n,
                  double* xyz_out, double* w_out, int* buffer_out, DevBuf<unsigned long long>& part,
                  CatalogScan* out, CatalogBox& box, cudaStream_t s) {
  const int64_t per = (int64_t)kScanBlock * kScanUnroll;
  const int64_t cap = 4 * (int64_t)sm_count();
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(cap, (3 * n + per - 1) / per));
  const size_t words = (size_t)kCatalogScanWords * cap;
  // the arrival counter sits behind the partial results
  if (part.n < words + 1) {
    part.reserve(words + 1);
    GR_CUDA_TRY(cudaMemsetAsync(part.p, 0, sizeof(unsigned long long) * (words + 1), s));
  }
  unsigned int* arrived = reinterpret_cast<unsigned int*>(part.p + words);
  if (n > 0) {
    if (xyz != xyz_out)
      catalog_scan_kernel<true><<<blocks, kScanBlock, 0, s>>>(xyz, w, buffer, n_data, n, xyz_out, w_out,
                                                              buffer_out, part.p, arrived, out);
    else
      catalog_scan_kernel<false><<<blocks, kScanBlock, 0, s>>>(xyz, w, buffer, n_data, n, nullptr, nullptr,
                                                               nullptr, part.p, arrived, out);
    GR_CHECK_LAUNCH();
  }
  GR_CUDA_TRY(cudaStreamSynchronize(s));
  box = box_of_scan(*out, n);
}

void CellIndex::build(const double* d_xyz, const double* d_w, const int* d_buffer, int64_t n_pts,
                      int64_t n_data_pts, const CatalogBox& cat_box, double rmax, cudaStream_t s,
                      ZeroList z, int sub, double dense_per_cell) {
  if (!cat_box.finite) throw Error{-1, "catalogue has non-finite coordinates"};
  const bool auto_sub = sub == 0;
  if (sub != 2) sub = 1;
  n = n_pts;
  n_data = n_data_pts;
  has_buffer = d_buffer ? 1 : 0;
  launches = 0;
  box = cat_box;
  coord_max = box.coord_max;
  // cells at least rmax (sub 2: rmax/2) wide; the cell table stays O(N)
  GridGeom g;
  {
    const int64_t cells1 = make_grid_geom(box.lo, box.hi, rmax, 2048, std::max<int64_t>(4 * n, 4096), g);
    per_cell_rmax = cells1 > 0 ? (double)n / (double)cells1 : 0.0;
    if (auto_sub) sub = (dense_per_cell > 0.0 && per_cell_rmax >= dense_per_cell) ? 2 : 1;
  }
  const int64_t total =
      make_grid_geom(box.lo, box.hi, rmax / sub, 2048, std::max<int64_t>(4 * n, 4096), g);
  grid.nx = g.nc[0];
  grid.ny = g.nc[1];
  grid.nz = g.nc[2];
  grid.ncell = total;
  grid.sub = sub;

  cell_start.reserve(total + 1);
  pos4.reserve(n);
  posd.reserve(n);
  w.reserve(n);
  orig.reserve(n);
  flags.reserve(n);
  cell_key.reserve(n);

  if (n > 0 && n <= kSmallIndex && small_index_smem(n, total) <= kSmallIndexSmem) {
    const size_t smem = small_index_smem(n, total);
    GR_CUDA_TRY(cudaFuncSetAttribute(index_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kSmallIndexSmem));
    index_small_kernel<<<(unsigned)((n + kSmallShare - 1) / kSmallShare), kSmallThreads, smem, s>>>(
        d_xyz, d_w, d_buffer, (int)n, (int)n_data, g, (int)total, z, pos4.p, posd.p, w.p, orig.p,
        flags.p, cell_key.p, cell_start.p);
    launches = 1;
    GR_CHECK_LAUNCH();
    return;
  }
  cell_count.reserve(total + 1);
  key_orig.reserve(n);
  slot.reserve(n);
  tmp_perm.reserve(n);
  cell_start64.reserve(total + 1);
  z.add(cell_count.p, sizeof(int) * (total + 1));
  zero_async(z, s);
  launches++;
  if (n > 0) {
    cell_assign_kernel<<<blocks_for(n, 256), 256, 0, s>>>(d_xyz, n, g, key_orig.p, slot.p,
                                                         cell_count.p);
    launches++;
  }
  GR_CHECK_LAUNCH();
  // cell starts as 64-bit offsets and, in the same pass, the 32-bit copy
  // the kernels read
  scan_i32_to_i64(cell_count.p, cell_start64.p, total, s, scan_tmp, cell_start.p);
  launches += 2;
  if (n > 0) {
    cell_scatter_kernel<<<blocks_for(n, 256), 256, 0, s>>>(n, key_orig.p, slot.p, cell_start64.p,
                                                          tmp_perm.p);
    cell_order_gather_kernel<<<blocks_for(total * 32, 256), 256, 0, s>>>(
        total, cell_start64.p, tmp_perm.p, d_xyz, d_w, d_buffer, n_data, pos4.p, posd.p, w.p,
        orig.p, flags.p, cell_key.p);
    launches += 2;
  }
  GR_CHECK_LAUNCH();
}

int sm_count() {
  constexpr int kDev = 64;
  static std::atomic<int> cache[kDev];
  int dev = 0;
  GR_CUDA_TRY(cudaGetDevice(&dev));
  if (dev >= 0 && dev < kDev) {
    const int v = cache[dev].load(std::memory_order_relaxed);
    if (v > 0) return v;
  }
  int v = 0;
  GR_CUDA_TRY(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev));
  if (v < 1) v = 1;
  if (dev >= 0 && dev < kDev) cache[dev].store(v, std::memory_order_relaxed);
  return v;
}

int64_t make_grid_geom(const double lo[3], const double hi[3], double rmax, int max_per_axis,
                       int64_t max_cells, GridGeom& g) {
  double cell_min = rmax * 1.000001;
  if (!(cell_min > 0)) cell_min = 1e300;
  int64_t total = 1;
  for (int d = 0; d < 3; ++d) {
    const double span = hi[d] - lo[d];
    double k = std::floor(span / cell_min);
    if (!(k >= 1)) k = 1;
    if (k > max_per_axis) k = max_per_axis;
    g.nc[d] = (int)k;
    g.lo[d] = lo[d];
    g.inv_cs[d] = 1.0 / (span > 0 ? span / k : 1.0);
    total *= (int64_t)k;
  }
  while (total > max_cells && total > 1) {
    int d = 0;
    for (int k = 1; k < 3; ++k)
      if (g.nc[k] > g.nc[d]) d = k;
    g.nc[d] = std::max(1, g.nc[d] / 2);
    const double span = hi[d] - lo[d];
    g.inv_cs[d] = 1.0 / (span > 0 ? span / g.nc[d] : 1.0);
    total = (int64_t)g.nc[0] * g.nc[1] * g.nc[2];
  }
  return total;
}

DevCatalog CellIndex::view() const {
  DevCatalog c;
  c.pos4 = pos4.p;
  c.posd = posd.p;
  c.w = w.p;
  c.orig = orig.p;
  c.flags = flags.p;
  c.cell_key = cell_key.p;
  c.cell_start = cell_start.p;
  c.n = (int)n;
  c.n_data = (int)n_data;
  c.has_buffer = has_buffer;
  c.grid = grid;
  c.cell_region = nullptr;
  c.region_grid = nullptr;
  c.region_cell_off = nullptr;
  return c;
}

// ------------------------------------------------------------------- scan --
namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;
// Up to this many tiles a block of the second pass adds the sums of the tiles
// before its own itself (8 KB at most); beyond it they are scanned first.
// The launch spared and the smaller tiles (1,024 against 4,096 items): 17,600
// cells 14.9 -> 7.5 us.
constexpr int64_t kScanFlat = 1024;

template <typename T>
__device__ __forceinline__ int64_t block_exclusive_scan(int64_t v, int64_t* warp_tot, int64_t& total) {
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int64_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int64_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_tot[wid] = x;
  __syncthreads();
  if (wid == 0) {
    int nw = blockDim.x >> 5;
    int64_t t = lane < nw ? warp_tot[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int64_t y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    if (lane < nw) warp_tot[lane] = t;
  }
  __syncthreads();
  int64_t before = wid > 0 ? warp_tot[wid - 1] : 0;
  total = warp_tot[(blockDim.x >> 5) - 1];
  return before + x - v;
}

template <typename T>
__global__ void scan_tile_sums(const T* __restrict__ in, int64_t n, int64_t* __restrict__ sums) {
  __shared__ int64_t warp_tot[32];
  int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int64_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k)
    if (base + k < n) s += (int64_t)in[base + k];
  int64_t total;
  block_exclusive_scan<T>(s, warp_tot, total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

template <typename T>
__global__ void scan_tile_apply(const T* __restrict__ in, int64_t n, const int64_t* __restrict__ offs,
                                const int64_t* __restrict__ sums, int64_t* __restrict__ out,
                                int* __restrict__ out32) {
  __shared__ int64_t warp_tot[32];
  int64_t first = offs ? offs[blockIdx.x] : 0;
  if (sums) {
    int64_t v = 0;
    for (int k = threadIdx.x; k < (int)blockIdx.x; k += kScanThreads) v += sums[k];
    block_exclusive_scan<T>(v, warp_tot, first);
    __syncthreads();
  }
  int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int64_t v[kScanItems];
  int64_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = (base + k < n) ? (int64_t)in[base + k] : 0;
    s += v[k];
  }
  int64_t total;
  int64_t ex = block_exclusive_scan<T>(s, warp_tot, total) + first;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k < n) {
      out[base + k] = ex;
      if (out32) out32[base + k] = (int)ex;
    }
    ex += v[k];
  }
  // the last element of the whole array writes the grand total at out[n]
  if (base <= n - 1 && n - 1 < base + kScanItems) {
    out[n] = ex;
    if (out32) out32[n] = (int)ex;
  }
}

// Exclusive scan of in[0, n) into out[0, n] (out[n] = the total); out32,
// when given, receives the same values as 32-bit integers.
template <typename T>
void scan_impl(const T* in, int64_t* out, int64_t n, cudaStream_t s, DevBuf<int64_t>& tmp,
               size_t tmp_off, int* out32 = nullptr) {
  if (n <= 0) {
    GR_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(int64_t), s));
    if (out32) GR_CUDA_TRY(cudaMemsetAsync(out32, 0, sizeof(int), s));
    return;
  }
  int64_t tiles = (n + kScanTile - 1) / kScanTile;
  if (tiles == 1) {
    scan_tile_apply<T><<<1, kScanThreads, 0, s>>>(in, n, nullptr, nullptr, out, out32);
    GR_CHECK_LAUNCH();
    return;
  }
  int64_t* sums = tmp.p + tmp_off;
  int64_t* offs = sums + tiles;
  scan_tile_sums<T><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, n, sums);
  GR_CHECK_LAUNCH();
  const bool flat = tiles <= kScanFlat;
  if (!flat) scan_impl<int64_t>(sums, offs, tiles, s, tmp, tmp_off + 2 * tiles + 1);
  scan_tile_apply<T><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, n, flat ? nullptr : offs,
                                                              flat ? sums : nullptr, out, out32);
  GR_CHECK_LAUNCH();
}

size_t scan_tmp_need(int64_t n) {
  size_t need = 0;
  while (n > kScanTile) {
    int64_t tiles = (n + kScanTile - 1) / kScanTile;
    need += 2 * tiles + 1;
    n = tiles;
  }
  return need + 1;
}

}  // namespace

namespace {

__global__ void zero_many_kernel(ZeroList z) {
  zero_list(z, blockIdx.x * (size_t)blockDim.x + threadIdx.x, (size_t)gridDim.x * blockDim.x);
}

// Results of a call to pinned host memory; values of fixed-point sums are
// their limbs times inv (inverses of powers of two, so one rounding, as the
// host's fix_value).  split: (lo, hi) are the split limbs of fix_red, worth
// hi * 2^32 + lo (fix_split_value).
__global__ void results_kernel(ResultList r) {
  const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t nthr = (int64_t)gridDim.x * blockDim.x;
  for (int k = 0; k < r.n; ++k) {
    const ResultList::Part& a = r.part[k];
    if (a.per == 0) {
      for (int64_t i = tid; i < a.n; i += nthr) a.out[i] = a.lo[i];
      continue;
    }
    for (int64_t i = tid; i < a.n; i += nthr) {
      unsigned long long l = a.lo[i * a.stride], h = a.hi[i * a.stride];
      if (a.split) {
        // (signed h) << 32 as 128 bits, plus l
        const long long hs = (long long)h;
        const unsigned long long L = (unsigned long long)hs << 32;
        unsigned long long H = (unsigned long long)(hs >> 32);
        const unsigned long long L2 = L + l;
        H += L2 < L ? 1ull : 0ull;
        l = L2;
        h = H;
      }
      const int64_t c = i / a.per;
      const double is = c == 0 ? a.inv[0] : (c == 1 ? a.inv[1] : (c == 2 ? a.inv[2] : a.inv[3]));
      a.out[i] = (unsigned long long)__double_as_longlong(fix_to_double(l, h, is));
    }
  }
}

}  // namespace

void zero_async(const ZeroList& z, cudaStream_t s) {
  if (z.n == 0) return;
  size_t total = 0;
  for (int k = 0; k < z.n; ++k) total += z.bytes[k];
  const size_t threads = 256;
  size_t blocks = (total / 16 + threads - 1) / threads;
  if (blocks < 1) blocks = 1;
  if (blocks > (size_t)8 * sm_count()) blocks = (size_t)8 * sm_count();
  zero_many_kernel<<<(unsigned)blocks, (unsigned)threads, 0, s>>>(z);
  GR_CHECK_LAUNCH();
}

void results_async(const ResultList& r, cudaStream_t s) {
  int64_t most = 0;
  for (int k = 0; k < r.n; ++k) most = std::max(most, r.part[k].n);
  if (most == 0) return;
  const int blocks = (int)std::min<int64_t>((most + 255) / 256, 2 * (int64_t)sm_count());
  results_kernel<<<blocks, 256, 0, s>>>(r);
  GR_CHECK_LAUNCH();
}

void scan_i64(const int64_t* in, int64_t* out, int64_t n, cudaStream_t s, DevBuf<int64_t>& tmp) {
  size_t need = scan_tmp_need(n);
  if (tmp.n < need) tmp.reserve(need);
  scan_impl<int64_t>(in, out, n, s, tmp, 0);
}

void scan_i32_to_i64(const int* in, int64_t* out, int64_t n, cudaStream_t s, DevBuf<int64_t>& tmp,
                     int* out32) {
  size_t need = scan_tmp_need(n);
  if (tmp.n < need) tmp.reserve(need);
  scan_impl<int>(in, out, n, s, tmp, 0, out32);
}

}  // namespace gr

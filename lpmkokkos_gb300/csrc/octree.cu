// octree.cu -- device build of the Morton octree of pbosler/lpmKokkos.
//
// The same tree as the reference's (Zhou et al. 2011, listings 1-2; file:line per step below), from the
// sorted keys alone.  With the points in key order, point i opens a new cell of level l where its
// key's first 3 l bits differ from the point's before it; the first level at which they differ
// therefore gives all levels at once:
//   * the cells of level l, in order, are those points; their number, times 8 (complete sibling
//     sets), is the node count of level l + 1;
//   * the cell that point i belongs to at level l has the rank (openings at level l up to i) - 1;
//   * a non-empty node of level l + 1 is 8 rank_l + octant, its points run to the next opening, and the
//     set of its children is number rank_(l+1).
// So every level is counted, placed and filled in the same few launches instead of bottom-up, a
// scan and a read-back per level (about 70 launches before).  All data are integers or exact
// copies of FP64 inputs, so the result equals the serial restatement bit for bit.
//
// The neighbour walk reads the parent level at base_address(l-1) + index (the reference reads the
// level-local index as a global row, right only at level 1), and the neighbour tables follow from
// their geometric definition (the reference's ChildLUT differs in row 0, columns 18-20 and 24-26,
// which drop the +x bit).

#include "octree.hpp"

#include <cub/cub.cuh>

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cstdio>
#include <mutex>

#include "engine_core.hpp"
#include "lpm_octree.h"

namespace lpm {
namespace {

constexpr int kBlock = 256;
constexpr int kLevels = kOctreeMaxDepth + 1;
constexpr double kZeroTol = 1.0e-14;  // ZERO_TOL, src/LpmDefs.hpp:99

// Doubles as integers of the same order (-0 as 0): comparisons without the FP64 pipe, which takes
// 64 times as long for one as the FP32 pipe.  NaN, which no comparison holds for, is the smallest.
__device__ __forceinline__ long long orderOf(double v) {
  const long long b = __double_as_longlong(v);
  const long long mag = b & 0x7fffffffffffffffll;
  if (mag == 0) return 0;
  if (mag > 0x7ff0000000000000ll) return LLONG_MIN;
  return b < 0 ? ~mag : b;
}
__device__ __forceinline__ double valueOf(long long o) {
  return __longlong_as_double(o < 0 ? (~o | (long long)0x8000000000000000ull) : o);
}

// BoxFunctor / BBoxReducer (src/LpmBox3d.hpp:84-160): min and max per axis, as ordered integers in
// box[0..5] = {min x, reversed max x, min y, ...} (all minima, biased to unsigned, all ones before; NaN
// left out).  With REC the points are the FP32 hi / lo records of the sources, which are also written
// out in FP64.
template <bool REC>
__global__ void __launch_bounds__(kBlock) boxKernel(const double* __restrict__ x, int64_t si, int64_t sc,
                                                    const float4* __restrict__ sp0, const float4* __restrict__ sp1,
                                                    int64_t n, double* __restrict__ pos,
                                                    unsigned long long* __restrict__ box) {
  __shared__ long long sh[kBlock / 32][6];
  long long v[6];
  for (int k = 0; k < 6; ++k) v[k] = LLONG_MAX;
  for (int64_t i = (int64_t)blockIdx.x * kBlock + threadIdx.x; i < n; i += (int64_t)gridDim.x * kBlock) {
    double p[3];
    if (REC) {
      const float4 a = sp0[i], b = sp1[i];
      p[0] = (double)a.x + (double)b.x;
      p[1] = (double)a.y + (double)b.y;
      p[2] = (double)a.z + (double)b.z;
      for (int c = 0; c < 3; ++c) pos[3 * i + c] = p[c];
    } else {
      for (int c = 0; c < 3; ++c) p[c] = x[i * si + c * sc];
    }
    for (int c = 0; c < 3; ++c) {
      const long long o = orderOf(p[c]);
      if (o == LLONG_MIN) continue;
      v[2 * c] = min(v[2 * c], o);
      v[2 * c + 1] = min(v[2 * c + 1], ~o);  // ~o reverses the order
    }
  }
  for (int k = 0; k < 6; ++k)
    for (int d = 16; d > 0; d >>= 1) v[k] = min(v[k], __shfl_xor_sync(0xffffffffu, v[k], d));
  if ((threadIdx.x & 31) == 0)
    for (int k = 0; k < 6; ++k) sh[threadIdx.x >> 5][k] = v[k];
  __syncthreads();
  if (threadIdx.x < 6) {
    long long m = sh[0][threadIdx.x];
    for (int w = 1; w < kBlock / 32; ++w) m = min(m, sh[w][threadIdx.x]);
    atomicMin(box + threadIdx.x, (unsigned long long)m ^ 0x8000000000000000ull);
  }
}

// compute_key_for_point (src/LpmOctreeUtil.hpp:57-81) with box2cube (src/LpmBox3d.hpp:290-303): the same
// comparisons and centre updates.
__device__ __forceinline__ void cubeOf(const double* __restrict__ b, double (&c)[3], double& half) {
  double xmin = b[0], xmax = b[1], ymin = b[2], ymax = b[3], zmin = b[4], zmax = b[5];
  const double dx = xmax - xmin, dy = ymax - ymin, dz = zmax - zmin;
  const double lo = fmin(fmin(dx, dy), dz), hi = fmax(fmax(dx, dy), dz);
  if (fabs(hi / lo - 1.0) > kZeroTol) {
    const double h = 0.5 * hi;
    const double mx = 0.5 * (xmin + xmax), my = 0.5 * (ymin + ymax), mz = 0.5 * (zmin + zmax);
    xmin = mx - h; xmax = mx + h; ymin = my - h; ymax = my + h; zmin = mz - h; zmax = mz + h;
  }
  c[0] = 0.5 * (xmin + xmax); c[1] = 0.5 * (ymin + ymax); c[2] = 0.5 * (zmin + zmax);
  half = 0.5 * (xmax - xmin);
}

// One block: the box in FP64, and per axis the centres that a point's key is formed with:
// split[axis][k], k = 1..2^depth - 1, is the centre that the bits of k above its last 1 lead to.
__global__ void __launch_bounds__(kBlock) splitsKernel(const unsigned long long* __restrict__ obox, int depth,
                                                       double* __restrict__ box, long long* __restrict__ split) {
  __shared__ double sb[6];
  if (threadIdx.x < 6) {
    const long long o = (long long)(obox[threadIdx.x] ^ 0x8000000000000000ull);
    const bool mx = threadIdx.x & 1;
    // (a cloud of NaNs keeps the start of the reduction)
    const double v = o == LLONG_MAX ? (mx ? -DBL_MAX : DBL_MAX) : valueOf(mx ? ~o : o);
    sb[threadIdx.x] = v;
    box[threadIdx.x] = v;
  }
  __syncthreads();
  double c0[3], half0;
  cubeOf(sb, c0, half0);
  const int m = 1 << depth;
  for (int q = threadIdx.x; q < 3 * m; q += kBlock) {
    const int axis = q / m, k = q % m;
    if (k == 0) continue;
    const int lev = depth - (__ffs(k) - 1);  // 1 = the root's centre
    double c = c0[axis], h = half0;
    for (int i = 1; i < lev; ++i) {
      h *= 0.5;
      c += (k >> (depth - i)) & 1 ? h : -h;
    }
    split[q] = isnan(c) ? LLONG_MAX : orderOf(c);  // no comparison with a NaN holds
  }
}

__device__ __forceinline__ uint32_t spread(uint32_t v) {  // 10 bits -> every third bit
  v = (v | (v << 16)) & 0x030000ffu;
  v = (v | (v << 8)) & 0x0300f00fu;
  v = (v | (v << 4)) & 0x030c30c3u;
  return (v | (v << 2)) & 0x09249249u;
}

// EncodeFunctor (src/LpmOctreeKernels.hpp:27-47): keys and point ids.
__global__ void __launch_bounds__(kBlock) keysKernel(const double* __restrict__ x, int64_t si, int64_t sc, int64_t n,
                                                     int depth, const long long* __restrict__ split,
                                                     uint32_t* __restrict__ keys, int* __restrict__ ids) {
  extern __shared__ long long sSplit[];
  const int m = 1 << depth;
  for (int q = threadIdx.x; q < 3 * m; q += kBlock) sSplit[q] = split[q];
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * kBlock + threadIdx.x; i < n; i += (int64_t)gridDim.x * kBlock) {
    const double p[3] = {x[i * si], x[i * si + sc], x[i * si + 2 * sc]};
    uint32_t key = 0;
    for (int a = 0; a < 3; ++a) {
      const long long o = orderOf(p[a]);
      int k = 0;
      if (o != LLONG_MIN)
        for (int b = m >> 1; b > 0; b >>= 1)  // level by level, the reference's comparisons
          if (sSplit[a * m + k + b] <= o) k += b;
      key |= spread((uint32_t)k) << (2 - a);
    }
    keys[i] = key;
    ids[i] = (int)i;
  }
}

// The first level at which point i's cell differs from the one of the point before it (0 for the first
// point, kLevels if they share the leaf).
__device__ __forceinline__ int openLevel(const uint32_t* __restrict__ keys, int64_t i, int64_t n, int depth) {
  if (i >= n) return kLevels;
  if (i == 0) return 0;
  const uint32_t x = keys[i] ^ keys[i - 1];
  return x ? depth - (31 - __clz(x)) / 3 : kLevels;
}

// Openings per level of each block of kBlock points: hist[level][block].
__global__ void __launch_bounds__(kBlock) openKernel(const uint32_t* __restrict__ keys, int64_t n, int depth, int nb,
                                                     int* __restrict__ hist) {
  __shared__ int cnt[kLevels];
  if (threadIdx.x < kLevels) cnt[threadIdx.x] = 0;
  __syncthreads();
  const int lev = openLevel(keys, (int64_t)blockIdx.x * kBlock + threadIdx.x, n, depth);
  for (int l = 0; l <= depth; ++l) {
    const unsigned w = __ballot_sync(0xffffffffu, lev <= l);
    if ((threadIdx.x & 31) == 0 && w) atomicAdd(&cnt[l], __popc(w));
  }
  __syncthreads();
  if (threadIdx.x <= depth) hist[(size_t)threadIdx.x * nb + blockIdx.x] = cnt[threadIdx.x];
}

// hist[level] to exclusive sums over the blocks, one warp per level; cells[level] = the number of cells,
// counts[level] = the number of nodes (complete sibling sets).
__global__ void __launch_bounds__(32 * kLevels) offsetsKernel(int nb, int depth, int* __restrict__ hist,
                                                              int* __restrict__ cells, int* __restrict__ counts) {
  const int lev = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lev > depth) return;
  int* h = hist + (size_t)lev * nb;
  int run = 0;
  for (int b0 = 0; b0 < nb; b0 += 128) {  // four values a lane
    int v[4], sum = 0;
    for (int k = 0; k < 4; ++k) {
      const int b = b0 + 4 * lane + k;
      v[k] = b < nb ? h[b] : 0;
      sum += v[k];
    }
    int incl = sum;
    for (int d = 1; d < 32; d <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += o;
    }
    int at = run + incl - sum;
    for (int k = 0; k < 4; ++k) {
      const int b = b0 + 4 * lane + k;
      if (b < nb) h[b] = at;
      at += v[k];
    }
    run += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) {
    cells[lev] = run;
    if (lev < depth) counts[lev + 1] = 8 * run;
    if (lev == 0) counts[0] = 1;
  }
}

// Where each level's cells and nodes are stored.
struct LevelBases {
  int cell[kLevels + 1];
  int node[kLevels + 1];
};

// Per cell: its first point, and the rank of its parent cell.  Per point: PermuteFunctor
// (src/LpmOctreeKernels.hpp:49-72) and its leaf.
__global__ void __launch_bounds__(kBlock) placeKernel(const uint32_t* __restrict__ keys, const int* __restrict__ ids,
                                                      int64_t n, int depth, int nb, const int* __restrict__ hist,
                                                      const LevelBases lb, int* __restrict__ first,
                                                      int* __restrict__ up, const double* __restrict__ x, int64_t si,
                                                      int64_t sc, double* __restrict__ sorted, int* __restrict__ leaf) {
  __shared__ int warpCnt[kLevels][kBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t i = (int64_t)blockIdx.x * kBlock + threadIdx.x;
  const int lev = openLevel(keys, i, n, depth);
  int rank[kLevels];
#pragma unroll
  for (int l = 0; l < kLevels; ++l) {
    if (l > depth) break;
    const unsigned w = __ballot_sync(0xffffffffu, lev <= l);
    rank[l] = __popc(w & (0xffffffffu >> (31 - lane))) - 1;
    if (lane == 0) warpCnt[l][warp] = __popc(w);
  }
  __syncthreads();
  if (i >= n) return;
#pragma unroll
  for (int l = 0; l < kLevels; ++l) {
    if (l > depth) break;
    int r = hist[(size_t)l * nb + blockIdx.x] + rank[l];
    for (int w = 0; w < warp; ++w) r += warpCnt[l][w];
    rank[l] = r;
    if (lev <= l) {
      first[lb.cell[l] + r] = (int)i;
      up[lb.cell[l] + r] = l > 0 ? rank[l > 0 ? l - 1 : 0] : 0;
    }
    if (l == depth) leaf[i] = 8 * rank[l > 0 ? l - 1 : 0] + (int)(keys[i] & 7u);
  }
  if (sorted) {
    const int64_t id = ids[i];
    for (int c = 0; c < 3; ++c) sorted[3 * i + c] = x[id * si + c * sc];
  }
}

// Key algebra of src/LpmOctreeUtil.hpp:83-135 (keys at max-depth resolution).
__device__ __forceinline__ uint32_t prefixOf(uint32_t key, int lev, int depth) {
  const int drop = 3 * (depth - lev);
  return lev == 0 ? 0u : (key >> drop) << drop;
}

// The nodes (src/LpmOctreeKernels.hpp:233-369, src/LpmNodeArrayInternal.cpp:13-52): eight threads per
// cell of levels 0..depth-1, thread c its child node c of the level below, empty or not; the root.
__global__ void __launch_bounds__(kBlock) nodesKernel(const uint32_t* __restrict__ pkeys, int64_t n, int depth,
                                                      const LevelBases lb, const int* __restrict__ cells,
                                                      const int* __restrict__ first, const int* __restrict__ up,
                                                      uint32_t* __restrict__ keys, int2* __restrict__ pt,
                                                      int* __restrict__ parents, int* __restrict__ kids) {
  const int q = blockIdx.x * kBlock + threadIdx.x;
  const int at = q >> 3, c = q & 7;
  int lev = 0;
  while (lev + 1 < depth && at >= lb.cell[lev + 1]) ++lev;
  const int r = at - lb.cell[lev];
  if (r >= cells[lev]) return;
  const int i = first[lb.cell[lev] + r];
  const uint32_t own = pkeys[i], prefix = prefixOf(own, lev, depth);
  const int node = lev == 0 ? 0 : 8 * up[lb.cell[lev] + r] + (int)((own >> (3 * (depth - lev))) & 7u);
  if (lev == 0 && c == 0) {
    keys[0] = 0;
    parents[0] = -1;
    pt[0] = make_int2(0, (int)n);
  }
  if (lev == 0) kids[c] = c;
  // the child cell of octant c, if it has points: its cells follow each other from the one that this
  // cell's first point opens
  const int cellsBelow = cells[lev + 1];
  const int* firstB = first + lb.cell[lev + 1];
  const int* upB = up + lb.cell[lev + 1];
  const int shift = 3 * (depth - lev - 1);
  int lo = 0, hi = cellsBelow;  // the first child cell: the one whose first point is i
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (firstB[mid] < i) lo = mid + 1;
    else hi = mid;
  }
  int m = -1;
  for (int k = lo; k < min(lo + 8, cellsBelow) && upB[k] == r; ++k)
    if ((int)((pkeys[firstB[k]] >> shift) & 7u) == c) m = k;
  const size_t g = (size_t)lb.node[lev + 1] + 8 * (size_t)r + c;
  keys[g] = prefix + ((uint32_t)c << shift);
  parents[g] = node;
  pt[g] = m < 0 ? make_int2(-1, 0)
                : make_int2(firstB[m], (m + 1 < cellsBelow ? firstB[m + 1] : (int)n) - firstB[m]);
  for (int k = 0; k < 8; ++k) kids[8 * g + k] = m < 0 || lev + 1 == depth ? -1 : 8 * m + k;
}

// NeighborhoodFunctor (src/LpmOctreeKernels.hpp:371-400) at level lev, parent level arrays at their own
// base.  Neighbour j = 9a + 3b + c of a node with local key i = 4x + 2y + z (offsets (a-1, b-1, c-1)):
// along an axis with bit s and offset o, its parent lies po = floor((s + o) / 2) cells over, and it
// is that cell's child s + o - 2 po (src/LpmOctreeLUT.hpp:70-137 tabulates the same).  27 threads a
// node: the lists are written coalesced.
__global__ void __launch_bounds__(kBlock) neighborsKernel(const uint32_t* __restrict__ keys,
                                                          const int* __restrict__ parents, int m, int lev, int depth,
                                                          const int* __restrict__ upNbrs,
                                                          const int* __restrict__ upKids, int* __restrict__ nbrs) {
  const int64_t q = (int64_t)blockIdx.x * kBlock + threadIdx.x;
  if (q >= 27 * (int64_t)m) return;
  const int t = (int)(q / 27), j = (int)(q % 27);
  if (lev == 0) {
    nbrs[q] = j == 13 ? 0 : -1;
    return;
  }
  const int i = (int)((keys[t] >> (3 * (depth - lev))) & 7u);
  const int off[3] = {j / 9 - 1, (j / 3) % 3 - 1, j % 3 - 1};
  int pj = 0, cj = 0;
  for (int a = 0; a < 3; ++a) {
    const int s = ((i >> (2 - a)) & 1) + off[a];
    const int po = s < 0 ? -1 : (s > 1 ? 1 : 0);
    pj = 3 * pj + po + 1;
    cj = 2 * cj + (s - 2 * po);
  }
  const int h = upNbrs[27 * (size_t)parents[t] + pj];
  nbrs[q] = h != -1 ? upKids[8 * (size_t)h + cj] : -1;
}

inline unsigned blocksFor(int64_t n) { return (unsigned)((n + kBlock - 1) / kBlock); }

void check(cudaError_t e, const char* what) {
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    fail(e == cudaErrorMemoryAllocation ? LPM_ERR_OUT_OF_MEMORY : LPM_ERR_CUDA, "octree %s: %s", what,
         cudaGetErrorString(e));
  }
}

// Octrees take their two blocks of memory from one pool per device, which keeps at most kPoolKeeps
// bytes of freed blocks for the next tree (a build would otherwise wait for the system's allocator
// each time: about a millisecond) and returns the rest when the device is next synchronised.
constexpr int kMaxDevices = 64;
constexpr uint64_t kPoolKeeps = uint64_t(64) << 20;

cudaMemPool_t poolOf(int dev) {
  static std::mutex mu;
  static cudaMemPool_t pools[kMaxDevices] = {};  // (kept until the process ends)
  std::lock_guard<std::mutex> lk(mu);
  if (!pools[dev]) {
    cudaMemPoolProps p{};
    p.allocType = cudaMemAllocationTypePinned;
    p.location.type = cudaMemLocationTypeDevice;
    p.location.id = dev;
    cudaMemPool_t pool = nullptr;
    check(cudaMemPoolCreate(&pool, &p), "memory pool");
    uint64_t keep = kPoolKeeps;
    check(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep), "memory pool");
    pools[dev] = pool;
  }
  return pools[dev];
}

// Carves arrays out of one block, 256-byte aligned; with a null block it only adds up.
struct Carver {
  char* p;
  size_t at = 0;
  template <typename T>
  T* take(size_t count) {
    T* r = reinterpret_cast<T*>(p ? p + at : nullptr);
    at += (std::max<size_t>(1, count) * sizeof(T) + 255) / 256 * 256;
    return r;
  }
};

}  // namespace

void* Octree::grow(Buf& b, size_t bytes, cudaStream_t s) {
  if (b.bytes < bytes) {
    if (b.p) check(cudaFreeAsync(b.p, s), "free");
    b = Buf{};
    int dev = 0;
    check(cudaGetDevice(&dev), "device query");
    if (dev < 0 || dev >= kMaxDevices) fail(LPM_ERR_NOT_SUPPORTED, "octree: device ordinal %d >= %d", dev, kMaxDevices);
    check(cudaMallocFromPoolAsync(&b.p, bytes, poolOf(dev), s), "allocation");
    b.bytes = bytes;
  }
  return b.p;
}

void Octree::release(cudaStream_t s) {
  for (Buf* b : {&work_, &out_}) {
    if (b->p) cudaFreeAsync(b->p, s);
    *b = Buf{};
  }
  dcount = nullptr;
  nnodes = 0;
}

Octree::~Octree() {
  if (!work_.p && !out_.p) return;  // released in stream order: nothing to wait for
  cudaDeviceSynchronize();          // any stream may still read the arrays
  release(nullptr);
}

// Box, keys, sort and the counts of every level, on the device.
void Octree::sortAndCount(const Points& X, cudaStream_t s) {
  const unsigned nb = blocksFor(n);
  const int m = 1 << depth;
  size_t tsort = 0;
  check(cub::DeviceRadixSort::SortPairs(nullptr, tsort, (uint32_t*)nullptr, (uint32_t*)nullptr, (int*)nullptr,
                                        (int*)nullptr, (int)n, 0, 3 * depth, s),
        "sort size");
  Carver c{nullptr};
  for (int pass = 0; pass < 2; ++pass) {
    if (pass == 1) c = Carver{static_cast<char*>(grow(work_, c.at, s))};
    obox_ = c.take<unsigned long long>(6);
    box_ = c.take<double>(6);
    dcount = c.take<int>(kLevels + 1);
    cells_ = c.take<int>(kLevels + 1);
    split_ = c.take<long long>(3 * (size_t)m);
    keys1_ = c.take<uint32_t>(n);
    keys2_ = c.take<uint32_t>(n);
    ids1_ = c.take<int>(n);
    hist_ = c.take<int>((size_t)(depth + 1) * nb);
    temp_ = c.take<char>(tsort);
    pos_ = X.rec0 ? c.take<double>(3 * (size_t)n) : nullptr;
    ids2_ = c.take<int>(n);
  }
  check(cudaMemsetAsync(obox_, 0xff, 6 * sizeof(long long), s), "clear");
  const unsigned boxBlocks = std::min(nb, 608u);
  if (X.rec0)
    boxKernel<true><<<boxBlocks, kBlock, 0, s>>>(nullptr, 0, 0, X.rec0, X.rec1, n, pos_, obox_);
  else
    boxKernel<false><<<boxBlocks, kBlock, 0, s>>>(X.x, X.si, X.sc, nullptr, nullptr, n, nullptr, obox_);
  splitsKernel<<<1, kBlock, 0, s>>>(obox_, depth, box_, split_);
  dbox = box_;
  const double* x = X.rec0 ? pos_ : X.x;
  const int64_t si = X.rec0 ? 3 : X.si, sc = X.rec0 ? 1 : X.sc;
  keysKernel<<<std::min(nb, 1216u), kBlock, 3 * (size_t)m * sizeof(long long), s>>>(x, si, sc, n, depth, split_, keys1_,
                                                                                    ids1_);
  // stable: points of one key stay in input order (the reference sorts key << 32 | id)
  check(cub::DeviceRadixSort::SortPairs(temp_, tsort, keys1_, keys2_, ids1_, ids2_, (int)n, 0, 3 * depth, s), "sort");
  openKernel<<<nb, kBlock, 0, s>>>(keys2_, n, depth, (int)nb, hist_);
  offsetsKernel<<<1, 32 * kLevels, 0, s>>>((int)nb, depth, hist_, cells_, dcount);
}

// The arrays, level l's nodes at base[l] and its cells (scratch) at cell[l] of `ncells`.
void Octree::fill(const Points& X, const int* cell, int64_t ncells, bool neighbors, bool wantSorted, bool clearPt,
                  cudaStream_t s) {
  const unsigned nb = blocksFor(n);
  int *first = nullptr, *up = nullptr;
  Carver c{nullptr};
  for (int pass = 0; pass < 2; ++pass) {
    if (pass == 1) c = Carver{static_cast<char*>(grow(out_, c.at, s))};
    first = c.take<int>(ncells);
    up = c.take<int>(ncells);
    keys = c.take<uint32_t>(nnodes);
    ptInds = c.take<int2>(nnodes);
    parents = c.take<int>(nnodes);
    kids = c.take<int>(8 * (size_t)nnodes);
    nbrs = neighbors ? c.take<int>(27 * (size_t)nnodes) : nullptr;
    sorted = wantSorted ? c.take<double>(3 * (size_t)n) : nullptr;
    ptInLeaf = c.take<int>(n);
  }
  origIds = ids2_;
  if (clearPt) check(cudaMemsetAsync(ptInds, 0, sizeof(int2) * (size_t)nnodes, s), "clear");  // empty past the counts
  LevelBases lb{};
  for (int l = 0; l <= depth; ++l) {
    lb.cell[l] = cell[l];
    lb.node[l] = base[l];
  }
  const double* x = X.rec0 ? pos_ : X.x;
  placeKernel<<<nb, kBlock, 0, s>>>(keys2_, ids2_, n, depth, (int)nb, hist_, lb, first, up, x, X.rec0 ? 3 : X.si,
                                    X.rec0 ? 1 : X.sc, sorted, ptInLeaf);
  nodesKernel<<<blocksFor(8 * (int64_t)cell[depth]), kBlock, 0, s>>>(keys2_, n, depth, lb, cells_, first, up, keys,
                                                                      ptInds, parents, kids);
}

void Octree::build(const double* x, int64_t si, int64_t sc, int64_t npts, int maxDepth, bool neighbors,
                   cudaStream_t s) {
  if (maxDepth < 1 || maxDepth > kOctreeMaxDepth) fail(LPM_ERR_INVALID_ARGUMENT, "octree depth must be 1..%d", kOctreeMaxDepth);
  if (npts <= 0 || npts > INT32_MAX) fail(LPM_ERR_INVALID_ARGUMENT, "octree: 1..2^31-1 points");
  depth = maxDepth;
  n = npts;
  const Points X{x, si, sc, nullptr, nullptr};
  sortAndCount(X, s);
  // the level sizes and the box
  int h[2 * (kLevels + 1)] = {};
  check(cudaMemcpyAsync(h, cells_, sizeof(int) * (depth + 1), cudaMemcpyDeviceToHost, s), "read-back");
  check(cudaMemcpyAsync(box, box_, sizeof(box), cudaMemcpyDeviceToHost, s), "read-back");
  check(cudaStreamSynchronize(s), "synchronise");
  int cell[kLevels + 1] = {};
  int64_t ncells = 0;
  nnodes = 0;
  for (int l = 0; l <= depth; ++l) {  // concatenation as Tree::initNodes (src/LpmOctree.cpp:45-75)
    cell[l] = (int)ncells;
    ncells += h[l];
    npl[l] = l == 0 ? 1 : 8 * h[l - 1];
    base[l] = (int)nnodes;
    nnodes += npl[l];
  }
  if (nnodes > INT32_MAX / 8) fail(LPM_ERR_NOT_SUPPORTED, "octree: %lld nodes", (long long)nnodes);
  fill(X, cell, ncells, neighbors, true, false, s);
  if (neighbors)
    for (int l = 0; l <= depth; ++l) {
      const size_t b = (size_t)base[l], u = l > 0 ? (size_t)base[l - 1] : 0;
      neighborsKernel<<<blocksFor(27 * (int64_t)npl[l]), kBlock, 0, s>>>(keys + b, parents + b, npl[l], l, depth,
                                                                         nbrs + 27 * u, kids + 8 * u, nbrs + 27 * b);
    }
  check(cudaGetLastError(), "launch");
  check(cudaStreamSynchronize(s), "synchronise");  // callers read the arrays on any stream
}

void Octree::buildOnDevice(const Points& X, int64_t npts, int maxDepth, bool wantSorted, cudaStream_t s) {
  if (maxDepth < 1 || maxDepth > kOctreeMaxDepth) fail(LPM_ERR_INVALID_ARGUMENT, "octree depth must be 1..%d", kOctreeMaxDepth);
  if (npts <= 0 || npts > INT32_MAX / 8) fail(LPM_ERR_INVALID_ARGUMENT, "octree: 1..2^28-1 points");
  depth = maxDepth;
  n = npts;
  // capacities: a level holds complete sibling sets of at most 8^l nodes, and at most 8 per cell of
  // the level above (<= n cells)
  int cell[kLevels + 1] = {};
  int64_t total = 0, ncells = 0;
  for (int l = 0; l <= depth; ++l) {
    int64_t c = 1;
    for (int k = 0; k < l && c < 8 * n; ++k) c *= 8;
    gbase[l] = base[l] = (int)std::min<int64_t>(total, INT32_MAX);
    cell[l] = (int)std::min<int64_t>(ncells, INT32_MAX);
    npl[l] = 0;  // counts live on the device (dcount)
    total += std::min<int64_t>(c, l == 0 ? 1 : 8 * n);
    ncells += std::min<int64_t>(c, n);
  }
  if (total > INT32_MAX / 8) fail(LPM_ERR_NOT_SUPPORTED, "octree: %lld nodes of fixed-level capacity", (long long)total);
  gbase[depth + 1] = (int)total;
  nnodes = total;
  sortAndCount(X, s);
  fill(X, cell, ncells, false, wantSorted, true, s);
  check(cudaGetLastError(), "launch");
}

}  // namespace lpm

struct lpm_octree {
  lpm::Octree tree;
  int device = 0;
  bool fixed = false;  // LPM_OCTREE_FIXED_LEVELS: counts and box still on the device
};

extern "C" {

int lpm_octree_build(const double* x, int64_t x_si, int64_t x_sc, int64_t n, int max_depth, int neighbors,
                     lpm_octree** out, lpm_stream_t stream) {
  if (!out) return LPM_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  if (!x || n <= 0 || n > INT32_MAX || x_si < 0 || x_sc < 0 || max_depth < 1 || max_depth > lpm::kOctreeMaxDepth)
    return LPM_ERR_INVALID_ARGUMENT;
  const bool fixed = neighbors & LPM_OCTREE_FIXED_LEVELS;
  if ((neighbors & ~(LPM_OCTREE_NEIGHBORS | LPM_OCTREE_FIXED_LEVELS)) ||
      (fixed && (neighbors & LPM_OCTREE_NEIGHBORS)) || (fixed && n > INT32_MAX / 8))
    return LPM_ERR_INVALID_ARGUMENT;
  lpm_octree* t = new (std::nothrow) lpm_octree();
  if (!t) return LPM_ERR_OUT_OF_MEMORY;
  try {
    lpm::check(cudaGetDevice(&t->device), "device");
    t->fixed = fixed;
    if (fixed)
      t->tree.buildOnDevice(lpm::Octree::Points{x, x_si, x_sc, nullptr, nullptr}, n, max_depth, true,
                            (cudaStream_t)stream);
    else
      t->tree.build(x, x_si, x_sc, n, max_depth, neighbors & LPM_OCTREE_NEIGHBORS, (cudaStream_t)stream);
  } catch (const lpm::Error& e) {
    std::fprintf(stderr, "lpm_octree_build: %s\n", e.msg.c_str());
    delete t;
    return e.code;
  } catch (const std::exception& e) {
    std::fprintf(stderr, "lpm_octree_build: %s\n", e.what());
    delete t;
    return lpm::fromStd(e).code;
  }
  *out = t;
  return LPM_OK;
}

int lpm_octree_info(const lpm_octree* t, int* max_depth, int64_t* nnodes_total, int64_t* npoints,
                    int32_t* nnodes_per_level, int32_t* base_address, double* box) {
  if (!t) return LPM_ERR_INVALID_ARGUMENT;
  lpm::Octree& T = const_cast<lpm_octree*>(t)->tree;
  if (t->fixed) {  // the sync-free build left its level counts and box on the device
    int cnt[lpm::kOctreeMaxDepth + 2] = {};
    if (cudaSetDevice(t->device) != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess ||
        cudaMemcpy(cnt, T.dcount, sizeof(int) * (T.depth + 1), cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(T.box, T.dbox, sizeof(T.box), cudaMemcpyDeviceToHost) != cudaSuccess)
      return LPM_ERR_CUDA;
    for (int l = 0; l <= T.depth; ++l) T.npl[l] = cnt[l];
  }
  if (max_depth) *max_depth = T.depth;
  if (nnodes_total) *nnodes_total = T.nnodes;
  if (npoints) *npoints = T.n;
  for (int l = 0; l <= T.depth; ++l) {
    if (nnodes_per_level) nnodes_per_level[l] = T.npl[l];
    if (base_address) base_address[l] = T.base[l];
  }
  if (box)
    for (int c = 0; c < 6; ++c) box[c] = T.box[c];
  return LPM_OK;
}

int lpm_octree_arrays(const lpm_octree* t, const uint32_t** keys, const int32_t** pt_inds, const int32_t** parents,
                      const int32_t** kids, const int32_t** neighbors, const double** sorted_pts,
                      const int32_t** orig_ids, const int32_t** pt_in_leaf) {
  if (!t) return LPM_ERR_INVALID_ARGUMENT;
  const lpm::Octree& T = t->tree;
  if (keys) *keys = T.keys;
  if (pt_inds) *pt_inds = reinterpret_cast<const int32_t*>(T.ptInds);
  if (parents) *parents = T.parents;
  if (kids) *kids = T.kids;
  if (neighbors) *neighbors = T.nbrs;
  if (sorted_pts) *sorted_pts = T.sorted;
  if (orig_ids) *orig_ids = T.origIds;
  if (pt_in_leaf) *pt_in_leaf = T.ptInLeaf;
  return LPM_OK;
}

int lpm_octree_destroy(lpm_octree* t) {
  if (!t) return LPM_ERR_INVALID_ARGUMENT;
  cudaSetDevice(t->device);
  delete t;
  return LPM_OK;
}

}  // extern "C"

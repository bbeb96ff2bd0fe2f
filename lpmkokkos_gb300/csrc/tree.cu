// tree.cu -- the tree-code evaluation (tree.hpp): source octree, upward pass (cluster centres,
// radii, gnomonic charts and proxy charges), target-tile geometry, interaction lists, and the
// host orchestration around the gathered pair kernel (pair_kernels.cu).
//
// Proxy charges use the barycentric form of Lagrange interpolation at Chebyshev points of the
// second kind, t_a = cos(pi a / n), weights (-1)^a (halved at both ends) (Berrut & Trefethen,
// "Barycentric Lagrange interpolation", SIAM Review 46(3), 2004), in the tensor-product form
// of the barycentric Lagrange tree code (Wang, Krasny & Tlupova, Commun. Comput. Phys. 28(4),
// 2020), here on a per-cluster gnomonic chart of the sphere.  All reductions run in a fixed
// order, so an evaluation is reproducible bit for bit.

#include "tree_eval.hpp"

#include <cub/cub.cuh>

#include <algorithm>
#include <cstring>
#include <cfloat>
#include <climits>
#include <cmath>
#include <mutex>
#include <numeric>
#include <utility>
#include <vector>

namespace lpm {
namespace {

constexpr int kBlock = 256;
constexpr int kUpThreads = 128;
constexpr int kMaxDegree = 10;            // (n+1)^2 <= 121 proxies: one thread per proxy charge
constexpr int kMaxNodes1D = kMaxDegree + 1;
// A chart covers sources within ~37 degrees of its centre direction: an octant (54.7 degrees)
// stretches its gnomonic chart 3x at the edge and its degree-8 interpolant then errs by 1e-5.
constexpr double kMinChartCos = 0.8;

__device__ __forceinline__ bool sane(double x, double y, double z) {
  const double r2 = x * x + y * y + z * z;
  return r2 >= 0.25 && r2 <= 4.0;  // false for NaN
}

// Fixed-order block reductions (warp shuffles, then the warps' partials in order).
// FP32: FP64 runs at 1/64 of the FP32 rate on GB300, and in a kernel whose work per block is
// short, FP64 reductions over every thread are a large share of the FP64 pipe.
template <int NT>
__device__ __forceinline__ float blockSumF(float v, float* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
  for (int w = 0; w < NT / 32; ++w) t += sh[w];
  return t;
}
template <int NT>
__device__ __forceinline__ float blockMaxF(float v, float* sh) {
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_down_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = -FLT_MAX;
  for (int w = 0; w < NT / 32; ++w) t = fmaxf(t, sh[w]);
  return t;
}
__device__ __forceinline__ void kahanAddF(float& h, float& c, float v) {
  const float y = v - c;
  const float t = h + y;
  c = (t - h) - y;
  h = t;
}

__global__ void gatherSources(const int* __restrict__ orig, const float4* __restrict__ sp0,
                              const float4* __restrict__ sp1, const int* __restrict__ srcSlot, int ns,
                              float4* __restrict__ tsp0, float4* __restrict__ tsp1, int* __restrict__ inv,
                              int* __restrict__ tslot) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= ns) return;
  const int o = orig[k];
  tsp0[k] = sp0[o];
  tsp1[k] = sp1[o];
  tslot[k] = srcSlot[o];
  inv[o] = k;
}

__global__ void sortedSelf(const int* __restrict__ self, const int* __restrict__ inv, int nslots,
                           int* __restrict__ out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nslots) return;
  const int s = self[t];
  out[t] = s >= 0 ? inv[s] : -1;
}

// Centroid and radius of each target tile over its vertices and leaf faces.  Masked parent
// faces do not shape the tile: on the icosahedral mesh a parent's centre lies within ~1e-6 of its
// middle child's, its velocity is near-singular in the reference's formula, and after a step it
// runs away (its bounding sphere would then admit no far field).  Parents are still evaluated with their tile's
// list; a cubed-sphere parent sits on its children's shared corner, inside the tile.
// One warp per tile (tiles hold at most a few hundred slots); the butterfly reductions leave the
// same value in every lane.
__device__ __forceinline__ double warpSumAll(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
constexpr int kGeomTilesPerBlock = kBlock / 32;
constexpr int kGeomPerLane = kTreeShape.threads * kTreeShape.k / 32;

// Whether a slot's position shapes its tile: near the sphere (sane), decided in FP32 except close to
// the bounds, where FP64 decides (an FP64 instruction takes the time of 64 FP32 ones).
__device__ __forceinline__ bool saneFast(double x, double y, double z) {
  const float fx = (float)x, fy = (float)y, fz = (float)z;
  const float r2 = fx * fx + fy * fy + fz * fz;
  if (r2 > 0.2501f && r2 < 3.9999f) return true;
  if (r2 < 0.2499f || r2 > 4.0001f) return false;
  return sane(x, y, z);  // and NaN
}

__global__ void __launch_bounds__(kBlock) tileGeometry(const double* __restrict__ tx, int n,
                                                       const int2* __restrict__ tiles, int ntiles,
                                                       const int* __restrict__ perm, int64_t na,
                                                       const uint8_t* __restrict__ mask,
                                                       float4* __restrict__ geom) {
  const int lane = threadIdx.x & 31;
  const int tile = blockIdx.x * kGeomTilesPerBlock + (threadIdx.x >> 5);
  if (tile >= ntiles) return;  // the whole warp
  const int2 tr = tiles[tile];
  const int t0 = tr.x, cnt = tr.y;  // cnt <= 32 kGeomPerLane
  double px[kGeomPerLane], py[kGeomPerLane], pz[kGeomPerLane];
  bool shapes[kGeomPerLane];
#pragma unroll
  for (int k = 0; k < kGeomPerLane; ++k) {
    const int q = lane + 32 * k, slot = t0 + q;
    shapes[k] = false;
    if (q < cnt) {
      px[k] = tx[slot]; py[k] = tx[n + slot]; pz[k] = tx[2 * n + slot];
      const int id = perm[slot];
      shapes[k] = !(mask && id >= na && mask[id - na]);
    }
  }
  double sx = 0, sy = 0, sz = 0;
  int sc = 0;
#pragma unroll
  for (int k = 0; k < kGeomPerLane; ++k) {
    shapes[k] = shapes[k] && saneFast(px[k], py[k], pz[k]);
    if (shapes[k]) { sx += px[k]; sy += py[k]; sz += pz[k]; ++sc; }
  }
  sx = warpSumAll(sx);
  sy = warpSumAll(sy);
  sz = warpSumAll(sz);
  sc = __reduce_add_sync(0xffffffffu, sc);
  if (sc == 0) {
    if (lane == 0) geom[tile] = make_float4(0.f, 0.f, 0.f, INFINITY);
    return;
  }
  const double cx = sx / sc, cy = sy / sc, cz = sz / sc;
  double r2 = 0.0;
#pragma unroll
  for (int k = 0; k < kGeomPerLane; ++k)
    if (shapes[k]) {
      const double x = px[k], y = py[k], z = pz[k];
      r2 = fmax(r2, (x - cx) * (x - cx) + (y - cy) * (y - cy) + (z - cz) * (z - cz));
    }
  // (non-negative: ordered as its bits)
  unsigned long long m = (unsigned long long)__double_as_longlong(r2);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  r2 = __longlong_as_double((long long)m);
  // FP32 for the traversal's acceptance test; the 1e-6 margin covers the rounded centre
  if (lane == 0) geom[tile] = make_float4((float)cx, (float)cy, (float)cz, (float)(sqrt(r2) + 1e-6));
}

// Chebyshev points of the second kind t_a = cos(pi a / n) and their barycentric weights.
struct Cheb {
  double t[kMaxNodes1D];
  double w[kMaxNodes1D];
};

Cheb chebFor(int n) {
  Cheb c{};
  for (int a = 0; a <= n; ++a) {
    c.t[a] = std::cos(kPi * a / n);
    c.w[a] = ((a & 1) ? -1.0 : 1.0) * ((a == 0 || a == n) ? 0.5 : 1.0);
  }
  c.t[0] = 1.0;
  c.t[n] = -1.0;
  return c;
}

// Barycentric Lagrange basis at u in [-1, 1] (second form; forward stable at Chebyshev points,
// Higham 2004), in FP32: the proxy charges are stored as floats, and the basis needs no more.
// scale multiplies every value (the source weight for the xi factor, 1 for eta).
__device__ __forceinline__ void basisF(float u, int n, const float* t, const float* w, float scale, float* L) {
  float den = 0.f;
  int hit = -1;
  for (int a = 0; a <= n; ++a) {
    const float d = u - t[a];
    if (d == 0.f) hit = a;
    L[a] = w[a] / d;
    den += L[a];
  }
  if (hit >= 0) {
    for (int a = 0; a <= n; ++a) L[a] = a == hit ? scale : 0.f;
    return;
  }
  const float r = scale / den;
  for (int a = 0; a <= n; ++a) L[a] *= r;
}

// A cluster's chart, from the node geometry for the charges (FP32) and the proxies (FP64).
struct Chart {
  double u[3], e1[3], e2[3];            // centre direction and tangent frame
  double mx, my, hx, hy;                // chart rectangle: middle and half widths
  float uh[3], ul[3], f1[3], f2[3];     // the centre direction in hi / lo parts, the frame
  float fmx, fmy, fihx, fihy;           // middle and reciprocal half widths
};

// The charges are summed in chunks of kUpThreads sources.  Chunk c of node g has the scratch slot
// slotOf(level base, its first point, its index in the level) + c: unique, because the nodes of a level
// follow each other in point order, and a node's chunks are at most its points / kUpThreads + 1.
constexpr int kMaxTreeLevels = kOctreeMaxDepth + 1;
struct ChunkSlots {
  int nodeBase[kMaxTreeLevels + 1];  // first node of each level; total past the last
  int slotBase[kMaxTreeLevels];      // first slot of each level
  int depth;
};
__device__ __forceinline__ int slotOf(const ChunkSlots& cs, int g, int firstPoint) {
  int lev = 0;
  while (lev < cs.depth && g >= cs.nodeBase[lev + 1]) ++lev;
  return cs.slotBase[lev] + firstPoint / kUpThreads + (g - cs.nodeBase[lev]);
}

// Upward pass in three kernels.  One CTA per node summed everything before: the largest nodes of level
// 2 (some 12,000 of 327,680 sources, 94 chunks one after the other) took the whole pass's time, 254 us
// per level-7 evaluation, while the GPU was idle; now 112 us, with the same sums in the same order.
//
// 1. One CTA per octree node: centre and radius of the node's sources; for nodes with more than
// (n+1)^2 sources all within ~37 degrees of the centre direction, the gnomonic chart.
__global__ void __launch_bounds__(kUpThreads) nodeGeometry(const int2* __restrict__ ptInds, int degree, int firstNode,
                                                           const ChunkSlots cs, const float4* __restrict__ sp0,
                                                           float4* __restrict__ geom, int* __restrict__ approx,
                                                           Chart* __restrict__ charts, int* __restrict__ owner) {
  __shared__ float shf[kUpThreads / 32];
  const int g = blockIdx.x;
  const int2 pt = ptInds[g];
  const int n1 = degree + 1, P = n1 * n1;
  if (pt.y == 0 || g < firstNode) {
    // empty; or the root and the octants, whose sources span more than any chart allows (their
    // geometry would only ever open them, so they are opened unconditionally: infinite radius)
    if (threadIdx.x == 0) { geom[g] = make_float4(0.f, 0.f, 0.f, pt.y == 0 ? -1.f : INFINITY); approx[g] = 0; }
    return;
  }
  const int k0 = pt.x, k1 = pt.x + pt.y;
  // Every per-source loop reads the sources' FP32 hi/lo records (sp0/sp1, key order), not their
  // FP64 positions: FP64 runs at 1/64 of the FP32 rate on GB300, and with FP64 sums, differences
  // and conversions per source this pass was FP64-pipe bound.  The centroid only has to lie near
  // the cluster (the radius and chart extents are measured from it); each thread sums its hi
  // parts in FP32, the block in FP64.
  float fsx = 0.f, fsy = 0.f, fsz = 0.f;
#pragma unroll 8
  for (int k = k0 + threadIdx.x; k < k1; k += kUpThreads) {
    const float4 a = sp0[k];
    fsx += a.x; fsy += a.y; fsz += a.z;
  }
  const float tsx = blockSumF<kUpThreads>(fsx, shf);
  const float tsy = blockSumF<kUpThreads>(fsy, shf);
  const float tsz = blockSumF<kUpThreads>(fsz, shf);
  // centre and chart frame, c^ and two tangent directions: FP64, so by one warp
  __shared__ double sU[3], sE1[3], sE2[3], sC[3];
  __shared__ bool sCand;
  if (threadIdx.x < 32) {
    const double sx = tsx, sy = tsy, sz = tsz;
    const double cx = sx / pt.y, cy = sy / pt.y, cz = sz / pt.y;
    const double cn = sqrt(cx * cx + cy * cy + cz * cz);
    const bool cand = pt.y > P && cn > 1e-3;
    double ux = 0, uy = 0, uz = 1, e1x = 1, e1y = 0, e1z = 0, e2x = 0, e2y = 1, e2z = 0;
    if (cand) {
      ux = cx / cn; uy = cy / cn; uz = cz / cn;
      const double ax = fabs(ux) < 0.9 ? 1.0 : 0.0, ay = 1.0 - ax;  // a = x^ or y^
      e1x = uy * 0.0 - uz * ay; e1y = uz * ax - ux * 0.0; e1z = ux * ay - uy * ax;  // c^ x a
      const double e1n = sqrt(e1x * e1x + e1y * e1y + e1z * e1z);
      e1x /= e1n; e1y /= e1n; e1z /= e1n;
      e2x = uy * e1z - uz * e1y; e2y = uz * e1x - ux * e1z; e2z = ux * e1y - uy * e1x;
    }
    if (threadIdx.x == 0) {
      sCand = cand;
      sC[0] = cx; sC[1] = cy; sC[2] = cz;
      sU[0] = ux; sU[1] = uy; sU[2] = uz;
      sE1[0] = e1x; sE1[1] = e1y; sE1[2] = e1z;
      sE2[0] = e2x; sE2[1] = e2y; sE2[2] = e2z;
    }
  }
  __syncthreads();
  const bool cand = sCand;
  // Radius, chart test and chart extents in FP32 (FP64 runs at 1/64 of the FP32 rate): the radius
  // only enters the acceptance test and the extents only bound the interpolation interval, so
  // ~1e-7 absolute errors are absorbed by the margins below.
  const float fcx = (float)sC[0], fcy = (float)sC[1], fcz = (float)sC[2];
  const float fux = (float)sU[0], fuy = (float)sU[1], fuz = (float)sU[2];
  const float f1x = (float)sE1[0], f1y = (float)sE1[1], f1z = (float)sE1[2];
  const float f2x = (float)sE2[0], f2y = (float)sE2[1], f2z = (float)sE2[2];
  float r2 = 0.f, dmin = FLT_MAX, xmin = FLT_MAX, xmax = -FLT_MAX, ymin = FLT_MAX, ymax = -FLT_MAX;
#pragma unroll 4
  for (int k = k0 + threadIdx.x; k < k1; k += kUpThreads) {
    const float4 a = sp0[k];
    const float x = a.x, y = a.y, z = a.z;  // hi parts: within 6e-8 of the position
    r2 = fmaxf(r2, (x - fcx) * (x - fcx) + (y - fcy) * (y - fcy) + (z - fcz) * (z - fcz));
    if (cand) {
      const float d = x * fux + y * fuy + z * fuz;
      dmin = fminf(dmin, d);
      if (d > 0.f) {
        const float rd = __frcp_rn(d);
        const float xi = (x * f1x + y * f1y + z * f1z) * rd, eta = (x * f2x + y * f2y + z * f2z) * rd;
        xmin = fminf(xmin, xi); xmax = fmaxf(xmax, xi); ymin = fminf(ymin, eta); ymax = fmaxf(ymax, eta);
      }
    }
  }
  const float tr2 = blockMaxF<kUpThreads>(r2, shf);
  const float tdmin = -blockMaxF<kUpThreads>(-dmin, shf);
  const float txlo = -blockMaxF<kUpThreads>(-xmin, shf), txhi = blockMaxF<kUpThreads>(xmax, shf);
  const float tylo = -blockMaxF<kUpThreads>(-ymin, shf), tyhi = blockMaxF<kUpThreads>(ymax, shf);
  if (threadIdx.x >= 32) return;
  const double rad = sqrt((double)tr2) + 1e-6;  // covers the FP32 rounding
  const bool valid = cand && (double)tdmin >= kMinChartCos && txhi > txlo && tyhi > tylo;
  if (threadIdx.x == 0) {
    geom[g] = make_float4(fcx, fcy, fcz, (float)rad);  // rad's 1e-6 margin covers the rounding
    approx[g] = valid ? 1 : 0;
  }
  if (!valid) return;
  // widen the rectangle by the FP32 error of the extents (|xi|, |eta| <= 0.75 on a valid chart)
  constexpr double kPad = 1e-6;
  const double xlo = (double)txlo - kPad, xhi = (double)txhi + kPad, ylo = (double)tylo - kPad, yhi = (double)tyhi + kPad;
  const double mx = 0.5 * (xlo + xhi), hx = 0.5 * (xhi - xlo);
  const double my = 0.5 * (ylo + yhi), hy = 0.5 * (yhi - ylo);
  if (threadIdx.x == 0) {
    Chart& C = charts[g];
    for (int c = 0; c < 3; ++c) {
      C.u[c] = sU[c]; C.e1[c] = sE1[c]; C.e2[c] = sE2[c];
      C.uh[c] = (float)sU[c];
      C.ul[c] = (float)(sU[c] - (double)(float)sU[c]);
      C.f1[c] = (float)sE1[c];
      C.f2[c] = (float)sE2[c];
    }
    C.mx = mx; C.my = my; C.hx = hx; C.hy = hy;
    C.fmx = (float)mx; C.fmy = (float)my; C.fihx = (float)(1.0 / hx); C.fihy = (float)(1.0 / hy);
  }
  const int slot = slotOf(cs, g, k0);
  for (int c = threadIdx.x; c < (pt.y + kUpThreads - 1) / kUpThreads; c += 32) owner[slot + c] = g;
}

// 2. One CTA per chunk of a node's sources: its FP32 basis values and, one thread per proxy, the
// chunk's charges sum_j w_j L_a(xi_j) L_b(eta_j), sources in index order.
__global__ void __launch_bounds__(kUpThreads) nodeCharges(const int2* __restrict__ ptInds, int degree, const Cheb C,
                                                          const ChunkSlots cs, const float4* __restrict__ sp0,
                                                          const float4* __restrict__ sp1,
                                                          const Chart* __restrict__ charts,
                                                          const int* __restrict__ owner, float* __restrict__ sums) {
  __shared__ float sL[kUpThreads][2 * kMaxNodes1D];
  __shared__ float sT[kMaxNodes1D], sBw[kMaxNodes1D];
  const int g = owner[blockIdx.x];
  if (g < 0) return;
  if (threadIdx.x <= degree) {
    sT[threadIdx.x] = (float)C.t[threadIdx.x];
    sBw[threadIdx.x] = (float)C.w[threadIdx.x];
  }
  const int2 pt = ptInds[g];
  const int n1 = degree + 1, P = n1 * n1, t = threadIdx.x;
  const int c0 = pt.x + ((int)blockIdx.x - slotOf(cs, g, pt.x)) * kUpThreads, k1 = pt.x + pt.y;
  __syncthreads();
  const int k = c0 + t;
  if (k < k1) {
    // chart coordinates from the offset d = x - c^: x.c^ = 1 + d.c^ and x.e = d.e for the
    // tangent directions, so every FP32 product is of the offset's size and the coordinates
    // carry ~1e-7 of it, not of |x|.  d from hi/lo parts: the hi difference is exact when the
    // coordinates are within a factor 2 (a cluster within ~37 degrees of c^), the lo parts
    // add the rest.
    const Chart& H = charts[g];
    const float fux = H.uh[0], fuy = H.uh[1], fuz = H.uh[2];
    const float4 a = sp0[k], b = sp1[k];
    const float dx = (a.x - fux) + (b.x - H.ul[0]), dy = (a.y - fuy) + (b.y - H.ul[1]), dz = (a.z - fuz) + (b.z - H.ul[2]);
    const float rd = __frcp_rn(1.f + (dx * fux + dy * fuy + dz * fuz));
    const float uxi = ((dx * H.f1[0] + dy * H.f1[1] + dz * H.f1[2]) * rd - H.fmx) * H.fihx;
    const float ueta = ((dx * H.f2[0] + dy * H.f2[1] + dz * H.f2[2]) * rd - H.fmy) * H.fihy;
    basisF(uxi, degree, sT, sBw, a.w, &sL[t][0]);  // w L_a(xi): one FMA per proxy below
    basisF(ueta, degree, sT, sBw, 1.f, &sL[t][n1]);
  }
  __syncthreads();
  if (t < P) {  // Kahan-compensated FP32 over the chunk (the FP32 pipe; FP64 is 1/64 of it)
    const int ia = t / n1, ib = t % n1;
    const int m = min(kUpThreads, k1 - c0);
    float h = 0.f, c = 0.f;
#pragma unroll 8
    for (int j = 0; j < m; ++j) {
      const float y = sL[j][ia] * sL[j][n1 + ib] - c;
      const float tt = h + y;
      c = (tt - h) - y;
      h = tt;
    }
    sums[(size_t)blockIdx.x * P + t] = h - c;
  }
}

// 3. One CTA per node with a chart: its charges Q_ab, the chunks' sums added with compensation in order
// (one thread per proxy), and the proxy records at sp0/sp1[ns + g (n+1)^2 + ab].
__global__ void __launch_bounds__(kUpThreads) nodeProxies(const int2* __restrict__ ptInds, int degree, const Cheb C,
                                                          const ChunkSlots cs, int ns, const int* __restrict__ approx,
                                                          const Chart* __restrict__ charts,
                                                          const float* __restrict__ sums, float4* __restrict__ sp0,
                                                          float4* __restrict__ sp1) {
  const int g = blockIdx.x;
  const int n1 = degree + 1, P = n1 * n1, t = threadIdx.x;
  if (t >= P || !approx[g]) return;
  const int2 pt = ptInds[g];
  const int chunks = (pt.y + kUpThreads - 1) / kUpThreads;
  const float* q0 = sums + (size_t)slotOf(cs, g, pt.x) * P + t;
  float qh = 0.f, qc = 0.f;
#pragma unroll 8
  for (int c = 0; c < chunks; ++c) kahanAddF(qh, qc, q0[(size_t)c * P]);
  const int ia = t / n1, ib = t % n1;
  const Chart& H = charts[g];
  const double q = (double)qh - (double)qc;
  const double xi = H.mx + H.hx * C.t[ia], eta = H.my + H.hy * C.t[ib];
  double px = H.u[0] + xi * H.e1[0] + eta * H.e2[0], py = H.u[1] + xi * H.e1[1] + eta * H.e2[1],
         pz = H.u[2] + xi * H.e1[2] + eta * H.e2[2];
  const double ip = 1.0 / sqrt(px * px + py * py + pz * pz);
  px *= ip; py *= ip; pz *= ip;
  const float hx0 = __double2float_rn(px), hy0 = __double2float_rn(py), hz0 = __double2float_rn(pz);
  const int slot = ns + g * P + t;
  sp0[slot] = make_float4(hx0, hy0, hz0, __double2float_rn(q));
  sp1[slot] = make_float4(__double2float_rn(px - (double)hx0), __double2float_rn(py - (double)hy0),
                          __double2float_rn(pz - (double)hz0), __double2float_rn(1.0 - (px * px + py * py + pz * pz)));
}

struct Levels {
  int base[kOctreeMaxDepth + 2];
};

// An evaluation's flags and whole-number statistics on the device, zeroed before it.
struct TreeFlags {
  int overflow, stackErr;
  int counter, pad;  // the pair kernel's work counter
  unsigned long long pairs, farPairs, farLen;
  long long total;
};

constexpr int kWarpStack = 4096;  // per-warp node stack: <= 256 entries per level for depth <= 10

// Interaction lists, one warp per target tile, the tree walked 32 nodes at a time: each step
// pops up to 32 stacked nodes (one per lane), tests them, places their kids on the stack and
// their list entries in lane order (warp prefix sums), and writes each entry's index range with
// the whole warp.  The order is a function of the data alone, so the lists are reproducible.
// FILL = false: list length and far-field length per tile; FILL = true: the flattened index
// list at listOff[tile], contiguous direct ranges merged.  A stack overflow (impossible for the
// depths the tree code builds) sets *err instead of writing out of bounds.
template <bool FILL>
__global__ void __launch_bounds__(32) traverse(const float4* __restrict__ tileGeom, int ntiles,
                                               const float4* __restrict__ geom, const int* __restrict__ approx,
                                               const int2* __restrict__ ptInds, const int* __restrict__ kids,
                                               Levels lv, int depth, float theta2, int P, int ns,
                                               const int2* __restrict__ tiles, int64_t* __restrict__ lens,
                                               int64_t* __restrict__ listOff, int* __restrict__ list,
                                               TreeFlags* __restrict__ flags) {
  __shared__ int stack[kWarpStack];
  const int tile = blockIdx.x;
  const int lane = threadIdx.x;
  if (tile >= ntiles) return;
  if (FILL && flags->overflow) {
    // the lists do not fit their buffer: every tile's list becomes the identity list of all sorted
    // sources, the exact direct sum (the buffer holds at least ns), written by all tiles' warps
    if (lane == 0) { listOff[tile] = 0; lens[tile] = ns; }
    for (int64_t i = (int64_t)tile * 32 + lane; i < ns; i += (int64_t)ntiles * 32) list[i] = (int)i;
    return;
  }
  const float4 tg = tileGeom[tile];
  if (lane == 0) stack[0] = 0;  // the root (level 0, global index 0)
  __syncwarp();
  int sp = 1;
  int64_t len = 0, far = 0;
  int64_t o = FILL ? listOff[tile] : 0;
  int rs = 0, rl = 0;  // pending direct range (FILL)
  while (sp > 0) {
    const int n = min(32, sp);
    const int b0 = sp - n;
    const int g = lane < n ? stack[b0 + lane] : -1;
    __syncwarp();
    sp = b0;
    int kind = 0;  // 0 nothing, 1 far, 2 direct, 3 open
    int2 pt = make_int2(0, 0);
    int lev = 0;
    if (g >= 0) {
      pt = ptInds[g];
      if (pt.y > 0) {
        // (r_tile + r_node) < theta |c_tile - c_node|, squared and in FP32 (FP64 runs at 1/64
        // of the FP32 rate; the radii carry 1e-6 margins); an infinite radius never passes
        const float4 ng = geom[g];
        const float dx = tg.x - ng.x, dy = tg.y - ng.y, dz = tg.z - ng.z;
        const float rr = tg.w + ng.w;
        const bool mac = rr * rr < theta2 * (dx * dx + dy * dy + dz * dz);
        while (lev < depth && g >= lv.base[lev + 1]) ++lev;
        if (mac && approx[g]) kind = 1;
        else if (mac && pt.y <= P) kind = 2;      // well separated but smaller than its proxy set
        else if (lev < depth) kind = 3;           // too close, or no valid chart: open the node
        else kind = 2;                            // a leaf
      }
    }
    // kids of opened nodes onto the stack (lane order, ascending child order)
    int nk = 0, kidv[8];
    if (kind == 3)
      for (int c = 0; c < 8; ++c) {
        const int k = kids[8 * g + c];
        if (k >= 0) kidv[nk++] = lv.base[lev + 1] + k;
      }
    int incl = nk;
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += v;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    if (sp + total > kWarpStack) {  // cannot happen for depth <= 10; never write out of bounds
      if (lane == 0) atomicExch(&flags->stackErr, 1);
      break;
    }
    for (int c = 0; c < nk; ++c) stack[sp + incl - nk + c] = kidv[c];
    sp += total;
    __syncwarp();
    // list entries in lane order
    const unsigned emit = __ballot_sync(0xffffffffu, kind == 1 || kind == 2);
    unsigned m = emit;
    while (m) {
      const int src = __ffs(m) - 1;
      m &= m - 1;
      const int kd = __shfl_sync(0xffffffffu, kind, src);
      const int st = __shfl_sync(0xffffffffu, pt.x, src);
      const int ct = __shfl_sync(0xffffffffu, pt.y, src);
      const int gg = __shfl_sync(0xffffffffu, g, src);
      if (kd == 1) {
        len += P;
        far += P;
        if (FILL) {
          for (int k = lane; k < rl; k += 32) list[o + k] = rs + k;
          o += rl;
          rl = 0;
          const int p0 = ns + gg * P;
          for (int k = lane; k < P; k += 32) list[o + k] = p0 + k;
          o += P;
        }
      } else {
        len += ct;
        if (FILL) {
          if (rl > 0 && rs + rl == st) {
            rl += ct;
          } else {
            for (int k = lane; k < rl; k += 32) list[o + k] = rs + k;
            o += rl;
            rs = st;
            rl = ct;
          }
        }
      }
    }
  }
  if (FILL) {
    for (int k = lane; k < rl; k += 32) list[o + k] = rs + k;
  } else if (lane == 0) {
    lens[tile] = len;
    // statistics: whole numbers, so the order of the additions does not matter
    const unsigned long long tc = (unsigned long long)tiles[tile].y;
    atomicAdd(&flags->pairs, tc * (unsigned long long)len);
    atomicAdd(&flags->farPairs, tc * (unsigned long long)far);
    atomicAdd(&flags->farLen, (unsigned long long)far);
  }
}

// Between the two traversals, one CTA: the lists' offsets (their exclusive sums) and total, whether they
// fit the buffer (cap entries), the report to the host, and the work items (each tile's list in
// nchunks parts), longest lists first to 1/kLenBuckets of the longest: the order only shapes the
// schedule.  One launch in the place of a scan, an eight-pass sort and six small kernels (105 us
// per level-7 evaluation, now 18 us).
constexpr int kPlanThreads = 1024;
constexpr int kLenBuckets = 512;

__global__ void __launch_bounds__(kPlanThreads) planLists(const int64_t* __restrict__ lens, int ntiles, int nchunks,
                                                          int64_t cap, int64_t* __restrict__ off,
                                                          int* __restrict__ order, TreeFlags* __restrict__ flags,
                                                          TreeWatch* __restrict__ w) {
  using Scan = cub::BlockScan<long long, kPlanThreads>;
  using Reduce = cub::BlockReduce<long long, kPlanThreads>;
  using Scan32 = cub::BlockScan<int, kPlanThreads>;
  __shared__ union {
    typename Scan::TempStorage scan;
    typename Reduce::TempStorage reduce;
    typename Scan32::TempStorage scan32;
  } sh;
  __shared__ long long sMax;
  __shared__ int sBucket[kLenBuckets];
  const int t = threadIdx.x;
  const int per = (ntiles + kPlanThreads - 1) / kPlanThreads, t0 = min(ntiles, t * per), t1 = min(ntiles, t0 + per);
  long long sum = 0, mx = 0;
  for (int i = t0; i < t1; ++i) {
    const long long l = lens[i];
    sum += l;
    mx = max(mx, l);
  }
  long long at = 0, total = 0;
  Scan(sh.scan).ExclusiveSum(sum, at, total);
  __syncthreads();
  mx = Reduce(sh.reduce).Reduce(mx, [](long long a, long long b) { return a > b ? a : b; });
  if (t == 0) {
    sMax = mx;
    flags->total = total;
    flags->overflow = total > cap ? 1 : 0;
    if (w) {  // mapped host memory, read without a synchronisation before a later evaluation
      if (total > w->maxTotal) w->maxTotal = total;
      if (total > cap) w->overflow = 1;
      if (flags->stackErr) w->stackErr = 1;
    }
  }
  if (t < kLenBuckets) sBucket[t] = 0;
  __syncthreads();
  const float scale = (float)kLenBuckets / ((float)sMax + 1.f);
  auto bucketOf = [&](long long l) { return kLenBuckets - 1 - min(kLenBuckets - 1, (int)((float)l * scale)); };
  for (int i = t0; i < t1; ++i) {
    const long long l = lens[i];
    off[i] = at;
    at += l;
    atomicAdd(&sBucket[bucketOf(l)], 1);
  }
  __syncthreads();
  int first = 0;
  Scan32(sh.scan32).ExclusiveSum(t < kLenBuckets ? sBucket[t] : 0, first);
  __syncthreads();
  if (t < kLenBuckets) sBucket[t] = first;
  __syncthreads();
  for (int i = t0; i < t1; ++i) {
    const int p = atomicAdd(&sBucket[bucketOf(lens[i])], 1);
    for (int c = 0; c < nchunks; ++c) order[(size_t)p * nchunks + c] = i * nchunks + c;
  }
}

inline unsigned blocks(int64_t n, int b = kBlock) { return (unsigned)((n + b - 1) / b); }

void ck(cudaError_t e, const char* what) {
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    fail(e == cudaErrorMemoryAllocation ? LPM_ERR_OUT_OF_MEMORY : LPM_ERR_CUDA, "tree code %s: %s", what,
         cudaGetErrorString(e));
  }
}

}  // namespace

int treeDepthFor(int64_t n, int leafPoints) {
  int d = 1;
  while (d < kOctreeMaxDepth && 4.7 * std::pow(4.0, d) * std::max(1, leafPoints) < (double)n) ++d;
  return d;
}

template <typename T>
T* TreeEval::grow(Buf& b, size_t count, cudaStream_t s) {
  const size_t bytes = std::max<size_t>(1, count) * sizeof(T);
  if (b.bytes < bytes) {
    if (b.p) ck(cudaFreeAsync(b.p, s), "free");
    b.p = nullptr;
    b.bytes = 0;
    const size_t want = bytes + bytes / 4;
    ck(cudaMallocAsync(&b.p, want, s), "allocation");
    b.bytes = want;
  }
  return static_cast<T*>(b.p);
}

// Report slots in mapped host memory, allocated in blocks and recycled: freeing mapped memory
// would synchronise the device, and a slot may still be written by kernels in flight when its
// evaluator goes away.  A slot returns to the pool only once the work queued before its release
// has completed (a host function on that stream) or after a device synchronisation.
class WatchPool {
 public:
  static WatchPool& get() {
    static WatchPool* p = new WatchPool();  // lives as long as the process (host functions may run late)
    return *p;
  }
  void take(TreeWatch** host, TreeWatch** dev) {
    std::lock_guard<std::mutex> lk(mu_);
    if (free_.empty()) {
      constexpr int kBlock = 64;
      void* h = nullptr;
      ck(cudaHostAlloc(&h, sizeof(TreeWatch) * kBlock, cudaHostAllocMapped | cudaHostAllocPortable),
         "host allocation");
      void* d = nullptr;
      ck(cudaHostGetDevicePointer(&d, h, 0), "mapped pointer");
      for (int i = kBlock - 1; i >= 0; --i)
        free_.emplace_back(static_cast<TreeWatch*>(h) + i, static_cast<TreeWatch*>(d) + i);
    }
    *host = free_.back().first;
    *dev = free_.back().second;
    free_.pop_back();
    std::memset(*host, 0, sizeof(TreeWatch));
  }
  void give(TreeWatch* host, TreeWatch* dev) {
    std::lock_guard<std::mutex> lk(mu_);
    free_.emplace_back(host, dev);
  }
  struct Pending {
    TreeWatch* host;
    TreeWatch* dev;
  };
  static void CUDART_CB giveLater(void* p) {  // host function: no CUDA calls
    Pending* q = static_cast<Pending*>(p);
    get().give(q->host, q->dev);
    delete q;
  }

 private:
  std::mutex mu_;
  std::vector<std::pair<TreeWatch*, TreeWatch*>> free_;
};

TreeEval::~TreeEval() {
  bool held = false;
  for (Buf* b : all_) held = held || b->p;
  if (held) {  // not released in stream order: wait for the device, then free
    cudaDeviceSynchronize();
    for (Buf* b : all_)
      if (b->p) cudaFree(b->p);
  }
  if (watch_) WatchPool::get().give(watch_, dWatch_);
}

void TreeEval::release(cudaStream_t s) {
  for (Buf* b : all_) {
    if (b->p) ck(cudaFreeAsync(b->p, s), "free");
    b->p = nullptr;
    b->bytes = 0;
  }
  tree_.release(s);
  if (watch_) {
    auto* q = new WatchPool::Pending{watch_, dWatch_};
    const cudaError_t e = cudaLaunchHostFunc(s, WatchPool::giveLater, q);
    if (e != cudaSuccess) {
      delete q;  // the slot is dropped, not reused
      ck(e, "host function");
    }
    watch_ = nullptr;
    dWatch_ = nullptr;
  }
  partial_ = nullptr;
  listCap_ = 0;
  devAt_ = nullptr;
  hDev_ = TreeDev{};
  statsOnDevice_ = false;
  ++generation_;
}

void TreeEval::ensureWatch() {
  if (watch_) return;
  WatchPool::get().take(&watch_, &dWatch_);
}

bool TreeEval::poll() {
  if (!watch_) return false;
  volatile TreeWatch* w = watch_;
  if (w->stackErr) {
    w->stackErr = 0;
    fail(LPM_ERR_INTERNAL, "tree code: traversal stack overflow (octree depth %d)", tree_.depth);
  }
  if (!w->overflow) return false;
  // an evaluation since the last poll did not fit its lists (it summed every source instead):
  // room for the largest total seen, with headroom, from the next evaluation on
  listCap_ = std::max<int64_t>(listCap_, (int64_t)(1.25 * (double)w->maxTotal) + 4096);
  w->overflow = 0;
  ++generation_;
  return true;
}

const TreeStats& TreeEval::stats() {
  if (statsOnDevice_) {
    TreeFlags f{};
    int cnt[kOctreeMaxDepth + 1] = {};
    ck(cudaDeviceSynchronize(), "synchronise");
    ck(cudaMemcpy(&f, bFlags.p, sizeof(f), cudaMemcpyDeviceToHost), "read-back");
    if (hDev_.ns > 0)
      ck(cudaMemcpy(cnt, tree_.dcount, sizeof(int) * (size_t)(tree_.depth + 1), cudaMemcpyDeviceToHost), "read-back");
    // with overflowing lists every tile took every source
    stats_.pairs = f.overflow ? (double)hDev_.nslots * hDev_.ns : (double)f.pairs;
    stats_.farPairs = f.overflow ? 0.0 : (double)f.farPairs;
    stats_.directPairs = stats_.pairs - stats_.farPairs;
    stats_.farClusters = f.overflow ? 0 : (int64_t)(f.farLen / (unsigned long long)statsP_);
    stats_.nodes = 0;
    for (int c : cnt) stats_.nodes += c;
  }
  return stats_;
}

void TreeEval::evaluate(SolvePlan& Pl, const TreeParams& tp, const PairShape& shape, bool psi, bool precise,
                        bool rcpApprox, int slots, int grid, PairTimer* timer, cudaStream_t s) {
  if (tp.degree < 2 || tp.degree > kMaxDegree) fail(LPM_ERR_INVALID_ARGUMENT, "tree code: degree must be 2..%d", kMaxDegree);
  if (!(tp.theta > 0.0 && tp.theta < 1.0)) fail(LPM_ERR_INVALID_ARGUMENT, "tree code: theta must be in (0, 1)");
  if (!treePairShapeSupported(shape)) fail(LPM_ERR_NOT_SUPPORTED, "tree code: plan built for another launch shape");
  const int ns = Pl.ns, nslots = Pl.nslots, ntiles = Pl.nTreeTiles;
  const int P = (tp.degree + 1) * (tp.degree + 1);
  ensureWatch();
  // reports of earlier evaluations (no synchronisation); never while the stream is captured, where
  // a report arriving now would make the capture grow a buffer (callers poll before capturing)
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  ck(cudaStreamIsCapturing(s, &cap), "capture status");
  if (cap == cudaStreamCaptureStatusNone) poll();
  direct_ = false;
  stats_ = TreeStats{};
  statsOnDevice_ = true;
  // phase timing (with the context's timer): events at the phase boundaries, read at the end
  cudaEvent_t ev[5] = {};
  if (timer)
    for (auto& e : ev) e = timer->get();
  auto mark = [&](int i) {
    if (timer) ck(cudaEventRecord(ev[i], s), "event");
  };
  mark(0);

  const int* selfSorted = nullptr;
  int* tslot = nullptr;
  int nnodes = 0;
  float4* tsp0 = nullptr;
  float4* tsp1 = nullptr;
  float4* geom = nullptr;
  int* approx = nullptr;
  int depth = 0;
  if (ns > 0) {
    // 1-3. octree over the stage positions (fixed-level layout, counts on the device), sources in
    // key order
    depth = treeDepthFor(ns, tp.leafPoints);
    tree_.buildOnDevice(Octree::Points{nullptr, 0, 0, Pl.stage.sp0, Pl.stage.sp1}, ns, depth, false, s);
    mark(1);
    nnodes = (int)tree_.nnodes;  // capacity: nodes past a level's count are empty
    stats_.depth = depth;
    const size_t nrec = (size_t)ns + (size_t)nnodes * P;
    tsp0 = grow<float4>(bSp0, nrec, s);
    tsp1 = grow<float4>(bSp1, nrec, s);
    int* inv = grow<int>(bInv, ns, s);
    tslot = grow<int>(bSlot, ns, s);
    gatherSources<<<blocks(ns), kBlock, 0, s>>>(tree_.origIds, Pl.stage.sp0, Pl.stage.sp1, Pl.stage.srcSlot, ns, tsp0,
                                                tsp1, inv, tslot);
    int* ss = grow<int>(bSelf, nslots, s);
    sortedSelf<<<blocks(nslots), kBlock, 0, s>>>(Pl.dev.self, inv, nslots, ss);
    selfSorted = ss;
    // 4. upward pass (empty nodes return at once)
    geom = grow<float4>(bGeom, nnodes, s);
    approx = grow<int>(bApprox, nnodes, s);
    const int firstNode = depth >= 2 ? tree_.base[2] : nnodes;
    const Cheb cheb = chebFor(tp.degree);
    ChunkSlots cs{};
    cs.depth = depth;
    int nslotsUp = 0;
    for (int l = 0; l <= depth + 1; ++l) cs.nodeBase[l] = l <= depth ? tree_.base[l] : nnodes;
    for (int l = 0; l <= depth; ++l) {
      cs.slotBase[l] = nslotsUp;
      if (l >= 2) nslotsUp += ns / kUpThreads + 1 + cs.nodeBase[l + 1] - cs.nodeBase[l];
    }
    Chart* charts = grow<Chart>(bCharts, nnodes, s);
    int* owner = grow<int>(bOwner, nslotsUp, s);
    float* sums = grow<float>(bSums, (size_t)std::max(1, nslotsUp) * P, s);
    ck(cudaMemsetAsync(owner, 0xff, sizeof(int) * (size_t)std::max(1, nslotsUp), s), "memset");
    nodeGeometry<<<nnodes, kUpThreads, 0, s>>>(tree_.ptInds, tp.degree, firstNode, cs, tsp0, geom, approx, charts, owner);
    if (nslotsUp > 0) {
      nodeCharges<<<nslotsUp, kUpThreads, 0, s>>>(tree_.ptInds, tp.degree, cheb, cs, tsp0, tsp1, charts, owner, sums);
      nodeProxies<<<nnodes, kUpThreads, 0, s>>>(tree_.ptInds, tp.degree, cheb, cs, ns, approx, charts, sums, tsp0, tsp1);
    }
    mark(2);
  } else {
    mark(1);
    mark(2);
    int* ss = grow<int>(bSelf, nslots, s);
    ck(cudaMemsetAsync(ss, 0xff, sizeof(int) * (size_t)nslots, s), "memset");  // -1: no sources
    selfSorted = ss;
    tsp0 = grow<float4>(bSp0, 1, s);
    tsp1 = grow<float4>(bSp1, 1, s);
    tslot = grow<int>(bSlot, 1, s);
  }
  // 5. tiles
  float4* tgeom = grow<float4>(bTileGeom, ntiles, s);
  const float theta2 = (float)(tp.theta * tp.theta);
  tileGeometry<<<(ntiles + kGeomTilesPerBlock - 1) / kGeomTilesPerBlock, kBlock, 0, s>>>(
      Pl.stage.tx, nslots, Pl.treeTiles, ntiles, Pl.stage.perm, Pl.io.na, Pl.mask, tgeom);
  // 6. interaction lists: lengths, offsets (a device scan), the work order (a device sort) and
  // the indices -- nothing read back but the very first total, which sizes the list buffer
  int64_t* lens = grow<int64_t>(bLen, ntiles, s);
  Levels lv{};
  for (int l = 0; l <= tree_.depth; ++l) lv.base[l] = tree_.base[l];
  lv.base[tree_.depth + 1] = nnodes;
  TreeFlags* flags = grow<TreeFlags>(bFlags, 1, s);
  ck(cudaMemsetAsync(flags, 0, sizeof(TreeFlags), s), "memset");
  if (ns > 0)
    traverse<false><<<ntiles, 32, 0, s>>>(tgeom, ntiles, geom, approx, tree_.ptInds, tree_.kids, lv, tree_.depth,
                                          theta2, P, ns, Pl.treeTiles, lens, nullptr, nullptr, flags);
  else
    ck(cudaMemsetAsync(lens, 0, sizeof(int64_t) * ntiles, s), "memset");
  mark(3);
  int64_t* off = grow<int64_t>(bOff, ntiles, s);
  // Work items: each tile's list in `nchunks` parts (enough items for ~8 waves of CTAs), each
  // part with its own partial chunk.
  const int nchunks = std::max(1, std::min(16, (8 * std::max(1, slots) + ntiles - 1) / std::max(1, ntiles)));
  const int nitems = ntiles * nchunks;
  int* order = grow<int>(bOrder, nitems, s);
  if (listCap_ == 0) {  // the first evaluation sizes the list buffer (its one synchronisation)
    planLists<<<1, kPlanThreads, 0, s>>>(lens, ntiles, nchunks, 0, off, order, flags, nullptr);
    long long total = 0;
    ck(cudaMemcpyAsync(&total, &flags->total, sizeof(total), cudaMemcpyDeviceToHost, s), "read-back");
    ck(cudaStreamSynchronize(s), "synchronise");
    listCap_ = std::max<int64_t>((int64_t)(1.25 * (double)total) + 4096, ns);  // >= ns: the fallback
    ++generation_;
  }
  int* oldList = static_cast<int*>(bList.p);
  int* list = grow<int>(bList, (size_t)listCap_, s);
  if (list != oldList) ++generation_;
  planLists<<<1, kPlanThreads, 0, s>>>(lens, ntiles, nchunks, listCap_, off, order, flags, dWatch_);
  if (ns > 0)
    traverse<true><<<ntiles, 32, 0, s>>>(tgeom, ntiles, geom, approx, tree_.ptInds, tree_.kids, lv, tree_.depth,
                                         theta2, P, ns, Pl.treeTiles, lens, off, list, flags);
  statsP_ = P;
  mark(4);
  // 7. the gathered pair kernel
  double* partial = grow<double>(bPartial, (size_t)nchunks * 5 * std::max(1, nslots), s);
  TreeDev hd;
  std::memset(&hd, 0, sizeof(hd));  // compared byte for byte with the last upload below
  hd.tx = Pl.stage.tx;
  hd.sp0 = tsp0;
  hd.sp1 = tsp1;
  hd.self = selfSorted;
  hd.tiles = Pl.treeTiles;
  hd.srcSlot = tslot;
  hd.tileCentre = Pl.treeCentres;
  hd.listOff = off;
  hd.list = list;
  hd.order = order;
  hd.partial = partial;
  hd.listLen = lens;
  hd.nslots = nslots;
  hd.ntiles = ntiles;
  hd.nchunks = nchunks;
  hd.ns = ns;
  hd.eps2 = Pl.eps2;
  TreeDev* dd = grow<TreeDev>(bDev, 1, s);
  if (dd != devAt_ || std::memcmp(&hd, &hDev_, sizeof(hd)) != 0) {  // unchanged between evaluations of a plan
    hDev_ = hd;
    devAt_ = dd;
    ck(cudaMemcpyAsync(dd, &hDev_, sizeof(hd), cudaMemcpyHostToDevice, s), "upload");
    ++generation_;
  }
  partial_ = partial;
  nchunks_ = nchunks;
  int* counter = &flags->counter;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (timer) {
    e0 = timer->get();
    e1 = timer->get();
    ck(cudaEventRecord(e0, s), "event");
  }
  ck(launchTreePair(shape, psi, precise, rcpApprox, dd, nitems, counter,
                    std::min(nitems, std::max(1, grid > 0 ? grid : slots)), s),
     "pair launch");
  if (timer) {
    ck(cudaEventRecord(e1, s), "event");
    timer->pending.emplace_back(e0, e1);
    // phases (the traversals end before the pair kernel starts)
    ck(cudaEventSynchronize(ev[4]), "event");
    float a = 0.f, b = 0.f, c = 0.f, d = 0.f;
    ck(cudaEventElapsedTime(&a, ev[0], ev[1]), "event");
    ck(cudaEventElapsedTime(&b, ev[1], ev[2]), "event");
    ck(cudaEventElapsedTime(&c, ev[2], ev[3]), "event");
    ck(cudaEventElapsedTime(&d, ev[3], ev[4]), "event");
    stats_.buildMs = a;
    stats_.upwardMs = b;
    stats_.listMs = c + d;  // tile geometry and count traversal, then offsets, order and the fill
    for (auto& e : ev) timer->pool.push_back(e);
  }
}

}  // namespace lpm

// Periodic ghost images, cell list and ConnectivityMap CSR on the device,
// for every member of a batch in one launch per stage.
//
// Replaces, for one FluidNodeList in a periodic box:
//   PlanarBoundary::setGhostNodes     src/Boundary/PlanarBoundary.cc:114-181
//   PlanarBoundary::updateGhostNodes  src/Boundary/PlanarBoundary.cc:361-395
//   NestedGridNeighbor + Neighbor precull (superset generation only)
//   ConnectivityMap::computeConnectivity src/Neighbor/ConnectivityMap.cc:521-890
//
// Compiled with -fmad=false: the ghost positions and the neighbor predicate
// |H_i r_ij|^2 <= kappa^2 || |H_j r_ij|^2 <= kappa^2 are evaluated in the
// reference's FP64 operation order, so neighbor sets are bit-identical.
//
// The build is sized on the device: the ghost counts, the cell grid, the
// entry count and the longest list are produced by kernels into each member's
// scalar slots and read there by the next kernels; launches are sized for the
// buffer capacities.  The host plans the capacities from the previous build,
// launches every stage, and reads the sizes back once at the end; a capacity
// overflow sets an error bit and the build is redone with larger buffers.
//
// Kernels and their bounds:
//   ghost_cluster                            all ghost passes of a small member
//                                            by one cluster: barrier latency
//   ghost_passes_fused                       ... of a large one by one
//                                            cooperative launch: the same
//   ghost_hmax / ghost_flag / ghost_scatter  O(N+G) streaming, HBM bound
//   node_bounds / cell_index / cell_scatter  O(N+G) streaming + atomics
//   nbr_thread<COUNT|FILL>                   thread per node (cell-sorted
//                                            order) over the 27 neighbouring
//                                            cells; 16-byte candidate records
//                                            shared by a warp through L1
//   nbr_cell<COUNT|FILL>                     block per cell, for large
//                                            candidate sets: the window
//                                            staged and ordered once per cell
//   nbr_crowded<COUNT|FILL>                  ... warp per node of the cells too
//                                            crowded for it
//   nbr_walk<COUNT|FILL>                     warp per node over cells of half
//                                            a reach, for denser sets
#include <cstdio>
#include <cstring>
#include <climits>

#include <cooperative_groups.h>
#include <math_constants.h>

#include "problem.cuh"

namespace sphgpu {

namespace {

constexpr int kGhostThreads = 256;
// blocks per member of the streaming passes (member-local grid stride)
constexpr int64_t kStreamBlocks = 148*4;
constexpr float kFilterTol = 1.0e-3f;
constexpr double kFilterTolPerSpread = 2.0e-5;
// shared memory for the per-thread lists of a 32-thread block (larger lists
// take the warp schedule)
constexpr size_t kMaxListSmem = 200*1024;
// blocks of 256 threads per SM the thread walk is compiled for
#ifndef NBR_THREAD_MIN_BLOCKS
#define NBR_THREAD_MIN_BLOCKS 4
#endif

__device__ __forceinline__ unsigned long long orderedBits(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return (b & 0x8000000000000000ULL) ? ~b : (b | 0x8000000000000000ULL);
}
__device__ __forceinline__ double fromOrderedBits(unsigned long long b) {
  const unsigned long long r = (b & 0x8000000000000000ULL) ? (b & 0x7fffffffffffffffULL) : ~b;
  return __longlong_as_double((long long)r);
}

__device__ __forceinline__ V3 nodePos(const Member& M, int64_t k) {
  const int64_t n = M.n;
  if (k < n) return V3{M.S[S_X*n + k], M.S[S_Y*n + k], M.S[S_Z*n + k]};
  const int64_t g = k - n;
  return V3{M.gpos[g], M.gpos[M.gcap + g], M.gpos[2*M.gcap + g]};
}
__device__ __forceinline__ Sym nodeH(const Member& M, int64_t k) {
  const int64_t n = M.n;
  const int64_t r = k < n ? k : M.groot[k - n];
  const double* S = M.S;
  return Sym{S[(S_H + 0)*n + r], S[(S_H + 1)*n + r], S[(S_H + 2)*n + r],
             S[(S_H + 3)*n + r], S[(S_H + 4)*n + r], S[(S_H + 5)*n + r]};
}

// internal + ghost nodes of the current build
__device__ __forceinline__ int64_t allNodes(const Member& M) { return M.n + scalI(M.scal, SC_G); }

__device__ __forceinline__ Grid loadGrid(const Member& M) {
  const double* s = M.scal + SC_GRID;
  Grid g;
  g.lo[0] = s[0]; g.lo[1] = s[1]; g.lo[2] = s[2];
  g.cell = s[3];
  g.dim[0] = (int)scalI(M.scal, SC_GRID + 4);
  g.dim[1] = (int)scalI(M.scal, SC_GRID + 5);
  g.dim[2] = (int)scalI(M.scal, SC_GRID + 6);
  g.filterTol = (float)s[7];
  g.reach = (float)M.scal[SC_REACH];
  return g;
}

// ---------------------------------------------------------------- ghosts
// Start of a build: no ghosts yet.
__global__ void build_init_kernel(const Member* mem, int nmem) {
  const int m = blockIdx.x*blockDim.x + threadIdx.x;
  if (m >= nmem) return;
  double* s = mem[m].scal;
  setScalI(s, SC_NTOT, mem[m].n);
  setScalI(s, SC_G, 0);
  s[SC_HMAX] = 0.0;
  for (int b = 0; b < 6; ++b) s[SC_PHMAX + b] = 0.0;
  s[SC_LMAXALL] = 0.0;
  unsigned long long* bb = reinterpret_cast<unsigned long long*>(s + SC_BOUNDS);
  for (int a = 0; a < 3; ++a) { bb[a] = ~0ULL; bb[3 + a] = 0ULL; }
  bb[6] = 0ULL;
}

// 1/min(eig(H)) (hmaxi[i]) and max(eig(H)) (hmaxi[n + i]) of every internal
// node, once per build (ghosts share their root's H, so every boundary pass,
// the cell size and the pre-test records read them from here); the bounding
// box of the internal nodes and the largest 1/min(eig(H)) (SC_BOUNDS); the
// largest max(eig(H)) of the problem (with the largest 1/min(eig(H)) it
// bounds the FP32 pre-test error).
// Fixed grid (member-local grid stride): each thread accumulates its nodes'
// bounds, then one set of atomics per block.
__global__ void __launch_bounds__(kGhostThreads) node_hmax_kernel(const Member* mem, BlockMap bm) {
  const MemberBlock mb = memberBlock(bm);
  const Member& M = mem[mb.m];
  double lmax = 0.0, h = 0.0;
  double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
  for (int64_t i = mb.block*(int64_t)blockDim.x + threadIdx.x; i < M.n; i += (int64_t)mb.blocks*blockDim.x) {
    const V3 ev = eigenValues(nodeH(M, i));
    const double hi1 = 1.0/vmin(ev);
    M.hmaxi[i] = hi1;
    h = fmax(h, hi1);
    double l = vmax(ev);
    M.hmaxi[M.n + i] = l;
    if (!(l < 1.0e300)) l = 1.0e300;           // degenerate H: no FP32 pre-test
    lmax = dmax(lmax, l);
    const V3 r = nodePos(M, i);
    lo[0] = fmin(lo[0], r.x); lo[1] = fmin(lo[1], r.y); lo[2] = fmin(lo[2], r.z);
    hi[0] = fmax(hi[0], r.x); hi[1] = fmax(hi[1], r.y); hi[2] = fmax(hi[2], r.z);
  }
  for (int o = 16; o > 0; o >>= 1) {
    lmax = dmax(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
    h = fmax(h, __shfl_xor_sync(0xffffffffu, h, o));
    for (int a = 0; a < 3; ++a) {
      lo[a] = fmin(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
      hi[a] = fmax(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
    }
  }
  __shared__ double sh[kGhostThreads/32][8];
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    for (int a = 0; a < 3; ++a) { sh[w][a] = lo[a]; sh[w][3 + a] = hi[a]; }
    sh[w][6] = h;
    sh[w][7] = lmax;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int ww = 1; ww < (int)(blockDim.x >> 5); ++ww) {
      for (int a = 0; a < 3; ++a) { lo[a] = fmin(lo[a], sh[ww][a]); hi[a] = fmax(hi[a], sh[ww][3 + a]); }
      h = fmax(h, sh[ww][6]);
      lmax = dmax(lmax, sh[ww][7]);
    }
    unsigned long long* out = reinterpret_cast<unsigned long long*>(M.scal + SC_BOUNDS);
    if (h > 0.0) {
      for (int a = 0; a < 3; ++a) {
        atomicMin(out + a, orderedBits(lo[a]));
        atomicMax(out + 3 + a, orderedBits(hi[a]));
      }
      atomicMax(out + 6, orderedBits(h));
    }
    if (lmax > 0.0)
      atomicMax(reinterpret_cast<unsigned long long*>(M.scal + SC_LMAXALL),
                (unsigned long long)__double_as_longlong(lmax));
  }
}

__device__ __forceinline__ double nodeHmax(const Member& M, int64_t k) {
  return M.hmaxi[k < M.n ? k : M.groot[k - M.n]];
}

// Items of a member in a fixed grid: member-local grid stride.
#define FOR_ITEMS(t, count) \
  for (int64_t t = mb.block*(int64_t)blockDim.x + threadIdx.x; t < (count); t += (int64_t)mb.blocks*blockDim.x)

// Internal nodes within kernelExtent*max(1/min(eig(H))) of a periodic plane
// (with a relative margin): the only internal nodes a boundary pass can
// image or count into its hmax.  Flags into counts[0:n].
__global__ void __launch_bounds__(kGhostThreads) near_flag_kernel(const Member* mem, BlockMap bm) {
  const MemberBlock mb = memberBlock(bm);
  const Member& M = mem[mb.m];
  const unsigned long long* bb = reinterpret_cast<const unsigned long long*>(M.scal + SC_BOUNDS);
  const double reach = M.prm.kernelExtent*fromOrderedBits(bb[6])*(1.0 + 1.0e-6);
  FOR_ITEMS(i, M.n) {
    const V3 r = nodePos(M, i);
    int f = 0;
    for (int a = 0; a < 3; ++a) {
      if (!M.prm.bcs.periodic[a]) continue;
      const PlanarBC& bc = M.prm.bcs.bc[2*a];
      if (dmin(minimumDistance(bc.exit, r), minimumDistance(bc.enter, r)) <= reach) f = 1;
    }
    M.counts[i] = f;
  }
}

// The near-plane list, ascending, into cidx[0:nnear] (cidx is free until
// the cell pass), and its length.
__global__ void __launch_bounds__(kGhostThreads) near_list_kernel(const Member* mem, BlockMap bm) {
  const MemberBlock mb = memberBlock(bm);
  const Member& M = mem[mb.m];
  FOR_ITEMS(i, M.n) {
    if (M.counts[i]) M.cidx[M.offsets[i]] = (int32_t)i;
  }
  if (mb.block == 0 && threadIdx.x == 0) setScalI(M.scal, SC_NNEAR, M.offsets[M.n]);
}

// Item t of a boundary pass: the near-plane internal nodes in ascending
// order, then the ghosts made so far in creation order (the order in which
// the reference visits a NodeList's nodes).
__device__ __forceinline__ int64_t passItems(const Member& M) {
  return scalI(M.scal, SC_NNEAR) + scalI(M.scal, SC_NTOT) - M.n;
}
__device__ __forceinline__ int64_t passNode(const Member& M, int64_t t, int64_t nnear) {
  return t < nnear ? (int64_t)M.cidx[t] : M.n + (t - nnear);
}

// hmax of PlanarBoundary::setGhostNodes: max 1/min(eig(H)) over nodes within
// kernelExtent*hmaxi of either plane.
__global__ void __launch_bounds__(kGhostThreads) ghost_hmax_kernel(const Member* mem, BlockMap bm, int b) {
  const MemberBlock mb = memberBlock(bm);
  const Member& M = mem[mb.m];
  double best = 0.0;
  if (M.prm.bcs.periodic[b >> 1]) {
    const PlanarBC& bc = M.prm.bcs.bc[b];
    const int64_t nnear = scalI(M.scal, SC_NNEAR);
    FOR_ITEMS(t, passItems(M)) {
      const int64_t k = passNode(M, t, nnear);
      const V3 r = nodePos(M, k);
      const double hmaxi = nodeHmax(M, k);
      if (dmin(minimumDistance(bc.exit, r), minimumDistance(bc.enter, r)) < M.prm.kernelExtent*hmaxi)
        best = dmax(best, hmaxi);
    }
  }
  for (int o = 16; o > 0; o >>= 1) best = dmax(best, __shfl_xor_sync(0xffffffffu, best, o));
  if ((threadIdx.x & 31) == 0 && best > 0.0)
    atomicMax(reinterpret_cast<unsigned long long*>(M.scal + SC_HMAX), (unsigned long long)__double_as_longlong(best));
}

__global__ void __launch_bounds__(kGhostThreads) ghost_flag_kernel(const Member* mem, BlockMap bm, int b) {
  const MemberBlock mb = memberBlock(bm);
  const Member& M = mem[mb.m];
  const double hmax = M.scal[SC_HMAX];
  const bool on = M.prm.bcs.periodic[b >> 1] && hmax > 0.0;
  const int64_t nnear = scalI(M.scal, SC_NNEAR);
  FOR_ITEMS(t, passItems(M)) {
    int f = 0;
    if (on) {
      const V3 r = nodePos(M, passNode(M, t, nnear));
      const double disti = signedDistance(M.prm.bcs.bc[b].exit, r)/hmax;
      f = (disti >= 0.0 && disti <= M.prm.kernelExtent) ? 1 : 0;
    }
    M.counts[t] = f;
  }
}

__global__ void __launch_bounds__(kGhostThreads) ghost_scatter_kernel(const Member* mem, BlockMap bm, int b) {
  const MemberBlock mb = memberBlock(bm);
  const Member& M = mem[mb.m];
  const int64_t n = M.n;
  const int64_t ntot = scalI(M.scal, SC_NTOT);
  const int64_t nnear = scalI(M.scal, SC_NNEAR);
  const PlanarBC& bc = M.prm.bcs.bc[b];
  const int axis = b >> 1;
  FOR_ITEMS(t, passItems(M)) {
    if (!M.counts[t]) continue;
    const int64_t k = passNode(M, t, nnear);
    const int64_t g = (ntot - n) + M.offsets[t];     // ghost index of the new image
    if (g >= M.gcap) {
      atomicOr(M.err, DERR_GHOST_CAPACITY);
      continue;
    }
    const V3 gp = mapPositionThroughPlanes(nodePos(M, k), bc.exit, bc.enter);
    const int32_t root = k < n ? (int32_t)k : M.groot[k - n];
    uint32_t code = k < n ? 0u : M.gcode[k - n];
    if ((code >> (2*axis)) & 3u) atomicOr(M.err, DERR_GHOST_CHAIN);
    code |= (uint32_t)((b & 1) + 1) << (2*axis);
    M.groot[g] = root;
    M.gcode[g] = code;
    M.gpos[g] = gp.x; M.gpos[M.gcap + g] = gp.y; M.gpos[2*M.gcap + g] = gp.z;
  }
}

// After a boundary pass: the new images join the node set (at most up to the
// ghost capacity; beyond it the build is redone), hmax restarts.
__global__ void ghost_advance_kernel(const Member* mem, int nmem) {
  const int m = blockIdx.x*blockDim.x + threadIdx.x;
  if (m >= nmem) return;
  const Member& M = mem[m];
  int64_t g = scalI(M.scal, SC_NTOT) - M.n + scalI(M.scal, SC_TOTAL);
  if (g > M.gcap) {
    atomicOr(M.err, DERR_GHOST_CAPACITY);
    g = M.gcap;
  }
  setScalI(M.scal, SC_NTOT, M.n + g);
  setScalI(M.scal, SC_G, g);
  M.scal[SC_HMAX] = 0.0;
}

// ---------------------------------------------------------------- fused ghost passes
// The six boundary passes in one launch.  A boundary's images follow from its
// hmax alone, item by item, so a thread keeps the images its near-plane nodes
// (roots) have so far as a bit set and only the passes' hmax are exchanged:
// one barrier per pass, and one for the counts at the end.
//
// An image is named by the plane it was mapped through on each axis (0 none,
// 1 or 2): e = x + 3 y + 9 z.  The reference's pass order (x, y, z, each plane 1
// then 2; in a pass the nodes first, then the images made so far in their
// order) makes the images come by ascending e, and those of one e by
// ascending root: their place is the images of smaller e plus the smaller
// roots that have this one.  Position, order and error bits are those of the
// per-pass launches.  Measured (B200, whole launch; before, two barriers a pass
// and every pass re-reading nodes and images): 124,550 nodes 80 -> 57 us,
// Kelvin-Helmholtz 128^3 121 -> 65 us; bound by the seven grid barriers.
__device__ __forceinline__ int64_t imin64(int64_t a, int64_t b) { return a < b ? a : b; }
constexpr int kFusedGhostMembers = 4;
constexpr int kGhostCodes = 27;                         // 1 (the root itself) + 26 images
constexpr int kRootThreads = 1024;
constexpr int kFusedGhostBlocks = 148;
constexpr int kBarrierPolls = 1 << 23;

// Grid barrier of a cooperative launch (every block resident).  bar[0]
// counts arrivals, bar[1] is the generation.  A block that polls more than
// kBarrierPolls times records DERR_BARRIER in every member and returns
// false; its launch then ends without finishing the passes.
__device__ bool grid_barrier(unsigned int* bar, const Member* mem, int nm) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    ok = 1;
    volatile unsigned int* gen = bar + 1;
    const unsigned int g0 = *gen;
    __threadfence();
    if (atomicAdd(bar, 1u) == gridDim.x - 1) {
      atomicExch(bar, 0u);
      __threadfence();
      atomicAdd(bar + 1, 1u);
    } else {
      int polls = 0;
      while (*gen == g0) {
        if (++polls > kBarrierPolls) {
          for (int m = 0; m < nm; ++m) atomicOr(mem[m].err, DERR_BARRIER);
          ok = 0;
          break;
        }
      }
    }
    __threadfence();
  }
  __syncthreads();
  return ok != 0;
}


__device__ __forceinline__ uint32_t imageCode(int e) {
  return (uint32_t)(e % 3) | (uint32_t)(e/3 % 3) << 2 | (uint32_t)(e/9) << 4;
}

// image codes with 0 and with 1 on each axis
__device__ constexpr uint32_t digitMask(int axis, int digit) {
  uint32_t m = 0;
  const int step = axis == 0 ? 1 : (axis == 1 ? 3 : 9);
  for (int e = 0; e < kGhostCodes; ++e) if (e/step % 3 == digit) m |= 1u << e;
  return m;
}

// The periodic planes lie across their axis, so a plane's test of an item sees
// the item's coordinate along that axis only, which mapping along the others
// leaves as the root's: the root's own position stands for all its images with
// 0 on the axis, and its image through plane 1 for those with 1.

// largest share of a root's items (itself and its images so far) in the hmax
// of boundary b (ghost_hmax_kernel's test)
__device__ __forceinline__ double rootShare(const Member& M, const V3& r, double h, uint32_t items, int b) {
  const PlanarBC bc = M.prm.bcs.bc[b];
  const double lim = M.prm.kernelExtent*h;
  bool f = dmin(minimumDistance(bc.exit, r), minimumDistance(bc.enter, r)) < lim;
  if ((b & 1) && !f && (items & (b == 1 ? digitMask(0, 1) : (b == 3 ? digitMask(1, 1) : digitMask(2, 1))))) {
    const PlanarBC& one = M.prm.bcs.bc[b - 1];
    const V3 x = mapPositionThroughPlanes(r, one.exit, one.enter);
    f = dmin(minimumDistance(bc.exit, x), minimumDistance(bc.enter, x)) < lim;
  }
  return f ? h : 0.0;
}

// the items boundary b images (ghost_flag_kernel's test) join the set
__device__ __forceinline__ uint32_t rootImages(const Member& M, const V3& r, double hmax, uint32_t items, int b) {
  if (!(hmax > 0.0)) return items;
  const PlanarBC bc = M.prm.bcs.bc[b];
  const int axis = b >> 1, step = axis == 0 ? 1 : (axis == 1 ? 3 : 9);
  const uint32_t d0 = axis == 0 ? digitMask(0, 0) : (axis == 1 ? digitMask(1, 0) : digitMask(2, 0));
  const uint32_t d1 = axis == 0 ? digitMask(0, 1) : (axis == 1 ? digitMask(1, 1) : digitMask(2, 1));
  auto imaged = [&](const V3& x) {
    const double disti = signedDistance(bc.exit, x)/hmax;
    return disti >= 0.0 && disti <= M.prm.kernelExtent;
  };
  uint32_t all = items;
  if (imaged(r)) all |= (items & d0) << (((b & 1) + 1)*step);
  if ((b & 1) && (items & d1)) {
    const PlanarBC& one = M.prm.bcs.bc[b - 1];
    if (imaged(mapPositionThroughPlanes(r, one.exit, one.enter))) atomicOr(M.err, DERR_GHOST_CHAIN);
  }
  return all;
}

// roots of the chunk per image code: cnt[e] (shared)
__device__ __forceinline__ void countImages(const Member& M, int64_t c0, int64_t c1, int* cnt) {
  if (threadIdx.x < 32) cnt[threadIdx.x] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int64_t base = c0; base < c1; base += kRootThreads) {
    const int64_t t = base + threadIdx.x;
    const uint32_t items = t < c1 ? (uint32_t)M.counts[t] : 0u;
    int mine = 0;
    for (uint32_t codes = __reduce_or_sync(0xffffffffu, items) & ~1u; codes; codes &= codes - 1) {
      const int e = __ffs(codes) - 1;
      const unsigned bal = __ballot_sync(0xffffffffu, items >> e & 1u);
      if (lane == e) mine = __popc(bal);
    }
    if (mine) atomicAdd(cnt + lane, mine);
  }
  __syncthreads();
}

// the images of the chunk's roots; next[e] (shared): ghost index of the
// chunk's first image of code e
__device__ __forceinline__ void writeImages(const Member& M, int64_t c0, int64_t c1, int64_t* next, int (*warpCnt)[32]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int64_t base = c0; base < c1; base += kRootThreads) {
    const int64_t t = base + threadIdx.x;
    uint32_t items = t < c1 ? (uint32_t)M.counts[t] & ~1u : 0u;
    const uint32_t codes = __reduce_or_sync(0xffffffffu, items);
    int mine = 0;
    for (uint32_t left = codes; left; left &= left - 1) {
      const int e = __ffs(left) - 1;
      const unsigned bal = __ballot_sync(0xffffffffu, items >> e & 1u);
      if (lane == e) mine = __popc(bal);
    }
    warpCnt[w][lane] = mine;
    __syncthreads();
    // lane e: the first index of this warp's images of code e
    int64_t at = next[lane];
    {
      int pre = 0;
#pragma unroll 8
      for (int k = 0; k < kRootThreads/32; ++k) pre += k < w ? warpCnt[k][lane] : 0;
      at += pre;
    }
    if (codes) {
      int32_t root = 0;
      V3 r{0.0, 0.0, 0.0};
      if (items) {
        root = __ldcg(M.cidx + t);
        r = nodePos(M, root);
      }
      for (uint32_t left = codes; left; left &= left - 1) {
        const int e = __ffs(left) - 1;
        const bool has = items >> e & 1u;
        const unsigned bal = __ballot_sync(0xffffffffu, has);
        const int64_t first = __shfl_sync(0xffffffffu, at, e);
        if (!has) continue;
        const int64_t g = first + __popc(bal & ((1u << lane) - 1u));
        if (g >= M.gcap) {
          atomicOr(M.err, DERR_GHOST_CAPACITY);
          continue;
        }
        const uint32_t code = imageCode(e);
        const V3 gp = ghostPosition(M.prm.bcs, r, code);
        M.groot[g] = root;
        M.gcode[g] = code;
        M.gpos[g] = gp.x; M.gpos[M.gcap + g] = gp.y; M.gpos[2*M.gcap + g] = gp.z;
      }
    }
    __syncthreads();
    if (w == 0) {
      int sum = 0;
#pragma unroll 8
      for (int k = 0; k < kRootThreads/32; ++k) sum += warpCnt[k][lane];
      next[lane] += sum;
    }
    __syncthreads();
  }
}

// sizes after the passes
__device__ __forceinline__ void endGhosts(const Member& M, int64_t G) {
  if (G > M.gcap) {
    atomicOr(M.err, DERR_GHOST_CAPACITY);
    G = M.gcap;
  }
  setScalI(M.scal, SC_NTOT, M.n + G);
  setScalI(M.scal, SC_G, G);
  M.scal[SC_HMAX] = 0.0;
}

__device__ __forceinline__ double blockMax(double x, double* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int o = 16; o > 0; o >>= 1) x = dmax(x, __shfl_xor_sync(0xffffffffu, x, o));
  __syncthreads();
  if (lane == 0) red[w] = x;
  __syncthreads();
  x = red[lane];
  for (int o = 16; o > 0; o >>= 1) x = dmax(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}

// A cooperative launch over the near-plane lists of a batch of a few members;
// fuse: the barrier (2 words), then the per-block counts of each member and code.
__global__ void __launch_bounds__(kRootThreads, 1) ghost_passes_fused_kernel(const Member* mem, int nm, unsigned int* fuse) {
  unsigned int* bar = fuse;
  int* blk = reinterpret_cast<int*>(fuse + 2);            // [member][code][block]
  const int nb = gridDim.x, kb = blockIdx.x;
  __shared__ double red[32];
  __shared__ int cnt[32], warpCnt[kRootThreads/32][32];
  __shared__ int64_t next[32];
  for (int b = 0; b < 6; ++b) {
    bool any = false;
    for (int m = 0; m < nm; ++m) any = any || mem[m].prm.bcs.periodic[b >> 1];
    if (!any && b > 0) continue;
    for (int m = 0; m < nm; ++m) {
      const Member& M = mem[m];
      const int64_t nnear = scalI(M.scal, SC_NNEAR), chunk = (nnear + nb - 1)/nb;
      const int64_t c0 = imin64(nnear, kb*chunk), c1 = imin64(nnear, c0 + chunk);
      double best = 0.0;
      for (int64_t t = c0 + threadIdx.x; t < c1; t += kRootThreads) {
        if (b == 0) M.counts[t] = 1;
        if (!M.prm.bcs.periodic[b >> 1]) continue;
        const int64_t k = M.cidx[t];
        best = dmax(best, rootShare(M, nodePos(M, k), M.hmaxi[k], (uint32_t)M.counts[t], b));
      }
      best = blockMax(best, red);
      if (threadIdx.x == 0 && best > 0.0)
        atomicMax(reinterpret_cast<unsigned long long*>(M.scal + SC_PHMAX + b), (unsigned long long)__double_as_longlong(best));
    }
    if (!any) continue;
    if (!grid_barrier(bar, mem, nm)) return;
    for (int m = 0; m < nm; ++m) {
      const Member& M = mem[m];
      if (!M.prm.bcs.periodic[b >> 1]) continue;
      const int64_t nnear = scalI(M.scal, SC_NNEAR), chunk = (nnear + nb - 1)/nb;
      const int64_t c0 = imin64(nnear, kb*chunk), c1 = imin64(nnear, c0 + chunk);
      const double hmax = __longlong_as_double((long long)__ldcg(reinterpret_cast<const unsigned long long*>(M.scal + SC_PHMAX + b)));
      for (int64_t t = c0 + threadIdx.x; t < c1; t += kRootThreads)
        M.counts[t] = (int32_t)rootImages(M, nodePos(M, M.cidx[t]), hmax, (uint32_t)M.counts[t], b);
    }
  }
  for (int m = 0; m < nm; ++m) {
    const Member& M = mem[m];
    const int64_t nnear = scalI(M.scal, SC_NNEAR), chunk = (nnear + nb - 1)/nb;
    const int64_t c0 = imin64(nnear, kb*chunk), c1 = imin64(nnear, c0 + chunk);
    countImages(M, c0, c1, cnt);
    if (threadIdx.x < kGhostCodes) blk[(m*kGhostCodes + threadIdx.x)*nb + kb] = cnt[threadIdx.x];
    __syncthreads();
  }
  if (!grid_barrier(bar, mem, nm)) return;
  for (int m = 0; m < nm; ++m) {
    const Member& M = mem[m];
    const int64_t nnear = scalI(M.scal, SC_NNEAR), chunk = (nnear + nb - 1)/nb;
    const int64_t c0 = imin64(nnear, kb*chunk), c1 = imin64(nnear, c0 + chunk);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // warp e: the images of code e in the blocks before this one, and in all
    int before = 0, total = 0;
    if (w < kGhostCodes) {
      for (int k = lane; k < nb; k += 32) {
        const int c = __ldcg(blk + (m*kGhostCodes + w)*nb + k);
        total += c;
        if (k < kb) before += c;
      }
    }
    before = __reduce_add_sync(0xffffffffu, before);
    total = __reduce_add_sync(0xffffffffu, total);
    if (lane == 0) { warpCnt[0][w] = before; warpCnt[1][w] = total; }
    __syncthreads();
    if (w == 0) {
      const int64_t mine = warpCnt[1][lane];
      int64_t incl = mine;
      for (int o = 1; o < 32; o <<= 1) {
        const int64_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      next[lane] = incl - mine + warpCnt[0][lane];
      if (lane == 31 && kb == 0) endGhosts(M, incl);
    }
    __syncthreads();
    writeImages(M, c0, c1, next, warpCnt);
  }
}

// ---------------------------------------------------------------- cells
// Uniform grid of cells of edge >= kappa*max(1/lambda_min(H)) (the margin
// covers the libm difference of the eigenvalue solve for anisotropic H),
// enlarged until the cells fit the cell buffers (larger cells only widen the
// candidate set).  Also resets the walk's counters and sets the FP32
// pre-test tolerance: only when max h / min h over the problem is <= 100.
__device__ void setGrid(const Member& M) {
  const unsigned long long* bb = reinterpret_cast<const unsigned long long*>(M.scal + SC_BOUNDS);
  double lo[3], hi[3];
  for (int a = 0; a < 3; ++a) { lo[a] = fromOrderedBits(bb[a]); hi[a] = fromOrderedBits(bb[3 + a]); }
  const double hmaxAll = fromOrderedBits(bb[6]);
  // ghosts lie within kappa*hmax (<= kappa*hmaxAll) beyond the periodic
  // planes; elsewhere they share their root's coordinates
  const double reach = M.prm.kernelExtent*hmaxAll*1.001 + 1.0e-300;
  for (int a = 0; a < 3; ++a) {
    if (!M.prm.bcs.periodic[a]) continue;
    const PlanarBC& bc = M.prm.bcs.bc[2*a];
    const double p0 = (&bc.enter.point.x)[a], p1 = (&bc.exit.point.x)[a];
    lo[a] = fmin(lo[a], fmin(p0, p1) - reach);
    hi[a] = fmax(hi[a], fmax(p0, p1) + reach);
  }
  const int sub = M.grid.sub > 1 ? M.grid.sub : 1;
  double cell = M.prm.kernelExtent*hmaxAll*1.001/sub;
  if (!(cell > 0.0) || !(cell < 1.0e300)) {
    atomicOr(M.err, DERR_NONPOSITIVE);
    cell = 1.0;
  }
  const int64_t maxCells = M.cellcap < ((int64_t)1 << 26) ? M.cellcap : ((int64_t)1 << 26);
  int64_t dim[3] = {1, 1, 1}, ncells = 1;
  bool covered = true;
  {
    // cells at the natural size, for the next build's capacity
    double want = 1.0;
    for (int a = 0; a < 3; ++a) want *= fmin((hi[a] - lo[a])/cell + 1.0, (double)(1 << 20));
    setScalI(M.scal, SC_CELLSWANTED, want < 1.0e15 ? (int64_t)want : (int64_t)1 << 50);
  }
  for (int attempt = 0; attempt < 200; ++attempt) {
    ncells = 1;
    for (int a = 0; a < 3; ++a) {
      const double d = (hi[a] - lo[a])/cell;
      const int64_t mm = d < 1.0e6 ? (int64_t)d + 1 : (int64_t)1 << 20;
      dim[a] = mm < (1 << 20) ? mm : (1 << 20);
      ncells *= dim[a];
    }
    if (ncells <= maxCells) break;
    cell *= 1.26;
  }
  for (int a = 0; a < 3; ++a) covered = covered && dim[a] < (1 << 20);
  double* s = M.scal + SC_GRID;
  s[0] = lo[0]; s[1] = lo[1]; s[2] = lo[2];
  s[3] = cell;
  for (int a = 0; a < 3; ++a) setScalI(M.scal, SC_GRID + 4 + a, dim[a]);
  // largest h over smallest h of the problem (>= every node's condition number)
  // and the cells' edge over the kernel reach where the capacity enlarged them:
  // the FP32 pre-test's relative error is below 2e-6 times their product (the
  // offsets are rounded at the size of a cell).  The band is ten times that,
  // 1e-3 at most, and the pre-test is off beyond a product of 100, and where
  // the grid ends before the box does (the offsets in its last cells have any
  // size).
  const double natural = M.prm.kernelExtent*hmaxAll*1.001/sub;
  const double spread = hmaxAll*M.scal[SC_LMAXALL]*fmax(1.0, cell/natural);
  s[7] = (M.grid.filterTol > 0.0f && covered && spread > 0.0 && spread <= 100.0)
             ? fmin((double)M.grid.filterTol, kFilterTolPerSpread*fmax(spread, 1.0)) : 0.0;
  // the largest kernel reach in cells (<= sub), for the walks' pruning
  M.scal[SC_REACH] = M.prm.kernelExtent*hmaxAll/cell;
  setScalI(M.scal, SC_NCELLS, ncells);
  setScalI(M.scal, SC_MAXCOUNT, 0);
  setScalI(M.scal, SC_PAIRS, 0);
  setScalI(M.scal, SC_CROWDED, 0);
}

__global__ void grid_kernel(const Member* mem, int nmem) {
  const int m = blockIdx.x*blockDim.x + threadIdx.x;
  if (m < nmem) setGrid(mem[m]);
}

// ---------------------------------------------------------------- small members
// The build up to the cell grid (hmax, bounds, near-plane list, the six
// boundary passes, the grid) in one launch with a cluster of 8 blocks per
// member, for members of at most kClusterNodes nodes.
//
// Why: the work is a few thousand items, but as separate launches it was nine
// kernels with a cooperative one among them.  Measured (B200): 4,096-node Sod
// tube, the nine launches 100 us, here 45 us.  Beyond kClusterNodes the eight
// blocks' passes over all nodes take longer than the launches saved (124,550
// nodes: 262 us against about 85).  The blocks of a cluster exchange their counts and
// maxima through each other's shared memory and meet at the hardware's cluster
// barrier.  Block k takes the k-th contiguous chunk of every list, so the
// near-plane list, the images, their order and the error bits are those of the
// separate launches.
namespace cg = cooperative_groups;
constexpr int kClusterBlocks = 8;
constexpr int kClusterThreads = kRootThreads;
#ifndef CLUSTER_NODES
#define CLUSTER_NODES 32768
#endif
constexpr int64_t kClusterNodes = CLUSTER_NODES;

struct ClusterShared {
  double hmax[6];                 // this block's share of each pass's hmax
  double bounds[8];               // lo[3], hi[3], largest 1/min(eig(H)), largest max(eig(H))
  int count;                      // near-plane nodes of this block's chunk
  int before, total;              // ... of the blocks before, of all
  double all;                     // the cluster's maximum
  int images[32];                 // images of this block's chunk, by code
  int64_t next[32];
  int warp[32], warpCnt[kClusterThreads/32][32];
  double red[32][8];
};

// flagged items of the block's chunk [c0, c1)
template<class Flag>
__device__ __forceinline__ int clusterCount(int64_t c0, int64_t c1, Flag flag) {
  int cnt = 0;
  for (int64_t base = c0; base < c1; base += kClusterThreads) {
    const int64_t t = base + threadIdx.x;
    cnt += __syncthreads_count(t < c1 && flag(t));
  }
  return cnt;
}

// put(t, k): item t is the chunk's k-th flagged one
template<class Flag, class Put>
__device__ __forceinline__ void clusterScatter(ClusterShared& sh, int64_t c0, int64_t c1, Flag flag, Put put) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int done = 0;
  for (int64_t base = c0; base < c1; base += kClusterThreads) {
    const int64_t t = base + threadIdx.x;
    const bool f = t < c1 && flag(t);
    const unsigned bal = __ballot_sync(0xffffffffu, f);
    __syncthreads();
    if (lane == 0) sh.warp[w] = __popc(bal);
    __syncthreads();
    const int c = sh.warp[lane];
    const int off = done + __reduce_add_sync(0xffffffffu, lane < w ? c : 0);
    done += __reduce_add_sync(0xffffffffu, c);
    if (f) put(t, off + __popc(bal & ((1u << lane) - 1u)));
  }
}

__global__ void __cluster_dims__(kClusterBlocks, 1, 1) __launch_bounds__(kClusterThreads, 1) ghost_cluster_kernel(const Member* mem) {
  __shared__ ClusterShared sh;
  cg::cluster_group cl = cg::this_cluster();
  const Member& M = mem[blockIdx.x/kClusterBlocks];
  const int rank = (int)cl.block_rank();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t n = M.n;
  // 1/min(eig(H)), max(eig(H)), the bounds (node_hmax_kernel)
  {
    double v[8] = {1e300, 1e300, 1e300, -1e300, -1e300, -1e300, 0.0, 0.0};
    for (int64_t i = rank*(int64_t)kClusterThreads + threadIdx.x; i < n; i += kClusterBlocks*kClusterThreads) {
      const V3 ev = eigenValues(nodeH(M, i));
      const double hi1 = 1.0/vmin(ev);
      M.hmaxi[i] = hi1;
      v[6] = fmax(v[6], hi1);
      double l = vmax(ev);
      M.hmaxi[n + i] = l;
      if (!(l < 1.0e300)) l = 1.0e300;           // degenerate H: no FP32 pre-test
      v[7] = dmax(v[7], l);
      const V3 r = nodePos(M, i);
      v[0] = fmin(v[0], r.x); v[1] = fmin(v[1], r.y); v[2] = fmin(v[2], r.z);
      v[3] = fmax(v[3], r.x); v[4] = fmax(v[4], r.y); v[5] = fmax(v[5], r.z);
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      for (int o = 16; o > 0; o >>= 1) {
        const double x = __shfl_xor_sync(0xffffffffu, v[c], o);
        v[c] = c < 3 ? fmin(v[c], x) : (c < 7 ? fmax(v[c], x) : dmax(v[c], x));
      }
      if (lane == 0) sh.red[w][c] = v[c];
    }
    __syncthreads();
    if (w < 8) {
      double x = sh.red[lane][w];
      for (int o = 16; o > 0; o >>= 1) {
        const double y = __shfl_xor_sync(0xffffffffu, x, o);
        x = w < 3 ? fmin(x, y) : fmax(x, y);
      }
      if (lane == 0) sh.bounds[w] = x;
    }
  }
  cl.sync();
  if (w == 0) {
    // one warp reads the other blocks' shared memory
    double b[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      double x = cl.map_shared_rank(&sh, lane % kClusterBlocks)->bounds[c];
      for (int o = kClusterBlocks/2; o > 0; o >>= 1) {
        const double y = __shfl_xor_sync(0xffffffffu, x, o);
        x = c < 3 ? fmin(x, y) : fmax(x, y);
      }
      b[c] = x;
    }
    if (lane == 0) sh.all = b[6];
    if (rank == 0 && lane == 0) {
    unsigned long long* out = reinterpret_cast<unsigned long long*>(M.scal + SC_BOUNDS);
    for (int a = 0; a < 3; ++a) {
      out[a] = b[6] > 0.0 ? orderedBits(b[a]) : ~0ULL;
      out[3 + a] = b[6] > 0.0 ? orderedBits(b[3 + a]) : 0ULL;
    }
    out[6] = b[6] > 0.0 ? orderedBits(b[6]) : 0ULL;
    M.scal[SC_LMAXALL] = b[7];
    }
  }
  __syncthreads();
  const double hAll = sh.all;
  // the near-plane list, ascending (near_flag_kernel, near_list_kernel)
  const double nearReach = M.prm.kernelExtent*fromOrderedBits(hAll > 0.0 ? orderedBits(hAll) : 0ULL)*(1.0 + 1.0e-6);
  auto isNear = [&](int64_t i) {
    const V3 r = nodePos(M, i);
    bool f = false;
    for (int a = 0; a < 3; ++a) {
      if (!M.prm.bcs.periodic[a]) continue;
      const PlanarBC& bc = M.prm.bcs.bc[2*a];
      if (dmin(minimumDistance(bc.exit, r), minimumDistance(bc.enter, r)) <= nearReach) f = true;
    }
    return f;
  };
  int64_t before = 0, nnear = 0;
  {
    const int64_t chunk = (n + kClusterBlocks - 1)/kClusterBlocks;
    const int64_t c0 = imin64(n, rank*chunk), c1 = imin64(n, c0 + chunk);
    const int cnt = clusterCount(c0, c1, isNear);
    if (threadIdx.x == 0) sh.count = cnt;
    cl.sync();
    if (w == 0) {
      const int c = lane < kClusterBlocks ? cl.map_shared_rank(&sh, lane)->count : 0;
      const int pre = __reduce_add_sync(0xffffffffu, lane < rank ? c : 0), all = __reduce_add_sync(0xffffffffu, c);
      if (lane == 0) { sh.before = pre; sh.total = all; }
    }
    __syncthreads();
    before = sh.before;
    nnear = sh.total;
    clusterScatter(sh, c0, c1, isNear, [&](int64_t i, int64_t k) { M.cidx[before + k] = (int32_t)i; });
    cl.sync();
  }
  // the boundary passes (ghost_passes_fused_kernel)
  const int64_t chunk = (nnear + kClusterBlocks - 1)/kClusterBlocks;
  const int64_t c0 = imin64(nnear, rank*chunk), c1 = imin64(nnear, c0 + chunk);
  for (int64_t t = c0 + threadIdx.x; t < c1; t += kRootThreads) M.counts[t] = 1;
  for (int b = 0; b < 6; ++b) {
    if (!M.prm.bcs.periodic[b >> 1]) continue;
    double best = 0.0;
    for (int64_t t = c0 + threadIdx.x; t < c1; t += kRootThreads) {
      const int64_t k = __ldcg(M.cidx + t);
      best = dmax(best, rootShare(M, nodePos(M, k), __ldcg(M.hmaxi + k), (uint32_t)M.counts[t], b));
    }
    best = blockMax(best, &sh.red[0][0]);
    if (threadIdx.x == 0) sh.hmax[b] = best;
    cl.sync();
    if (w == 0) {
      double x = cl.map_shared_rank(&sh, lane % kClusterBlocks)->hmax[b];
      for (int o = kClusterBlocks/2; o > 0; o >>= 1) x = dmax(x, __shfl_xor_sync(0xffffffffu, x, o));
      if (lane == 0) sh.all = x;
    }
    __syncthreads();
    const double hmax = sh.all;
    for (int64_t t = c0 + threadIdx.x; t < c1; t += kRootThreads)
      M.counts[t] = (int32_t)rootImages(M, nodePos(M, __ldcg(M.cidx + t)), hmax, (uint32_t)M.counts[t], b);
  }
  countImages(M, c0, c1, sh.images);
  cl.sync();
  if (w == 0) {
    int64_t mine = 0, pre = 0;
    for (int k = 0; k < kClusterBlocks; ++k) {
      const int c = cl.map_shared_rank(&sh, k)->images[lane];
      if (k < rank) pre += c;
      mine += c;
    }
    int64_t incl = mine;
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    sh.next[lane] = incl - mine + pre;
    if (lane == 31 && rank == 0) {
      setScalI(M.scal, SC_NNEAR, nnear);
      endGhosts(M, incl);
    }
  }
  __syncthreads();
  writeImages(M, c0, c1, sh.next, sh.warpCnt);
  if (rank == 0 && threadIdx.x == 0) setGrid(M);
  cl.sync();                      // no block leaves while another may read its shared memory
}

__device__ __forceinline__ int cellCoord(double x, double lo, double cell, int dim) {
  int c = int((x - lo)/cell);
  return c < 0 ? 0 : (c >= dim ? dim - 1 : c);
}

__global__ void __launch_bounds__(kGhostThreads) cell_zero_kernel(const Member* mem, BlockMap bm) {
  const MemberBlock mb = memberBlock(bm);
  const Member& M = mem[mb.m];
  FOR_ITEMS(c, scalI(M.scal, SC_NCELLS)) M.cellFill[c] = 0;
}

__global__ void __launch_bounds__(kGhostThreads) cell_index_kernel(const Member* mem, BlockMap bm) {
  const MemberBlock mb = memberBlock(bm);
  const Member& M = mem[mb.m];
  const Grid g = loadGrid(M);
  FOR_ITEMS(k, allNodes(M)) {
    const V3 r = nodePos(M, k);
    const int cx = cellCoord(r.x, g.lo[0], g.cell, g.dim[0]);
    const int cy = cellCoord(r.y, g.lo[1], g.cell, g.dim[1]);
    const int cz = cellCoord(r.z, g.lo[2], g.cell, g.dim[2]);
    const int c = (cz*g.dim[1] + cy)*g.dim[0] + cx;
    M.cidx[k] = c;
    atomicAdd(M.cellFill + c, 1);
  }
}

// Cell-ordered candidate arrays (Problem::cand), one slot per node:
//   pre     [candcap] float4:   FP32 offsets of the position from the lower
//                               corner of the node's cell, and
//                               k2hi/min eig(H)^2 (k2hi the upper edge of the
//                               pre-test band): beyond that r^2 the node's own
//                               eta^2 lies above the band
//   lmax    [candcap] float:    FP32 max eig(H)
// Both are in units of the cell edge, as every length of the FP32 tests is: r^2
// and its bounds are then of order one, and no FP32 square overflows or
// vanishes whatever the problem's unit of length (a centimetre with kernels of
// 1e20 cm, say).
// and sortedIdx[slot], the node of each slot.  The walks read only `pre` for
// most candidates; `lmax` when the i-side test alone does not decide, and
// the FP64 position and H of the node (state, ghost positions) for the
// candidates the FP32 pre-test cannot decide.
struct NbrArrays {
  const float4* pre;
  const float* lmax;
};

__device__ __forceinline__ NbrArrays nbrArrays(const Member& M) {
  const double* c = static_cast<const double*>(M.cand);
  NbrArrays a;
  a.pre = reinterpret_cast<const float4*>(c);
  a.lmax = reinterpret_cast<const float*>(c + 2*M.candcap);
  return a;
}

__device__ __forceinline__ float symEta2F(const float* h, float x, float y, float z) {
  const float ex = __fmaf_rn(h[0], x, __fmaf_rn(h[1], y, h[2]*z));
  const float ey = __fmaf_rn(h[1], x, __fmaf_rn(h[3], y, h[4]*z));
  const float ez = __fmaf_rn(h[2], x, __fmaf_rn(h[4], y, h[5]*z));
  return __fmaf_rn(ex, ex, __fmaf_rn(ey, ey, ez*ez));
}

// The walking node: FP32 H and cell offsets for the pre-test (in cell edges),
// its cell, its sorted slot and node index (the exact test re-reads its FP64
// state).
struct Walker {
  float hf[6];
  float lam2;          // isotropic H = lam I: lam^2 (then eta_i^2 = lam^2 |r|^2)
  float T;             // k2hi/min eig(H)^2: beyond r^2 = T the node's own eta^2 exceeds the band
  bool iso;
  float ox, oy, oz;
  int cx, cy, cz;
  int32_t slot;
  int32_t idx;
};

// Walker of sorted slot s; idx >= n marks a ghost slot (no walk).
__device__ __forceinline__ Walker makeWalker(const Member& M, const NbrArrays& a, const Grid& g, int32_t s) {
  Walker w;
  w.slot = s;
  w.idx = __ldg(M.sortedIdx + s);
  if (w.idx >= M.n) return w;
  const V3 r = nodePos(M, w.idx);
  const Sym H = nodeH(M, w.idx);
  w.hf[0] = (float)(H.xx*g.cell); w.hf[1] = (float)(H.xy*g.cell); w.hf[2] = (float)(H.xz*g.cell);
  w.hf[3] = (float)(H.yy*g.cell); w.hf[4] = (float)(H.yz*g.cell); w.hf[5] = (float)(H.zz*g.cell);
  w.iso = H.xy == 0.0 && H.xz == 0.0 && H.yz == 0.0 && H.xx == H.yy && H.xx == H.zz;
  w.lam2 = w.hf[0]*w.hf[0];
  const float4 p = __ldg(a.pre + s);
  w.ox = p.x; w.oy = p.y; w.oz = p.z;
  w.T = p.w;
  w.cx = cellCoord(r.x, g.lo[0], g.cell, g.dim[0]);
  w.cy = cellCoord(r.y, g.lo[1], g.cell, g.dim[1]);
  w.cz = cellCoord(r.z, g.lo[2], g.cell, g.dim[2]);
  return w;
}

// Square of the distance, in cells, beyond which a walk leaves candidates out:
// the largest kernel reach, a relative margin, and `slack` for the rounding of
// the FP32 offsets (which counts where the cells' capacity made them many times
// a reach).
__device__ __forceinline__ float reachBound2(float reach, float slack) {
  const float r = reach*1.00005f + slack;
  return r*r;
}

// Distance, in cells, from a walker at fraction f of its cell to the cell d
// cells away along one axis (0 for its own cell); a lower bound for every
// node of that cell.
__device__ __forceinline__ float axisGap(int d, float f) {
  return d > 0 ? fmaxf(0.0f, (float)d - f) : (d < 0 ? fmaxf(0.0f, (float)(-d - 1) + f) : 0.0f);
}

// One x-row of the walk window: the candidate slot range [start, end) of its
// cells x0..x1 (contiguous in the sorted order), trimmed with SUB > 1 to
// the cells within the kernel reach, and the ends of its first cells (a
// candidate's cell follows from its slot).
template<int SUB>
struct Row {
  int32_t start, end;  // slots (every slot index fits in 32 bits)
  int32_t e[2*SUB];
  int x0;
};

template<int SUB>
__device__ __forceinline__ Row<SUB> loadRow(const Member& M, const Grid& g, const Walker& w, int y, int z,
                                            float fx, float gyz, float rc2) {
  int x0 = w.cx - SUB > 0 ? w.cx - SUB : 0;
  int x1 = w.cx + SUB < g.dim[0] - 1 ? w.cx + SUB : g.dim[0] - 1;
  if (SUB > 1) {
    // the gaps grow with |x - cx|: trim the far cells at both ends
    while (x0 < w.cx) { const float gx = axisGap(x0 - w.cx, fx); if (gx*gx + gyz <= rc2) break; ++x0; }
    while (x1 > w.cx) { const float gx = axisGap(x1 - w.cx, fx); if (gx*gx + gyz <= rc2) break; --x1; }
  }
  const int64_t* cs = M.cellStart + (int64_t)(z*g.dim[1] + y)*g.dim[0] + x0;
  const int nx = x1 - x0 + 1;
  Row<SUB> r;
  r.x0 = x0;
  r.start = (int32_t)cs[0];
  r.end = (int32_t)cs[nx];
#pragma unroll
  for (int c = 0; c < 2*SUB; ++c) r.e[c] = c + 1 < nx ? (int32_t)cs[c + 1] : r.end;
  return r;
}

template<int SUB>
__device__ __forceinline__ float rowDxc(const Row<SUB>& r, const Walker& w, int32_t k) {
  int xc = r.x0 - w.cx;
#pragma unroll
  for (int c = 0; c < 2*SUB; ++c) xc += (k >= r.e[c]);
  return (float)xc;
}

// The exact FP64 predicate for nodes i and j (the walks reach it for the
// few candidates the pre-test leaves undecided).
__device__ __forceinline__ bool exactTest(const Member& M, int32_t i, int32_t j, double k2) {
  const int64_t n = M.n;
  const double* S = M.S;
  const V3 ri{S[S_X*n + i], S[S_Y*n + i], S[S_Z*n + i]};     // the walker is an internal node
  const V3 rj = nodePos(M, j);
  const V3 rij{ri.x - rj.x, ri.y - rj.y, ri.z - rj.z};
  const Sym Hi{S[(S_H + 0)*n + i], S[(S_H + 1)*n + i], S[(S_H + 2)*n + i],
               S[(S_H + 3)*n + i], S[(S_H + 4)*n + i], S[(S_H + 5)*n + i]};
  return mag2(sdot(Hi, rij)) <= k2 || mag2(sdot(nodeH(M, j), rij)) <= k2;
}

// ConnectivityMap predicate |H_i r_ij|^2 <= kappa^2 || |H_j r_ij|^2 <= kappa^2
// (src/Neighbor/ConnectivityMapInline.hh:169-186) for candidate slot k, whose
// cell corner lies at (dxc, dyc, dzc) from the walker's, in cells.
// With tol > 0 a FP32 pre-test decides every pair whose eta^2 lies clearly
// outside the band kappa^2 (1 -+ tol): eta_i^2 from the FP32 H_i, eta_j^2
// bounded by min/max eig(H_j)^2 |r_ij|^2, r_ij from the cell offsets.  The
// pre-test error is below 2e-6 (max h/min h over the problem) relative, and
// tol is ten times that (grid_kernel), so it never decides a
// pair the exact test would decide otherwise.  Undecided pairs take the
// exact FP64 test in the reference's operation order.  eta^2 of either node
// lies in [min eig(H)^2 r^2, max eig(H)^2 r^2]: a candidate beyond the band
// for the smaller of the two minimum eigenvalues is rejected from r^2 alone
// (most candidates of the window); each record carries that r^2 bound,
// k2hi/min eig(H)^2, so the test is one comparison with the larger of the
// two nodes' bounds.
__device__ __forceinline__ bool candTest(const Member& M, const NbrArrays& a, const Walker& w, int32_t k,
                                         float dxc, float dyc, float dzc, double k2, float k2lo, float k2hi,
                                         bool pretest) {
  if (pretest) {
    const float4 c = __ldg(a.pre + k);
    const float fx = (w.ox - c.x) - dxc, fy = (w.oy - c.y) - dyc, fz = (w.oz - c.z) - dzc;
    const float r2 = __fmaf_rn(fx, fx, __fmaf_rn(fy, fy, fz*fz));
    if (r2 > fmaxf(w.T, c.w)) return false;
    float e2i;
    if (w.iso) e2i = w.lam2*r2;          // the common case: H = lam I
    else e2i = symEta2F(w.hf, fx, fy, fz);
    if (e2i <= k2lo) return true;
    if (e2i > k2hi && r2 > c.w) return false;
    const float lm = __ldg(a.lmax + k);
    if (lm*lm*r2 <= k2lo) return true;
  }
  return exactTest(M, w.idx, __ldg(M.sortedIdx + k), k2);
}

__global__ void __launch_bounds__(kGhostThreads) cell_scatter_kernel(const Member* mem, BlockMap bm) {
  const MemberBlock mb = memberBlock(bm);
  const Member& M = mem[mb.m];
  const Grid g = loadGrid(M);
  double* base = static_cast<double*>(M.cand);
  float4* pre = reinterpret_cast<float4*>(base);
  float* lmax = reinterpret_cast<float*>(base + 2*M.candcap);
  // the pre-test's upper band edge, as the walks form it
  const float k2f = (float)(M.prm.kernelExtent*M.prm.kernelExtent);
  const double k2hi = (double)(k2f*(1.0f + g.filterTol));
  const double inv = 1.0/g.cell;
  FOR_ITEMS(k, allNodes(M)) {
    const int c = M.cidx[k];
    const int64_t slot = M.cellStart[c] + atomicAdd(M.cellFill + c, 1);
    M.sortedIdx[slot] = (int32_t)k;
    const V3 r = nodePos(M, k);
    const int cx = cellCoord(r.x, g.lo[0], g.cell, g.dim[0]);
    const int cy = cellCoord(r.y, g.lo[1], g.cell, g.dim[1]);
    const int cz = cellCoord(r.z, g.lo[2], g.cell, g.dim[2]);
    const int64_t root = k < M.n ? k : M.groot[k - M.n];
    const double hm = M.hmaxi[root]*inv;
    pre[slot] = make_float4((float)((r.x - (g.lo[0] + cx*g.cell))*inv), (float)((r.y - (g.lo[1] + cy*g.cell))*inv),
                            (float)((r.z - (g.lo[2] + cz*g.cell))*inv), (float)(k2hi*hm*hm));
    lmax[slot] = (float)(M.hmaxi[M.n + root]*g.cell);
  }
}

// Thread per internal node, nodes taken in cell-sorted order so that the
// threads of a warp share their candidate rows (L1 broadcast).  The 27
// neighbouring cells are walked as 9 x-rows (three cells each, contiguous in
// the sorted order) and the ConnectivityMap predicate is applied.
// COUNT pass: per-node counts and their maximum.  FILL pass: the neighbor
// indices are insertion-sorted into a per-thread shared-memory list of
// capacity `cap` (element c of thread t at lst[c*blockDim + t], conflict
// free) and stored ascending at offsets[i].
// A member with a stash (Grid::stashCap > 0) builds its lists in the COUNT
// pass too and stores them ascending in the stash, element c of sorted slot s
// at stash[c*stashStride + s]; nbr_compact_thread_kernel then moves them to
// offsets[i], and the FILL pass does not run for it.
template<bool FILL, int SUB>
__global__ void __launch_bounds__(256, SUB == 1 ? NBR_THREAD_MIN_BLOCKS : 1) nbr_thread_kernel(const Member* mem, BlockMap bm, int cap, int maxNbr) {
  extern __shared__ int32_t lst[];
  const MemberBlock mb = memberBlock(bm);
  const Member& M = mem[mb.m];
  const int tid = threadIdx.x;
  const int bd = blockDim.x;
  const int64_t s = mb.block*bd + tid;
  const int64_t n = M.n;
  const NbrArrays a = nbrArrays(M);
  const Grid g = loadGrid(M);
  bool active = s < allNodes(M);
  Walker me;
  if (active) {
    me = makeWalker(M, a, g, (int32_t)s);
    active = me.idx < n;
  }
  // list capacity: the shared-memory list (FILL) or the member's stash (COUNT)
  const int lcap = FILL ? cap : M.grid.stashCap;
  const bool collect = FILL || lcap > 0;
  int count = 0, above = 0;
  if (active) {
    const double k2 = M.prm.kernelExtent*M.prm.kernelExtent;
    const float k2f = (float)k2;
    const bool pretest = g.filterTol > 0.0f;
    const float k2lo = k2f*(1.0f - g.filterTol), k2hi = k2f*(1.0f + g.filterTol);
    const int32_t i = me.idx;
    // window of +-SUB cells; with SUB > 1 the rows and cells farther than the
    // largest kernel reach (in cells, with a margin) are skipped
    const float rc2 = reachBound2(g.reach, 1.0e-6f);
    auto accept = [&](int32_t k) {
      if (collect) {
        const int32_t j = __ldg(M.sortedIdx + k);
        if (count < lcap) {
          int p = count;
          while (p > 0) {
            const int32_t prev = lst[(p - 1)*bd + tid];
            if (prev < j) break;
            lst[p*bd + tid] = prev;
            --p;
          }
          lst[p*bd + tid] = j;
        }
        above += (j > i);
      }
      ++count;
    };
    {
      const float fx = me.ox, fy = me.oy, fz = me.oz;
      for (int dz = -SUB; dz <= SUB; ++dz) {
        const int z = me.cz + dz;
        if (z < 0 || z >= g.dim[2]) continue;
        const float gz = axisGap(dz, fz);
        const float dzc = (float)dz;
        for (int dy = -SUB; dy <= SUB; ++dy) {
          const int y = me.cy + dy;
          if (y < 0 || y >= g.dim[1]) continue;
          const float gy = axisGap(dy, fy);
          const float gyz = gy*gy + gz*gz;
          if (SUB > 1 && gyz > rc2) continue;
          const float dyc = (float)dy;
          const Row<SUB> row = loadRow<SUB>(M, g, me, y, z, fx, gyz, rc2);
          for (int32_t k = row.start; k < row.end; ++k) {
            if (k != s && candTest(M, a, me, k, rowDxc<SUB>(row, me, k), dyc, dzc, k2, k2lo, k2hi, pretest))
              accept(k);
          }
        }
      }
    }
    if (!FILL) {
      M.counts[i] = count;
      if (count > maxNbr) atomicOr(M.err, DERR_NBR_CAPACITY);
      if (lcap > 0) {
        const int64_t stride = M.grid.stashStride;
        if (count > lcap || s >= stride) {
          atomicOr(M.err, DERR_LIST_CAPACITY);
        } else {
          int32_t* stash = reinterpret_cast<int32_t*>(M.pacc);
          for (int c = 0; c < count; ++c) stash[c*stride + s] = lst[c*bd + tid];
        }
      }
    } else {
      const int64_t o = M.offsets[i];
      if (count > cap) atomicOr(M.err, DERR_LIST_CAPACITY);
      else if (o + count > M.ecap) atomicOr(M.err, DERR_ENTRY_CAPACITY);
      else for (int c = 0; c < count; ++c) M.nbr[o + c] = lst[c*bd + tid];
    }
  }
  if (!FILL) {
    int m = count;
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((tid & 31) == 0 && m > 0) atomicMax(reinterpret_cast<int*>(M.scal + SC_MAXCOUNT), m);
  }
  if (collect) {
    unsigned long long b = (unsigned long long)above;
    for (int o = 16; o > 0; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
    if ((tid & 31) == 0 && b) atomicAdd(reinterpret_cast<unsigned long long*>(M.scal + SC_PAIRS), b);
  }
}

// Stashed lists (thread schedule) to the CSR: thread per sorted slot, eight
// entries loaded before the first is stored (one after the other the loads'
// latency bound it; Kelvin-Helmholtz 128^3 60 -> 42 us).
__global__ void __launch_bounds__(256) nbr_compact_thread_kernel(const Member* mem, BlockMap bm) {
  const MemberBlock mb = memberBlock(bm);
  const Member& M = mem[mb.m];
  const int64_t s = mb.block*blockDim.x + threadIdx.x;
  if (s >= allNodes(M)) return;
  const int32_t i = M.sortedIdx[s];
  if (i >= M.n) return;
  const int count = M.counts[i];
  const int64_t stride = M.grid.stashStride;
  if (count > M.grid.stashCap || s >= stride) return;   // not stashed: the count pass flagged it
  const int64_t o = M.offsets[i];
  if (o + count > M.ecap) {
    atomicOr(M.err, DERR_ENTRY_CAPACITY);
    return;
  }
  const int32_t* stash = reinterpret_cast<const int32_t*>(M.pacc);
  int32_t* to = M.nbr + o;
  for (int base = 0; base < count; base += 8) {
    int32_t v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (base + u < count) v[u] = __ldg(stash + (base + u)*stride + s);
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (base + u < count) to[base + u] = v[u];
  }
}

// Stashed lists (warp schedule) to the CSR: warp per internal node, the list
// of node i at stash[i*stashCap : i*stashCap + count].  Four loads per lane in
// flight: Sod 256x32x32 121 -> 82 us (3 TB/s), 24 tubes 570 -> 410 us.
__global__ void __launch_bounds__(256) nbr_compact_warp_kernel(const Member* mem, BlockMap bm) {
  const MemberBlock mb = memberBlock(bm);
  const Member& M = mem[mb.m];
  const int lane = threadIdx.x & 31;
  const int64_t i = (mb.block*(int64_t)blockDim.x + threadIdx.x) >> 5;
  if (i >= M.n) return;
  const int count = M.counts[i];
  if (count > M.grid.stashCap) return;       // not stashed: the count pass flagged it
  const int64_t o = M.offsets[i];
  if (o + count > M.ecap) {
    if (lane == 0) atomicOr(M.err, DERR_ENTRY_CAPACITY);
    return;
  }
  const int32_t* stash = reinterpret_cast<const int32_t*>(M.pacc) + i*(int64_t)M.grid.stashCap;
  int32_t* to = M.nbr + o;
  for (int base = 0; base < count; base += 128) {
    int32_t v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int t = base + 32*u + lane;
      if (t < count) v[u] = __ldg(stash + t);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int t = base + 32*u + lane;
      if (t < count) to[t] = v[u];
    }
  }
}

// One warp walks the neighbouring cells of the node in sorted slot s (nothing
// for a ghost slot): apply the ConnectivityMap predicate, count (FILL=false)
// or collect, sort ascending and store (FILL=true) the neighbor indices.
// `cap` is the capacity of the warp's list sbuf (a power of two >= 32), R its
// row table.  A member with a stash (Grid::stashCap > 0) collects and sorts
// in the COUNT pass and stores the list of node i at stash[i*stashCap];
// nbr_compact_warp_kernel moves it to offsets[i].
template<int SUB>
struct RowTable {
  static constexpr int NR = (2*SUB + 1)*(2*SUB + 1);
  static constexpr int RW = 3 + 2*SUB;                // start, first candidate number, x0, cell ends
  int32_t v[NR*RW];
};

template<bool FILL, int SUB>
__device__ __forceinline__ void walkWarp(const Member& M, const Grid& g, int64_t s, int32_t* sbuf, int cap, int maxNbr,
                                      int32_t* R) {
  const int lane = threadIdx.x & 31;
  const int scap = FILL ? 0 : M.grid.stashCap;
  const bool collect = FILL || scap > 0;
  const NbrArrays a = nbrArrays(M);
  const Walker me = makeWalker(M, a, g, (int32_t)s);
  if (me.idx >= M.n) return;
  const int32_t i = me.idx;
  const double k2 = M.prm.kernelExtent*M.prm.kernelExtent;
  const float k2f = (float)k2;
  const bool pretest = g.filterTol > 0.0f;
  const float k2lo = k2f*(1.0f - g.filterTol), k2hi = k2f*(1.0f + g.filterTol);
  const float rc2 = reachBound2(g.reach, 1.0e-6f);
  const float fx = me.ox, fy = me.oy, fz = me.oz;
  // The window's rows, one per lane (rows outside the grid or, with SUB > 1,
  // beyond the kernel reach are empty), their candidates numbered in one
  // sequence by a warp scan: the lanes then take 32 consecutive candidates at
  // a time across row ends, so a warp iteration tests 32 candidates however
  // short the rows are.
  constexpr int NR = RowTable<SUB>::NR, RW = RowTable<SUB>::RW;
  int len = 0;
  if (lane < NR) {
    const int dy = lane % (2*SUB + 1) - SUB, dz = lane/(2*SUB + 1) - SUB;
    const int y = me.cy + dy, z = me.cz + dz;
    if (y >= 0 && y < g.dim[1] && z >= 0 && z < g.dim[2]) {
      const float gy = axisGap(dy, fy), gz = axisGap(dz, fz);
      const float gyz = gy*gy + gz*gz;
      if (SUB == 1 || gyz <= rc2) {
        const Row<SUB> row = loadRow<SUB>(M, g, me, y, z, fx, gyz, rc2);
        len = row.end > row.start ? row.end - row.start : 0;
        R[lane*RW] = row.start;
        R[lane*RW + 2] = row.x0;
#pragma unroll
        for (int c = 0; c < 2*SUB; ++c) R[lane*RW + 3 + c] = row.e[c];
      }
    }
  }
  int incl = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane < NR) R[lane*RW + 1] = incl - len;
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  __syncwarp();
  int count = 0;
  int r = 0;                                          // the lane's row (lanes only move forward)
  for (int base = 0; base < total; base += 32) {
    const int t = base + lane;
    bool pass = false;
    int32_t k = 0;
    if (t < total) {
      while (r + 1 < NR && R[(r + 1)*RW + 1] <= t) ++r;
      const int32_t* row = R + r*RW;
      k = row[0] + (t - row[1]);
      if (k != s) {
        int xc = row[2] - me.cx;
#pragma unroll
        for (int c = 0; c < 2*SUB; ++c) xc += (k >= row[3 + c]);
        const float dyc = (float)(r % (2*SUB + 1) - SUB), dzc = (float)(r/(2*SUB + 1) - SUB);
        pass = candTest(M, a, me, k, (float)xc, dyc, dzc, k2, k2lo, k2hi, pretest);
      }
    }
    const unsigned ballot = __ballot_sync(0xffffffffu, pass);
    if (collect && pass) {
      const int pos = count + __popc(ballot & ((1u << lane) - 1u));
      if (pos < cap) sbuf[pos] = __ldg(M.sortedIdx + k);
    }
    count += __popc(ballot);
  }
  if (!FILL) {
    if (lane == 0) {
      M.counts[i] = count;
      if (count > maxNbr) atomicOr(M.err, DERR_NBR_CAPACITY);
      atomicMax(reinterpret_cast<int*>(M.scal + SC_MAXCOUNT), count);
    }
    if (scap == 0) return;
    if (count > scap) {
      if (lane == 0) atomicOr(M.err, DERR_LIST_CAPACITY);
      return;
    }
  }
  const int64_t o = FILL ? M.offsets[i] : 0;
  if (FILL && (count > cap || o + count > M.ecap)) {
    if (lane == 0) atomicOr(M.err, count > cap ? DERR_LIST_CAPACITY : DERR_ENTRY_CAPACITY);
    return;
  }
  int32_t* out = FILL ? M.nbr + o : reinterpret_cast<int32_t*>(M.pacc) + i*(int64_t)scap;
  // bitonic sort of sbuf[0:count] (padded to a power of two)
  int size = 32;
  while (size < count) size <<= 1;
  for (int t = count + lane; t < size; t += 32) sbuf[t] = INT_MAX;
  __syncwarp();
  for (int k = 2; k <= size; k <<= 1) {
    for (int jj = k >> 1; jj > 0; jj >>= 1) {
      for (int t = lane; t < size; t += 32) {
        const int ixj = t ^ jj;
        if (ixj > t) {
          const int32_t u = sbuf[t], v = sbuf[ixj];
          const bool up = (t & k) == 0;
          if ((u > v) == up) { sbuf[t] = v; sbuf[ixj] = u; }
        }
      }
      __syncwarp();
    }
  }
  int above = 0;
  for (int t = lane; t < count; t += 32) {
    const int32_t j = sbuf[t];
    out[t] = j;
    above += (j > (int32_t)i);
  }
  for (int sh = 16; sh > 0; sh >>= 1) above += __shfl_xor_sync(0xffffffffu, above, sh);
  if (lane == 0 && above)
    atomicAdd(reinterpret_cast<unsigned long long*>(M.scal + SC_PAIRS), (unsigned long long)above);
}

// (a call of its own where a kernel's registers are meant for other work)
template<bool FILL>
__device__ __noinline__ void walkWarpCall(const Member& M, const Grid& g, int64_t s, int32_t* sbuf, int cap, int maxNbr,
                                          int32_t* R) {
  walkWarp<FILL, 1>(M, g, s, sbuf, cap, maxNbr, R);
}

// A warp per sorted slot (walkWarp), cells of half a kernel reach.
template<bool FILL>
__global__ void __launch_bounds__(256) nbr_walk_kernel(const Member* mem, BlockMap bm, int cap, int maxNbr) {
  extern __shared__ int32_t sbuf_all[];
  __shared__ RowTable<2> rows[256/32];
  const MemberBlock mb = memberBlock(bm);
  const Member& M = mem[mb.m];
  const int wib = threadIdx.x >> 5;
  const bool collect = FILL || M.grid.stashCap > 0;
  const int64_t s = (mb.block*(int64_t)blockDim.x + threadIdx.x) >> 5;
  if (s >= allNodes(M)) return;
  walkWarp<FILL, 2>(M, loadGrid(M), s, sbuf_all + (collect ? wib*cap : 0), cap, maxNbr, rows[wib].v);
}

// ---------------------------------------------------------------- cell walk
// A block per cell of one kernel reach: the candidates of the 27
// neighbouring cells are staged in shared memory once for all walkers of the
// cell, in node order, and each warp then tests them for four walkers at a
// time and appends the ones that pass with a ballot, so every list comes out
// ascending without a sort of its own.
//
// Why this split: a walker of the Sod tube (27 nodes per cell) has 743
// candidates for 115 neighbors.  With a warp per walker each of the 27
// walkers of a cell gathered the same candidates from L1/L2 and sorted its
// own list.  Here the gather and the ordering are shared by the cell, the
// candidates farther from the cell than the kernel reach are left out first
// (743 -> 570), and a test is a 16-byte shared-memory read and about twenty
// instructions for 32 candidates.  The cells' slots are brought into node
// order once (cell_order_kernel), so that a block only merges 27 sorted runs:
// along x, then y, then z, each element finding its rank by bisection in the
// two other runs.
//
// Measured (B200): Sod 256x32x32 (262,144 nodes, 115 neighbors) 680 us against
// 1,939 us with a warp per node; 24 tubes of the ensemble together 2.81 against
// 8.92 ms.  Bound by the latency of its steps between barriers (32 warps per
// SM, about half of the cycles issue): the merges' bisections, then the tests
// and the lists' stores.  Other forms, against 699 us at the time: the bisections
// in the two other runs one after the other and a warp per 32 elements of one
// run, 786 (the merges took 23,000 of a cell's 60,000 cycles); the 27 cells'
// loads ahead of the first test, 786 (the registers spill); a list's places from
// a scan of its words' counts instead of one after the other, 702.
constexpr int kCellThreads = 256;
constexpr int kCellWarps = kCellThreads/32;
constexpr int kCellCand = 1536;                        // nodes of the 27 cells that can be staged (more: crowded)
constexpr int kCellTest = 1024;                        // of them within the reach of the cell: a ballot word per lane
constexpr int kCellSort = 128;                         // nodes of a cell kept in node order (more: crowded)
constexpr int kWalkers = 4;                            // walkers a warp tests at a time
constexpr int64_t kCellBlocks = 148*16;                // blocks of a member, at most

// The slots of one cell into node order (a warp per cell, 32*E >= its nodes).
template<int E>
__device__ __forceinline__ void orderCell(const Member& M, int32_t s0, int count) {
  double* base = static_cast<double*>(M.cand);
  float4* pre = reinterpret_cast<float4*>(base);
  float* lmax = reinterpret_cast<float*>(base + 2*M.candcap);
  const int lane = threadIdx.x & 31;
  int32_t key[E];
  float4 p[E];
  float lm[E];
  int rank[E];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int t = 32*e + lane;
    key[e] = t < count ? M.sortedIdx[s0 + t] : INT_MAX;
    if (t < count) { p[e] = pre[s0 + t]; lm[e] = lmax[s0 + t]; }
    rank[e] = 0;
  }
  for (int l = 0; l < 32; ++l) {
#pragma unroll
    for (int f = 0; f < E; ++f) {
      const int32_t o = __shfl_sync(0xffffffffu, key[f], l);
#pragma unroll
      for (int e = 0; e < E; ++e) rank[e] += o < key[e];
    }
  }
  __syncwarp();
#pragma unroll
  for (int e = 0; e < E; ++e) {
    if (32*e + lane >= count) continue;
    M.sortedIdx[s0 + rank[e]] = key[e];
    pre[s0 + rank[e]] = p[e];
    lmax[s0 + rank[e]] = lm[e];
  }
}

__global__ void __launch_bounds__(256) cell_order_kernel(const Member* mem, BlockMap bm) {
  const MemberBlock mb = memberBlock(bm);
  const Member& M = mem[mb.m];
  const int64_t ncells = scalI(M.scal, SC_NCELLS);
  const int64_t stride = (int64_t)mb.blocks*(blockDim.x >> 5);
  for (int64_t c = mb.block*(blockDim.x >> 5) + (threadIdx.x >> 5); c < ncells; c += stride) {
    const int32_t s0 = (int32_t)M.cellStart[c];
    const int count = (int)M.cellStart[c + 1] - s0;
    if (count < 2 || count > kCellSort) continue;
    if (count <= 32) orderCell<1>(M, s0, count);
    else if (count <= 64) orderCell<2>(M, s0, count);
    else orderCell<kCellSort/32>(M, s0, count);
  }
}

// Elements below k of the ascending runs a[0 : la) and b[0 : lb), summed (the
// two bisections' reads overlap).
__device__ __forceinline__ int rankInTwo(const int32_t* a, int la, const int32_t* b, int lb, int32_t k) {
  int x = 0, y = 0;
  const int most = la > lb ? la : lb;
  for (int w = most > 0 ? 1 << (31 - __clz(most)) : 0; w > 0; w >>= 1) {
    const bool ga = x + w <= la && a[x + w - 1] < k, gb = y + w <= lb && b[y + w - 1] < k;
    x += ga ? w : 0;
    y += gb ? w : 0;
  }
  return x + y;
}

// Merge of the ascending runs 3g, 3g + 1, 3g + 2 (run r at [start[r],
// start[r + 1])) of every g from (key, src) to (keyTo, srcTo), each element at
// the rank it has among the three.
// own (the last merge): the final place of the element staged at ownAt + m
// goes to own[m], m < ownLen.
template<int RUNS>
__device__ __forceinline__ void mergeRuns(const int32_t* key, const uint16_t* src, int32_t* keyTo, uint16_t* srcTo,
                                          const int* start, uint16_t* own = nullptr, int ownAt = 0, int ownLen = 0) {
  const int count = start[RUNS];
  for (int t = threadIdx.x; t < count; t += kCellThreads) {
    int r = 0;
#pragma unroll
    for (int q = 1; q < RUNS; ++q) r += start[q] <= t;
    const int g = r - r % 3;
    const int o1 = r == g ? g + 1 : g, o2 = r == g + 2 ? g + 1 : g + 2;
    const int a1 = start[o1], a2 = start[o2];
    const int32_t k = key[t];
    const uint16_t from = src[t];
    const int to = start[g] + (t - start[r]) +
                   rankInTwo(key + a1, start[o1 + 1] - a1, key + a2, start[o2 + 1] - a2, k);
    keyTo[to] = k;
    srcTo[to] = from;
    if (own != nullptr && (unsigned)(from - ownAt) < (unsigned)ownLen) own[from - ownAt] = (uint16_t)to;
  }
}

// The walker's side of the test (lengths in cells).
struct CellWalker {
  float x, y, z;
  float T;             // r^2 above both nodes' T: not neighbors
  float A;             // r^2 at most either node's A: neighbors
  int32_t idx;
};

// A pair between the bounds: the FP32 form of H_i, then the exact test.
__device__ __noinline__ bool cellUndecided(const Member& M, int32_t i, int32_t j, double cell, float fx, float fy,
                                           float fz, float cT, double k2, float k2lo, float k2hi, bool pretest) {
  if (pretest) {
    const Sym H = nodeH(M, i);
    const float hf[6] = {(float)(H.xx*cell), (float)(H.xy*cell), (float)(H.xz*cell),
                         (float)(H.yy*cell), (float)(H.yz*cell), (float)(H.zz*cell)};
    const float r2 = __fmaf_rn(fx, fx, __fmaf_rn(fy, fy, fz*fz));
    const float e2i = symEta2F(hf, fx, fy, fz);
    if (e2i <= k2lo) return true;
    if (e2i > k2hi && r2 > cT) return false;
  }
  return exactTest(M, i, j, k2);
}

struct CellShared {
  float4 pre[kCellCand];            // offsets from the cell's corner, T
  float acc[kCellCand];             // A
  int32_t key[2][kCellCand];        // node index
  uint16_t src[2][kCellCand];       // position in pre before the merges
  uint16_t own[kCellSort];          // place of the cell's own nodes after the merges
};

template<bool FILL>
__global__ void __launch_bounds__(kCellThreads, 4) nbr_cell_kernel(const Member* mem, BlockMap bm, int cap, int maxNbr) {
  extern __shared__ float4 cellSmem[];
  CellShared& sh = *reinterpret_cast<CellShared*>(cellSmem);
  __shared__ int32_t cellS0[27];
  __shared__ int cellLen[27], cellAt[28];       // staged nodes of each cell, their first position
  __shared__ int rowAt[10], planeAt[4];
  __shared__ int crowded, listAt;
  const MemberBlock mb = memberBlock(bm);
  const Member& M = mem[mb.m];
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  const int64_t n = M.n;
  const NbrArrays a = nbrArrays(M);
  const int ncells = (int)scalI(M.scal, SC_NCELLS);   // at most 2^26 (grid_kernel)
  const int scap = FILL ? 0 : M.grid.stashCap;
  const double k2 = M.prm.kernelExtent*M.prm.kernelExtent;
  const float filterTol = (float)M.scal[SC_GRID + 7];
  const float k2f = (float)k2;
  const bool pretest = filterTol > 0.0f;
  const float k2lo = k2f*(1.0f - filterTol), k2hi = k2f*(1.0f + filterTol);
  const double cell = M.scal[SC_GRID + 3];
  const int dim0 = (int)scalI(M.scal, SC_GRID + 4), dim1 = (int)scalI(M.scal, SC_GRID + 5),
            dim2 = (int)scalI(M.scal, SC_GRID + 6);
  // no candidate farther than the largest kernel reach can pass (the slack
  // covers the FP32 offsets and a walker at the tolerance of `outside`)
  const float reach2 = reachBound2((float)M.scal[SC_REACH], 1.2e-5f);
  int most = 0;
  unsigned above = 0;
  for (int c = (int)mb.block; c < ncells; c += mb.blocks) {
    const int32_t s0 = (int32_t)M.cellStart[c], s1 = (int32_t)M.cellStart[c + 1];
    // (also the barrier between the last cell's tests and this one's staging)
    bool any = false, outside = false;
    for (int32_t s = s0 + tid; s < s1; s += kCellThreads) {
      if (M.sortedIdx[s] >= n) continue;
      any = true;
      // a node clamped into the grid's outermost cells may lie outside its cell
      const float4 p = a.pre[s];
      const float lo = -1.0e-5f, hi = 1.00001f;
      outside = outside || fminf(p.x, fminf(p.y, p.z)) < lo || fmaxf(p.x, fmaxf(p.y, p.z)) > hi;
    }
    if (!__syncthreads_or(any)) continue;
    if (tid == 0) crowded = 0;
    const float rc2 = __syncthreads_or(outside) ? CUDART_INF_F : reach2;
    const int cyz = c/dim0, cx = c - cyz*dim0, cz = cyz/dim1, cy = cyz - cz*dim1;
    if (wib == 0) {
      // the 27 cells, x fastest: first slot and nodes, and an upper bound of each run's position
      int len = 0;
      if (lane < 27) {
        const int x = cx + lane % 3 - 1, y = cy + (lane/3) % 3 - 1, z = cz + lane/9 - 1;
        int32_t first = 0;
        if (x >= 0 && x < dim0 && y >= 0 && y < dim1 && z >= 0 && z < dim2) {
          const int64_t* cs = M.cellStart + ((int64_t)z*dim1 + y)*dim0 + x;
          first = (int32_t)cs[0];
          len = (int)cs[1] - first;
        }
        cellS0[lane] = first;
        cellLen[lane] = len;
        if (len > kCellSort) crowded = 1;
      }
      int incl = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      if (lane < 28) cellAt[lane] = incl - len;
      if (lane == 31 && incl > kCellCand) crowded = 1;
    }
    __syncthreads();
    // too many to stage or to merge: a warp per walker, its list sorted by itself
    // (nbr_crowded_kernel; the fill pass has the counting pass's list)
    auto walkAlone = [&]() {
      if (!FILL) {
        if (tid == 0) listAt = (int)atomicAdd(reinterpret_cast<unsigned long long*>(M.scal + SC_CROWDED),
                                              (unsigned long long)(s1 - s0));
        __syncthreads();
        if (M.grid.crowdList) for (int32_t s = s0 + tid; s < s1; s += kCellThreads) M.cidx[listAt + (s - s0)] = s;
      }
      if (M.grid.crowdList) return;
      int32_t* rows = reinterpret_cast<int32_t*>(cellSmem) + wib*(cap + RowTable<1>::NR*RowTable<1>::RW);
      const Grid g = loadGrid(M);
      for (int32_t s = s0 + wib; s < s1; s += kCellWarps) {
        walkWarpCall<FILL>(M, g, s, rows + RowTable<1>::NR*RowTable<1>::RW, cap, maxNbr, rows);
        __syncwarp();
      }
    };
    if (crowded) { walkAlone(); continue; }
    // stage the cells, a warp each: offsets from this cell's corner; the
    // nodes beyond the reach of this cell's box left out
    for (int q = wib; q < 27; q += kCellWarps) {
      const int len = cellLen[q], at = cellAt[q];
      const int32_t first = cellS0[q];
      const float ox = (float)(q % 3 - 1), oy = (float)((q/3) % 3 - 1), oz = (float)(q/9 - 1);
      int kept = 0;
      for (int base = 0; base < len; base += 32) {
        const int t = base + lane;
        bool keep = false;
        float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (t < len) {
          p = a.pre[first + t];
          p.x += ox; p.y += oy; p.z += oz;
          const float gx = fmaxf(fmaxf(-p.x, p.x - 1.0f), 0.0f), gy = fmaxf(fmaxf(-p.y, p.y - 1.0f), 0.0f),
                      gz = fmaxf(fmaxf(-p.z, p.z - 1.0f), 0.0f);
          keep = q == 13 || gx*gx + gy*gy + gz*gz <= rc2;   // (the own nodes' places follow their slots)
        }
        const unsigned bal = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          const int pos = at + kept + __popc(bal & ((1u << lane) - 1u));
          const float lm = a.lmax[first + t];
          sh.pre[pos] = p;
          sh.acc[pos] = pretest ? __fdividef(k2lo, lm*lm) : -1.0f;
          sh.key[0][pos] = M.sortedIdx[first + t];
        }
        kept += __popc(bal);
      }
      if (lane == 0) cellLen[q] = kept;
    }
    __syncthreads();
    // rows: three cells along x each, closed up
    if (tid < 10) {
      int at = 0;
      for (int q = 0; q < 3*tid; ++q) at += cellLen[q];
      rowAt[tid] = at;
      if (tid % 3 == 0) planeAt[tid/3] = at;
    }
    __syncthreads();
    const int count = rowAt[9];
    if (count > kCellTest) { walkAlone(); continue; }
    for (int q = wib; q < 27; q += kCellWarps) {
      const int len = cellLen[q], at = cellAt[q], r = q/3, o1 = 3*r + (q + 1) % 3, o2 = 3*r + (q + 2) % 3;
      for (int t = lane; t < len; t += 32) {
        const int32_t k = sh.key[0][at + t];
        const int to = rowAt[r] + t + rankInTwo(sh.key[0] + cellAt[o1], cellLen[o1], sh.key[0] + cellAt[o2], cellLen[o2], k);
        sh.key[1][to] = k;
        sh.src[1][to] = (uint16_t)(at + t);
      }
    }
    __syncthreads();
    mergeRuns<9>(sh.key[1], sh.src[1], sh.key[0], sh.src[0], rowAt);
    __syncthreads();
    mergeRuns<3>(sh.key[0], sh.src[0], sh.key[1], sh.src[1], planeAt, sh.own, cellAt[13], cellLen[13]);
    __syncthreads();
    const int32_t* key = sh.key[1];
    const uint16_t* src = sh.src[1];
    const unsigned mine = 1u << lane, below = mine - 1u;
    // kWalkers walkers per warp at a time
    for (int32_t s = s0 + kWalkers*wib; s < s1; s += kWalkers*kCellWarps) {
      CellWalker w[kWalkers];
      int cnt[kWalkers];
      bool some = false;
#pragma unroll
      for (int q = 0; q < kWalkers; ++q) {
        cnt[q] = 0;
        const int32_t i = s + q < s1 ? M.sortedIdx[s + q] : -1;
        const bool on = i >= 0 && i < n;
        some = some || on;
        const float4 p = a.pre[on ? s + q : s0];
        const float lm = a.lmax[on ? s + q : s0];
        // an empty place tests like any other and is not stored; without the
        // pre-test every candidate is left to the exact test
        w[q] = CellWalker{p.x, p.y, p.z, pretest ? p.w : CUDART_INF_F, pretest ? __fdividef(k2lo, lm*lm) : -1.0f, on ? i : -1};
      }
      if (!some) continue;
      const int batches = (count + 31) >> 5;              // at most 32
      // the last batch's places that hold a candidate
      const unsigned filled = 0xffffffffu >> (32*batches - count);
      // the batch's ballots, kept by the lane of the batch's number
      unsigned sure[kWalkers], open[kWalkers];
#pragma unroll
      for (int q = 0; q < kWalkers; ++q) { sure[q] = 0; open[q] = 0; }
      for (int b = 0; b < batches; ++b) {
        const int t = 32*b + lane;
        const int at = src[t < count ? t : count - 1];
        const float4 cnd = sh.pre[at];
        const float cA = sh.acc[at];
#pragma unroll
        for (int q = 0; q < kWalkers; ++q) {
          const float fx = w[q].x - cnd.x, fy = w[q].y - cnd.y, fz = w[q].z - cnd.z;
          const float r2 = __fmaf_rn(fx, fx, __fmaf_rn(fy, fy, fz*fz));
          const unsigned in = __ballot_sync(0xffffffffu, r2 <= fmaxf(w[q].A, cA));
          const unsigned near = __ballot_sync(0xffffffffu, r2 <= fmaxf(w[q].T, cnd.w));
          if (lane == b) { sure[q] = in; open[q] = near & ~in; }
        }
      }
#pragma unroll
      for (int q = 0; q < kWalkers; ++q) {
        const int32_t i = w[q].idx;
        if (i < 0) continue;
        if (lane == batches - 1) { sure[q] &= filled; open[q] &= filled; }
        // the walker itself is no neighbor
        const int self = sh.own[s + q - s0];
        if (self >> 5 == lane) { sure[q] &= ~(1u << (self & 31)); open[q] &= ~(1u << (self & 31)); }
        // pairs between the bounds, each lane its own batch's
        while (open[q]) {
          const int bit = __ffs(open[q]) - 1;
          open[q] &= open[q] - 1;
          const int t = 32*lane + bit, at = src[t];
          if (cellUndecided(M, i, key[t], cell, w[q].x - sh.pre[at].x, w[q].y - sh.pre[at].y, w[q].z - sh.pre[at].z,
                            sh.pre[at].w, k2, k2lo, k2hi, pretest))
            sure[q] |= 1u << bit;
        }
        __syncwarp();
        int32_t* out = nullptr;
        int lim = 0;
        if (FILL) {
          const int64_t o = M.offsets[i];
          lim = M.counts[i];
          out = M.nbr + o;
          if (o + lim > M.ecap) {
            if (lane == 0) atomicOr(M.err, DERR_ENTRY_CAPACITY);
            lim = 0;
          }
        } else if (scap > 0) {
          out = reinterpret_cast<int32_t*>(M.pacc) + i*(int64_t)scap;
          lim = scap;
        }
        // neighbors after the walker in node order: its own pairs
        const int before = 32*lane <= self ? self - 32*lane : 0;
        above += __popc(before >= 32 ? 0u : sure[q] >> before);
        if (lim > 0) {
          for (int b = 0; b < batches; ++b) {
            const unsigned word = __shfl_sync(0xffffffffu, sure[q], b);
            const int pos = cnt[q] + __popc(word & below);
            if ((word & mine) && pos < lim) out[pos] = key[32*b + lane];
            cnt[q] += __popc(word);
          }
        } else {
          cnt[q] += __reduce_add_sync(0xffffffffu, __popc(sure[q]));
        }
      }
      if (!FILL) {
#pragma unroll
        for (int q = 0; q < kWalkers; ++q) {
          if (w[q].idx < 0) continue;
          if (lane == 0) {
            M.counts[w[q].idx] = cnt[q];
            if (cnt[q] > maxNbr) atomicOr(M.err, DERR_NBR_CAPACITY);
            if (scap > 0 && cnt[q] > scap) atomicOr(M.err, DERR_LIST_CAPACITY);
          }
          most = cnt[q] > most ? cnt[q] : most;
        }
      }
    }
  }
  // the pairs of this pass's lists (a counting pass without lists leaves them to the fill pass)
  unsigned long long pairs = FILL || scap > 0 ? above : 0;
  for (int o = 16; o > 0; o >>= 1) pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
  if (lane == 0) {
    if (!FILL && most > 0) atomicMax(reinterpret_cast<int*>(M.scal + SC_MAXCOUNT), most);
    if (pairs) atomicAdd(reinterpret_cast<unsigned long long*>(M.scal + SC_PAIRS), pairs);
  }
}

// The slots of the cell walk's crowded cells (listed in cidx, which is free
// after the counting sort), a warp each over the whole grid.
//
// Why: the cell's own block has eight warps for them, so a problem whose nodes
// lie in a few cells, or in one clump, would leave most of the chip idle behind
// chains of dozens of walks.  The launch is left out while no build has seen a
// crowded cell (Problem::crowd).  One slot a warp: in a loop over the list on a
// fixed grid the walk is 20% slower (64^3 nodes at 216 a cell 20.2 against 16.8 ms).
// Measured (B200, whole build, the cell's block -> the list): 16^3 nodes at nPerh 3
// 6.1 -> 0.7 ms, 64^3 nodes with 4,000 of them in a clump 12.0 -> 2.4 ms.
template<bool FILL>
__global__ void __launch_bounds__(256, 3) nbr_crowded_kernel(const Member* mem, BlockMap bm, int cap, int maxNbr) {
  extern __shared__ int32_t sbuf_all[];
  __shared__ RowTable<1> rows[256/32];
  const MemberBlock mb = memberBlock(bm);
  const Member& M = mem[mb.m];
  const int wib = threadIdx.x >> 5;
  const bool collect = FILL || M.grid.stashCap > 0;
  const int64_t w = (mb.block*(int64_t)blockDim.x + threadIdx.x) >> 5;
  if (w >= scalI(M.scal, SC_CROWDED)) return;
  walkWarp<FILL, 1>(M, loadGrid(M), M.cidx[w], sbuf_all + (collect ? wib*cap : 0), cap, maxNbr, rows[wib].v);
}


int64_t grow(int64_t v) { return v + v/4 + 1024; }

// Cells of one kernel reach of the last build's grid (0: no build yet).
double reach_cells(const Problem& p) {
  const int sub = p.lastNbrCells > 0 ? p.lastNbrCells : 1;
  return p.cellsWanted > 0 ? (double)p.cellsWanted/(double)(sub*sub*sub) : 0.0;
}

// Capacities for the next build, from the previous one (or first estimates).
// captured: for a graph that replays the build.
int plan_capacities(Batch& b, bool captured = false) {
  for (Problem* pp : b.mem) {
    Problem& p = *pp;
    const int64_t oldg = p.gcap, oldc = p.candcap, olde = p.ecap, oldcells = p.cellcap;
    // sizes of the last build, else the caller's hints, else built-in guesses
    const int64_t G = p.G > 0 ? p.G : p.hintG;
    const int64_t E = p.E > 0 ? p.E : p.hintE;
    if (G > 0) SPH_TRY(ensure_capacity_ghosts(p, grow(G)));
    // schedule: the cell walk (half-reach cells: a warp per node) once the
    // 27-cell candidate set of the last build kept 32 lanes busy, or once a thread's list would not fit in
    // shared memory
    const double cells1 = reach_cells(p);
    const double candPerNode = cells1 > 0.0 ? 27.0*(double)(p.n + p.G)/cells1 : 0.0;
    const int req = p.nbrSchedule != NBR_SCHEDULE_AUTO ? p.nbrSchedule : b.nbrSchedule;
    p.fillSchedule = (req == NBR_SCHEDULE_WARP || (req == NBR_SCHEDULE_AUTO && candPerNode > 384.0) ||
                      sizeof(int32_t)*32*(size_t)(p.fillCap > 8 ? p.fillCap : 64) > kMaxListSmem)
                         ? NBR_SCHEDULE_WARP : NBR_SCHEDULE_THREAD;
    // cells per kernel reach: one unless requested (half-reach cells test
    // fewer candidates but walk more rows; the autotuner measures both) or a
    // quarter of the slots lay in cells too crowded for the cell walk: half-reach
    // cells have no such limit.  Measured (B200, lattice 64^3, build): nPerh 1.8
    // (47 nodes a cell) cell walk 1.25 ms, half-reach cells 2.79; 1.85 (51) 4.41 with the
    // crowded cells' list, 2.82; nPerh 3 (216) 24.0, 14.3
    const int reqCells = p.nbrCells != 0 ? p.nbrCells : b.nbrCells;
    if (candPerNode < 0.8*p.denseSet) p.denseSet = 0.0;
    p.grid.sub = reqCells != 0 ? reqCells : (p.fillSchedule == NBR_SCHEDULE_WARP && p.denseSet > 0.0 ? 2 : 1);
    // (before the first cell walk an eager build lists what it finds; a captured
    // one would launch the empty list in every replay: its first replay tells)
    const bool cellWalk = p.fillSchedule == NBR_SCHEDULE_WARP && p.grid.sub == 1;
    p.grid.crowdList = cellWalk && (p.crowd > 0 || (p.crowd < 0 && !captured)) ? 1 : 0;
    const int sub = p.grid.sub;
    // cells the grid wants at this subdivision (the last build's, rescaled), else the hint
    const int64_t cells = cells1 > 0.0 ? (int64_t)(cells1*sub*sub*sub) + 1 : p.hintCells;
    // grow (with slack) when the buffers hold less than the wanted cells, and
    // once when the first measured count replaces the first build's guess (so
    // that a later small drift of h does not reallocate mid-run)
    const int64_t cellsNeed = cells > 0 ? grow(cells) : p.candcap/2 + 64;
    const int64_t cellsMin = cells > 0 ? cells + cells/32 + 64 : cellsNeed;
    const bool firstMeasured = cells > 0 && !p.cellsMeasured;
    if (cells > 0) p.cellsMeasured = true;
    if (cellsMin + 1 > p.cellcap || (firstMeasured && cellsNeed + 1 > p.cellcap)) {
      cudaStreamSynchronize(b.stream);
      void* old[] = {p.cellStart, p.cellFill};
      dev_free_all(old, 2);
      p.cellStart = nullptr; p.cellFill = nullptr;
      p.cellcap = cellsNeed + 1;
      if (dev_alloc(reinterpret_cast<void**>(&p.cellStart), sizeof(int64_t)*(p.cellcap + 1)) != cudaSuccess ||
          dev_alloc(reinterpret_cast<void**>(&p.cellFill), sizeof(int32_t)*p.cellcap) != cudaSuccess) {
        p.cellcap = 0;
        set_error("cell list allocation failed");
        return SPHGPU_ERR_NOMEM;
      }
    }
    // without a hint the first build guesses 32 entries per node; an overflow redoes it
    SPH_TRY(ensure_capacity_entries(p, E > 0 ? E + E/8 : 32*p.n));
    if (p.fillCap < 8) p.fillCap = p.maxCount > 0 ? p.maxCount + p.maxCount/4 + 8 : 64;
    if (kScanBlocks + 1 > p.blockSumsCap) SPH_TRY(ensure_block_sums(p, kScanBlocks + 1));
    if (p.gcap != oldg || p.candcap != oldc || p.ecap != olde || p.cellcap != oldcells) b.memDirty = true;
    if (p.fillSchedule == NBR_SCHEDULE_THREAD && sizeof(int32_t)*32*(size_t)p.fillCap > kMaxListSmem)
      p.fillSchedule = NBR_SCHEDULE_WARP;
    p.grid.filterTol = p.nbrFilter ? kFilterTol : 0.0f;
    // single pass: the lists go to the pair-acceleration buffer (free until
    // the next derivative evaluation rewrites it) when they fit there
    // (thread schedule: one row per sorted slot, internal and ghost, sized
    // from the last build's ghosts; a slot beyond it flags the build for a redo)
    const int64_t rows = G > 0 ? p.n + grow(G) : p.candcap;
    p.grid.stashStride = rows < p.candcap ? rows : p.candcap;
    const int64_t slots = p.fillSchedule == NBR_SCHEDULE_WARP ? p.n : p.grid.stashStride;
    p.grid.stashCap = (p.pacc != nullptr && p.nbrStash && (int64_t)p.fillCap*slots <= 6*p.ecap) ? p.fillCap : 0;
  }
  b.memDirty = true;
  return SPHGPU_OK;
}

}  // namespace

// Mirrors the capacity rules a new problem goes through: sphgpu_create sizes
// the ghost and (n + ghost) buffers for n/2 + 4096 ghosts, plan_capacities
// grows them from the planned sizes, ensure_capacity_* add their own slack,
// and the mixed and CRKSPH records follow the (n + ghost) capacity.
int64_t planned_bytes(const sphgpu_config& cfg, int64_t n, int64_t G, int64_t E, int64_t ncells) {
  auto ghostCap = [](int64_t need) { return need + need/2 + 1024; };  // ensure_capacity_ghosts
  Problem p;
  p.cfg = cfg;
  p.n = n;
  p.prm.W.n = cfg.num_points;
  p.gcap = ghostCap(n/2 + 4096);
  if (G > 0 && grow(G) > p.gcap) p.gcap = ghostCap(grow(G));
  p.candcap = n + p.gcap;
  p.cellcap = (ncells > 0 ? grow(ncells) : p.candcap/2 + 64) + 1;
  const int64_t eneed = E > 0 ? E + E/8 : 32*n;
  p.ecap = eneed + eneed/8 + 1024;                                       // ensure_capacity_entries
  p.blockSumsCap = kScanBlocks + 1 + 64;                                // ensure_block_sums
  if (cfg.precision == SPHGPU_PRECISION_MIXED) p.mreccap = p.candcap;
  if (cfg.hydro == SPHGPU_HYDRO_CRKSPH) p.creccap = p.candcap;
  double marker = 0.0;                          // problem_bytes only tests these for null
  if (cfg.compatibleEnergyEvolution) p.pacc = &marker;
  if (cfg.precision == SPHGPU_PRECISION_MIXED) p.coefF = reinterpret_cast<float*>(&marker);
  if (cfg.hydro == SPHGPU_HYDRO_CRKSPH) { p.K = &marker; p.Kheld = &marker; }
  const int64_t b = problem_bytes(p);
  p.pacc = nullptr; p.coefF = nullptr; p.K = nullptr; p.Kheld = nullptr;
  return b;
}

namespace {

// Grid of the fused ghost passes: every block must be resident at once.
int fused_ghost_grid() {
  static int grid = -1;
  if (grid < 0) {
    int dev = 0, sms = 0, occ = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, ghost_passes_fused_kernel, kRootThreads, 0) != cudaSuccess) {
      cudaGetLastError();
      grid = 0;
    } else {
      grid = sms*occ < kFusedGhostBlocks ? sms*occ : kFusedGhostBlocks;
    }
  }
  return grid;
}

// The fused passes for this build: by the schedule, or (automatic) for a
// batch of at most kFusedGhostMembers members.  Their scratch is allocated
// outside a capture; a captured build without it takes the per-pass launches.
bool use_fused_ghost_passes(Batch& b) {
  const int nm = (int)b.mem.size();
  if (b.ghostPasses == 1 || nm > kFusedGhostMembers || fused_ghost_grid() <= 0) return false;
  if (b.d_fuse == nullptr) {
    if (b.capturing) return false;
    const size_t bytes = 2*sizeof(unsigned int) + sizeof(int)*(size_t)kFusedGhostMembers*kGhostCodes*kFusedGhostBlocks;
    if (dev_alloc(reinterpret_cast<void**>(&b.d_fuse), bytes) != cudaSuccess) { cudaGetLastError(); return false; }
    if (cudaMemset(b.d_fuse, 0, bytes) != cudaSuccess) { cudaGetLastError(); return false; }
  }
  return true;
}

int launch_fused_ghost_passes(Batch& b) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3((unsigned)fused_ghost_grid());
  lc.blockDim = dim3(kRootThreads);
  lc.dynamicSmemBytes = 0;
  lc.stream = b.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  lc.attrs = attr;
  lc.numAttrs = 1;
  const int nm = (int)b.mem.size();
  return cuda_status(cudaLaunchKernelEx(&lc, ghost_passes_fused_kernel, (const Member*)b.d_mem, nm, b.d_fuse),
                     "fused ghost passes");
}

int launch_build(Batch& b) {
  cudaStream_t st = b.stream;
  const int nm = (int)b.mem.size();
  for (Problem* p : b.mem) p->paccReady = false;   // the walk parks its lists in pacc
  // (a captured build reads the descriptor slot uploaded before the capture)
  if (!b.capturing && !b.buildPlanned) SPH_TRY(batch_upload(b));
  b.buildPlanned = false;
  // ---- ghosts: six planar boundaries in order, sizes kept on the device
  // fixed grids: at most kStreamBlocks blocks per member, member-local stride
  auto fixedItems = [](int64_t cap) { return cap < kStreamBlocks*kGhostThreads ? cap : kStreamBlocks*kGhostThreads; };
  BlockMap nmap, cap;
  unsigned ngrid = 0, capGrid = 0;
  SPH_TRY(batch_map_items(b, [&](const Problem& p) { return fixedItems(p.n); }, kGhostThreads, &nmap, &ngrid));
  SPH_TRY(batch_map_items(b, [&](const Problem& p) { return fixedItems(p.candcap); }, kGhostThreads, &cap, &capGrid));
  bool anyPeriodic = false;
  for (Problem* p : b.mem) for (int a = 0; a < 3; ++a) anyPeriodic = anyPeriodic || p->prm.bcs.periodic[a];
  bool small = b.ghostPasses == 0;
  for (Problem* p : b.mem) small = small && p->n <= kClusterNodes;
  if (small) {
    // (the first pass's schedule value: all six passes in one launch)
    if (anyPeriodic) b.lastGhostPasses = 2;
    ghost_cluster_kernel<<<nm*kClusterBlocks, kClusterThreads, 0, st>>>(b.d_mem); batch_count_launch(b);
  } else {
    build_init_kernel<<<(nm + 127)/128, 128, 0, st>>>(b.d_mem, nm); batch_count_launch(b);
    if (ngrid) { node_hmax_kernel<<<ngrid, kGhostThreads, 0, st>>>(b.d_mem, nmap); batch_count_launch(b); }
    if (anyPeriodic) {
      // the boundary passes visit only the internal nodes near a periodic plane
      near_flag_kernel<<<ngrid, kGhostThreads, 0, st>>>(b.d_mem, nmap); batch_count_launch(b);
      SPH_TRY(batch_scan(b, SCAN_COUNTS));
      near_list_kernel<<<ngrid, kGhostThreads, 0, st>>>(b.d_mem, nmap); batch_count_launch(b);
    }
    const bool fused = anyPeriodic && use_fused_ghost_passes(b);
    if (anyPeriodic) b.lastGhostPasses = fused ? 2 : 1;
    if (fused) {
      // (the barrier's arrival counter is back at zero after every completed
      // barrier; a build that reported a timed-out barrier clears it)
      SPH_TRY(launch_fused_ghost_passes(b));
      batch_count_launch(b);
    }
    for (int bnd = 0; bnd < 6 && !fused; ++bnd) {
      bool any = false;
      for (Problem* p : b.mem) any = any || p->prm.bcs.periodic[bnd >> 1];
      if (!any) continue;
      ghost_hmax_kernel<<<capGrid, kGhostThreads, 0, st>>>(b.d_mem, cap, bnd); batch_count_launch(b);
      ghost_flag_kernel<<<capGrid, kGhostThreads, 0, st>>>(b.d_mem, cap, bnd); batch_count_launch(b);
      SPH_TRY(batch_scan(b, SCAN_FLAGS));
      ghost_scatter_kernel<<<capGrid, kGhostThreads, 0, st>>>(b.d_mem, cap, bnd); batch_count_launch(b);
      ghost_advance_kernel<<<(nm + 127)/128, 128, 0, st>>>(b.d_mem, nm); batch_count_launch(b);
    }
    grid_kernel<<<(nm + 127)/128, 128, 0, st>>>(b.d_mem, nm); batch_count_launch(b);
  }
  // ---- counting sort of all nodes by cell
  BlockMap cm;
  unsigned cgrid = 0;
  SPH_TRY(batch_map_items(b, [&](const Problem& p) { return fixedItems(p.cellcap); }, kGhostThreads, &cm, &cgrid));
  cell_zero_kernel<<<cgrid, kGhostThreads, 0, st>>>(b.d_mem, cm); batch_count_launch(b);
  cell_index_kernel<<<capGrid, kGhostThreads, 0, st>>>(b.d_mem, cap); batch_count_launch(b);
  SPH_TRY(batch_scan(b, SCAN_CELLS));
  cell_zero_kernel<<<cgrid, kGhostThreads, 0, st>>>(b.d_mem, cm); batch_count_launch(b);
  cell_scatter_kernel<<<capGrid, kGhostThreads, 0, st>>>(b.d_mem, cap); batch_count_launch(b);
  // ---- neighbor counts, offsets, lists
  int maxNbr = 0, tcap = 1, wmax = 0;
  bool tstash = false, wstash = false, alone = false;
  for (Problem* p : b.mem) {
    maxNbr = p->maxNbr > maxNbr ? p->maxNbr : maxNbr;
    if (p->fillSchedule == NBR_SCHEDULE_WARP) {
      wmax = p->fillCap > wmax ? p->fillCap : wmax;
      wstash = wstash || p->grid.stashCap > 0;
      alone = alone || p->grid.crowdList == 0;
    } else {
      tcap = p->fillCap > tcap ? p->fillCap : tcap;
      tstash = tstash || p->grid.stashCap > 0;
    }
  }
  const int wthreads = 256;
  // a thread's list lives in shared memory: fewer threads per block for long lists
  int fthreads = 256;
  while (fthreads > 32 && sizeof(int32_t)*(size_t)fthreads*tcap > 96*1024) fthreads >>= 1;
  // bitonic sort pads each warp's list to a power of two >= 32
  int wcap = 32;
  while (wcap < wmax) wcap <<= 1;
  auto thread = [](const Problem& p) { return p.fillSchedule != NBR_SCHEDULE_WARP; };
  for (Problem* p : b.mem) {
    p->lastNbrSchedule = p->fillSchedule;
    p->lastNbrPasses = p->grid.stashCap > 0 ? 1 : 2;
  }
  b.lastNbrSchedule = nm ? b.mem[0]->lastNbrSchedule : 0;
  const size_t tsmem = sizeof(int32_t)*(size_t)fthreads*tcap;
  const size_t wsmem = sizeof(int32_t)*(wthreads/32)*(size_t)wcap;
  // the cell walk's staging area, at least a list and a row table per warp
  // where a block may walk a crowded cell itself
  const size_t clists = sizeof(int32_t)*kCellWarps*(size_t)(wcap + RowTable<1>::NR*RowTable<1>::RW);
  const size_t cstage = sizeof(CellShared);
  const size_t csmem = alone && clists > cstage ? clists : cstage;
  auto smemAttr = [](auto* kernel, size_t bytes) -> int {
    if (bytes <= 48*1024) return SPHGPU_OK;
    return cuda_status(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes),
                       "nbr smem attribute");
  };
  SPH_TRY(smemAttr(nbr_thread_kernel<false, 1>, tsmem)); SPH_TRY(smemAttr(nbr_thread_kernel<true, 1>, tsmem));
  SPH_TRY(smemAttr(nbr_thread_kernel<false, 2>, tsmem)); SPH_TRY(smemAttr(nbr_thread_kernel<true, 2>, tsmem));
  SPH_TRY(smemAttr(nbr_cell_kernel<false>, csmem)); SPH_TRY(smemAttr(nbr_cell_kernel<true>, csmem));
  SPH_TRY(smemAttr(nbr_walk_kernel<false>, wsmem)); SPH_TRY(smemAttr(nbr_walk_kernel<true>, wsmem));
  SPH_TRY(smemAttr(nbr_crowded_kernel<false>, wsmem)); SPH_TRY(smemAttr(nbr_crowded_kernel<true>, wsmem));
  // One walk launch per (schedule, cell subdivision) present.  pass 0: count
  // (and the lists of members with a stash); pass 1: fill (members without).
  auto walk = [&](bool threadSched, int sub, bool fill) -> int {
    BlockMap map;
    unsigned grid = 0;
    const int threads = threadSched ? (fill || tstash ? fthreads : 256) : (sub == 1 ? kCellThreads : wthreads);
    SPH_TRY(batch_map_items(b, [&](const Problem& p) {
      if (thread(p) != threadSched || p.grid.sub != sub || (fill && p.grid.stashCap)) return (int64_t)0;
      if (threadSched) return p.candcap;
      // the cell walk: a block per cell up to kCellBlocks, each striding over the member's cells
      if (sub == 1) return kCellThreads*(p.cellcap < kCellBlocks ? p.cellcap : kCellBlocks);
      return 32*p.candcap; }, threads, &map, &grid));
    if (!grid) return SPHGPU_OK;
    if (threadSched) {
      const bool lists = fill || tstash;
      const size_t smem = lists ? tsmem : 0;
      const int c = lists ? tcap : 0;
      if (sub == 1) {
        if (fill) nbr_thread_kernel<true, 1><<<grid, threads, smem, st>>>(b.d_mem, map, c, maxNbr);
        else nbr_thread_kernel<false, 1><<<grid, threads, smem, st>>>(b.d_mem, map, c, maxNbr);
      } else {
        if (fill) nbr_thread_kernel<true, 2><<<grid, threads, smem, st>>>(b.d_mem, map, c, maxNbr);
        else nbr_thread_kernel<false, 2><<<grid, threads, smem, st>>>(b.d_mem, map, c, maxNbr);
      }
    } else {
      const bool lists = fill || wstash;
      const size_t smem = sub == 1 ? csmem : (lists ? wsmem : 0);
      const int c = lists || sub == 1 ? wcap : 0;
      if (sub == 1) {
        if (fill) nbr_cell_kernel<true><<<grid, threads, smem, st>>>(b.d_mem, map, c, maxNbr);
        else nbr_cell_kernel<false><<<grid, threads, smem, st>>>(b.d_mem, map, c, maxNbr);
      } else {
        if (fill) nbr_walk_kernel<true><<<grid, threads, smem, st>>>(b.d_mem, map, c, maxNbr);
        else nbr_walk_kernel<false><<<grid, threads, smem, st>>>(b.d_mem, map, c, maxNbr);
      }
    }
    batch_count_launch(b);
    if (threadSched || sub != 1) return SPHGPU_OK;
    SPH_TRY(batch_map_items(b, [&](const Problem& p) {
      if (thread(p) || p.grid.sub != 1 || !p.grid.crowdList || (fill && p.grid.stashCap)) return (int64_t)0;
      return 32*p.candcap; }, wthreads, &map, &grid));
    if (!grid) return SPHGPU_OK;
    const size_t smem = fill || wstash ? wsmem : 0;
    if (fill) nbr_crowded_kernel<true><<<grid, wthreads, smem, st>>>(b.d_mem, map, wcap, maxNbr);
    else nbr_crowded_kernel<false><<<grid, wthreads, smem, st>>>(b.d_mem, map, wcap, maxNbr);
    batch_count_launch(b);
    return SPHGPU_OK;
  };
  {
    // the cell walk reads its cells in node order
    BlockMap om;
    unsigned ogrid = 0;
    SPH_TRY(batch_map_items(b, [&](const Problem& p) {
      return thread(p) || p.grid.sub != 1 ? (int64_t)0 : fixedItems(32*p.cellcap); }, kGhostThreads, &om, &ogrid));
    if (ogrid) { cell_order_kernel<<<ogrid, kGhostThreads, 0, st>>>(b.d_mem, om); batch_count_launch(b); }
  }
  for (int sub = 1; sub <= 2; ++sub) {
    SPH_TRY(walk(true, sub, false));
    SPH_TRY(walk(false, sub, false));
  }
  SPH_TRY(batch_scan(b, SCAN_COUNTS));
  // lists to the CSR: compaction of the stashes, fill pass for the rest
  BlockMap ctmap, cwmap;
  unsigned ctgrid = 0, cwgrid = 0;
  SPH_TRY(batch_map_items(b, [&](const Problem& p) { return thread(p) && p.grid.stashCap ? p.candcap : (int64_t)0; },
                          256, &ctmap, &ctgrid));
  SPH_TRY(batch_map_items(b, [&](const Problem& p) { return !thread(p) && p.grid.stashCap ? 32*p.n : (int64_t)0; },
                          256, &cwmap, &cwgrid));
  if (ctgrid) { nbr_compact_thread_kernel<<<ctgrid, 256, 0, st>>>(b.d_mem, ctmap); batch_count_launch(b); }
  if (cwgrid) { nbr_compact_warp_kernel<<<cwgrid, 256, 0, st>>>(b.d_mem, cwmap); batch_count_launch(b); }
  for (int sub = 1; sub <= 2; ++sub) {
    SPH_TRY(walk(true, sub, true));
    SPH_TRY(walk(false, sub, true));
  }
  return cuda_status(cudaGetLastError(), "neighbor build");
}

}  // namespace

// The build's launches alone, for a CUDA-graph capture of the whole step:
// capacities planned beforehand (plan_build), no read-back; a capacity
// overflow sets the member's error flag on the device instead.
int plan_build(Batch& b, bool captured) { return plan_capacities(b, captured); }
int launch_build_captured(Batch& b) { return launch_build(b); }

// After a build: whether the cell walk has met crowded cells, and whether they
// hold so much of the problem that it had better not be used.  Once it has, the
// problem keeps the list (a run whose clump comes and goes is not captured
// anew each time).
void note_crowd(Problem& p, int64_t crowdedSlots) {
  if (p.fillSchedule != NBR_SCHEDULE_WARP || p.grid.sub != 1) return;
  if (crowdedSlots > 0) p.crowd = 1;
  else if (p.crowd < 0) p.crowd = 0;
  if (4*crowdedSlots > p.n + p.G && reach_cells(p) > 0.0) p.denseSet = 27.0*(double)(p.n + p.G)/reach_cells(p);
}

// Ghosts and ConnectivityMap of every member: all stages launched with the
// sizes kept on the device, then one read-back of the sizes; a capacity
// overflow grows the buffers and repeats the build.
int build_connectivity(Batch& b) {
  const int nm = (int)b.mem.size();
  for (Problem* p : b.mem) {
    if (p->n + p->gcap > INT_MAX) { set_error("too many nodes for 32-bit neighbor indices"); return SPHGPU_ERR_CAPACITY; }
  }
  for (int attempt = 0; attempt < 6; ++attempt) {
    if (!(attempt == 0 && b.buildPlanned)) SPH_TRY(plan_capacities(b));
    SPH_TRY(launch_build(b));
    if (b.afterBuildLaunch) {
      const std::function<int()> f = std::move(b.afterBuildLaunch);
      b.afterBuildLaunch = nullptr;
      SPH_TRY(f());
    }
    const int slots[8] = {SC_G, SC_TOTAL, SC_MAXCOUNT, SC_PAIRS, SC_NCELLS, SC_CELLSWANTED, -1, SC_CROWDED};
    std::vector<double> r;
    SPH_TRY(batch_gather(b, slots, 8, r));
    bool redo = false;
    for (int m = 0; m < nm; ++m) {
      Problem& p = *b.mem[m];
      const int herr = (int)r[m*8 + 6];
      p.G = asI64(r[m*8]);
      p.ntot = p.n + p.G;
      p.E = asI64(r[m*8 + 1]);
      note_rows(p);
      p.maxCount = asI32(r[m*8 + 2]);
      p.pairs = asI64(r[m*8 + 3]);
      p.ncells = asI64(r[m*8 + 4]);
      p.cellsWanted = asI64(r[m*8 + 5]);
      p.lastNbrCells = p.grid.sub;
      note_crowd(p, asI64(r[m*8 + 7]));
      if (herr) cudaMemsetAsync(p.d_err, 0, sizeof(int), b.stream);
      if ((herr & DERR_NBR_CAPACITY) || p.maxCount > p.maxNbr) {
        set_error("a node has more neighbors than max_neighbors");
        return SPHGPU_ERR_CAPACITY;
      }
      if (herr & DERR_GHOST_CHAIN) {
        set_error("a ghost image was imaged twice through one periodic axis");
        return SPHGPU_ERR_UNSUPPORTED;
      }
      if (herr & DERR_NONPOSITIVE) {
        set_error("non-positive or non-finite smoothing scale");
        return SPHGPU_ERR_NUMERIC;
      }
      if (herr & DERR_BARRIER) {
        if (b.d_fuse) cudaMemsetAsync(b.d_fuse, 0, 2*sizeof(unsigned int), b.stream);
        set_error("neighbor build: a grid barrier of the fused ghost passes timed out");
        return SPHGPU_ERR_CUDA;
      }
      if (herr & DERR_GHOST_CAPACITY) { p.G = 2*p.gcap; redo = true; }        // ghost count unknown: double
      if (herr & DERR_ENTRY_CAPACITY) redo = true;                           // p.E is the true entry count
      if (herr & DERR_LIST_CAPACITY) { p.fillCap = p.maxCount + p.maxCount/4 + 8; redo = true; }
      else if (p.fillCap > p.maxCount + p.maxCount/2 + 16) p.fillCap = 0;   // re-plan a tighter list
    }
    if (!redo) return SPHGPU_OK;
    SPH_CHECK(cudaStreamSynchronize(b.stream));
  }
  set_error("neighbor build: capacities did not converge");
  return SPHGPU_ERR_CAPACITY;
}

}  // namespace sphgpu

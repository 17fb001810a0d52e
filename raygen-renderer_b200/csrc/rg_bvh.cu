// rg_bvh.cu - scene preparation and binned-SAH BVH build on the device.
//
// Reference: RayRenderer::transformScene / transformObject
// (rayrenderer.cpp:157-363), RenderMeshTriangle::precalc (raycommon.cpp:128-149)
// and TriangleBVH::build / buildRecursive (bvh.cpp:76-231).
//
// The reference builds top-down and recursively on one CPU thread: widest
// centroid axis, 16 bins, leaf <= 4, cost 1 + 1.5 (A_L N_L + A_R N_R)/A_P
// against 1.5 N.  Here the same split rule (bin count a parameter, 32 by
// default) runs breadth-first over nodes of more than kSubtree primitives: every
// level bins all open nodes at once, picks splits one warp per node and moves the
// primitives by a stable partition; below that size one block splits a node to
// the end in shared memory.  Leaves hold at most kMaxLeaf (8) triangles:
// where the reference would keep a larger leaf, the best SAH bin (or, for
// coincident centroids, an index median) splits it further.
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <climits>
#include <cub/device/device_scan.cuh>
#include <cuda_fp16.h>

#include <cfloat>
#include <vector>

#include "rg_device.cuh"
#include "rg_host.h"

namespace rg {

namespace {

__device__ __forceinline__ uint32_t fenc(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float fdec(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

struct BNode {
  float bmin[3], bmax[3];
  float cmin[3], cmax[3];
  int start, count;
  int left;      // first child (right = left + 1), -1 for leaves
  int axis;
  int binSlot;   // slot in the level's bin array while open
  int splitBin;  // bins <= splitBin go left; -2 = index median split
};

struct BinData {  // ordered-uint encoded bounds, 16 words
  uint32_t bmin[3], bmax[3], cmin[3], cmax[3];
  uint32_t count;
  uint32_t pad[3];
};

// device counters of a build
enum BuildCounter { C_NODES = 0, C_BUILD_ERROR = 1, C_SMALL = 2, C_BUILD_COUNTERS = 3 };

// ---- triangle preparation -------------------------------------------------
// World -> view (camera translation; angles handled on the host by rotating
// the input), edges, geometric normal, bounds, occluder bits.
__global__ void k_prepTriangles(int n, const float* __restrict__ pos, const float* __restrict__ nrm,
                                const float* __restrict__ uv, const int* __restrict__ triMesh,
                                const int* __restrict__ meshObj, const int* __restrict__ objMat,
                                const DevMaterial* __restrict__ mats, const float* __restrict__ view,
                                float4* __restrict__ verts, float4* __restrict__ shade, float2* __restrict__ uvOut,
                                float4* __restrict__ bmin, float4* __restrict__ bmax) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float* p = pos + (size_t)i * 9;
  const float* q = nrm + (size_t)i * 9;
  V3 v[3], nn[3];
  for (int k = 0; k < 3; k++) {
    const V3 w = v3(p[k * 3], p[k * 3 + 1], p[k * 3 + 2]);
    // p_view = [p 1] * M (row vector, M row-major 4x4), non-contracted
    v[k].x = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(w.x, view[0]), __fmul_rn(w.y, view[4])), __fmul_rn(w.z, view[8])), view[12]);
    v[k].y = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(w.x, view[1]), __fmul_rn(w.y, view[5])), __fmul_rn(w.z, view[9])), view[13]);
    v[k].z = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(w.x, view[2]), __fmul_rn(w.y, view[6])), __fmul_rn(w.z, view[10])), view[14]);
    const V3 m = v3(q[k * 3], q[k * 3 + 1], q[k * 3 + 2]);
    // normals: [n 0] * inverse-transpose(M); M is rigid here, so its 3x3 block
    V3 r;
    r.x = __fadd_rn(__fadd_rn(__fmul_rn(m.x, view[0]), __fmul_rn(m.y, view[4])), __fmul_rn(m.z, view[8]));
    r.y = __fadd_rn(__fadd_rn(__fmul_rn(m.x, view[1]), __fmul_rn(m.y, view[5])), __fmul_rn(m.z, view[9]));
    r.z = __fadd_rn(__fadd_rn(__fmul_rn(m.x, view[2]), __fmul_rn(m.y, view[6])), __fmul_rn(m.z, view[10]));
    const float l = __fsqrt_rn(dot_rn(r, r));
    nn[k] = l > 0.0f ? v3(__fdiv_rn(r.x, l), __fdiv_rn(r.y, l), __fdiv_rn(r.z, l)) : r;
  }
  const V3 e1 = sub_rn(v[1], v[0]), e2 = sub_rn(v[2], v[0]);
  const V3 pd = cross_rn(sub_rn(v[1], v[0]), sub_rn(v[2], v[1]));
  const float pl = __fsqrt_rn(dot_rn(pd, pd));
  const V3 gn = pl > 0.0f ? v3(__fdiv_rn(pd.x, pl), __fdiv_rn(pd.y, pl), __fdiv_rn(pd.z, pl)) : pd;
  const int mesh = triMesh[i];
  const DevMaterial mt = mats[objMat[meshObj[mesh]]];
  uint32_t occ = kOccAll;
  if (mt.transparency < 0.01f && mt.emission <= 0.0f) occ |= kOccArea;
  if (mt.emission <= 0.0f && (mt.transparency < 0.01f || mt.refraction > 0.1f)) occ |= kOccPoint;
  if (mt.transparency < 0.01f) occ |= kOccAO;
  if (mt.emission <= 0.0f && mt.transparency < 0.01f && mt.refraction <= 0.1f) occ |= kOccVol;
  verts[(size_t)i * 3 + 0] = make_float4(v[0].x, v[0].y, v[0].z, __int_as_float(mesh));
  verts[(size_t)i * 3 + 1] = make_float4(e1.x, e1.y, e1.z, __uint_as_float(occ));
  verts[(size_t)i * 3 + 2] = make_float4(e2.x, e2.y, e2.z, 0.0f);
  shade[(size_t)i * 3 + 0] = make_float4(nn[0].x, nn[0].y, nn[0].z, nn[1].x);
  shade[(size_t)i * 3 + 1] = make_float4(nn[1].y, nn[1].z, nn[2].x, nn[2].y);
  shade[(size_t)i * 3 + 2] = make_float4(nn[2].z, gn.x, gn.y, gn.z);
  if (uvOut) {
    for (int k = 0; k < 3; k++) uvOut[(size_t)i * 3 + k] = uv ? make_float2(uv[(size_t)i * 6 + k * 2], uv[(size_t)i * 6 + k * 2 + 1]) : make_float2(0, 0);
  }
  const V3 lo = v3(fminf(v[0].x, fminf(v[1].x, v[2].x)), fminf(v[0].y, fminf(v[1].y, v[2].y)), fminf(v[0].z, fminf(v[1].z, v[2].z)));
  const V3 hi = v3(fmaxf(v[0].x, fmaxf(v[1].x, v[2].x)), fmaxf(v[0].y, fmaxf(v[1].y, v[2].y)), fmaxf(v[0].z, fmaxf(v[1].z, v[2].z)));
  bmin[i] = make_float4(lo.x, lo.y, lo.z, 0.0f);
  bmax[i] = make_float4(hi.x, hi.y, hi.z, 0.0f);
}

// ---- root bounds -------------------------------------------------------------
__global__ void k_initBounds(uint32_t* out) {  // identities, as k_rootBounds reduces into them
  const int k = threadIdx.x;
  if (k < 12) out[k] = (k / 3) % 2 == 0 ? 0xFFFFFFFFu : 0u;
}

__global__ void k_rootBounds(int n, const float4* __restrict__ bmin, const float4* __restrict__ bmax, uint32_t* out) {
  // out: bmin[3] bmax[3] cmin[3] cmax[3] (encoded)
  float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
  float clo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, chi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4 a = bmin[i], b = bmax[i];
    const float av[3] = {a.x, a.y, a.z}, bv[3] = {b.x, b.y, b.z};
    for (int k = 0; k < 3; k++) {
      lo[k] = fminf(lo[k], av[k]);
      hi[k] = fmaxf(hi[k], bv[k]);
      const float c = (av[k] + bv[k]) * 0.5f;
      clo[k] = fminf(clo[k], c);
      chi[k] = fmaxf(chi[k], c);
    }
  }
  for (int k = 0; k < 3; k++) {
    for (int o = 16; o > 0; o >>= 1) {
      lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
      hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
      clo[k] = fminf(clo[k], __shfl_xor_sync(0xffffffffu, clo[k], o));
      chi[k] = fmaxf(chi[k], __shfl_xor_sync(0xffffffffu, chi[k], o));
    }
  }
  if ((threadIdx.x & 31) == 0) {
    for (int k = 0; k < 3; k++) {
      atomicMin(&out[k], fenc(lo[k]));
      atomicMax(&out[3 + k], fenc(hi[k]));
      atomicMin(&out[6 + k], fenc(clo[k]));
      atomicMax(&out[9 + k], fenc(chi[k]));
    }
  }
}

// rootOpen: 0 a leaf, 1 open for the levels (task 0 of level 0), 2 small enough for k_subtrees.
__global__ void k_initRoot(int n, const uint32_t* rb, BNode* nodes, int* primIdx, int* primNode, int rootOpen, int* counters,
                           int* levelCount, int* tasks, int* smallTasks) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    counters[C_NODES] = 1;
    counters[C_BUILD_ERROR] = 0;
    counters[C_SMALL] = rootOpen == 2 ? 1 : 0;
    levelCount[0] = rootOpen == 1 ? 1 : 0;
    tasks[0] = 0;
    smallTasks[0] = 0;
    BNode r;
    for (int k = 0; k < 3; k++) {
      r.bmin[k] = fdec(rb[k]); r.bmax[k] = fdec(rb[3 + k]);
      r.cmin[k] = fdec(rb[6 + k]); r.cmax[k] = fdec(rb[9 + k]);
    }
    r.start = 0; r.count = n; r.left = -1; r.axis = 0; r.binSlot = 0; r.splitBin = -1;
    nodes[0] = r;
  }
  if (i < n) {
    primIdx[i] = i;
    primNode[i] = rootOpen == 1 ? 0 : -1;
  }
}

// Task counts live on the device (`count`, of which this launch takes [first, first + most)), so
// that levels can be launched before the previous ones have run.
__device__ __forceinline__ int tasksOf(const int* count, int first, int most) { return max(0, min(*count - first, most)); }

__device__ __forceinline__ int widestAxis(const BNode& nd) {  // bvh.cpp:125-131
  const float ex = nd.cmax[0] - nd.cmin[0], ey = nd.cmax[1] - nd.cmin[1], ez = nd.cmax[2] - nd.cmin[2];
  int axis = 0;
  if (ey > ex) axis = 1;
  if (ez > ((axis == 0) ? ex : ey)) axis = 2;
  return axis;
}

// Prepare open nodes of a level: pick the widest centroid axis.
__global__ void k_prepareLevel(const int* count, int first, int most, const int* tasks, BNode* nodes, BinData* bins, int nbins,
                               bool resetBins) {
  const int numTasks = tasksOf(count, first, most);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < numTasks) {
    BNode& nd = nodes[tasks[first + t]];
    nd.axis = widestAxis(nd);
    nd.binSlot = t;
  }
  // reset bins (one thread per bin) unless the split kernel leaves them reset
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (resetBins && b < numTasks * nbins) {
    BinData z;
    for (int k = 0; k < 3; k++) {
      z.bmin[k] = 0xFFFFFFFFu; z.bmax[k] = 0u; z.cmin[k] = 0xFFFFFFFFu; z.cmax[k] = 0u;
    }
    z.count = 0; z.pad[0] = z.pad[1] = z.pad[2] = 0;
    bins[b] = z;
  }
}

__device__ __forceinline__ int binOf(const BNode& nd, float c, int nbins) {
  const float cmin = nd.cmin[nd.axis];
  const float ext = nd.cmax[nd.axis] - cmin;
  const float scale = (float)nbins / ext;
  int b = (int)((c - cmin) * scale);
  if (b < 0) b = 0;
  if (b >= nbins) b = nbins - 1;
  return b;
}

__device__ __forceinline__ float axisOf(const float4& v, int a) { return a == 0 ? v.x : (a == 1 ? v.y : v.z); }

// Primitives binned per block (build-time overridable (-D) for sweeps).
#ifndef RG_BIN_CHUNK
#define RG_BIN_CHUNK 1024  // swept: 1024 / 2048 / 4096 / 16384 -> 12.5 / 13.0 / 13.9 / 19.4 ms (4M triangles)
#endif
constexpr int kBinChunk = RG_BIN_CHUNK;
// Largest leaf of the 8-wide BVH (<= 4: a node's leaves address at most 32 triangles
// through its 32-bit triangle mask); build-time overridable (-D) for sweeps.
#ifndef RG_WIDE_MAX_LEAF
#define RG_WIDE_MAX_LEAF 4
#endif
constexpr int kWideMaxLeaf = RG_WIDE_MAX_LEAF;
static_assert(kWideMaxLeaf >= 1 && kWideMaxLeaf <= 4, "8 leaves of at most 4 triangles fill the 32-bit mask");
constexpr int kMaxBins = 64;
// Nodes of at most this many primitives are split to the end by one thread block
// (k_subtrees); larger ones level by level over the whole device.  A level reads every
// primitive and costs six launches; below this size the levels were 40% of the build of 4M
// triangles and nearly all of a small scene's.
#ifndef RG_SUBTREE
#define RG_SUBTREE 1024
#endif
constexpr int kSubtree = RG_SUBTREE;
static_assert(kSubtree >= kBinChunk, "k_bin: a chunk reaches into at most two open nodes");

// One primitive's bounds and centroid into a bin in shared memory (ordered-uint encoded).
__device__ __forceinline__ void binPrim(uint32_t (&sb)[13], const uint32_t (&v)[12], uint32_t count) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    atomicMin(&sb[k], v[k]);
    atomicMax(&sb[3 + k], v[3 + k]);
    atomicMin(&sb[6 + k], v[6 + k]);
    atomicMax(&sb[9 + k], v[9 + k]);
  }
  atomicAdd(&sb[12], count);
}

// Bins of the open nodes of a level.  Open nodes hold more than kBinChunk primitives in
// consecutive places, so a block's chunk reaches into at most two of them; it bins them in
// shared memory and adds the bins that got any to the nodes' bins in global memory.
// Neighbouring primitives mostly fall into the same bin, whose 13 shared-memory atomics
// then serialise over the warp: the lanes of the bins of up to three leading lanes are
// reduced in registers first.  bmin / bmax are in the current primitive order (they move
// with primIdx in the partition), so the pass reads them coalesced.
__global__ void __launch_bounds__(256) k_bin(int n, const int* __restrict__ primNode, const BNode* __restrict__ nodes,
                                             const float4* __restrict__ bmin, const float4* __restrict__ bmax,
                                             BinData* bins, int nbins, const int* __restrict__ err) {
  __shared__ uint32_t sb[2][kMaxBins][13];
  __shared__ int sNode[2];  // lowest and highest open node id of the chunk
  const bool failed = *err != 0;
  const int first = blockIdx.x * kBinChunk;
  const int last = min(n, first + kBinChunk);
  if (threadIdx.x == 0) {
    sNode[0] = INT_MAX;
    sNode[1] = -1;
  }
  for (int b = threadIdx.x; b < 2 * nbins; b += blockDim.x) {
    uint32_t* r = sb[b / nbins][b % nbins];
    for (int k = 0; k < 3; k++) {
      r[k] = r[6 + k] = 0xFFFFFFFFu;
      r[3 + k] = r[9 + k] = 0u;
    }
    r[12] = 0u;
  }
  __syncthreads();
  {
    int lo = INT_MAX, hi = -1;
    for (int i = first + threadIdx.x; i < last; i += blockDim.x) {
      const int nd = primNode[i];
      if (nd >= 0) {
        lo = min(lo, nd);
        hi = max(hi, nd);
      }
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if ((threadIdx.x & 31) == 0 && hi >= 0) {
      atomicMin(&sNode[0], lo);
      atomicMax(&sNode[1], hi);
    }
  }
  __syncthreads();
  const int nodeA = sNode[0], nodeB = sNode[1];
  if (nodeB < 0 || failed) return;
  const BNode ndA = nodes[nodeA], ndB = nodes[nodeB];
  const bool onA = ndA.binSlot >= 0 && ndA.cmax[ndA.axis] - ndA.cmin[ndA.axis] >= 1e-12f;
  const bool onB = ndB.binSlot >= 0 && ndB.cmax[ndB.axis] - ndB.cmin[ndB.axis] >= 1e-12f;
  const int lane = threadIdx.x & 31;
  for (int i0 = first; i0 < last; i0 += blockDim.x) {  // whole warps: i0 is the block's
    const int i = i0 + threadIdx.x;
    const int nd = i < last ? primNode[i] : -1;
    const bool isA = nd == nodeA, in = nd >= 0 && (isA ? onA : onB);
    int slot = -1;  // bin of the two nodes' bins
    uint32_t v[12];
    if (in) {
      const float4 lo = bmin[i], hi = bmax[i];
      const float4 c = make_float4((lo.x + hi.x) * 0.5f, (lo.y + hi.y) * 0.5f, (lo.z + hi.z) * 0.5f, 0.0f);
      const BNode& N = isA ? ndA : ndB;
      slot = (isA ? 0 : kMaxBins) + binOf(N, axisOf(c, N.axis), nbins);
      v[0] = fenc(lo.x); v[1] = fenc(lo.y); v[2] = fenc(lo.z);
      v[3] = fenc(hi.x); v[4] = fenc(hi.y); v[5] = fenc(hi.z);
      v[6] = v[9] = fenc(c.x); v[7] = v[10] = fenc(c.y); v[8] = v[11] = fenc(c.z);
    }
    unsigned left = __ballot_sync(0xffffffffu, in);
    for (int r = 0; r < 3 && left; r++) {
      const int lead = __ffs(left) - 1;
      const unsigned same = __ballot_sync(0xffffffffu, slot == __shfl_sync(0xffffffffu, slot, lead));
      if ((same >> lane) & 1u) {
        uint32_t w[12];
#pragma unroll
        for (int k = 0; k < 3; k++) {
          w[k] = __reduce_min_sync(same, v[k]);
          w[3 + k] = __reduce_max_sync(same, v[3 + k]);
          w[6 + k] = __reduce_min_sync(same, v[6 + k]);
          w[9 + k] = __reduce_max_sync(same, v[9 + k]);
        }
        if (lane == lead) binPrim(sb[slot / kMaxBins][slot % kMaxBins], w, __popc(same));
      }
      left &= ~same;
    }
    if ((left >> lane) & 1u) binPrim(sb[slot / kMaxBins][slot % kMaxBins], v, 1u);
  }
  __syncthreads();
  for (int b = threadIdx.x; b < 2 * nbins; b += blockDim.x) {
    const uint32_t* r = sb[b / nbins][b % nbins];
    if (r[12] == 0) continue;
    BinData& nb = bins[(size_t)(b < nbins ? ndA.binSlot : ndB.binSlot) * nbins + b % nbins];
    for (int k = 0; k < 3; k++) {
      atomicMin(&nb.bmin[k], r[k]);
      atomicMax(&nb.bmax[k], r[3 + k]);
      atomicMin(&nb.cmin[k], r[6 + k]);
      atomicMax(&nb.cmax[k], r[9 + k]);
    }
    atomicAdd(&nb.count, r[12]);
  }
}

// Binning for more than 32 bins, where nodes of any size are open: shared-memory bins for a
// block inside one node, global atomics across nodes.
__global__ void __launch_bounds__(256) k_binAny(int n, const int* __restrict__ primNode, const BNode* __restrict__ nodes,
                                             const float4* __restrict__ bmin, const float4* __restrict__ bmax,
                                             BinData* bins, int nbins, const int* __restrict__ err) {
  if (*err) return;
  __shared__ uint32_t sb[kMaxBins][13];
  const int first = blockIdx.x * kBinChunk;
  if (first >= n) return;
  const int last = min(n, first + kBinChunk) - 1;
  const int nodeA = primNode[first], nodeB = primNode[last];
  const bool uniform = (nodeA == nodeB) && nodeA >= 0;
  if (uniform) {
    for (int b = threadIdx.x; b < nbins; b += blockDim.x) {
      for (int k = 0; k < 3; k++) {
        sb[b][k] = 0xFFFFFFFFu; sb[b][3 + k] = 0u; sb[b][6 + k] = 0xFFFFFFFFu; sb[b][9 + k] = 0u;
      }
      sb[b][12] = 0;
    }
    __syncthreads();
    const BNode nd = nodes[nodeA];
    if (nd.binSlot < 0) return;
    const float ext = nd.cmax[nd.axis] - nd.cmin[nd.axis];
    if (ext >= 1e-12f) {
      for (int i = first + threadIdx.x; i <= last; i += blockDim.x) {
        const float4 lo = bmin[i], hi = bmax[i];
        const float4 c = make_float4((lo.x + hi.x) * 0.5f, (lo.y + hi.y) * 0.5f, (lo.z + hi.z) * 0.5f, 0.0f);
        const int b = binOf(nd, axisOf(c, nd.axis), nbins);
        atomicMin(&sb[b][0], fenc(lo.x)); atomicMin(&sb[b][1], fenc(lo.y)); atomicMin(&sb[b][2], fenc(lo.z));
        atomicMax(&sb[b][3], fenc(hi.x)); atomicMax(&sb[b][4], fenc(hi.y)); atomicMax(&sb[b][5], fenc(hi.z));
        atomicMin(&sb[b][6], fenc(c.x)); atomicMin(&sb[b][7], fenc(c.y)); atomicMin(&sb[b][8], fenc(c.z));
        atomicMax(&sb[b][9], fenc(c.x)); atomicMax(&sb[b][10], fenc(c.y)); atomicMax(&sb[b][11], fenc(c.z));
        atomicAdd(&sb[b][12], 1u);
      }
    }
    __syncthreads();
    BinData* nb = bins + (size_t)nd.binSlot * nbins;
    for (int b = threadIdx.x; b < nbins; b += blockDim.x) {
      if (sb[b][12] == 0) continue;
      for (int k = 0; k < 3; k++) {
        atomicMin(&nb[b].bmin[k], sb[b][k]);
        atomicMax(&nb[b].bmax[k], sb[b][3 + k]);
        atomicMin(&nb[b].cmin[k], sb[b][6 + k]);
        atomicMax(&nb[b].cmax[k], sb[b][9 + k]);
      }
      atomicAdd(&nb[b].count, sb[b][12]);
    }
    return;
  }
  for (int i = first + threadIdx.x; i <= last; i += blockDim.x) {
    const int node = primNode[i];
    if (node < 0) continue;
    const BNode& nd = nodes[node];
    if (nd.binSlot < 0) continue;
    const float ext = nd.cmax[nd.axis] - nd.cmin[nd.axis];
    if (ext < 1e-12f) continue;
    const float4 lo = bmin[i], hi = bmax[i];
    const float4 c = make_float4((lo.x + hi.x) * 0.5f, (lo.y + hi.y) * 0.5f, (lo.z + hi.z) * 0.5f, 0.0f);
    const int b = binOf(nd, axisOf(c, nd.axis), nbins);
    BinData& bd = bins[(size_t)nd.binSlot * nbins + b];
    atomicMin(&bd.bmin[0], fenc(lo.x)); atomicMin(&bd.bmin[1], fenc(lo.y)); atomicMin(&bd.bmin[2], fenc(lo.z));
    atomicMax(&bd.bmax[0], fenc(hi.x)); atomicMax(&bd.bmax[1], fenc(hi.y)); atomicMax(&bd.bmax[2], fenc(hi.z));
    atomicMin(&bd.cmin[0], fenc(c.x)); atomicMin(&bd.cmin[1], fenc(c.y)); atomicMin(&bd.cmin[2], fenc(c.z));
    atomicMax(&bd.cmax[0], fenc(c.x)); atomicMax(&bd.cmax[1], fenc(c.y)); atomicMax(&bd.cmax[2], fenc(c.z));
    atomicAdd(&bd.count, 1u);
  }
}

__device__ __forceinline__ float areaOf(const float lo[3], const float hi[3]) {
  const float dx = hi[0] - lo[0], dy = hi[1] - lo[1], dz = hi[2] - lo[2];
  return 2.0f * (dx * dy + dy * dz + dz * dx);
}

// Split decision per open node (bvh.cpp:133-211 cost model).
__global__ void k_split(const int* count, int firstTask, int most, const int* __restrict__ tasks, BNode* nodes,
                        const BinData* __restrict__ bins, int nbins, int* nodeCounter, int* nextTasks, int* nextCount,
                        int maxLeaf) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= tasksOf(count, firstTask, most)) return;
  const int id = tasks[firstTask + t];
  BNode nd = nodes[id];
  const BinData* nb = bins + (size_t)nd.binSlot * nbins;
  const float ext = nd.cmax[nd.axis] - nd.cmin[nd.axis];
  int best = -1;
  float bestCost = (float)nd.count * 1.5f;
  float forcedCost = FLT_MAX;
  int forced = -1;
  // sweeps
  float la[kMaxBins];
  int lc[kMaxBins];
  if (ext >= 1e-12f) {
    float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    int c = 0;
    for (int i = 0; i < nbins - 1; i++) {
      if (nb[i].count > 0) {
        for (int k = 0; k < 3; k++) { lo[k] = fminf(lo[k], fdec(nb[i].bmin[k])); hi[k] = fmaxf(hi[k], fdec(nb[i].bmax[k])); }
      }
      c += nb[i].count;
      la[i] = c > 0 ? areaOf(lo, hi) : 0.0f;
      lc[i] = c;
    }
    const float pa = areaOf(nd.bmin, nd.bmax);
    const float invPa = pa > 0.0f ? 1.0f / pa : 0.0f;
    float rlo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, rhi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    int rc = 0;
    for (int i = nbins - 1; i > 0; i--) {
      if (nb[i].count > 0) {
        for (int k = 0; k < 3; k++) { rlo[k] = fminf(rlo[k], fdec(nb[i].bmin[k])); rhi[k] = fmaxf(rhi[k], fdec(nb[i].bmax[k])); }
      }
      rc += nb[i].count;
      const float ra = rc > 0 ? areaOf(rlo, rhi) : 0.0f;
      const int s = i - 1;
      if (lc[s] == 0 || rc == 0) continue;
      const float cost = 1.0f + 1.5f * invPa * (la[s] * (float)lc[s] + ra * (float)rc);
      if (cost < bestCost || (cost == bestCost && best >= 0 && s < best)) { bestCost = cost; best = s; }
      if (cost < forcedCost || (cost == forcedCost && s < forced)) { forcedCost = cost; forced = s; }
    }
  }
  int split = best;
  if (split < 0 && nd.count > maxLeaf) split = forced >= 0 ? forced : -2;  // -2: index median
  nd.binSlot = -1;
  if (split == -1) {
    nd.left = -1;
    nodes[id] = nd;
    return;
  }
  const int left = atomicAdd(nodeCounter, 2);
  BNode ch[2];
  int cnt[2];
  if (split == -2) {
    cnt[0] = nd.count / 2;
    cnt[1] = nd.count - cnt[0];
    for (int s = 0; s < 2; s++) {
      for (int k = 0; k < 3; k++) {
        ch[s].bmin[k] = nd.bmin[k]; ch[s].bmax[k] = nd.bmax[k];
        ch[s].cmin[k] = nd.cmin[k]; ch[s].cmax[k] = nd.cmax[k];
      }
    }
  } else {
    for (int s = 0; s < 2; s++) {
      float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
      float clo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, chi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
      int c = 0;
      const int b0 = s == 0 ? 0 : split + 1, b1 = s == 0 ? split + 1 : nbins;
      for (int b = b0; b < b1; b++) {
        if (nb[b].count == 0) continue;
        c += nb[b].count;
        for (int k = 0; k < 3; k++) {
          lo[k] = fminf(lo[k], fdec(nb[b].bmin[k])); hi[k] = fmaxf(hi[k], fdec(nb[b].bmax[k]));
          clo[k] = fminf(clo[k], fdec(nb[b].cmin[k])); chi[k] = fmaxf(chi[k], fdec(nb[b].cmax[k]));
        }
      }
      cnt[s] = c;
      for (int k = 0; k < 3; k++) { ch[s].bmin[k] = lo[k]; ch[s].bmax[k] = hi[k]; ch[s].cmin[k] = clo[k]; ch[s].cmax[k] = chi[k]; }
    }
  }
  for (int s = 0; s < 2; s++) {
    ch[s].start = nd.start + (s == 0 ? 0 : cnt[0]);
    ch[s].count = cnt[s];
    ch[s].left = -1;
    ch[s].axis = 0;
    ch[s].binSlot = -1;
    ch[s].splitBin = -1;
    nodes[left + s] = ch[s];
    if (cnt[s] > 4) {  // BVH_LEAF_SIZE (bvh.cpp:23): larger children stay open
      const int slot = atomicAdd(nextCount, 1);
      nextTasks[slot] = left + s;
    }
  }
  nd.left = left;
  nd.splitBin = split;
  nodes[id] = nd;
}

// The same split decision with one warp per open node (nbins <= 32: lane b holds
// bin b).  Left and right bounds come from inclusive warp scans of min / max (exact,
// so the same values as the sequential sweeps), the cost of each split from the
// same formula, and the choice is the lowest bin index of the lowest cost, as the
// sweeps choose.  The warp then resets its bins for the next use, so levels need
// no separate clear.
__device__ __forceinline__ void resetBin(BinData* b) {
  uint4* w = reinterpret_cast<uint4*>(b);
  w[0] = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u);  // bmin x y z, bmax x
  w[1] = make_uint4(0u, 0u, 0xFFFFFFFFu, 0xFFFFFFFFu);           // bmax y z, cmin x y
  w[2] = make_uint4(0xFFFFFFFFu, 0u, 0u, 0u);                    // cmin z, cmax x y z
  w[3] = make_uint4(0u, 0u, 0u, 0u);                             // count, pad
}

__global__ void k_resetBins(size_t count, BinData* bins) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) resetBin(bins + i);
}

template <bool MIN>
__device__ __forceinline__ float warpScanF(float v, int lane, bool reverse) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float u = reverse ? __shfl_down_sync(0xffffffffu, v, o) : __shfl_up_sync(0xffffffffu, v, o);
    const bool in = reverse ? lane + o < 32 : lane >= o;
    if (in) v = MIN ? fminf(v, u) : fmaxf(v, u);
  }
  return v;
}

__device__ __forceinline__ int warpScanI(int v, int lane, bool reverse) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = reverse ? __shfl_down_sync(0xffffffffu, v, o) : __shfl_up_sync(0xffffffffu, v, o);
    if (reverse ? lane + o < 32 : lane >= o) v += u;
  }
  return v;
}

// Split of node nd from its bins, lane b's bin in (cnt, b*, c*): ordered-uint bounds of the
// primitives and of their centroids, identities when empty.  All lanes return the split (bin,
// -1 leaf, -2 index median) and the children's counts and bounds (bmin, bmax, cmin, cmax).
// A cost that is no number (a box of NaN, an area that overflows) compares with nothing and
// can leave the lanes with different splits.  Lane 0's is the split; the node is refused (split
// -1) where another lane would put its bin on the other side.
struct WarpSplit {
  int split;
  bool refused;
  int count[2];
  float bounds[2][12];
};
__device__ __forceinline__ WarpSplit decideSplit(const BNode& nd, int nbins, int maxLeaf, int cnt, const uint32_t (&bin)[12]) {
  const int lane = threadIdx.x & 31;
  const bool any = cnt > 0;
  float blo[3], bhi[3];
  for (int k = 0; k < 3; k++) {
    blo[k] = any ? fdec(bin[k]) : FLT_MAX;
    bhi[k] = any ? fdec(bin[3 + k]) : -FLT_MAX;
  }
  // left: bins 0..lane, right: bins lane..nbins-1
  float llo[3], lhi[3], rlo[3], rhi[3];
  for (int k = 0; k < 3; k++) {
    llo[k] = warpScanF<true>(blo[k], lane, false);
    lhi[k] = warpScanF<false>(bhi[k], lane, false);
    rlo[k] = warpScanF<true>(blo[k], lane, true);
    rhi[k] = warpScanF<false>(bhi[k], lane, true);
  }
  const int lc = warpScanI(cnt, lane, false), total = __shfl_sync(0xffffffffu, lc, 31), rc = total - lc;
  // split s = lane: left = bins 0..s, right = bins s+1..nbins-1 (the right sums of lane s + 1)
  float rl[3], rh[3];
  for (int k = 0; k < 3; k++) {
    rl[k] = __shfl_down_sync(0xffffffffu, rlo[k], 1);
    rh[k] = __shfl_down_sync(0xffffffffu, rhi[k], 1);
  }
  const float pa = areaOf(nd.bmin, nd.bmax);
  const float invPa = pa > 0.0f ? 1.0f / pa : 0.0f;
  float cost = FLT_MAX;
  const bool valid = lane < nbins - 1 && lc > 0 && rc > 0;
  if (valid) {
    const float la = areaOf(llo, lhi), ra = areaOf(rl, rh);
    cost = 1.0f + 1.5f * invPa * (la * (float)lc + ra * (float)rc);
  }
  // lowest cost, then lowest split index
  float bc = cost;
  int bs = valid ? lane : 0x7fffffff;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float oc = __shfl_xor_sync(0xffffffffu, bc, o);
    const int os = __shfl_xor_sync(0xffffffffu, bs, o);
    if (oc < bc || (oc == bc && os < bs)) { bc = oc; bs = os; }
  }
  const int forced = bs == 0x7fffffff ? -1 : bs;
  const int best = (forced >= 0 && bc < (float)nd.count * 1.5f) ? forced : -1;
  WarpSplit r;
  r.split = best;
  if (best < 0 && nd.count > maxLeaf) r.split = forced >= 0 ? forced : -2;  // -2: index median
  const int own = r.split;
  r.split = __shfl_sync(0xffffffffu, own, 0);
  const bool same = !any || r.split < 0 || (own >= 0 && (lane <= own) == (lane <= r.split));
  r.refused = !__all_sync(0xffffffffu, same);
  if (r.refused) r.split = -1;
  const int at = r.split >= 0 ? r.split : 0;
  const int lcAt = __shfl_sync(0xffffffffu, lc, at);
  r.count[0] = r.split >= 0 ? lcAt : nd.count / 2;
  r.count[1] = (r.split >= 0 ? total : nd.count) - r.count[0];
  for (int k = 0; k < 3; k++) {
    // bounds: the scans at the split; centroid bounds: reductions of each side's bins
    const float l0 = __shfl_sync(0xffffffffu, llo[k], at), l1 = __shfl_sync(0xffffffffu, lhi[k], at),
                r0 = __shfl_sync(0xffffffffu, rl[k], at), r1 = __shfl_sync(0xffffffffu, rh[k], at);
    const bool onL = lane <= at;
    const uint32_t cl0 = __reduce_min_sync(0xffffffffu, any && onL ? bin[6 + k] : 0xFFFFFFFFu),
                   cl1 = __reduce_max_sync(0xffffffffu, any && onL ? bin[9 + k] : 0u),
                   cr0 = __reduce_min_sync(0xffffffffu, any && !onL ? bin[6 + k] : 0xFFFFFFFFu),
                   cr1 = __reduce_max_sync(0xffffffffu, any && !onL ? bin[9 + k] : 0u);
    const bool med = r.split < 0;
    r.bounds[0][k] = med ? nd.bmin[k] : l0;
    r.bounds[0][3 + k] = med ? nd.bmax[k] : l1;
    r.bounds[0][6 + k] = med ? nd.cmin[k] : fdec(cl0);
    r.bounds[0][9 + k] = med ? nd.cmax[k] : fdec(cl1);
    r.bounds[1][k] = med ? nd.bmin[k] : r0;
    r.bounds[1][3 + k] = med ? nd.bmax[k] : r1;
    r.bounds[1][6 + k] = med ? nd.cmin[k] : fdec(cr0);
    r.bounds[1][9 + k] = med ? nd.cmax[k] : fdec(cr1);
  }
  return r;
}

// Child `side` of a split node (one lane each).
__device__ __forceinline__ void writeChild(BNode* nodes, int left, int side, int start, const WarpSplit& sp) {
  BNode c;
  for (int k = 0; k < 3; k++) {
    c.bmin[k] = side ? sp.bounds[1][k] : sp.bounds[0][k];
    c.bmax[k] = side ? sp.bounds[1][3 + k] : sp.bounds[0][3 + k];
    c.cmin[k] = side ? sp.bounds[1][6 + k] : sp.bounds[0][6 + k];
    c.cmax[k] = side ? sp.bounds[1][9 + k] : sp.bounds[0][9 + k];
  }
  c.start = start + (side ? sp.count[0] : 0);
  c.count = side ? sp.count[1] : sp.count[0];
  c.left = -1;
  c.axis = 0;
  c.binSlot = -1;
  c.splitBin = -1;
  nodes[left + side] = c;
}

// Split decisions of a level, one warp per open node; the warp resets the bins it read.
// Children above kSubtree primitives stay open for the next level, smaller ones that can
// still split (BVH_LEAF_SIZE 4, bvh.cpp:23) go to the block-wise pass.
__global__ void __launch_bounds__(128) k_splitWarp(const int* count, int first, int most, const int* __restrict__ tasks,
                                                  BNode* nodes, BinData* bins, int nbins, int* nodeCounter, int* nextTasks,
                                                  int* nextCount, int* smallTasks, int* smallCount, int maxLeaf,
                                                  int* err) {
  const int t = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (t >= tasksOf(count, first, most)) return;
  const int id = tasks[first + t];
  const BNode nd = nodes[id];
  BinData* nb = bins + (size_t)nd.binSlot * nbins;
  int cnt = 0;
  uint32_t bin[12];
  for (int k = 0; k < 12; k++) bin[k] = 0u;
  if (lane < nbins) {
    const BinData b = nb[lane];
    cnt = (int)b.count;
    for (int k = 0; k < 3; k++) {
      bin[k] = b.bmin[k];
      bin[3 + k] = b.bmax[k];
      bin[6 + k] = b.cmin[k];
      bin[9 + k] = b.cmax[k];
    }
    resetBin(nb + lane);
  }
  const WarpSplit sp = decideSplit(nd, nbins, maxLeaf, cnt, bin);
  int left = -1;
  if (lane == 0) {
    if (sp.refused) atomicCAS(err, 0, kErrPartition);
    if (sp.split != -1) left = atomicAdd(nodeCounter, 2);
    nodes[id].binSlot = -1;
    nodes[id].left = left;
    nodes[id].splitBin = sp.split;
  }
  if (sp.split == -1) return;
  left = __shfl_sync(0xffffffffu, left, 0);
  if (lane < 2) {
    writeChild(nodes, left, lane, nd.start, sp);
    const int c = lane ? sp.count[1] : sp.count[0];
    if (c > kSubtree) nextTasks[atomicAdd(nextCount, 1)] = left + lane;
    else if (c > 4) smallTasks[atomicAdd(smallCount, 1)] = left + lane;
  }
}

// Nodes of at most kSubtree primitives: one block splits each to the end, level by level with
// a warp per node, bounds and order in shared memory.  The same bins, costs and stable
// partition as the device-wide levels, so the tree is the same.  Bound by the latency of a
// node's scans and reductions (about 1 us) over the nodes of a block's deepest chain.
constexpr int kSubThreads = 256;
__global__ void __launch_bounds__(kSubThreads) k_subtrees(const int* __restrict__ count, const int* __restrict__ tasks,
                                                          BNode* nodes, int* primIdx, const float4* __restrict__ bmin,
                                                          const float4* __restrict__ bmax, int nbins, int* nodeCounter,
                                                          int maxLeaf, int* err) {
  constexpr int kWarps = kSubThreads / 32, kList = kSubtree / 5 + 1;  // nodes of five primitives and more
  __shared__ float sB[6][kSubtree];
  __shared__ int sIdx[kSubtree];
  __shared__ uint16_t sPerm[2][kSubtree];
  __shared__ uint32_t sBins[kWarps][32][13];
  __shared__ int sList[2][kList];
  __shared__ int sCount[2], sBase;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) sBase = *(volatile int*)err ? 0 : *count;  // one answer for the block: others may set it
  __syncthreads();
  const int numTasks = sBase;
  __syncthreads();
  for (int task = blockIdx.x; task < numTasks; task += gridDim.x) {
    const int root = tasks[task];
    const int start = nodes[root].start, n = nodes[root].count;
    for (int i = threadIdx.x; i < n; i += kSubThreads) {
      const float4 lo = bmin[start + i], hi = bmax[start + i];
      sB[0][i] = lo.x; sB[1][i] = lo.y; sB[2][i] = lo.z;
      sB[3][i] = hi.x; sB[4][i] = hi.y; sB[5][i] = hi.z;
      sIdx[i] = primIdx[start + i];
      sPerm[0][i] = (uint16_t)i;
    }
    if (threadIdx.x == 0) {
      sList[0][0] = root;
      sCount[0] = 1;
    }
    for (int cur = 0;; cur ^= 1) {
      __syncthreads();
      const int L = sCount[cur];
      if (L == 0) break;
      if (threadIdx.x == 0) {
        sBase = atomicAdd(nodeCounter, 2 * L);  // ids for every node of this level to split
        sCount[cur ^ 1] = 0;
      }
      __syncthreads();
      for (int e = warp; e < L; e += kWarps) {
        const int id = sList[cur][e], left = sBase + 2 * e;
        BNode nd = nodes[id];
        nd.axis = widestAxis(nd);
        const int s0 = nd.start - start;
        const bool flat = !(nd.cmax[nd.axis] - nd.cmin[nd.axis] >= 1e-12f);
        uint32_t (&bins)[32][13] = sBins[warp];
        for (int k = 0; k < 3; k++) {
          bins[lane][k] = bins[lane][6 + k] = 0xFFFFFFFFu;
          bins[lane][3 + k] = bins[lane][9 + k] = 0u;
        }
        bins[lane][12] = 0u;
        __syncwarp();
        auto binAt = [&](int p) {
          return binOf(nd, (sB[nd.axis][p] + sB[3 + nd.axis][p]) * 0.5f, nbins);
        };
        if (!flat)
          for (int j = lane; j < nd.count; j += 32) {
            const int p = sPerm[0][s0 + j];
            uint32_t v[12];
            for (int k = 0; k < 3; k++) {
              const float lo = sB[k][p], hi = sB[3 + k][p];
              v[k] = fenc(lo);
              v[3 + k] = fenc(hi);
              v[6 + k] = v[9 + k] = fenc((lo + hi) * 0.5f);
            }
            binPrim(bins[binAt(p)], v, 1u);
          }
        __syncwarp();
        uint32_t bin[12];
        for (int k = 0; k < 12; k++) bin[k] = bins[lane][k];
        const WarpSplit sp = decideSplit(nd, nbins, maxLeaf, lane < nbins ? (int)bins[lane][12] : 0, bin);
        if (lane == 0) {
          if (sp.refused) atomicCAS(err, 0, kErrPartition);
          nodes[id].axis = nd.axis;
          nodes[id].binSlot = -1;
          nodes[id].left = sp.split == -1 ? -1 : left;
          nodes[id].splitBin = sp.split;
        }
        if (sp.split == -1) {  // its two ids stay unused
          if (lane < 2) nodes[left + lane].left = -1;
          continue;
        }
        if (lane < 2) {
          writeChild(nodes, left, lane, nd.start, sp);
          if ((lane ? sp.count[1] : sp.count[0]) > 4) sList[cur ^ 1][atomicAdd(&sCount[cur ^ 1], 1)] = left + lane;
        }
        // stable partition of the node's places through the second order array
        int nl = 0;
        for (int j0 = 0; j0 < nd.count; j0 += 32) {
          const int j = j0 + lane;
          const bool in = j < nd.count;
          const int p = in ? sPerm[0][s0 + j] : 0;
          const bool toLeft = in && (sp.split == -2 ? j < sp.count[0] : binAt(p) <= sp.split);
          const unsigned m = __ballot_sync(0xffffffffu, toLeft);
          const int before = nl + __popc(m & ((1u << lane) - 1u));
          const int to = toLeft ? before : sp.count[0] + j - before;
          if (in && to < nd.count) sPerm[1][s0 + to] = (uint16_t)p;
          nl += __popc(m);
        }
        __syncwarp();
        if (nl == sp.count[0]) {  // else not every place was written: the order stays
          for (int j = lane; j < nd.count; j += 32) sPerm[0][s0 + j] = sPerm[1][s0 + j];
        } else if (lane == 0) {
          atomicCAS(err, 0, kErrPartition);
        }
        __syncwarp();
      }
    }
    for (int i = threadIdx.x; i < n; i += kSubThreads) primIdx[start + i] = sIdx[sPerm[0][i]];
    __syncthreads();  // before the next task's data overwrite this one's
  }
}

// Partition, pass 1: flag 1 for a primitive that goes to the left child of its
// node (the split bin, or the first half of the node's range for a median split).
// A pass of its own: computed inside the prefix sum the flags cost more (4M primitives 66
// against 31 + 12 us, 20k 31 against 10).
__global__ void k_partitionFlags(int n, const int* __restrict__ primNode, const BNode* __restrict__ nodes,
                                 const float4* __restrict__ bmin, const float4* __restrict__ bmax, int nbins,
                                 int* __restrict__ flags, const int* __restrict__ err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const bool failed = *err != 0;
  int node = primNode[i];
  if (failed) node = -1;
  int flag = 0;
  if (node >= 0) {
    const BNode& nd = nodes[node];
    if (nd.left >= 0) {
      if (nd.splitBin == -2) {
        flag = (i - nd.start) < nd.count / 2 ? 1 : 0;
      } else {
        const float c = (axisOf(bmin[i], nd.axis) + axisOf(bmax[i], nd.axis)) * 0.5f;
        flag = binOf(nd, c, nbins) <= nd.splitBin ? 1 : 0;
      }
    }
  }
  flags[i] = flag;
}

// Partition, pass 2 (after an exclusive scan of the flags into `before`): a stable
// scatter of each split node's primitives into its children's ranges, with their
// bounds; primitives of closed nodes and new leaves stay where they are.  No
// atomics, so the order (and the BVH) is the same on every run.  A primitive past its
// child's range is an error of the build; it is not written, and the kernels launched behind
// take every primitive, also one that was never written, as closed.
__global__ void k_partitionScatter(int n, const int* __restrict__ primIdx, const int* __restrict__ primNode,
                                   const BNode* __restrict__ nodes, const float4* __restrict__ bmin,
                                   const float4* __restrict__ bmax, const int* __restrict__ flags,
                                   const int* __restrict__ before, int* __restrict__ outIdx, int* __restrict__ outNode,
                                   float4* __restrict__ outMin, float4* __restrict__ outMax, int openCount, int* err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const bool failed = *err != 0;
  int node = primNode[i];
  if (failed) node = -1;
  int pos = i, outN = -1;
  if (node >= 0) {
    const BNode& nd = nodes[node];
    if (nd.left >= 0) {
      const int leftBefore = before[i] - before[nd.start];
      const int side = flags[i] ? 0 : 1;
      const int rank = side == 0 ? leftBefore : (i - nd.start) - leftBefore;
      const BNode& cn = nodes[nd.left + side];
      if (rank >= cn.count) {
        atomicCAS(err, 0, kErrPartition);
        return;
      }
      pos = cn.start + rank;
      outN = cn.count > openCount ? nd.left + side : -1;  // smaller ones are closed for the levels
    }
  }
  outIdx[pos] = primIdx[i];
  outNode[pos] = outN;
  outMin[pos] = bmin[i];
  outMax[pos] = bmax[i];
}

__global__ void k_innerFlags(int numNodes, const BNode* __restrict__ nodes, int* flags) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < numNodes) flags[i] = nodes[i].left >= 0 ? 1 : 0;
}

__device__ __forceinline__ float inflateLo(float x) { return x - fmaxf(fabsf(x), 1.0f) * 2e-6f; }
__device__ __forceinline__ float inflateHi(float x) { return x + fmaxf(fabsf(x), 1.0f) * 2e-6f; }

__global__ void k_emitNodes(int numNodes, const BNode* __restrict__ nodes, const int* __restrict__ travIdx,
                            float4* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= numNodes) return;
  const BNode nd = nodes[i];
  if (nd.left < 0) return;
  const BNode a = nodes[nd.left], b = nodes[nd.left + 1];
  int refs[2];
  const BNode* cs[2] = {&a, &b};
  for (int s = 0; s < 2; s++) {
    const BNode& c = *cs[s];
    if (c.left >= 0) refs[s] = travIdx[nd.left + s];
    else refs[s] = ~((c.start << 3) | (c.count - 1));
  }
  float4* o = out + (size_t)travIdx[i] * 4;
  o[0] = make_float4(inflateLo(a.bmin[0]), inflateHi(a.bmax[0]), inflateLo(a.bmin[1]), inflateHi(a.bmax[1]));
  o[1] = make_float4(inflateLo(b.bmin[0]), inflateHi(b.bmax[0]), inflateLo(b.bmin[1]), inflateHi(b.bmax[1]));
  o[2] = make_float4(inflateLo(a.bmin[2]), inflateHi(a.bmax[2]), inflateLo(b.bmin[2]), inflateHi(b.bmax[2]));
  o[3] = make_float4(__int_as_float(refs[0]), __int_as_float(refs[1]), 0.0f, 0.0f);
}

__global__ void k_gather(int n, const int* __restrict__ primIdx, const float4* __restrict__ vIn,
                         const float4* __restrict__ sIn, const float2* __restrict__ uvIn, float4* __restrict__ vOut,
                         float4* __restrict__ sOut, float2* __restrict__ uvOut, int* __restrict__ orig) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int p = primIdx[i];
  for (int k = 0; k < 3; k++) {
    vOut[(size_t)i * 3 + k] = vIn[(size_t)p * 3 + k];
    sOut[(size_t)i * 3 + k] = sIn[(size_t)p * 3 + k];
    if (uvOut) uvOut[(size_t)i * 3 + k] = uvIn[(size_t)p * 3 + k];
  }
  orig[i] = p;
}


// ---- 8-wide BVH (collapse of the binary build) ---------------------------------
// Node (128 B = kNode8Vec float4; word k is stored at word k ^ (node index % 8)):
//   (childBase, triBase, meta[0..3], meta[4..7])
//   (origin x, y, z, scale | inner mask)
//   per axis x, y, z: 8 half lo planes, 8 half hi planes of the child boxes
// A plane lies at origin + scale * half value; scale is a power of two (its exponent
// bits, in place) that maps the node's extent to at most 2^15, so thin axes keep
// their precision, and planes are rounded outward.  meta[s] = (count << 5) | offset: a
// leaf of `count` (1..4) triangles at triBase + offset; 0 for an inner child, stored at
// childBase + (inner slots below s), and for an empty slot, which has an inverted box.
// Slots are assigned per octant: a child whose centre lies on the negative side
// of the node centre along axis k prefers slots with bit k set, so visiting hit
// slots in descending order of (slot XOR ray octant) is roughly front to back.
// Eight lanes collapse one task (binary node task.x becomes wide node task.y), a lane per child
// and then per slot: one thread per node took 53 us a level, the latency of its chain of
// node reads and 8 x 8 slot scores, whatever the number of nodes.  Nodes past maxNodes8 are
// counted and their children followed, but not written (the host then sizes the array and
// repeats).
__global__ void __launch_bounds__(128) k_collapse(const int* __restrict__ count, const int2* __restrict__ tasks,
                                                  const BNode* __restrict__ nodes, const int* __restrict__ primIdx,
                                                  float4* __restrict__ nodes8, int* counters, int2* __restrict__ nextTasks,
                                                  int* nextCount, int* __restrict__ triOrder, int maxNodes8,
                                                  const int* __restrict__ err) {
  constexpr unsigned kAll = 0xffffffffu;
  const int numTasks = *err ? 0 : *count;
  const int lane = threadIdx.x & 7, shift = threadIdx.x & 24;  // lane of the node's eight, their place in the warp
  auto of = [&](auto v, int l) { return __shfl_sync(kAll, v, l, 8); };
  auto minOf = [&](float v) {
    for (int o = 4; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(kAll, v, o));
    return v;
  };
  auto maxOf = [&](float v) {
    for (int o = 4; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kAll, v, o));
    return v;
  };
  auto sumOf = [&](float v) {
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(kAll, v, o);
    return v;
  };
  const int stride = (int)(gridDim.x * blockDim.x) >> 3;
  // whole warps: a group past the last task goes along without one
  for (int t0 = (int)(blockIdx.x * blockDim.x + (threadIdx.x & ~31)) >> 3; t0 < numTasks; t0 += stride) {
    const int t = t0 + (shift >> 3);
    const bool on = t < numTasks;
    const int2 task = on ? tasks[t] : make_int2(0, 0);
    // children by opening the inner child of the largest area until there are eight
    int id = -1, left = -1, cnt = 0, first = 0;
    float bmin[3] = {0, 0, 0}, bmax[3] = {0, 0, 0}, area = -1.0f;
    auto load = [&](int node) {
      const BNode& c = nodes[node];
      id = node;
      left = c.left;
      cnt = c.count;
      first = c.start;
      for (int k = 0; k < 3; k++) {
        bmin[k] = c.bmin[k];
        bmax[k] = c.bmax[k];
      }
      area = left >= 0 ? areaOf(bmin, bmax) : -1.0f;
    };
    int nc = on ? 1 : 0;
    const int rootLeft = on ? nodes[task.x].left : -1;
    if (on) {
      if (rootLeft < 0) {
        if (lane == 0) load(task.x);
      } else {
        nc = 2;
        if (lane < 2) load(rootLeft + lane);
      }
    }
    for (int it = 0; it < 6; it++) {
      const float best = maxOf(area);
      const unsigned m = (__ballot_sync(kAll, area == best && best >= 0.0f) >> shift) & 0xffu;
      if (__ballot_sync(kAll, m != 0 && nc < 8) == 0) break;
      const int who = m ? __ffs(m) - 1 : 0;  // the first of equal areas
      const int l = of(left, who);
      if (m && nc < 8) {
        if (lane == who) load(l);
        else if (lane == nc) load(l + 1);
        nc++;
      }
    }
    // node bounds of the widened child boxes, their centre, and greedy octant slots
    const bool mine = lane < nc;
    float lo[3], hi[3], ctr[3], cc[3];
    for (int k = 0; k < 3; k++) {
      lo[k] = minOf(mine ? inflateLo(bmin[k]) : FLT_MAX);
      hi[k] = maxOf(mine ? inflateHi(bmax[k]) : -FLT_MAX);
      ctr[k] = 0.5f * (lo[k] + hi[k]);
      cc[k] = 0.5f * (bmin[k] + bmax[k]);
    }
    int slot = -1;
    unsigned used = 0;
    for (int it = 0; it < 8; it++) {
      float bestS = -INFINITY;
      int bs = -1;
      if (mine && slot < 0)
        for (int sl = 0; sl < 8; sl++) {
          if ((used >> sl) & 1u) continue;
          const float sc = (cc[0] - ctr[0]) * ((sl & 1) ? -1.0f : 1.0f) + (cc[1] - ctr[1]) * ((sl & 2) ? -1.0f : 1.0f) +
                           (cc[2] - ctr[2]) * ((sl & 4) ? -1.0f : 1.0f);
          if (bs < 0 || sc > bestS) { bestS = sc; bs = sl; }
        }
      const bool cand = bs >= 0;
      const float top = maxOf(cand ? bestS : -INFINITY);
      unsigned m = (__ballot_sync(kAll, cand && bestS == top) >> shift) & 0xffu;
      const unsigned anyCand = (__ballot_sync(kAll, cand) >> shift) & 0xffu;
      if (__ballot_sync(kAll, anyCand != 0) == 0) break;
      if (!m) m = anyCand;  // scores that are no numbers: any order will do
      const int who = m ? __ffs(m) - 1 : 0;
      const int s = of(bs, who);
      if (m) {
        used |= 1u << s;
        if (lane == who) slot = s;
      }
    }
    // from here a lane stands for slot `lane`
    int from = -1;
    for (int j = 0; j < 8; j++)
      if (of(slot, j) == lane) from = j;
    const bool full = from >= 0;
    const int src = full ? from : lane;
    const int cId = of(id, src), cLeft = of(left, src), cCnt = of(cnt, src), cFirst = of(first, src);
    float cMin[3], cMax[3];
    for (int k = 0; k < 3; k++) {
      cMin[k] = of(bmin[k], src);
      cMax[k] = of(bmax[k], src);
    }
    const bool inner = full && cLeft >= 0, leaf = full && cLeft < 0;
    const unsigned innerMask = (__ballot_sync(kAll, inner) >> shift) & 0xffu;
    const int ni = __popc(innerMask), rank = __popc(innerMask & ((1u << lane) - 1u));
    int off = leaf ? cCnt : 0;  // triangles of the slots up to this one
    for (int o = 1; o < 8; o <<= 1) {
      const int up = __shfl_up_sync(kAll, off, o, 8);
      if (lane >= o) off += up;
    }
    const int ntri = of(off, 7);
    off -= leaf ? cCnt : 0;
    int childBase = 0, triBase = 0, taskBase = 0;
    if (lane == 0 && on) {
      if (ni) {
        childBase = atomicAdd(&counters[0], ni);
        taskBase = atomicAdd(nextCount, ni);
      }
      triBase = atomicAdd(&counters[1], ntri);
    }
    childBase = of(childBase, 0);
    triBase = of(triBase, 0);
    taskBase = of(taskBase, 0);
    if (on && inner) nextTasks[taskBase + rank] = make_int2(cId, childBase + rank);
    if (on && leaf)
      for (int q = 0; q < cCnt; q++) triOrder[triBase + off + q] = primIdx[cFirst + q];
    // The origin of the planes is, per axis, the node's low end, centre or high end: the one
    // closest to the planes of thin boxes (walls, floors, lamps), whose rounding matters most
    // because rays start and end at such surfaces.
    // margin: against the slab test's rounding, which is up to 2 x 2^-24 of the planes' distance from
    // their origin besides a part that grows with the ray's way to the box (kNearScale)
    float org[3], margin[3], ext = 0.0f;
    for (int k = 0; k < 3; k++) {
      const float cand[3] = {ctr[k], lo[k], hi[k]}, thin = (hi[k] - lo[k]) * (1.0f / 256.0f);
      float best = FLT_MAX;
      org[k] = ctr[k];
      for (int q = 0; q < 3; q++) {
        const float cost =
            sumOf(full ? (fabsf(cMin[k] - cand[q]) + fabsf(cMax[k] - cand[q])) / (cMax[k] - cMin[k] + thin) : 0.0f);
        if (cost < best) {
          best = cost;
          org[k] = cand[q];
        }
      }
      const float e = fmaxf(__fsub_ru(hi[k], org[k]), __fsub_ru(org[k], lo[k]));
      margin[k] = e * (8.0f / 16777216.0f);
      ext = fmaxf(ext, __fadd_ru(e, margin[k]));
    }
    // planes as half values, rounded outward; an empty slot keeps an inverted box, and a node
    // that is not of finite size has boxes that every ray enters
    const bool finite = ext < 1e30f;
    int exponent = 0;
    if (finite) frexpf(ext, &exponent);  // ext < 2^exponent
    exponent = max(exponent - 15, -126);
    const float scale = ldexpf(1.0f, exponent), toHalf = ldexpf(1.0f, -exponent);
    uint32_t meta = leaf ? (uint32_t)((cCnt << 5) | off) << (8 * (lane & 3)) : 0u;
    meta |= __shfl_xor_sync(kAll, meta, 1);
    meta |= __shfl_xor_sync(kAll, meta, 2);
    const uint32_t meta1 = of(meta, 4);
    if (!on || task.y >= maxNodes8) continue;
    float4* o = nodes8 + (size_t)task.y * kNode8Vec;
    const int sw = task.y & 7;
    for (int k = 0; k < 3; k++)
      for (int h = 0; h < 2; h++) {
        __half v = __float2half_rn(h ? -65504.0f : 65504.0f);
        if (full) {
          if (!finite) v = h ? __float2half_ru(INFINITY) : __float2half_rd(-INFINITY);
          else if (h) v = __float2half_ru(__fsub_ru(inflateHi(cMax[k]) + margin[k], org[k]) * toHalf);
          else v = __float2half_rd(__fsub_rd(inflateLo(cMin[k]) - margin[k], org[k]) * toHalf);
        }
        reinterpret_cast<__half*>(o + ((2 + 2 * k + h) ^ sw))[lane] = v;
      }
    if (lane == 0) {
      o[0 ^ sw] = make_float4(__int_as_float(childBase), __int_as_float(triBase), __uint_as_float(meta), __uint_as_float(meta1));
      o[1 ^ sw] = make_float4(finite ? org[0] : 0.0f, finite ? org[1] : 0.0f, finite ? org[2] : 0.0f,
                              __uint_as_float(__float_as_uint(scale) | innerMask));
    }
  }
}

__global__ void k_initCollapse(int* counters, int* levelCount, int2* tasks) {
  counters[0] = 1;  // nodes: the root
  counters[1] = 0;  // triangles
  levelCount[0] = 1;
  tasks[0] = make_int2(0, 0);
}

inline int gridFor(long long n, int block) { return (int)((n + block - 1) / block); }

}  // namespace

// Per-level host timing of the build, printed to stderr when RG_TRACE_HOST is set.
struct BuildTrace {
  bool on = std::getenv("RG_TRACE_HOST") != nullptr;
  std::chrono::steady_clock::time_point last = std::chrono::steady_clock::now();
  void mark(const char* what, int level, int tasks) {
    if (!on) return;
    const auto t = std::chrono::steady_clock::now();
    std::fprintf(stderr, "[rg] bvh %-10s %3d: %8d tasks %8.3f ms\n", what, level, tasks,
                 std::chrono::duration<double, std::milli>(t - last).count());
    last = t;
  }
};

// The build's working arrays; a scene rebuilt in place keeps them, so a build no
// larger than the last allocates nothing (DevBuf::alloc only grows).
struct BvhScratch {
  DevBuf<float4> vTmp, sTmp, lo, hi, lo2, hi2;
  DevBuf<float2> uvTmp;
  DevBuf<uint32_t> rb;
  DevBuf<BNode> nodes;
  DevBuf<int> idxA, idxB, nodeA, nodeB, tasksA, tasksB, smallTasks, counters, levelCount, pflags, pbefore;
  DevBuf<BinData> bins;
  DevBuf<unsigned char> scanTmp, tmp;
  DevBuf<int2> ta, tb;
  DevBuf<int> order, c8, flags, trav;
};

void freeBvhScratch(BvhScratch* s) { delete s; }

// Builds the view-space triangle arrays and the BVH of a scene whose world-space inputs are already
// on the device (DeviceScene::in*).  Grids of looping kernels count the 148 SMs of a B200.
rg_status buildDeviceBvh(DeviceScene& ds, int nbins, bool wide, cudaStream_t st, std::string& err) {
  BuildTrace trace;
  const int n = ds.numTris;
  nbins = nbins < 2 ? 2 : (nbins > kMaxBins ? kMaxBins : nbins);
  ds.rootIsLeaf = 0;
  ds.rootLeafRef = 0;
  ds.numNodes = 0;
  if (n == 0) return RG_OK;
  if (!ds.scratch) ds.scratch = new BvhScratch();
  BvhScratch& X = *ds.scratch;
  DevBuf<float4> &vTmp = X.vTmp, &sTmp = X.sTmp, &lo = X.lo, &hi = X.hi, &lo2 = X.lo2, &hi2 = X.hi2;
  DevBuf<float2>& uvTmp = X.uvTmp;
  if (!vTmp.alloc((size_t)n * 3) || !sTmp.alloc((size_t)n * 3) || !lo.alloc(n) || !hi.alloc(n)) {
    err = "out of device memory (triangle staging)";
    return RG_ERR_OUT_OF_MEMORY;
  }
  if (ds.hasUV && !uvTmp.alloc((size_t)n * 3)) {
    err = "out of device memory (triangle staging)";
    return RG_ERR_OUT_OF_MEMORY;
  }
  trace.mark("alloc stage", 0, n);
  k_prepTriangles<<<gridFor(n, 256), 256, 0, st>>>(n, ds.inPos.p, ds.inNrm.p, ds.hasUV ? ds.inUV.p : nullptr,
                                                   ds.inTriMesh.p, ds.meshObj.p, ds.objMat.p, ds.mats.p, ds.view.p,
                                                   vTmp.p, sTmp.p, ds.hasUV ? uvTmp.p : nullptr, lo.p, hi.p);
  // root bounds
  DevBuf<uint32_t>& rb = X.rb;
  if (!rb.alloc(12)) {
    err = "out of device memory (BVH build)";
    return RG_ERR_OUT_OF_MEMORY;
  }
  k_initBounds<<<1, 32, 0, st>>>(rb.p);
  k_rootBounds<<<std::min(gridFor(n, 256), 1184), 256, 0, st>>>(n, lo.p, hi.p, rb.p);
  const size_t maxNodes = 2 * (size_t)n + 1;
  // up to 32 bins: nodes of at most kSubtree primitives are left to k_subtrees, and one warp
  // per larger node decides its split
  const bool warpSplit = nbins <= 32;
  const int openCount = warpSplit ? kSubtree : 4;  // more primitives than this stay open for the levels
  const int maxOpen = n / (openCount + 1) + 1;     // open nodes of a level
  // bins for at most chunkTasks open nodes at a time (<= 256 MB)
  const int chunkTasks = (int)std::min<size_t>((size_t)maxOpen, ((size_t)256 << 20) / (sizeof(BinData) * nbins));
  DevBuf<BNode>& nodes = X.nodes;
  DevBuf<int> &idxA = X.idxA, &idxB = X.idxB, &nodeA = X.nodeA, &nodeB = X.nodeB, &tasksA = X.tasksA,
  &tasksB = X.tasksB, &smallTasks = X.smallTasks, &counters = X.counters, &levelCount = X.levelCount,
  &pflags = X.pflags, &pbefore = X.pbefore;
  DevBuf<BinData>& bins = X.bins;
  trace.mark("prep kern", 0, n);
  constexpr int kMaxLevels = 200;
  if (!nodes.alloc(maxNodes) || !idxA.alloc(n) || !idxB.alloc(n) || !nodeA.alloc(n) || !nodeB.alloc(n) ||
      !lo2.alloc(n) || !hi2.alloc(n) || !pflags.alloc(n) || !pbefore.alloc(n) || !tasksA.alloc((size_t)maxOpen + 1) ||
      !tasksB.alloc((size_t)maxOpen + 1) || !smallTasks.alloc((size_t)n / 5 + 2) || !counters.alloc(C_BUILD_COUNTERS) ||
      !levelCount.alloc(kMaxLevels + 2) || !bins.alloc((size_t)chunkTasks * nbins)) {
    err = "out of device memory (BVH build)";
    return RG_ERR_OUT_OF_MEMORY;
  }
  const int rootOpen = n <= 4 ? 0 : (n > openCount ? 1 : 2);
  cudaMemsetAsync(levelCount.p, 0, sizeof(int) * (kMaxLevels + 2), st);
  k_initRoot<<<gridFor(n, 256), 256, 0, st>>>(n, rb.p, nodes.p, idxA.p, nodeA.p, rootOpen, counters.p, levelCount.p,
                                              tasksA.p, smallTasks.p);
  int* curIdx = idxA.p;
  int* curNode = nodeA.p;
  int* altIdx = idxB.p;
  int* altNode = nodeB.p;
  int* curTasks = tasksA.p;
  int* nxtTasks = tasksB.p;
  float4* curLo = lo.p;
  float4* curHi = hi.p;
  float4* altLo = lo2.p;
  float4* altHi = hi2.p;
  int levels = 0;
  trace.mark("alloc tree", 0, n);
  if (rootOpen == 1) {
    if (warpSplit) {  // k_splitWarp resets the bins it reads, so they start reset once here
      const size_t nb = (size_t)chunkTasks * nbins;
      k_resetBins<<<(unsigned)((nb + 255) / 256), 256, 0, st>>>(nb, bins.p);
    }
    // scratch of the partition's prefix sum
    size_t scanBytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, scanBytes, pflags.p, pbefore.p, n, st);
    DevBuf<unsigned char>& scanTmp = X.scanTmp;
    if (!scanTmp.alloc(scanBytes + 16)) {
      err = "out of device memory (BVH build)";
      return RG_ERR_OUT_OF_MEMORY;
    }
    // The levels a balanced tree takes to reach openCount, and two, are launched without
    // waiting (task counts stay on the device; a level without tasks copies the primitives);
    // then the host looks at the count before each further level.
    int ahead = 2;
    for (long long c = n; c > openCount; c = (c + 1) / 2) ahead++;
    int numTasks = 1;
    while (numTasks > 0) {
      const int most = (int)std::min<long long>(levels < 31 ? 1ll << levels : (long long)maxOpen, maxOpen);
      const int* count = levelCount.p + levels;
      int* nextCount = levelCount.p + levels + 1;
      for (int c0 = 0; c0 < most; c0 += chunkTasks) {
        const int nt = std::min(chunkTasks, most - c0);
        k_prepareLevel<<<gridFor(warpSplit ? nt : (long long)nt * nbins, 256), 256, 0, st>>>(count, c0, nt, curTasks, nodes.p,
                                                                                          bins.p, nbins, !warpSplit);
        if (warpSplit) {
          k_bin<<<gridFor(n, kBinChunk), 256, 0, st>>>(n, curNode, nodes.p, curLo, curHi, bins.p, nbins,
                                                   counters.p + C_BUILD_ERROR);
          k_splitWarp<<<gridFor((long long)nt * 32, 128), 128, 0, st>>>(
              count, c0, nt, curTasks, nodes.p, bins.p, nbins, counters.p + C_NODES, nxtTasks, nextCount, smallTasks.p,
              counters.p + C_SMALL, wide ? kWideMaxLeaf : kMaxLeaf, counters.p + C_BUILD_ERROR);
        } else {
          k_binAny<<<gridFor(n, kBinChunk), 256, 0, st>>>(n, curNode, nodes.p, curLo, curHi, bins.p, nbins,
                                                   counters.p + C_BUILD_ERROR);
          k_split<<<gridFor(nt, 128), 128, 0, st>>>(count, c0, nt, curTasks, nodes.p, bins.p, nbins, counters.p + C_NODES,
                                                     nxtTasks, nextCount, wide ? kWideMaxLeaf : kMaxLeaf);
        }
      }
      k_partitionFlags<<<gridFor(n, 256), 256, 0, st>>>(n, curNode, nodes.p, curLo, curHi, nbins, pflags.p,
                                                          counters.p + C_BUILD_ERROR);
      cub::DeviceScan::ExclusiveSum(scanTmp.p, scanBytes, pflags.p, pbefore.p, n, st);
      k_partitionScatter<<<gridFor(n, 256), 256, 0, st>>>(n, curIdx, curNode, nodes.p, curLo, curHi, pflags.p, pbefore.p, altIdx,
                                                          altNode, altLo, altHi, openCount, counters.p + C_BUILD_ERROR);
      std::swap(curIdx, altIdx);
      std::swap(curNode, altNode);
      std::swap(curLo, altLo);
      std::swap(curHi, altHi);
      std::swap(curTasks, nxtTasks);
      levels++;
      if (levels >= ahead) {
        cudaMemcpyAsync(&numTasks, nextCount, sizeof(int), cudaMemcpyDeviceToHost, st);
        if (cudaStreamSynchronize(st) != cudaSuccess) {
          err = "BVH build level failed";
          return RG_ERR_CUDA;
        }
        trace.mark("levels", levels, numTasks);
        if (numTasks > 0 && levels >= kMaxLevels) {
          err = "BVH build did not converge";
          return RG_ERR_DEVICE_STATUS;
        }
      }
    }
  }
  if (warpSplit && n > 4)
    k_subtrees<<<std::min(n / 5 + 1, 148 * 8), kSubThreads, 0, st>>>(counters.p + C_SMALL, smallTasks.p, nodes.p, curIdx,
                                                                    curLo, curHi, nbins, counters.p + C_NODES,
                                                                    wide ? kWideMaxLeaf : kMaxLeaf,
                                                                    counters.p + C_BUILD_ERROR);
  ds.buildLevels = levels;
  if (!ds.triVerts.alloc((size_t)n * 3) || !ds.triShade.alloc((size_t)n * 3) || !ds.triOrig.alloc(n)) {
    err = "out of device memory (triangles)";
    return RG_ERR_OUT_OF_MEMORY;
  }
  if (ds.hasUV && !ds.triUV.alloc((size_t)n * 3)) {
    err = "out of device memory (triangles)";
    return RG_ERR_OUT_OF_MEMORY;
  }
  trace.mark("alloc tris", 0, n);
  if (wide) {
    // collapse to the 8-wide layout, level by level, the task counts on the device; an inner
    // binary node has five primitives or more, which bounds the tasks of a level
    ds.bvhWidth = 8;
    DevBuf<int2> &ta = X.ta, &tb = X.tb;
    DevBuf<int> &order = X.order, &c8 = X.c8;
    // the node array: as allocated, or about what scenes need (0.08-0.13 nodes a triangle)
    int cap = (int)std::max<size_t>(ds.nodes8.n / kNode8Vec, (size_t)n / 7 + 64);
    if (!ta.alloc((size_t)n / 5 + 2) || !tb.alloc((size_t)n / 5 + 2) || !order.alloc(n) || !c8.alloc(2) ||
        !ds.nodes8.alloc((size_t)cap * kNode8Vec)) {
      err = "out of device memory (wide BVH)";
      return RG_ERR_OUT_OF_MEMORY;
    }
    int h8[2] = {0, 0}, buildErr = 0;  // nodes, triangles
    for (int pass = 0;; pass++) {
      cudaMemsetAsync(levelCount.p, 0, sizeof(int) * (kMaxLevels + 2), st);
      k_initCollapse<<<1, 1, 0, st>>>(c8.p, levelCount.p, ta.p);
      int2* cur = ta.p;
      int2* nxt = tb.p;
      int more = 1, lv = 0, ahead = 2;
      for (long long c = n; c > 4; c /= 6) ahead++;
      while (more > 0) {
        const long long most = std::min<long long>((long long)n / 5 + 2, lv < 10 ? 1ll << (3 * lv) : (long long)n);
        k_collapse<<<(int)std::min<long long>((most + 15) / 16, 148 * 16), 128, 0, st>>>(
            levelCount.p + lv, cur, nodes.p, curIdx, ds.nodes8.p, c8.p, nxt, levelCount.p + lv + 1, order.p, cap,
            counters.p + C_BUILD_ERROR);
        std::swap(cur, nxt);
        if (++lv < ahead) continue;
        cudaMemcpyAsync(&more, levelCount.p + lv, sizeof(int), cudaMemcpyDeviceToHost, st);
        cudaMemcpyAsync(h8, c8.p, sizeof(h8), cudaMemcpyDeviceToHost, st);
        cudaMemcpyAsync(&buildErr, counters.p + C_BUILD_ERROR, sizeof(int), cudaMemcpyDeviceToHost, st);
        if (cudaStreamSynchronize(st) != cudaSuccess) {
          err = "wide BVH collapse failed";
          return RG_ERR_CUDA;
        }
        trace.mark("collapse", lv, h8[0]);
        if (buildErr != 0) {
          err = "BVH build scatter error " + std::to_string(buildErr);
          return RG_ERR_DEVICE_STATUS;
        }
        if (more > 0 && lv >= kMaxLevels) {
          err = "wide BVH collapse did not converge";
          return RG_ERR_DEVICE_STATUS;
        }
      }
      if (h8[0] <= cap || pass > 0) break;
      cap = h8[0];  // more nodes than the array held: once more with the exact size
      if (!ds.nodes8.alloc((size_t)cap * kNode8Vec)) {
        err = "out of device memory (wide BVH)";
        return RG_ERR_OUT_OF_MEMORY;
      }
    }
    if (h8[1] != n || h8[0] < 1 || h8[0] > cap) {
      err = "wide BVH collapse error (nodes " + std::to_string(h8[0]) + ", triangles " + std::to_string(h8[1]) + ")";
      return RG_ERR_DEVICE_STATUS;
    }
    ds.numNodes8 = h8[0];
    ds.numNodes = 0;
    k_gather<<<gridFor(n, 256), 256, 0, st>>>(n, order.p, vTmp.p, sTmp.p, ds.hasUV ? uvTmp.p : nullptr, ds.triVerts.p,
                                              ds.triShade.p, ds.hasUV ? ds.triUV.p : nullptr, ds.triOrig.p);
    if (cudaStreamSynchronize(st) != cudaSuccess) {
      err = std::string("BVH gather failed: ") + cudaGetErrorString(cudaGetLastError());
      return RG_ERR_CUDA;
    }
    trace.mark("gather", 0, n);
    return RG_OK;
  }
  // binary traversal layout
  int numNodes = 0, buildErr = 0;
  cudaMemcpyAsync(&numNodes, counters.p + C_NODES, sizeof(int), cudaMemcpyDeviceToHost, st);
  cudaMemcpyAsync(&buildErr, counters.p + C_BUILD_ERROR, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (cudaStreamSynchronize(st) != cudaSuccess) {
    err = "BVH build failed";
    return RG_ERR_CUDA;
  }
  if (buildErr != 0) {
    err = "BVH build scatter error " + std::to_string(buildErr);
    return RG_ERR_DEVICE_STATUS;
  }
  ds.bvhWidth = 2;
  DevBuf<int> &flags = X.flags, &trav = X.trav;
  if (!flags.alloc(numNodes) || !trav.alloc(numNodes)) {
    err = "out of device memory (BVH layout)";
    return RG_ERR_OUT_OF_MEMORY;
  }
  k_innerFlags<<<gridFor(numNodes, 256), 256, 0, st>>>(numNodes, nodes.p, flags.p);
  size_t tmpBytes = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, tmpBytes, flags.p, trav.p, numNodes, st);
  DevBuf<unsigned char>& tmp = X.tmp;
  if (!tmp.alloc(tmpBytes + 16)) {
    err = "out of device memory (BVH layout)";
    return RG_ERR_OUT_OF_MEMORY;
  }
  cub::DeviceScan::ExclusiveSum(tmp.p, tmpBytes, flags.p, trav.p, numNodes, st);
  int lastFlag = 0, lastTrav = 0;
  cudaMemcpyAsync(&lastFlag, flags.p + numNodes - 1, sizeof(int), cudaMemcpyDeviceToHost, st);
  cudaMemcpyAsync(&lastTrav, trav.p + numNodes - 1, sizeof(int), cudaMemcpyDeviceToHost, st);
  cudaStreamSynchronize(st);
  const int numInner = lastFlag + lastTrav;
  ds.numNodes = numInner;
  if (numInner == 0) {
    ds.rootIsLeaf = 1;
    ds.rootLeafRef = ~((0 << 3) | (n - 1));
    if (!ds.nodes.alloc(4)) {
      err = "out of device memory (BVH nodes)";
      return RG_ERR_OUT_OF_MEMORY;
    }
  } else {
    if (!ds.nodes.alloc((size_t)numInner * 4)) {
      err = "out of device memory (BVH nodes)";
      return RG_ERR_OUT_OF_MEMORY;
    }
    k_emitNodes<<<gridFor(numNodes, 256), 256, 0, st>>>(numNodes, nodes.p, trav.p, ds.nodes.p);
  }
  k_gather<<<gridFor(n, 256), 256, 0, st>>>(n, curIdx, vTmp.p, sTmp.p, ds.hasUV ? uvTmp.p : nullptr, ds.triVerts.p,
                                            ds.triShade.p, ds.hasUV ? ds.triUV.p : nullptr, ds.triOrig.p);
  if (cudaStreamSynchronize(st) != cudaSuccess) {
    err = std::string("BVH build failed: ") + cudaGetErrorString(cudaGetLastError());
    return RG_ERR_CUDA;
  }
  return RG_OK;
}

}  // namespace rg

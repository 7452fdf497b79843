// Stages (a) and (b) over a table of render jobs.
//
// A job is one (mesh, camera, resolution) view.  Every kernel here covers
// all jobs of a batch in one launch: items of all jobs share one index space
// (vertices, tets, external-face blocks, visible faces, screen tiles), and a
// binary search over a prefix of per-job counts maps an item to its job.
// Counts known on the host (vertices, tets, faces, tiles) are prefixed on the
// host; counts produced on the device (visible faces, rays) by
// prefix_kernel.  Nothing waits on the host between stages, so a batch is one
// stream-ordered chain of launches (and can be captured as a CUDA graph).
#pragma once
#include "vfr_types.cuh"

namespace vfr {

// Largest j with pref[j] <= g (pref[0] = 0, pref has n+1 entries, g < pref[n]).
__device__ __forceinline__ uint32_t job_of(const uint32_t* __restrict__ pref, uint32_t n, uint32_t g) {
  uint32_t lo = 0, hi = n;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(pref + mid) <= g) lo = mid; else hi = mid;
  }
  return lo;
}

// The same for one g per warp, 32 steps of the search at a time: called by the
// whole warp.
__device__ __forceinline__ uint32_t job_of_warp(const uint32_t* __restrict__ pref, uint32_t n, uint32_t g) {
  uint32_t lo = 0;
  while (n > 1) {  // the job is one of lo .. lo + n - 1, and pref[lo] <= g
    const uint32_t step = (n + 31u) / 32u, at = step * (threadIdx.x & 31u);
    const uint32_t below = __ballot_sync(0xffffffffu, at < n && __ldg(pref + lo + at) <= g);
    const uint32_t skip = step * (uint32_t)(__popc(below) - 1);
    lo += skip;
    n = min(step, n - skip);
  }
  return lo;
}

__device__ __forceinline__ float job_maxedge(const JobDev& J) {
  return J.use_mv ? __uint_as_float(J.ctr->maxedge_bits) : J.maxEdge_in;
}

__global__ void init_jobs_kernel(const JobDev* __restrict__ jobs, uint32_t njobs,
                                 uint32_t* __restrict__ queue) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j == 0) {
    queue[0] = 0;  // the traversal's ray queue
    queue[1] = 0;  // the composited mode's entry-arena cursor
    queue[2] = 0;  // blocks done of compact_kernel (see prefix_by_last_block)
    queue[3] = 0;  // and of raylist_kernel
  }
  if (j >= njobs) return;
  ViewCounters v;
  v.nvis = 0; v.nrays = 0; v.nentries = 0; v.status = 0; v.steps = 0;
  v.maxedge_bits = 0; v.rays_done = 0; v.nbins = 0;
  for (int k = 0; k < 4; ++k) { v.mm[k] = 0xffffffffu; v.mm[4 + k] = 0u; }
  *jobs[j].ctr = v;
}

// Before stages (b) and (c) run again on the visible faces of one stage (a):
// their counts start from 0 as after init_jobs_kernel (raylist_kernel appends
// to nrays, and the traversal's queue still holds the last run's rays).  What
// stage (a) found stays: the visible faces, and an id out of range.
__global__ void reproject_kernel(const JobDev* __restrict__ jobs, uint32_t njobs,
                                 uint32_t* __restrict__ queue) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < 4u) queue[j] = 0;
  if (j >= njobs) return;
  ViewCounters& v = *jobs[j].ctr;
  v.nrays = 0;
  v.nentries = 0;
  v.status &= kDevRange;
  v.steps = 0;
  v.rays_done = 0;
  v.nbins = 0;
}

// ------------------------------------------------------------ view set-up

// The view set-up kernels give each job a range of blocks (bpref: prefix of
// blocks per job), so a block reduces within one job and ends with one
// atomic per counter.

__device__ __forceinline__ float warp_min(float v) {
  for (int o = 16; o; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
  for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// rotateVolume (vfRayPreComp.cc:886-906) of one vertex.
__device__ __forceinline__ float4 rotated(const float4* rows, float4 v) {
  float r[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float acc = 0.0f;
    acc = fadd(acc, fmul(rows[a].x, v.x));
    acc = fadd(acc, fmul(rows[a].y, v.y));
    acc = fadd(acc, fmul(rows[a].z, v.z));
    acc = fadd(acc, fmul(rows[a].w, 1.0f));
    r[a] = acc;
  }
  return make_float4(r[0], r[1], r[2], v.w);
}

// The min/max of the rotated vertices that normalizeVertices needs, for every
// job with a model-view.  Nothing is written: view_normalize_kernel rotates
// again, and a batch's views (16 bytes per vertex and view, more than L2
// holds) cross DRAM once instead of three times (64 views of the carved 64^3
// mesh: 168 -> 126 us for the two kernels).
__global__ void __launch_bounds__(256) view_rotate_kernel(const JobDev* __restrict__ jobs,
                                                          uint32_t njobs,
                                                          const uint32_t* __restrict__ bpref) {
  const uint32_t j = job_of(bpref, njobs, blockIdx.x);
  const JobDev& J = jobs[j];
  const uint32_t lb = blockIdx.x - bpref[j], nb = bpref[j + 1] - bpref[j];
  const float4 rows[3] = {J.m0, J.m1, J.m2};
  float mn[4] = {INFINITY, INFINITY, INFINITY, INFINITY};
  float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
  for (uint32_t i = lb * blockDim.x + threadIdx.x; i < J.nV; i += nb * blockDim.x) {
    const float4 o = rotated(rows, J.vert_in[i]);
    const float c[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      mn[k] = fminf(mn[k], c[k]);
      mx[k] = fmaxf(mx[k], c[k]);
    }
  }
  // one pair of atomics per block and coordinate: warps reduce, then the
  // block through shared memory
  __shared__ float s_mm[8][8];
  const uint32_t w = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float a = warp_min(mn[k]), b = warp_max(mx[k]);
    if ((threadIdx.x & 31u) == 0) {
      s_mm[w][k] = a;
      s_mm[w][4 + k] = b;
    }
  }
  __syncthreads();
  if (threadIdx.x < 8) {
    const uint32_t k = threadIdx.x;
    float v = s_mm[0][k];
    for (uint32_t i = 1; i < (blockDim.x >> 5); ++i)
      v = k < 4 ? fminf(v, s_mm[i][k]) : fmaxf(v, s_mm[i][k]);
    if (k < 4) atomicMin(&J.ctr->mm[k], f2ord(v));
    else atomicMax(&J.ctr->mm[k], f2ord(v));
  }
}

// rotateVolume and normalizeVertices (vfRayPreComp.cc:84-145) with each view's
// min/max.
__global__ void __launch_bounds__(256) view_normalize_kernel(const JobDev* __restrict__ jobs,
                                                             uint32_t njobs,
                                                             const uint32_t* __restrict__ bpref) {
  const uint32_t j = job_of(bpref, njobs, blockIdx.x);
  const JobDev& J = jobs[j];
  const uint32_t lb = blockIdx.x - bpref[j], nb = bpref[j + 1] - bpref[j];
  const float4 rows[3] = {J.m0, J.m1, J.m2};
  float mn[4], mx[4], cen[3];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    mn[k] = ord2f(J.ctr->mm[k]);
    mx[k] = ord2f(J.ctr->mm[4 + k]);
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    cen[k] = (float)ddiv((double)fadd(mn[k], mx[k]), 2.0);
    mx[k] = fsub(mx[k], cen[k]);
    mn[k] = fsub(mn[k], cen[k]);
  }
  float maxCoord = (mx[1] > mx[2]) ? mx[1] : mx[2];
  maxCoord = (mx[0] > maxCoord) ? mx[0] : maxCoord;
  const float sc = (float)ddiv(1.0, (double)maxCoord);
  const float ss = (float)ddiv(1.0, (double)fsub(mx[3], mn[3]));
  for (uint32_t i = lb * blockDim.x + threadIdx.x; i < J.nV; i += nb * blockDim.x) {
    float4 p = rotated(rows, J.vert_in[i]);
    p.x = fmul(fsub(p.x, cen[0]), sc);
    p.y = fmul(fsub(p.y, cen[1]), sc);
    p.z = fmul(fsub(p.z, cen[2]), sc);
    p.w = fmul(fsub(p.w, mn[3]), ss);
    J.vview[i] = p;
  }
}

// A mesh edge's squared length; infinite where an id is out of range (checked
// build), so that no edges are listed as long and every view meets this one.
__host__ __device__ __forceinline__ float edge_sq(const float4* vert, uint32_t nV, uint2 e) {
  if (id_bad(e.x, nV) || id_bad(e.y, nV)) return INFINITY;
  const float4 a = vert[e.x], b = vert[e.y];
  const float x = a.x - b.x, y = a.y - b.y, z = a.z - b.z;
  return x * x + y * y + z * z;
}
struct LongEdge {
  const float4* vert;
  uint32_t nV;
  float least;  // squared length
  __host__ __device__ bool operator()(unsigned long long k) const {
    // the two ids as they lie in memory (little-endian: the high word second)
    return edge_sq(vert, nV, make_uint2((uint32_t)k, (uint32_t)(k >> 32))) >= least;
  }
};

// Keys of the 6 edges of every tet, (min id << 32) | max id, to be sorted and
// made unique into the mesh's distinct edges.
__global__ void __launch_bounds__(256) edge_keys_kernel(const uint4* __restrict__ tet, uint32_t nT,
                                                        unsigned long long* __restrict__ keys) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nT) return;
  const uint4 id = tet[t];
  const uint32_t v[4] = {id.x, id.y, id.z, id.w};
  const int E[6][2] = {{0, 1}, {0, 2}, {0, 3}, {1, 2}, {1, 3}, {2, 3}};
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const uint32_t a = v[E[k][0]], b = v[E[k][1]];
    keys[6 * (size_t)t + k] = (unsigned long long)min(a, b) << 32 | max(a, b);
  }
}

// The longest edge's squared length and the largest coordinate of the
// vertices, as float bits.
__global__ void __launch_bounds__(256) edge_extent_kernel(const uint2* __restrict__ edges, uint32_t n,
                                                          const float4* __restrict__ vert,
                                                          uint32_t nV, uint32_t* __restrict__ out) {
  const uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  float sq = 0.0f, co = 0.0f;
  for (uint32_t i = i0; i < n; i += step) sq = fmaxf(sq, edge_sq(vert, nV, edges[i]));
  for (uint32_t i = i0; i < nV; i += step) {
    const float4 v = vert[i];
    co = fmaxf(co, fmaxf(fabsf(v.x), fmaxf(fabsf(v.y), fabsf(v.z))));
  }
  sq = warp_max(sq);
  co = warp_max(co);
  if ((threadIdx.x & 31u) == 0) {
    atomicMax(out, __float_as_uint(sq));
    atomicMax(out + 1, __float_as_uint(co));
  }
}

// ------------------------------------------------------------ stage (a)

// buildLmt's maxEdgeLength (vfRayPreComp.cc:810-836) over each view's
// vertices.  The reference visits the 6 edges of every tet; an edge shared by
// several tets gives the same length in each (its difference vector at most
// changes sign), so the maximum over the mesh's distinct edges is the same
// float, at about a seventh of the work.
//
// Where the model-view is a similarity (a rotation, with any scale), the
// view's longest edge is one of the mesh's long ones: a view keeps all
// lengths in proportion up to its rounding, so only the edges within
// kLongEdge of the mesh's longest, which the edge list starts with, can be
// the view's longest.  long_edges_suffice bounds how far a length can be off
// its proportion.  64 views of the carved 64^3 mesh: 315 -> 11
// us.
constexpr float kLongEdge = 1.0f - 0x1p-9f;  // of the squared length
__device__ __forceinline__ bool long_edges_suffice(const JobDev& J) {
  if (!J.nLong) return false;
  const double u = 0x1p-24;
  const float4 m[3] = {J.m0, J.m1, J.m2};
  double g[6], s2 = 0, reach = 0, half = 0;
#pragma unroll
  for (int a = 0, q = 0; a < 3; ++a) {
#pragma unroll
    for (int b = a; b < 3; ++b, ++q)
      g[q] = (double)m[a].x * m[b].x + (double)m[a].y * m[b].y + (double)m[a].z * m[b].z;
    // rotated coordinates are within 5 u of this (three products, four sums)
    reach = fmax(reach, ((double)fabsf(m[a].x) + fabsf(m[a].y) + fabsf(m[a].z)) * J.vertMax + fabsf(m[a].w));
    half = fmax(half, 0.5 * ((double)ord2f(J.ctr->mm[4 + a]) - ord2f(J.ctr->mm[a])));
  }
  s2 = (g[0] + g[3] + g[5]) / 3.0;
  // M M^T = s2 (1 + E): squared lengths keep proportion within 1 +- 3 eta
  const double eta = fmax(fmax(fmax(fabs(g[0] - s2), fabs(g[3] - s2)), fabs(g[5] - s2)),
                          fmax(fmax(fabs(g[1]), fabs(g[2])), fabs(g[4]))) / s2;
  // normalised: scaled by 1 / half, coordinates at most 1; each end of an
  // edge is off by rounding in its 3 coordinates, its length by 8 u besides
  const double length = sqrt(s2) * J.edgeMax / half;
  const double eps = 16.0 * u + 3.5 * (10.0 * u * reach / half + 4.0 * u) / length;
  return 8.0 * eta + 2.5 * eps < 0x1p-11;  // false for a NaN too; half the margin of kLongEdge
}

__device__ __forceinline__ void view_maxedge(const JobDev* __restrict__ jobs, uint32_t njobs,
                                             const uint32_t* __restrict__ bpref, uint32_t block) {
  const uint32_t j = job_of(bpref, njobs, block);
  const JobDev& J = jobs[j];
  const uint32_t lb = block - bpref[j], nb = bpref[j + 1] - bpref[j];
  const uint32_t n = long_edges_suffice(J) ? J.nLong : J.nEdges;
  if (lb * blockDim.x >= n) return;
  // the rounded square root is monotone, so the largest rounded length is
  // the rounded root of the largest squared length: one root per thread
  float best_sq = 0.0f;
  for (uint32_t e = lb * blockDim.x + threadIdx.x; e < n; e += nb * blockDim.x) {
    const uint2 ed = __ldg(J.edges + e);
    if (id_bad(ed.x, J.nV) || id_bad(ed.y, J.nV)) {
      atomicOr(&J.ctr->status, kDevRange);
      continue;
    }
    const float4 a = J.vview[ed.x], b = J.vview[ed.y];
    const float e0 = fsub(a.x, b.x), e1 = fsub(a.y, b.y), e2 = fsub(a.z, b.z);
    const float sq = fadd(fadd(fmul(e0, e0), fmul(e1, e1)), fmul(e2, e2));
    if (sq > best_sq) best_sq = sq;
  }
  float best = __fsqrt_rn(best_sq);
  __shared__ float s_best[32];
  best = warp_max(best);
  if ((threadIdx.x & 31u) == 0) s_best[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (uint32_t i = 1; i < (blockDim.x >> 5); ++i) best = fmaxf(best, s_best[i]);
    atomicMax(&J.ctr->maxedge_bits, __float_as_uint(best));
  }
}

__global__ void __launch_bounds__(256) view_maxedge_kernel(const JobDev* __restrict__ jobs,
                                                           uint32_t njobs,
                                                           const uint32_t* __restrict__ bpref) {
  view_maxedge(jobs, njobs, bpref, blockIdx.x);
}

// findVisibleFaces (vfRayKernelCPU.cc:51-132), one thread per external face;
// each block of 1024 faces belongs to one job (bpref: blocks per job).  The
// blocks after the ext_blocks first take the views' longest edge (epref: edge
// blocks per job): both need only the view's vertices, and where the blocks
// of both fit the device at once, one launch saves 5 us of a small view's
// chain.  A larger grid runs view_maxedge_kernel, whose smaller blocks gather
// edges faster (32 views of the carved 64^3 mesh: 0.26 ms less).
__global__ void __launch_bounds__(1024) visible_kernel(const JobDev* __restrict__ jobs,
                                                       uint32_t njobs,
                                                       const uint32_t* __restrict__ bpref,
                                                       uint32_t ext_blocks,
                                                       const uint32_t* __restrict__ epref) {
  if (blockIdx.x >= ext_blocks) {
    view_maxedge(jobs, njobs, epref, blockIdx.x - ext_blocks);
    return;
  }
  const uint32_t j = job_of(bpref, njobs, blockIdx.x);
  const JobDev& J = jobs[j];
  const uint32_t lb = blockIdx.x - bpref[j];
  const uint32_t e = lb * blockDim.x + threadIdx.x;
  int vis = 0;
  if (e < J.nExt) {
    const uint2 tf = J.extf[e];
    bool bad = id_bad(tf.x, J.nT);
    uint4 id = J.tet[bad ? 0u : tf.x];
    bad = bad || id_bad(id.x, J.nV) || id_bad(id.y, J.nV) || id_bad(id.z, J.nV) ||
          id_bad(id.w, J.nV);
    if (bad) {
      id = make_uint4(0u, 0u, 0u, 0u);
      atomicOr(&J.ctr->status, kDevRange);
    }
    const float4 v0 = J.vert[sel4(id, tf.y & 3u)];
    const float4 v1 = J.vert[sel4(id, (tf.y + 1) & 3u)];
    const float4 v2 = J.vert[sel4(id, (tf.y + 2) & 3u)];
    const float4 op = J.vert[sel4(id, (tf.y + 3) & 3u)];
    Plane P;
    face_plane(v0, v1, v2, P);
    const float faceZ = plane_eval(op.x, op.y, P.zx, P.zy, P.zz);
    if (faceZ < op.z || bad) P.sx = -1.0f;  // :128 invisible sentinel
    vis = (P.sx != -1.0f);
    float4* pl = J.planes + kPlaneStride * (size_t)e;
    pl[0] = make_float4(P.zx, P.zy, P.zz, P.sx);
    pl[1] = make_float4(P.sy, P.sz, v0.x, v0.y);
    pl[2] = make_float4(v1.x, v1.y, v2.x, v2.y);
  }
  const int cnt = __syncthreads_count(vis);
  if (threadIdx.x == 0) J.blk[lb] = (uint32_t)cnt;
}

// Exclusive prefix of a per-job device count (0: visible faces, 1: rays) into
// out[0..njobs], by one block of 256 or 1024 threads.
__device__ __forceinline__ void prefix_block(const JobDev* __restrict__ jobs, uint32_t njobs,
                                             int which, uint32_t* __restrict__ out) {
  __shared__ uint32_t s[32];
  __shared__ uint32_t s_carry;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (uint32_t base = 0; base < njobs; base += blockDim.x) {
    const uint32_t j = base + threadIdx.x;
    uint32_t v = 0;
    if (j < njobs) {
      const ViewCounters* c = jobs[j].ctr;
      v = __ldcg(which == 0 ? &c->nvis : &c->nrays);  // other blocks' writes
    }
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) s[warp] = x;
    __syncthreads();
    if (warp == 0) {
      const uint32_t c = lane < (blockDim.x >> 5) ? s[lane] : 0u;
      uint32_t z = c;
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, z, o);
        if (lane >= (uint32_t)o) z += y;
      }
      s[lane] = z - c;
    }
    __syncthreads();
    const uint32_t carry = s_carry;
    if (j < njobs) out[j] = carry + s[warp] + x - v;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) s_carry = carry + s[warp] + x;
    __syncthreads();
  }
  if (threadIdx.x == 0) out[njobs] = s_carry;
}

// Called at the end of a kernel that produces a per-job count: the block that
// finishes last makes its prefix, which saves a one-block launch (3 us of a
// small view's chain each).  done counts the finished blocks (zeroed by
// init_jobs_kernel); every block's counts are fenced before its arrival.
// done is null where the grid is more than one wave of blocks: there the
// blocks' fences, each waiting for its block's stores, cost more than the
// launch (a 1024x768 view gains nothing, 32 views at 512^2 lose 0.04 ms).
__device__ __forceinline__ void prefix_by_last_block(const JobDev* __restrict__ jobs,
                                                     uint32_t njobs, int which,
                                                     uint32_t* __restrict__ out,
                                                     uint32_t* __restrict__ done) {
  __shared__ bool s_last;
  if (!done) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(done, 1u) == gridDim.x - 1u;
  }
  __syncthreads();
  if (s_last) {
    __threadfence();
    prefix_block(jobs, njobs, which, out);
    if (threadIdx.x == 0) *done = 0;
  }
}

__global__ void __launch_bounds__(1024) prefix_kernel(const JobDev* __restrict__ jobs, uint32_t njobs,
                                                      int which, uint32_t* __restrict__ out) {
  prefix_block(jobs, njobs, which, out);
}

// Ordered compaction (main.cc:93-138, vfRay.cu:355-388): a block's offset is
// the sum of the counts of the job's blocks before it; inside the block,
// warp ballots and a warp-count prefix place each face at its rank.
__global__ void __launch_bounds__(1024) compact_kernel(const JobDev* __restrict__ jobs,
                                                       uint32_t njobs,
                                                       const uint32_t* __restrict__ bpref,
                                                       uint32_t* __restrict__ vis_pref,
                                                       uint32_t* __restrict__ done) {
  __shared__ uint32_t s_warp[32];
  __shared__ uint32_t s_base;
  const uint32_t j = job_of(bpref, njobs, blockIdx.x);
  const JobDev& J = jobs[j];
  const uint32_t lb = blockIdx.x - bpref[j];
  const uint32_t nb = bpref[j + 1] - bpref[j];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t part = 0;
  const uint32_t nwarps = blockDim.x >> 5;  // blocks of 256 or 1024 threads
  for (uint32_t b = threadIdx.x; b < lb; b += blockDim.x) part += J.blk[b];
  for (int o = 16; o; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if (lane == 0) s_warp[warp] = part;
  __syncthreads();
  if (warp == 0) {
    uint32_t x = lane < nwarps ? s_warp[lane] : 0u;
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) s_base = x;
  }
  __syncthreads();
  const uint32_t e = lb * blockDim.x + threadIdx.x;
  const bool vis = e < J.nExt && J.planes[kPlaneStride * (size_t)e].w != -1.0f;
  const uint32_t m = __ballot_sync(0xffffffffu, vis);
  if (lane == 0) s_warp[warp] = __popc(m);
  __syncthreads();
  if (warp == 0) {
    const uint32_t c = lane < nwarps ? s_warp[lane] : 0u;
    uint32_t x = c;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= (uint32_t)o) x += y;
    }
    s_warp[lane] = x - c;
    if (lb == nb - 1 && lane == 31) J.ctr->nvis = s_base + x;
  }
  __syncthreads();
  if (vis) J.vis_ext[s_base + s_warp[warp] + __popc(m & ((1u << lane) - 1u))] = e;
  prefix_by_last_block(jobs, njobs, 0, vis_pref, done);
}

// ------------------------------------------------------------ stage (b)

// projectVisibleFaces (vfRayKernelCPU.cc:136-169): the pixel bounding box of
// a face from its vertex xy, which stage (a) stores with the plane (p1.zw,
// p2.xy, p2.zw); min starts at res - 1 and max at 0 as in the reference.
__device__ __forceinline__ uint4 face_box(const float4& p1, const float4& p2, uint32_t W,
                                          uint32_t H) {
  uint32_t bx = W - 1, by = H - 1, bz = 0, bw = 0;
  const float xs[3] = {p1.z, p2.x, p2.z}, ys[3] = {p1.w, p2.y, p2.w};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const uint32_t ix = to_pixel(xs[k], W), iy = to_pixel(ys[k], H);
    if (ix < bx) bx = ix;
    if (iy < by) by = iy;
    if (ix > bz) bz = ix;
    if (iy > bw) bw = iy;
  }
  return make_uint4(bx, by, bz, bw);
}

// A face as the rasteriser covers it: job, ext-face index, clipped box (x in
// a, y in d), entry edges, scalar plane, the pixel coordinates' reciprocals.
struct __align__(16) RasterFace {
  uint4 a;
  float4 b, c, d;
  double2 r;
};

// projectVisibleFaces (vfRayKernelCPU.cc:136-169) + the pixel coverage of
// vfRay's face loop (:248-274): persistent warps over the visible faces of
// all jobs, covering one face at a time with their lanes over the pixels of
// the face's bounding box in chunks of rh rows x (32 / rh) columns (rh = the box height
// rounded up to a power of two, at most 32).  The reference walks a column
// y-ascending and stops it at the first covered pixel whose entry scalar is
// out of [0,1] (:274); here the lanes of a column ballot that condition and a
// pixel is dropped if it or a pixel above it in its column has it (carried
// across row chunks of taller boxes).  The reference lets the last visible
// face in order write a pixel; visible order is ext-face order, so the
// winner is the largest ext-face index reaching it: atomicMax.  Pixels
// outside the image are clipped (the reference would write past its buffer
// there).  Reference mode; the composited mode's entry lists come from the
// screen-tile kernels below.
__global__ void __launch_bounds__(256, 4) raster_kernel(const JobDev* __restrict__ jobs, uint32_t njobs,
                                                     const uint32_t* __restrict__ vpref) {
  __shared__ RasterFace s_face[256];
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  const uint32_t total = vpref[njobs];
  // A warp takes up to 32 consecutive visible faces at a time.  Each lane
  // loads and sets up one of them (plane, box, entry edges: 32 independent
  // load chains in flight instead of one), then the warp covers the faces one
  // after another with the setup broadcast from the lane that made it
  // (1.25 -> 0.83 ms for 64 views at 512^2 against one warp per face, 0.60
  // with the broadcast below; 56 registers, 4 CTAs per SM).  Covering is serial in a warp, so where there
  // are fewer than 32 faces per launched warp -- a single view has a few
  // thousand to a few ten thousand -- each warp takes only its share.  The
  // broadcasts are shared-memory reads of one record (five wide loads; 22
  // shuffles a face took 700 us instead of 597 for those 64 views).
  const uint32_t per = min(32u, (total + nwarps - 1u) / nwarps);
  for (uint32_t g0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * per; g0 < total;
       g0 += nwarps * per) {
    const uint32_t g = lane < per ? g0 + lane : total;
    bool has = false;
    uint32_t j = 0, e = 0, bx = 0, by = 0, xe = 0, ye = 0;
    EntryEdges E = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    float sa = 0.0f, sb = 0.0f, sc = 0.0f;
    double rW = 0.0, rH = 0.0;
    if (g < total) {
      j = job_of(vpref, njobs, g);
      const JobDev& J = jobs[j];
      const uint32_t i = g - vpref[j];
      const uint32_t W = J.W, H = J.H;
      e = J.vis_ext[i];
      if (id_bad(e, J.nExt)) {
        atomicOr(&J.ctr->status, kDevRange);
      } else {
        // the face's plane and vertex xy, written by stage (a): one dependent
        // load after the visible list instead of the face -> tet -> vertex chain
        const float4* pl = J.planes + kPlaneStride * (size_t)e;
        const float4 p0 = pl[0], p1 = pl[1], p2 = pl[2];
        const uint4 box = face_box(p1, p2, W, H);
        J.bbox[i] = box;
        bx = box.x;
        by = box.y;
        xe = min(box.z, W - 1);
        ye = min(box.w, H - 1);
        has = bx <= xe && by <= ye;  // else the box lies entirely outside the image
        E = entry_edges(make_float4(p1.z, p1.w, 0.0f, 0.0f), make_float4(p2.x, p2.y, 0.0f, 0.0f),
                        make_float4(p2.z, p2.w, 0.0f, 0.0f));
        sa = p0.w;
        sb = p1.x;
        sc = p1.y;
        rW = __drcp_rn((double)(float)(W - 1u));
        rH = __drcp_rn((double)(float)(H - 1u));
      }
    }
    // the setup to shared memory, a record per face, read back by the whole
    // warp with broadcast loads
    if (has) {
      RasterFace& f = s_face[threadIdx.x];
      f.a = make_uint4(j, e, bx, xe);
      f.b = make_float4(E.v0x, E.v0y, E.e1x, E.e1y);
      f.c = make_float4(E.e2x, E.e2y, E.cx, sa);
      f.d = make_float4(sb, sc, __uint_as_float(by), __uint_as_float(ye));
      f.r = make_double2(rW, rH);
    }
    const uint32_t faces = __ballot_sync(0xffffffffu, has);
    __syncwarp();
    for (uint32_t todo = faces; todo; todo &= todo - 1u) {
      const RasterFace& f = s_face[(threadIdx.x & ~31u) + (uint32_t)__ffs(todo) - 1u];
      const uint4 fa = f.a;
      const float4 fb = f.b, fc = f.c, fd = f.d;
      const double2 fr = f.r;
      const uint32_t fj = fa.x, fe = fa.y, fbx = fa.z, fxe = fa.w;
      const uint32_t fby = __float_as_uint(fd.z), fye = __float_as_uint(fd.w);
      const EntryEdges F = {fb.x, fb.y, fb.z, fb.w, fc.x, fc.y, fc.z};
      const float fsa = fc.w, fsb = fd.x, fsc = fd.y;
      const double frW = fr.x, frH = fr.y;
      const uint32_t W = jobs[fj].W;
      int32_t* const winner = jobs[fj].winner;
      const uint32_t h = fye - fby + 1;
      const uint32_t rh = h >= 32 ? 32u : (h <= 1 ? 1u : 1u << (32 - __clz(h - 1)));
      const uint32_t cw = 32u / rh;
      const uint32_t r = lane % rh, c = lane / rh;
      const uint32_t seg = (rh == 32 ? 0xffffffffu : ((1u << rh) - 1u)) << (c * rh);  // my column
      const uint32_t upto = seg & (lane == 31 ? 0xffffffffu : ((2u << lane) - 1u));   // rows <= mine
      for (uint32_t x0 = fbx; x0 <= fxe; x0 += cw) {
        const uint32_t px = x0 + c;
        const float ox = obj_coord_r(px, frW);
        bool carried = false;  // a kill in an earlier row chunk of this column (rh == 32)
        for (uint32_t y0 = fby; y0 <= fye; y0 += rh) {
          const uint32_t py = y0 + r;
          const bool live = px <= fxe && py <= fye;
          bool inside = false, ok = false;
          if (live) {
            const float oy = obj_coord_r(py, frH);
            inside = entry_inside(F, ox, oy);
            const float sp = plane_eval(ox, oy, fsa, fsb, fsc);
            ok = (sp >= 0.0f) && (sp <= 1.0f);
          }
          const uint32_t kill = __ballot_sync(0xffffffffu, live && inside && !ok);
          if (live && inside && ok && !carried && !(kill & upto))
            atomicMax(&winner[py * W + px], (int32_t)fe);
          carried = carried || (kill & seg);
        }
      }
    }
    __syncwarp();  // the records are written again
  }
}

// ------------------------------------------------------------ stage (b), composited mode
//
// Every visible face covering a pixel (entry scalar in [0, 1]) is an entry
// of that pixel's ray.  The faces are binned into screen tiles of 16 x 16
// pixels (count, scan, fill: one atomic per face and tile), then one CTA per
// tile stages the tile's faces in shared memory, and each thread tests its
// pixel against them and writes its pixel's entry list in descending
// (depth, face) order -- the order the traversal takes the segments in.

constexpr uint32_t kTile = 16;

// Bin pass over the visible faces of all jobs: kFill = false counts the
// screen tiles each face's box overlaps (and stores the box), kFill = true
// writes the face's visible index into each tile's bin.  tpref: prefix of
// the jobs' tile counts.
template <bool kFill>
__global__ void __launch_bounds__(256) bin_kernel(const JobDev* __restrict__ jobs, uint32_t njobs,
                                                  const uint32_t* __restrict__ vpref,
                                                  const uint32_t* __restrict__ tpref,
                                                  uint32_t* __restrict__ tile_cnt,
                                                  const uint32_t* __restrict__ tile_off,
                                                  uint32_t* __restrict__ tile_cur,
                                                  uint32_t* __restrict__ bins, uint32_t bin_cap) {
  const uint32_t total = vpref[njobs];
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t g0 = blockIdx.x * blockDim.x; g0 < total; g0 += stride) {
    const uint32_t g = g0 + threadIdx.x;
    uint32_t j = 0, n = 0;
    if (g < total) {
      j = job_of(vpref, njobs, g);
      const JobDev& J = jobs[j];
      const uint32_t i = g - vpref[j];
      const uint32_t e = J.vis_ext[i];
      const bool bad = id_bad(e, J.nExt);
      if (bad) atomicOr(&J.ctr->status, kDevRange);
      const float4* pl = J.planes + kPlaneStride * (size_t)(bad ? 0u : e);
      uint4 b = face_box(pl[1], pl[2], J.W, J.H);
      if (bad) b = make_uint4(1u, 1u, 0u, 0u);  // an empty box: no tiles
      if (!kFill) J.bbox[i] = b;
      const uint32_t xe = min(b.z, J.W - 1), ye = min(b.w, J.H - 1);
      if (b.x <= xe && b.y <= ye) {
        const uint32_t tpx = (J.W + kTile - 1) / kTile, base = tpref[j];
        for (uint32_t ty = b.y / kTile; ty <= ye / kTile; ++ty)
          for (uint32_t tx = b.x / kTile; tx <= xe / kTile; ++tx) {
            const uint32_t t = base + ty * tpx + tx;
            if (!kFill) {
              atomicAdd(&tile_cnt[t], 1u);
            } else {
              const uint32_t slot = tile_off[t] + atomicAdd(&tile_cur[t], 1u);
              if (slot < bin_cap) bins[slot] = i;
            }
            ++n;
          }
      }
    }
    if (!kFill) {  // per job the (face, tile) pairs, one atomic per job and warp
      const uint32_t act = __activemask();
      const uint32_t peers = __match_any_sync(act, g < total ? j : 0xffffffffu);
      const uint32_t sum = __reduce_add_sync(peers, n);
      if (g < total && (threadIdx.x & 31u) == (uint32_t)(__ffs(peers) - 1) && sum)
        atomicAdd(&jobs[j].ctr->nbins, sum);
    }
  }
}

// A face as the tile kernel tests it: its box, entry edges, depth and
// scalar planes, ext-face index, and the tet and entry face a segment
// starting at it enters (tet << 2 | face).
struct TileFace {
  uint4 box;
  EntryEdges E;
  float zx, zy, zz, sx, sy, sz;
  uint32_t e, tf;
};

// One CTA per screen tile (a block-stride loop over the tiles of all jobs),
// one thread per pixel.  Pass 1 counts each pixel's entries; a block scan
// and one atomic on the batch's entry cursor give each pixel its list's
// place; pass 2 inserts each entry into its pixel's list in descending
// (depth, face) order.  The entry test is the rasteriser's own: the pixel in
// the face's box (clipped to the image), inside the entry face (inclusive,
// vfRayKernelCPU.cc:258-268), entry scalar in [0, 1].  Lists that do not
// fit the arena are left empty and counted, and the caller renders again
// with room (as with bins past their capacity).
__global__ void __launch_bounds__(256) tile_kernel(const JobDev* __restrict__ jobs, uint32_t njobs,
                                                   const uint32_t* __restrict__ tpref,
                                                   const uint32_t* __restrict__ tile_off,
                                                   const uint32_t* __restrict__ bins,
                                                   uint32_t bin_cap, uint4* __restrict__ ent,
                                                   uint32_t ent_cap, uint32_t* __restrict__ cursor) {
  __shared__ TileFace F[256];
  __shared__ uint32_t s_warp[8];
  __shared__ uint32_t s_base;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t ntiles = tpref[njobs];
  for (uint32_t g = blockIdx.x; g < ntiles; g += gridDim.x) {
    const uint32_t j = job_of(tpref, njobs, g);
    const JobDev& J = jobs[j];
    const uint32_t lt = g - tpref[j], W = J.W, H = J.H;
    const uint32_t tpx = (W + kTile - 1) / kTile;
    // a warp's pixels are an 8 x 4 block of the tile
    const uint32_t wx = (lt % tpx) * kTile + (warp & 1u) * 8u, wy = (lt / tpx) * kTile + (warp >> 1) * 4u;
    const uint32_t px = wx + (lane & 7u), py = wy + (lane >> 3);
    const bool live = px < W && py < H;
    const double rW = __drcp_rn((double)(float)(W - 1u)), rH = __drcp_rn((double)(float)(H - 1u));
    const float ox = obj_coord_r(px, rW), oy = obj_coord_r(py, rH);
    const uint32_t b0 = min(tile_off[g], bin_cap), b1 = min(tile_off[g + 1], bin_cap);
    auto covers = [&](const TileFace& f) {
      return px >= f.box.x && px <= f.box.z && py >= f.box.y && py <= f.box.w &&
             entry_inside(f.E, ox, oy) && [&] {
               const float sp = plane_eval(ox, oy, f.sx, f.sy, f.sz);
               return (sp >= 0.0f) && (sp <= 1.0f);
             }();
    };
    // which of the staged faces 32 w .. 32 w + 31 have a box that meets the
    // warp's pixels, one face per lane: the others need no test at any pixel
    // (an 801x600 view of the carved 48^3 mesh: 45 -> 38 us against testing
    // every face at every pixel; with 16 x 2 pixels per warp fewer faces drop
    // out.  Selecting each next entry over the mask in shared memory, with no
    // insertion in the arena, was slower: 41 us)
    auto meets = [&](uint32_t w, uint32_t m) {
      const uint32_t k = 32u * w + lane;
      bool ov = false;
      if (k < m) {
        const uint4 b = F[k].box;
        ov = b.x <= wx + 7u && b.z >= wx && b.y <= wy + 3u && b.w >= wy;
      }
      return __ballot_sync(0xffffffffu, ov);
    };
    auto stage = [&](uint32_t c) {  // faces c .. c+255 of the bin into shared memory
      __syncthreads();
      if (c + tid < b1) {
        uint32_t i = bins[c + tid];
        bool bad = id_bad(i, J.ctr->nvis);
        uint32_t e = J.vis_ext[bad ? 0u : i];
        bad = bad || id_bad(e, J.nExt);
        if (bad) {
          i = e = 0;
          atomicOr(&J.ctr->status, kDevRange);
        }
        const float4* pl = J.planes + kPlaneStride * (size_t)e;
        const float4 p0 = pl[0], p1 = pl[1], p2 = pl[2];
        TileFace f;
        f.box = bad ? make_uint4(1u, 1u, 0u, 0u) : J.bbox[i];  // bad: covers nothing
        f.box.z = min(f.box.z, W - 1);
        f.box.w = min(f.box.w, H - 1);
        f.E = entry_edges(make_float4(p1.z, p1.w, 0.0f, 0.0f), make_float4(p2.x, p2.y, 0.0f, 0.0f),
                          make_float4(p2.z, p2.w, 0.0f, 0.0f));
        f.zx = p0.x;
        f.zy = p0.y;
        f.zz = p0.z;
        f.sx = p0.w;
        f.sy = p1.x;
        f.sz = p1.y;
        f.e = e;
        const uint2 tf = J.extf[e];
        f.tf = (tf.x << 2) | (tf.y & 3u);
        F[tid] = f;
      }
      __syncthreads();
      return min(256u, b1 - c);
    };
    // pass 1: entries per pixel.  A tile whose bin fits one staged chunk
    // (the common case) also keeps which of the chunk's faces cover each
    // pixel, as a 256-bit mask in registers, so that pass 2 neither stages
    // nor tests the faces again.
    const bool one_chunk = b1 - b0 <= 256u;
    uint32_t cov[8];
    uint32_t count = 0;
    for (uint32_t c = b0; c < b1; c += 256) {
      const uint32_t m = stage(c);  // every thread: stage() synchronises the block
#pragma unroll
      for (uint32_t w = 0; w < 8; ++w) {  // w is a constant after unrolling: cov stays in registers
        uint32_t bits = 0;
        if (32u * w < m)
          for (uint32_t todo = meets(w, m); todo; todo &= todo - 1u) {
            const uint32_t k = (uint32_t)__ffs(todo) - 1u;
            if (live && covers(F[32u * w + k])) bits |= 1u << k;
          }
        cov[w] = bits;
        count += __popc(bits);
      }
    }
    if (b1 == b0) {
#pragma unroll
      for (uint32_t w = 0; w < 8; ++w) cov[w] = 0;
    }
    // block scan of the counts
    uint32_t x = count;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
      const uint32_t c = lane < 8 ? s_warp[lane] : 0u;
      uint32_t z = c;
      for (int o = 1; o < 8; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, z, o);
        if (lane >= (uint32_t)o) z += y;
      }
      if (lane < 8) s_warp[lane] = z - c;
      if (lane == 7) {
        s_base = atomicAdd(cursor, z);
        atomicAdd(&J.ctr->nentries, z);
      }
    }
    __syncthreads();
    const uint32_t off = s_base + s_warp[warp] + x - count;
    const bool fits = off + count <= ent_cap;
    // VFR_DEV_OVERFLOW: a list or this tile's bin did not fit
    if ((live && count && !fits) || (tid == 0 && tile_off[g + 1] > bin_cap))
      atomicOr(&J.ctr->status, 16u);
    if (live) {
      const uint32_t p = py * W + px;
      J.ent_off[p] = fits ? off : 0u;
      J.ent_cnt[p] = fits ? count : 0u;
    }
    // pass 2: each pixel's entries, inserted in descending (depth, face) order
    uint32_t n = 0;
    // each entry also carries what its segment starts from (the face's tet
    // and entry face, the back colour's TF entry), so the traversal starts a
    // segment without going back through the plane and the external face
    auto insert = [&](const TileFace& f) {
      const float z = plane_eval(ox, oy, f.zx, f.zy, f.zz);
      const uint32_t cbi = (uint32_t)fmul(255.0f, plane_eval(ox, oy, f.sx, f.sy, f.sz));
      uint32_t q = n++;
      while (q > 0) {
        const uint4 a = ent[off + q - 1];
        const float za = __uint_as_float(a.x);
        if (za > z || (za == z && a.y > f.e)) break;
        ent[off + q] = a;
        --q;
      }
      ent[off + q] = make_uint4(__float_as_uint(z), f.e, f.tf, cbi);
    };
    if (one_chunk) {  // F still holds the chunk pass 1 staged
      if (live && fits && count) {
#pragma unroll
        for (uint32_t w = 0; w < 8; ++w)
          for (uint32_t bits = cov[w]; bits; bits &= bits - 1u)
            insert(F[32u * w + (uint32_t)(__ffs(bits) - 1)]);
      }
    } else {
      for (uint32_t c = b0; c < b1; c += 256) {
        const uint32_t m = stage(c);
        for (uint32_t w = 0; 32u * w < m; ++w)
          for (uint32_t todo = meets(w, m); todo; todo &= todo - 1u) {
            const TileFace& f = F[32u * w + (uint32_t)__ffs(todo) - 1u];
            if (live && fits && count && covers(f)) insert(f);
          }
      }
    }
  }
}

// Ray lists: the pixels with an entry face, as start records (RayStart),
// in screen tiles of 32 pixels
// (tw x 32/tw, one warp per tile, tiles of all jobs in one index space) so
// that neighbouring rays, which walk neighbouring tets, are neighbours in the
// list and share warps.  A job's rows of tiles are taken from the middle of
// the image outwards: rays near the silhouette are the shortest, and with
// them last the traversal's tail, when its queue is empty and lanes run dry,
// is shorter.  The block's warps of one job take their places in the list
// with one atomic (a warp each made the counter the bottleneck: 69 us for
// 2048^2).  Pixels without a ray are cleared in the outputs here (the
// reference zero-fills its image, main.cc:194).
__global__ void __launch_bounds__(256) raylist_kernel(const JobDev* __restrict__ jobs, uint32_t njobs,
                                                      const uint32_t* __restrict__ tpref, int mode,
                                                      uint32_t tw, uint32_t* __restrict__ ray_pref,
                                                      uint32_t* __restrict__ done) {
  __shared__ uint32_t s_job[8], s_count[8], s_base[8];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const bool any = g < tpref[njobs];  // else a warp past the last tile: no pixels
  const uint32_t j = any ? job_of_warp(tpref, njobs, g) : njobs - 1u;
  const JobDev& J = jobs[j];
  const uint32_t tile = any ? g - tpref[j] : 0u;
  const uint32_t th = 32u / tw;
  const uint32_t tx = (J.W + tw - 1) / tw, ty = (J.H + th - 1) / th;
  // row k of the order is the middle row, the one above it, the one below, ...
  const uint32_t k = tile / tx, row = (k & 1u) ? ty / 2u - (k + 1u) / 2u : ty / 2u + k / 2u;
  const uint32_t x = (tile % tx) * tw + (lane % tw), y = row * th + (lane / tw);
  bool has = false;
  uint32_t p = 0;
  RayStart rs = {0u, 0u, 0u, 0u};
  const bool inside = any && x < J.W && y < J.H;
  if (inside) {
    p = y * J.W + x;
    rs.p = p;
    if (mode == 0) {
      // the winning face's segment start, computed as the traversal would
      // (vfRayKernelCPU.cc:250-279): object coordinates of the pixel, the
      // plane's depth and scalar there, the face's tet and entry face
      const int32_t w = J.winner[p];
      has = w >= 0;
      if (has && id_bad((uint32_t)w, J.nExt)) {
        atomicOr(&J.ctr->status, kDevRange);
        has = false;
      }
      if (has) {
        const float4* pl = J.planes + kPlaneStride * (size_t)w;
        const float4 p0 = pl[0], p1 = pl[1];
        const float ox = obj_coord_r(x, __drcp_rn((double)(float)(J.W - 1u))),
                    oy = obj_coord_r(y, __drcp_rn((double)(float)(J.H - 1u)));
        const uint2 tf = J.extf[w];
        rs.tf = (tf.x << 2) | (tf.y & 3u);
        rs.zp = __float_as_uint(plane_eval(ox, oy, p0.x, p0.y, p0.z));
        rs.cbi = (uint32_t)fmul(255.0f, plane_eval(ox, oy, p0.w, p1.x, p1.y));
        if (id_bad(tf.x, J.nT)) {
          atomicOr(&J.ctr->status, kDevRange);
          has = false;
        }
      }
    } else {
      has = J.ent_cnt[p] > 0;
    }
  }
  const uint32_t m = __ballot_sync(0xffffffffu, has);
  if (lane == 0) {
    s_job[warp] = j;
    s_count[warp] = (uint32_t)__popc(m);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (uint32_t w = 0; w < 8u;) {
      uint32_t e = w, n = 0;  // warps w .. e-1: one job
      for (; e < 8u && s_job[e] == s_job[w]; ++e) n += s_count[e];
      uint32_t base = n ? atomicAdd(&jobs[s_job[w]].ctr->nrays, n) : 0u;
      for (; w < e; ++w) {
        s_base[w] = base;
        base += s_count[w];
      }
    }
  }
  __syncthreads();
  if (has) J.rays[s_base[warp] + __popc(m & ((1u << lane) - 1u))] = rs;
  if (inside && !has) {
    if (J.rgb8) {
      uint8_t* o = J.rgb8 + 3 * (size_t)p;
      o[0] = 0; o[1] = 0; o[2] = 0;
    }
    if (J.rgba) J.rgba[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (J.steps) J.steps[p] = 0;
  }
  prefix_by_last_block(jobs, njobs, 1, ray_pref, done);
}

// Exclusive scan of the batch's entry-count arena (composited mode): block
// scans, then each block adds the sums of the blocks before it.
__global__ void __launch_bounds__(1024) scan_blocks_kernel(const uint32_t* __restrict__ in,
                                                           uint32_t n, uint32_t* __restrict__ out,
                                                           uint32_t* __restrict__ sums) {
  __shared__ uint32_t s[32];
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t v = i < n ? in[i] : 0u;
  uint32_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  if (lane == 31) s[warp] = x;
  __syncthreads();
  if (warp == 0) {
    const uint32_t c = lane < (blockDim.x >> 5) ? s[lane] : 0u;
    uint32_t z = c;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, z, o);
      if (lane >= (uint32_t)o) z += y;
    }
    s[lane] = z - c;
    if (lane == 31) sums[blockIdx.x] = z;
  }
  __syncthreads();
  if (i < n) out[i] = x - v + s[warp];
}

__global__ void __launch_bounds__(1024) scan_add_kernel(uint32_t* __restrict__ out, uint32_t n,
                                                        const uint32_t* __restrict__ sums,
                                                        uint32_t* __restrict__ total) {
  __shared__ uint32_t s[32];
  __shared__ uint32_t s_base;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t part = 0;
  for (uint32_t b = threadIdx.x; b < blockIdx.x; b += blockDim.x) part += sums[b];
  for (int o = 16; o; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if (lane == 0) s[warp] = part;
  __syncthreads();
  if (warp == 0) {
    uint32_t x = lane < (blockDim.x >> 5) ? s[lane] : 0u;
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) s_base = x;
  }
  __syncthreads();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] += s_base;
  if (total && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *total = s_base + sums[blockIdx.x];
}

}  // namespace vfr

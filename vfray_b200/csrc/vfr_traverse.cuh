// Stage (c): tet-to-tet traversal with partial pre-integration
// (vfRayKernelCPU.cc:173-566), one lane per ray, persistent warps.
//
// Per-lane state machine: a lane walks up to two tets per loop pass; when its
// ray ends it writes the pixel, and once enough lanes of the warp are idle
// the warp refills them from the batch's single ray queue (one
// warp-aggregated atomicAdd), so lanes do not wait for the longest ray of
// their warp.  The kernel is bound by instruction issue, so the step is
// written to keep lanes converged: its arithmetic is branch-free, its rare
// exact fallbacks (psi coordinate, exp, plane re-solve) are taken in one
// block after the fast path, and every way a step can end is a status
// rather than an early return.  The current tet's 4 vertices live in shared
// memory, one slot each per thread, and a per-ray map of 4 bytes names the
// slot of each vertex in the entry face's rotation (r_j = local vertex
// (f + j) & 3): the three exit candidates (f+1, f+2, f+3) are candidate i =
// (r_i, r_i+1, r_i+2).  Moving to the next tet stores its one new vertex in
// the slot of the vertex left behind and permutes the map's bytes.  Once the
// exit face is known, a step issues its two loads together: the next tet's
// 32-byte walk record and the one vertex the next tet does not share with
// this one (its id is in this tet's record), so one memory round trip per
// step.
#pragma once
#include "vfr_jobs.cuh"

namespace vfr {

// One exit candidate (vfRayKernelCPU.cc:312-348), branch-free.  The slack
// test (double)(c1+c2) <= (double)cr + 1e-12 (:341-342) is decided in float:
// for a float sum s and cr >= 0x2b8cbccd (faces below RDELTA are skipped) it
// holds exactly when s - cr rounded to float is at most 0x2b8cbccc, the
// largest float below 1e-12.  For s <= cr both hold; for cr < s <= 2cr the
// difference is exact (Sterbenz) and a multiple of ulp(cr) >= 2^-63, and no
// such multiple lies within the double rounding error of cr + 1e-12 (below
// 2^(k-28) for multiples of 2^k) of 1e-12, whose distance to the multiples of
// 2^-63 is 2^-67.8; for s > 2cr the difference exceeds cr > 1e-12.
//
// The reference swaps v1 and v2 and negates cr when cr < 0 (:323-330).  Its
// products then become c1' = v2x v0y - v2y v0x = -c2 and c2' = -c1 exactly
// (rounded products and differences are symmetric), and its sum and slack
// difference are the negations of the unswapped ones.  So the swap is a sign
// flip of (c1, c2, sum - cr): applied by xor-ing the sign of cr into them.
__device__ __forceinline__ bool exit_test(const float4& a, const float4& b, const float4& c,
                                          float ox, float oy) {
  const float v1x = fsub(b.x, a.x), v1y = fsub(b.y, a.y);
  const float v2x = fsub(c.x, a.x), v2y = fsub(c.y, a.y);
  const float cr = fsub(fmul(v1x, v2y), fmul(v1y, v2x));
  const bool skip = below_rdelta(cr);
  const float v0x = fsub(ox, a.x), v0y = fsub(oy, a.y);
  const float c1 = fsub(fmul(v1x, v0y), fmul(v1y, v0x));
  const float c2 = fsub(fmul(v0x, v2y), fmul(v0y, v2x));
  const float d = fsub(fadd(c1, c2), cr);
  const uint32_t sg = __float_as_uint(cr) & 0x80000000u;
  const float c1s = __uint_as_float(__float_as_uint(c1) ^ sg);
  const float c2s = __uint_as_float(__float_as_uint(c2) ^ sg);
  const float ds = __uint_as_float(__float_as_uint(d) ^ sg);
  return !skip && (c1s >= 0.0f) && (c2s >= 0.0f) && (ds <= __uint_as_float(0x2b8cbcccu));
}

// Per-CTA copies of the small tables: the transfer function (RGBA, one
// 16-byte read per step: the front's; the back's is the previous front's and
// stays in registers), and 2^(-k/64), k = 0..511, for zeta_fast.  Divergent
// shared reads are what the step must be sparing with: the L1 data pipe,
// which serves them and the mesh loads, is its tightest resource (139
// wavefronts per warp and step, 87 % of the pipe, with the colours as
// doubles and alpha as three tables read for the front and for the back).
struct SharedTables {
  float4 tf[256];
  double e2[kExpEntries];
};

// A ray's walk is a function of its state (tet, entry face) alone: the pixel
// is fixed, so a state that comes back means the reference's while loop
// never ends (a cycle among tets around a projected edge, which the
// inclusive exit tests with slack allow on meshes whose tets list their
// vertices in arbitrary order).  Rays longer than kWatchSteps iterations are
// watched: the state is saved at every power-of-two iteration count and
// compared with the state of every later iteration (Brent), which stops a
// cycling ray within about two periods.  Shorter rays pay one comparison
// per pass of two steps.  The oracle applies the same rule, so steps stay
// comparable.
constexpr uint32_t kWatchSteps = 4095;

// The watched state of each thread's ray (tet << 2 | entry face, ~0 =
// none), in shared memory: it is written when a segment starts and read
// only by watched iterations, so it takes no register of the step.
__shared__ uint32_t s_watch_saved[256];

// The current tet's 4 vertices, per thread, in 4 slots.  A ray's map has one
// byte per vertex, in the order r_3, r_0, r_1, r_2 of the entry face's
// rotation (r_j = vertex (f + j) & 3): the vertex opposite the entry face
// first.  Rotating the map right by i bytes puts the exit face i's vertices
// (r_i, r_i+1, r_i+2) in bytes 1-3 and the vertex the step leaves behind,
// r_i+3, in byte 0; the permutation code of the walk record then reorders
// bytes 1-3 for the next tet (perm_selector), whose new vertex takes byte
// 0's slot.  A byte is the second byte of the vertex's 16-bit shared-memory
// address, slot * 4096 + thread * 16 from the 256-byte aligned start of
// s_vtx, so one byte permutation with the thread's low address byte gives an
// address that the load takes as it is.  (With 2-bit fields, a shift and a
// mask per vertex and a 64-bit table of permutations, the map cost about 20
// integer instructions more per step; with offsets into the array, which the
// compiler adds to its base, 10 more: 8.21 -> 8.12 ms for 32 views.)
__shared__ __align__(256) float4 s_vtx[4][256];
__device__ __forceinline__ uint32_t identity_map() {
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(s_vtx) >> 8;
  return 0x20100030u + ((threadIdx.x >> 4) + base) * 0x01010101u;
}
// The thread's low offset byte, held in a register rather than read from
// the thread index at each use.
__device__ __forceinline__ uint32_t thread_low() {
  uint32_t low = (threadIdx.x & 15u) << 4;
  asm volatile("" : "+r"(low));
  return low;
}
__device__ __forceinline__ uint32_t vtx_at(uint32_t map, uint32_t low, uint32_t byte) {
  return __byte_perm(map, low, 0x5504u | byte << 4);
}
__device__ __forceinline__ float4 vtx(uint32_t at) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at));
  return v;
}
__device__ __forceinline__ f32x2 vtx_xy(uint32_t at) {
  f32x2 v;
  asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(at));
  return v;
}
__device__ __forceinline__ void set_vtx(uint32_t at, float4 v) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at), "f"(v.x), "f"(v.y), "f"(v.z),
               "f"(v.w));
}

// The exit face of the step from rotated vertices (bytes of the map): the
// i in 1..3 of the first candidate (r_i, r_i+1, r_i+2) the exit test accepts
// (:310-350), 0 if none does.
static __device__ __noinline__ uint32_t exit_face_exact(uint32_t map, uint32_t low, float ox, float oy) {
  const float4 r3 = vtx(vtx_at(map, low, 0)), r0 = vtx(vtx_at(map, low, 1)),
               r1 = vtx(vtx_at(map, low, 2)), r2 = vtx(vtx_at(map, low, 3));
  return exit_test(r1, r2, r3, ox, oy)   ? 1u
         : exit_test(r2, r3, r0, ox, oy) ? 2u
         : exit_test(r3, r0, r1, ox, oy) ? 3u
                                         : 0u;
}

// The same from the signs of the six cross products of the vertices' offsets
// from the ray, A_j = r_j - o: x_ab = A_a x A_b.  In real arithmetic a
// candidate (a, b, c) has c1 = x_ab, c2 = x_ca, cr - c1 - c2 = x_bc, so the
// ray lies inside it when the three have one sign.  With M the largest
// component of the A_j and u = 2^-24, a computed cross product is within
// 6.1 u M^2 of the real one, and the exit test's own c1, c2, cr and slack
// difference (differences of vertices, at most 2M, each rounded) are within
// 16, 16, 32 and 80 u M^2 of theirs.  So when all six products exceed
// 2^-17 M^2 + 2e-12 = 128 u M^2 + 2e-12 in magnitude, each of them and each
// of the test's quantities has its real sign, the slack difference is on its
// side of 1e-12, an accepted candidate's cr is above RDELTA, and a candidate
// is accepted exactly when its three products have one sign: of two products
// of different sign, one fails the test whatever cr's sign is.  When the
// entry face (r_0, r_1, r_2) holds the ray too, exactly one candidate does:
// the ray is strictly inside it, and -A_3 lies in one of the three sectors
// the A_j cut the plane into.  sure says that all this holds (NaN and
// infinite coordinates fail it); about one step in 2^13 is not sure and
// takes the exact tests (every step of a lattice seen along its axes, where
// two vertices of each tet lie in front of one another).
//
// 40 instructions instead of 66 for three exact tests, with the six
// products shared between the candidates.
__device__ __forceinline__ uint32_t exit_face(uint32_t map, uint32_t low, float ox, float oy,
                                              bool& sure) {
  const f32x2 o = pack2(ox, oy);
  float a0x, a0y, a1x, a1y, a2x, a2y, a3x, a3y;
  unpack2(sub2(vtx_xy(vtx_at(map, low, 1)), o), a0x, a0y);
  unpack2(sub2(vtx_xy(vtx_at(map, low, 2)), o), a1x, a1y);
  unpack2(sub2(vtx_xy(vtx_at(map, low, 3)), o), a2x, a2y);
  unpack2(sub2(vtx_xy(vtx_at(map, low, 0)), o), a3x, a3y);
  auto cross = [](float ax, float ay, float bx, float by) {
    return __fmaf_rn(ax, by, -fmul(ay, bx));
  };
  const float x01 = cross(a0x, a0y, a1x, a1y), x02 = cross(a0x, a0y, a2x, a2y);
  const float x12 = cross(a1x, a1y, a2x, a2y), x03 = cross(a0x, a0y, a3x, a3y);
  const float x13 = cross(a1x, a1y, a3x, a3y), x23 = cross(a2x, a2y, a3x, a3y);
  const float M = max3_abs(max3_abs(a0x, a0y, a1x), max3_abs(a1y, a2x, a2y), max3_abs(a3x, a3y, 0.0f));
  const float least = min3_abs(min3_abs(x01, x02, x12), min3_abs(x03, x13, x23), x23);
  // sign bits: 01, 12, 20 alike (x20 = -x02); 12, 23, 31 alike; 23, 30, 02 alike
  const uint32_t b01 = __float_as_uint(x01), b02 = __float_as_uint(x02), b12 = __float_as_uint(x12);
  const uint32_t b03 = __float_as_uint(x03), b13 = __float_as_uint(x13), b23 = __float_as_uint(x23);
  const int entry = (int)(~(b01 ^ b12) & (b12 ^ b02));
  const int in1 = (int)(~(b12 ^ b23) & (b23 ^ b13));
  const int in2 = (int)(~(b23 ^ b02) & (b23 ^ b03));
  sure = least > __fmaf_rn(fmul(M, M), 0x1p-17f, 2e-12f) && entry < 0;
  return in1 < 0 ? 1u : (in2 < 0 ? 2u : 3u);
}

// Composited mode: the pixel's entry list (first, count), the next entry to
// take and the depth where the last segment left the mesh, in shared memory:
// only a segment's end reads them, and the step needs the registers (spills
// 46 -> 22 bytes at 3 CTAs per SM then; now 16).
__shared__ uint32_t s_ea[256], s_en[256], s_de[256];
__shared__ float s_exit_z[256];

struct Ray {
  uint32_t map;                // slots of the rotated vertices in s_vtx, a byte each
  uint32_t low;                // the thread's low offset byte in a slot
  WalkRec w;                   // walk record of the current tet
  const WalkRec* walk;         // this job's mesh and view vertices
  const float4* vert;
  uint32_t j, nT;
  uint32_t nV;                 // checked build: vertex ids are compared with it
  uint32_t watch;              // min(kWatchSteps, step cap): longer rays are checked
  float maxEdge, rmaxEdge;     // maxEdgeLength and its correctly rounded reciprocal
  float4 cb;                   // colorBack (RGBA)
  uint32_t t, f, p, iters;
  float ox, oy, zp;
  float ar, ag, ab, tr, lastZ;
  // served form: the job (its table entry lives in the server's arena) and
  // its completion flag
  const JobDev* jp;
  uint32_t* done;
};

// Read-only loads of the mesh through the non-coherent path (the arrays are
// not written while the traversal runs).  The record is one 32-byte load:
// lanes in different tets cost the L1 data pipe 17 wavefronts fewer per warp
// than two 16-byte loads of the same sector (122 -> 104 per step).
__device__ __forceinline__ WalkRec ldg_walk(const WalkRec* w, uint32_t t) {
  WalkRec r;
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r.n.x), "=r"(r.n.y), "=r"(r.n.z), "=r"(r.n.w), "=r"(r.q.x), "=r"(r.q.y), "=r"(r.q.z),
        "=r"(r.q.w)
      : "l"(w + t));
  return r;
}

// The four vertices of a tet in the slots, rotated by its entry face f.
__device__ __forceinline__ void set_vertices(Ray& R, uint4 id, uint32_t f) {
  const uint32_t ident = identity_map();
  set_vtx(vtx_at(ident, R.low, 1), __ldg(R.vert + sel4(id, f)));
  set_vtx(vtx_at(ident, R.low, 2), __ldg(R.vert + sel4(id, (f + 1) & 3u)));
  set_vtx(vtx_at(ident, R.low, 3), __ldg(R.vert + sel4(id, (f + 2) & 3u)));
  set_vtx(vtx_at(ident, R.low, 0), __ldg(R.vert + sel4(id, (f + 3) & 3u)));
  R.map = ident;
}

// Start a segment in tet t through its face f, with entry depth zp and the
// back colour's transfer-function entry cbi (:256-279).  False (checked build
// only): the tet or one of its vertex ids is out of range, and nothing was
// loaded.
__device__ __forceinline__ bool begin_segment_at(const SharedTables& S, const JobDev& J, Ray& R,
                                                 uint32_t t, uint32_t f, float zp, uint32_t cbi) {
  if (id_bad(t, J.nT)) return false;
  R.t = t;
  R.f = f;
  const uint4 id = __ldg(J.tet + t);
  if (id_bad(id.x, J.nV) || id_bad(id.y, J.nV) || id_bad(id.z, J.nV) || id_bad(id.w, J.nV))
    return false;
  R.w = ldg_walk(R.walk, t);
  set_vertices(R, id, f);
  R.zp = zp;
  R.lastZ = zp;
  R.cb = S.tf[cbi];
  s_watch_saved[threadIdx.x] = 0xffffffffu;  // a new segment walks other states
  return true;
}


// Composited mode: the pixel's next entry in its list, which stage (b)
// wrote in descending (depth, face) order, skipping entries above the depth
// where the previous segment left the mesh.  Returns false when the list is
// done (or, checked build only, holds an id out of range: VFR_DEV_RANGE).
__device__ __forceinline__ bool next_entry(const SharedTables& S, const JobDev& J, Ray& R,
                                           uint32_t& status) {
  bool bad = false;
  const uint32_t ea = s_ea[threadIdx.x], en = s_en[threadIdx.x];
  const float exit_z = s_exit_z[threadIdx.x];
  uint32_t de = s_de[threadIdx.x];
  bool started = false;
  while (de < en) {
    if (id_bad(ea + de, J.ent_cap)) {
      bad = true;
      break;
    }
    const uint4 q = J.ent[ea + de];
    ++de;
    const float z = __uint_as_float(q.x);
    if (z > exit_z) continue;  // behind the ray already
    // stage (b) resolved the segment's start: tet << 2 | entry face, and the
    // back colour's transfer-function entry
    started = begin_segment_at(S, J, R, q.z >> 2, q.z & 3u, z, q.w);
    bad = !started;
    break;
  }
  s_de[threadIdx.x] = de;
  if (bad) status |= kDevRange;
  return started;
}

__device__ __forceinline__ void finish_pixel(const JobDev& J, const Ray& R) {
  float c[3] = {R.ar, R.ag, R.ab};
#pragma unroll
  for (int k = 0; k < 3; ++k) c[k] = (c[k] > 1.0f) ? 1.0f : c[k];  // :546-548
  if (J.rgb8) {
    uint8_t* o = J.rgb8 + 3 * (size_t)R.p;
#pragma unroll
    for (int k = 0; k < 3; ++k) o[k] = (uint8_t)__float2int_rz(fmul(255.0f, c[k]));  // :550-552
  }
  if (J.rgba) J.rgba[R.p] = make_float4(c[0], c[1], c[2], fsub(1.0f, R.tr));
  if (J.steps) J.steps[R.p] = R.iters;
}

enum StepResult : uint32_t {
  kContinue = 0, kSegmentEnd = 1, kReload = 2, kCycle = 3, kCap = 4, kRange = 5
};

// The step cap of a ray of this job: the option, or 4 nT + 64 (a walk that
// repeats no state has at most 4 nT iterations).
__device__ __forceinline__ uint32_t step_cap_of(const TraverseParams& P, uint32_t nT) {
  return P.step_cap ? P.step_cap : min(4u * nT + 64u, 0x7fffffffu);
}

// Rare: an iteration beyond the watch threshold.  The cap, then Brent's
// check of the state this iteration starts from (R.t, R.f are still the
// current tet and entry face).
__device__ __forceinline__ uint32_t watched_step(const TraverseParams& P, Ray& R) {
  if (R.iters > step_cap_of(P, R.nT)) return kCap;
  const uint32_t key = (R.t << 2) | R.f;  // nT < 2^30 (checked at upload)
  uint32_t& saved = s_watch_saved[threadIdx.x];
  if (key == saved) return kCycle;
  if ((R.iters & (R.iters - 1u)) == 0u) saved = key;
  return kContinue;
}

// The step's depth difference and extinctions from the exit face's depth zn
// and scalar sn at the pixel (:437-457): dz = |zPrev - zNext| (0 below
// RDELTA) / maxEdgeLength, the front's colour and alpha, tau of the
// front and of the back.  The step ends when sn is outside [0, 1] (:446).
//
// The fast form divides dz by maxEdgeLength through its reciprocal
// (Markstein's correction, as in face_plane_pairs): dz is 0 or at least
// 1e-12 and maxEdgeLength between 2^-100 and 2^80 (another one gets a NaN
// reciprocal in start_ray, and a dz that overflows gives NaN, both of which
// fail the psi coordinates' certificate), so nothing underflows.  Its
// transfer-function entry (uint)(255 sn) (:452) is read off the truncated
// sum with 2^23, and any sn indexes the table in range.
template <bool kExact>
__device__ __forceinline__ void extinction(const SharedTables& S, const Ray& R, float zn, float sn,
                                           float maxEdge, bool& end, float4& front, float& taux,
                                           float& tauy) {
  float dz = fabsf(fsub(R.zp, zn));
  dz = below_rdelta(dz) ? 0.0f : dz;
  end = end || (sn < 0.0f) || (sn > 1.0f);
  const float v = fmul(255.0f, sn);
  uint32_t tfi;
  if (kExact) {
    dz = fdiv(dz, maxEdge);
    tfi = min((uint32_t)v, 255u);
  } else {
    const float q0 = fmul(dz, R.rmaxEdge);
    dz = __fmaf_rn(__fmaf_rn(-maxEdge, q0, dz), R.rmaxEdge, q0);
    tfi = __float_as_uint(__fadd_rz(v, 0x1p23f)) & 255u;
  }
  front = S.tf[tfi];
  taux = fmul(front.w, dz);
  tauy = fmul(R.cb.w, dz);
}

// zeta's argument -(tau_f*0.5 + tau_b*0.5), in double (:459).  Halving is
// exact and commutes with rounding (a double sum of two floats is never
// subnormal), so it is the sum times -0.5.
__device__ __forceinline__ double zeta_arg(float taux, float tauy) {
  return dmul(dadd((double)taux, (double)tauy), -0.5);
}

// The reference's own exponential; not inlined, so that its registers are not
// the step's.
static __device__ __noinline__ float zeta_exact(float taux, float tauy) {
  return (float)exp(zeta_arg(taux, tauy));
}

struct StepColour {
  float r, g, b, t;
};

// The segment's own colour (:473-476): front (1 - psi) + back (psi - zeta),
// in double, per channel rounded to float.
__device__ __forceinline__ float3 segment_colour(const Ray& R, const float4& front, float psif,
                                                 float zeta) {
  const double psi = (double)psif;
  const double ca = dsub(1.0, psi), cbk = dsub(psi, (double)zeta);
  return make_float3((float)dadd(dmul((double)front.x, ca), dmul((double)R.cb.x, cbk)),
                     (float)dadd(dmul((double)front.y, ca), dmul((double)R.cb.y, cbk)),
                     (float)dadd(dmul((double)front.z, ca), dmul((double)R.cb.z, cbk)));
}

// The step's colour and transparency (:477-483) as the reference computes
// them: keep = 1 - a in double with a = (float)(1.0 - zeta).
__device__ __forceinline__ StepColour composite_exact(const Ray& R, float3 f, float zeta) {
  const double keep = dsub(1.0, (double)fsub(1.0f, zeta));
  StepColour o;
  o.r = (float)dadd((double)f.x, dmul(keep, (double)R.ar));
  o.g = (float)dadd((double)f.y, dmul(keep, (double)R.ag));
  o.b = (float)dadd((double)f.z, dmul(keep, (double)R.ab));
  o.t = fmul(R.tr, zeta);
  return o;
}

// The same for zeta in [0, 1].  1 - a is then a float: zeta rounded to a
// multiple of 2^-24 (exact in float: a is 1 - zeta or a multiple of 2^-24),
// its product with a float is exact in double, and the reference's result is
// that sum rounded to double and then to float.  One FMA rounds it once: the
// two differ only where the double rounding lands on a midpoint between
// floats, which takes a sum of more than 53 bits (the accumulated channel
// below a 32nd of the new one) and 28 equal bits in a row, and there the FMA
// is the one nearer to the exact sum.  3 instructions instead of 15, 9 of
// them conversions.
__device__ __forceinline__ StepColour composite_fast(const Ray& R, float3 f, float zeta) {
  const float keep = fsub(1.0f, fsub(1.0f, zeta));
  StepColour o;
  o.r = __fmaf_rn(keep, R.ar, f.x);
  o.g = __fmaf_rn(keep, R.ag, f.y);
  o.b = __fmaf_rn(keep, R.ab, f.z);
  o.t = fmul(R.tr, zeta);
  return o;
}

// One iteration of the reference's while loop (:302-542).  The ways it can
// end before compositing (no exit face, scalar or psi coordinate out of
// range; a cycle or the step cap in watched iterations; an id out of range
// in the checked build) are folded into one flag and the arithmetic runs on
// for every lane; the colour is only committed while the flag says to go
// on, so no lane takes an early branch.  The exact fallbacks of the
// plane, zeta and the psi coordinates are gathered into one rare block
// after the fast path, so the step from the exit tests to the advance is
// one straight run of code that the compiler schedules as a whole.
//
// kWatched: the iteration is past the watch threshold and checked for a
// cycle first (its verdict ends the step like the cap: nothing of it is
// committed).  The loop below takes the unwatched form, which carries no
// trace of the check, for every pass that stays below the threshold.
template <bool kWatched, bool kServe = false>
__device__ __forceinline__ uint32_t step(const TraverseParams& P, const SharedTables& S, Ray& R) {
  ++R.iters;
  const uint32_t wst = kWatched ? watched_step(P, R) : (uint32_t)kContinue;
  bool end = wst != kContinue;
  bool sure;
  uint32_t i = exit_face(R.map, R.low, R.ox, R.oy, sure);
  if (!sure) i = exit_face_exact(R.map, R.low, R.ox, R.oy);
  end = end || i == 0;  // :353 no exit face
  const uint32_t ex = (R.f + i) & 3u;
  const bool xo = (ex & 1u) != 0u, xh = (ex & 2u) != 0u;
  const uint32_t tn = xh ? (xo ? R.w.n.w : R.w.n.z) : (xo ? R.w.n.y : R.w.n.x);
  const uint32_t q = xh ? (xo ? R.w.q.w : R.w.q.z) : (xo ? R.w.q.y : R.w.q.x);
  // both loads of the step, issued before the plane solve that hides them,
  // whatever the exit: tn and the vertex word are valid ids for every face
  // (a boundary face's record names the tet itself and vertex 0; the mesh's
  // ids were validated at upload), so no branch cuts the step.  The checked
  // build compares them first.
  bool bad = id_bad(tn, R.nT) || id_bad(q & 0x07ffffffu, R.nV);
  end = end || bad;
  WalkRec N = R.w;
  float4 nv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (!bad) {
    N = ldg_walk(R.walk, tn);
    nv = __ldg(R.vert + (q & 0x07ffffffu));
  }
  // exit face (ex, ex+1, ex+2) = (r_i, r_i+1, r_i+2): bytes 1-3 of the
  // rotated map
  const uint32_t m = __funnelshift_r(R.map, R.map, 8u * i);
  const float4 a = vtx(vtx_at(m, R.low, 1)), b = vtx(vtx_at(m, R.low, 2)),
               c = vtx(vtx_at(m, R.low, 3));
  // fast path: every quantity from its branch-free estimate, with a flag
  // where the estimate may differ from the reference's value
  float zn, sn;
  const bool plane_ok = face_depth_fast(a, b, c, R.ox, R.oy, P.neg0, zn, sn);
  const bool end0 = end;
  float4 front;
  float taux, tauy;
  extinction<false>(S, R, zn, sn, R.maxEdge, end, front, taux, tauy);
  bool z_ok, psi_ok;
  float zeta = zeta_fast(taux, tauy, S.e2, z_ok);
  const uint32_t pij = psi_coords_fast(taux, tauy, psi_ok);
  StepColour col = composite_fast(R, segment_colour(R, front, __ldg(P.psi + pij), zeta), zeta);
  // rare: the exact path for the lanes whose plane, zeta or psi coordinate
  // was not certified (a plane with a zero or tiny coefficient; about one psi
  // coordinate in 2^12), before anything is committed.  Not rare for a lattice
  // seen along its axes, fields constant in places or opaque transfer
  // functions, so it takes the double exponential and the double psi
  // coordinates only where their own estimates are not certain: a 512^2 view
  // of the 64^3 lattice 1,446 -> 1,283 us, 1024x768 of a field clamped at 0
  // 1,750 -> 1,630, of one with 100 times the extinction 1,256 -> 1,176.
  if ((!plane_ok && !end0) || (!end && !(z_ok && psi_ok))) {
    if (!plane_ok) {
      Plane nf;
      face_plane_ieee(a, b, c, nf);
      zn = plane_eval(R.ox, R.oy, nf.zx, nf.zy, nf.zz);
      sn = plane_eval(R.ox, R.oy, nf.sx, nf.sy, nf.sz);
    }
    end = end0;
    extinction<true>(S, R, zn, sn, job_maxedge(kServe ? *R.jp : P.jobs[R.j]), end, front, taux,
                     tauy);
    zeta = zeta_fast(taux, tauy, S.e2, z_ok);
    uint32_t at = psi_coords_fast(taux, tauy, psi_ok);
    if (!(z_ok && taux >= 0.0f && tauy >= 0.0f)) zeta = zeta_exact(taux, tauy);
    if (!(psi_ok && taux < 1000.0f && tauy < 1000.0f)) {
      const int ci = psi_coord_double(taux), cj = psi_coord_double(tauy);
      end = end || (ci | cj) < 0;  // :468
      at = (uint32_t)max(ci, 0) * 512u + (uint32_t)max(cj, 0);
    }
    col = composite_exact(R, segment_colour(R, front, __ldg(P.psi + at), zeta), zeta);
  }
  if (!end) {
    R.ar = col.r;
    R.ag = col.g;
    R.ab = col.b;
    R.tr = col.t;
    R.lastZ = zn;
    R.cb = front;
  }
  // :535 the ray leaves the mesh through a boundary face; it and a face whose
  // vertices the records could not match by id (the walk goes on, but the
  // caller loads the next tet's vertices first) have these two bits clear
  const bool go_on = !end && (q & 0x60000000u) != 0u;
  // advance to tn through its face fn: the exit face's vertices in tn's order
  // (permutation code), the loaded vertex in the slot of the one left
  // behind.  Done whatever the status: once a ray's segment ends, nothing
  // reads its walk state before begin_segment sets it again.
  const uint32_t fn = (q >> 27) & 3u;
  set_vtx(vtx_at(m, R.low, 0), nv);
  R.map = __byte_perm(m, 0u, perm_selector(q >> 29));
  R.w = N;
  R.t = tn;
  R.f = fn;
  R.zp = zn;
  if (wst != kContinue) return wst;
  if (bad) return kRange;
  // kCodeMismatch is the only one of the two with the top bit set
  return go_on ? (uint32_t)kContinue : kSegmentEnd + (end ? 0u : q >> 31);
}

// Rare (a face whose neighbour lists other vertices): the vertices of the tet
// the step moved to, in the entry face's rotation.  False (checked build
// only): an id is out of range.
template <bool kServe>
__device__ __forceinline__ bool reload(const TraverseParams& P, Ray& R) {
  const uint4 id = __ldg((kServe ? R.jp->tet : P.jobs[R.j].tet) + R.t);
  if (id_bad(id.x, R.nV) || id_bad(id.y, R.nV) || id_bad(id.z, R.nV) || id_bad(id.w, R.nV))
    return false;
  set_vertices(R, id, R.f);
  return true;
}

// Start the ray of the job's local ray index `local`: its pixel, the
// pixel's object coordinates, and its first segment -- the winning entry
// face's, from the start record stage (b) wrote (reference mode: three
// levels of dependent loads, the record, then the tet and its walk record,
// then the vertices), or the first entry of the pixel's list (composited
// mode; kMode 2 takes the mode from the job).  Returns whether the ray
// walks; a composited pixel without a usable entry is finished here.
template <int kMode>
__device__ __forceinline__ bool start_ray(const TraverseParams& P, const SharedTables& S,
                                          const JobDev& J, Ray& R, uint32_t local,
                                          uint32_t& status) {
  R.walk = J.walk;
  R.vert = J.vert;
  R.nT = J.nT;
  R.nV = J.nV;
  R.watch = min(kWatchSteps, step_cap_of(P, J.nT));
  R.maxEdge = job_maxedge(J);
  R.rmaxEdge = R.maxEdge >= 0x1p-100f ? __frcp_rn(R.maxEdge) : __uint_as_float(0x7fffffffu);
  const RayStart rs = J.rays[local];
  R.p = rs.p;
  if (id_bad(R.p, J.W * J.H)) {
    status |= kDevRange;
    return false;
  }
  const uint32_t x = R.p % J.W, y = R.p / J.W;
  R.ox = obj_coord(x, J.W);
  R.oy = obj_coord(y, J.H);
  R.ar = R.ag = R.ab = 0.0f;
  R.tr = 1.0f;
  R.iters = 0;
  const bool ref = kMode == 0 || (kMode == 2 && J.mode == 0);
  if (ref) {  // stage (b) resolved the winning face's segment start
    if (!begin_segment_at(S, J, R, rs.tf >> 2, rs.tf & 3u, __uint_as_float(rs.zp), rs.cbi)) {
      status |= kDevRange;
      return false;
    }
    return true;
  }
  s_ea[threadIdx.x] = J.ent_off[R.p];
  s_en[threadIdx.x] = J.ent_cnt[R.p];
  s_exit_z[threadIdx.x] = INFINITY;
  s_de[threadIdx.x] = 0;
  if (next_entry(S, J, R, status)) return true;
  finish_pixel(J, R);
  return false;
}

// Per-lane tallies of tet-walk steps and status bits, flushed to the job's
// counters when the lane moves to another job and at the end.
struct Tally {
  uint32_t j;
  unsigned long long steps;
  uint32_t status;
};

__device__ __forceinline__ void flush(const TraverseParams& P, Tally& T) {
  if (T.j != 0xffffffffu) {
    ViewCounters* c = P.jobs[T.j].ctr;
    if (T.steps) atomicAdd(&c->steps, T.steps);
    if (T.status) atomicOr(&c->status, T.status);
  }
  T.steps = 0;
  T.status = 0;
}

__device__ __forceinline__ void load_tables(const TraverseParams& P, SharedTables& S) {
  for (uint32_t i = threadIdx.x; i < 256; i += blockDim.x) S.tf[i] = P.tf[i];
  // 2^(-k/64) from the table of 2^(j/64), j = 0..63, scaled by a power of two
  for (uint32_t k = threadIdx.x; k < kExpEntries; k += blockDim.x)
    S.e2[k] = P.e2tab[(64u - (k & 63u)) & 63u] * (1.0 / (double)(1u << ((k + 63u) >> 6)));
  __syncthreads();
}

// kMinBlocks: CTAs of 256 threads the register budget must allow per SM
// (2: no spills; 3: 80 registers, 16 to 24 bytes spilled to L1).
template <int kMode, int kMinBlocks>
__global__ void __launch_bounds__(256, kMinBlocks) traverse_kernel(TraverseParams P) {
  __shared__ SharedTables S;
  load_tables(P, S);
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lt_mask = (1u << lane) - 1u;
  const uint32_t nrays = P.ray_pref[P.njobs];
  const uint32_t refill = P.refill ? P.refill : 1u;
  // A warp's first 32 rays are its share of the front of the list, the queue
  // hands out the rest: thousands of warps taking their first rays from one
  // counter at once serialise there for several microseconds, which is most
  // of a small view's start.  Consecutive chunks go to different CTAs, so a
  // list with fewer chunks than warps spreads over the device.  (A lane
  // without a job has had no ray; if the warp's first chunk left it none, the
  // list is exhausted for the warp.)
  Tally T = {0xffffffffu, 0ull, 0u};
  bool active = false, exhausted = false;
  Ray R;
  R.low = thread_low();
  for (;;) {
    const uint32_t idle = __ballot_sync(0xffffffffu, !active);
    if (idle && !exhausted && ((uint32_t)__popc(idle) >= refill || idle == 0xffffffffu)) {
      const uint32_t leader = __ffs(idle) - 1u, k = __popc(idle);
      uint32_t base = 0;
      if (lane == leader)
        base = T.j == 0xffffffffu ? 32u * ((threadIdx.x >> 5) * gridDim.x + blockIdx.x)
                                  : gridDim.x * blockDim.x + atomicAdd(P.queue, k);
      base = __shfl_sync(0xffffffffu, base, leader);
      if (base + k >= nrays) exhausted = true;
      if (!active) {
        const uint32_t g = base + __popc(idle & lt_mask);
        if (g < nrays) {
          const uint32_t j = job_of(P.ray_pref, P.njobs, g);
          const JobDev& J = P.jobs[j];
          if (j != T.j) {
            flush(P, T);
            T.j = j;
          }
          R.j = j;
          active = start_ray<kMode>(P, S, J, R, g - P.ray_pref[j], T.status);
        }
      }
    }
    if (!__any_sync(0xffffffffu, active)) {
      if (exhausted) break;
      continue;
    }
    if (!active) continue;
    // two steps per pass of the loop: the refill test runs half as often.
    // A pass that would reach the watch threshold takes one watched step
    // instead (rare: rays longer than kWatchSteps iterations).
    uint32_t res;
    if (R.iters + 2u <= R.watch) {
      res = step<false>(P, S, R);
      if (res == kContinue) res = step<false>(P, S, R);
    } else {
      res = step<true>(P, S, R);
    }
    if (res == kContinue) continue;
    if (res == kReload) {
      if (reload<false>(P, R)) continue;
      res = kRange;
    }
    if (res == kSegmentEnd) {
      if (kMode == 1) {
        s_exit_z[threadIdx.x] = R.lastZ;
        if (next_entry(S, P.jobs[R.j], R, T.status)) continue;
      }
      finish_pixel(P.jobs[R.j], R);
    } else if (res == kCycle || res == kCap) {
      // the pixel keeps what the ray composited before it was stopped
      T.status |= res == kCycle ? 32u : 2u;  // VFR_DEV_CYCLE, VFR_DEV_STEP_CAP
      finish_pixel(P.jobs[R.j], R);
    } else {
      T.status |= 4u;
    }
    T.steps += R.iters;
    active = false;
  }
  flush(P, T);
}

// ---------------------------------------------------------------- served

// A served ray has ended: its steps and status go to its job's counters,
// then its count of finished rays; the lane that finishes the job's last ray
// sets the job's completion flag in mapped host memory.  Each lane's pixel
// and counter writes are fenced before its count, and the last lane fences
// at system scope before the flag, so everything the job wrote is visible
// to the host's copy once the flag is.
__device__ __forceinline__ void served_ray_done(const Ray& R, uint32_t status) {
  ViewCounters* c = R.jp->ctr;
  atomicAdd(&c->steps, (unsigned long long)R.iters);
  if (status) atomicOr(&c->status, status);
  __threadfence();
  const uint32_t n = atomicAdd(&c->rays_done, 1u) + 1u;
  if (n == *(volatile const uint32_t*)&c->nrays) {
    __threadfence_system();
    *(volatile uint32_t*)R.done = 1u;
  }
}

// A segment-table entry read through L2 only (ld.global.cg): entries are
// 40 bytes, several to a cache line, and each is written (once per epoch)
// after this launch may already have cached the line for an earlier entry.
__device__ __forceinline__ SegDev load_seg(const SegDev* p) {
  static_assert(sizeof(SegDev) == 40, "segment-table entry layout");
  const unsigned long long* w = reinterpret_cast<const unsigned long long*>(p);
  SegDev d;
  unsigned long long* o = reinterpret_cast<unsigned long long*>(&d);
#pragma unroll
  for (int i = 0; i < 5; ++i) o[i] = __ldcg(w + i);
  return d;
}

// The same for every lane of the warp whose ray ended in this pass (fin),
// aggregated per job: one fence and one atomic per job and pass.  Called by
// the whole warp.  The lanes' pixel writes are ordered before the leader's
// fence by __syncwarp, and the leader's count after its fence.
__device__ __forceinline__ void served_rays_done(const Ray& R, bool fin, uint32_t status) {
  const uint32_t finm = __ballot_sync(0xffffffffu, fin);
  if (!finm) return;
  if (fin) {
    const uint32_t peers = __match_any_sync(finm, (unsigned long long)(uintptr_t)R.jp);
    // steps as two 16-bit halves, so the 32-bit warp sums cannot overflow
    const uint32_t lo = __reduce_add_sync(peers, R.iters & 0xffffu);
    const uint32_t hi = __reduce_add_sync(peers, R.iters >> 16);
    const uint32_t st = __reduce_or_sync(peers, status);
    __syncwarp(peers);
    if ((threadIdx.x & 31u) == (uint32_t)(__ffs(peers) - 1)) {
      ViewCounters* c = R.jp->ctr;
      atomicAdd(&c->steps, ((unsigned long long)hi << 16) + lo);
      if (st) atomicOr(&c->status, st);
      __threadfence();
      const uint32_t n = atomicAdd(&c->rays_done, (uint32_t)__popc(peers)) + __popc(peers);
      if (n == *(volatile const uint32_t*)&c->nrays) {
        __threadfence_system();
        *(volatile uint32_t*)R.done = 1u;
      }
    }
  }
}

// The served form's persistent traversal: one long-lived launch whose warps
// take rays from the published segments in order, oldest first, while the
// host publishes new ones (requests admitted while this launch runs fold
// into it).  A warp holds its place in the segment table: it takes rays from
// its current entry with one atomicAdd on the entry's head and moves on once
// the entry is drained.  Jobs of either mode may be mixed (kMode 2 per job).
// A warp with nothing to do polls for newly published segments: it leaves
// when the host's stop flag is set, or sets VFR_DEV_QUEUE in the control
// word and leaves when it has found nothing for idle_limit microseconds
// (%globaltimer) -- a bounded wait, so a launch never outlives its work by
// much more than that.  The host relaunches it when work arrives after it
// left.
template <int kMinBlocks>
__global__ void __launch_bounds__(256, kMinBlocks) serve_kernel(ServeParams SP) {
  const TraverseParams& P = SP.T;
  __shared__ SharedTables S;
  load_tables(P, S);
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lt_mask = (1u << lane) - 1u;
  const uint32_t refill = P.refill ? P.refill : 1u;
  uint32_t cur = SP.first;  // this warp's entry of the segment table
  // Polling costs: a warp with nothing to do polls the publication count and
  // the stop word (device memory) with plain loads by one lane, backing off
  // from 256 ns to 256 us between polls, and a warp whose claim found
  // nothing while some of its lanes still walk waits 32 passes before it
  // tries again -- thousands of warps polling back to back would make those
  // L2 lines hot spots that slow everything, the preparation kernels beside
  // this launch included.
  unsigned long long idle_since = 0;  // %globaltimer (ns) when the warp found nothing (0: busy)
  uint32_t backoff = 256, quiet = 0;
  bool active = false;
  Ray R;
  R.low = thread_low();
  for (;;) {
    const uint32_t idle = __ballot_sync(0xffffffffu, !active);
    uint32_t seg = 0xffffffffu;
    if (quiet) --quiet;
    if (idle && (idle == 0xffffffffu || ((uint32_t)__popc(idle) >= refill && quiet == 0))) {
      const uint32_t leader = __ffs(idle) - 1u, k = __popc(idle);
      uint32_t base = 0, nr = 0;
      if (lane == leader) {
        const uint32_t pub = *(volatile const uint32_t*)&SP.ctl->published;
        if (cur < pub) {
          // with the publisher's release, the entries below pub are visible
          __threadfence();
          while (cur < pub) {
            SegDev* sg = SP.segs + cur;
            const uint32_t b = atomicAdd(&sg->head, k);
            const uint32_t n = __ldcg(&sg->nrays);  // written before the entry was published
            if (b < n) {
              base = b;
              nr = n;
              seg = cur;
              break;
            }
            ++cur;  // drained: the next entry
          }
        }
      }
      cur = __shfl_sync(0xffffffffu, cur, leader);
      seg = __shfl_sync(0xffffffffu, seg, leader);
      base = __shfl_sync(0xffffffffu, base, leader);
      nr = __shfl_sync(0xffffffffu, nr, leader);
      __syncwarp();  // the leader's fence after the publication orders the lanes' reads
      if (seg == 0xffffffffu) quiet = 32;
      if (seg != 0xffffffffu && !active) {
        const uint32_t g = base + __popc(idle & lt_mask);
        if (g < nr) {
          const SegDev sg = load_seg(SP.segs + seg);
          const uint32_t j = job_of(sg.ray_pref, sg.njobs, g);
          R.jp = sg.jobs + j;
          R.done = sg.done + j;
          uint32_t status = 0;
          active = start_ray<2>(P, S, *R.jp, R, g - sg.ray_pref[j], status);
          if (!active) served_ray_done(R, status);
        }
      }
    }
    if (!__any_sync(0xffffffffu, active)) {
      if (seg == 0xffffffffu) {  // nothing published to take: wait, boundedly
        // lane 0's reads decide for the warp, which leaves together
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        now = __shfl_sync(0xffffffffu, now, 0);
        const uint32_t stop = lane == 0 ? *(volatile const uint32_t*)&SP.ctl->stop : 0u;
        if (__shfl_sync(0xffffffffu, stop, 0)) break;
        if (!idle_since) {
          idle_since = now;
        } else if (now - idle_since > 1000ull * SP.idle_limit) {
          if (lane == 0) atomicOr(&SP.ctl->status, 8u);  // VFR_DEV_QUEUE
          break;
        }
        __nanosleep(backoff);
        backoff = min(2u * backoff, 262144u);
      }
      continue;
    }
    idle_since = 0;
    backoff = 256;
    // every lane goes on to served_rays_done, which syncs the whole warp
    uint32_t res = kContinue;
    if (active) {
      if (R.iters + 2u <= R.watch) {
        res = step<false, true>(P, S, R);
        if (res == kContinue) res = step<false, true>(P, S, R);
      } else {
        res = step<true, true>(P, S, R);
      }
    }
    uint32_t status = 0;
    bool fin = false;
    if (active && res == kReload) res = reload<true>(P, R) ? (uint32_t)kContinue : (uint32_t)kRange;
    if (active && res != kContinue) {
      fin = true;
      if (res == kSegmentEnd) {
        if (R.jp->mode == 1) {
          s_exit_z[threadIdx.x] = R.lastZ;
          fin = !next_entry(S, *R.jp, R, status);
        }
        if (fin) finish_pixel(*R.jp, R);
      } else if (res == kCycle || res == kCap) {
        status = res == kCycle ? 32u : 2u;
        finish_pixel(*R.jp, R);
      } else {
        status = 4u;
      }
    }
    served_rays_done(R, fin, status);
    active = active && !fin;
  }
}

// Publishes a prepared segment: its table entry, then (release) the count
// of published entries the served launch acquires.  Jobs without rays are
// complete now: their pixels were cleared by stage (b).
__global__ void publish_kernel(SegDev* segs, ServeCtl* ctl, uint32_t seq, const JobDev* jobs,
                               const uint32_t* ray_pref, uint32_t* done, uint32_t njobs) {
  if (threadIdx.x == 0) {
    SegDev d;
    d.jobs = jobs;
    d.ray_pref = ray_pref;
    d.done = done;
    d.njobs = njobs;
    d.nrays = ray_pref[njobs];
    d.head = 0;
    d.pad = 0;
    segs[seq] = d;
  }
  __syncthreads();
  for (uint32_t j = threadIdx.x; j < njobs; j += blockDim.x)
    if (ray_pref[j + 1] == ray_pref[j]) {
      __threadfence_system();
      *(volatile uint32_t*)(done + j) = 1u;
    }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(&ctl->published), "r"(seq + 1u) : "memory");
  }
}

}  // namespace vfr

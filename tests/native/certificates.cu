// The shortcuts of the traversal step, as the product's own device functions
// (the headers of vfray_b200/csrc, compiled here), against the plain forms
// they stand for: wherever a shortcut says that its result is certain, the
// plain form must give the same bits.  Prints one line per check:
//
//   name  cases  certified  mismatches
//
// Everything indexes arrays by thread or by table ranges only; the inputs are
// made from the case number.
#include <cstdio>
#include <cmath>
#include <string>
#include <vector>

#include "vfr_traverse.cuh"

using namespace vfr;

struct Count {
  unsigned long long cases, sure, bad;
};

__device__ unsigned long long mix(unsigned long long x) {  // splitmix64
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}
struct Rng {
  unsigned long long s;
  __device__ uint32_t u() { return (uint32_t)(mix(s++) >> 32); }
  __device__ float unit() { return (float)(u() >> 8) * 0x1p-24f; }  // [0, 1)
  __device__ float sym() { return 2.0f * unit() - 1.0f; }
};
__device__ float pow2(int e) { return ldexpf(1.0f, e); }

__device__ void tally(Count* c, bool sure, bool bad) {
  const uint32_t all = __activemask();
  const uint32_t s = __popc(__ballot_sync(all, sure)), b = __popc(__ballot_sync(all, bad));
  if ((int)(threadIdx.x & 31u) == __ffs(all) - 1) {
    atomicAdd(&c->cases, (unsigned long long)__popc(all));
    atomicAdd(&c->sure, (unsigned long long)s);
    atomicAdd(&c->bad, (unsigned long long)b);
  }
}
__device__ bool same(float a, float b) {  // bits, but for the sign of a zero
  return __float_as_uint(a) == __float_as_uint(b) || (a == 0.0f && b == 0.0f);
}
__device__ unsigned long long id() { return blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; }
__device__ unsigned long long stride() { return gridDim.x * (unsigned long long)blockDim.x; }

// every float of a range of bit patterns, both signs
__global__ void reciprocal(Count* c, uint32_t lo, uint32_t hi) {
  for (unsigned long long i = lo + id(); i <= hi; i += stride()) {
    const float b = __uint_as_float((uint32_t)i);
    tally(c, true, rcp_newton(b) != __frcp_rn(b) || rcp_newton(-b) != __frcp_rn(-b));
  }
}

// A triangle of size 2^-span about a ray, scalars of one scale: depth and
// scalar at the ray against the IEEE plane.
__global__ void planes(Count* c, unsigned long long n, int scalar_exp, int zeros, f32x2 neg0) {
  for (unsigned long long i = id(); i < n; i += stride()) {
    Rng r{i * 64ull + 1ull};
    const float size = pow2(-(int)(r.u() % 14u)), ox = r.sym(), oy = r.sym(), oz = r.sym();
    const float sc = pow2(scalar_exp) * (0.5f + r.unit());
    float4 v[3];
    for (int k = 0; k < 3; ++k)
      v[k] = make_float4(ox + size * r.sym(), oy + size * r.sym(), oz + size * r.sym(), sc * r.unit());
    if (zeros & 1) v[1].w = v[0].w, v[2].w = v[0].w;  // a constant scalar
    if (zeros & 2) v[1].z = v[0].z, v[2].z = v[0].z;  // a constant depth
    float z, s;
    const bool ok = face_depth_fast(v[0], v[1], v[2], ox, oy, neg0, z, s);
    Plane p;
    face_plane_ieee(v[0], v[1], v[2], p);
    const float ez = plane_eval(ox, oy, p.zx, p.zy, p.zz), es = plane_eval(ox, oy, p.sx, p.sy, p.sz);
    tally(c, ok, ok && !(same(z, ez) && same(s, es)));
  }
}

// Every extinction below 1000, from 0 up, against the double form; its
// partner is another of the range.
__global__ void psi(Count* c, uint32_t hi) {
  for (unsigned long long i = id(); i < hi; i += stride()) {
    const float x = __uint_as_float((uint32_t)i);
    const float y = __uint_as_float((uint32_t)(mix(i) % hi));
    bool ok;
    const uint32_t at = psi_coords_fast(x, y, ok);
    const int ci = psi_coord_double(x), cj = psi_coord_double(y);
    tally(c, ok, (ok && (ci < 0 || cj < 0 || at != (uint32_t)ci * 512u + (uint32_t)cj)) || at >= 1u << 18);
  }
}

// Pairs of extinctions of any size against the double exponential: half the
// pairs with a sum below 16, the others of all exponents; with pow2s, powers
// of two and their sums (whose products with 32 / ln2 have short significands).
__global__ void zeta(Count* c, unsigned long long n, const double* e2tab, bool pow2s) {
  __shared__ SharedTables S;
  TraverseParams P = {};
  __shared__ float4 zero[256];
  zero[threadIdx.x] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  __syncthreads();
  P.tf = zero;
  P.e2tab = e2tab;
  load_tables(P, S);
  for (unsigned long long i = id(); i < n; i += stride()) {
    Rng r{i * 8ull + 3ull};
    float x, y;
    if (pow2s) {
      x = pow2((int)(r.u() % 277u) - 149);
      y = (i & 1u) ? 0.0f : pow2((int)(r.u() % 277u) - 149);
    } else if (i & 1u) {
      x = 16.0f * r.unit() * pow2(-(int)(r.u() % 24u));
      y = 16.0f * r.unit() * pow2(-(int)(r.u() % 24u));
    } else {
      x = __uint_as_float(r.u() & 0x7fffffffu);  // infinities and NaN too
      y = __uint_as_float(r.u() & 0x7fffffffu);
    }
    bool ok;
    const float z = zeta_fast(x, y, S.e2, ok);
    tally(c, ok, ok && z != (float)exp(zeta_arg(x, y)));
  }
}

// The exit face: a ray inside the entry face's outline, by a margin of
// 2^-(0..30) of the face's size, and a fourth vertex anywhere about it.
// lattice: all offsets are multiples of 2^-2, so that products are often 0.
__global__ void __launch_bounds__(256) exits(Count* c, unsigned long long n, int kind) {
  const uint32_t ident = identity_map(), low = thread_low();
  for (unsigned long long i = id(); i < n; i += stride()) {
    Rng r{i * 32ull + 7ull};
    const float ox = kind ? 0.25f * (float)(int)(r.u() % 9u) - 1.0f : r.sym(), oy = kind ? 0.5f : r.sym();
    const float size = kind ? 1.0f : pow2(-(int)(r.u() % 16u));
    float4 v[4];
    for (int k = 0; k < 4; ++k) {
      const float x = kind ? 0.25f * (float)((int)(r.u() % 9u) - 4) : r.sym();
      const float y = kind ? 0.25f * (float)((int)(r.u() % 9u) - 4) : r.sym();
      v[k] = make_float4(ox + size * x, oy + size * y, 0.0f, 0.0f);
    }
    if (!kind && (i & 1u)) {  // the ray next to the edge from vertex 0 to 1
      const float t = r.unit(), off = size * r.sym() * pow2(-(int)(r.u() % 31u));
      const float ex = v[1].x - v[0].x, ey = v[1].y - v[0].y;
      const float mx = v[0].x + t * ex - off * ey - ox, my = v[0].y + t * ey + off * ex - oy;
      for (int k = 0; k < 4; ++k) v[k].x -= mx, v[k].y -= my;
    }
    if (kind == 2) v[3] = v[(int)(r.u() % 3u)];  // in front of one of the entry face's vertices
    // bytes of the map: r_3, r_0, r_1, r_2
    set_vtx(vtx_at(ident, low, 1), v[0]);
    set_vtx(vtx_at(ident, low, 2), v[1]);
    set_vtx(vtx_at(ident, low, 3), v[2]);
    set_vtx(vtx_at(ident, low, 0), v[3]);
    bool sure;
    const uint32_t face = exit_face(ident, low, ox, oy, sure);
    tally(c, sure, sure && face != exit_face_exact(ident, low, ox, oy));
  }
}

// The step's depth difference and table entries: the fast form against the
// IEEE one, where the extinctions it gives are in the certified range.
__global__ void __launch_bounds__(256) extinctions(Count* c, unsigned long long n) {
  __shared__ SharedTables S;
  for (uint32_t k = threadIdx.x; k < 256u; k += blockDim.x)
    S.tf[k] = make_float4((float)k, 0.0f, 0.0f, 1.0f + (float)k);
  __syncthreads();
  for (unsigned long long i = id(); i < n; i += stride()) {
    Rng r{i * 16ull + 5ull};
    Ray R;
    R.zp = r.sym();
    R.maxEdge = (1.0f + r.unit()) * pow2((int)(r.u() % 178u) - 99);
    R.rmaxEdge = __frcp_rn(R.maxEdge);
    R.cb = make_float4(0.0f, 0.0f, 0.0f, r.unit());
    const float zn = (i & 1u) ? R.zp + r.sym() * pow2(-(int)(r.u() % 40u)) : r.sym();
    const float sn = (i & 7u) ? r.unit() : (float)(r.u() % 256u) / 255.0f;
    bool ea = false, eb = false, ok;
    float4 fa, fb;
    float ax, ay, bx, by;
    extinction<false>(S, R, zn, sn, R.maxEdge, ea, fa, ax, ay);
    extinction<true>(S, R, zn, sn, R.maxEdge, eb, fb, bx, by);
    psi_coords_fast(ax, ay, ok);
    ok = ok && ax < 1000.0f && ay < 1000.0f;
    tally(c, ok, ok && (ea != eb || fa.x != fb.x || ax != bx || ay != by));
  }
}

// A channel in one FMA against the reference's two roundings: at most one
// unit in the last place apart (certified), and never the farther one from
// the exact sum, which is a double here (no more than 53 bits).
__global__ void channels(Count* c, unsigned long long n) {
  for (unsigned long long i = id(); i < n; i += stride()) {
    Rng r{i * 8ull + 11ull};
    Ray R;
    R.ar = R.ag = R.ab = r.unit() * pow2(-(int)(r.u() % 8u));
    R.tr = r.unit();
    const float zeta = fminf(1.0f, r.unit() + 0.004f), f = r.unit() * pow2(-(int)(r.u() % 8u));
    const StepColour a = composite_fast(R, make_float3(f, f, f), zeta);
    const StepColour b = composite_exact(R, make_float3(f, f, f), zeta);
    const int d = __float_as_int(a.r) - __float_as_int(b.r);
    tally(c, d == 0, d < -1 || d > 1 || a.t != b.t || a.r != a.g || a.g != a.b);
  }
}

static bool run(const char* name, const std::string& what, void (*launch)(Count*)) {
  Count *d, h = {};
  if (cudaMalloc(&d, sizeof h) != cudaSuccess) return false;
  cudaMemset(d, 0, sizeof h);
  if (what.empty() || what == name) {
    launch(d);
    if (cudaDeviceSynchronize() != cudaSuccess) {
      std::printf("%s: %s\n", name, cudaGetErrorString(cudaGetLastError()));
      return false;
    }
    cudaMemcpy(&h, d, sizeof h, cudaMemcpyDeviceToHost);
    std::printf("%s %llu %llu %llu\n", name, h.cases, h.sure, h.bad);
  }
  cudaFree(d);
  return true;
}

static double* g_e2;
constexpr f32x2 kNeg0 = 0x8000000080000000ull;
constexpr unsigned long long kMany = 1ull << 27;

template <int kExp, int kZeros>
static void planes_of(Count* c) { planes<<<2048, 256>>>(c, kMany >> 2, kExp, kZeros, kNeg0); }
template <int kKind>
static void exits_of(Count* c) { exits<<<1024, 256>>>(c, kMany, kKind); }

int main(int argc, char** argv) {
  const std::string only = argc > 1 ? argv[1] : "";
  double e2[64];
  for (int j = 0; j < 64; ++j) e2[j] = (double)std::exp2l((long double)j / 64.0L);
  if (cudaMalloc(&g_e2, sizeof e2) != cudaSuccess) return 1;
  cudaMemcpy(g_e2, e2, sizeof e2, cudaMemcpyHostToDevice);
  bool ok = true;
  // 2^-41 .. 2^125
  ok = ok && run("reciprocal", only, [](Count* c) { reciprocal<<<2048, 256>>>(c, 86u << 23, 252u << 23); });
  ok = ok && run("planes", only, planes_of<0, 0>);
  ok = ok && run("planes_scalar_2^-30", only, planes_of<-30, 0>);
  ok = ok && run("planes_scalar_2^-60", only, planes_of<-60, 0>);
  ok = ok && run("planes_scalar_2^-80", only, planes_of<-80, 0>);
  ok = ok && run("planes_scalar_2^-100", only, planes_of<-100, 0>);
  ok = ok && run("planes_scalar_2^-118", only, planes_of<-118, 0>);
  ok = ok && run("planes_scalar_2^-140", only, planes_of<-140, 0>);
  ok = ok && run("planes_constant_scalar", only, planes_of<0, 1>);
  ok = ok && run("planes_constant_depth", only, planes_of<0, 2>);
  ok = ok && run("psi", only, [](Count* c) { psi<<<2048, 256>>>(c, 0x447a0000u); });
  ok = ok && run("zeta", only, [](Count* c) { zeta<<<2048, 256>>>(c, kMany, g_e2, false); });
  ok = ok && run("zeta_powers_of_two", only, [](Count* c) { zeta<<<256, 256>>>(c, kMany >> 4, g_e2, true); });
  ok = ok && run("exits", only, exits_of<0>);
  ok = ok && run("exits_lattice", only, exits_of<1>);
  ok = ok && run("exits_edge_on", only, exits_of<2>);
  ok = ok && run("extinctions", only, [](Count* c) { extinctions<<<1024, 256>>>(c, kMany); });
  ok = ok && run("channels", only, [](Count* c) { channels<<<1024, 256>>>(c, kMany); });
  return ok ? 0 : 1;
}

// Helpers of the render library shared by its .cc and .cu files.
#pragma once
#include <cstdint>
#include <string>

#ifdef __CUDACC__
#define VFR_HOST_DEVICE __host__ __device__
#else
#define VFR_HOST_DEVICE
#endif

namespace vfr {

// Permutation codes.  The walk names a tet's vertices by a 4-byte map
// (vfr_traverse.cuh) whose bytes 1-3 are the exit face's vertices 0-2 in the
// current tet's order, and moves to the next tet with one byte permutation:
// byte 1 + k of the new map is the vertex at place k of the shared face in
// the next tet's order.  The codes are numbered so that the permutation's
// selector, 4 bits per byte, comes from one multiplication, one addition and
// a mask; byte 0 keeps its place.  (Found by searching multiplier and
// addend; 0 and 4, which give no permutation, mark the special faces.)
constexpr uint32_t kCodeMismatch = 4u;
VFR_HOST_DEVICE inline uint32_t perm_selector(uint32_t code) {
  return (code * 0x115bu + 0x11au) & 0x3330u;
}
// the code of the permutation (p0, p1, p2) of (0, 1, 2), 0 if it is none
inline uint32_t perm_code(uint32_t p0, uint32_t p1, uint32_t p2) {
  const uint32_t want = (p0 + 1u) << 4 | (p1 + 1u) << 8 | (p2 + 1u) << 12;
  for (uint32_t c = 1; c < 8; ++c)
    if (c != kCodeMismatch && perm_selector(c) == want) return c;
  return 0u;
}

// Ids in range, adjacency that points back, external faces that are boundary
// faces (vfr_validate.cc).
bool validate_mesh(const uint32_t* tet4, const uint32_t* con4, uint32_t nV, uint32_t nT,
                   const uint32_t* extf2, uint32_t nExt, std::string& why);

// Walk records: per tet 8 words (4 neighbour ids, 4 packed opposite-vertex
// words); nV must be below 2^27 (vfr_validate.cc).
bool build_walk(const uint32_t* tet4, const uint32_t* con4, uint32_t nV, uint32_t nT,
                uint32_t* walk8, std::string& why);

}  // namespace vfr

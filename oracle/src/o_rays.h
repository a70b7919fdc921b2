// ORACLE (test infrastructure only).  Ray queries of the CPU restatement: the closest hit, or whether
// anything is hit, among a scene's triangles.  With the reference's own SBVH at hand
// (oracle/_ref/libksref_sbvh.so, KS_REF_SBVH) it answers them; without it a tree of the oracle's own
// does (o_rays.cpp).  Both make the same watertight triangle test, so they differ only where two
// triangles are hit at equal distances, and in the work that they count.
#pragma once
#include <cstdint>

namespace oracle::rays
{

// A candidate hit on triangle tri at barycentrics (u, v) of vertices 1 and 2 counts when the filter says so.
using Filter = int (*)(void *user, uint32_t tri, float u, float v);

// counts: nodes whose box is tested, triangles tested, stack overflows.
struct Tree
{
    virtual ~Tree() = default;
    // ray: origin, tmin, direction, tmax.  The triangle (~0u: none), or for any-hit queries 1 / 0.  Tests
    // both sides of a triangle.
    virtual uint32_t query(const float ray[8], bool any_hit, float *t, float *bary, uint64_t *counts, Filter filter,
                           void *user) const = 0;
    // The same query by the tree's other implementation where it has one (the reference's own, against its
    // restatement that counts); counts nothing and takes no filter.
    virtual uint32_t query_plain(const float ray[8], bool any_hit, float *t, float *bary) const = 0;
    virtual void bound(float out[6]) const = 0;
};

// Null on invalid input (no triangles).
Tree *build(const float *verts, uint32_t n_verts, const uint32_t *idx, uint32_t n_tris, uint32_t max_prims,
            uint32_t buckets, float trav_weight, float alpha);

// Whether build() makes the reference's SBVH.
bool is_reference();

} // namespace oracle::rays

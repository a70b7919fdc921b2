// ORACLE (test infrastructure only).  See o_rays.h.
#include "o_rays.h"
#include "o_math.h"

#include <algorithm>
#include <array>
#include <cstddef>
#include <numeric>
#include <vector>

#ifdef KS_REF_SBVH
extern "C" {
int ksref_sbvh_build(const float *, uint32_t, const uint32_t *, uint32_t, uint32_t, uint32_t, float, float, void **,
                     uint32_t *, uint32_t *);
uint32_t ksref_sbvh_intersect1(void *, const float *, int, float *, float *);
uint32_t ksref_sbvh_intersect1_counted(void *, const float *, int, int, float *, float *, uint64_t *,
                                       int (*)(void *, uint32_t, float, float), void *);
void ksref_sbvh_bound(void *, float *);
void ksref_sbvh_destroy(void *);
}
#endif

namespace oracle::rays
{
#ifdef KS_REF_SBVH
namespace
{
struct ReferenceTree final : Tree
{
    void *h = nullptr;
    ~ReferenceTree() override
    {
        if (h)
            ksref_sbvh_destroy(h);
    }
    uint32_t query(const float ray[8], bool any_hit, float *t, float *bary, uint64_t *counts, Filter filter,
                   void *user) const override
    {
        return ksref_sbvh_intersect1_counted(h, ray, any_hit, 2, t, bary, counts, filter, user);
    }
    uint32_t query_plain(const float ray[8], bool any_hit, float *t, float *bary) const override
    {
        return ksref_sbvh_intersect1(h, ray, any_hit, t, bary);
    }
    void bound(float out[6]) const override { ksref_sbvh_bound(h, out); }
};
} // namespace

Tree *build(const float *verts, uint32_t n_verts, const uint32_t *idx, uint32_t n_tris, uint32_t max_prims,
            uint32_t buckets, float trav_weight, float alpha)
{
    auto *t = new ReferenceTree;
    uint32_t nodes, prims;
    if (ksref_sbvh_build(verts, n_verts, idx, n_tris, max_prims, buckets, trav_weight, alpha, &t->h, &nodes, &prims) == 0)
        return t;
    delete t;
    return nullptr;
}

bool is_reference() { return true; }

#else
namespace
{

// The watertight test of Woop, Benthin and Wald (Watertight Ray/Triangle Intersection, JCGT 2013): the
// triangle sheared into the ray's frame, the edge functions as differences of products with an error
// term, again in 64 bits where one is zero.
struct Shear
{
    int x, y, z;
    float sx, sy, sz;
    explicit Shear(V3 d)
    {
        z = 0;
        for (int k = 1; k < 3; ++k)
            if (std::fabs(d[k]) > std::fabs(d[z]))
                z = k;
        x = (z + 1) % 3;
        y = (z + 2) % 3;
        if (d[z] < 0.0f)
            std::swap(x, y);
        sx = d[x] / d[z];
        sy = d[y] / d[z];
        sz = 1.0f / d[z];
    }
};

float products_difference(float a, float b, float c, float d) // a b - c d
{
    const float cd = c * d;
    return std::fma(a, b, -cd) + std::fma(-c, d, cd);
}

bool hit_triangle(const Shear &s, V3 o, float tmin, float tmax, const V3 v[3], float &t, float bary[3])
{
    float x[3], y[3], z[3];
    for (int k = 0; k < 3; ++k) {
        const V3 p = v[k] - o;
        x[k] = p[s.x] - s.sx * p[s.z];
        y[k] = p[s.y] - s.sy * p[s.z];
        z[k] = s.sz * p[s.z];
    }
    float e[3]; // edge function opposite vertex k
    for (int k = 0; k < 3; ++k) {
        const int a = (k + 1) % 3, b = (k + 2) % 3;
        e[k] = products_difference(y[a], x[b], y[b], x[a]);
    }
    if (e[0] == 0.0f || e[1] == 0.0f || e[2] == 0.0f)
        for (int k = 0; k < 3; ++k) {
            const int a = (k + 1) % 3, b = (k + 2) % 3;
            e[k] = (float)((double)x[b] * (double)y[a] - (double)y[b] * (double)x[a]);
        }
    const bool below = e[0] < 0.0f || e[1] < 0.0f || e[2] < 0.0f, above = e[0] > 0.0f || e[1] > 0.0f || e[2] > 0.0f;
    if (below && above)
        return false;
    const float det = e[0] + e[1] + e[2];
    if (det == 0.0f)
        return false;
    const float scaled = e[0] * z[0] + e[1] * z[1] + e[2] * z[2];
    if (det < 0.0f ? (scaled >= tmin * det || scaled <= tmax * det) : (scaled <= tmin * det || scaled >= tmax * det))
        return false;
    const float inv = 1.0f / det;
    for (int k = 0; k < 3; ++k)
        bary[k] = e[k] * inv;
    t = scaled * inv;
    return true;
}

// A binary tree over the triangles' boxes, split at the median of the centres' longest axis: shallow
// (its stack has a bound) and the same for every choice of SBVH options.
class MedianTree final : public Tree
{
    struct Node
    {
        float lo[3], hi[3];
        uint32_t first, count; // count > 0: a leaf's triangles; else the children are this + 1 and first
    };
    static constexpr uint32_t kLeaf = 4;
    static constexpr int kStack = 64;
    std::vector<V3> corners_; // three per triangle, in tree order
    std::vector<uint32_t> ids_;
    std::vector<Node> nodes_;

    void make(std::vector<uint32_t> &order, const std::vector<std::array<float, 6>> &box, uint32_t begin, uint32_t end)
    {
        const uint32_t me = (uint32_t)nodes_.size();
        nodes_.emplace_back();
        Node n;
        float clo[3], chi[3];
        for (int a = 0; a < 3; ++a) {
            n.lo[a] = clo[a] = inf;
            n.hi[a] = chi[a] = -inf;
        }
        for (uint32_t k = begin; k < end; ++k) {
            const auto &b = box[order[k]];
            for (int a = 0; a < 3; ++a) {
                n.lo[a] = std::min(n.lo[a], b[a]);
                n.hi[a] = std::max(n.hi[a], b[3 + a]);
                const float c = 0.5f * b[a] + 0.5f * b[3 + a];
                clo[a] = std::min(clo[a], c);
                chi[a] = std::max(chi[a], c);
            }
        }
        n.first = begin;
        n.count = end - begin;
        if (n.count > kLeaf) {
            int axis = 0;
            for (int a = 1; a < 3; ++a)
                if (chi[a] - clo[a] > chi[axis] - clo[axis])
                    axis = a;
            const uint32_t mid = begin + n.count / 2;
            std::nth_element(order.begin() + begin, order.begin() + mid, order.begin() + end,
                             [&](uint32_t p, uint32_t q) {
                                 const float c = 0.5f * box[p][axis] + 0.5f * box[p][3 + axis];
                                 const float d = 0.5f * box[q][axis] + 0.5f * box[q][3 + axis];
                                 return c != d ? c < d : p < q;
                             });
            n.count = 0;
            make(order, box, begin, mid);
            n.first = (uint32_t)nodes_.size();
            make(order, box, mid, end);
        }
        nodes_[me] = n;
    }

    // Entry time of a box, or infinity.  Plane times have three roundings, each at most 2^-24 of the value:
    // the far ones are moved out by 2^-21 of theirs so that no box holding a hit is missed.
    static float enter(const Node &n, V3 o, V3 inv, float tmin, float tmax)
    {
        for (int a = 0; a < 3; ++a) {
            float near = (n.lo[a] - o[a]) * inv[a], far = (n.hi[a] - o[a]) * inv[a];
            if (std::signbit(inv[a]))
                std::swap(near, far);
            far += std::fabs(far) * 0x1p-21f;
            // 0 * inf: the ray lies in a plane of the box, which bounds nothing
            if (near > tmin)
                tmin = near;
            if (far < tmax)
                tmax = far;
        }
        return tmin <= tmax ? tmin : inf;
    }

public:
    MedianTree(const float *verts, const uint32_t *idx, uint32_t n)
    {
        std::vector<std::array<float, 6>> box(n);
        ids_.resize(n);
        std::iota(ids_.begin(), ids_.end(), 0u);
        for (uint32_t t = 0; t < n; ++t)
            for (int a = 0; a < 3; ++a) {
                const float p = verts[3 * idx[3 * t] + a], q = verts[3 * idx[3 * t + 1] + a], r = verts[3 * idx[3 * t + 2] + a];
                box[t][a] = std::min(p, std::min(q, r));
                box[t][3 + a] = std::max(p, std::max(q, r));
            }
        nodes_.reserve(n);
        make(ids_, box, 0, n);
        corners_.reserve(3 * (size_t)n);
        for (uint32_t t : ids_)
            for (int k = 0; k < 3; ++k) {
                const float *v = verts + 3 * (size_t)idx[3 * (size_t)t + k];
                corners_.emplace_back(v[0], v[1], v[2]);
            }
    }

    uint32_t query(const float ray[8], bool any_hit, float *t_out, float *bary_out, uint64_t *counts, Filter filter,
                   void *user) const override
    {
        const V3 o(ray[0], ray[1], ray[2]), d(ray[4], ray[5], ray[6]);
        const V3 inv(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
        const float tmin = ray[3];
        float tmax = ray[7];
        const Shear shear(d);
        uint32_t result = ~0u;
        struct Entry
        {
            uint32_t node;
            float t;
        } stack[kStack];
        int sp = 0;
        auto visit = [&](uint32_t i) {
            ++counts[0];
            return enter(nodes_[i], o, inv, tmin, tmax);
        };
        float t0 = visit(0);
        if (t0 < inf)
            stack[sp++] = {0, t0};
        while (sp > 0) {
            const Entry e = stack[--sp];
            if (e.t > tmax)
                continue;
            const Node &n = nodes_[e.node];
            if (n.count == 0) {
                const uint32_t l = e.node + 1, r = n.first;
                const float tl = visit(l), tr = visit(r);
                const bool left_near = tl <= tr;
                const Entry near = left_near ? Entry{l, tl} : Entry{r, tr}, far = left_near ? Entry{r, tr} : Entry{l, tl};
                if (far.t < inf)
                    stack[sp++] = far;
                if (near.t < inf)
                    stack[sp++] = near;
                continue;
            }
            for (uint32_t k = n.first; k < n.first + n.count; ++k) {
                ++counts[1];
                float t, b[3];
                if (!hit_triangle(shear, o, tmin, ray[7], &corners_[3 * (size_t)k], t, b))
                    continue;
                const uint32_t id = ids_[k];
                // equal distances: the lower triangle
                if (!any_hit && (result != ~0u ? (t > tmax || (t == tmax && id > result)) : !(t < tmax)))
                    continue;
                if (filter && !filter(user, id, b[1], b[2]))
                    continue;
                if (any_hit)
                    return 1u;
                tmax = t;
                result = id;
                *t_out = t;
                std::copy(b, b + 3, bary_out);
            }
        }
        return any_hit ? 0u : result;
    }

    uint32_t query_plain(const float ray[8], bool any_hit, float *t, float *bary) const override
    {
        uint64_t counts[3] = {0, 0, 0};
        return query(ray, any_hit, t, bary, counts, nullptr, nullptr);
    }

    void bound(float out[6]) const override
    {
        std::copy(nodes_[0].lo, nodes_[0].lo + 3, out);
        std::copy(nodes_[0].hi, nodes_[0].hi + 3, out + 3);
    }
};

} // namespace

Tree *build(const float *verts, uint32_t, const uint32_t *idx, uint32_t n_tris, uint32_t, uint32_t, float, float)
{
    return verts && idx && n_tris ? new MedianTree(verts, idx, n_tris) : nullptr;
}

bool is_reference() { return false; }
#endif

} // namespace oracle::rays

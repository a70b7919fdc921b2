// Parallel SBVH builder for sm_100a.
//
// Produces the same tree as the reference's sequential builder ksc::SBVH::build
// (cuda/sbvh.cu:81-440): same SAH object-split estimate (:81-136), same spatial-split estimate
// (:138-216) and skip test (:132-134), same leaf rule (:351-354), same reference un-splitting
// (:257-287), same depth-first flattening (:375-393).  Every split decision of the reference
// depends only on the *multiset* of references of a node (min/max unions, integer counts, and
// per-reference tests against fixed per-node values), so the tree can be built breadth-first,
// one level of nodes at a time, with all references of the level processed in parallel:
//
//   per level:  bounds -> prep -> object bins -> object eval -> spatial bins -> decide
//               -> spatial classes -> spatial costs -> count -> scan -> scatter -> children
//
// Floating-point expressions are written exactly as in the reference (std::min/std::max
// argument order, std::lerp, float(count) * area, ...) and the translation unit is compiled with
// -fmad=false, so every cost and comparison rounds as on the reference's host.
// Min/max accumulation across threads uses an order-preserving integer encoding of floats and
// integer atomics, which is exact and deterministic.  Only the order of primitives inside a leaf
// can differ from the reference (it depends on std::partition's swap order).
#include "ks_scan.cuh"
#include "ks_scene.h"
#include "ks_traverse4.cuh"

#include <algorithm>
#include <cstring>

namespace ksb
{
namespace
{

constexpr int kMaxBuckets = 16;
// References per work item (one warp each).  The serial steps of a warp, not the bandwidth, bound the upper levels'
// kernels.  Builds of 82 K, 328 K and 1.3 M triangles: items of 1024 4.1, 5.4 and 10.3 ms, 512 3.5, 4.6 and 9.7, 256 3.3,
// 4.5 and 9.65, 128 3.1, 4.5 and 10.3 (more atomics on the nodes' tables).
#ifndef KS_BUILD_CHUNK
#define KS_BUILD_CHUNK 256
#endif
constexpr uint32_t kChunk = KS_BUILD_CHUNK;
constexpr int kEvalLanes = 16; // lanes that evaluate a node's splits, one each
static_assert(kMaxBuckets <= kEvalLanes, "a lane per split");
constexpr int kWarpsPerBlock = 8;

enum NodeKind : int
{
    kPending = 0,
    kLeaf = 1,
    kObject = 2,
    kSpatial = 3,
};

struct BRef
{
    float4 lo; // min xyz, original triangle index (bits) in w
    float4 hi; // max xyz
};

struct LevelNode
{
    uint32_t ref_begin, ref_count, build_id, first_item;
};

struct Item
{
    uint32_t node, begin, count, single;
};

struct NodeInfo
{
    float bmin[3], bmax[3], cmin[3], cmax[3];
    int kind, dim, skip;
    int os_bucket;
    float os_cost;
    float osL[6], osR[6];
    int ss_bucket;
    float ss_cost;
    float ssL[6], ssR[6];
    float clip[kMaxBuckets + 1];
    float split_clip;
    int n1, n2;
    float full_cost, saL, saR;
    uint32_t cls[3];
    uint32_t n_left, n_right;
};

struct BuildRec
{
    float bmin[3], bmax[3];
    uint32_t left, right, axis, leaf;
    uint32_t leaf_begin, leaf_count;
    uint32_t size, prims;
    uint32_t dfs, prim_off;
};

struct Params
{
    uint32_t max_prims;
    uint32_t buckets;
    float trav_weight;
    float alpha;
};

// ---- float helpers with the reference's host semantics -------------------------------------
KS_D float smin(float a, float b) { return (b < a) ? b : a; } // std::min(a, b)
KS_D float smax(float a, float b) { return (a < b) ? b : a; } // std::max(a, b)

// Order-preserving map float -> uint32 (total order, -0 < +0), exact round trip.
KS_D uint32_t f2o(float f)
{
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
KS_D float o2f(uint32_t o) { return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o); }
constexpr uint32_t kOInf = 0xFF800000u;    // f2o(+inf): identity for min
constexpr uint32_t kONegInf = 0x007FFFFFu; // f2o(-inf): identity for max

KS_D float surface_area(const float mn[3], const float mx[3])
{
    float ex = mx[0] - mn[0], ey = mx[1] - mn[1], ez = mx[2] - mn[2];
    return 2.0f * (ex * ey + ey * ez + ex * ez);
}
KS_D void box_empty(float b[6])
{
    b[0] = b[1] = b[2] = kInf;
    b[3] = b[4] = b[5] = -kInf;
}
KS_D void box_expand(float b[6], const float o[6])
{
    for (int k = 0; k < 3; ++k) {
        b[k] = smin(b[k], o[k]);
        b[3 + k] = smax(b[3 + k], o[3 + k]);
    }
}
KS_D float ref_lo(const BRef &r, int d) { return d == 0 ? r.lo.x : (d == 1 ? r.lo.y : r.lo.z); }
KS_D float ref_hi(const BRef &r, int d) { return d == 0 ? r.hi.x : (d == 1 ? r.hi.y : r.hi.z); }
KS_D float ref_center(const BRef &r, int d) { return 0.5f * (ref_lo(r, d) + ref_hi(r, d)); }

// Bucket of a reference for the object split (cuda/sbvh.cu:98-100).
KS_D uint32_t object_bucket(const BRef &r, const NodeInfo &n, uint32_t buckets)
{
    int d = n.dim;
    float ext = n.cmax[d] - n.cmin[d];
    float off = ext == 0.0f ? 0.0f : (ref_center(r, d) - n.cmin[d]) / ext;
    uint32_t b = (uint32_t)floorf((float)buckets * off);
    return b < buckets - 1 ? b : buckets - 1;
}

// Reference un-splitting decision for a straddling reference (cuda/sbvh.cu:257-287).
// Returns 0 = move left, 1 = move right, 2 = split.
KS_D int unsplit_decision(const BRef &r, const NodeInfo &n)
{
    float rb[6] = {r.lo.x, r.lo.y, r.lo.z, r.hi.x, r.hi.y, r.hi.z};
    float jl[6], jr[6];
    for (int k = 0; k < 6; ++k) {
        jl[k] = n.ssL[k];
        jr[k] = n.ssR[k];
    }
    // join(a, b) = AABB3(min(a.min, b.min), max(a.max, b.max)) with ksc::min/max = std::min/max
    for (int k = 0; k < 3; ++k) {
        jl[k] = smin(jl[k], rb[k]);
        jl[3 + k] = smax(jl[3 + k], rb[3 + k]);
        jr[k] = smin(jr[k], rb[k]);
        jr[3 + k] = smax(jr[3 + k], rb[3 + k]);
    }
    float move_left = surface_area(jl, jl + 3) * (float)n.n1 + n.saR * (float)(n.n2 - 1);
    float move_right = n.saL * (float)(n.n1 - 1) + surface_area(jr, jr + 3) * (float)n.n2;
    float m = smin(n.full_cost, smin(move_left, move_right));
    if (m == move_left)
        return 0;
    if (m == move_right)
        return 1;
    return 2;
}

// Destination of a reference: bit0 = goes left, bit1 = goes right, bit2 = to leaf pool.
KS_D int ref_destination(const BRef &r, const NodeInfo &n, uint32_t buckets)
{
    if (n.kind == kLeaf)
        return 4;
    if (n.kind == kObject)
        return object_bucket(r, n, buckets) <= (uint32_t)n.os_bucket ? 1 : 2;
    int d = n.dim;
    if (ref_hi(r, d) <= n.split_clip)
        return 1;
    if (ref_lo(r, d) >= n.split_clip)
        return 2;
    int u = unsplit_decision(r, n);
    return u == 0 ? 1 : (u == 1 ? 2 : 3);
}

// ---- kernels --------------------------------------------------------------------------------

__global__ void k_init_refs(const float *verts, const uint32_t *idx, uint32_t tri_begin, uint32_t n_tris, BRef *refs)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_tris)
        return;
    float b[6];
    box_empty(b);
    for (int v = 0; v < 3; ++v) {
        uint32_t vi = idx[3 * (tri_begin + i) + v];
        float p[6] = {verts[3 * vi], verts[3 * vi + 1], verts[3 * vi + 2], 0, 0, 0};
        p[3] = p[0];
        p[4] = p[1];
        p[5] = p[2];
        box_expand(b, p);
    }
    refs[i].lo = make_float4(b[0], b[1], b[2], __uint_as_float(tri_begin + i));
    refs[i].hi = make_float4(b[3], b[4], b[5], 0.0f);
}

KS_D uint32_t item_count(uint32_t refs) { return (refs + kChunk - 1) / kChunk; }

// The work items of every node, and its accumulators' start: kEvalLanes lanes a node.
__global__ void k_items_fill(LevelNode *nodes, uint32_t n, const uint32_t *item_off, Item *items, uint32_t *bnd,
                             uint32_t *obj, uint32_t *sp, NodeInfo *info, uint32_t buckets)
{
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) / kEvalLanes, lane = threadIdx.x % kEvalLanes;
    if (i >= n)
        return;
    const uint32_t ref_begin = nodes[i].ref_begin, ref_count = nodes[i].ref_count;
    const uint32_t first = item_off[i], cnt = item_off[i + 1] - first;
    for (uint32_t k = lane; k < cnt; k += kEvalLanes) {
        Item it;
        it.node = i;
        it.begin = ref_begin + k * kChunk;
        uint32_t rem = ref_count - k * kChunk;
        it.count = rem < kChunk ? rem : kChunk;
        it.single = cnt == 1;
        items[first + k] = it;
    }
    if (lane == 0)
        nodes[i].first_item = first;
    if (lane < 3)
        info[i].cls[lane] = 0;
    if (cnt == 1)
        return; // single work item: every accumulator is written with plain stores
    if (lane < 12)
        bnd[12 * i + lane] = (lane < 3 || (lane >= 6 && lane < 9)) ? kOInf : kONegInf;
    for (uint32_t k = lane; k < buckets * 7; k += kEvalLanes) {
        const uint32_t f = k % 7;
        obj[(size_t)i * buckets * 7 + k] = f == 0 ? 0u : (f < 4 ? kOInf : kONegInf);
    }
    for (uint32_t k = lane; k < buckets * 8; k += kEvalLanes) {
        const uint32_t f = k % 8;
        sp[(size_t)i * buckets * 8 + k] = f < 2 ? 0u : (f < 5 ? kOInf : kONegInf);
    }
}

KS_D float warp_min(float v)
{
    for (int o = 16; o > 0; o >>= 1)
        v = smin(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
KS_D float warp_max(float v)
{
    for (int o = 16; o > 0; o >>= 1)
        v = smax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Node bounds and centroid bounds (cuda/sbvh.cu:308-313, 330-333).
__global__ void k_bounds(const Item *items, const uint32_t *n_items, const BRef *refs, uint32_t *bnd)
{
    uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= *n_items)
        return;
    Item it = items[w];
    float v[12];
    for (int k = 0; k < 3; ++k) {
        v[k] = kInf;
        v[3 + k] = -kInf;
        v[6 + k] = kInf;
        v[9 + k] = -kInf;
    }
    for (uint32_t j = lane; j < it.count; j += 32) {
        BRef r = refs[it.begin + j];
        float lo[3] = {r.lo.x, r.lo.y, r.lo.z}, hi[3] = {r.hi.x, r.hi.y, r.hi.z};
        for (int k = 0; k < 3; ++k) {
            v[k] = smin(v[k], lo[k]);
            v[3 + k] = smax(v[3 + k], hi[k]);
            float c = 0.5f * (lo[k] + hi[k]);
            v[6 + k] = smin(v[6 + k], c);
            v[9 + k] = smax(v[9 + k], c);
        }
    }
    for (int k = 0; k < 3; ++k) {
        v[k] = warp_min(v[k]);
        v[3 + k] = warp_max(v[3 + k]);
        v[6 + k] = warp_min(v[6 + k]);
        v[9 + k] = warp_max(v[9 + k]);
    }
    if (lane < 12) {
        float x = v[0];
        for (int k = 1; k < 12; ++k)
            if ((int)lane == k)
                x = v[k];
        bool is_min = lane < 3 || (lane >= 6 && lane < 9);
        uint32_t *dst = bnd + 12 * it.node + lane;
        if (it.single)
            *dst = f2o(x);
        else if (is_min)
            atomicMin(dst, f2o(x));
        else
            atomicMax(dst, f2o(x));
    }
}

__device__ float g_root_sa;

// Leaf tests before any split estimate (cuda/sbvh.cu:301-338) + node record.
__global__ void k_prep(const LevelNode *nodes, uint32_t n, const uint32_t *bnd, NodeInfo *info, BuildRec *recs,
                       int is_root_level)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    NodeInfo &ni = info[i];
    for (int k = 0; k < 3; ++k) {
        ni.bmin[k] = o2f(bnd[12 * i + k]);
        ni.bmax[k] = o2f(bnd[12 * i + 3 + k]);
        ni.cmin[k] = o2f(bnd[12 * i + 6 + k]);
        ni.cmax[k] = o2f(bnd[12 * i + 9 + k]);
    }
    if (is_root_level)
        g_root_sa = surface_area(ni.bmin, ni.bmax);
    BuildRec &rec = recs[nodes[i].build_id];
    for (int k = 0; k < 3; ++k) {
        rec.bmin[k] = ni.bmin[k];
        rec.bmax[k] = ni.bmax[k];
    }
    ni.kind = kPending;
    ni.skip = 1;
    if (nodes[i].ref_count == 1) {
        ni.kind = kLeaf;
        return;
    }
    float ex = ni.cmax[0] - ni.cmin[0], ey = ni.cmax[1] - ni.cmin[1], ez = ni.cmax[2] - ni.cmin[2];
    int dim = (ex >= ey && ex >= ez) ? 0 : ((ey >= ex && ey >= ez) ? 1 : 2);
    ni.dim = dim;
    if (ni.cmax[dim] == ni.cmin[dim])
        ni.kind = kLeaf;
}

// Object-split bucket statistics (cuda/sbvh.cu:95-102).
__global__ void k_obj_bins(const Item *items, const uint32_t *n_items, const BRef *refs, const NodeInfo *info,
                           uint32_t buckets, uint32_t *obj)
{
    __shared__ uint32_t sbins[kWarpsPerBlock][kMaxBuckets * 7];
    uint32_t wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t w = blockIdx.x * kWarpsPerBlock + wl;
    if (w >= *n_items)
        return;
    Item it = items[w];
    const NodeInfo &ni = info[it.node];
    if (ni.kind != kPending)
        return;
    uint32_t *sb = sbins[wl];
    for (uint32_t k = lane; k < buckets * 7; k += 32) {
        uint32_t f = k % 7;
        sb[k] = f == 0 ? 0u : (f < 4 ? kOInf : kONegInf);
    }
    __syncwarp();
    for (uint32_t j = lane; j < it.count; j += 32) {
        BRef r = refs[it.begin + j];
        uint32_t b = object_bucket(r, ni, buckets);
        uint32_t *o = sb + b * 7;
        atomicAdd(o, 1u);
        atomicMin(o + 1, f2o(r.lo.x));
        atomicMin(o + 2, f2o(r.lo.y));
        atomicMin(o + 3, f2o(r.lo.z));
        atomicMax(o + 4, f2o(r.hi.x));
        atomicMax(o + 5, f2o(r.hi.y));
        atomicMax(o + 6, f2o(r.hi.z));
    }
    __syncwarp();
    uint32_t *dst = obj + (size_t)it.node * buckets * 7;
    for (uint32_t k = lane; k < buckets * 7; k += 32) {
        uint32_t f = k % 7;
        if (it.single)
            dst[k] = sb[k];
        else if (f == 0)
            atomicAdd(dst + k, sb[k]);
        else if (f < 4)
            atomicMin(dst + k, sb[k]);
        else
            atomicMax(dst + k, sb[k]);
    }
}

// Picks the cheapest split of a bucket table (cuda/sbvh.cu:104-130, 190-216) with kEvalLanes lanes, one split each,
// and writes it (all lanes of the warp call; a group without a node passes its own flag).
// lc, rc, box: a bucket's counts for the left and the right side, and its bounds.
// Bound by the latency of its table reads: a thread per node went over the table 15 times (k_obj_eval and k_decide
// 1.02 + 0.44 ms of the build of a level-7 icosphere's 327680 triangles, 21 us for the root alone; now 0.42 + 0.16).
template <typename LeftCount, typename RightCount, typename BoxOf>
KS_D void best_split(bool active, uint32_t lane, uint32_t buckets, float travw, float node_sa, LeftCount lc, RightCount rc,
                     BoxOf box, int &best_bucket, float &best_cost, float bl[6], float br[6])
{
    float L[6], R[6], cost = kInf;
    box_empty(L);
    box_empty(R);
    if (active && lane + 1 < buckets) {
        uint32_t c0 = 0, c1 = 0;
        for (uint32_t j = 0; j < buckets; ++j) {
            float b[6];
            box(j, b);
            if (j <= lane) {
                box_expand(L, b);
                c0 += lc(j);
            } else {
                box_expand(R, b);
                c1 += rc(j);
            }
        }
        cost = travw + ((float)c0 * surface_area(L, L + 3) + (float)c1 * surface_area(R, R + 3)) / node_sa;
        // the first split stands even where its cost is not a number; a later one then never wins
        if (lane > 0 && !(cost == cost))
            cost = kInf;
    }
    uint32_t best = lane;
    float best_c = cost;
    for (int o = 1; o < kEvalLanes; o <<= 1) {
        const float c = __shfl_xor_sync(0xffffffffu, best_c, o);
        const uint32_t l = __shfl_xor_sync(0xffffffffu, best, o);
        // the lower split unless the higher one is cheaper
        if (l > best ? c < best_c : !(best_c < c)) {
            best = l;
            best_c = c;
        }
    }
    if (active && lane == best) {
        best_bucket = (int)lane;
        best_cost = cost;
        for (int k = 0; k < 6; ++k) {
            bl[k] = L[k];
            br[k] = R[k];
        }
    }
    __syncwarp();
}

__global__ void k_obj_eval(uint32_t n, const uint32_t *obj, NodeInfo *info, Params p)
{
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) / kEvalLanes, lane = threadIdx.x % kEvalLanes;
    const bool active = i < n && info[i].kind == kPending;
    NodeInfo &ni = info[i < n ? i : 0];
    const uint32_t *o = obj + (size_t)(i < n ? i : 0) * p.buckets * 7;
    float node_sa = surface_area(ni.bmin, ni.bmax);
    auto cnt = [&](uint32_t j) { return o[j * 7]; };
    auto box = [&](uint32_t j, float b[6]) {
        for (int k = 0; k < 6; ++k)
            b[k] = o2f(o[j * 7 + 1 + k]);
    };
    best_split(active, lane, p.buckets, p.trav_weight, node_sa, cnt, cnt, box, ni.os_bucket, ni.os_cost, ni.osL, ni.osR);
    if (!active)
        return;
    // skipSpatialSplit (cuda/sbvh.cu:132-134)
    float imn[3], imx[3];
    bool empty = false;
    for (int k = 0; k < 3; ++k) {
        imn[k] = smax(ni.osL[k], ni.osR[k]);
        imx[k] = smin(ni.osL[3 + k], ni.osR[3 + k]);
    }
    if (imn[0] > imx[0] || imn[1] > imx[1] || imn[2] > imx[2])
        empty = true; // intersect() returns an empty AABB3, whose is_empty() is true
    float isa = empty ? 0.0f : surface_area(imn, imx);
    const int skip = (isa / g_root_sa <= p.alpha) ? 1 : 0;
    if (lane == 0)
        ni.skip = skip;
    if (!skip) {
        int d = ni.dim;
        for (uint32_t b = lane; b <= p.buckets; b += kEvalLanes)
            ni.clip[b] = std_lerp(ni.bmin[d], ni.bmax[d], (float)b / (float)p.buckets);
    }
}

// Spatial-split bucket statistics (cuda/sbvh.cu:154-176).
__global__ void k_sp_bins(const Item *items, const uint32_t *n_items, const BRef *refs, const NodeInfo *info,
                          uint32_t buckets, uint32_t *sp)
{
    __shared__ uint32_t sbins[kWarpsPerBlock][kMaxBuckets * 8];
    uint32_t wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t w = blockIdx.x * kWarpsPerBlock + wl;
    if (w >= *n_items)
        return;
    Item it = items[w];
    const NodeInfo &ni = info[it.node];
    if (ni.kind != kPending || ni.skip)
        return;
    uint32_t *sb = sbins[wl];
    for (uint32_t k = lane; k < buckets * 8; k += 32) {
        uint32_t f = k % 8;
        sb[k] = f < 2 ? 0u : (f < 5 ? kOInf : kONegInf);
    }
    __syncwarp();
    int d = ni.dim;
    for (uint32_t j = lane; j < it.count; j += 32) {
        BRef r = refs[it.begin + j];
        float lo[3] = {r.lo.x, r.lo.y, r.lo.z}, hi[3] = {r.hi.x, r.hi.y, r.hi.z};
        uint32_t enter = buckets - 1, exit = 0;
        for (uint32_t b = 0; b < buckets; ++b) {
            if (lo[d] > ni.clip[b + 1])
                continue;
            if (hi[d] < ni.clip[b])
                break;
            exit = exit < b ? b : exit;   // std::max(exit, b)
            enter = b < enter ? b : enter; // std::min(enter, b)
            float cl[3] = {lo[0], lo[1], lo[2]}, ch[3] = {hi[0], hi[1], hi[2]};
            cl[d] = smax(cl[d], ni.clip[b]);
            ch[d] = smin(ch[d], ni.clip[b + 1]);
            uint32_t *s = sb + b * 8;
            for (int k = 0; k < 3; ++k) {
                atomicMin(s + 2 + k, f2o(cl[k]));
                atomicMax(s + 5 + k, f2o(ch[k]));
            }
        }
        atomicAdd(sb + enter * 8 + 0, 1u);
        atomicAdd(sb + exit * 8 + 1, 1u);
    }
    __syncwarp();
    uint32_t *dst = sp + (size_t)it.node * buckets * 8;
    for (uint32_t k = lane; k < buckets * 8; k += 32) {
        uint32_t f = k % 8;
        if (it.single)
            dst[k] = sb[k];
        else if (f < 2)
            atomicAdd(dst + k, sb[k]);
        else if (f < 5)
            atomicMin(dst + k, sb[k]);
        else
            atomicMax(dst + k, sb[k]);
    }
}

// Spatial estimate + leaf/object/spatial decision (cuda/sbvh.cu:347-360).
__global__ void k_decide(const LevelNode *nodes, uint32_t n, const uint32_t *sp, NodeInfo *info, Params p)
{
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) / kEvalLanes, lane = threadIdx.x % kEvalLanes;
    const bool active = i < n && info[i].kind == kPending;
    NodeInfo &ni = info[i < n ? i : 0];
    const bool skip = ni.skip;
    const uint32_t *s = sp + (size_t)(i < n ? i : 0) * p.buckets * 8;
    float node_sa = surface_area(ni.bmin, ni.bmax);
    auto enter = [&](uint32_t j) { return s[j * 8 + 0]; };
    auto exitc = [&](uint32_t j) { return s[j * 8 + 1]; };
    auto box = [&](uint32_t j, float b[6]) {
        for (int k = 0; k < 6; ++k)
            b[k] = o2f(s[j * 8 + 2 + k]);
    };
    best_split(active && !skip, lane, p.buckets, p.trav_weight, node_sa, enter, exitc, box, ni.ss_bucket, ni.ss_cost, ni.ssL,
               ni.ssR);
    if (!active || lane)
        return;
    uint32_t ref_count = nodes[i].ref_count;
    float leaf_cost = (float)ref_count;
    if (ref_count <= p.max_prims && leaf_cost <= ni.os_cost && (skip || leaf_cost <= ni.ss_cost)) {
        ni.kind = kLeaf;
        return;
    }
    if (skip || ni.os_cost <= ni.ss_cost) {
        ni.kind = kObject;
    } else {
        ni.kind = kSpatial;
        int d = ni.dim;
        ni.split_clip = std_lerp(ni.bmin[d], ni.bmax[d], (float)(ni.ss_bucket + 1) / (float)p.buckets);
    }
}

// Left / right / straddling counts of a spatial split (cuda/sbvh.cu:242-251).
__global__ void k_sp_classes(const Item *items, const uint32_t *n_items, const BRef *refs, NodeInfo *info)
{
    uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= *n_items)
        return;
    Item it = items[w];
    NodeInfo &ni = info[it.node];
    if (ni.kind != kSpatial)
        return;
    uint32_t c[3] = {0, 0, 0};
    int d = ni.dim;
    for (uint32_t j = lane; j < it.count; j += 32) {
        BRef r = refs[it.begin + j];
        if (ref_hi(r, d) <= ni.split_clip)
            c[0]++;
        else if (ref_lo(r, d) >= ni.split_clip)
            c[1]++;
        else
            c[2]++;
    }
    for (int k = 0; k < 3; ++k) {
        uint32_t v = c[k];
        for (int o = 16; o > 0; o >>= 1)
            v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0 && v)
            atomicAdd(&ni.cls[k], v);
    }
}

__global__ void k_sp_costs(uint32_t n, NodeInfo *info)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    NodeInfo &ni = info[i];
    if (ni.kind != kSpatial)
        return;
    // n1 = rightStart (left + straddling), n2 = N - leftEnd (right + straddling) (cuda/sbvh.cu:256-258)
    ni.n1 = (int)(ni.cls[0] + ni.cls[2]);
    ni.n2 = (int)(ni.cls[1] + ni.cls[2]);
    ni.saL = surface_area(ni.ssL, ni.ssL + 3);
    ni.saR = surface_area(ni.ssR, ni.ssR + 3);
    ni.full_cost = ni.saL * (float)ni.n1 + ni.saR * (float)ni.n2;
}

// Per work item: how many references go left, right, or into the leaf pool: three arrays of n_max entries, zero past
// the level's items.
__global__ void k_count(const Item *items, const uint32_t *n_items, uint32_t n_max, const BRef *refs,
                        const NodeInfo *info, uint32_t buckets, uint32_t *counts)
{
    uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= n_max)
        return;
    uint32_t l = 0, r = 0, p = 0;
    if (w < *n_items) {
        const Item it = items[w];
        const NodeInfo &ni = info[it.node];
        for (uint32_t j = lane; j < it.count; j += 32) {
            int dst = ref_destination(refs[it.begin + j], ni, buckets);
            l += dst & 1;
            r += (dst >> 1) & 1;
            p += (dst >> 2) & 1;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        l += __shfl_xor_sync(0xffffffffu, l, o);
        r += __shfl_xor_sync(0xffffffffu, r, o);
        p += __shfl_xor_sync(0xffffffffu, p, o);
    }
    if (lane == 0) {
        counts[w] = l;
        counts[n_max + w] = r;
        counts[2 * n_max + w] = p;
    }
}

// Child reference counts of every node, from the per-item scans.  A spatial split that leaves
// one side empty trips the reference's assertion (cuda/sbvh.cu:295); such a node falls back to
// its object split and the level is recounted.
__global__ void k_child_counts(uint32_t n, const uint32_t *item_off, const uint32_t *sl, const uint32_t *sr,
                               NodeInfo *info, uint32_t *flag, uint32_t *split)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    NodeInfo &ni = info[i];
    uint32_t a = item_off[i], b = item_off[i + 1];
    ni.n_left = sl[b] - sl[a];
    ni.n_right = sr[b] - sr[a];
    if (ni.kind == kSpatial && (ni.n_left == 0 || ni.n_right == 0)) {
        ni.kind = kObject;
        atomicAdd(flag, 1u);
    }
    split[i] = ni.kind != kLeaf;
}

// What the host reads of a level: references left and right, to leaves, splits, nodes that fell back.
__global__ void k_totals(const uint32_t *sl, const uint32_t *sr, const uint32_t *spool, const uint32_t *split,
                         const uint32_t *flag, uint32_t *out)
{
    const uint32_t *src[5] = {sl, sr, spool, split, flag};
    if (threadIdx.x < 5)
        out[threadIdx.x] = *src[threadIdx.x];
}

__global__ void k_scatter(const Item *items, const uint32_t *n_items, const BRef *refs, const NodeInfo *info,
                          uint32_t buckets, const uint32_t *sl, const uint32_t *sr, const uint32_t *spool,
                          uint32_t left_total, BRef *next, uint32_t pool_base, uint32_t *pool)
{
    uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= *n_items)
        return;
    Item it = items[w];
    const NodeInfo &ni = info[it.node];
    uint32_t ol = sl[w], orr = left_total + sr[w], op = pool_base + spool[w];
    uint32_t lt_mask = (1u << lane) - 1u;
    for (uint32_t j0 = 0; j0 < it.count; j0 += 32) {
        uint32_t j = j0 + lane;
        bool valid = j < it.count;
        BRef r;
        int dst = 0;
        if (valid) {
            r = refs[it.begin + j];
            dst = ref_destination(r, ni, buckets);
        }
        uint32_t bl = __ballot_sync(0xffffffffu, dst & 1);
        uint32_t br = __ballot_sync(0xffffffffu, (dst >> 1) & 1);
        uint32_t bp = __ballot_sync(0xffffffffu, (dst >> 2) & 1);
        if (dst & 4)
            pool[op + __popc(bp & lt_mask)] = __float_as_uint(r.lo.w);
        if (dst & 1) {
            BRef x = r;
            if (dst == 3) {
                int d = ni.dim;
                if (d == 0)
                    x.hi.x = ni.split_clip;
                else if (d == 1)
                    x.hi.y = ni.split_clip;
                else
                    x.hi.z = ni.split_clip;
            }
            next[ol + __popc(bl & lt_mask)] = x;
        }
        if (dst & 2) {
            BRef x = r;
            if (dst == 3) {
                int d = ni.dim;
                if (d == 0)
                    x.lo.x = ni.split_clip;
                else if (d == 1)
                    x.lo.y = ni.split_clip;
                else
                    x.lo.z = ni.split_clip;
            }
            next[orr + __popc(br & lt_mask)] = x;
        }
        ol += __popc(bl);
        orr += __popc(br);
        op += __popc(bp);
    }
}

__global__ void k_children(const LevelNode *nodes, uint32_t n, const NodeInfo *info, const uint32_t *split_scan,
                           uint32_t n_split, const uint32_t *sl, const uint32_t *sr, const uint32_t *spool,
                           uint32_t left_total, uint32_t pool_base, uint32_t next_build_base, BuildRec *recs,
                           LevelNode *next_nodes, uint32_t *next_items)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const NodeInfo &ni = info[i];
    LevelNode nd = nodes[i];
    BuildRec &rec = recs[nd.build_id];
    if (ni.kind == kLeaf) {
        rec.leaf = 1;
        rec.left = rec.right = 0;
        rec.axis = 0;
        rec.leaf_begin = pool_base + spool[nd.first_item];
        rec.leaf_count = nd.ref_count;
        return;
    }
    uint32_t k = split_scan[i];
    LevelNode L, R;
    L.ref_begin = sl[nd.first_item];
    L.ref_count = ni.n_left;
    L.build_id = next_build_base + k;
    L.first_item = 0;
    R.ref_begin = left_total + sr[nd.first_item];
    R.ref_count = ni.n_right;
    R.build_id = next_build_base + n_split + k;
    R.first_item = 0;
    next_nodes[k] = L;
    next_nodes[n_split + k] = R;
    next_items[k] = item_count(L.ref_count);
    next_items[n_split + k] = item_count(R.ref_count);
    rec.leaf = 0;
    rec.left = L.build_id;
    rec.right = R.build_id;
    rec.axis = (uint32_t)ni.dim;
}

// ---- flattening ------------------------------------------------------------------------------

__global__ void k_subtree(BuildRec *recs, uint32_t begin, uint32_t end)
{
    uint32_t i = begin + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= end)
        return;
    BuildRec &r = recs[i];
    if (r.leaf) {
        r.size = 1;
        r.prims = r.leaf_count;
    } else {
        r.size = 1 + recs[r.left].size + recs[r.right].size;
        r.prims = recs[r.left].prims + recs[r.right].prims;
    }
}

__global__ void k_dfs(BuildRec *recs, uint32_t begin, uint32_t end)
{
    uint32_t i = begin + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= end)
        return;
    BuildRec &r = recs[i];
    if (i == 0) {
        r.dfs = 0;
        r.prim_off = 0;
    }
    if (!r.leaf) {
        BuildRec &L = recs[r.left];
        BuildRec &R = recs[r.right];
        L.dfs = r.dfs + 1;
        L.prim_off = r.prim_off;
        R.dfs = r.dfs + 1 + L.size;
        R.prim_off = r.prim_off + L.prims;
    }
}

__global__ void k_emit(const BuildRec *recs, uint32_t n, const uint32_t *pool, RefNode *out, uint32_t *prims,
                       uint32_t *interior_flag)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const BuildRec &r = recs[i];
    RefNode node;
    for (int k = 0; k < 3; ++k) {
        node.bmin[k] = r.bmin[k];
        node.bmax[k] = r.bmax[k];
    }
    node.axis = r.leaf ? 0 : r.axis;
    node.right = r.leaf ? 0 : recs[r.right].dfs;
    node.prim_offset = r.prim_off;
    out[r.dfs] = node;
    interior_flag[r.dfs] = r.leaf ? 0u : 1u;
    if (r.leaf)
        for (uint32_t k = 0; k < r.leaf_count; ++k)
            prims[r.prim_off + k] = pool[r.leaf_begin + k];
}

// Traversal layout: one 64-byte record per interior node (DFS order), children boxes inline.
// Leaf children carry their primitive count (the count the reference's traversal derives from
// primOffset differences, cuda/sbvh.cu:546-552).
// Also marks each leaf child's last primitive (kLastPrim in the w component of its second vertex,
// written after k_prim_tris), where the resumable traversal ends the leaf, and writes the leaf's box.
__global__ void k_trav(const BuildRec *recs, uint32_t n, const uint32_t *interior_scan, TravNode *trav,
                       float4 *prim_tris, float4 *leaf_box)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const BuildRec &p = recs[i];
    if (p.leaf)
        return;
    const BuildRec &L = recs[p.left];
    const BuildRec &R = recs[p.right];
    auto ref_of = [&](const BuildRec &c) { return c.leaf ? (kLeafBit | c.prim_off) : interior_scan[c.dfs]; };
    TravNode t;
    t.a = make_float4(L.bmin[0], L.bmin[1], L.bmin[2], L.bmax[0]);
    t.b = make_float4(L.bmax[1], L.bmax[2], R.bmin[0], R.bmin[1]);
    t.c = make_float4(R.bmin[2], R.bmax[0], R.bmax[1], R.bmax[2]);
    t.d = make_uint4(ref_of(L), ref_of(R), L.prims | (p.axis << 30), R.prims);
    trav[interior_scan[p.dfs]] = t;
    for (const BuildRec *c : {&L, &R}) {
        if (!c->leaf || !c->prims)
            continue;
        prim_tris[3 * (size_t)(c->prim_off + c->prims - 1) + 1].w = __uint_as_float(kLastPrim);
        leaf_box[2 * (size_t)c->prim_off] = make_float4(c->bmin[0], c->bmin[1], c->bmin[2], 0.0f);
        leaf_box[2 * (size_t)c->prim_off + 1] = make_float4(c->bmax[0], c->bmax[1], c->bmax[2], 0.0f);
    }
}

// recs[0] is the root: the box of the leaf when the whole tree is one.
__global__ void k_prim_tris(const uint32_t *prims, uint32_t n_prims, const float *verts, const uint32_t *idx,
                            const BuildRec *recs, float4 *out, float4 *leaf_box)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_prims)
        return;
    uint32_t t = prims[i];
    float4 v[3];
    for (int k = 0; k < 3; ++k) {
        uint32_t vi = idx[3 * t + k];
        v[k] = make_float4(verts[3 * vi], verts[3 * vi + 1], verts[3 * vi + 2], 0.0f);
    }
    v[0].w = __uint_as_float(t);
    if (i + 1 == n_prims) // ends the last leaf (the whole tree may be one)
        v[1].w = __uint_as_float(kLastPrim);
    if (i == 0) {
        leaf_box[0] = make_float4(recs[0].bmin[0], recs[0].bmin[1], recs[0].bmin[2], 0.0f);
        leaf_box[1] = make_float4(recs[0].bmax[0], recs[0].bmax[1], recs[0].bmax[2], 0.0f);
    }
    out[3 * i + 0] = v[0];
    out[3 * i + 1] = v[1];
    out[3 * i + 2] = v[2];
}

inline unsigned grid_for(uint64_t n, unsigned block) { return (unsigned)((n + block - 1) / block); }

} // namespace

// One SBVH over the triangles [tri_begin, tri_begin + n_tris) of the global arrays; primitive
// references keep global triangle indices.
struct RangeOut
{
    DevBuf<RefNode> ref_nodes;
    DevBuf<uint32_t> prims;
    DevBuf<TravNode> trav;
    DevBuf<float4> prim_tris, leaf_box;
    uint32_t n_nodes = 0, n_prims = 0, n_trav = 0, n_levels = 0;
    float bound[6] = {0, 0, 0, 0, 0, 0};
};

// `done` (may be null) is recorded on the stream after the last build kernel, before the scratch
// buffers are released.
// Scratch of build_range, kept by the context between builds: growing these buffers level by level
// costs a few hundred allocations per build (each replaced buffer's cudaFree waits for the
// device), so a context reuses them; they grow to the largest tree built on it and are freed with
// the context.
struct BuildScratch
{
    DevBuf<BRef> refs_a, refs_b;
    DevBuf<LevelNode> nodes_a, nodes_b;
    DevBuf<Item> items;
    DevBuf<NodeInfo> info;
    DevBuf<uint32_t> bnd, obj, sp, item_cnt, item_off, counts, count_scan, split_flag, split_scan, pool, flag, totals;
    DevBuf<uint32_t> interior_flag, interior_scan;
    DevBuf<uint32_t> wide_binary, wide_child, wide_level;
    DevBuf<float> wide_bound;
    DevBuf<BuildRec> recs;
    ScanScratch scan;
    uint32_t *h_totals = nullptr; // pinned
    ~BuildScratch()
    {
        if (h_totals)
            cudaFreeHost(h_totals);
    }
};

static BuildScratch &build_scratch(ks_context *ctx)
{
    if (!ctx->build_cache)
        ctx->build_cache = std::make_shared<BuildScratch>();
    return *static_cast<BuildScratch *>(ctx->build_cache.get());
}

static ks_status build_range(ks_context *ctx, const float *verts, const uint32_t *indices, uint32_t tri_begin,
                             uint32_t n_tris, const Params &p, RangeOut &out, cudaEvent_t done = nullptr)
{
    cudaStream_t st = ctx->stream;
    BuildScratch &bs = build_scratch(ctx);
    auto &refs_a = bs.refs_a, &refs_b = bs.refs_b;
    auto &nodes_a = bs.nodes_a, &nodes_b = bs.nodes_b;
    auto &items = bs.items;
    auto &info = bs.info;
    auto &bnd = bs.bnd, &obj = bs.obj, &sp = bs.sp, &item_cnt = bs.item_cnt, &item_off = bs.item_off;
    auto &counts = bs.counts, &count_scan = bs.count_scan;
    auto &split_flag = bs.split_flag, &split_scan = bs.split_scan, &pool = bs.pool, &flag = bs.flag;
    auto &recs = bs.recs;
    auto &scan = bs.scan;

    size_t ref_cap = (size_t)n_tris * 2 + 1024;
    KS_CUDA_TRY(ctx, refs_a.reserve(ref_cap));
    KS_CUDA_TRY(ctx, refs_b.reserve(ref_cap));
    KS_CUDA_TRY(ctx, pool.reserve(ref_cap));
    size_t rec_cap = (size_t)n_tris * 4 + 1024;
    KS_CUDA_TRY(ctx, recs.reserve(rec_cap));
    KS_CUDA_TRY(ctx, flag.reserve(1));
    KS_CUDA_TRY(ctx, bs.totals.reserve(5));
    if (!bs.h_totals)
        KS_CUDA_TRY(ctx, cudaMallocHost((void **)&bs.h_totals, sizeof(uint32_t) * 5));

    k_init_refs<<<grid_for(n_tris, 256), 256, 0, st>>>(verts, indices, tri_begin, n_tris, refs_a.ptr);
    LevelNode root{0, n_tris, 0, 0};
    KS_CUDA_TRY(ctx, nodes_a.reserve(1));
    KS_CUDA_TRY(ctx, cudaMemcpyAsync(nodes_a.ptr, &root, sizeof(root), cudaMemcpyHostToDevice, st));
    const uint32_t root_items = (n_tris + kChunk - 1) / kChunk;
    KS_CUDA_TRY(ctx, item_cnt.reserve(1));
    KS_CUDA_TRY(ctx, cudaMemcpyAsync(item_cnt.ptr, &root_items, sizeof(uint32_t), cudaMemcpyHostToDevice, st));

    uint32_t n_active = 1, n_refs = n_tris, build_base = 0, pool_used = 0;
    std::vector<uint32_t> level_begin;
    BRef *cur = refs_a.ptr, *nxt = refs_b.ptr;
    DevBuf<BRef> *cur_buf = &refs_a, *nxt_buf = &refs_b;
    DevBuf<LevelNode> *cur_nodes = &nodes_a, *nxt_nodes = &nodes_b;
    int level = 0;
    while (n_active > 0) {
        level_begin.push_back(build_base);
        if ((size_t)build_base + n_active > rec_cap)
            return fail(ctx, KS_ERR_OUT_OF_MEMORY, "sbvh build: node record capacity exceeded");
        // work items (the last kernel of the level before counted them); the host knows no more than their bound
        KS_CUDA_TRY(ctx, item_off.reserve(n_active + 1));
        KS_CUDA_TRY(ctx, exclusive_scan(item_cnt.ptr, item_off.ptr, n_active, scan, st));
        const uint32_t max_items = n_active + n_refs / kChunk;
        const uint32_t *n_items = item_off.ptr + n_active;
        KS_CUDA_TRY(ctx, items.reserve(max_items));
        KS_CUDA_TRY(ctx, info.reserve(n_active));
        KS_CUDA_TRY(ctx, bnd.reserve((size_t)n_active * 12));
        KS_CUDA_TRY(ctx, obj.reserve((size_t)n_active * p.buckets * 7));
        KS_CUDA_TRY(ctx, sp.reserve((size_t)n_active * p.buckets * 8));
        const unsigned wgrid = grid_for((uint64_t)max_items * 32, 256);
        const unsigned wgrid8 = grid_for(max_items, kWarpsPerBlock);
        const unsigned eval_grid = grid_for((uint64_t)n_active * kEvalLanes, 128);
        k_items_fill<<<eval_grid, 128, 0, st>>>(cur_nodes->ptr, n_active, item_off.ptr, items.ptr, bnd.ptr, obj.ptr, sp.ptr,
                                                info.ptr, p.buckets);
        k_bounds<<<wgrid, 256, 0, st>>>(items.ptr, n_items, cur, bnd.ptr);
        k_prep<<<grid_for(n_active, 128), 128, 0, st>>>(cur_nodes->ptr, n_active, bnd.ptr, info.ptr, recs.ptr + 0,
                                                        level == 0);
        k_obj_bins<<<wgrid8, kWarpsPerBlock * 32, 0, st>>>(items.ptr, n_items, cur, info.ptr, p.buckets, obj.ptr);
        k_obj_eval<<<eval_grid, 128, 0, st>>>(n_active, obj.ptr, info.ptr, p);
        k_sp_bins<<<wgrid8, kWarpsPerBlock * 32, 0, st>>>(items.ptr, n_items, cur, info.ptr, p.buckets, sp.ptr);
        k_decide<<<eval_grid, 128, 0, st>>>(cur_nodes->ptr, n_active, sp.ptr, info.ptr, p);
        k_sp_classes<<<wgrid, 256, 0, st>>>(items.ptr, n_items, cur, info.ptr);
        k_sp_costs<<<grid_for(n_active, 128), 128, 0, st>>>(n_active, info.ptr);
        KS_CUDA_TRY(ctx, counts.reserve((size_t)max_items * 3));
        KS_CUDA_TRY(ctx, count_scan.reserve(((size_t)max_items + 1) * 3));
        KS_CUDA_TRY(ctx, split_flag.reserve(n_active));
        KS_CUDA_TRY(ctx, split_scan.reserve(n_active + 1));
        const uint32_t *sl = count_scan.ptr, *sr = sl + max_items + 1, *spool = sr + max_items + 1;
        for (int pass = 0;; ++pass) {
            k_count<<<wgrid, 256, 0, st>>>(items.ptr, n_items, max_items, cur, info.ptr, p.buckets, counts.ptr);
            KS_CUDA_TRY(ctx, exclusive_scan(counts.ptr, count_scan.ptr, max_items, scan, st, 3));
            KS_CUDA_TRY(ctx, cudaMemsetAsync(flag.ptr, 0, 4, st));
            k_child_counts<<<grid_for(n_active, 128), 128, 0, st>>>(n_active, item_off.ptr, sl, sr, info.ptr, flag.ptr,
                                                                    split_flag.ptr);
            KS_CUDA_TRY(ctx, exclusive_scan(split_flag.ptr, split_scan.ptr, n_active, scan, st));
            k_totals<<<1, 32, 0, st>>>(sl + max_items, sr + max_items, spool + max_items, split_scan.ptr + n_active,
                                       flag.ptr, bs.totals.ptr);
            KS_CUDA_TRY(ctx, cudaMemcpyAsync(bs.h_totals, bs.totals.ptr, sizeof(uint32_t) * 5, cudaMemcpyDeviceToHost, st));
            KS_CUDA_TRY(ctx, cudaStreamSynchronize(st));
            if (!bs.h_totals[4])
                break;
            if (pass > 0)
                return fail(ctx, KS_ERR_INVALID_ARGUMENT, "sbvh build: degenerate split could not be resolved");
        }
        const uint32_t left_total = bs.h_totals[0], right_total = bs.h_totals[1], leaf_total = bs.h_totals[2];
        const uint32_t n_split = bs.h_totals[3];
        size_t next_refs = (size_t)left_total + right_total;
        if (next_refs > nxt_buf->count) {
            // grow the next-level buffer (contents are rewritten by the scatter)
            KS_CUDA_TRY(ctx, nxt_buf->alloc(next_refs + next_refs / 2));
            nxt = nxt_buf->ptr;
        }
        if ((size_t)pool_used + leaf_total > pool.count)
            return fail(ctx, KS_ERR_OUT_OF_MEMORY, "sbvh build: leaf pool capacity exceeded");
        k_scatter<<<wgrid, 256, 0, st>>>(items.ptr, n_items, cur, info.ptr, p.buckets, sl, sr, spool, left_total, nxt, pool_used, pool.ptr);
        KS_CUDA_TRY(ctx, nxt_nodes->reserve((size_t)2 * n_split + 1));
        KS_CUDA_TRY(ctx, item_cnt.reserve((size_t)2 * n_split + 1));
        uint32_t next_build_base = build_base + n_active;
        k_children<<<grid_for(n_active, 128), 128, 0, st>>>(cur_nodes->ptr, n_active, info.ptr, split_scan.ptr, n_split,
                                                            sl, sr, spool, left_total, pool_used, next_build_base,
                                                            recs.ptr, nxt_nodes->ptr, item_cnt.ptr);
        // the level's node list is read by k_children above; keep the swap after it
        KS_CUDA_TRY(ctx, cudaGetLastError());
        pool_used += leaf_total;
        build_base = next_build_base;
        n_active = 2 * n_split;
        n_refs = (uint32_t)next_refs;
        std::swap(cur, nxt);
        std::swap(cur_buf, nxt_buf);
        std::swap(cur_nodes, nxt_nodes);
        ++level;
        if ((uint32_t)level > (ctx->limits.sbvh_max_levels ? ctx->limits.sbvh_max_levels : 4096u))
            return fail(ctx, KS_ERR_WATCHDOG, "sbvh build: level limit reached");
    }
    const uint32_t n_nodes = build_base;
    level_begin.push_back(build_base);
    // subtree sizes bottom-up, DFS numbering top-down
    for (int l = (int)level_begin.size() - 2; l >= 0; --l) {
        uint32_t b = level_begin[l], e = level_begin[l + 1];
        k_subtree<<<grid_for(e - b, 256), 256, 0, st>>>(recs.ptr, b, e);
    }
    for (size_t l = 0; l + 1 < level_begin.size(); ++l) {
        uint32_t b = level_begin[l], e = level_begin[l + 1];
        k_dfs<<<grid_for(e - b, 256), 256, 0, st>>>(recs.ptr, b, e);
    }
    KS_CUDA_TRY(ctx, out.ref_nodes.alloc(n_nodes));
    KS_CUDA_TRY(ctx, out.prims.alloc(pool_used));
    auto &interior_flag = bs.interior_flag, &interior_scan = bs.interior_scan;
    KS_CUDA_TRY(ctx, interior_flag.reserve(n_nodes));
    KS_CUDA_TRY(ctx, interior_scan.reserve(n_nodes + 1));
    k_emit<<<grid_for(n_nodes, 256), 256, 0, st>>>(recs.ptr, n_nodes, pool.ptr, out.ref_nodes.ptr, out.prims.ptr,
                                                   interior_flag.ptr);
    KS_CUDA_TRY(ctx, exclusive_scan(interior_flag.ptr, interior_scan.ptr, n_nodes, scan, st));
    uint32_t n_trav = 0;
    KS_CUDA_TRY(ctx, cudaMemcpyAsync(&n_trav, interior_scan.ptr + n_nodes, 4, cudaMemcpyDeviceToHost, st));
    KS_CUDA_TRY(ctx, cudaStreamSynchronize(st));
    KS_CUDA_TRY(ctx, out.trav.alloc(n_trav > 0 ? n_trav : 1));
    // records past the end are read (not used) with the last leaf, by the lanes of a group (ks_traverse4.cuh)
    KS_CUDA_TRY(ctx, out.prim_tris.alloc(((size_t)pool_used + kPrimPad) * 3));
    KS_CUDA_TRY(ctx, cudaMemsetAsync(out.prim_tris.ptr + 3 * (size_t)pool_used, 0, sizeof(float4) * 3 * kPrimPad, st));
    KS_CUDA_TRY(ctx, out.leaf_box.alloc((size_t)pool_used * 2));
    k_prim_tris<<<grid_for(pool_used, 256), 256, 0, st>>>(out.prims.ptr, pool_used, verts, indices, recs.ptr,
                                                          out.prim_tris.ptr, out.leaf_box.ptr);
    k_trav<<<grid_for(n_nodes, 256), 256, 0, st>>>(recs.ptr, n_nodes, interior_scan.ptr, out.trav.ptr,
                                                   out.prim_tris.ptr, out.leaf_box.ptr);
    KS_CUDA_TRY(ctx, cudaGetLastError());
    if (done)
        KS_CUDA_TRY(ctx, cudaEventRecord(done, st));
    RefNode root_node;
    KS_CUDA_TRY(ctx, cudaMemcpyAsync(&root_node, out.ref_nodes.ptr, sizeof(RefNode), cudaMemcpyDeviceToHost, st));
    KS_CUDA_TRY(ctx, cudaStreamSynchronize(st));
    for (int k = 0; k < 3; ++k) {
        out.bound[k] = root_node.bmin[k];
        out.bound[3 + k] = root_node.bmax[k];
    }
    out.n_nodes = n_nodes;
    out.n_prims = pool_used;
    out.n_trav = n_trav;
    out.n_levels = (uint32_t)level_begin.size() - 1;
    return KS_OK;
}

// ---- the renderer's 4-wide view (Wide4Node) ----------------------------------------------------
// Built from the binary nodes level by level.  A wide node opens its binary node: two children, then
// the interior child of the largest area replaced by its own two, until there are 4 or only leaves
// (`even`: each interior child replaced once instead).
// k_wide4_alloc finds each node's interior children and gives them nodes of the next level (one atomic
// per node); k_wide4_fill then writes all nodes at once, opening each the same way again.
struct Opened4
{
    float lo[4][3], hi[4][3];
    uint32_t ref[4];
    int n;
};

__device__ __forceinline__ void open4(const TravNode *__restrict__ nodes, uint32_t ref, bool even, Opened4 &c)
{
    float area[4]; // of interior children
    auto put = [&](int at, const TravNode &t, int side) {
        const float4 A = t.a, B = t.b, C = t.c;
        const float l0[3] = {A.x, A.y, A.z}, h0[3] = {A.w, B.x, B.y};
        const float l1[3] = {B.z, B.w, C.x}, h1[3] = {C.y, C.z, C.w};
        for (int a = 0; a < 3; ++a) {
            c.lo[at][a] = side ? l1[a] : l0[a];
            c.hi[at][a] = side ? h1[a] : h0[a];
        }
        c.ref[at] = side ? t.d.y : t.d.x;
        const float x = c.hi[at][0] - c.lo[at][0], y = c.hi[at][1] - c.lo[at][1], z = c.hi[at][2] - c.lo[at][2];
        area[at] = x * y + y * z + z * x;
    };
    {
        const TravNode t = nodes[ref];
        put(0, t, 0);
        put(1, t, 1);
    }
    c.n = 2;
    int next = 0; // even: the child to replace
    while (c.n < 4) {
        int best = -1;
        if (even) {
            while (next < c.n && (c.ref[next] & kLeafBit))
                ++next;
            best = next < c.n ? next : -1;
            next += 2; // past what takes its place
        } else {
            for (int k = 0; k < c.n; ++k)
                if (!(c.ref[k] & kLeafBit) && (best < 0 || area[k] > area[best]))
                    best = k;
        }
        if (best < 0)
            break;
        const TravNode t = nodes[c.ref[best]];
        for (int k = c.n; k > best + 1; --k) { // the two children take their parent's place
            for (int a = 0; a < 3; ++a) {
                c.lo[k][a] = c.lo[k - 1][a];
                c.hi[k][a] = c.hi[k - 1][a];
            }
            c.ref[k] = c.ref[k - 1];
            area[k] = area[k - 1];
        }
        put(best, t, 0);
        put(best + 1, t, 1);
        ++c.n;
    }
}

// Level `level` of the view: binary[i] is wide node i's binary node (kLeafBit: a tree that is one
// leaf), level_n[l] the nodes of level l (complete below `level` + 1), child[i] the first child.
__global__ void k_wide4_alloc(const TravNode *__restrict__ nodes, uint32_t level, bool even, uint32_t *level_n,
                              uint32_t *binary, uint32_t *child)
{
    uint32_t begin = 0;
    for (uint32_t l = 0; l < level; ++l)
        begin += level_n[l];
    const uint32_t n = level_n[level], next = begin + n;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t ref = binary[begin + i];
        if (ref & kLeafBit) {
            child[begin + i] = 0;
            continue;
        }
        Opened4 c;
        open4(nodes, ref, even, c);
        uint32_t inner = 0;
        for (int k = 0; k < c.n; ++k)
            inner += (c.ref[k] & kLeafBit) ? 0u : 1u;
        uint32_t at = inner ? next + atomicAdd(&level_n[level + 1], inner) : 0u;
        child[begin + i] = at;
        for (int k = 0; k < c.n; ++k)
            if (!(c.ref[k] & kLeafBit))
                binary[at++] = c.ref[k];
    }
}

// root_bound: the root's box, read when the tree is one leaf.
__global__ void k_wide4_fill(const TravNode *__restrict__ nodes, uint32_t n, bool even, const uint32_t *__restrict__ binary,
                             const uint32_t *__restrict__ child, const float *__restrict__ root_bound, Wide4Node *out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const uint32_t ref = binary[i];
    Opened4 c;
    if (ref & kLeafBit) {
        c.n = 1;
        for (int a = 0; a < 3; ++a) {
            c.lo[0][a] = root_bound[a];
            c.hi[0][a] = root_bound[3 + a];
        }
        c.ref[0] = ref;
    } else {
        open4(nodes, ref, even, c);
    }
    Wide4Node w;
    float *plane = reinterpret_cast<float *>(w.plane);
    uint32_t next = child[i];
    for (int k = 0; k < 4; ++k) {
        for (int a = 0; a < 3; ++a) {
            plane[8 * a + k] = k < c.n ? c.lo[k][a] : kInf;
            plane[8 * a + 4 + k] = k < c.n ? c.hi[k][a] : -kInf;
        }
        w.ref[k] = k >= c.n ? kLeafBit : (c.ref[k] & kLeafBit) ? c.ref[k] : next++;
        w.pad[k] = 0;
    }
    out[i] = w;
}

// The view of the tree over `nodes` whose root is root_ref with box root_bound (6 floats), into out (node 0:
// the root).  Launches kWide4Chunk levels between two looks at the counts (a level without nodes costs its
// launch, some 2 us); max_levels: levels of the binary tree, at most kMaxBinaryLevels, and no fewer than the view's.
static ks_status build_wide4(ks_context *ctx, BuildScratch &bs, const TravNode *nodes, uint32_t n_trav, uint32_t root_ref,
                             const float *root_bound, uint32_t max_levels, DevBuf<Wide4Node> &out)
{
    constexpr uint32_t kWide4Chunk = 16;
    cudaStream_t st = ctx->stream;
    const uint32_t levels = std::max(max_levels, kMaxWideLevels) + kWide4Chunk + 1, one = 1;
    KS_CUDA_TRY(ctx, bs.wide_binary.reserve((size_t)n_trav + 1));
    KS_CUDA_TRY(ctx, bs.wide_child.reserve((size_t)n_trav + 1));
    KS_CUDA_TRY(ctx, bs.wide_level.reserve(levels));
    KS_CUDA_TRY(ctx, bs.wide_bound.reserve(6));
    KS_CUDA_TRY(ctx, cudaMemcpyAsync(bs.wide_binary.ptr, &root_ref, sizeof(uint32_t), cudaMemcpyHostToDevice, st));
    KS_CUDA_TRY(ctx, cudaMemcpyAsync(bs.wide_bound.ptr, root_bound, sizeof(float) * 6, cudaMemcpyHostToDevice, st));
    std::vector<uint32_t> count;
    bool even = false;
    while (true) {
        count.assign(levels, 0);
        count[0] = 1;
        KS_CUDA_TRY(ctx, cudaMemsetAsync(bs.wide_level.ptr, 0, sizeof(uint32_t) * levels, st));
        KS_CUDA_TRY(ctx, cudaMemcpyAsync(bs.wide_level.ptr, &one, sizeof(uint32_t), cudaMemcpyHostToDevice, st));
        uint32_t done = 0;
        while (done < levels && count[done]) {
            const uint32_t end = std::min(done + kWide4Chunk, max_levels);
            if (end == done)
                return fail(ctx, KS_ERR_WATCHDOG, "sbvh build: 4-wide level limit reached");
            for (; done < end; ++done)
                k_wide4_alloc<<<(unsigned)ctx->sm_count * 4, 128, 0, st>>>(nodes, done, even, bs.wide_level.ptr,
                                                                           bs.wide_binary.ptr, bs.wide_child.ptr);
            KS_CUDA_TRY(ctx, cudaMemcpyAsync(count.data(), bs.wide_level.ptr, sizeof(uint32_t) * levels,
                                             cudaMemcpyDeviceToHost, st));
            KS_CUDA_TRY(ctx, cudaStreamSynchronize(st));
        }
        if (count[kMaxWideLevels] == 0)
            break;
        if (even)
            return fail(ctx, KS_ERR_WATCHDOG, "sbvh build: 4-wide levels exceed the traversal stack");
        even = true;
    }
    uint32_t n = 0;
    for (uint32_t c : count)
        n += c;
    KS_CUDA_TRY(ctx, out.alloc(n));
    k_wide4_fill<<<grid_for(n, 128), 128, 0, st>>>(nodes, n, even, bs.wide_binary.ptr, bs.wide_child.ptr,
                                                   bs.wide_bound.ptr, out.ptr);
    KS_CUDA_TRY(ctx, cudaGetLastError());
    return KS_OK;
}

// The exact traversal's 4-wide steps: wide node i holds the children of interior node i, each interior child
// replaced by its own two children (2 to 4 slots, in order).
__global__ void k_widen(const TravNode *nodes, uint32_t n, WideNode *wide)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    WideNode w;
    for (int a = 0; a < 3; ++a) {
        w.lo[a] = make_float4(kInf, kInf, kInf, kInf); // unused slots: an empty box, never hit
        w.hi[a] = make_float4(-kInf, -kInf, -kInf, -kInf);
    }
    w.ref = make_uint4(kLeafBit, kLeafBit, kLeafBit, kLeafBit);
    w.pad = make_uint4(0, 0, 0, 0);
    float *lo = reinterpret_cast<float *>(w.lo), *hi = reinterpret_cast<float *>(w.hi);
    uint32_t *ref = reinterpret_cast<uint32_t *>(&w.ref);
    int m = 0;
    auto put = [&](const TravNode &nd, int side) {
        const float4 A = nd.a, B = nd.b, C = nd.c;
        const float l0[3] = {A.x, A.y, A.z}, h0[3] = {A.w, B.x, B.y};
        const float l1[3] = {B.z, B.w, C.x}, h1[3] = {C.y, C.z, C.w};
        for (int a = 0; a < 3; ++a) {
            lo[4 * a + m] = side ? l1[a] : l0[a];
            hi[4 * a + m] = side ? h1[a] : h0[a];
        }
        ref[m] = side ? nd.d.y : nd.d.x;
        ++m;
    };
    const TravNode nd = nodes[i];
    for (int side = 0; side < 2; ++side) {
        const uint32_t r = side ? nd.d.y : nd.d.x;
        if (r & kLeafBit) {
            put(nd, side);
        } else {
            const TravNode c = nodes[r];
            put(c, 0);
            put(c, 1);
        }
    }
    wide[i] = w;
}

cudaError_t make_wide_steps(ks_scene *scene)
{
    const cudaError_t e = scene->wide_steps.alloc(scene->n_trav > 0 ? scene->n_trav : 1);
    if (e != cudaSuccess || scene->n_trav == 0)
        return e;
    k_widen<<<grid_for(scene->n_trav, 256), 256, 0, scene->ctx->stream>>>(scene->trav_nodes.ptr, scene->n_trav,
                                                                          scene->wide_steps.ptr);
    return cudaGetLastError();
}

// BLAS concatenation: interior refs move by the node base, leaf refs by the slot base.
__global__ void k_offset_trav(const TravNode *src, uint32_t n, uint32_t node_base, uint32_t slot_base, TravNode *dst)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    TravNode t = src[i];
    t.d.x = (t.d.x & kLeafBit) ? (kLeafBit | ((t.d.x & ~kLeafBit) + slot_base)) : t.d.x + node_base;
    t.d.y = (t.d.y & kLeafBit) ? (kLeafBit | ((t.d.y & ~kLeafBit) + slot_base)) : t.d.y + node_base;
    dst[i] = t;
}

// ---- TLAS over instance boxes (host, binned SAH; leaves of at most 2 instances) ---------------
struct InstBox
{
    float lo[3], hi[3], c[3];
    uint32_t id;
};

struct TlasBuilder
{
    std::vector<InstBox> items;
    std::vector<TravNode> nodes;

    static void unite(float *lo, float *hi, const InstBox &b)
    {
        for (int k = 0; k < 3; ++k) {
            lo[k] = std::min(lo[k], b.lo[k]);
            hi[k] = std::max(hi[k], b.hi[k]);
        }
    }
    static float area(const float *lo, const float *hi)
    {
        float dx = hi[0] - lo[0], dy = hi[1] - lo[1], dz = hi[2] - lo[2];
        return 2.0f * (dx * dy + dy * dz + dz * dx);
    }
    // returns (ref, count); box of the subtree in lo/hi
    std::pair<uint32_t, uint32_t> build(uint32_t b, uint32_t e, float *lo, float *hi)
    {
        for (int k = 0; k < 3; ++k) {
            lo[k] = kInf;
            hi[k] = -kInf;
        }
        for (uint32_t i = b; i < e; ++i)
            unite(lo, hi, items[i]);
        if (e - b <= 2)
            return {kLeafBit | b, e - b};
        float clo[3] = {kInf, kInf, kInf}, chi[3] = {-kInf, -kInf, -kInf};
        for (uint32_t i = b; i < e; ++i)
            for (int k = 0; k < 3; ++k) {
                clo[k] = std::min(clo[k], items[i].c[k]);
                chi[k] = std::max(chi[k], items[i].c[k]);
            }
        int axis = 0;
        for (int k = 1; k < 3; ++k)
            if (chi[k] - clo[k] > chi[axis] - clo[axis])
                axis = k;
        uint32_t mid = (b + e) / 2;
        float ext = chi[axis] - clo[axis];
        if (ext > 0.0f) {
            constexpr int kBins = 12;
            float blo[kBins][3], bhi[kBins][3];
            uint32_t bcnt[kBins] = {};
            for (int q = 0; q < kBins; ++q)
                for (int k = 0; k < 3; ++k) {
                    blo[q][k] = kInf;
                    bhi[q][k] = -kInf;
                }
            auto bin_of = [&](const InstBox &x) {
                int q = (int)((x.c[axis] - clo[axis]) / ext * kBins);
                return std::min(std::max(q, 0), kBins - 1);
            };
            for (uint32_t i = b; i < e; ++i) {
                int q = bin_of(items[i]);
                ++bcnt[q];
                unite(blo[q], bhi[q], items[i]);
            }
            float best = kInf;
            int best_q = -1;
            for (int q = 1; q < kBins; ++q) {
                float llo[3] = {kInf, kInf, kInf}, lhi[3] = {-kInf, -kInf, -kInf};
                float rlo[3] = {kInf, kInf, kInf}, rhi[3] = {-kInf, -kInf, -kInf};
                uint32_t nl = 0, nr = 0;
                for (int j = 0; j < kBins; ++j) {
                    if (!bcnt[j])
                        continue;
                    float *L = j < q ? llo : rlo, *H = j < q ? lhi : rhi;
                    for (int k = 0; k < 3; ++k) {
                        L[k] = std::min(L[k], blo[j][k]);
                        H[k] = std::max(H[k], bhi[j][k]);
                    }
                    (j < q ? nl : nr) += bcnt[j];
                }
                if (!nl || !nr)
                    continue;
                float cost = area(llo, lhi) * nl + area(rlo, rhi) * nr;
                if (cost < best) {
                    best = cost;
                    best_q = q;
                }
            }
            if (best_q > 0) {
                auto it = std::partition(items.begin() + b, items.begin() + e,
                                         [&](const InstBox &x) { return bin_of(x) < best_q; });
                mid = (uint32_t)(it - items.begin());
            }
        }
        if (mid == b || mid == e) {
            mid = (b + e) / 2;
            std::nth_element(items.begin() + b, items.begin() + mid, items.begin() + e,
                             [&](const InstBox &x, const InstBox &y) { return x.c[axis] < y.c[axis]; });
        }
        uint32_t me = (uint32_t)nodes.size();
        nodes.emplace_back();
        float llo[3], lhi[3], rlo[3], rhi[3];
        auto L = build(b, mid, llo, lhi);
        auto R = build(mid, e, rlo, rhi);
        TravNode &n = nodes[me];
        n.a = make_float4(llo[0], llo[1], llo[2], lhi[0]);
        n.b = make_float4(lhi[1], lhi[2], rlo[0], rlo[1]);
        n.c = make_float4(rlo[2], rhi[0], rhi[1], rhi[2]);
        n.d = make_uint4(L.first, R.first, L.second | ((uint32_t)axis << 30), R.second);
        return {me, 0u};
    }
};

static ks_status build_instanced(ks_scene *scene, const Params &p)
{
    ks_context *ctx = scene->ctx;
    cudaStream_t st = ctx->stream;
    const SceneHost &h = scene->host;
    const uint32_t n_protos = scene->n_protos;
    std::vector<RangeOut> blas(n_protos);
    uint32_t total_trav = 0, total_slots = 0;
    for (uint32_t q = 0; q < n_protos; ++q) {
        uint32_t b = h.proto_tri_begin[q], n = h.proto_tri_end[q] - b;
        ks_status s = build_range(ctx, scene->verts.ptr, scene->indices.ptr, b, n, p, blas[q]);
        if (s != KS_OK)
            return s;
        total_trav += blas[q].n_trav;
        total_slots += blas[q].n_prims;
    }
    KS_CUDA_TRY(ctx, scene->trav_nodes.alloc(total_trav > 0 ? total_trav : 1));
    KS_CUDA_TRY(ctx, scene->prim_tris.alloc((size_t)total_slots * 3));
    std::vector<uint4> roots(n_protos);
    std::vector<float> pbound(6 * (size_t)n_protos);
    uint32_t node_base = 0, slot_base = 0;
    for (uint32_t q = 0; q < n_protos; ++q) {
        const RangeOut &r = blas[q];
        if (r.n_trav)
            k_offset_trav<<<grid_for(r.n_trav, 256), 256, 0, st>>>(r.trav.ptr, r.n_trav, node_base, slot_base,
                                                                  scene->trav_nodes.ptr + node_base);
        KS_CUDA_TRY(ctx, cudaMemcpyAsync(scene->prim_tris.ptr + 3 * (size_t)slot_base, r.prim_tris.ptr,
                                         sizeof(float4) * 3 * (size_t)r.n_prims, cudaMemcpyDeviceToDevice, st));
        roots[q] = make_uint4(r.n_trav ? node_base : (kLeafBit | slot_base), r.n_prims, 0, 0);
        std::memcpy(&pbound[6 * (size_t)q], r.bound, sizeof(r.bound));
        node_base += r.n_trav;
        slot_base += r.n_prims;
    }
    KS_CUDA_TRY(ctx, cudaGetLastError());
    // 4-wide steps over the concatenated BLAS nodes (their refs are already global)
    KS_CUDA_TRY(ctx, scene->wide_steps.alloc(total_trav > 0 ? total_trav : 1));
    if (total_trav > 0)
        k_widen<<<grid_for(total_trav, 256), 256, 0, st>>>(scene->trav_nodes.ptr, total_trav, scene->wide_steps.ptr);
    // instance boxes: the 8 corners of the prototype box, transformed, padded by a relative epsilon
    TlasBuilder tb;
    for (uint32_t i = 0; i < scene->n_instances; ++i) {
        const float *xf = &h.inst_xf[12 * (size_t)i];
        const float *pb = &pbound[6 * (size_t)h.inst_proto[i]];
        InstBox ib{{kInf, kInf, kInf}, {-kInf, -kInf, -kInf}, {0, 0, 0}, i};
        for (int c = 0; c < 8; ++c) {
            f3 corner = mk(pb[(c & 1) ? 3 : 0], pb[(c & 2) ? 4 : 1], pb[(c & 4) ? 5 : 2]);
            f3 w = xf_point(xf, corner);
            float wv[3] = {w.x, w.y, w.z};
            for (int k = 0; k < 3; ++k) {
                ib.lo[k] = std::min(ib.lo[k], wv[k]);
                ib.hi[k] = std::max(ib.hi[k], wv[k]);
            }
        }
        for (int k = 0; k < 3; ++k) {
            float pad = 1e-6f * (ib.hi[k] - ib.lo[k] + std::fabs(ib.lo[k]) + std::fabs(ib.hi[k])) + 1e-30f;
            ib.lo[k] -= pad;
            ib.hi[k] += pad;
            ib.c[k] = 0.5f * (ib.lo[k] + ib.hi[k]);
        }
        tb.items.push_back(ib);
    }
    float lo[3], hi[3];
    auto root = tb.build(0, (uint32_t)tb.items.size(), lo, hi);
    std::vector<uint32_t> items(tb.items.size());
    for (size_t k = 0; k < items.size(); ++k)
        items[k] = tb.items[k].id;
    KS_CUDA_TRY(ctx, scene->tlas_nodes.alloc(std::max<size_t>(tb.nodes.size(), 1)));
    KS_CUDA_TRY(ctx, scene->tlas_items.alloc(items.size()));
    KS_CUDA_TRY(ctx, scene->proto_root.alloc(n_protos));
    KS_CUDA_TRY(ctx, scene->proto_bound.alloc(pbound.size()));
    if (!tb.nodes.empty())
        KS_CUDA_TRY(ctx, cudaMemcpyAsync(scene->tlas_nodes.ptr, tb.nodes.data(), sizeof(TravNode) * tb.nodes.size(),
                                         cudaMemcpyHostToDevice, st));
    KS_CUDA_TRY(ctx, cudaMemcpyAsync(scene->tlas_items.ptr, items.data(), sizeof(uint32_t) * items.size(),
                                     cudaMemcpyHostToDevice, st));
    KS_CUDA_TRY(ctx, cudaMemcpyAsync(scene->proto_root.ptr, roots.data(), sizeof(uint4) * roots.size(),
                                     cudaMemcpyHostToDevice, st));
    KS_CUDA_TRY(ctx, cudaMemcpyAsync(scene->proto_bound.ptr, pbound.data(), sizeof(float) * pbound.size(),
                                     cudaMemcpyHostToDevice, st));
    KS_CUDA_TRY(ctx, cudaStreamSynchronize(st));
    scene->tlas_root_ref = root.first;
    scene->tlas_root_count = root.second;
    for (int k = 0; k < 3; ++k) {
        scene->scene_bound[k] = lo[k];
        scene->scene_bound[3 + k] = hi[k];
    }
    scene->ref_nodes.release();
    scene->prims.release();
    scene->n_nodes = 0;
    scene->n_prims = total_slots;
    scene->n_trav = total_trav;
    scene->root_ref = 0;
    scene->root_count = 0;
    return KS_OK;
}

ks_status build_sbvh(ks_scene *scene, const ks_sbvh_options &o, float *build_ms)
{
    ks_context *ctx = scene->ctx;
    cudaStream_t st = ctx->stream;
    Params p;
    // option clamps (cuda/sbvh.cu:411-414)
    p.max_prims = std::min(o.max_prims_in_node, 8u);
    p.buckets = std::min(o.bucket_count, 16u);
    p.trav_weight = std::clamp(o.trav_weight, 0.0f, 10.0f);
    p.alpha = std::clamp(o.alpha, 0.0f, 1.0f);
    if (p.buckets < 2)
        return fail(ctx, KS_ERR_INVALID_ARGUMENT, "ks_scene_build_bvh: bucket_count must be >= 2");
    if (scene->n_tris == 0)
        return fail(ctx, KS_ERR_INVALID_ARGUMENT, "ks_scene_build_bvh: scene has no triangles");
    cudaEvent_t ev0, ev1, ev2, ev3;
    KS_CUDA_TRY(ctx, cudaEventCreate(&ev0));
    KS_CUDA_TRY(ctx, cudaEventCreate(&ev1));
    KS_CUDA_TRY(ctx, cudaEventCreate(&ev2));
    KS_CUDA_TRY(ctx, cudaEventCreate(&ev3));
    bool widened = false;
    KS_CUDA_TRY(ctx, cudaEventRecord(ev0, st));
    ks_status s = KS_OK;
    if (scene->n_instances > 0) {
        s = build_instanced(scene, p);
        if (s == KS_OK)
            cudaEventRecord(ev1, st);
    } else {
        RangeOut r;
        s = build_range(ctx, scene->verts.ptr, scene->indices.ptr, 0, scene->n_tris, p, r, ev1);
        if (s == KS_OK) {
            scene->ref_nodes.swap(r.ref_nodes);
            scene->prims.swap(r.prims);
            scene->trav_nodes.swap(r.trav);
            scene->prim_tris.swap(r.prim_tris);
            scene->leaf_box.swap(r.leaf_box);
            std::memcpy(scene->scene_bound, r.bound, sizeof(r.bound));
            scene->n_nodes = r.n_nodes;
            scene->n_prims = r.n_prims;
            scene->n_trav = r.n_trav;
            scene->root_count = r.n_prims;
            scene->root_ref = r.n_trav > 0 ? 0u : kLeafBit;
            // the renderer's 4-wide view of the tree, or the exact traversal's steps (timed with the build)
            scene->deep = r.n_levels > kMaxBinaryLevels;
            scene->coincident = false;
            scene->wide_nodes.release();
            scene->wide_steps.release();
            cudaEventRecord(ev2, st);
            if (!scene->deep) {
                s = build_wide4(ctx, build_scratch(ctx), scene->trav_nodes.ptr, r.n_trav, scene->root_ref, r.bound,
                                r.n_levels, scene->wide_nodes);
            } else if (make_wide_steps(scene) != cudaSuccess) {
                s = fail(ctx, KS_ERR_OUT_OF_MEMORY, "ks_scene_build_bvh: wide nodes");
            }
            cudaEventRecord(ev3, st);
            widened = s == KS_OK;
        }
    }
    float ms = 0;
    if (s == KS_OK) {
        cudaEventSynchronize(ev1);
        cudaEventElapsedTime(&ms, ev0, ev1);
        if (widened) {
            float mw = 0;
            cudaEventSynchronize(ev3);
            cudaEventElapsedTime(&mw, ev2, ev3);
            ms += mw;
        }
    } else {
        // a build that stopped early leaves its work on the stream: let it finish before the
        // scratch is reused, and keep no error of it for the next call
        cudaStreamSynchronize(st);
        cudaGetLastError();
    }
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
    cudaEventDestroy(ev2);
    cudaEventDestroy(ev3);
    if (s != KS_OK)
        return s;
    if (build_ms)
        *build_ms = ms;
    scene->bvh_built = true;
    return KS_OK;
}

} // namespace ksb

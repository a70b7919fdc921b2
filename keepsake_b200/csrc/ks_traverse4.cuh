// Traversal of the renderer's 4-wide view of the SBVH (Wide4Node): its ray queries on the device.
//
// The result of a query is the one that the 4-wide steps of ks_traverse.cuh give (the closest hit, or
// whether anything is hit: "the exact traversal" below), reached with cheaper steps, since the kernels
// are bound by the instructions they issue:
//   * the box test need only be conservative: one fused multiply-add per plane instead of a
//     subtraction, a product and a guard, with its rounding widened away (Trav4::set_ray);
//   * a closest-hit node's slots are sorted as integers, the entry time with the slot in its last two
//     bits; a pending child is that key and its parent's index, and its ref is read when it is visited.
// What keeps the result:
//   * a triangle that is hit counts when slab() accepts its leaf's box, which is when the exact
//     traversal tests the triangle at all (a leaf's box passes only if every box above it does);
//   * which of several hits is the closest does not depend on the visiting order unless two of them
//     are nearly equally far: within rounding of each other, or one nearer than the other's box is
//     entered.  Within a leaf the order is the exact traversal's; where two leaves are concerned Trav4 keeps
//     what is needed to see it, and such a ray is traced again in the exact traversal's order (retrace).
//     That is about one ray in a million of the mesh frame (no two surfaces in one plane); a scene with
//     many goes over to the exact steps (kAgainShare).
// Trees too deep for the stack keep the exact traversal, whose stack overflow is an error status, and so do
// instanced scenes: beside the state of their upper level this one's does not fit the registers (closest hit
// over 400 instances at 1080p x 4: 22.0 ms by the exact traversal, 23.8 by this one at its best).
#pragma once
#include "ks_traverse.cuh"

namespace ksb
{

// Deepest SBVH (levels) with this view: the exact traversal pushes at most 3 entries per two levels, so
// up to here it never outgrows kWideStackDepth.  This one pushes at most 3 per level of the view; where opening
// the largest child first gives more levels than that allows, the view opens evenly (build_wide4).  A sphere of
// 81920 triangles, 512 x 512 x 4, beside nested clusters (58 levels) 3.3 ms, beside a chain (114 levels, the exact
// steps) 3.9 ms; with both on binary nodes widened at each visit 9.6 and 10.2 ms.
constexpr uint32_t kMaxBinaryLevels = 2 * (kWideStackDepth / 3), kMaxWideLevels = kWideStackDepth / 3;

KS_D float max3f(float a, float b, float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
KS_D float min3f(float a, float b, float c)
{
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Relative slack of the box test, of the ray's end, of the pruning distance and of the tie test (Trav4).
// An entry time that is compared with the ray's end may lie above slab()'s by 3 roundings (2^-24 each; the
// padding by the origin vanishes at the origin) and, on the stack, by the slot number in its last two bits (3 ulp).
constexpr float kMaxInv = 1e30f; // 1 / d is clamped to it
constexpr float kBoxSlack = 0x1p-20f, kRangeSlack = 0x1p-18f, kPruneSlack = 0x1p-12f, kTieSlack = 0x1p-20f;

// What the traversal reads: the nodes, and per leaf (at its first primitive slot) its box, 2 float4.
struct Tree4
{
    const Wide4Node *nodes;
    const float4 *leaf_box;
};

struct Trav4
{
    RayQuery ray;            // tmax: as the query gave it
    TriHelper th;
    f3 inv;                  // 1 / d
    f3 o_in, inv_out, o_out; // t of an entry plane: b inv - o_in; of an exit plane: b inv_out - o_out
    uint32_t ref;            // the node or leaf to visit
    int sp;
    float limit;             // boxes and triangles beyond it are skipped: no less than what ends the query
    Hit hit;
    float entry;             // entry time of the hit's leaf
    float second;            // distance of the closest other hit seen

    KS_D bool at_leaf() const { return (ref & kLeafBit) != 0; }

    // The plane equations.  Against slab()'s t = (b - o) * inv the fused form is off by at most
    // 2^-24 |o inv| per rounded constant and a few 2^-24 |t|: the offsets are moved out by
    // 2^-22 |o inv|, exit planes are scaled by 1 + 2^-20.  A zero component's infinite 1 / d is
    // clamped, which keeps the products finite: inside its slab the interval stays at least +-1e30
    // times the distance to the planes, outside it starts beyond every other exit.
    KS_D void set_ray(f3 d)
    {
        auto axis = [&](float o, float dc, float &iv, float &oi, float &io, float &oo) {
            iv = 1.0f / dc;
            if (!(fabsf(iv) <= kMaxInv))
                iv = copysignf(kMaxInv, iv);
            const float oc = o * iv, pad = fabsf(oc) * 0x1p-22f;
            oi = oc + pad;
            io = iv * (1.0f + kBoxSlack);
            oo = oc * (1.0f + kBoxSlack) - pad;
            if (ray.tmin < 0.0f) // negative distances: the scale would move exit planes inwards
                oo += ray.tmin * 0x1p-18f;
        };
        axis(ray.o.x, d.x, inv.x, o_in.x, inv_out.x, o_out.x);
        axis(ray.o.y, d.y, inv.y, o_in.y, inv_out.y, o_out.y);
        axis(ray.o.z, d.z, inv.z, o_in.z, inv_out.z, o_out.z);
    }
};

// The query's own 1 / d: what set_ray clamped was infinite.  (Or the component was a nonzero one below
// 1e-30, whose slab a ray leaves within a distance of 1e-25 of its plane: infinity decides the same.)
KS_D BoxHelper exact_helper(const Trav4 &s)
{
    auto own = [](float iv) { return fabsf(iv) == kMaxInv ? copysignf(kInf, iv) : iv; };
    return box_helper_of(mk(own(s.inv.x), own(s.inv.y), own(s.inv.z)));
}

// Whether another visiting order could have found another closest hit: one within rounding of it, or
// nearer than its leaf is entered (a leaf is skipped when the ray enters it beyond the hit at hand).
KS_D bool ambiguous(const Trav4 &s)
{
    const float far = fmaxf(s.hit.t, s.entry);
    return s.hit.tri != ~0u && (!(s.second > far + fabsf(far) * kTieSlack) ||
                                s.entry > s.hit.t + fabsf(s.hit.t) * (0.5f * kPruneSlack));
}

// False when the ray misses the root box.
KS_D bool trav_begin(Trav4 &s, const RayQuery &ray, uint32_t root, uint32_t root_count, const float root_bmin[3],
                     const float root_bmax[3])
{
    s.hit.tri = s.hit.slot = ~0u;
    s.ray = ray;
    s.th = make_tri_helper(ray.d);
    s.set_ray(ray.d);
    s.limit = ray.tmax + fabsf(ray.tmax) * kRangeSlack;
    s.entry = 0.0f;
    s.second = kInf;
    s.sp = 0;
    s.ref = root;
    float t0, t1;
    return root_count != 0 && slab(ray, make_box_helper(ray.d), root_bmin, root_bmax, t0, t1) && t0 < ray.tmax &&
           t1 > ray.tmin;
}

// The next pending child; false when there is none.  Closest hit: entries are (parent index, key), dropped
// beyond the limit.  Any hit: the child's ref.
template <bool kAnyHit>
KS_D bool trav4_pop(const Wide4Node *__restrict__ nodes, Trav4 &s, const TravStack &stack)
{
    while (s.sp > 0) {
        const uint2 e = stack.get(--s.sp);
        if constexpr (kAnyHit) {
            s.ref = e.x;
            return true;
        } else if (__uint_as_float(e.y) <= s.limit) {
            s.ref = __ldg(&nodes[e.x].ref[e.y & 3u]);
            return true;
        }
    }
    return false;
}

// Visits node s.ref: descends to a child and returns true, or returns false when none is hit.
// Any-hit queries take the children in slot order (why: trav_descend).
template <bool kAnyHit>
KS_D bool trav4_node(const Wide4Node *__restrict__ nodes, Trav4 &s, TravStack &stack, TravCount *count)
{
    if (count)
        count->nodes += 2; // 128 bytes: two 64-byte node units
    const uint32_t at = s.ref;
    const uintptr_t n = reinterpret_cast<uintptr_t>(nodes + at);
    // the entry plane of an axis is its upper one (16 bytes on) when the direction is negative
    auto plane = [&](uint32_t axis, uint32_t upper) {
        return __ldg(reinterpret_cast<const float4 *>((n | (upper & 16u)) + 32u * axis));
    };
    const uint32_t ux = __float_as_uint(s.inv.x) >> 27, uy = __float_as_uint(s.inv.y) >> 27,
                   uz = __float_as_uint(s.inv.z) >> 27;
    const float4 ax = plane(0, ux), ay = plane(1, uy), az = plane(2, uz);
    const float4 bx = plane(0, ~ux), by = plane(1, ~uy), bz = plane(2, ~uz);
    const float ex[4] = {ax.x, ax.y, ax.z, ax.w}, ey[4] = {ay.x, ay.y, ay.z, ay.w}, ez[4] = {az.x, az.y, az.z, az.w};
    const float lx[4] = {bx.x, bx.y, bx.z, bx.w}, ly[4] = {by.x, by.y, by.z, by.w}, lz[4] = {bz.x, bz.y, bz.z, bz.w};
    float t_in[4];
    bool ok[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        t_in[k] = max3f(fmaf(ex[k], s.inv.x, -s.o_in.x), fmaf(ey[k], s.inv.y, -s.o_in.y),
                        fmaxf(fmaf(ez[k], s.inv.z, -s.o_in.z), s.ray.tmin));
        const float t_out = min3f(fmaf(lx[k], s.inv_out.x, -s.o_out.x), fmaf(ly[k], s.inv_out.y, -s.o_out.y),
                                  fminf(fmaf(lz[k], s.inv_out.z, -s.o_out.z), s.limit));
        ok[k] = t_in[k] <= t_out;
    }
    if constexpr (kAnyHit) {
        const uint4 child = __ldg(reinterpret_cast<const uint4 *>(n + 96));
        const uint32_t ref[4] = {child.x, child.y, child.z, child.w};
        // the first slot hit next, the others below it on the stack, the last one deepest
        const int top = s.sp + (int)ok[0] + (int)ok[1] + (int)ok[2] + (int)ok[3] - 1;
        if (top < s.sp)
            return false;
        s.ref = ok[0] ? ref[0] : (ok[1] ? ref[1] : (ok[2] ? ref[2] : ref[3]));
        int put = s.sp;
#pragma unroll
        for (int k = 3; k >= 1; --k)
            if (ok[k] && put < top)
                stack.set(put++, ref[k], 0.0f);
        s.sp = top;
    } else {
        // t_in >= tmin >= 0 in a render: the bits order like the times (a negative tmin only costs order)
        uint32_t key[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            key[k] = ok[k] ? ((__float_as_uint(t_in[k]) & ~3u) | (uint32_t)k) : ~0u;
        auto cex = [&](int i, int j) {
            const uint32_t lo = min(key[i], key[j]), hi = max(key[i], key[j]);
            key[i] = lo;
            key[j] = hi;
        };
        cex(0, 1);
        cex(2, 3);
        cex(0, 2);
        cex(1, 3);
        cex(1, 2);
        if (key[0] == ~0u)
            return false;
        const int top = s.sp + (key[1] != ~0u) + (key[2] != ~0u) + (key[3] != ~0u);
        if (top <= kSmemStack) {
            uint2 *e = stack.sm + top * kTravBlock;
#pragma unroll
            for (int r = 1; r < 4; ++r)
                if (key[r] != ~0u)
                    e[-r * kTravBlock] = make_uint2(at, key[r]);
        } else {
            for (int r = 3; r >= 1; --r)
                if (key[r] != ~0u)
                    stack.set(top - r, at, __uint_as_float(key[r]));
        }
        s.sp = top;
        s.ref = __ldg(&nodes[at].ref[key[0] & 3u]);
    }
    return true;
}

// The box of a leaf in slab()'s own arithmetic: whether the exact traversal tests the leaf, and when
// the ray enters it.
KS_D bool leaf_reached(const float4 *__restrict__ leaf_box, const Trav4 &s, uint32_t first, float &entry)
{
    const float4 lo = __ldg(leaf_box + 2 * (size_t)first), hi = __ldg(leaf_box + 2 * (size_t)first + 1);
    const float bmin[3] = {lo.x, lo.y, lo.z}, bmax[3] = {hi.x, hi.y, hi.z};
    float t1;
    return slab(s.ray, exact_helper(s), bmin, bmax, entry, t1) && t1 > s.ray.tmin && entry < s.ray.tmax;
}

// Whether the hit at hand is one of the leaf that starts at `first`, of which `slot` is tested.
KS_D bool in_leaf(const Trav4 &s, uint32_t first, uint32_t slot)
{
    return s.hit.slot - first < slot - first; // no hit yet: slot ~0u
}

// The range in which primitive `slot` of a leaf is tested.  After a hit in the same leaf it ends there, as in
// the exact traversal: the order within a leaf is the same, so which of a leaf's nearly equal hits stays
// (a mesh given twice has its copies in one leaf) is no question of the order of leaves.
KS_D RayQuery leaf_range(const Trav4 &s, uint32_t first, uint32_t slot)
{
    RayQuery q = s.ray;
    q.tmax = in_leaf(s, first, slot) ? s.hit.t : fminf(q.tmax, s.limit);
    return q;
}

// Takes note of a closest-hit ray's hit on a triangle of a leaf that starts at `first` and that the ray enters
// at `entry`.
KS_D void trav4_take(Trav4 &s, const Hit &h, float entry, uint32_t first)
{
    if (h.tri == s.hit.tri) {
        s.entry = fminf(s.entry, entry); // the same triangle through another of its leaves
    } else if (s.hit.tri == ~0u || h.t < s.hit.t) {
        if (s.hit.tri != ~0u && !in_leaf(s, first, h.slot))
            s.second = fminf(s.second, s.hit.t);
        s.entry = entry;
        s.limit = fminf(s.limit, h.t + fabsf(h.t) * kPruneSlack);
        s.hit = h;
    } else {
        s.second = fminf(s.second, h.t);
    }
}

// Tests the leaf at hand; true when an any-hit query found an occluder.
template <bool kAnyHit, class Alpha>
KS_D bool trav4_leaf(const float4 *__restrict__ leaf_box, const float4 *__restrict__ tris, Trav4 &s, int culling,
                     TravCount *count, const Alpha &alpha)
{
    const uint32_t first = s.ref & ~kLeafBit;
    uint32_t slot = first;
    bool last;
    do {
        if (count)
            count->tris++;
        const float4 *p = tris + 3 * (size_t)slot;
        const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
        last = __float_as_uint(b.w) != 0u;
        const f3 v0 = mk(a.x, a.y, a.z), v1 = mk(b.x, b.y, b.z), v2 = mk(c.x, c.y, c.z);
        const uint32_t tri = __float_as_uint(a.w);
        const RayQuery q = kAnyHit ? s.ray : leaf_range(s, first, slot);
        float t, b0, b1, b2;
        if (!cull_tri(q, v0, v1, v2, culling) && isect_tri(q, s.th, v0, v1, v2, t, b0, b1, b2)) {
            float entry;
            if (kAnyHit) {
                if (leaf_reached(leaf_box, s, first, entry) && alpha(tri, b1, b2, s.ray)) {
                    s.hit.tri = tri;
                    return true;
                }
            } else if (t < q.tmax && leaf_reached(leaf_box, s, first, entry) && alpha(tri, b1, b2, s.ray)) {
                trav4_take(s, Hit{tri, slot, t, b0, b1, b2}, entry, first);
            }
        }
        ++slot;
    } while (!last);
    return false;
}

// One step (a node or a leaf); true when the traversal of the ray is over.
template <bool kAnyHit, class Alpha = NoAlpha>
KS_D bool trav_step(const Tree4 &tree, const float4 *__restrict__ tris, Trav4 &s, TravStack &stack, int culling, int &,
                    TravCount *count, const Alpha &alpha = Alpha{})
{
    if (s.at_leaf()) {
        if (trav4_leaf<kAnyHit>(tree.leaf_box, tris, s, culling, count, alpha))
            return true;
    } else {
        if (trav4_node<kAnyHit>(tree.nodes, s, stack, count))
            return false;
    }
    return !trav4_pop<kAnyHit>(tree.nodes, s, stack);
}

// ---- one ray per group of 4 lanes -------------------------------------------------------------
// A queue shorter than the GPU takes the time of its longest ray, whatever the throughput: some hundred
// rays along a bumpy surface took 100 to 170 us a launch, one dependent step after the other.  Here the 4
// lanes of a group follow one ray: a lane tests one slot of a node or one triangle of a leaf, so a step's
// chain is that of one box instead of four, a sort and three pushes.  Every lane holds the ray's state
// (the same values); the same tests make the same hits.  The stack is the group's, in shared memory.
constexpr int kGroup = 4, kGroupStack = kWideStackDepth; // entries of (ref, entry time)

struct GroupStack
{
    uint2 *e;
};
#define KS_GROUP_STACK(name)                                                                                     \
    __shared__ uint2 name##_smem[kTravBlock / kGroup][kGroupStack];                                             \
    const GroupStack name{name##_smem[threadIdx.x / kGroup]}

// One ray from trav_begin to its end; `mask`: the group's lanes.
template <bool kAnyHit, class Alpha>
KS_D void group_trace(const Tree4 &tree, const float4 *__restrict__ tris, Trav4 &s, const GroupStack &stack,
                      uint32_t mask, int culling, TravCount *count, const Alpha &alpha)
{
    const uint32_t lane = threadIdx.x & 31u, k = lane & (kGroup - 1u), shift = lane & ~(kGroup - 1u);
    while (true) {
        if (!s.at_leaf()) {
            if (k == 0)
                count->nodes += 2;
            const float *n = reinterpret_cast<const float *>(tree.nodes + s.ref) + k;
            const int ux = s.inv.x < 0.0f ? 4 : 0, uy = s.inv.y < 0.0f ? 4 : 0, uz = s.inv.z < 0.0f ? 4 : 0;
            const float ex = __ldg(n + ux), ey = __ldg(n + 8 + uy), ez = __ldg(n + 16 + uz);
            const float lx = __ldg(n + 4 - ux), ly = __ldg(n + 12 - uy), lz = __ldg(n + 20 - uz);
            const uint32_t ref = __float_as_uint(__ldg(n + 24));
            const float t_in = max3f(fmaf(ex, s.inv.x, -s.o_in.x), fmaf(ey, s.inv.y, -s.o_in.y),
                                     fmaxf(fmaf(ez, s.inv.z, -s.o_in.z), s.ray.tmin));
            const float t_out = min3f(fmaf(lx, s.inv_out.x, -s.o_out.x), fmaf(ly, s.inv_out.y, -s.o_out.y),
                                      fminf(fmaf(lz, s.inv_out.z, -s.o_out.z), s.limit));
            const bool ok = t_in <= t_out;
            const uint32_t hits = (__ballot_sync(mask, ok) >> shift) & ((1u << kGroup) - 1u);
            if (hits) {
                const int n_hit = __popc(hits);
                int rank; // among the slots hit: by time, any-hit queries by slot
                if constexpr (kAnyHit) {
                    rank = __popc(hits & ((1u << k) - 1u));
                } else {
                    const uint32_t key = ok ? ((__float_as_uint(t_in) & ~3u) | k) : ~0u;
                    rank = 0;
#pragma unroll
                    for (int x = 1; x < kGroup; ++x)
                        rank += __shfl_xor_sync(mask, key, x) < key ? 1 : 0;
                }
                if (ok && rank > 0)
                    stack.e[s.sp + n_hit - 1 - rank] = make_uint2(ref, __float_as_uint(t_in));
                const uint32_t first = (__ballot_sync(mask, ok && rank == 0) >> shift) & ((1u << kGroup) - 1u);
                s.ref = __shfl_sync(mask, ref, (int)(shift + __ffs(first) - 1u));
                s.sp += n_hit - 1;
                __syncwarp(mask);
                continue;
            }
        } else {
            const uint32_t first = s.ref & ~kLeafBit;
            uint32_t base = first;
            bool last = false;
            while (!last) {
                // the record past the leaf's last is another leaf's or the array's padding: read, not used
                const uint32_t slot = base + k;
                const float4 *p = tris + 3 * (size_t)slot;
                const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
                const uint32_t ends =
                    (__ballot_sync(mask, __float_as_uint(b.w) != 0u) >> shift) & ((1u << kGroup) - 1u);
                last = ends != 0u;
                const bool mine = !last || (int)k < __ffs(ends);
                const f3 v0 = mk(a.x, a.y, a.z), v1 = mk(b.x, b.y, b.z), v2 = mk(c.x, c.y, c.z);
                Hit h;
                h.tri = __float_as_uint(a.w);
                h.slot = slot;
                float entry = 0.0f;
                bool take = false;
                auto test = [&]() {
                    const RayQuery q = kAnyHit ? s.ray : leaf_range(s, first, slot);
                    return !cull_tri(q, v0, v1, v2, culling) &&
                           isect_tri(q, s.th, v0, v1, v2, h.t, h.b0, h.b1, h.b2) && (kAnyHit || h.t < q.tmax);
                };
                if (mine) {
                    count->tris++;
                    take = test() && leaf_reached(tree.leaf_box, s, first, entry) && alpha(h.tri, h.b1, h.b2, s.ray);
                }
                uint32_t found = (__ballot_sync(mask, take) >> shift) & ((1u << kGroup) - 1u);
                if constexpr (kAnyHit) {
                    if (found) {
                        s.hit.tri = 0u;
                        return;
                    }
                } else {
                    while (found) { // in the leaf's order, as one lane would
                        const int src = (int)(shift + __ffs(found) - 1u);
                        Hit g;
                        g.tri = __shfl_sync(mask, h.tri, src);
                        g.slot = __shfl_sync(mask, h.slot, src);
                        g.t = __shfl_sync(mask, h.t, src);
                        g.b0 = __shfl_sync(mask, h.b0, src);
                        g.b1 = __shfl_sync(mask, h.b1, src);
                        g.b2 = __shfl_sync(mask, h.b2, src);
                        trav4_take(s, g, __shfl_sync(mask, entry, src), first);
                        found &= found - 1u;
                        if (found) {
                            const bool later = (found >> k) & 1u;
                            found = (__ballot_sync(mask, later && test()) >> shift) & ((1u << kGroup) - 1u);
                        }
                    }
                }
                base += kGroup;
            }
        }
        // the next pending child
        bool more = false;
        while (s.sp > 0 && !more) {
            const uint2 e = stack.e[--s.sp];
            s.ref = e.x;
            more = kAnyHit || __uint_as_float(e.y) <= s.limit;
        }
        __syncwarp(mask);
        if (!more)
            return;
    }
}

// The closest hit by the exact traversal's own order: the 4-wide steps over boxes read from the
// binary nodes.  Out of line and called from other kernels than the traversal's: a call there would
// cost its registers and its stack their places (measured: 1.3 x the time).
struct Retraced
{
    Hit hit;
    int overflow;
};
template <class Alpha = NoAlpha>
static __device__ __noinline__ Retraced retrace(const TravNode *nodes, const float4 *tris, uint32_t root_ref,
                                                uint32_t root_count, const float *bmin, const float *bmax, RayQuery q,
                                                int culling, Alpha alpha = Alpha{})
{
    TravState s;
    LocalStack stack;
    Retraced r;
    r.overflow = 0;
    if (trav_begin(s, q, root_ref, root_count, bmin, bmax))
        while (!trav_step<false>(reinterpret_cast<const LazyWide *>(nodes), tris, s, stack, culling, r.overflow, nullptr,
                                 alpha)) {
        }
    r.hit = s.hit;
    return r;
}
} // namespace ksb

// pg_traverse_warp.cuh - warp-cooperative BVH traversal: each lane walks its
// own ray down the four-wide BVH, the warp tests the rays' leaf triangles
// together.
//
// Why: with one ray per lane and each lane testing its own leaves, a warp
// instruction of the triangle test had 6-7 lanes active (a step meets about one
// triangle per ray on average, but the slowest lane meets ten).  Here a step
// appends the leaves its rays meet to a list in shared memory and four lanes
// take each leaf, one triangle per lane: eight leaves per pass, neighbouring
// lanes reading neighbouring triangles.
//
// The hit is the one trav_step finds, bit for bit: a ray visits the same nodes in
// the same order against the same best t, each node's boxes are met or dropped by
// box_enter's arithmetic (lane_boxes), the triangle test's is the same, and the
// least (t, id) of a step's accepted triangles does not depend on the order they are
// tested in.  Meeting more boxes than box_enter would not do: it drops a box whose
// plane holds the origin of a ray that does not move along that axis (0 x infinity),
// and a triangle in such a box is then no hit.  trav_step stays for renders that
// count their work and for single rays inside divergent code.
//
// Both sides of an SM were near their limits with the slab test and the pair
// list of the first version (ncu, second bounce of the Cornell box: 21 warp
// instructions per ray and node at 70 % of the issue slots, 66 % of the L1 data
// pipe's wavefronts; now 73-77 % and 72-80 %, 23-25 lanes active).
#pragma once

#include "pg_traverse.cuh"

namespace pg {

constexpr unsigned kFullWarp = 0xffffffffu;
constexpr int kSharedStack = 12;  // stack entries per lane in shared memory, deeper ones local
constexpr int kLaneDeep = kStackSize - kSharedStack;

// One warp's shared memory.
struct WarpTrav {
    uint2 leaf[128];                // a met leaf: {first triangle, its ray's lane | triangles << 8}
    float4 ray_a[32], ray_b[32];    // the lanes' rays for the triangle test: {origin, Sx}, {Sy, Sz, tmin, axis}
    float2 best[32];                // best t of each lane's ray and its primitive (any hit: PG_NO_HIT until occluded)
    float2 uv[32];                  // barycentrics of the best hit
    int stack[kSharedStack][32];
};

// A lane's ray during a traversal.  A child's slab distances are (plane + neg_org)
// inv; the planes of axis i that the ray meets first start at byte near[i] of a
// node, the others at 48 + 32 i - near[i].
struct LaneRay {
    float inv[3], neg_org[3];
    float tmin, tmax;  // tmax: best t so far for closest-hit queries
    int near[3];
    int node, sp;
    bool odd;          // the planes' order does not follow from inv (lane_boxes)
};

__device__ __forceinline__ void lane_push(LaneRay &st, WarpTrav &W, int *deep, int lane, int x) {
    if (st.sp >= kStackSize) return;
    if (st.sp < kSharedStack)
        W.stack[st.sp][lane] = x;
    else
        deep[st.sp - kSharedStack] = x;
    ++st.sp;
}
__device__ __forceinline__ int lane_pop(LaneRay &st, const WarpTrav &W, const int *deep, int lane) {
    --st.sp;
    return st.sp < kSharedStack ? W.stack[st.sp][lane] : deep[st.sp - kSharedStack];
}

// Starts a lane's query (trav_begin's rules: the spheres first).  Returns true
// when it is already decided (any hit: a sphere occludes).
template <bool kAny>
__device__ __forceinline__ bool lane_begin(const DevScene &S, LaneRay &st, WarpTrav &W, int lane, const float o[3],
                                           const float d[3], float tmin, float tmax) {
    const RayPre r = ray_setup(o, d);
    st.tmin = tmin;
    st.tmax = tmax;
    st.node = 0;
    st.sp = 0;
    uint32_t id = PG_NO_HIT;
    for (uint32_t i = 0; i < S.n_spheres; ++i) {
        float t;
        if (sphere_intersect(r, S.spheres[i], tmin, st.tmax, t)) {
            id = PG_SPHERE_BIT | i;
            if (kAny) break;
            st.tmax = t;
        }
    }
    st.odd = false;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        st.inv[i] = r.inv[i];
        st.neg_org[i] = -o[i];
        st.near[i] = 16 * i + (r.inv[i] < 0.0f ? 48 : 0);
        st.odd |= !(fabsf(r.inv[i]) < INFINITY) || r.inv[i] == 0.0f || !(fabsf(o[i]) < INFINITY);
    }
    // the rotation that takes axis kz to z; ray_setup's swap of x and y for
    // d[kz] < 0 is kept as a flag (tri_test)
    const bool flip = d[r.kz] < 0.0f;
    W.ray_a[lane] = make_float4(o[0], o[1], o[2], flip ? r.Sy : r.Sx);
    W.ray_b[lane] = make_float4(flip ? r.Sx : r.Sy, r.Sz, tmin, __int_as_float(r.kz | (flip ? 4 : 0)));
    W.best[lane] = make_float2(st.tmax, __uint_as_float(id));
    W.uv[lane] = make_float2(0.0f, 0.0f);
    return kAny && id != PG_NO_HIT;
}

// The edge functions of a ray in the form lane_begin stores: tri_intersect's
// arithmetic with axes rotated, not swapped.  A swap of x and y negates U, V, W,
// det and T exactly, so t is the same.  Returns whether the ray's line passes
// through the triangle; T / det is then t.
struct TriEdges {
    float V, W, det, T;
};
__device__ __forceinline__ bool tri_edges(const float4 &ra, const float4 &rb, const float4 &v0, const float4 &v1,
                                          const float4 &v2, TriEdges &x) {
    const int axis = __float_as_int(rb.w);
    const bool z0 = (axis & 3) == 0, z1 = (axis & 3) == 1;
    auto rotate = [&](const float4 &p, float &px, float &py, float &pz) {
        const float a = __fsub_rn(p.x, ra.x), b = __fsub_rn(p.y, ra.y), c = __fsub_rn(p.z, ra.z);
        pz = z0 ? a : (z1 ? b : c);
        px = z0 ? b : (z1 ? c : a);
        py = z0 ? c : (z1 ? a : b);
    };
    float Akx, Aky, Akz, Bkx, Bky, Bkz, Ckx, Cky, Ckz;
    rotate(v0, Akx, Aky, Akz);
    rotate(v1, Bkx, Bky, Bkz);
    rotate(v2, Ckx, Cky, Ckz);
    const float Sx = ra.w, Sy = rb.x, Sz = rb.y;
    const float Ax = __fmaf_rn(-Sx, Akz, Akx), Ay = __fmaf_rn(-Sy, Akz, Aky);
    const float Bx = __fmaf_rn(-Sx, Bkz, Bkx), By = __fmaf_rn(-Sy, Bkz, Bky);
    const float Cx = __fmaf_rn(-Sx, Ckz, Ckx), Cy = __fmaf_rn(-Sy, Ckz, Cky);
    float U = __fsub_rn(__fmul_rn(Cx, By), __fmul_rn(Cy, Bx));
    float V = __fsub_rn(__fmul_rn(Ax, Cy), __fmul_rn(Ay, Cx));
    float W = __fsub_rn(__fmul_rn(Bx, Ay), __fmul_rn(By, Ax));
    if (fminf(fminf(fabsf(U), fabsf(V)), fabsf(W)) == 0.0f) {
        // an edge function exactly zero: redo them in double (exact products), the
        // difference taken as ray_setup's axes take it (the sign of a zero is then theirs)
        const bool flip = (axis & 4) != 0;
        auto edge = [flip](float a, float b, float c, float d) {
            const double p = __dmul_rn((double)a, (double)b), q = __dmul_rn((double)c, (double)d);
            return flip ? -(float)__dsub_rn(q, p) : (float)__dsub_rn(p, q);
        };
        U = edge(Cx, By, Cy, Bx);
        V = edge(Ax, Cy, Ay, Cx);
        W = edge(Bx, Ay, By, Ax);
    }
    x.V = V;
    x.W = W;
    x.det = __fadd_rn(__fadd_rn(U, V), W);
    x.T = __fmaf_rn(W, __fmul_rn(Sz, Ckz), __fmaf_rn(V, __fmul_rn(Sz, Bkz), __fmul_rn(U, __fmul_rn(Sz, Akz))));
    const bool mixed = fminf(fminf(U, V), W) < 0.0f && fmaxf(fmaxf(U, V), W) > 0.0f;
    return !mixed && x.det != 0.0f;
}
// The barycentrics V / det, W / det as ray_setup's swapped axes give them: all
// three negated, which matters for the sign of a zero.
__device__ __forceinline__ float2 tri_uv(const float4 &rb, const TriEdges &x) {
    const bool flip = (__float_as_int(rb.w) & 4) != 0;
    const float dn = flip ? -x.det : x.det;
    return make_float2(__fdiv_rn(flip ? -x.V : x.V, dn), __fdiv_rn(flip ? -x.W : x.W, dn));
}

// Tests the triangles of the lanes' met leaves (leaf[j]: child j of the lane's
// node is one, ref[j] names it), all lanes of the warp together.  Updates
// W.best and W.uv (closest: the least (t, id); any: the primitive of an
// occluded ray).  Lanes without a triangle test one all the same (the array
// has four spare ones) and drop the result: no branch around the loads.
template <bool kAny>
__device__ __forceinline__ void warp_leaves(const DevScene &S, WarpTrav &W, int lane, const bool (&leaf)[4],
                                            const int (&ref)[4]) {
    const unsigned below = (1u << lane) - 1u;
    // leaves of more than four triangles go on in further rounds
    for (int skip = 0;; skip += 4) {
        int n = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int left = leaf_count(ref[j]) - skip;
            const bool on = leaf[j] && left > 0;
            const unsigned m = __ballot_sync(kFullWarp, on);
            if (on)
                W.leaf[n + __popc(m & below)] = make_uint2((uint32_t)(leaf_first(ref[j]) + skip),
                                                           (uint32_t)lane | ((uint32_t)min(left, 4) << 8));
            n += __popc(m);
        }
        if (n == 0) return;
        __syncwarp();
        for (int base = 0; base < n; base += 8) {
            const int q = base + (lane >> 2);
            uint2 lf = W.leaf[q];  // past n: stale words of earlier lists, or zeros
            const bool on = q < n && (uint32_t)(lane & 3) < (lf.y >> 8);
            lf.x = on ? lf.x + (uint32_t)(lane & 3) : 0u;
            const int src = (int)(lf.y & 31u);
            const float4 *tri = S.tris + 3 * (size_t)lf.x;
            const float4 v0 = __ldg(tri), v1 = __ldg(tri + 1), v2 = __ldg(tri + 2);
            const float4 ra = W.ray_a[src], rb = W.ray_b[src];
            const float2 bst = W.best[src];
            const float bt = bst.x;
            const uint32_t bid = __float_as_uint(bst.y), id = __float_as_uint(v0.w);
            TriEdges x;
            bool acc = tri_edges(ra, rb, v0, v1, v2, x) && on;
            float t = 0.0f;
            if (acc) {
                t = __fdiv_rn(x.T, x.det);
                // one ulp above the best t, so an equal t is seen and the lower id wins
                const float lim = (kAny || bid == PG_NO_HIT) ? bt : __uint_as_float(__float_as_uint(bt) + 1u);
                acc = t > rb.z && t < lim && (kAny || t < bt || id < bid);
                const uint32_t tex = __float_as_uint(v1.w);
                if (tex != 0u && acc) {
                    const float2 uv = tri_uv(rb, x);
                    acc = alpha_keep(S, ra.x, id, tex, uv.x, uv.y, t);
                }
            }
            if (!__any_sync(kFullWarp, acc)) continue;
            if (kAny) {
                if (acc) W.best[src].y = __uint_as_float(id);
                __syncwarp();
            } else {
                // t > tmin >= 0: its bits order as the numbers do
                if (acc) atomicMin(reinterpret_cast<unsigned *>(&W.best[src].x), __float_as_uint(t));
                __syncwarp();
                const bool win = acc && W.best[src].x == t;
                if (win && t < bt) W.best[src].y = __uint_as_float(PG_NO_HIT);  // closer than every earlier hit
                __syncwarp();
                if (win) atomicMin(reinterpret_cast<unsigned *>(&W.best[src].y), id);
                __syncwarp();
                if (win && __float_as_uint(W.best[src].y) == id) W.uv[src] = tri_uv(rb, x);
                __syncwarp();
            }
        }
        __syncwarp();  // the list is read before the next round (or step) writes it
        if (!S.big_leaves) return;
    }
}

// The lane's node: its children's references, which are met (the entry
// distance in e, +inf if not): box_enter's decisions and distances.  Its difference
// and product for each plane, two children to a packed instruction.  Where inv and
// the origin are finite and inv is not zero, a slab's smaller distance is the
// one of the plane that inv's sign names; otherwise distances may be NaN, and
// box_enter's minimum and maximum of the two are taken.  One multiply-add a plane
// with padded offsets, which meets more boxes than box_enter, took 18.0 ms for the
// Cornell frame (these 18.2) and 573 us for 2 M incoherent rays (595).
__device__ __forceinline__ void lane_boxes(const DevScene &S, const LaneRay &st, float (&e)[4], int (&ref)[4]) {
    const char *np = reinterpret_cast<const char *>(S.nodes + st.node);
    float4 nr[3], fr[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        nr[i] = __ldg(reinterpret_cast<const float4 *>(np + st.near[i]));
        fr[i] = __ldg(reinterpret_cast<const float4 *>(np + (48 + 32 * i) - st.near[i]));
    }
    const int4 rf = __ldg(reinterpret_cast<const int4 *>(np + 96));
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float2 o = make_float2(st.neg_org[i], st.neg_org[i]), v = make_float2(st.inv[i], st.inv[i]);
        auto distances = [&](float4 &p) {
            const float2 a = __fmul2_rn(__fadd2_rn(make_float2(p.x, p.y), o), v);
            const float2 b = __fmul2_rn(__fadd2_rn(make_float2(p.z, p.w), o), v);
            p = make_float4(a.x, a.y, b.x, b.y);
        };
        distances(nr[i]);
        distances(fr[i]);
    }
    if (st.odd) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const float4 a = nr[i], b = fr[i];
            nr[i] = make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z), fminf(a.w, b.w));
            fr[i] = make_float4(fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z), fmaxf(a.w, b.w));
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float te = fmaxf(fmaxf(f4(nr[0], j), f4(nr[1], j)), fmaxf(f4(nr[2], j), st.tmin));
        const float tx = fminf(fminf(f4(fr[0], j), f4(fr[1], j)), fminf(f4(fr[2], j), st.tmax));
        ref[j] = i4(rf, j);
        e[j] = te <= __fmul_rn(tx, 1.0000004f) && ref[j] != kNoChild ? te : INFINITY;
    }
}

// One BVH node for every lane with a ray (have), all lanes of the warp
// together.  Returns true when the lane's traversal is over.
template <bool kAny>
__device__ __forceinline__ bool warp_step(const DevScene &S, LaneRay &st, WarpTrav &W, int *deep, int lane,
                                          bool have) {
    float e[4] = {INFINITY, INFINITY, INFINITY, INFINITY};
    int ref[4] = {0, 0, 0, 0};
    if (have) lane_boxes(S, st, e, ref);
    bool leaf[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        leaf[j] = e[j] != INFINITY && ref[j] < 0;
        if (ref[j] < 0) e[j] = INFINITY;
    }
    warp_leaves<kAny>(S, W, lane, leaf, ref);
    if (!have) return false;
    if (kAny) {
        if (__float_as_uint(W.best[lane].y) != PG_NO_HIT) return true;
    } else {
        st.tmax = W.best[lane].x;
        // nearest first, ties by slot (neighbours exchanged, as trav_step's insertion sort)
        auto order = [&](int a, int b) {
            if (e[a] > e[b]) {
                const float x = e[a];
                e[a] = e[b];
                e[b] = x;
                const int y = ref[a];
                ref[a] = ref[b];
                ref[b] = y;
            }
        };
        order(0, 1);
        order(1, 2);
        order(2, 3);
        order(0, 1);
        order(1, 2);
        order(0, 1);
    }
    // the first met child is next, the others are pushed so the following one is on top
    if (kAny) {
        // slot order: close the gaps
#pragma unroll
        for (int pass = 3; pass > 0; --pass)
#pragma unroll
            for (int j = 0; j < pass; ++j) {
                const bool gap = e[j] == INFINITY;
                e[j] = gap ? e[j + 1] : e[j];
                ref[j] = gap ? ref[j + 1] : ref[j];
                e[j + 1] = gap ? INFINITY : e[j + 1];
            }
    }
    const int n = (e[0] != INFINITY) + (e[1] != INFINITY) + (e[2] != INFINITY) + (e[3] != INFINITY);
    int next = ref[0];
    if (st.sp + 3 <= kSharedStack) {
        if (n > 1) {
            int *top = &W.stack[st.sp + n - 2][lane];
            top[0] = ref[1];
            if (n > 2) top[-32] = ref[2];
            if (n > 3) top[-64] = ref[3];
        }
        st.sp += n - 1;
        if (n == 0) {
            if (st.sp < 0) return true;
            next = W.stack[st.sp][lane];
        }
    } else if (n > 0) {
        if (n > 3) lane_push(st, W, deep, lane, ref[3]);
        if (n > 2) lane_push(st, W, deep, lane, ref[2]);
        if (n > 1) lane_push(st, W, deep, lane, ref[1]);
    } else {
        next = lane_pop(st, W, deep, lane);
    }
    st.node = next;
    return false;
}

// The lane's closest hit after its traversal.
__device__ __forceinline__ pg_hit lane_hit(const WarpTrav &W, int lane) {
    pg_hit h;
    h.t = W.best[lane].x;
    h.u = W.uv[lane].x;
    h.v = W.uv[lane].y;
    h.prim = __float_as_uint(W.best[lane].y);
    return h;
}

}  // namespace pg

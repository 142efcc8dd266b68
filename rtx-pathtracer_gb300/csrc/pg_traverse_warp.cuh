// pg_traverse_warp.cuh - warp-cooperative BVH traversal: each lane walks its
// own ray down the four-wide BVH, the warp tests the rays' leaf triangles
// together.
//
// Why: with one ray per lane and each lane testing its own leaves, a warp
// instruction of the triangle test had 6-7 lanes active (a step meets about one
// triangle per ray on average, but the slowest lane meets ten), and every
// lane's node loads touch a cache line of their own.  Here a step appends its
// (ray, triangle) pairs to a list in shared memory and the 32 lanes take the
// pairs in turn, so the test runs with nearly full warps and neighbouring lanes
// read neighbouring triangles of one leaf.
//
// The hit is the one trav_step finds, bit for bit: a step tests the same boxes
// against the best t at its start and the same triangles (every triangle of
// every leaf whose box is met), visits inner children in the same order, and the
// closest hit is the least (t, id) of the accepted ones, whatever the order they
// are tested in.  trav_step stays for rays counted one by one and for single
// rays inside divergent code.
#pragma once

#include "pg_traverse.cuh"

namespace pg {

constexpr unsigned kFullWarp = 0xffffffffu;
constexpr int kPairsPerLane = 16;                  // four leaves of four triangles per round
constexpr int kPairBits = 27;                      // triangle index of a packed pair; the ray's lane above
constexpr uint32_t kMaxPairTris = 1u << kPairBits;
constexpr int kSharedStack = 8;                    // stack entries per lane in shared memory, deeper ones local

// One warp's shared memory.
struct WarpTrav {
    uint32_t pair[32 * kPairsPerLane];  // (lane << kPairBits) | triangle, in lane order
    int stack[kSharedStack][32];
    float t[32];                        // best t of each lane's ray
    uint32_t id[32];                    // its primitive (any hit: PG_NO_HIT until occluded)
    float u[32], v[32];
};

// A lane's ray during a traversal.  The best primitive and its barycentrics
// are in the warp's shared memory.
struct LaneRay {
    RayPre r;
    float tmin, tmax;  // tmax: best t so far for closest-hit queries
    int node, sp;
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
    st.r = ray_setup(o, d);
    st.tmin = tmin;
    st.tmax = tmax;
    st.node = 0;
    st.sp = 0;
    uint32_t id = PG_NO_HIT;
    for (uint32_t i = 0; i < S.n_spheres; ++i) {
        float t;
        if (sphere_intersect(st.r, S.spheres[i], tmin, st.tmax, t)) {
            id = PG_SPHERE_BIT | i;
            if (kAny) break;
            st.tmax = t;
        }
    }
    W.t[lane] = st.tmax;
    W.id[lane] = id;
    W.u[lane] = W.v[lane] = 0.0f;
    return kAny && id != PG_NO_HIT;
}

// Tests the triangles [first[j], first[j] + cnt[j]) of every lane's leaves
// against that lane's ray, all lanes of the warp together.  Updates W.t, W.id,
// W.u, W.v (closest: the least (t, id); any: W.id of an occluded ray) and the
// lane's st.tmax.
template <bool kAny>
__device__ __forceinline__ void warp_leaves(const DevScene &S, LaneRay &st, WarpTrav &W, int lane, int (&first)[4],
                                            int (&cnt)[4]) {
    while (__any_sync(kFullWarp, (cnt[0] | cnt[1] | cnt[2] | cnt[3]) != 0)) {
        // this round's pairs: up to four triangles of each leaf
        int c = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) c += min(cnt[j], 4);
        int incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFullWarp, incl, o);
            if (lane >= o) incl += y;
        }
        const int total = __shfl_sync(kFullWarp, incl, 31);
        uint32_t at = (uint32_t)(incl - c);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = min(cnt[j], 4);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k < n) W.pair[at + k] = ((uint32_t)lane << kPairBits) | (uint32_t)(first[j] + k);
            at += (uint32_t)n;
            first[j] += n;
            cnt[j] -= n;
        }
        __syncwarp();
        for (int base = 0; base < total; base += 32) {
            const bool on = base + lane < total;
            const uint32_t pr = on ? W.pair[base + lane] : 0u;
            const int src = (int)(pr >> kPairBits);
            const uint32_t ti = pr & (kMaxPairTris - 1u);
            RayPre r;
#pragma unroll
            for (int i = 0; i < 3; ++i) r.org[i] = __shfl_sync(kFullWarp, st.r.org[i], src);
            r.Sx = __shfl_sync(kFullWarp, st.r.Sx, src);
            r.Sy = __shfl_sync(kFullWarp, st.r.Sy, src);
            r.Sz = __shfl_sync(kFullWarp, st.r.Sz, src);
            const int kk = __shfl_sync(kFullWarp, st.r.kx | (st.r.ky << 2) | (st.r.kz << 4), src);
            r.kx = kk & 3;
            r.ky = (kk >> 2) & 3;
            r.kz = kk >> 4;
            const float tmin = __shfl_sync(kFullWarp, st.tmin, src);
            const float bt = W.t[src];
            const uint32_t bid = W.id[src];
            float t = 0.0f, u = 0.0f, v = 0.0f;
            uint32_t id = 0;
            bool acc = false;
            if (on) {
                const float4 v0 = __ldg(&S.tris[3 * (size_t)ti]), v1 = __ldg(&S.tris[3 * (size_t)ti + 1]),
                             v2 = __ldg(&S.tris[3 * (size_t)ti + 2]);
                id = __float_as_uint(v0.w);
                const uint32_t tex = __float_as_uint(v1.w);
                // one ulp above the best t, so an equal t is seen and the lower id wins
                const float lim = (kAny || bid == PG_NO_HIT) ? bt : __uint_as_float(__float_as_uint(bt) + 1u);
                acc = tri_intersect(r, v0, v1, v2, tmin, lim, t, u, v) &&
                      (kAny || t < bt || (t == bt && id < bid)) &&
                      (tex == 0u || alpha_keep(S, r.org[0], id, tex, u, v, t));
            }
            if (!__any_sync(kFullWarp, acc)) continue;
            if (kAny) {
                if (acc) W.id[src] = id;
                __syncwarp();
            } else {
                // t > tmin >= 0: its bits order as the numbers do
                if (acc) atomicMin(reinterpret_cast<unsigned *>(&W.t[src]), __float_as_uint(t));
                __syncwarp();
                const bool win = acc && W.t[src] == t;
                if (win && t < bt) W.id[src] = PG_NO_HIT;  // closer than every earlier hit
                __syncwarp();
                if (win) atomicMin(&W.id[src], id);
                __syncwarp();
                if (win && W.id[src] == id) {
                    W.u[src] = u;
                    W.v[src] = v;
                }
                __syncwarp();
            }
        }
        __syncwarp();  // the pairs are read before the next round (or step) writes them
    }
    if (!kAny) st.tmax = W.t[lane];
}

// One BVH node for every lane with a ray (have), all lanes of the warp
// together.  Returns true when the lane's traversal is over.
template <bool kAny>
__device__ __forceinline__ bool warp_step(const DevScene &S, LaneRay &st, WarpTrav &W, int *deep, int lane,
                                          bool have) {
    float e[4];
    int first[4], cnt[4], inner[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        e[j] = INFINITY;
        first[j] = cnt[j] = 0;
        inner[j] = -1;
    }
    if (have) {
        const DevBvhNode *np = S.nodes + st.node;
        const float4 lox = __ldg(&np->lox), loy = __ldg(&np->loy), loz = __ldg(&np->loz);
        const float4 hix = __ldg(&np->hix), hiy = __ldg(&np->hiy), hiz = __ldg(&np->hiz);
        const int4 child = __ldg(&np->child), count = __ldg(&np->count);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            e[j] = box_enter(st.r, f4(lox, j), f4(loy, j), f4(loz, j), f4(hix, j), f4(hiy, j), f4(hiz, j), st.tmin,
                             st.tmax);
            const bool met = e[j] != INFINITY;
            const int n = i4(count, j), c = i4(child, j);
            first[j] = c;
            cnt[j] = met && n > 0 ? n : 0;
            inner[j] = met && n <= 0 ? c : -1;
            if (inner[j] < 0) e[j] = INFINITY;
        }
    }
    warp_leaves<kAny>(S, st, W, lane, first, cnt);
    if (!have) return false;
    if (kAny && W.id[lane] != PG_NO_HIT) return true;
    if (!kAny) {
        // nearest first, ties in slot order: adjacent exchanges keep equal keys in place
#pragma unroll
        for (int pass = 3; pass > 0; --pass)
#pragma unroll
            for (int j = 0; j < pass; ++j)
                if (e[j] > e[j + 1]) {
                    const float x = e[j];
                    e[j] = e[j + 1];
                    e[j + 1] = x;
                    const int y = inner[j];
                    inner[j] = inner[j + 1];
                    inner[j + 1] = y;
                }
    }
    // the first child is next, the others are pushed so the next nearest is on top
    int next = -1;
#pragma unroll
    for (int j = 3; j >= 0; --j)
        if (inner[j] >= 0) {
            if (next >= 0) lane_push(st, W, deep, lane, next);
            next = inner[j];
        }
    if (next < 0) {
        if (st.sp == 0) return true;
        next = lane_pop(st, W, deep, lane);
    }
    st.node = next;
    return false;
}

}  // namespace pg

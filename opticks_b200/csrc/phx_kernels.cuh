// phx_kernels.cuh : device-side scene description, closest-hit traversal and the per-photon
// bounce loop shared by the plain, batched and adjoint kernels.
#pragma once
#include "phx_pod.h"
#include "phx_vec.cuh"
#include "phx_csg.cuh"
#include "phx_physics.cuh"

#define PHX_BVH_STACK 48
// leaf steps are taken when leaf-ready lanes x this weight >= node-ready lanes (or no node work is left)
#ifndef PHX_TRACE_LEAF_WEIGHT
#define PHX_TRACE_LEAF_WEIGHT 1
#endif

struct PhxScene {
    const phx_bvh4_node* bvh;   // root at 0
    const phx_leaf* leaves;     // the global leaves (tested first by every ray: boxes spanning much of the
                                // scene), then the hierarchy's
    const float4* leaf_sph;     // world bounding sphere (centre, radius) of each
    const float4* global_q;     // two rows per global leaf: parameters of a plain leaf under the identity
                                // instance, and its typecode (word 0; 0: any other leaf)
    const float4* inst_inv;     // (num_inst*4) rows of the world->object 4x4 (row-vector convention)
    PhxCsgCtx csg;
    float4 cull;                // ball no hierarchy leaf reaches: centre xyz, radius^2 (0: none)
    int num_global;
    unsigned kind_mask;         // bits of phx_leaf.node_offset that hold the leaf's kind (PHX_LEAF_KIND)
    int bvh_empty;              // no hierarchy leaves
    int empty;                  // no leaves at all
};

struct PhxBest {
    float t;
    int leaf;                   // index into the scene's leaves; < 0 : none
    float3 n;                   // object-frame normal
};

// Can the ray segment (tmin, tmax) meet the ball (centre, radius)?  The radius is padded on the
// host beyond FP32 error, so a false answer never hides a hit of the leaf inside the ball.
PHX_D bool phx_ball_overlaps(const float4 b, const float3& o, const float3& d, float tmin, float tmax)
{
    const float3 oc = make_float3(b.x - o.x, b.y - o.y, b.z - o.z);
    const float dd = dot(d, d);
    const float tc = dot(oc, d) / dd;
    const float3 q = oc - tc * d;
    if (dot(q, q) > b.w * b.w) return false;
    const float h = b.w * rsqrtf(dd);
    return tc + h >= tmin && tc - h <= tmax;
}

// No hit of what the ball (centre, radius) holds can lie on the ray beyond tmin: the line passes it by, or
// it lies behind the origin.  The margin grows with the origin's distance as the FP32 error of the
// leaves' own discriminants does, a hundred times wider.  False for any NaN, and where the products of a
// very long or short direction leave the FP32 range (the leaves' own, smaller products may not).
PHX_D bool phx_ball_missed(const float4 b, const float3& o, const float3& d, float tmin)
{
    const float3 oc = make_float3(b.x - o.x, b.y - o.y, b.z - o.z);
    const float dd = dot(d, d), bd = dot(oc, d), cc = dot(oc, oc);
    const float rr = b.w * b.w + 1e-5f * cc;
    const float cd = cc * dd;
    return (dd > 1e-30f && cd < 3e38f && cd - bd * bd > rr * dd) || (bd < 0.f && tmin >= 0.f && cc > rr);
}

// IS program of CSGOptiX/CSGOptiX7.cu:896-967 for one (instance, prim) leaf: object-frame
// intersect_prim, keep the closest hit.  `li` indexes the scene's leaves, L is that record.
// The usual prims (PHX_KIND_LEAF, PHX_KIND_TREE3) are evaluated inline where PHX_CV_INLINE says so: the
// kind comes with the leaf, so the chain of dependent node loads that finds it out and the calls per
// leaf go away.  Identity and lposcost of the hit are looked up once a ray (phx_best_prd), not at every
// closer hit.  With the plain global leaves below: 10M-photon detector event 13.15 -> 12.27 ms, 2^20 rays
// through the detector 443 -> 402 us.
template <int CV>
PHX_D void phx_test_leaf(const PhxScene& S, const int li, const int4 L, const float3& o, const float3& d, float tmin, PhxBest& B,
                         unsigned& status)
{
    const float4* q = S.inst_inv + 4 * L.x;
    const float4 m[4] = { __ldg(q + 0), __ldg(q + 1), __ldg(q + 2), __ldg(q + 3) };
    const float3 lo = fx_point(m, o);
    const float3 ld = fx_dir(m, d);
    const int root = (int)((unsigned)L.y & ~S.kind_mask);
    float4 is;
    bool valid;
    if constexpr (PHX_CV_INLINE(CV)) {
        const unsigned kind = ((unsigned)L.y & S.kind_mask) >> PHX_LEAF_KIND;
        if (kind >= PHX_KIND_TREE3) {
            is = intersect_tree3_fast(S.csg.node, S.csg.itra, root, kind - PHX_KIND_TREE3 + 1u, tmin, lo, ld, status);
            valid = is.w > 0.f;
        } else if (kind == PHX_KIND_LEAF) {
            is = leaf_fast(S.csg.node, S.csg.itra, root, tmin, lo, ld);
            valid = is.w > tmin;
        } else if constexpr ((CV & PHX_CV_PLAIN) != 0) {
            return;
        } else {
            const PhxPrimHit h = intersect_prim_any<CV>(S.csg.node, S.csg.itra, S.csg.plan, root, tmin, lo, ld);
            is = h.is;
            valid = h.valid;
            status |= h.status;
        }
    } else {
        valid = intersect_prim<CV>(is, S.csg, root, tmin, lo, ld, status);
    }
    // OptiX's interval rule: a report outside [tmin, tmax] is ignored (a convexpolyhedron wholly
    // behind the ray reports valid with t = 0, CSG/csg_intersect_leaf_convexpolyhedron.h:85-101)
    if (valid && is.w >= tmin && is.w < B.t) {
        B.t = is.w;
        B.leaf = li;
        B.n = make_float3(is.x, is.y, is.z);
    }
}

// the hierarchy leaves [first, first + count) (counted from the first hierarchy leaf)
template <int CV>
PHX_D void phx_test_range(const PhxScene& S, int first, int count, const float3& o, const float3& d, float tmin, PhxBest& B, unsigned& status)
{
#pragma unroll 1
    for (int li = S.num_global + first; li < S.num_global + first + count; li++) {
        const int4 L = __ldg(reinterpret_cast<const int4*>(S.leaves + li));
        if (phx_ball_overlaps(__ldg(S.leaf_sph + li), o, d, tmin, B.t)) phx_test_leaf<CV>(S, li, L, o, d, tmin, B, status);
    }
}

// Global leaf g if it has a parameter row (false: it has none)
template <bool POLISH>
PHX_D bool phx_test_plain_global(const PhxScene& S, int g, const float3& o, const float3& d, float tmin, PhxBest& B)
{
    const float4 q0 = __ldg(S.global_q + 2 * g);
    const unsigned tc = __float_as_uint(__ldg(&S.global_q[2 * g + 1].x));
    if (tc != PHX_CSG_SPHERE && tc != PHX_CSG_BOX3) return false;
    float4 is;
    bool valid;
    if (tc == PHX_CSG_SPHERE) valid = leaf_sphere<POLISH>(is, q0, tmin, o, d);
    else { is = leaf_box3(q0, tmin, o, d); valid = is.w > tmin; }
    if (valid && is.w < B.t) {
        B.t = is.w;
        B.leaf = g;
        B.n = make_float3(is.x, is.y, is.z);
    }
    return true;
}

// The global leaves, in order.  Plain spheres and boxes of the world solid (identity instance, no
// node transform, no complement: the usual volumes around a detector) are solved from their parameter
// row, without the instance transform, the node loads and the dispatch of the general leaf.
template <int CV>
PHX_D void phx_test_globals(const PhxScene& S, const float3& o, const float3& d, float tmin, PhxBest& B, unsigned& status)
{
#pragma unroll 1
    for (int g = 0; g < S.num_global; g++) {
        if (!phx_test_plain_global<PHX_CV_P(CV)>(S, g, o, d, tmin, B)) {
            const int4 L = __ldg(reinterpret_cast<const int4*>(S.leaves + g));
            if (phx_ball_overlaps(__ldg(S.leaf_sph + g), o, d, tmin, B.t)) phx_test_leaf<CV>(S, g, L, o, d, tmin, B, status);
        }
    }
}

// A ray's slab constants: reciprocal direction and -origin/direction per axis, each as a pair of
// equal floats (the operand form of the packed FP32 instructions), and the byte offset of the box
// side the ray meets first in a node's (lo, hi) row pair of the axis.
struct PhxSlabs {
    unsigned long long ix, iy, iz, ox, oy, oz;
    unsigned nx, ny, nz;
};

PHX_D unsigned long long phx_pair(float a, float b)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
PHX_D void phx_unpair(unsigned long long v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
PHX_D unsigned long long phx_fma2(unsigned long long a, unsigned long long b, unsigned long long c)
{
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
PHX_D float phx_max3(float a, float b, float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
PHX_D float phx_min3(float a, float b, float c)
{
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// zero direction components are nudged, so every reciprocal is finite
PHX_D void phx_ray_slabs(const float3& o, const float3& d, PhxSlabs& R)
{
    const float3 dd = make_float3(fabsf(d.x) < 1e-30f ? copysignf(1e-30f, d.x) : d.x,
                                  fabsf(d.y) < 1e-30f ? copysignf(1e-30f, d.y) : d.y,
                                  fabsf(d.z) < 1e-30f ? copysignf(1e-30f, d.z) : d.z);
    const float3 inv = make_float3(1.f / dd.x, 1.f / dd.y, 1.f / dd.z);
    R.ix = phx_pair(inv.x, inv.x); R.iy = phx_pair(inv.y, inv.y); R.iz = phx_pair(inv.z, inv.z);
    const float3 oi = make_float3(-o.x * inv.x, -o.y * inv.y, -o.z * inv.z);
    R.ox = phx_pair(oi.x, oi.x); R.oy = phx_pair(oi.y, oi.y); R.oz = phx_pair(oi.z, oi.z);
    R.nx = (__float_as_uint(inv.x) >> 31) << 4;
    R.ny = (__float_as_uint(inv.y) >> 31) << 4;
    R.nz = (__float_as_uint(inv.z) >> 31) << 4;
}

// Visit BVH4 node ni: slab-test its four children against [tmin, tmax] and push the hit ones
// (inner nodes and leaf ranges) far-to-near, so that the nearest is taken next.  A visit is bound by
// issue and by its L1 loads (12 a ray on the detector's water rays), so it is kept short: the near and
// far side of each axis are chosen by address instead of by min and max, two children share each
// multiply-add (packed FP32), three-input min and max close the interval, and the pushed distance is the
// sort key itself.  10M-photon detector event 13.77 -> 13.15 ms against four unpacked slab tests.
PHX_D void phx_visit_node(const PhxScene& S, int ni, const PhxSlabs& R, float tmin, float tmax, int2* stk, int& sp, unsigned& status)
{
    const char* nb = reinterpret_cast<const char*>(S.bvh + ni);
    const ulonglong2 nx = __ldg(reinterpret_cast<const ulonglong2*>(nb + R.nx));
    const ulonglong2 fx = __ldg(reinterpret_cast<const ulonglong2*>(nb + (R.nx ^ 16u)));
    const ulonglong2 ny = __ldg(reinterpret_cast<const ulonglong2*>(nb + 32 + R.ny));
    const ulonglong2 fy = __ldg(reinterpret_cast<const ulonglong2*>(nb + 32 + (R.ny ^ 16u)));
    const ulonglong2 nz = __ldg(reinterpret_cast<const ulonglong2*>(nb + 64 + R.nz));
    const ulonglong2 fz = __ldg(reinterpret_cast<const ulonglong2*>(nb + 64 + (R.nz ^ 16u)));
    const int4 ch = __ldg(reinterpret_cast<const int4*>(nb + 96));
    const int cha[4] = { ch.x, ch.y, ch.z, ch.w };
    unsigned key[4];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        float x0[2], x1[2], y0[2], y1[2], z0[2], z1[2];
        phx_unpair(phx_fma2(h ? nx.y : nx.x, R.ix, R.ox), x0[0], x0[1]);
        phx_unpair(phx_fma2(h ? fx.y : fx.x, R.ix, R.ox), x1[0], x1[1]);
        phx_unpair(phx_fma2(h ? ny.y : ny.x, R.iy, R.oy), y0[0], y0[1]);
        phx_unpair(phx_fma2(h ? fy.y : fy.x, R.iy, R.oy), y1[0], y1[1]);
        phx_unpair(phx_fma2(h ? nz.y : nz.x, R.iz, R.oz), z0[0], z0[1]);
        phx_unpair(phx_fma2(h ? fz.y : fz.x, R.iz, R.oz), z1[0], z1[1]);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int c = 2 * h + q;
            const float tnear = phx_max3(fmaxf(x0[q], y0[q]), z0[q], tmin);
            const float tfar = phx_min3(fminf(x1[q], y1[q]), z1[q], tmax);
            // slab arithmetic slack: boxes are padded on the host, and a relative slack here.
            // key: the near distance's bits (not negative: they order like the floats) with the
            // child slot in the two low bits, all ones for a missed child (sorts last)
            const unsigned k = ((unsigned)max(__float_as_int(tnear), 0) & 0x7ffffffcu) | (unsigned)c;
            key[c] = cha[c] != 0 && tnear <= fmaf(tfar, 1.00001f, 1e-4f) ? k : 0xffffffffu;
        }
    }
    unsigned k0 = key[0], k1 = key[1], k2 = key[2], k3 = key[3], t;
    t = min(k0, k1); k1 = max(k0, k1); k0 = t;
    t = min(k2, k3); k3 = max(k2, k3); k2 = t;
    t = min(k0, k2); k2 = max(k0, k2); k0 = t;
    t = min(k1, k3); k3 = max(k1, k3); k1 = t;
    t = min(k1, k2); k2 = max(k1, k2); k1 = t;
    const unsigned ks[4] = { k0, k1, k2, k3 };
#pragma unroll
    for (int j = 3; j >= 0; j--) {
        const unsigned k = ks[j];
        if (k == 0xffffffffu) continue;
        if (sp >= PHX_BVH_STACK) { status |= PHX_STATUS_BVH_STACK; continue; }
        // the pushed distance is the key's, at most a few ulp below the near distance (tmin bounds
        // it where that is negative), so that no entry is dropped too early
        const int child = k & 2u ? (k & 1u ? cha[3] : cha[2]) : (k & 1u ? cha[1] : cha[0]);
        stk[sp] = make_int2(child, k < 4u ? __float_as_int(tmin) : (int)(k & ~3u));
        sp++;
    }
}

// The segment [tmin, t] lies inside the ball no hierarchy leaf reaches: skip the hierarchy.
PHX_D bool phx_culled(const PhxScene& S, const float3& o, const float3& d, float tmin, float t)
{
    if (!(S.cull.w > 0.f)) return false;
    const float3 c = make_float3(S.cull.x, S.cull.y, S.cull.z);
    const float3 p0 = o + tmin * d - c;
    const float3 p1 = o + t * d - c;
    return dot(p0, p0) < S.cull.w && dot(p1, p1) < S.cull.w;
}

// PRD of a closest hit (CH program CSGOptiX/CSGOptiX7.cu:776-874, lposcost of the IS program), or of a miss
PHX_D void phx_best_prd(const PhxScene& S, const PhxBest& B, const float3& o, const float3& d, PhxPRD& prd)
{
    if (B.leaf < 0) {
        prd.gp_bd = 0xffffffffu;
        prd.ii_id = 0xffffffffu;
        prd.normal = make_float3(0.f, 0.f, 0.f);
        prd.distance = 0.f;
        prd.lposcost = 0.f;
        return;
    }
    const int4 L = __ldg(reinterpret_cast<const int4*>(S.leaves + B.leaf));
    const float4* q = S.inst_inv + 4 * L.x;
    const float4 m[4] = { __ldg(q + 0), __ldg(q + 1), __ldg(q + 2), __ldg(q + 3) };
    prd.normal = fx_normal(m, B.n);
    prd.distance = B.t;
    const float3 lpos = fx_at(fx_point(m, o), B.t, fx_dir(m, d));
    prd.lposcost = lpos.z / sqrtf(fx_mix(lpos.x, lpos.x, lpos.y, lpos.y, lpos.z, lpos.z));
    prd.gp_bd = (unsigned)L.z;
    prd.ii_id = (unsigned)L.w;
}

// Closest hit over all (instance, prim) leaves: restates optixTrace over the IAS with the
// IS program CSGOptiX/CSGOptiX7.cu:896-967 (object-frame intersect_prim, lposcost) and the
// CH program :776-874 (object->world normal, iindex<<16|identity, globalPrimIdx<<16|boundary).
// The global leaves are tested first, then the hierarchy is traversed unless the segment
// [tmin, closest so far] lies inside the ball no hierarchy leaf reaches.
// Returns false for a miss (prd boundary 0xffff).
template <int CV>
PHX_D bool phx_trace(const PhxScene& S, const float3& o, const float3& d, float tmin, float tmax, PhxPRD& prd, unsigned& status)
{
    prd.gp_bd = 0xffffffffu;
    prd.ii_id = 0xffffffffu;
    prd.normal = make_float3(0.f, 0.f, 0.f);
    prd.distance = 0.f;
    prd.lposcost = 0.f;
    if (S.empty) return false;
    PhxBest B;
    B.t = tmax;
    B.leaf = -1;
    B.n = make_float3(0.f, 0.f, 0.f);
    phx_test_globals<CV>(S, o, d, tmin, B, status);
    if (!S.bvh_empty && !phx_culled(S, o, d, tmin, B.t)) {
        PhxSlabs R;
        phx_ray_slabs(o, d, R);
        int2 stk[PHX_BVH_STACK];     // node or leaf range, near distance bits
        int sp = 1;
        stk[0] = make_int2(0, __float_as_int(tmin));
        // Each step the lanes of the warp that traverse together vote: either the lanes whose next
        // entry is an inner node visit it, or the lanes whose next entry is a leaf range test it.
        // Every lane still takes its own entries in its own near-first order; the vote only
        // gathers the expensive leaf tests into steps where many lanes run them.
        const unsigned mask = __activemask();
        for (;;) {
            int2 top = make_int2(0, 0);
            while (sp > 0 && __int_as_float((top = stk[sp - 1]).y) > B.t) sp--;
            const bool leaf_top = sp > 0 && top.x < 0;
            const unsigned want_leaf = __ballot_sync(mask, leaf_top);
            const unsigned want_node = __ballot_sync(mask, sp > 0 && !leaf_top);
            if (!(want_leaf | want_node)) break;
            const bool leaf_step = want_node == 0u || __popc(want_leaf) * PHX_TRACE_LEAF_WEIGHT >= __popc(want_node);
            if (sp == 0 || leaf_top != leaf_step) continue;
            sp--;
            const int ni = top.x;
            if (leaf_step) {
                const int enc = -ni - 1;
                phx_test_range<CV>(S, enc >> 3, (enc & 7) + 1, o, d, tmin, B, status);
                continue;
            }
            phx_visit_node(S, ni, R, tmin, B.t, stk, sp, status);
        }
    }
    phx_best_prd(S, B, o, d, prd);
    return B.leaf >= 0;
}

// A stream of rays traced by persistent warps.  Windows of 32 rays are taken first through the global
// leaves with all lanes (their PRDs are stored at once), and the rays that must walk the hierarchy are
// queued; lanes whose walk has ended take the next queued rays once `refill_idle` of them wait.  So the
// coherent part never runs in the few lanes that happen to be free, rays the cull ball keeps out of
// the hierarchy never hold a lane among walking ones, and a warp does not wait for its longest walk.
// Same arithmetic and order per ray as phx_trace.  2^20 rays anywhere in the detector (a quarter of them
// walk): 402 -> 160 us against one thread per ray (122 us in the plain variant, 16 warps per SM); a
// 1M-photon event's third round, where every ray walks, runs at 16.8 lanes instead of 12.7.
//   next()                       the warp's next window (its first ray; < 0: none left), warp-uniform
//   tag(base, lane, tag)         the lane's ray of a window: false past the end
//   load(tag, o, d, tmin)        its origin, direction and interval start
//   store(tag, prd)
// `queue`: 64 entries of the warp's own in shared memory (tag, closest hit so far).
template <int CV, class NEXT, class TAG, class LOAD, class STORE>
PHX_D void phx_trace_stream(const PhxScene& S, float tmax, int refill_idle, int2* queue, unsigned& status, NEXT next, TAG tag, LOAD load,
                            STORE store)
{
    const unsigned FULL = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned below = (1u << lane) - 1u;
    unsigned waiting = 0u;                // queued rays
    bool drained = false;                 // no window left
    bool has = false;                     // this lane walks a ray
    unsigned s = 0u;
    float3 o = make_float3(0.f, 0.f, 0.f), d = o;
    PhxSlabs R = {};
    float tmin = 0.f;
    PhxBest B;
    B.t = 0.f; B.leaf = -1; B.n = o;
    int2 stk[PHX_BVH_STACK];              // node or leaf range, near distance bits
    int sp = 0;
    for (;;) {
        const unsigned idle = __ballot_sync(FULL, !has);
        if (__popc(idle) >= refill_idle) {
            while (waiting < 32u && !drained) {
                const long long base = next();
                if (base < 0) { drained = true; break; }
                unsigned q;
                bool walk = false;
                float t = 0.f;
                if (tag(base, lane, q)) {
                    float3 qo, qd;
                    float qmin;
                    load(q, qo, qd, qmin);
                    PhxBest G;
                    G.t = tmax; G.leaf = -1; G.n = make_float3(0.f, 0.f, 0.f);
                    phx_test_globals<CV>(S, qo, qd, qmin, G, status);
                    PhxPRD prd;
                    phx_best_prd(S, G, qo, qd, prd);
                    store(q, prd);
                    walk = !S.bvh_empty && !phx_culled(S, qo, qd, qmin, G.t);
                    t = G.t;
                }
                const unsigned m = __ballot_sync(FULL, walk);
                if (walk) queue[waiting + __popc(m & below)] = make_int2((int)q, __float_as_int(t));
                waiting += __popc(m);
                __syncwarp();
            }
            const unsigned take = min((unsigned)__popc(idle), waiting);
            const unsigned rank = __popc(idle & below);
            if (!has && rank < take) {
                const int2 e = queue[waiting - take + rank];
                s = (unsigned)e.x;
                load(s, o, d, tmin);
                phx_ray_slabs(o, d, R);
                B.t = __int_as_float(e.y); B.leaf = -1;
                stk[0] = make_int2(0, __float_as_int(tmin));
                sp = 1;
                has = true;
            }
            waiting -= take;
            __syncwarp();
        }
        // finish the rays whose stacks are empty
        int2 top = make_int2(0, 0);
        if (has) {
            while (sp > 0 && __int_as_float((top = stk[sp - 1]).y) > B.t) sp--;
            if (sp == 0) {
                if (B.leaf >= 0) {
                    PhxPRD prd;
                    phx_best_prd(S, B, o, d, prd);
                    store(s, prd);
                }
                has = false;
            }
        }
        const bool leaf_top = has && top.x < 0;
        const unsigned want_leaf = __ballot_sync(FULL, leaf_top);
        const unsigned want_node = __ballot_sync(FULL, has && !leaf_top);
        if (!(want_leaf | want_node)) {
            if (drained && waiting == 0u) break;
            continue;
        }
        // one step: the lanes whose next entry is a leaf range, or those whose next entry is a node
        const bool leaf_step = want_node == 0u || __popc(want_leaf) * PHX_TRACE_LEAF_WEIGHT >= __popc(want_node);
        if (!has || leaf_top != leaf_step) continue;
        sp--;
        const int ni = top.x;
        if (leaf_step) {
            const int enc = -ni - 1;
            phx_test_range<CV>(S, enc >> 3, (enc & 7) + 1, o, d, tmin, B, status);
        } else {
            phx_visit_node(S, ni, R, tmin, B.t, stk, sp, status);
        }
    }
}

struct PhxLoopCfg {
    int max_bounce;
    float max_time;
    float tmin, tmin0, tmax;
    unsigned eps0_mask;
};

PHX_D void seq_add_nibble(unsigned long long* seqhis, unsigned long long* seqbnd, unsigned slot, unsigned flag, unsigned boundary)
{
    const unsigned iseq = slot / 16u;
    const unsigned shift = 4u * (slot - iseq * 16u);
    if (iseq < 2u) {
        const unsigned long long f = (unsigned long long)(__ffs((int)flag) & 0xf);
        const unsigned long long b = (unsigned long long)(boundary & 0xfu);
        if (iseq == 0u) { seqhis[0] |= f << shift; seqbnd[0] |= b << shift; }
        else            { seqhis[1] |= f << shift; seqbnd[1] |= b << shift; }
    }
}

// genstep of photon idx: the last g with off[g] <= idx (empty gensteps are skipped)
PHX_D int phx_find_genstep(const long long* off, int G, long long idx)
{
    int lo = 0, hi = G;   // off[lo] <= idx < off[hi]
    while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (__ldg(off + mid) <= idx) lo = mid; else hi = mid;
    }
    return lo;
}

// Advance a loaded XORWOW state by n steps: v <- M v over GF(2) with M = T^n (phx_rngjump.h), d <- d +
// 362437 n.  M comes as 4-bit group tables (phx_event_table): 40 lookups, each the XOR of up to four
// columns.  Same state as skipahead(n).
PHX_D void phx_rng_jump4(curandStateXORWOW& s, const uint32_t* __restrict__ T, unsigned long long n)
{
    uint32_t o0 = 0u, o1 = 0u, o2 = 0u, o3 = 0u, o4 = 0u;
    const uint32_t in[5] = { s.v[0], s.v[1], s.v[2], s.v[3], s.v[4] };
#pragma unroll 1
    for (int w = 0; w < 5; w++) {
        const uint32_t x = in[w];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const uint32_t* e = T + (size_t)((8 * w + q) * 16 + ((x >> (4 * q)) & 15u)) * PHX_JUMP_COLW;
            const uint4 a = __ldg(reinterpret_cast<const uint4*>(e));
            const uint32_t e4 = __ldg(e + 4);
            o0 ^= a.x; o1 ^= a.y; o2 ^= a.z; o3 ^= a.w; o4 ^= e4;
        }
    }
    s.v[0] = o0; s.v[1] = o1; s.v[2] = o2; s.v[3] = o3; s.v[4] = o4;
    s.d += (unsigned int)((362437ull * n) & 0xffffffffull);
}

// The event's jump matrix as 4-bit group tables, by one block of at least PHX_JUMP_THREADS threads.
// The event index is taken as hex digits: D holds, for digit position g and value v in 1..15, the
// group tables of T^(skip v 16^g) (k_jump_digits), and M is their product.  Four threads work on a
// column: the first digit's column is a table entry, each further digit is 40 lookups, ten a thread.
// `col`: 160 x 5 words of shared memory.  Bound by the latency of one dependent round of L2 lookups a
// digit: event indices up to 4095 take 5 us where composing the matrix column by column took 48.
#define PHX_JUMP_THREADS 640
PHX_D void phx_event_table(unsigned long long event, const uint32_t* __restrict__ D, uint32_t* T, uint32_t* col)
{
    const int t = threadIdx.x;
    if (t < PHX_JUMP_THREADS) {
        const int c = t >> 2, part = t & 3;
        uint32_t v[5] = { 0u, 0u, 0u, 0u, 0u };
        v[c >> 5] = 1u << (c & 31);
        bool first = true;
        for (int g = 0; g < PHX_JUMP_DIGITS; g++) {
            const unsigned x = (unsigned)(event >> (4 * g)) & 15u;
            if (!x) continue;
            const uint32_t* E = D + (size_t)(15 * g + (int)x - 1) * PHX_JUMP_NIBW;
            if (first) {
                const uint32_t* e = E + (size_t)((c >> 2) * 16 + (1 << (c & 3))) * PHX_JUMP_COLW;
                const uint4 a = __ldg(reinterpret_cast<const uint4*>(e));
                v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = __ldg(e + 4);
                first = false;
                continue;
            }
            uint32_t o[5] = { 0u, 0u, 0u, 0u, 0u };
#pragma unroll
            for (int w = 0; w < 5; w++)
#pragma unroll
                for (int h = 0; h < 2; h++) {            // groups 2 part and 2 part + 1 of word w
                    const int q = 2 * part + h;
                    const uint32_t* e = E + (size_t)((8 * w + q) * 16 + (int)((v[w] >> (4 * q)) & 15u)) * PHX_JUMP_COLW;
                    const uint4 a = __ldg(reinterpret_cast<const uint4*>(e));
                    const uint32_t e4 = __ldg(e + 4);
                    o[0] ^= a.x; o[1] ^= a.y; o[2] ^= a.z; o[3] ^= a.w; o[4] ^= e4;
                }
#pragma unroll
            for (int w = 0; w < 5; w++) {
                o[w] ^= __shfl_xor_sync(0xffffffffu, o[w], 1);
                v[w] = o[w] ^ __shfl_xor_sync(0xffffffffu, o[w], 2);
            }
        }
        if (part == 0)
            for (int w = 0; w < 5; w++) col[5 * c + w] = v[w];
    }
    __syncthreads();
    if (t < PHX_JUMP_BITS / 4 * 16) {
        const int g = t >> 4, k = t & 15;
        uint32_t o[5] = { 0u, 0u, 0u, 0u, 0u };
        for (int b = 0; b < 4; b++) {
            const uint32_t m = 0u - ((unsigned)(k >> b) & 1u);
            for (int w = 0; w < 5; w++) o[w] ^= col[5 * (4 * g + b) + w] & m;
        }
        uint4* dst = reinterpret_cast<uint4*>(T + (size_t)t * PHX_JUMP_COLW);
        dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
        dst[1] = make_uint4(o[4], 0u, 0u, 0u);
    }
}

// the digit tables of phx_event_table from the powers P_k = T^(skip 2^k): block 15 g + v - 1 composes
// the columns of T^(skip v 16^g) (once per engine)
__global__ void __launch_bounds__(PHX_JUMP_THREADS) k_jump_digits(const uint32_t* __restrict__ P, uint32_t* D)
{
    __shared__ uint32_t col[PHX_JUMP_BITS * 5];
    const int g = blockIdx.x / 15, x = blockIdx.x % 15 + 1, t = threadIdx.x;
    if (t < PHX_JUMP_BITS) {
        uint32_t v[5] = { 0u, 0u, 0u, 0u, 0u };
        v[t >> 5] = 1u << (t & 31);
        for (int k = 0; k < 4; k++) {
            if (!((x >> k) & 1)) continue;
            const uint32_t* Pk = P + (size_t)(4 * g + k) * PHX_JUMP_MATW;
            uint32_t o[5] = { 0u, 0u, 0u, 0u, 0u };
            for (int bit = 0; bit < PHX_JUMP_BITS; bit++) {
                const uint32_t m = 0u - ((v[bit >> 5] >> (bit & 31)) & 1u);
                for (int q = 0; q < 5; q++) o[q] ^= Pk[bit * PHX_JUMP_COLW + q] & m;
            }
            for (int q = 0; q < 5; q++) v[q] = o[q];
        }
        for (int q = 0; q < 5; q++) col[5 * t + q] = v[q];
    }
    __syncthreads();
    if (t < PHX_JUMP_BITS / 4 * 16) {
        uint32_t o[5] = { 0u, 0u, 0u, 0u, 0u };
        for (int b = 0; b < 4; b++) {
            const uint32_t m = 0u - ((unsigned)((t & 15) >> b) & 1u);
            for (int w = 0; w < 5; w++) o[w] ^= col[5 * (4 * (t >> 4) + b) + w] & m;
        }
        uint32_t* dst = D + (size_t)blockIdx.x * PHX_JUMP_NIBW + (size_t)t * PHX_JUMP_COLW;
        for (int q = 0; q < 8; q++) dst[q] = q < 5 ? o[q] : 0u;
    }
}

// the tables of every genstep's event (batched calls): one block per genstep
__global__ void __launch_bounds__(PHX_JUMP_THREADS) k_jump_tables(const int* ev, const uint32_t* __restrict__ D, uint32_t* T)
{
    __shared__ uint32_t col[PHX_JUMP_BITS * 5];
    phx_event_table((unsigned long long)(unsigned)ev[blockIdx.x], D, T + (size_t)blockIdx.x * PHX_JUMP_NIBW, col);
}

PHX_D void phx_load_rng(curandStateXORWOW& s, const uint32_t* rng, long long slots, long long slot)
{
    s.d = __ldg(rng + slot);
    s.v[0] = __ldg(rng + slots * 1 + slot);
    s.v[1] = __ldg(rng + slots * 2 + slot);
    s.v[2] = __ldg(rng + slots * 3 + slot);
    s.v[3] = __ldg(rng + slots * 4 + slot);
    s.v[4] = __ldg(rng + slots * 5 + slot);
    s.boxmuller_flag = 0;
    s.boxmuller_flag_double = 0;
    s.boxmuller_extra = 0.f;
    s.boxmuller_extra_double = 0.0;
}

PHX_D void phx_store_photon(phx_photon* out, const PhxPhoton& p)
{
    float4* o = reinterpret_cast<float4*>(out);
    o[0] = make_float4(p.pos.x, p.pos.y, p.pos.z, p.time);
    o[1] = make_float4(p.mom.x, p.mom.y, p.mom.z, __uint_as_float(p.hitcount_iindex));
    o[2] = make_float4(p.pol.x, p.pol.y, p.pol.z, p.wavelength);
    o[3] = make_float4(__uint_as_float(p.obf), __uint_as_float(p.identity), __uint_as_float(p.index), __uint_as_float(p.flagmask));
}

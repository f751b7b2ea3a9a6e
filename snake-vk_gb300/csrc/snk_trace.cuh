// snk_trace.cuh -- two-level traversal of 8-wide compressed BVHs.
//
// Replaces traceRayEXT (Core/res/shaders/RayGen.rgen:101-121, 164-176, 195-207;
// RayClosestHit.rchit:64-84), which runs on the driver's RT-core traversal in
// the reference.  Semantics (BVH independent, so every device and the CPU
// oracle agree bit for bit):
//   closest hit = the minimum of (t, instance, triangle) over all triangles
//                 with tmin < t < tmax under the watertight test;
//   any hit     = whether such a triangle exists.
// Box tests are only required to be conservative: child boxes are quantised
// outwards and accepted with a slack of BOX_SLACK of the exit distance.  tmin below 0 (or NaN) is taken as 0, as traceRayEXT
// requires tmin >= 0; entry distances are then never negative.
//
// Traversal scheme (Ylitie, Karras, Laine, HPG 2017): the current node group
// is (child_base, hit bits of internal children << 24 | imask) and the current
// primitive group is (prim_base, 32 primitive hit bits).  Groups are kept on a
// short per-thread stack in shared memory ([entry][thread] layout, conflict
// free) that spills to local memory; primitive groups carry PRIM_GROUP in the
// base word there.  Closest-hit rays visit children in the order of the slot
// index xor the ray octant, which the builder makes approximately front to back;
// any-hit rays visit them from the highest slot down.  Leaves of the instance BVH hold instance ids: on reaching one
// the ray is transformed into object space and the BLAS root is entered; when
// the stack unwinds to the entry depth, the world ray is restored.  Coherent rays
// (the camera rays of large views) can instead be traced 32 at a time by a whole
// warp (PacketTraverser, below), with the same results.
#pragma once
#include "snk_device.cuh"
#include "snk_lane_stack.h"

namespace snk {

constexpr uint32_t PRIM_GROUP = 0x80000000u;         // stack tag of a primitive group (bases are < 2^31)
// A child box is accepted when t_enter <= t_exit (1 + BOX_SLACK), the sign of one FMA
// (exact but for results that round to zero, which keep their sign).  The slack covers
// the 2-ulp reciprocal of the direction, the roundings relative to t of the plane
// offsets and the final rounding of each plane distance (about 6 ulps of t in all);
// with t_enter >= tmin >= 0 a negative t_exit (box behind the origin) is rejected.  The
// rounding relative to the node's size is covered by the planes (quant_child).
constexpr float BOX_SLACK = 3.814697265625e-6f;   // 2^-18

// device error word bits
constexpr unsigned ERR_STACK_OVERFLOW = 1u;
constexpr unsigned ERR_STEP_LIMIT = 2u;
constexpr unsigned ERR_BAD_INDEX = 4u;    // a node/primitive/instance index outside its array

struct NodeRay {
    float ox, oy, oz;
    float idx, idy, idz;
    uint32_t oct;   // bit i set when direction component i is negative
};

// Reciprocal for box tests only (they need to be conservative, not exact): one
// instruction, within 1 ulp, inside BOX_SLACK (which allows 2).
__device__ __forceinline__ float safe_rcp(float d) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(copysignf(fmaxf(fabsf(d), 1e-20f), d)));
    return r;
}

__device__ __forceinline__ NodeRay make_node_ray(V3 o, V3 d) {
    NodeRay r;
    r.ox = o.x; r.oy = o.y; r.oz = o.z;
    r.idx = safe_rcp(d.x); r.idy = safe_rcp(d.y); r.idz = safe_rcp(d.z);
    // sign bits (not d < 0): -0.0 has a negative reciprocal and must enter through the high plane
    r.oct = (__float_as_uint(d.x) >> 31) | ((__float_as_uint(d.y) >> 31) << 1) | ((__float_as_uint(d.z) >> 31) << 2);
    return r;
}

// Three-input maximum / minimum (one instruction on sm_100 and later; NaN inputs
// are ignored, as with fmaxf / fminf).
__device__ __forceinline__ float max3f(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// ((1 << len) - 1) << pos in one instruction
__device__ __forceinline__ uint32_t bit_mask(uint32_t pos, uint32_t len) {
    uint32_t d;
    asm("bmsk.clamp.b32 %0, %1, %2;" : "=r"(d) : "r"(pos), "r"(len));
    return d;
}

// Byte k of w as 1 + q 2^-15 (bits 8..15 of the mantissa of 1.0f): one byte permute.
__device__ __forceinline__ float byte_m(uint32_t w, uint32_t k) {
    return __uint_as_float(__byte_perm(w, 0x3F800000u, 0x7604u | (k << 4)));
}

// a plane byte as byte_m decodes it
__device__ __forceinline__ float byte_f(uint32_t q) { return __uint_as_float(0x3F800000u | (q << 8)); }

// Box tests of the 8 children of a node (words w0, w2, w3, w4) against ray r on
// [tmin, tmax]: bit s of the result is set when the box of slot s is hit.
// Near/far planes are swapped once per node by the ray octant; each plane costs a
// byte permute and half a packed FMA; the sign of t_exit (1 + BOX_SLACK) - t_enter
// decides, collected by one funnel shift per child.  Bound by issue and the ALU pipe
// (min/max, permutes): with the planes' pad in the tree instead of per-axis near and far
// offsets, and a sign instead of an integer compare, select and or per child, a 1080p
// frame of the sphere field took 2.054 instead of 2.105 ms, the 19.2 Mpx terrain batch
// 37.3 instead of 38.5 ms.
__device__ __forceinline__ uint32_t box_hits(const float4& w0, const float4& w2, const float4& w3, const float4& w4,
                                             const NodeRay& r, float tmin, float tmax) {
    const uint32_t e = __float_as_uint(w0.w);
    // per axis A = 2^15 x (grid step) / d (the node's exponent bytes carry the 2^15), B =
    // (p - o) / d - A rounded once; a plane byte q decodes as x = 1 + q 2^-15 (one byte
    // permute), so t = fma(x, A, B).  The part of B's rounding that is relative to A (at
    // most |A| 2^-23, 1/256 of a grid step) is covered by the 1/64 of a grid step by
    // which the planes lie outside the boxes (quant_child).
    const float ax = __uint_as_float((e << 23) & 0x7F800000u) * r.idx;
    const float ay = __uint_as_float((e << 15) & 0x7F800000u) * r.idy;
    const float az = __uint_as_float((e << 7) & 0x7F800000u) * r.idz;
    const float bx = __fmaf_rn(w0.x - r.ox, r.idx, -ax), by = __fmaf_rn(w0.y - r.oy, r.idy, -ay),
                bz = __fmaf_rn(w0.z - r.oz, r.idz, -az);
    const bool sx = r.oct & 1u, sy = r.oct & 2u, sz = r.oct & 4u;
    uint32_t lx0 = __float_as_uint(w2.x), lx1 = __float_as_uint(w2.y), ly0 = __float_as_uint(w2.z),
             ly1 = __float_as_uint(w2.w), lz0 = __float_as_uint(w3.x), lz1 = __float_as_uint(w3.y),
             hx0 = __float_as_uint(w3.z), hx1 = __float_as_uint(w3.w), hy0 = __float_as_uint(w4.x),
             hy1 = __float_as_uint(w4.y), hz0 = __float_as_uint(w4.z), hz1 = __float_as_uint(w4.w);
    // near / far plane words per axis (a negative direction enters through the high plane)
    uint32_t nx[2] = {sx ? hx0 : lx0, sx ? hx1 : lx1}, fx[2] = {sx ? lx0 : hx0, sx ? lx1 : hx1};
    uint32_t ny[2] = {sy ? hy0 : ly0, sy ? hy1 : ly1}, fy[2] = {sy ? ly0 : hy0, sy ? ly1 : hy1};
    uint32_t nz[2] = {sz ? hz0 : lz0, sz ? hz1 : lz1}, fz[2] = {sz ? lz0 : hz0, sz ? lz1 : hz1};
    uint32_t miss = 0;   // bit s: the box of slot s is missed
    // children s and s + 1 in one packed FMA per plane (sm_100 and later: two
    // binary32 FMAs per instruction, each rounded as fmaf)
    const float2 AX = make_float2(ax, ax), AY = make_float2(ay, ay), AZ = make_float2(az, az);
    const float2 BX = make_float2(bx, bx), BY = make_float2(by, by), BZ = make_float2(bz, bz);
#pragma unroll
    for (int s = 6; s >= 0; s -= 2) {
        const int h = s >> 2, k = s & 3;
        const float2 tnx = __ffma2_rn(make_float2(byte_m(nx[h], k), byte_m(nx[h], k + 1)), AX, BX);
        const float2 tny = __ffma2_rn(make_float2(byte_m(ny[h], k), byte_m(ny[h], k + 1)), AY, BY);
        const float2 tnz = __ffma2_rn(make_float2(byte_m(nz[h], k), byte_m(nz[h], k + 1)), AZ, BZ);
        const float2 tfx = __ffma2_rn(make_float2(byte_m(fx[h], k), byte_m(fx[h], k + 1)), AX, BX);
        const float2 tfy = __ffma2_rn(make_float2(byte_m(fy[h], k), byte_m(fy[h], k + 1)), AY, BY);
        const float2 tfz = __ffma2_rn(make_float2(byte_m(fz[h], k), byte_m(fz[h], k + 1)), AZ, BZ);
        const float tn0 = max3f(tnx.x, tny.x, fmaxf(tnz.x, tmin)), tn1 = max3f(tnx.y, tny.y, fmaxf(tnz.y, tmin));
        const float tf0 = min3f(tfx.x, tfy.x, fminf(tfz.x, tmax)), tf1 = min3f(tfx.y, tfy.y, fminf(tfz.y, tmax));
        miss = __funnelshift_l(__float_as_uint(__fmaf_rn(tf1, 1.0f + BOX_SLACK, -tn1)), miss, 1);
        miss = __funnelshift_l(__float_as_uint(__fmaf_rn(tf0, 1.0f + BOX_SLACK, -tn0)), miss, 1);
    }
    return ~miss & 0xFFu;
}

// Leaf slots of a single-primitive-leaf node (meta count bits 1: bit 5 of each
// byte), gathered from the four bytes of each meta word by a byte dot product.
__device__ __forceinline__ uint32_t leaf_slots(uint32_t meta0, uint32_t meta1) {
    const uint32_t l0 = (meta0 >> 5) & 0x01010101u, l1 = (meta1 >> 5) & 0x01010101u;
    return __dp4a(l1, 0x80402010u, __dp4a(l0, 0x08040201u, 0u));
}

// Child bits moved by octant oct: bit s to s ^ oct (three conditional swaps).  The groups
// of a single ray are taken from the highest bit down (one instruction finds it, the
// lowest one takes two), so that they are kept at s ^ oct ^ 7: that and the reciprocal in one
// instruction took the eight-view terrain batch from 33.7 to 32.9 ms.
__device__ __forceinline__ uint32_t visit_order(uint32_t x, uint32_t oct) {
    x = (oct & 1u) ? (((x & 0x55u) << 1) | ((x >> 1) & 0x55u)) : x;
    x = (oct & 2u) ? (((x & 0x33u) << 2) | ((x >> 2) & 0x33u)) : x;
    x = (oct & 4u) ? (((x & 0x0Fu) << 4) | ((x >> 4) & 0x0Fu)) : x;
    return x;
}

// Tests the 8 children of node idx.  ngroup <- (child_base, internal hits << 24 | imask)
// with internal hit bit of slot s at position s ^ oct ^ 7 (ORDERED) or s; tgroup <- (prim_base,
// primitive hits).  The internal-child bits are moved into visiting order with three
// conditional swaps when the order matters (closest hit; an any-hit
// ray stops at whichever occluder it meets first and skips the swaps), and only the
// hit leaf slots are expanded into primitive bits.
template <bool ORDERED, bool SINGLE>
__device__ __forceinline__ void intersect_node(const WideNode* __restrict__ nodes, uint32_t idx, const NodeRay& r,
                                               float tmin, float tmax, uint2& ngroup, uint2& tgroup) {
    const float4* np = reinterpret_cast<const float4*>(nodes + idx);
    float4 w0 = __ldg(np + 0), w1 = __ldg(np + 1), w2 = __ldg(np + 2), w3 = __ldg(np + 3), w4 = __ldg(np + 4);
    const uint32_t imask = __float_as_uint(w0.w) >> 24;
    const uint32_t meta0 = __float_as_uint(w1.z), meta1 = __float_as_uint(w1.w);
    const uint32_t hits = box_hits(w0, w2, w3, w4, r, tmin, tmax);
    // internal children (imask bits) in visiting order, the first one highest
    uint32_t x = hits & imask;
    if (ORDERED) x = visit_order(x, r.oct ^ 7u);
    ngroup = make_uint2(__float_as_uint(w1.x), (x << 24) | imask);
    if constexpr (SINGLE) {
        // every leaf holds one primitive, stored in slot order; primitive groups are
        // (prim_base, hit leaf slots << 24 | leaf slots), like node groups
        const uint32_t leafmask = leaf_slots(meta0, meta1);
        tgroup = make_uint2(__float_as_uint(w1.y), ((hits & leafmask) << 24) | leafmask);
    } else {
        // leaf children: (count << 5) | offset -> primitive bits; an empty slot (meta 0) adds none
        uint32_t leaves = hits & ~imask, hit_prim = 0;
        while (leaves) {
            const uint32_t s = __ffs(leaves) - 1;
            leaves &= leaves - 1u;
            const uint32_t m = __byte_perm(meta0, meta1, s) & 0xFFu;
            hit_prim |= bit_mask(m & 31u, m >> 5);
        }
        tgroup = make_uint2(__float_as_uint(w1.y), hit_prim);
    }
}

struct TraceResult { float t, u, v; uint32_t inst, prim; bool hit; };

struct TraceCounters { unsigned long long nodes, tris; };

// Short stack: entries [0, STACK_SH) live in shared memory at sh[k * nthreads + tid],
// deeper entries in a local array; at most lim (<= STACK_MAX) entries.  Rows
// STACK_SH .. STACK_SH + 4 of sh (TRACE_SH_ROWS rows in all) keep the world ray.
struct ShortStack {
    uint2* sh;
    uint2* spill;   // STACK_MAX - STACK_SH entries (a local array of the caller)
    uint32_t tid, nthreads;
    int sp, lim;
    __device__ __forceinline__ bool push(uint2 v) {
        if (sp >= lim) return false;
        if (sp < STACK_SH) sh[sp * nthreads + tid] = v;
        else spill[sp - STACK_SH] = v;
        sp++;
        return true;
    }
    __device__ __forceinline__ uint2 pop() {
        sp--;
        return sp < STACK_SH ? sh[sp * nthreads + tid] : spill[sp - STACK_SH];
    }
};

// Result of a finished ray (T: its traversal state); traversal errors are reported
// through the scene's error word and read as a miss.
template <class T>
__device__ __forceinline__ bool ray_result(const T& v, const SceneDev& S, TraceResult& res) {
    res.hit = false;
    res.t = -1.0f; res.u = 0.0f; res.v = 0.0f; res.inst = INVALID; res.prim = INVALID;
    if (v.err) {
        if (S.error_word) atomicOr(S.error_word, v.err);
        return false;
    }
    if (v.best_inst != INVALID) {
        res.hit = true;
        res.t = v.best_t; res.inst = v.best_inst; res.prim = v.best_prim; res.u = v.best_u; res.v = v.best_v;
    }
    return res.hit;
}

// Resumable traversal state of one ray.  The work is split into single units so
// a warp can vote each iteration which kind of unit its lanes execute together:
//   node_step()  intersect one internal child of the current node group
//   prim_step()  test one primitive of the current primitive group (a triangle,
//                or at the instance level: enter that instance's BLAS)
//   settle()     pop the stack until there is work again, leaving the BLAS
//                when its part of the stack is used up; true when finished
// SINGLE: every leaf of both levels holds one primitive (SceneDev::single_leaf);
// primitive groups are then (prim_base, hit leaf slots << 24 | leaf slots).  The
// general form (primitive offset bits from the meta bytes) is valid for any tree.
template <bool ANY, bool COUNT, bool SINGLE = false>
struct Traverser {
    static constexpr bool ORD = !ANY;   // visit children front to back (closest hit only)
    static constexpr uint32_t PTHR = SINGLE ? 0x00FFFFFFu : 0u;   // a primitive group is pending above this
    float tmin, tmax;    // (the world-space ray itself is kept in shared memory: save_world)
    NodeRay cr;          // ray of the current level (world or object space)
    WRay tr;             // object-space watertight set-up (in a BLAS, once k != INVALID)
    float best_t, best_u, best_v;
    uint32_t best_inst, best_prim;
    uint2 ngroup, tgroup;
    int level, blas_sp;
    uint32_t cur_inst, steps;
    unsigned err;
    bool done;
    ShortStack st;

    __device__ __forceinline__ void init(const SceneDev& S, V3 o_, V3 d_, float tmin_, float tmax_, uint2* sh,
                                         uint2* spill, uint32_t tid, uint32_t nthreads) {
        tmin = fmaxf(tmin_, 0.0f); tmax = tmax_;
        cr = make_node_ray(o_, d_);
        best_t = tmax; best_u = 0.0f; best_v = 0.0f; best_inst = INVALID; best_prim = INVALID;
        level = 0; blas_sp = 0; cur_inst = 0; steps = 0; err = 0; done = false;
        st.sh = sh; st.spill = spill; st.tid = tid; st.nthreads = nthreads; st.sp = 0;
        st.lim = S.stack_max < STACK_MAX ? S.stack_max : STACK_MAX;
        save_world(d_);
        ngroup = S.tlas_root == INVALID ? make_uint2(0u, 0u) : make_uint2(S.tlas_root, (1u << (24 + (ORD ? cr.oct ^ 7u : 0u))) | 1u);
        tgroup = make_uint2(0u, 0u);
    }

    __device__ __forceinline__ bool has_node() const { return ngroup.y > 0x00FFFFFFu; }
    __device__ __forceinline__ bool has_prim() const { return tgroup.y > PTHR; }

    __device__ __forceinline__ void fail(unsigned e) { err |= e; done = true; }

    // the world ray (origin, direction) and its node-test set-up, kept in shared
    // memory rows STACK_SH .. STACK_SH + 4 of this thread: read when the ray enters an
    // instance and when it leaves one
    __device__ __forceinline__ uint2& row(int k) const { return st.sh[(STACK_SH + k) * st.nthreads + st.tid]; }
    __device__ __forceinline__ void save_world(V3 d) {
        row(0) = make_uint2(__float_as_uint(cr.idx), __float_as_uint(cr.idy));
        row(1) = make_uint2(__float_as_uint(cr.idz), cr.oct);
        row(2) = make_uint2(__float_as_uint(cr.ox), __float_as_uint(cr.oy));
        row(3) = make_uint2(__float_as_uint(cr.oz), __float_as_uint(d.x));
        row(4) = make_uint2(__float_as_uint(d.y), __float_as_uint(d.z));
    }
    __device__ __forceinline__ void restore_world() {
        const uint2 a = row(0), b = row(1), c = row(2), e = row(3);
        cr.ox = __uint_as_float(c.x); cr.oy = __uint_as_float(c.y); cr.oz = __uint_as_float(e.x);
        cr.idx = __uint_as_float(a.x); cr.idy = __uint_as_float(a.y); cr.idz = __uint_as_float(b.x);
        cr.oct = b.y;
    }
    __device__ __forceinline__ void world_ray(V3& o, V3& d) const {
        const uint2 c = row(2), e = row(3), f = row(4);
        o = v3(__uint_as_float(c.x), __uint_as_float(c.y), __uint_as_float(e.x));
        d = v3(__uint_as_float(e.y), __uint_as_float(f.x), __uint_as_float(f.y));
    }

    // Pops a node or primitive group when none is pending (what is on the stack has work);
    // sets done when the ray is finished.
    __device__ __forceinline__ void settle() {
        if (!done && !has_node() && !has_prim()) {
            if (level == 1 && st.sp == blas_sp) { level = 0; restore_world(); }
            if (st.sp == 0) { done = true; return; }
            uint2 g = st.pop();
            if (g.x & PRIM_GROUP) tgroup = make_uint2(g.x & ~PRIM_GROUP, g.y);
            else ngroup = g;
        }
    }

    // The units are bound by issue and the branches cost as much as the arithmetic
    // between them: one pop instead of a loop, the pushes of both groups under one test of
    // the shared-memory part of the stack, and errors that are noted without leaving the
    // step (an index outside its array becomes 0) took the eight-view terrain batch from
    // 36.3 to 33.7 ms, a 1080p frame of the sphere field from 1.893 to 1.803 ms and two
    // ReSTIR frames from 14.84 to 14.29 ms.

    // puts the pending groups on the stack (primitives first); false: no room
    __device__ __forceinline__ bool push_groups(const SceneDev& S) {
        const bool pp = has_prim(), pn = has_node();
        if (st.sp <= min(STACK_SH, S.stack_max) - 2) {
            uint2* top = st.sh + st.sp * st.nthreads + st.tid;
            if (pp) *top = make_uint2(tgroup.x | PRIM_GROUP, tgroup.y);
            if (pp) top += st.nthreads;
            if (pn) *top = ngroup;
            st.sp += (int)pp + (int)pn;
            return true;
        }
        return (!pp || st.push(make_uint2(tgroup.x | PRIM_GROUP, tgroup.y))) && (!pn || st.push(ngroup));
    }

    __device__ __forceinline__ void node_step(const SceneDev& S, TraceCounters* ctr) {
        if (++steps > S.max_steps) fail(ERR_STEP_LIMIT);
        const uint32_t bit = 31u - __clz(ngroup.y);
        ngroup.y ^= 1u << bit;
        const uint32_t slot = (ORD ? bit ^ cr.oct ^ 7u : bit) & 7u;
        uint32_t child = ngroup.x + __popc(ngroup.y & ((1u << slot) - 1u));
        // a pending primitive group is postponed onto the stack, then what is left of the nodes
        if (!push_groups(S)) { fail(ERR_STACK_OVERFLOW); return; }
        tgroup = make_uint2(0u, 0u);
        if (COUNT) ctr->nodes++;
        if (child >= (level ? S.num_blas_nodes : S.num_tlas_nodes)) { fail(ERR_BAD_INDEX); child = 0; }
        intersect_node<ORD, SINGLE>(level ? S.blas_nodes : S.tlas_nodes, child, cr, tmin, best_t, ngroup, tgroup);
    }

    // enters the instance of instance-BVH primitive pidx (what is left of the instance
    // level is on the stack)
    __device__ __forceinline__ void enter_instance(const SceneDev& S, uint32_t pidx) {
        if (pidx >= S.num_tlas_prims) { fail(ERR_BAD_INDEX); pidx = 0; }
        uint32_t inst = __ldg(&S.tlas_prims[pidx]);
        if (inst >= S.num_instances) { fail(ERR_BAD_INDEX); inst = 0; }
        const float4* ip = reinterpret_cast<const float4*>(S.inst_trace + inst);
        float4 r0 = __ldg(ip), r1 = __ldg(ip + 1), r2 = __ldg(ip + 2);
        uint32_t root = __ldg(reinterpret_cast<const uint32_t*>(ip + 3));
        float inv[12] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w, r2.x, r2.y, r2.z, r2.w};
        V3 o, d;
        world_ray(o, d);
        V3 oo = xform_point_rn(inv, o);
        V3 od = xform_dir_rn(inv, d);
        cr = make_node_ray(oo, od);
        // the watertight set-up waits for the instance's first triangle test (many
        // instances are left without one); until then its shear slots hold the direction
        tr.k = INVALID; tr.Sx = od.x; tr.Sy = od.y; tr.Sz = od.z;
        blas_sp = st.sp;
        level = 1;
        cur_inst = inst;
        ngroup = make_uint2(root, (1u << (24 + (ORD ? cr.oct ^ 7u : 0u))) | 1u);
        tgroup = make_uint2(0u, 0u);
    }

    __device__ __forceinline__ void prim_step(const SceneDev& S, TraceCounters* ctr) {
        if (++steps > S.max_steps) { fail(ERR_STEP_LIMIT); return; }
        uint32_t pidx;
        if constexpr (SINGLE) {   // the primitive's rank among the node's leaf slots
            const uint32_t bit = 31u - __clz(tgroup.y);
            tgroup.y ^= 1u << bit;
            pidx = tgroup.x + __popc(tgroup.y & ((1u << (bit & 7u)) - 1u));
        } else {
            const uint32_t k = __ffs(tgroup.y) - 1;
            tgroup.y &= tgroup.y - 1u;
            pidx = tgroup.x + k;
        }
        if (level == 0) {
            if (!push_groups(S)) { fail(ERR_STACK_OVERFLOW); return; }
            enter_instance(S, pidx);
        } else {
            if (pidx >= S.num_tris) { fail(ERR_BAD_INDEX); pidx = 0; }
            if (COUNT) ctr->tris++;
            if (tr.k == INVALID) tr = wray_setup(v3(tr.Sx, tr.Sy, tr.Sz));
            const float4* tp = reinterpret_cast<const float4*>(S.tris + pidx);
            float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
            float va[3] = {a.x, a.y, a.z}, vb[3] = {b.x, b.y, b.z}, vc[3] = {c.x, c.y, c.z};
            float t, b1, b2;
            if (intersect_tri(tr, v3(cr.ox, cr.oy, cr.oz), va, vb, vc, tmin, tmax, &t, &b1, &b2)) {
                uint32_t prim = __float_as_uint(a.w);
                bool better = best_inst == INVALID || t < best_t ||
                              (t == best_t && (cur_inst < best_inst || (cur_inst == best_inst && prim < best_prim)));
                if (ANY || better) {
                    best_t = t; best_inst = cur_inst; best_prim = prim; best_u = b1; best_v = b2;
                }
                if (ANY) done = true;
            }
        }
    }

    __device__ __forceinline__ bool finish(const SceneDev& S, TraceResult& res) { return ray_result(*this, S, res); }
};

// ---- eight lanes per ray -----------------------------------------------------------
// The last rays of a queue, and the rays of a queue too small to fill the GPU, are bound
// by the latency of their dependent steps, not by issue: a warp with at most
// COOP_RAYS rays gives eight lanes to each.  A lane tests one child of a node, or the
// triangle of one leaf slot, and the lanes vote; everything else they do alike.  Hits
// equal the one-lane traversal's: boxes only cull, and the closest hit is the minimum
// of the tested triangles in the same (t, instance, triangle) order.  A ray gets there
// through a slot in shared memory (coop_save), so that the code that follows keeps no
// registers of the one-lane loop alive.  Its stack moves into the warp's shared stack
// rows, of which a group's eight columns hold the STACK_MAX entries (the finished rays
// no longer need theirs); its world-ray rows stay in its owner's column.  For
// single-primitive-leaf trees.
constexpr int COOP_RAYS = 4;
static_assert(STACK_SH * 8 >= STACK_MAX, "eight columns of the shared stack hold a whole stack");

struct CoopSlot {   // (the result comes back in best_*, the error bits in err)
    float tmin, tmax;
    NodeRay cr;
    WRay tr;
    float best_t, best_u, best_v;
    uint32_t best_inst, best_prim;
    uint2 ngroup, tgroup;
    int level, blas_sp, sp;
    uint32_t cur_inst, steps, ri, tid;
    unsigned err;
};

// an unfinished ray of this thread into a slot
template <class TV>
__device__ __forceinline__ void coop_save(CoopSlot& c, const TV& tv, uint32_t ri) {
    c.tmin = tv.tmin; c.tmax = tv.tmax;
    c.cr = tv.cr;
    c.tr = tv.tr;
    c.best_t = tv.best_t; c.best_u = tv.best_u; c.best_v = tv.best_v;
    c.best_inst = tv.best_inst; c.best_prim = tv.best_prim;
    c.ngroup = tv.ngroup; c.tgroup = tv.tgroup;
    c.level = tv.level; c.blas_sp = tv.blas_sp; c.sp = tv.st.sp;
    c.cur_inst = tv.cur_inst; c.steps = tv.steps; c.ri = ri; c.tid = threadIdx.x;
}

// Finishes the k <= COOP_RAYS rays saved in the warp's slots (all 32 lanes call this;
// spill: the one-lane traversal's local stack entries).  A call, so that the one-lane
// loops keep their registers (inlined, they spilled and big queues took 2 to 5 % longer).
template <bool ANY>
__device__ __noinline__ void coop_trace(CoopSlot* slots, uint32_t k_rays, const SceneDev& S, uint2* sh_stack,
                                        const uint2* spill, uint32_t nthreads) {
    using TV = Traverser<ANY, false, true>;
    TV tv;
    const uint32_t lane = threadIdx.x & 31u, base = threadIdx.x & ~31u, g = lane >> 3, slot = lane & 7u;
    auto entry = [&](uint32_t group, int e) -> uint2& {   // stack entry e of a group
        return sh_stack[(uint32_t)(e & 7) * nthreads + base + 8u * group + (uint32_t)(e >> 3)];
    };
    const bool valid = g < k_rays;
    __syncwarp();   // the slots are complete
    {   // the stacks into the groups' columns: first the entries in shared rows (entry `slot`
        // of this lane's group), once all are read, then the owners' local ones
        uint2 v = make_uint2(0u, 0u);
        const bool move = valid && (int)slot < slots[g].sp;
        if (move) v = sh_stack[slot * nthreads + slots[g].tid];
        __syncwarp();
        if (move) entry(g, (int)slot) = v;
        for (uint32_t r = 0; r < k_rays; r++)
            if (slots[r].tid == threadIdx.x)
                for (int e = STACK_SH; e < slots[r].sp; e++) entry(r, e) = spill[e - STACK_SH];
        __syncwarp();
    }
    if (valid) {
        const CoopSlot& c = slots[g];
        tv.tmin = c.tmin; tv.tmax = c.tmax;
        tv.cr = c.cr;
        tv.tr = c.tr;
        tv.best_t = c.best_t; tv.best_u = c.best_u; tv.best_v = c.best_v;
        tv.best_inst = c.best_inst; tv.best_prim = c.best_prim;
        tv.ngroup = c.ngroup; tv.tgroup = c.tgroup;
        tv.level = c.level; tv.blas_sp = c.blas_sp;
        tv.cur_inst = c.cur_inst; tv.steps = c.steps;
        tv.err = 0; tv.done = false;
        tv.st.sh = sh_stack; tv.st.tid = c.tid; tv.st.nthreads = nthreads; tv.st.sp = c.sp;
        tv.st.lim = S.stack_max < STACK_MAX ? S.stack_max : STACK_MAX;
        const unsigned gm = 0xFFu << (8u * g);
        auto push = [&](uint32_t x, uint32_t y) {
            if (tv.st.sp >= tv.st.lim) { tv.fail(ERR_STACK_OVERFLOW); return; }
            entry(g, tv.st.sp++) = make_uint2(x, y);   // (the group's lanes store the same value)
        };
        while (!tv.done) {
            if (!tv.has_node() && !tv.has_prim()) {
                if (tv.level == 1 && tv.st.sp == tv.blas_sp) { tv.level = 0; tv.restore_world(); }
                if (tv.st.sp == 0) break;
                const uint2 e = lanes_pop<uint2>([&](int k) { return entry(g, k); }, tv.st.sp, [&] { __syncwarp(gm); });
                if (e.x & PRIM_GROUP) tv.tgroup = make_uint2(e.x & ~PRIM_GROUP, e.y);
                else tv.ngroup = e;
                continue;
            }
            if (++tv.steps > S.max_steps) { tv.fail(ERR_STEP_LIMIT); break; }
            if (tv.has_prim() && tv.level == 1) {
                // the hit leaf slots' triangles, one per lane
                const uint32_t hit = tv.tgroup.y >> 24, leaves = tv.tgroup.y & 0xFFu;
                if (tv.tr.k == INVALID) tv.tr = wray_setup(v3(tv.tr.Sx, tv.tr.Sy, tv.tr.Sz));
                float t = 0.0f, b1 = 0.0f, b2 = 0.0f;
                uint32_t prim = INVALID;
                bool found = false, bad = false;
                if ((hit >> slot) & 1u) {
                    const uint32_t pidx = tv.tgroup.x + (uint32_t)__popc(leaves & ((1u << slot) - 1u));
                    bad = pidx >= S.num_tris;
                    if (!bad) {
                        const float4* tp = reinterpret_cast<const float4*>(S.tris + pidx);
                        const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
                        const float va[3] = {a.x, a.y, a.z}, vb[3] = {b.x, b.y, b.z}, vc[3] = {c.x, c.y, c.z};
                        found = intersect_tri(tv.tr, v3(tv.cr.ox, tv.cr.oy, tv.cr.oz), va, vb, vc, tv.tmin, tv.tmax, &t,
                                              &b1, &b2);
                        prim = __float_as_uint(a.w);
                    }
                }
                tv.tgroup = make_uint2(0u, 0u);
                if (__any_sync(gm, bad)) { tv.fail(ERR_BAD_INDEX); break; }
                unsigned f = __ballot_sync(gm, found);
                if (ANY) {
                    if (f) { tv.best_inst = tv.cur_inst; break; }
                } else {
                    for (; f; f &= f - 1u) {   // (rarely more than one)
                        const int l = __ffs(f) - 1;
                        const float tl = __shfl_sync(gm, t, l), ul = __shfl_sync(gm, b1, l), vl = __shfl_sync(gm, b2, l);
                        const uint32_t pl = __shfl_sync(gm, prim, l);
                        if (tv.best_inst == INVALID || tl < tv.best_t ||
                            (tl == tv.best_t && (tv.cur_inst < tv.best_inst ||
                                                 (tv.cur_inst == tv.best_inst && pl < tv.best_prim)))) {
                            tv.best_t = tl; tv.best_inst = tv.cur_inst; tv.best_prim = pl; tv.best_u = ul; tv.best_v = vl;
                        }
                    }
                }
                continue;
            }
            if (tv.has_prim()) {   // an instance
                const uint32_t k = __ffs(tv.tgroup.y >> 24) - 1;
                tv.tgroup.y &= ~(1u << (24 + k));
                const uint32_t pidx = tv.tgroup.x + (uint32_t)__popc(tv.tgroup.y & ((1u << k) - 1u));
                const uint32_t rest_x = tv.tgroup.x, rest_y = tv.tgroup.y;
                if (tv.has_prim()) push(rest_x | PRIM_GROUP, rest_y);
                if (!tv.done && tv.has_node()) push(tv.ngroup.x, tv.ngroup.y);
                if (tv.done) break;
                tv.enter_instance(S, pidx);
                continue;
            }
            // a node: one child per lane
            const uint32_t bit = 31u - __clz(tv.ngroup.y);
            tv.ngroup.y ^= 1u << bit;
            const uint32_t sl = (TV::ORD ? bit ^ tv.cr.oct ^ 7u : bit) & 7u;
            const uint32_t child = tv.ngroup.x + (uint32_t)__popc(tv.ngroup.y & ((1u << sl) - 1u) & 0xFFu);
            if (tv.has_node()) push(tv.ngroup.x, tv.ngroup.y);
            if (tv.done) break;
            if (child >= (tv.level ? S.num_blas_nodes : S.num_tlas_nodes)) { tv.fail(ERR_BAD_INDEX); break; }
            const WideNode* N = (tv.level ? S.blas_nodes : S.tlas_nodes) + child;
            const float4 w0 = __ldg(reinterpret_cast<const float4*>(N));
            const uint2 w1 = __ldg(reinterpret_cast<const uint2*>(N) + 2);
            const uint8_t* q = N->meta + slot;   // meta, then the planes: lo x y z, hi x y z, eight bytes each
            const uint32_t meta = __ldg(q);
            const uint32_t ox = tv.cr.oct & 1u ? 24u : 0u, oy = tv.cr.oct & 2u ? 24u : 0u, oz = tv.cr.oct & 4u ? 24u : 0u;
            const float nx = byte_f(__ldg(q + 8 + ox)), fx = byte_f(__ldg(q + 32 - ox));
            const float ny = byte_f(__ldg(q + 16 + oy)), fy = byte_f(__ldg(q + 40 - oy));
            const float nz = byte_f(__ldg(q + 24 + oz)), fz = byte_f(__ldg(q + 48 - oz));
            const uint32_t e = __float_as_uint(w0.w), imask = e >> 24;
            const float ax = __uint_as_float((e << 23) & 0x7F800000u) * tv.cr.idx;
            const float ay = __uint_as_float((e << 15) & 0x7F800000u) * tv.cr.idy;
            const float az = __uint_as_float((e << 7) & 0x7F800000u) * tv.cr.idz;
            const float bx = __fmaf_rn(w0.x - tv.cr.ox, tv.cr.idx, -ax), by = __fmaf_rn(w0.y - tv.cr.oy, tv.cr.idy, -ay),
                        bz = __fmaf_rn(w0.z - tv.cr.oz, tv.cr.idz, -az);
            const float tn = max3f(__fmaf_rn(nx, ax, bx), __fmaf_rn(ny, ay, by), fmaxf(__fmaf_rn(nz, az, bz), tv.tmin));
            const float tf = min3f(__fmaf_rn(fx, ax, bx), __fmaf_rn(fy, ay, by), fminf(__fmaf_rn(fz, az, bz), tv.best_t));
            const bool in = (int)__float_as_uint(__fmaf_rn(tf, 1.0f + BOX_SLACK, -tn)) >= 0;
            const uint32_t hits = (__ballot_sync(gm, in) >> (8u * g)) & 0xFFu;
            const uint32_t leaves = (__ballot_sync(gm, (meta & 0x20u) != 0u && !((imask >> slot) & 1u)) >> (8u * g)) & 0xFFu;
            uint32_t x = hits & imask;
            if (TV::ORD) x = visit_order(x, tv.cr.oct ^ 7u);
            tv.ngroup = make_uint2(w1.x, (x << 24) | imask);
            tv.tgroup = make_uint2(w1.y, ((hits & leaves) << 24) | leaves);
        }
    }
    __syncwarp();
    if (valid && slot == 0u) {
        CoopSlot& c = slots[g];
        c.best_t = tv.best_t; c.best_u = tv.best_u; c.best_v = tv.best_v;
        c.best_inst = tv.best_inst; c.best_prim = tv.best_prim;
        c.err = tv.err;
    }
    __syncwarp();
}

// ---- warp packets ------------------------------------------------------------
// Traversal of up to 32 coherent rays (one per lane) by the whole warp together,
// for queues whose neighbouring entries are neighbouring pixels (camera rays).
// Node groups and instance groups are uniform over the warp and carry the mask of
// the lanes whose rays hit one of their boxes: every node is tested by all lanes
// against their own rays (lanes outside the mask count no hits), and the children
// hit by any lane form the next group, visited in the order of the octant of the
// group's first lane.  A mesh node's hit triangles stay per lane and are tested
// before anything else, each lane its own, in as many rounds as the lane with the
// most.  Hits equal the per-ray traversal's: boxes only cull, and the closest hit
// is the minimum over the tested triangles in the same (t, instance, triangle)
// order.  The group stack is one array of PSTACK entries (base, bits, lane mask)
// per warp in shared memory (lanes_pop).  Each lane's world ray and its node-test
// set-up wait in shared-memory rows while the lane's ray is in an instance.  For
// single-primitive-leaf trees only.  A packet that runs past its stack or past
// 32x the per-ray step cap reports the same error bits as a ray would (all its
// rays then miss).
constexpr int PSTACK = 2 * STACK_MAX;

template <bool ANY, int NT>
struct PacketTraverser {
    static constexpr bool ORD = !ANY;
    static constexpr uint32_t FULL = 0xFFFFFFFFu;
    // per lane
    float tmin, tmax;
    uint2* rows;             // this thread's 5 shared-memory rows (stride NT): the world ray and its set-up
    NodeRay cr;              // node-test set-up of the current level's ray
    WRay tr;                 // object-space watertight set-up (in a mesh, once k != INVALID)
    float best_t, best_u, best_v;
    uint32_t best_inst, best_prim;
    uint32_t tbits;          // hit leaf slots of the current mesh node this lane still has to test
    // uniform over the warp
    uint4* stk;
    uint2 ngroup, tgroup;    // node group; instance group (leaves of the instance BVH)
    uint32_t nmask, tmask, live, lane_bit;
    uint32_t tri_base, tri_leaves;   // prim_base and leaf slots of the mesh node tbits refers to
    uint32_t woct, coct;     // visiting octant of the world level and of the current level
    int level, sp, blas_sp;
    uint32_t cur_inst, steps, step_limit;
    unsigned err;

    __device__ __forceinline__ uint2& row(int k) const { return rows[k * NT]; }
    __device__ __forceinline__ void restore_world() {
        const uint2 a = row(0), b = row(1), c = row(2), e = row(3);
        cr.ox = __uint_as_float(c.x); cr.oy = __uint_as_float(c.y); cr.oz = __uint_as_float(e.x);
        cr.idx = __uint_as_float(a.x); cr.idy = __uint_as_float(a.y); cr.idz = __uint_as_float(b.x);
        cr.oct = b.y;
    }

    __device__ __forceinline__ void init(const SceneDev& S, V3 o, V3 d, float tmin_, float tmax_, bool active,
                                         uint4* stack, uint2* world_rows) {
        tmin = fmaxf(tmin_, 0.0f); tmax = tmax_;
        cr = make_node_ray(o, d);
        rows = world_rows;
        row(0) = make_uint2(__float_as_uint(cr.idx), __float_as_uint(cr.idy));
        row(1) = make_uint2(__float_as_uint(cr.idz), cr.oct);
        row(2) = make_uint2(__float_as_uint(o.x), __float_as_uint(o.y));
        row(3) = make_uint2(__float_as_uint(o.z), __float_as_uint(d.x));
        row(4) = make_uint2(__float_as_uint(d.y), __float_as_uint(d.z));
        tr.k = INVALID; tr.Sx = 0.0f; tr.Sy = 0.0f; tr.Sz = 0.0f;
        best_t = tmax; best_u = 0.0f; best_v = 0.0f; best_inst = INVALID; best_prim = INVALID;
        tbits = 0;
        stk = stack;
        lane_bit = 1u << (threadIdx.x & 31u);
        live = __ballot_sync(FULL, active);
        woct = live ? __shfl_sync(FULL, cr.oct, __ffs(live) - 1) : 0u;
        coct = woct;
        level = 0; sp = 0; blas_sp = 0; cur_inst = 0; steps = 0; err = 0; tri_base = 0; tri_leaves = 0;
        step_limit = S.max_steps < 0x07FFFFFFu ? 32u * S.max_steps : 0xFFFFFFFFu;
        ngroup = (S.tlas_root == INVALID || !live) ? make_uint2(0u, 0u)
                                                   : make_uint2(S.tlas_root, (1u << (24 + (ORD ? woct : 0u))) | 1u);
        nmask = live;
        tgroup = make_uint2(0u, 0u);
        tmask = 0;
    }

    // (as in the single ray's units, an error is noted and ends the packet after the step)
    __device__ __forceinline__ void push(uint32_t x, uint32_t y, uint32_t mask) {
        if (sp >= PSTACK) { err |= ERR_STACK_OVERFLOW; sp = PSTACK - 1; }
        stk[sp++] = make_uint4(x, y, mask, 0u);
    }

    // one internal child of the node group, tested by every lane
    __device__ __forceinline__ void node_step(const SceneDev& S) {
        const uint32_t k = __ffs(ngroup.y >> 24) - 1;
        ngroup.y &= ~(1u << (24 + k));
        const uint32_t m = nmask & live;
        if (ANY && m == 0) { ngroup.y &= 0x00FFFFFFu; return; }   // the group's rays are all finished
        const uint32_t slot = ORD ? k ^ coct : k;
        uint32_t child = ngroup.x + __popc(ngroup.y & ((1u << slot) - 1u));
        if (ngroup.y > 0x00FFFFFFu) push(ngroup.x, ngroup.y, nmask);   // (instances go first: none is pending)
        if (child >= (level ? S.num_blas_nodes : S.num_tlas_nodes)) { err |= ERR_BAD_INDEX; child = 0; }
        const float4* np = reinterpret_cast<const float4*>((level ? S.blas_nodes : S.tlas_nodes) + child);
        const float4 w0 = __ldg(np + 0), w1 = __ldg(np + 1), w2 = __ldg(np + 2), w3 = __ldg(np + 3),
                     w4 = __ldg(np + 4);
        uint32_t hits = box_hits(w0, w2, w3, w4, cr, tmin, best_t);
        if (!(m & lane_bit)) hits = 0;
        const uint32_t imask = __float_as_uint(w0.w) >> 24;
        const uint32_t leaves = leaf_slots(__float_as_uint(w1.z), __float_as_uint(w1.w));
        const uint32_t hi = hits & imask, hl = hits & leaves;
        const uint32_t ui = __reduce_or_sync(FULL, hi);
        nmask = __ballot_sync(FULL, hi != 0u);
        ngroup = make_uint2(__float_as_uint(w1.x), ((ORD ? visit_order(ui, coct) : ui) << 24) | imask);
        if (level == 0) {
            const uint32_t ul = __reduce_or_sync(FULL, hl);
            tmask = __ballot_sync(FULL, hl != 0u);
            tgroup = make_uint2(__float_as_uint(w1.y), (ul << 24) | leaves);
        } else {
            tbits = hl;
            tri_base = __float_as_uint(w1.y);
            tri_leaves = leaves;
        }
    }

    // enter the next instance of the instance group (the lanes that hit its leaf box)
    __device__ __forceinline__ void inst_step(const SceneDev& S) {
        const uint32_t k = __ffs(tgroup.y >> 24) - 1;
        tgroup.y &= ~(1u << (24 + k));
        const uint32_t m = tmask & live;
        if (ANY && m == 0) { tgroup.y &= 0x00FFFFFFu; return; }
        uint32_t pidx = tgroup.x + __popc(tgroup.y & ((1u << k) - 1u));
        if (pidx >= S.num_tlas_prims) { err |= ERR_BAD_INDEX; pidx = 0; }
        uint32_t inst = __ldg(&S.tlas_prims[pidx]);
        if (inst >= S.num_instances) { err |= ERR_BAD_INDEX; inst = 0; }
        if (tgroup.y > 0x00FFFFFFu) push(tgroup.x | PRIM_GROUP, tgroup.y, tmask);
        if (ngroup.y > 0x00FFFFFFu) push(ngroup.x, ngroup.y, nmask);
        const float4* ip = reinterpret_cast<const float4*>(S.inst_trace + inst);
        const float4 r0 = __ldg(ip), r1 = __ldg(ip + 1), r2 = __ldg(ip + 2);
        const uint32_t root = __ldg(reinterpret_cast<const uint32_t*>(ip + 3));
        if (m & lane_bit) {
            const float inv[12] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w, r2.x, r2.y, r2.z, r2.w};
            const uint2 c = row(2), e = row(3), f = row(4);
            const V3 wo = v3(__uint_as_float(c.x), __uint_as_float(c.y), __uint_as_float(e.x));
            const V3 wd = v3(__uint_as_float(e.y), __uint_as_float(f.x), __uint_as_float(f.y));
            const V3 oo = xform_point_rn(inv, wo);
            const V3 od = xform_dir_rn(inv, wd);
            cr = make_node_ray(oo, od);
            // (the watertight set-up waits for the instance's first triangle test)
            tr.k = INVALID; tr.Sx = od.x; tr.Sy = od.y; tr.Sz = od.z;
        }
        coct = __shfl_sync(FULL, cr.oct, __ffs(m) - 1);
        blas_sp = sp;
        level = 1;
        cur_inst = inst;
        ngroup = make_uint2(root, (1u << (24 + (ORD ? coct : 0u))) | 1u);
        nmask = m;
        tgroup = make_uint2(0u, 0u);
        tmask = 0;
    }

    // every lane with a hit leaf slot left tests its next triangle
    __device__ __forceinline__ void tri_step(const SceneDev& S) {
        bool found = false;
        unsigned e = 0;
        if (tbits) {
            const uint32_t k = __ffs(tbits) - 1;
            tbits &= tbits - 1u;
            const uint32_t pidx = tri_base + __popc(tri_leaves & ((1u << k) - 1u));
            if (pidx >= S.num_tris) e = ERR_BAD_INDEX;
            if (tr.k == INVALID) tr = wray_setup(v3(tr.Sx, tr.Sy, tr.Sz));
            const float4* tp = reinterpret_cast<const float4*>(S.tris + (e ? 0u : pidx));
            const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
            const float va[3] = {a.x, a.y, a.z}, vb[3] = {b.x, b.y, b.z}, vc[3] = {c.x, c.y, c.z};
            float t, b1, b2;
            if (intersect_tri(tr, v3(cr.ox, cr.oy, cr.oz), va, vb, vc, tmin, tmax, &t, &b1, &b2)) {
                const uint32_t prim = __float_as_uint(a.w);
                const bool better = best_inst == INVALID || t < best_t ||
                                    (t == best_t && (cur_inst < best_inst || (cur_inst == best_inst && prim < best_prim)));
                if (ANY || better) {
                    best_t = t; best_inst = cur_inst; best_prim = prim; best_u = b1; best_v = b2;
                }
                found = true;
            }
        }
        err |= __reduce_or_sync(FULL, e);
        if (ANY) {
            const uint32_t f = __ballot_sync(FULL, found);
            live &= ~f;
            if (f & lane_bit) tbits = 0;
        }
    }

    // (a pop goes straight on to its step, and a mesh node's hit triangles are tested before
    // the next turn: a 1080p frame of the sphere field 1.798 -> 1.772 ms)
    __device__ __forceinline__ void run(const SceneDev& S) {
        for (;;) {
            if (err || live == 0) return;
            if (++steps > step_limit) { err |= ERR_STEP_LIMIT; return; }
            if (tgroup.y <= 0x00FFFFFFu && ngroup.y <= 0x00FFFFFFu) {
                if (level == 1 && sp == blas_sp) { level = 0; restore_world(); coct = woct; }
                if (sp == 0) return;
                const uint4 g = lanes_pop<uint4>([&](int k) { return stk[k]; }, sp, [] { __syncwarp(); });
                if (g.x & PRIM_GROUP) { tgroup = make_uint2(g.x & ~PRIM_GROUP, g.y); tmask = g.z; }
                else { ngroup = make_uint2(g.x, g.y); nmask = g.z; }
            }
            if (tgroup.y > 0x00FFFFFFu) {
                inst_step(S);
            } else {
                node_step(S);
                if (level == 1)
                    while (__any_sync(FULL, tbits != 0u)) tri_step(S);
            }
        }
    }

    // this lane's result; an error of the packet is reported once and read as a miss
    __device__ __forceinline__ bool finish(const SceneDev& S, TraceResult& res) {
        res.hit = false;
        res.t = -1.0f; res.u = 0.0f; res.v = 0.0f; res.inst = INVALID; res.prim = INVALID;
        if (err) {
            if (S.error_word && (threadIdx.x & 31u) == 0) atomicOr(S.error_word, err);
            return false;
        }
        if (best_inst != INVALID) {
            res.hit = true; res.t = best_t; res.inst = best_inst; res.prim = best_prim; res.u = best_u; res.v = best_v;
        }
        return res.hit;
    }
};

}  // namespace snk

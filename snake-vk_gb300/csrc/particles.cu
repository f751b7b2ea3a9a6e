// particles.cu -- scene collision queries of the particle update pass.
// Compiled with --fmad=false (exact binary32 operation order, as the oracle).
//
// Reference: Core/res/shaders/ParticleUpdate.rgen
//   TraceCollisionRay ......... :101-124 (from the particle's back, speed-weighted choice)
//   ConstrainOffsetWithScene .. :126-148
//   CalculateGravity .......... :150-165
//   main (scene part) ......... :151-166
// and ParticleUpdate.rchit:41-67 (contact normal / position / velocity).
// Every query is a closest-hit trace (the shader asks for the first hit found).  A
// query runs as three launches: its rays are set up (a particle's four side by side in
// the queue's four parts, so that a warp's rays are of one kind), traced by the
// persistent closest-hit kernel of the ray queries, and turned into contacts.  A thread
// per particle that traced its rays one after the other, without ray replacement, left
// lanes waiting for the longest of 32 particles: 100,000 particles took 250 us, now 169
// (set-up 6, trace 108, contacts 14, the rest the call).
#include "snk_frame.h"
#include "snk_shade.cuh"
#include "snk_particles.h"

namespace snk {
namespace {

constexpr int PBLK = 128;
constexpr float PARTICLE_DT = 1.0f / 120.0f;   // Particle.glsl:1

struct Contact {
    V3 n;
    float dist;
    V3 p;
    V3 v;
};

__device__ __forceinline__ void store(ContactOut* out, const Contact& c) {
    ContactOut o;
    o.n[0] = c.n.x; o.n[1] = c.n.y; o.n[2] = c.n.z; o.dist = c.dist;
    o.p[0] = c.p.x; o.p[1] = c.p.y; o.p[2] = c.p.z; o.pad0 = 0.0f;
    o.v[0] = c.v.x; o.v[1] = c.v.y; o.v[2] = c.v.z; o.pad1 = 0.0f;
    *out = o;
}

__device__ __forceinline__ Contact no_contact() {
    Contact c;
    c.n = v3(0.0f, 0.0f, 0.0f); c.p = c.n; c.v = c.n;
    c.dist = -1.0f;
    return c;
}

// ParticleUpdate.rchit of a ray's closest hit
__device__ __forceinline__ Contact contact_of(const SceneDev& S, const HitDev& r, V3 o, V3 d, float timestep) {
    if (!r.flags) return no_contact();
    Contact c;
    const InstShade& I = S.inst_shade[r.inst];
    const MeshInfo& M = S.meshes[I.mesh_id];
    const uint32_t* ix = S.indices + M.index_offset + 3ull * r.prim;
    const uint32_t i0 = M.vertex_offset + ix[0], i1 = M.vertex_offset + ix[1], i2 = M.vertex_offset + ix[2];
    const V3 p0 = load3(S.positions + 3ull * i0), p1 = load3(S.positions + 3ull * i1), p2 = load3(S.positions + 3ull * i2);
    const float b0 = (1.0f - r.u) - r.v;
    const V3 p = add(add(mul(p0, b0), mul(p1, r.u)), mul(p2, r.v));
    V3 nn;
    if (M.has_normals) {
        const V3 n0 = load3(S.normals + 3ull * i0), n1 = load3(S.normals + 3ull * i1), n2 = load3(S.normals + 3ull * i2);
        nn = add(add(mul(n0, b0), mul(n1, r.u)), mul(n2, r.v));
    } else {
        nn = cross(sub(p1, p0), sub(p2, p0));
    }
    c.n = normalize(mat3_mul(I.nmat, nn));
    c.p = add(o, mul(d, r.t));
    const V3 prev = xform_point(I.pm, p);
    c.v = v3((c.p.x - prev.x) / timestep, (c.p.y - prev.y) / timestep, (c.p.z - prev.z) / timestep);
    c.dist = r.t;
    return c;
}
// the same for queue entry e
__device__ __forceinline__ Contact contact_at(const SceneDev& S, const HitDev* hits, const float4* rays, size_t e,
                                              float timestep) {
    const HitDev r = hits[e];
    if (!r.flags) return no_contact();
    const float4 a = rays[2 * e], b = rays[2 * e + 1];
    return contact_of(S, r, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), timestep);
}

__device__ __forceinline__ void put_ray(float4* rays, size_t e, V3 o, V3 d, float tmax) {
    rays[2 * e] = make_float4(o.x, o.y, o.z, 0.0f);
    rays[2 * e + 1] = make_float4(d.x, d.y, d.z, tmax);
}

__global__ void __launch_bounds__(PBLK) k_contacts(SceneDev S, const HitDev* __restrict__ hits,
                                                   const float4* __restrict__ rays, uint32_t n, float timestep,
                                                   ContactOut* out) {
    const uint32_t i = blockIdx.x * PBLK + threadIdx.x;
    if (i < n) store(out + i, contact_at(S, hits, rays, i, timestep));
}

// entries k n + i: particle i's collision rays (k = 0, 1, 2; an empty one, which hits
// nothing, for a particle asleep or at rest) and its gravity ray (k = 3); the work counter
// of the trace that follows starts at 0
__global__ void __launch_bounds__(PBLK) k_particle_rays(const ParticleDev* __restrict__ P, uint32_t n, float4* rays,
                                                        uint32_t* work) {
    const uint32_t i = blockIdx.x * PBLK + threadIdx.x;
    if (i == 0) *work = 0u;
    if (i >= n) return;
    const ParticleDev q = P[i];
    const V3 pos = v3(q.pr.x, q.pr.y, q.pr.z), vel = v3(q.vel.x, q.vel.y, q.vel.z);
    const float rad = q.pr.w;
    const bool asleep = q.vel.w < 0.5f;   // IsParticleAsleep
    const float speed = length(vel);
    const V3 down = v3(0.0f, -1.0f, 0.0f);
    if (!asleep && speed > 0.0f && speed <= 3.0e38f) {
        const V3 vdir = v3(vel.x / speed, vel.y / speed, vel.z / speed);
        const V3 right = fabsf(dot(vdir, v3(0.0f, 1.0f, 0.0f))) > 0.99f ? cross(vdir, v3(0.0f, 0.0f, 1.0f))
                                                                      : cross(vdir, v3(0.0f, 1.0f, 0.0f));
        const V3 up = cross(right, vdir);
        const V3 dirs[3] = {vdir, right, up};
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const float len = k == 0 ? speed * PARTICLE_DT + rad * 2.0f : rad * 2.0f;
            put_ray(rays, (size_t)k * n + i, sub(pos, mul(dirs[k], rad)), dirs[k], len);
        }
    } else {
        for (int k = 0; k < 3; k++) put_ray(rays, (size_t)k * n + i, pos, down, -1.0f);
    }
    put_ray(rays, 3 * (size_t)n + i, pos, down, rad + 0.001f);
}

__global__ void __launch_bounds__(PBLK) k_particle_contacts(SceneDev S, const ParticleDev* __restrict__ P,
                                                            const HitDev* __restrict__ hits,
                                                            const float4* __restrict__ rays, uint32_t n, float timestep,
                                                            ContactOut* cand_out, float* gravity) {
    const uint32_t i = blockIdx.x * PBLK + threadIdx.x;
    if (i >= n) return;
    const float4 v4 = P[i].vel;
    const V3 vel = v3(v4.x, v4.y, v4.z);
    Contact cand = no_contact();
    float best = 0.0f;
    for (int k = 0; k < 3; k++) {
        const Contact c = contact_at(S, hits, rays, (size_t)k * n + i, timestep);
        const float w = length(sub(c.v, vel));
        if (c.dist > 0.0f && w > best) { best = w; cand = c; }
    }
    store(cand_out + i, cand);
    const HitDev& g = hits[3 * (size_t)n + i];
    gravity[i] = g.flags && g.t >= 0.0f ? 0.0f : -9.8f * PARTICLE_DT;
}

// the ray of offset i (an empty one for an offset of no length)
__global__ void __launch_bounds__(PBLK) k_constrain_rays(const ParticleDev* __restrict__ P, const float* __restrict__ off,
                                                         uint32_t n, float4* rays, uint32_t* work) {
    const uint32_t i = blockIdx.x * PBLK + threadIdx.x;
    if (i == 0) *work = 0u;
    if (i >= n) return;
    const float4 pr = P[i].pr;
    const V3 o = v3(off[3ull * i], off[3ull * i + 1], off[3ull * i + 2]), pos = v3(pr.x, pr.y, pr.z);
    const float len = length(o);
    if (!(len < 0.00001f)) put_ray(rays, i, pos, v3(o.x / len, o.y / len, o.z / len), len + pr.w);
    else put_ray(rays, i, pos, v3(0.0f, -1.0f, 0.0f), -1.0f);
}

__global__ void __launch_bounds__(PBLK) k_constrain(SceneDev S, const ParticleDev* __restrict__ P,
                                                    const float* __restrict__ off, const HitDev* __restrict__ hits,
                                                    const float4* __restrict__ rays, uint32_t n, float timestep,
                                                    float* out) {
    const uint32_t i = blockIdx.x * PBLK + threadIdx.x;
    if (i >= n) return;
    const V3 o = v3(off[3ull * i], off[3ull * i + 1], off[3ull * i + 2]);
    V3 res = v3(0.0f, 0.0f, 0.0f);
    if (!(length(o) < 0.00001f)) {
        const float rad = P[i].pr.w;
        const Contact c = contact_at(S, hits, rays, i, timestep);
        if (c.dist > 0.0f) {
            const float4 b = rays[2ull * i + 1];
            const float m = fmaxf(c.dist - rad * 0.9f, 0.0f), s = rad * 0.05f;
            res = add(mul(v3(b.x, b.y, b.z), m), mul(c.n, s));
        } else {
            res = o;
        }
    }
    out[3ull * i] = res.x; out[3ull * i + 1] = res.y; out[3ull * i + 2] = res.z;
}

inline unsigned pgrid(uint32_t n) { return (n + PBLK - 1) / PBLK; }

cudaError_t trace(const SceneDev& S, const ContactScratch& c, const float4* rays, uint32_t n, cudaStream_t s) {
    return launch_trace_rays(S, rays, n, c.hits, false, c.work, c.grid, c.tune, s);
}

}  // namespace

cudaError_t launch_contact_rays(const SceneDev& S, const float4* rays, uint32_t n, float timestep, ContactOut* out,
                                const ContactScratch& c, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(c.work, 0, sizeof(uint32_t), s);
    if (e == cudaSuccess) e = trace(S, c, rays, n, s);
    if (e != cudaSuccess) return e;
    k_contacts<<<pgrid(n), PBLK, 0, s>>>(S, c.hits, rays, n, timestep, out);
    return cudaGetLastError();
}

cudaError_t launch_particle_probe(const SceneDev& S, const ParticleDev* p, uint32_t n, float timestep,
                                  ContactOut* cand, float* gravity, const ContactScratch& c, cudaStream_t s) {
    k_particle_rays<<<pgrid(n), PBLK, 0, s>>>(p, n, c.rays, c.work);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = trace(S, c, c.rays, 4u * n, s);
    if (e != cudaSuccess) return e;
    k_particle_contacts<<<pgrid(n), PBLK, 0, s>>>(S, p, c.hits, c.rays, n, timestep, cand, gravity);
    return cudaGetLastError();
}

cudaError_t launch_particle_constrain(const SceneDev& S, const ParticleDev* p, const float* off, uint32_t n,
                                      float timestep, float* out, const ContactScratch& c, cudaStream_t s) {
    k_constrain_rays<<<pgrid(n), PBLK, 0, s>>>(p, off, n, c.rays, c.work);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = trace(S, c, c.rays, n, s);
    if (e != cudaSuccess) return e;
    k_constrain<<<pgrid(n), PBLK, 0, s>>>(S, p, off, c.hits, c.rays, n, timestep, out);
    return cudaGetLastError();
}

}  // namespace snk

// snk_particles.h -- device records and launches of the particle collision queries
// (particles.cu); layouts equal snk_particle / snk_contact of the C ABI.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "snk_frame.h"

namespace snk {

struct ParticleDev { float4 pr, vel, col; };
struct ContactOut { float n[3]; float dist; float p[3]; float pad0; float v[3]; float pad1; };
static_assert(sizeof(ParticleDev) == 48 && sizeof(ContactOut) == 48, "particle record layouts");

// scratch of one query: rays (2 float4 each) and hits of its queue, the trace's work
// counter, and how the trace is launched
struct ContactScratch {
    float4* rays;
    HitDev* hits;
    uint32_t items;   // of a part at most (particles, offsets or rays)
    uint32_t* work;
    int grid;
    TraceTuning tune;
};

// (rays: caller's; the particle queries set theirs up in the scratch: 4 per particle, 1 per offset)
cudaError_t launch_contact_rays(const SceneDev& S, const float4* rays, uint32_t n, float timestep, ContactOut* out,
                                const ContactScratch& c, cudaStream_t s);
cudaError_t launch_particle_probe(const SceneDev& S, const ParticleDev* p, uint32_t n, float timestep,
                                  ContactOut* cand, float* gravity, const ContactScratch& c, cudaStream_t s);
cudaError_t launch_particle_constrain(const SceneDev& S, const ParticleDev* p, const float* off, uint32_t n,
                                      float timestep, float* out, const ContactScratch& c, cudaStream_t s);

}  // namespace snk

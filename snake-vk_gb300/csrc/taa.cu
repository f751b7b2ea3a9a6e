// taa.cu -- temporal anti-aliasing resolve of the path tracer's radiance.
//
// Restates TAA_Resolve.comp (Core/res/shaders/TAA_Resolve.comp:12-86) and the
// history handling of TAA_ResolvePass (Core/src/renderpasses/TAA_ResolvePass.cpp:
// 6-56).  Compiled with --fmad=false: every operation is a binary32 basic
// operation in the shader's order, so the CPU oracle reproduces it bit for bit.
//
// Differences from the pass, by design:
//   * out-of-place: every pixel reads the unresolved frame (the shader resolves
//     img_current_frame in place, so a pixel's 3x3 neighbourhood may already hold
//     resolved values of neighbouring invocations);
//   * every pixel is resolved (the pass dispatches floor(W/8) x floor(H/8) groups
//     and leaves a right/bottom remainder unresolved when W or H is not a
//     multiple of 8);
//   * bilinear history/velocity fetches in FP32 with exact weights (texture units
//     quantise the weights to a few bits);
//   * the history starts as the first frame (the pass's history image starts
//     undefined).
//
// Kernel: 32x8 pixels per block, the 34x10 halo tile of the current frame staged
// in shared memory (coalesced float4 loads, issued first and held in registers
// until the motion-dependent gathers are in flight), history and previous
// velocity fetched through L1 (neighbouring pixels share texels).  88 B per
// pixel (16 current + 8 motion + 16 history + 8 previous motion in; 16 out, 16
// next history, 8 next previous motion).  The first frame reads itself as its history.
#include <cstring>
#include <string>

#include "snk_host.h"
#include "../../include/snk_pt.h"

namespace snk {
namespace {

constexpr int TX = 32, TY = 8;
constexpr int HALO = 2 * (TX + 2) + 2 * TY;
static_assert(HALO <= TX * TY, "one halo texel per thread");
// blocks between a block and the one whose texels it prefetches into L2: about twice
// as many as run at once
constexpr int PREFETCH_BLOCKS = 912;

struct TaaImages {
    const float4* cur;
    const float2* motion;
    const float4* hist;
    const float2* pmot;
    float4* out;        // may be null
    float4* hist_next;
    float2* pmot_next;
    int w, h;
    int ahead;          // rows of blocks from a block down to the one it prefetches for
};

// repeat addressing of a texel index in [-n, 2n): the coordinate is clamped to [0, 1], so
// the filter's texels are at most one image away
__device__ __forceinline__ int wrap_repeat(int i, int n) {
    if (i < 0) i += n;
    return i >= n ? i - n : i;
}

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

// two channels per addition, each rounded by itself (packed products feeding packed
// additions came back fused, so the products stay single)
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(*reinterpret_cast<unsigned long long*>(&a)),
        "l"(*reinterpret_cast<unsigned long long*>(&b)));
    return *reinterpret_cast<float2*>(&d);
}
// texture() with a linear filter and repeat addressing, in FP32: the four texels
// are fetched first (so that their loads are in flight together with the
// frame's tile), the weights are applied later
template <class T>
struct Bilinear {
    T t00, t10, t01, t11;
    float w00, w10, w01, w11;
    __device__ __forceinline__ void fetch(const T* __restrict__ img, int w, int h, float cu, float cv) {
        const float u = cu * (float)w - 0.5f, v = cv * (float)h - 0.5f;
        const float fu = floorf(u), fv = floorf(v);
        const float a = u - fu, b = v - fv;
        const int i0 = wrap_repeat((int)fu, w), i1 = wrap_repeat((int)fu + 1, w);
        const int j0 = wrap_repeat((int)fv, h), j1 = wrap_repeat((int)fv + 1, h);
        w00 = (1.0f - a) * (1.0f - b); w10 = a * (1.0f - b); w01 = (1.0f - a) * b; w11 = a * b;
        const uint32_t r0 = (uint32_t)(j0 * w), r1 = (uint32_t)(j1 * w);   // (an image has at most 2^30 texels)
        t00 = img[r0 + i0];
        t10 = img[r0 + i1];
        t01 = img[r1 + i0];
        t11 = img[r1 + i1];
    }
    // component k of the filtered value
    __device__ __forceinline__ float at(int k) const {
        const float* a = reinterpret_cast<const float*>(&t00);
        const float* b = reinterpret_cast<const float*>(&t10);
        const float* c = reinterpret_cast<const float*>(&t01);
        const float* d = reinterpret_cast<const float*>(&t11);
        return ((w00 * a[k] + w10 * b[k]) + w01 * c[k]) + w11 * d[k];
    }
};

// The resolve of one pixel from its neighbourhood's sums and bounds.
__device__ __forceinline__ float4 resolve_pixel(const float4 cur4, const float* mn, const float* mx, const float* m,
                                                const float* m2, const Bilinear<float4>& hb, const Bilinear<float2>& pb,
                                                float2 vel) {
    const float cur[3] = {cur4.x, cur4.y, cur4.z};
    const float inv9 = 1.0f / 9.0f, gamma = 0.55f, eps = 0.00000001f;
    float mu[3], minc[3], maxc[3], p[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        mu[c] = m[c] * inv9;
        const float sigma = sqrtf(fabsf(m2[c] * inv9 - mu[c] * mu[c]));
        minc[c] = mu[c] - gamma * sigma;
        maxc[c] = mu[c] + gamma * sigma;
        p[c] = fminf(fmaxf(mu[c], mn[c]), mx[c]);
    }
    // clip_aabb(minc, maxc, vec4(p, 1), vec4(hist, 1)); r.w stays 0
    float r[3];
#pragma unroll
    for (int c = 0; c < 3; c++) r[c] = fmaxf(hb.at(c), 0.0f) - p[c];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const float rmax = maxc[c] - p[c];
        if (r[c] > rmax + eps) {
            const float s = rmax / r[c];
            for (int k = 0; k < 3; k++) r[k] = r[k] * s;
        }
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const float rmin = minc[c] - p[c];
        if (r[c] < rmin - eps) {
            const float s = rmin / r[c];
            for (int k = 0; k < 3; k++) r[k] = r[k] * s;
        }
    }
    const float vx = pb.at(0) + vel.x, vy = pb.at(1) + vel.y;
    const float vlen = sqrtf(vx * vx + vy * vy);
    const float dis = fminf(fmaxf((vlen - 0.001f) * 10.0f, 0.0f), 1.0f);
    float fin[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const float hc = p[c] + r[c];
        const float f = cur[c] * (1.0f - 0.9f) + hc * 0.9f;
        fin[c] = f * (1.0f - dis) + mu[c] * dis;
    }
    return make_float4(fin[0], fin[1], fin[2], 1.0f);
}

// Bound by latency and issue: a thread waits for its motion, then for the texels that
// it points to, with 24 warps per SM to cover both, and runs some 570 instructions (the
// exact divisions and square roots among them).  So a block asks L2 for the texels of
// one that runs later, neither index needs a division, and the bounds take three
// operands at a time: a 1080p resolve whose images are partly in L2 43 us, 50 before (49
// without the prefetch); after an L2 flush 60 us, 72 before, 88 B per pixel at 3.0 TB/s.  (Two
// pixels per thread need 126 registers and were slower, as were 512-thread blocks; 64
// registers changed nothing.)
__global__ void __launch_bounds__(TX * TY) k_taa_resolve(TaaImages I) {
    __shared__ float4 tile[TY + 2][TX + 2];   // clamped to >= 0, as the neighbourhood takes it
    const int bx = blockIdx.x * TX, by = blockIdx.y * TY;
    const int t = threadIdx.y * TX + threadIdx.x;
    const int x = bx + threadIdx.x, y = by + threadIdx.y;
    const bool inside = x < I.w && y < I.h;
    const uint32_t pix = inside ? (uint32_t)(y * I.w + x) : 0u;
    auto texel = [&](int lx, int ly) {   // tile entry (lx, ly): the frame's texel, its edges repeated
        const int gx = min(max(bx + lx - 1, 0), I.w - 1), gy = min(max(by + ly - 1, 0), I.h - 1);
        return I.cur[(uint32_t)(gy * I.w + gx)];
    };
    auto positive = [](float4 c) { return make_float4(fmaxf(c.x, 0.0f), fmaxf(c.y, 0.0f), fmaxf(c.z, 0.0f), 0.0f); };
    // the loads that wait for nothing: this thread's texel and motion, one halo texel
    const float2 vel = inside ? I.motion[pix] : make_float2(0.0f, 0.0f);
    const float4 own = texel(threadIdx.x + 1, threadIdx.y + 1);
    float4 halo;
    int hx = 0, hy = 0;
    if (t < HALO) {
        if (t < 2 * (TX + 2)) {
            hx = t < TX + 2 ? t : t - (TX + 2);
            hy = t < TX + 2 ? 0 : TY + 1;
        } else {
            hx = (t & 1) * (TX + 1);
            hy = 1 + ((t - 2 * (TX + 2)) >> 1);
        }
        halo = texel(hx, hy);
    }
    {   // the later block's rows of the four images, one 128-byte line per thread: 4 lines
        // of the frame and of the history, 2 of each motion
        const int py = by + I.ahead * TY + (t & (TY - 1)), line = t / TY;
        const int px = line < 8 ? bx + 8 * (line & 3) : bx + 16 * (line & 1);
        if (line < 12 && py < I.h && px < I.w) {
            const uint32_t at = (uint32_t)(py * I.w + px);
            const void* p = line < 4 ? (const void*)(I.cur + at) : line < 8 ? (const void*)(I.hist + at)
                          : line < 10 ? (const void*)(I.motion + at) : (const void*)(I.pmot + at);
            asm volatile("prefetch.global.L2 [%0];" :: "l"(p));
        }
    }
    // then the reprojected history and previous velocity
    Bilinear<float4> hb;
    Bilinear<float2> pb;
    if (inside) {
        float u = ((float)x + 0.5f) / (float)I.w + vel.x;
        float v = ((float)y + 0.5f) / (float)I.h + vel.y;
        u = fminf(fmaxf(u, 0.0f), 1.0f);
        v = fminf(fmaxf(v, 0.0f), 1.0f);
        hb.fetch(I.hist, I.w, I.h, u, v);
        pb.fetch(I.pmot, I.w, I.h, u, v);
    }
    tile[threadIdx.y + 1][threadIdx.x + 1] = positive(own);
    if (t < HALO) tile[hy][hx] = positive(halo);
    __syncthreads();
    if (!inside) return;
    // neighbourhood sums in the shader's order (columns, then rows) and bounds
    float2 sxy = make_float2(0.0f, 0.0f), qxy = sxy;
    float sz = 0.0f, qz = 0.0f;
    float mn[3] = {9999.0f, 9999.0f, 9999.0f}, mx[3] = {-9999.0f, -9999.0f, -9999.0f};
#pragma unroll
    for (int ox = 0; ox < 3; ox++) {
        float4 col[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const float4 c = col[k] = tile[threadIdx.y + k][threadIdx.x + ox];
            sxy = add2(sxy, make_float2(c.x, c.y));
            qxy = add2(qxy, make_float2(c.x * c.x, c.y * c.y));
            sz = sz + c.z;
            qz = qz + c.z * c.z;
        }
        mn[0] = fminf(min3f(mn[0], col[0].x, col[1].x), col[2].x); mx[0] = fmaxf(max3f(mx[0], col[0].x, col[1].x), col[2].x);
        mn[1] = fminf(min3f(mn[1], col[0].y, col[1].y), col[2].y); mx[1] = fmaxf(max3f(mx[1], col[0].y, col[1].y), col[2].y);
        mn[2] = fminf(min3f(mn[2], col[0].z, col[1].z), col[2].z); mx[2] = fmaxf(max3f(mx[2], col[0].z, col[1].z), col[2].z);
    }
    const float m[3] = {sxy.x, sxy.y, sz}, m2[3] = {qxy.x, qxy.y, qz};
    const float4 o = resolve_pixel(own, mn, mx, m, m2, hb, pb, vel);
    if (I.out) I.out[pix] = o;
    I.hist_next[pix] = o;
    I.pmot_next[pix] = vel;
}

}  // namespace
}  // namespace snk

using namespace snk;

struct snk_taa {
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    uint32_t w = 0, h = 0;
    DBuf<float4> hist[2];
    DBuf<float2> pmot[2];
    DBuf<float4> stage_in, stage_out;
    DBuf<float2> stage_motion;
    int cur = 0;
    bool valid = false;
    std::string err;
};

namespace {
int taa_fail(snk_taa* t, int code, const std::string& msg) {
    if (t) t->err = msg;
    return code;
}
}  // namespace

extern "C" {

int snk_taa_create(int32_t device, void* stream, uint32_t width, uint32_t height, snk_taa** out) {
    if (!out || width == 0 || height == 0 || (uint64_t)width * height > (1ull << 30)) return SNK_ERR_INVALID_ARG;
    *out = nullptr;
    if (cudaSetDevice(device) != cudaSuccess) return SNK_ERR_CUDA;
    snk_taa* t = new snk_taa();
    t->device = device;
    t->w = width;
    t->h = height;
    if (stream) {
        t->stream = (cudaStream_t)stream;
    } else {
        if (cudaStreamCreateWithFlags(&t->stream, cudaStreamNonBlocking) != cudaSuccess) { delete t; return SNK_ERR_CUDA; }
        t->own_stream = true;
    }
    const size_t np = (size_t)width * height;
    for (int k = 0; k < 2; k++)
        if (t->hist[k].reserve(np) != cudaSuccess || t->pmot[k].reserve(np) != cudaSuccess) {
            if (t->own_stream) cudaStreamDestroy(t->stream);
            delete t;
            return SNK_ERR_OUT_OF_MEMORY;
        }
    *out = t;
    return SNK_OK;
}

int snk_taa_destroy(snk_taa* t) {
    if (!t) return SNK_OK;
    cudaSetDevice(t->device);
    cudaStreamSynchronize(t->stream);
    if (t->own_stream) cudaStreamDestroy(t->stream);
    delete t;
    return SNK_OK;
}

int snk_taa_reset(snk_taa* t) {
    if (!t) return SNK_ERR_INVALID_ARG;
    t->valid = false;
    return SNK_OK;
}

int snk_taa_resolve(snk_taa* t, const float* radiance, const float* motion, float* out, uint32_t memory) {
    if (!t || !radiance || !motion || !out || memory > SNK_MEM_HOST)
        return taa_fail(t, SNK_ERR_INVALID_ARG, "taa_resolve: bad arguments");
    if (cudaSetDevice(t->device) != cudaSuccess) return taa_fail(t, SNK_ERR_CUDA, "taa_resolve: device");
    const size_t np = (size_t)t->w * t->h;
    cudaStream_t st = t->stream;
    const float4* cur = reinterpret_cast<const float4*>(radiance);
    const float2* mot = reinterpret_cast<const float2*>(motion);
    if (memory == SNK_MEM_HOST) {
        if (t->stage_in.reserve(np) || t->stage_motion.reserve(np))
            return taa_fail(t, SNK_ERR_OUT_OF_MEMORY, "taa_resolve: staging");
        if (cudaMemcpyAsync(t->stage_in.p, radiance, np * sizeof(float4), cudaMemcpyHostToDevice, st) ||
            cudaMemcpyAsync(t->stage_motion.p, motion, np * sizeof(float2), cudaMemcpyHostToDevice, st))
            return taa_fail(t, SNK_ERR_CUDA, "taa_resolve: upload");
        cur = t->stage_in.p;
        mot = t->stage_motion.p;
    } else if (reinterpret_cast<uintptr_t>(radiance) % 16 || reinterpret_cast<uintptr_t>(motion) % 8 ||
               reinterpret_cast<uintptr_t>(out) % 16) {
        return taa_fail(t, SNK_ERR_INVALID_ARG, "taa_resolve: device buffers must be 16-byte (radiance, out) "
                                                "and 8-byte (motion) aligned");
    }
    const int nxt = t->cur ^ 1;
    TaaImages I;
    I.cur = cur;
    I.motion = mot;
    // first frame: the history is the current frame, the previous motion this frame's
    I.hist = t->valid ? t->hist[t->cur].p : cur;
    I.pmot = t->valid ? t->pmot[t->cur].p : mot;
    // in place (or host output): write the history only, then copy it out
    const bool direct = memory == SNK_MEM_DEVICE && out != radiance;
    I.out = direct ? reinterpret_cast<float4*>(out) : nullptr;
    I.hist_next = t->hist[nxt].p;
    I.pmot_next = t->pmot[nxt].p;
    I.w = (int)t->w;
    I.h = (int)t->h;
    dim3 grid((t->w + TX - 1) / TX, (t->h + TY - 1) / TY);
    I.ahead = (PREFETCH_BLOCKS + (int)grid.x - 1) / (int)grid.x;
    k_taa_resolve<<<grid, dim3(TX, TY), 0, st>>>(I);
    if (cudaGetLastError() != cudaSuccess) return taa_fail(t, SNK_ERR_CUDA, "taa_resolve: launch");
    if (!direct) {
        if (cudaMemcpyAsync(out, t->hist[nxt].p, np * sizeof(float4),
                            memory == SNK_MEM_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice, st))
            return taa_fail(t, SNK_ERR_CUDA, "taa_resolve: copy out");
    }
    if (memory == SNK_MEM_HOST && cudaStreamSynchronize(st) != cudaSuccess)
        return taa_fail(t, SNK_ERR_CUDA, "taa_resolve: synchronise");
    t->cur = nxt;
    t->valid = true;
    return SNK_OK;
}

int snk_taa_get_last_error(const snk_taa* t, char* buf, size_t len) {
    if (!t || !buf || len == 0) return SNK_ERR_INVALID_ARG;
    std::strncpy(buf, t->err.c_str(), len - 1);
    buf[len - 1] = 0;
    return SNK_OK;
}

}  // extern "C"

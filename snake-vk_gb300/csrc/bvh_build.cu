// bvh_build.cu -- GPU construction of 8-wide compressed BVHs.
//
// Replaces the driver-built acceleration structures of the reference:
//   BLAS::GenerateFromMeshData   Core/src/resources/TLAS.cpp:109-186 (per submesh, at load)
//   TLAS::BuildFromInstances     Core/src/resources/TLAS.cpp:10-87   (full rebuild every frame,
//                                Core/src/scene/TlasSystem.cpp:16-20,27-49)
//
// Pipeline (all on the device, one stream, no host round trip).  A build takes the
// primitives of any number of trees (the meshes of a scene, one after another; the
// instance BVH is one tree), so that loading many submeshes costs the launches and
// the dependent steps of one (50 small meshes: 807 launches and 29.3 ms one mesh and
// one host-read level at a time, 31 launches and 1.63 ms together; a 131,072-triangle
// terrain and a sphere 3.66 and 2.46 ms):
//   1. centroid bounds of each tree (block reduction + order-preserving atomics)
//   2. 63-bit Morton codes of the centroids (21 bits per axis)
//   3. sort of (tree, code, primitive) (project kernels below: a bitonic network in one
//      CTA's shared memory for one small tree, else an LSD radix sort, one kernel per digit)
//   4. binary radix trees (Karras, HPG 2012): one thread per internal node
//   5. boxes and leaf counts, bottom-up (atomic arrival flags), in the first of the
//      climbs below that runs
//   5b. treelet restructuring (Karras & Aila, HPG 2013): bottom-up over the binary
//      tree, every node whose subtree holds >= 7 primitives roots a treelet of 7
//      leaves (grown by opening the largest-area treelet leaf); one warp finds the
//      SAH-optimal binary topology of those 7 leaves by dynamic programming over
//      all 127 leaf subsets and every 2-partition of each, and rewrites the
//      treelet's 6 internal nodes in place.  Subtrees of at most leaf_max primitives
//      are costed as the leaves the collapse will make of them.  Repeated for a few
//      passes; the result is deterministic (each treelet depends only on its
//      finished subtrees, ties break on the lowest subset index).
//   5c. least-SAH choice of every wide node's children (bottom-up)
//   6. top-down collapse to 8-wide nodes, one warp per output node, level by
//      level: a node's children are the least-SAH choice or, with greedy collapse,
//      start as its binary children, of which the internal one
//      with the largest surface area and more than leaf_max primitives is replaced
//      by its two children until 8 children exist or none can be opened.  Children
//      with <= leaf_pack primitives (leaf_max <= leaf_pack <= 4) become leaves: a
//      full node keeps small subtrees as multi-primitive leaves instead of
//      spending a sparsely filled child node on them.  Children are assigned to the 8 slots greedily by how
//      well their centroid offset matches each octant corner, so that visiting
//      slot ^ ray_octant in increasing order is roughly front to back.  Child boxes
//      are quantised outwards to 8 bits per plane.
//   7. SAH cost of the result (for quality reporting).
//
// Binary node ids: internal node i of the tree whose primitives start at f is f + i
// (its root is f), the leaf at sorted position j is N + j, N the primitives of the
// whole build.
//
// The per-frame instance BVH of up to 1024 instances is built by one single-CTA
// launch instead (k_build_small: clustering in shared memory, then treelet passes
// and the same collapse).

#include <algorithm>

#include "snk_host.h"

namespace snk {
namespace {

constexpr int BLK = 256;

__device__ __forceinline__ unsigned enc_f(float f) {
    unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float dec_f(unsigned u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// loads of tree data written by other threads during the build: through L2 for
// global memory (G), plain for shared memory (the single-CTA builder)
template <bool G, class T>
__device__ __forceinline__ T ldx(const T* p) {
    if constexpr (G) return __ldcg(p);
    else return *p;
}

// the tree of primitive i / where tree t's primitives begin and end
__device__ __forceinline__ uint32_t tree_of(const BuildTrees& B, uint32_t i) {
    uint32_t lo = 0, hi = B.count - 1u;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1u) >> 1;
        if (__ldg(B.first + mid) <= i) lo = mid;
        else hi = mid - 1u;
    }
    return lo;
}
__device__ __forceinline__ uint32_t tree_begin(const BuildTrees& B, uint32_t t) {
    return B.count == 1u ? 0u : __ldg(B.first + t);
}
__device__ __forceinline__ uint32_t tree_end(const BuildTrees& B, uint32_t t) {
    return B.count == 1u ? B.total : __ldg(B.first + t + 1u);
}

// Centroid bounds of every tree, 6 words each (zero at the start): the largest ~enc of
// x, y, z (whose complement is the smallest) and the largest enc.  A block inside one
// tree reduces before its atomics.
__global__ void __launch_bounds__(BLK) k_centroid_bounds(const float4* __restrict__ lo, const float4* __restrict__ hi,
                                                         BuildTrees B, unsigned* cb) {
    __shared__ unsigned red[6][BLK / 32];
    const uint32_t b0 = blockIdx.x * BLK, i = b0 + threadIdx.x;
    const bool valid = i < B.total;
    const uint32_t last = min(b0 + BLK, B.total) - 1u;
    unsigned v[6] = {0u, 0u, 0u, 0u, 0u, 0u};
    if (valid) {
        const float4 a = lo[i], b = hi[i];
        const float c[3] = {0.5f * (a.x + b.x), 0.5f * (a.y + b.y), 0.5f * (a.z + b.z)};
        for (int k = 0; k < 3; k++) {
            const unsigned e = enc_f(c[k]);
            v[k] = ~e;
            v[3 + k] = e;
        }
    }
    const uint32_t t0 = tree_of(B, b0);
    if (last < tree_end(B, t0)) {
        for (int k = 0; k < 6; k++) {
            const unsigned m = __reduce_max_sync(0xFFFFFFFFu, v[k]);
            if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = m;
        }
        __syncthreads();
        if (threadIdx.x < 6) {
            unsigned m = 0u;
            for (int w = 0; w < BLK / 32; w++) m = max(m, red[threadIdx.x][w]);
            atomicMax(&cb[6ull * t0 + threadIdx.x], m);
        }
    } else if (valid) {
        unsigned* dst = cb + 6ull * tree_of(B, i);
        for (int k = 0; k < 6; k++) atomicMax(&dst[k], v[k]);
    }
}

__device__ __forceinline__ unsigned long long spread21(unsigned long long x) {
    x &= 0x1FFFFFull;
    x = (x | (x << 32)) & 0x1F00000000FFFFull;
    x = (x | (x << 16)) & 0x1F0000FF0000FFull;
    x = (x | (x << 8)) & 0x100F00F00F00F00Full;
    x = (x | (x << 4)) & 0x10C30C30C30C30C3ull;
    x = (x | (x << 2)) & 0x1249249249249249ull;
    return x;
}

// cb: encoded centroid bounds (min xyz, max xyz)
__device__ __forceinline__ unsigned long long morton_of(float4 a, float4 b, const unsigned* cb) {
    float c[3] = {0.5f * (a.x + b.x), 0.5f * (a.y + b.y), 0.5f * (a.z + b.z)};
    unsigned long long q[3];
    for (int k = 0; k < 3; k++) {
        float mn = dec_f(cb[k]), mx = dec_f(cb[3 + k]);
        float ext = mx - mn;
        float f = ext > 0.0f ? (c[k] - mn) / ext : 0.5f;
        f = fminf(fmaxf(f, 0.0f), 1.0f);
        q[k] = (unsigned long long)fminf(f * 2097152.0f, 2097151.0f);
    }
    return (spread21(q[0]) << 2) | (spread21(q[1]) << 1) | spread21(q[2]);
}

__device__ __forceinline__ int delta(const unsigned long long* __restrict__ k, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    unsigned long long a = k[i], b = k[j];
    if (a == b) return 64 + __clz((unsigned)(i ^ j));
    return __clzll(a ^ b);
}

__device__ __forceinline__ void karras_node(int i, const unsigned long long* __restrict__ keys, int n, uint32_t first,
                                            uint32_t total, int2* children, int* parent) {
    int d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
    int dmin = delta(keys, n, i, i - d);
    int lmax = 2;
    while (delta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
    int j = i + l * d;
    int dnode = delta(keys, n, i, j);
    int s = 0, t = l;
    do {
        t = (t + 1) >> 1;
        if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    int gamma = i + s * d + min(d, 0);
    const int left = (int)first + gamma + (min(i, j) == gamma ? (int)total : 0);
    const int right = (int)first + gamma + 1 + (max(i, j) == gamma + 1 ? (int)total : 0);
    const int self = (int)first + i;
    children[self] = make_int2(left, right);
    parent[left] = self;
    parent[right] = self;
}

// ---- radix sort of (tree, 63-bit Morton code, primitive) ------------------------------
// LSD radix sort with 8-bit digits, one kernel per digit: the code's eight, then the
// digits of the tree's number when a build has several trees.  Every pass is stable:
// the elements of one digit keep their current order.  A CTA owns a tile of the
// input; it adds up the digit counts of the tiles before its own (and of all tiles,
// for the digits' starts), then ranks a chunk of 1024 consecutive elements at a time:
// lanes holding the same digit find each other with __match_any_sync (their order
// within the warp is their lane order), every warp counts its digits in shared
// memory, and an exclusive scan of those counts over the warps gives each warp its
// start within the digit.  As it stores an element it counts the element's next digit
// for the tile it lands in, so a pass needs no counting or scanning launch of its own.
// Bound by latency at the sizes of a scene: tiles of 1024 put 131,072 elements on 128
// SMs, nine launches of about 9 us for 132,352 keys of two trees (tiles of 4096 and three
// launches per digit took 24 launches and 185 us).
constexpr int SORT_THREADS = 1024;
constexpr int SORT_WARPS = SORT_THREADS / 32;
constexpr int SORT_RADIX = 256;
constexpr int SORT_CODE_PASSES = 8;                // 64 bits (the codes use 63)
constexpr uint32_t SORT_TILES = 160;               // tiles of a pass, about one per SM

struct SortSmem {
    uint32_t wcnt[SORT_WARPS][SORT_RADIX];   // per-warp digit counts, then their exclusive scan
    uint32_t base[SORT_RADIX];               // next output position of each digit
    uint32_t total[SORT_RADIX];              // the current chunk's count of each digit
    uint32_t warp_sum[SORT_RADIX / 32];
};

// digit `pass` of an element: of its code, or of its tree's number
__device__ __forceinline__ uint32_t sort_digit(int pass, unsigned long long k, uint32_t v, const BuildTrees& B) {
    if (pass < SORT_CODE_PASSES) return (uint32_t)(k >> (8 * pass)) & (SORT_RADIX - 1u);
    return (tree_of(B, v) >> (8 * (pass - SORT_CODE_PASSES))) & (SORT_RADIX - 1u);
}

// Morton codes within each tree's centroid bounds; hist: digit 0 of every tile (zero at
// the start; null when the codes are not radix-sorted)
__global__ void k_morton(const float4* __restrict__ lo, const float4* __restrict__ hi, BuildTrees B, const unsigned* cb,
                         unsigned long long* keys, uint32_t* vals, uint32_t* hist, uint32_t tile_shift) {
    const uint32_t i = blockIdx.x * BLK + threadIdx.x;
    if (i >= B.total) return;
    const unsigned* c = cb + 6ull * tree_of(B, i);
    const unsigned bounds[6] = {~__ldg(c), ~__ldg(c + 1), ~__ldg(c + 2), __ldg(c + 3), __ldg(c + 4), __ldg(c + 5)};
    const unsigned long long k = morton_of(lo[i], hi[i], bounds);
    keys[i] = k;
    vals[i] = i;
    if (hist) atomicAdd(&hist[(size_t)(i >> tile_shift) * SORT_RADIX + sort_digit(0, k, i, B)], 1u);
}

// Output position of this thread's element (valid, digit d) in a chunk of one
// element per thread, in thread order; then base advances past the chunk.
__device__ __forceinline__ uint32_t rank_chunk(SortSmem& S, bool valid, uint32_t d) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int i = t; i < SORT_WARPS * SORT_RADIX; i += SORT_THREADS) (&S.wcnt[0][0])[i] = 0u;
    __syncthreads();
    const uint32_t key = valid ? d : (uint32_t)(SORT_RADIX + lane);   // lanes without an element match nobody
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, key);
    const uint32_t before = (uint32_t)__popc(peers & ((1u << lane) - 1u));
    if (valid && before == 0u) S.wcnt[warp][d] = (uint32_t)__popc(peers);
    __syncthreads();
    if (t < SORT_RADIX) {
        uint32_t run = 0;
#pragma unroll 8
        for (int w = 0; w < SORT_WARPS; w++) {
            const uint32_t c = S.wcnt[w][t];
            S.wcnt[w][t] = run;
            run += c;
        }
        S.total[t] = run;
    }
    __syncthreads();
    const uint32_t pos = valid ? S.base[d] + S.wcnt[warp][d] + before : 0u;
    __syncthreads();
    if (t < SORT_RADIX) S.base[t] += S.total[t];
    return pos;   // (the next chunk's first barrier orders the base update)
}

// One digit of the sort.  hist: this digit's counts, 256 per tile; hist_next: the next
// digit's, zero at the start (null at the last digit).  tile = 1 << tile_shift elements.
__global__ void __launch_bounds__(SORT_THREADS, 1) k_sort_pass(const unsigned long long* __restrict__ sk,
                                                             const uint32_t* __restrict__ sv, BuildTrees B, int pass,
                                                             uint32_t tile_shift, const uint32_t* __restrict__ hist,
                                                             uint32_t* hist_next, unsigned long long* dk, uint32_t* dv) {
    __shared__ SortSmem S;
    const uint32_t t = threadIdx.x, n = B.total;
    {   // four rows of counts at a time: the tiles before this one, and all of them
        const uint32_t d = t & (SORT_RADIX - 1u), group = t / SORT_RADIX;
        uint32_t before = 0, all = 0;
#pragma unroll 8
        for (uint32_t r = group; r < gridDim.x; r += SORT_THREADS / SORT_RADIX) {
            const uint32_t c = __ldg(&hist[(size_t)r * SORT_RADIX + d]);
            all += c;
            if (r < blockIdx.x) before += c;
        }
        S.wcnt[group][d] = before;
        S.wcnt[SORT_THREADS / SORT_RADIX + group][d] = all;
    }
    __syncthreads();
    const uint32_t lane = t & 31u;
    uint32_t before = 0, sum = 0, incl = 0;
    if (t < SORT_RADIX) {
        for (int g = 0; g < SORT_THREADS / SORT_RADIX; g++) {
            before += S.wcnt[g][t];
            sum += S.wcnt[SORT_THREADS / SORT_RADIX + g][t];
        }
        incl = sum;
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += u;
        }
        if (lane == 31u) S.warp_sum[t >> 5] = incl;
    }
    __syncthreads();
    if (t < SORT_RADIX) {
        uint32_t off = 0;
        for (uint32_t w = 0; w < (t >> 5); w++) off += S.warp_sum[w];
        S.base[t] = off + incl - sum + before;
    }
    __syncthreads();
    const uint32_t b0 = blockIdx.x << tile_shift, b1 = min(b0 + (1u << tile_shift), n);
    for (uint32_t c = b0; c < b1; c += SORT_THREADS) {
        const uint32_t i = c + t;
        const bool valid = i < b1;
        const unsigned long long k = valid ? sk[i] : 0ull;
        const uint32_t v = valid ? sv[i] : 0u;
        const uint32_t pos = rank_chunk(S, valid, valid ? sort_digit(pass, k, v, B) : 0u);
        if (valid) {
            dk[pos] = k;
            dv[pos] = v;
            if (hist_next)
                atomicAdd(&hist_next[(size_t)(pos >> tile_shift) * SORT_RADIX + sort_digit(pass + 1, k, v, B)], 1u);
        }
    }
}

// One tree of up to SORT_BITONIC_MAX primitives is sorted by one CTA in shared
// memory with a bitonic network (78 barrier-separated compare-exchange stages for
// 4096 entries, one launch instead of eight).  The network is not
// stable by itself, so it orders by (key, value): the values are the primitives'
// indices 0..n-1 in their input order, which makes the result the stable order.
// Entries past n are padded with the largest pair.  Rebuilding the BVH of 1,100 instances
// took 187 us with the network and 204 with the radix sort, 2,048 202 and 242, 3,000 240
// and 252, 4,096 246 and 252; a network of 8,192 has 91 stages of twice the work.
constexpr uint32_t SORT_BITONIC_MAX = 4096;

__global__ void __launch_bounds__(SORT_THREADS, 1) k_sort_bitonic(unsigned long long* keys, uint32_t* vals,
                                                                uint32_t n) {
    extern __shared__ __align__(16) unsigned char sort_smem[];
    uint32_t N = 2;
    while (N < n) N <<= 1;
    unsigned long long* sk = reinterpret_cast<unsigned long long*>(sort_smem);
    uint32_t* sv = reinterpret_cast<uint32_t*>(sk + N);
    for (uint32_t i = threadIdx.x; i < N; i += SORT_THREADS) {
        sk[i] = i < n ? keys[i] : ~0ull;
        sv[i] = i < n ? vals[i] : ~0u;
    }
    __syncthreads();
    for (uint32_t k = 2; k <= N; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t i = threadIdx.x; i < N / 2; i += SORT_THREADS) {
                const uint32_t lo = ((i & ~(j - 1u)) << 1) | (i & (j - 1u)), hi = lo + j;
                const unsigned long long ka = sk[lo], kb = sk[hi];
                const uint32_t va = sv[lo], vb = sv[hi];
                const bool a_greater = ka > kb || (ka == kb && va > vb);
                if (a_greater == ((lo & k) == 0u)) {   // ascending blocks put the smaller first
                    sk[lo] = kb; sk[hi] = ka;
                    sv[lo] = vb; sv[hi] = va;
                }
            }
            __syncthreads();
        }
    }
    for (uint32_t i = threadIdx.x; i < n; i += SORT_THREADS) {
        keys[i] = sk[i];
        vals[i] = sv[i];
    }
}

// one thread per primitive: internal node i of its tree, i its place in the tree (the
// last place has none); the root has no parent
__global__ void k_karras(const unsigned long long* __restrict__ keys, BuildTrees B, int2* children, int* parent) {
    const uint32_t g = blockIdx.x * BLK + threadIdx.x;
    if (g >= B.total) return;
    const uint32_t t = tree_of(B, g), first = tree_begin(B, t);
    const int n = (int)(tree_end(B, t) - first), i = (int)(g - first);
    if (i == 0) parent[n > 1 ? first : B.total + first] = -1;
    if (i < n - 1) karras_node(i, keys + first, n, first, B.total, children, parent);
}

// Arrival at a tree node during a climb: true for the second thread to arrive, which
// then sees what the first one (and the warp it acted for) had written.  One
// acquire-release addition: a sequentially consistent fence on each side of a relaxed
// one made every step of a climb wait longer (the collapse cost's climb over 132,352
// triangles 51 us, 43 so).
template <bool G>
__device__ __forceinline__ bool arrive_second(int* flag) {
    if constexpr (G) {
        int old;
        asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(old) : "l"(flag) : "memory");
        return (old & 1) != 0;
    } else {
        __threadfence_block();
        const bool second = (atomicAdd(flag, 1) & 1) != 0;
        __threadfence_block();
        return second;
    }
}

// box and primitive count of internal node p from its two finished children; returns the count
template <bool G>
__device__ __forceinline__ uint32_t join_children(int p, int2 ch, float4* node_lo, float4* node_hi,
                                                  uint32_t* leaf_count) {
    const float4 al = ldx<G>(&node_lo[ch.x]), ah = ldx<G>(&node_hi[ch.x]);
    const float4 bl = ldx<G>(&node_lo[ch.y]), bh = ldx<G>(&node_hi[ch.y]);
    const uint32_t cnt = ldx<G>(&leaf_count[ch.x]) + ldx<G>(&leaf_count[ch.y]);
    node_lo[p] = make_float4(fminf(al.x, bl.x), fminf(al.y, bl.y), fminf(al.z, bl.z), 0.0f);
    node_hi[p] = make_float4(fmaxf(ah.x, bh.x), fmaxf(ah.y, bh.y), fmaxf(ah.z, bh.z), 0.0f);
    leaf_count[p] = cnt;
    return cnt;
}
__device__ __forceinline__ void init_leaf(int node, uint32_t prim, const float4* __restrict__ plo,
                                          const float4* __restrict__ phi, float4* node_lo, float4* node_hi,
                                          uint32_t* leaf_count) {
    node_lo[node] = plo[prim];
    node_hi[node] = phi[prim];
    leaf_count[node] = 1;
}

// Climbs from every leaf: the second thread to arrive at a node completes it.  Every
// climb of a build adds 2 to the flag of each internal node, so the flags are zeroed
// once.
__global__ void k_bottom_up(const uint32_t* __restrict__ sorted, const float4* __restrict__ plo,
                            const float4* __restrict__ phi, int n, const int2* __restrict__ children,
                            const int* __restrict__ parent, int* flags, float4* node_lo, float4* node_hi,
                            uint32_t* leaf_count) {
    const int j = blockIdx.x * BLK + threadIdx.x;
    if (j >= n) return;
    init_leaf(n + j, sorted[j], plo, phi, node_lo, node_hi, leaf_count);
    for (int p = parent[n + j]; p >= 0; p = parent[p]) {
        if (!arrive_second<true>(&flags[p])) return;
        join_children<true>(p, children[p], node_lo, node_hi, leaf_count);
    }
}

__device__ __forceinline__ float half_area(float4 lo, float4 hi) {
    float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
    return dx * dy + dy * dz + dz * dx;
}

// ---- treelet restructuring -----------------------------------------------------
// Bound by latency: a climb towards the root is a chain of treelets, each of which
// waits for the one below it (about 20 on the way up a 131,072-triangle tree).  So a
// warp works one treelet out with all its lanes and as few dependent loads as it can:
// the four levels below the root are fetched a level at a time, before it is known which
// of their nodes will be opened (30 lanes, a node each; seven rounds of loads when every
// opening waited for its own), the subsets of each size are costed one per lane (four
// lanes share a subset of six leaves), and the six rewritten nodes are stored by six
// lanes.  A treelet whose present form costs no more than the best one stays as it is
// without the rewriting, the stores and the wait for them: 21 %, 63 % and 82 % of the
// treelets of the three passes.  Subtrees below seven primitives only need their cost,
// which each lane works out for its own node.  A node's parent, children and count are
// loaded before the arrival at it, not after.
// Loading 50 small meshes (150 passes then) took 58.1 ms with one lane growing and
// rewriting every treelet and small subtrees costed one after another, 29.3 ms with lane
// k opening and storing leaf and node k; a 131,072-triangle terrain and a sphere 5.77 and
// 3.66 ms.  With 64 registers (four blocks per SM) all of a large mesh's warps run at
// once: terrain and sphere 2.43 and 2.18 ms.  Four levels at a time, kept forms and the
// early loads: 1.885 and 1.658 ms (three passes about 250 and 170 us each), 50 small
// meshes, now built together, 1.452 and 1.279 ms; the trees' SAH costs agree to 1e-5.
constexpr int TL_LEAVES = 7;
constexpr int TL_SUBSETS = 1 << TL_LEAVES;
constexpr int TL_WARPS = BLK / 32;
constexpr float SAH_CI = 1.2f;   // binary internal node
constexpr float SAH_CT = 1.0f;   // primitive

// the subsets of 2 to 6 treelet leaves, by size
struct SubsetTable { uint8_t v[120]; };
constexpr SubsetTable make_subsets() {
    SubsetTable t{};
    int n = 0;
    for (int size = 2; size <= 6; size++)
        for (int s = 1; s < TL_SUBSETS; s++) {
            int c = 0;
            for (int k = 0; k < TL_LEAVES; k++) c += (s >> k) & 1;
            if (c == size) t.v[n++] = (uint8_t)s;
        }
    return t;
}
__device__ const SubsetTable TL_SUBS = make_subsets();
constexpr int TL_AT2 = 0, TL_AT3 = 21, TL_AT4 = 56, TL_AT5 = 91, TL_AT6 = 112;   // 21, 35, 35, 21 and 7 subsets

// the subsets a lane works out (0: none): one or two of each size, a quarter of one of size 6
struct TreeletLane { uint32_t s2, s3, s3b, s4, s4b, s5, s6; };
__device__ __forceinline__ TreeletLane treelet_lane() {
    const int lane = threadIdx.x & 31;
    const uint8_t* v = TL_SUBS.v;
    TreeletLane t;
    t.s2 = lane < 21 ? __ldg(v + TL_AT2 + lane) : 0u;
    t.s3 = __ldg(v + TL_AT3 + lane);
    t.s3b = lane < 3 ? __ldg(v + TL_AT3 + 32 + lane) : 0u;
    t.s4 = __ldg(v + TL_AT4 + lane);
    t.s4b = lane < 3 ? __ldg(v + TL_AT4 + 32 + lane) : 0u;
    t.s5 = lane < 21 ? __ldg(v + TL_AT5 + lane) : 0u;
    t.s6 = lane < 28 ? __ldg(v + TL_AT6 + (lane >> 2)) : 0u;
    return t;
}

struct TreeletSmem {
    float area[TL_SUBSETS];
    float cost[TL_SUBSETS];
    uint32_t count[TL_SUBSETS];
    uint8_t part[TL_SUBSETS];
    float4 lo[TL_LEAVES], hi[TL_LEAVES];   // leaf boxes (lo.w: cost, hi.w: primitive count)
    int leaf[TL_LEAVES];
};

// subtrees of at most leaf_max primitives become leaves of the wide BVH
__device__ __forceinline__ float node_cost(float area, uint32_t cnt, float split_cost, uint32_t leaf_max) {
    return cnt <= leaf_max ? SAH_CT * area * (float)cnt : SAH_CI * area + split_cost;
}

// The best of the PARTS unordered 2-partitions of subset sub (the part that holds its
// lowest leaf is enumerated, from the largest down: of equal costs the lowest part wins)
template <int PARTS>
__device__ __forceinline__ void treelet_subset(TreeletSmem& T, uint32_t sub, uint32_t leaf_max) {
    if (sub == 0u) return;
    const uint32_t low = sub & (0u - sub), rest = sub ^ low;
    uint32_t q = (rest - 1u) & rest, bp = low | q;
    float best = T.cost[bp] + T.cost[sub ^ bp];
#pragma unroll
    for (int i = 1; i < PARTS; i++) {
        q = (q - 1u) & rest;
        const uint32_t P = low | q;
        const float c = T.cost[P] + T.cost[sub ^ P];
        if (c <= best) { best = c; bp = P; }
    }
    T.cost[sub] = node_cost(T.area[sub], T.count[sub], best, leaf_max);
    T.part[sub] = (uint8_t)bp;
}

// minimum of (cost, part) over the lanes that differ in the lane bits up to `lanes`
__device__ __forceinline__ void treelet_min(float& best, uint32_t& bp, int lanes) {
    for (int o = lanes >> 1; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xFFFFFFFFu, best, o);
        const uint32_t op = __shfl_xor_sync(0xFFFFFFFFu, bp, o);
        if (ob < best || (ob == best && op < bp)) { best = ob; bp = op; }
    }
}

// Optimises the treelet rooted at `root` (children rc), a subtree of at least TL_LEAVES
// primitives (all 32 lanes of the warp call this).  Internal nodes have ids below nl.
template <bool G>
__device__ void treelet_optimise(int root, int2 rc, int nl, int2* children, int* parent, float4* node_lo,
                                 float4* node_hi, uint32_t* leaf_count, float* cost, TreeletSmem& T,
                                 const TreeletLane& mine, uint32_t leaf_max) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    // the four levels below the root, a round of loads for each: lanes 0 and 1 the root's
    // children, lanes 2 h + 2 and 2 h + 3 those of lane h
    int id = lane == 0 ? rc.x : rc.y, inner = root;   // lane k: a node / internal node k of the treelet
    float area = 0.0f;
    int2 ch = make_int2(0, 0);
    float4 lo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), hi = lo;
    auto fetch = [&](int c) {
        id = c;
        lo = ldx<G>(&node_lo[c]);
        hi = ldx<G>(&node_hi[c]);
        const float k = ldx<G>(&cost[c]);
        const uint32_t n = ldx<G>(&leaf_count[c]);
        if (c < nl) ch = ldx<G>(&children[c]);
        area = half_area(lo, hi);
        lo.w = k;
        hi.w = __uint_as_float(n);
    };
    bool have = lane < 2;
    if (have) fetch(id);
#pragma unroll
    for (int first = 2; first < 30; first = 2 * first + 2) {   // 2, 6, 14
        const int from = (lane >> 1) - 1;   // (lane - 2) / 2
        const int bx = __shfl_sync(FULL, ch.x, from), by = __shfl_sync(FULL, ch.y, from);
        const bool opens = __shfl_sync(FULL, have && id < nl, from);
        if (lane >= first && lane < 2 * first + 2 && opens) {
            have = true;
            fetch((lane & 1) ? by : bx);
        }
    }
    // grow: open the largest treelet leaf until there are seven; the children of a node of
    // the fourth level are fetched, into its lane and lane 30 or 31
    // (a subtree of >= 7 primitives always has an internal node to open; areas are >= 0)
    unsigned leaves = 3u;
    const float unchanged = __shfl_sync(FULL, lo.w, 0) + __shfl_sync(FULL, lo.w, 1);
    int spare = 30;
#pragma unroll
    for (int nleaf = 2; nleaf < TL_LEAVES; nleaf++) {
        const unsigned key = (((leaves >> lane) & 1u) && id < nl) ? __float_as_uint(area) + 1u : 0u;
        const unsigned mx = __reduce_max_sync(FULL, key);
        const int best = __ffs(__ballot_sync(FULL, key == mx)) - 1;
        const int opened = __shfl_sync(FULL, id, best);
        if (lane == nleaf - 1) inner = opened;
        if (best < 14) {
            leaves = (leaves & ~(1u << best)) | (3u << (2 * best + 2));
        } else {
            const int bx = __shfl_sync(FULL, ch.x, best), by = __shfl_sync(FULL, ch.y, best);
            if (lane == best || lane == spare) fetch(lane == best ? bx : by);
            leaves |= 1u << spare;
            spare++;
        }
    }
    if ((leaves >> lane) & 1u) {
        const int k = __popc(leaves & ((1u << lane) - 1u));
        T.lo[k] = lo;
        T.hi[k] = hi;
        T.leaf[k] = id;
    }
    __syncwarp();
    // areas and primitive counts of the subsets lane + 32 h: the union of the leaves
    // 0..4 in `lane`, then with leaf 5, leaf 6 and both
    {
        float4 a = make_float4(3.4e38f, 3.4e38f, 3.4e38f, 0.0f), z = make_float4(-3.4e38f, -3.4e38f, -3.4e38f, 0.0f);
        uint32_t cnt = 0;
        auto add = [&](int k) {
            const float4 l = T.lo[k], h = T.hi[k];
            a.x = fminf(a.x, l.x); a.y = fminf(a.y, l.y); a.z = fminf(a.z, l.z);
            z.x = fmaxf(z.x, h.x); z.y = fmaxf(z.y, h.y); z.z = fmaxf(z.z, h.z);
            cnt += __float_as_uint(h.w);
        };
#pragma unroll
        for (int k = 0; k < 5; k++)
            if ((lane >> k) & 1) add(k);
        const float4 a0 = a, z0 = z;
        const uint32_t c0 = cnt;
#pragma unroll
        for (int h = 0; h < 4; h++) {
            a = a0; z = z0; cnt = c0;
            if (h & 1) add(5);
            if (h & 2) add(6);
            const int sub = lane + 32 * h;
            T.area[sub] = half_area(a, z);
            T.count[sub] = cnt;
            if (__popc(sub) == 1) T.cost[sub] = T.lo[__ffs(sub) - 1].w;
        }
    }
    __syncwarp();
    treelet_subset<1>(T, mine.s2, leaf_max);
    __syncwarp();
    treelet_subset<3>(T, mine.s3, leaf_max);
    treelet_subset<3>(T, mine.s3b, leaf_max);
    __syncwarp();
    treelet_subset<7>(T, mine.s4, leaf_max);
    treelet_subset<7>(T, mine.s4b, leaf_max);
    __syncwarp();
    treelet_subset<15>(T, mine.s5, leaf_max);
    __syncwarp();
    {   // size 6: lanes 4 j .. 4 j + 3 share subset j's 31 partitions
        const uint32_t sub = mine.s6;
        float best = 3.4e38f;
        uint32_t bp = 0xFFFFFFFFu;
        if (sub) {
            const int gap = __ffs(sub ^ (TL_SUBSETS - 1)) - 1;   // the leaf it leaves out
            const uint32_t low = gap == 0 ? 2u : 1u, keep = gap == 0 ? 0u : (1u << gap) - 1u;
#pragma unroll
            for (uint32_t i = 0; i < 8; i++) {
                const uint32_t k = 4u * i + (uint32_t)(lane & 3), t = k << 1;
                if (k == 31u) break;   // (all of sub)
                const uint32_t P = low | (t & keep) | ((t & ~keep) << 1);
                const float c = T.cost[P] + T.cost[sub ^ P];
                if (c < best || (c == best && P < bp) || bp == 0xFFFFFFFFu) { best = c; bp = P; }
            }
        }
        treelet_min(best, bp, 4);
        if (sub && (lane & 3) == 0) {
            T.cost[sub] = node_cost(T.area[sub], T.count[sub], best, leaf_max);
            T.part[sub] = (uint8_t)bp;
        }
    }
    __syncwarp();
    {   // the full set: 63 partitions across the warp
        const uint32_t full = TL_SUBSETS - 1;
        uint32_t bp = 1u | ((uint32_t)lane << 1);
        float best = T.cost[bp] + T.cost[full ^ bp];
        if (lane < 31) {
            const uint32_t P = bp + 64u;
            const float c = T.cost[P] + T.cost[full ^ P];
            if (c < best) { best = c; bp = P; }
        }
        treelet_min(best, bp, 32);
        // (the costs of the nodes inside were stored when each was the root)
        const float area_root = T.area[full];
        const uint32_t n_root = T.count[full];
        if (!(best < unchanged)) {
            if (lane == 0) cost[root] = node_cost(area_root, n_root, unchanged, leaf_max);
            __syncwarp();
            return;
        }
        if (lane == 0) {
            T.cost[full] = node_cost(area_root, n_root, best, leaf_max);
            T.part[full] = (uint8_t)bp;
        }
    }
    __syncwarp();
    // rewrite the treelet's six internal nodes: every lane follows the partitions (the
    // nodes' subsets in order, a byte each), lane k keeps and stores node k
    unsigned long long queue = TL_SUBSETS - 1;
    uint32_t sub = 0u, part = 0u;
    int at0 = 0, at1 = 0, next = 1;
#pragma unroll
    for (int k = 0; k < TL_LEAVES - 1; k++) {
        const uint32_t u = (uint32_t)(queue >> (8 * k)) & 0xFFu, a = T.part[u], b = u ^ a;
        const int i0 = next;
        if (__popc(a) > 1) queue |= (unsigned long long)a << (8 * next++);
        const int i1 = next;
        if (__popc(b) > 1) queue |= (unsigned long long)b << (8 * next++);
        if (lane == k) { sub = u; part = a; at0 = i0; at1 = i1; }
    }
    int2 kids;
    kids.x = __shfl_sync(FULL, inner, at0);
    kids.y = __shfl_sync(FULL, inner, at1);
    if (__popc(part) == 1) kids.x = T.leaf[__ffs(part) - 1];
    if (__popc(sub ^ part) == 1) kids.y = T.leaf[__ffs(sub ^ part) - 1];
    if (lane < TL_LEAVES - 1) {
        children[inner] = kids;
        parent[kids.x] = inner;
        parent[kids.y] = inner;
        float4 a = make_float4(3.4e38f, 3.4e38f, 3.4e38f, 0.0f), z = make_float4(-3.4e38f, -3.4e38f, -3.4e38f, 0.0f);
#pragma unroll
        for (int k = 0; k < TL_LEAVES; k++) {
            if (!((sub >> k) & 1u)) continue;
            const float4 l = T.lo[k], h = T.hi[k];
            a.x = fminf(a.x, l.x); a.y = fminf(a.y, l.y); a.z = fminf(a.z, l.z);
            z.x = fmaxf(z.x, h.x); z.y = fmaxf(z.y, h.y); z.z = fmaxf(z.z, h.z);
        }
        node_lo[inner] = a;
        node_hi[inner] = z;
        leaf_count[inner] = T.count[sub];
        cost[inner] = T.cost[sub];
    }
    __syncwarp();
}

// One restructuring pass, leaf j of this thread (every lane of the warp calls
// it): each thread climbs towards the root; the second thread to reach a node costs
// it, or hands its treelet to the whole warp when it holds at least seven
// primitives.  FIRST: the climb also makes the boxes and counts (the boxes and counts
// of the leaves are in place).  Every pass adds 2 to the flag of each internal node.
template <bool G, bool FIRST>
__device__ void treelet_climb(int j, int n, int nl, int2* children, int* parent, int* flags, float4* node_lo,
                              float4* node_hi, uint32_t* leaf_count, float* cost, TreeletSmem& T, uint32_t leaf_max) {
    const TreeletLane mine = treelet_lane();
    bool active = j < n;
    int p = -1, up = -1;   // the node to arrive at, and its parent (no treelet below changes either)
    if (active) {
        const int cur = nl + j;
        cost[cur] = SAH_CT * half_area(node_lo[cur], node_hi[cur]);
        p = ldx<G>(&parent[cur]);
        active = p >= 0;
    }
    while (true) {
        bool ready = false, big = false;
        int2 ch = make_int2(0, 0);
        if (active) {
            // (nothing below p changes these, and what is above comes later)
            up = ldx<G>(&parent[p]);
            ch = ldx<G>(&children[p]);
            uint32_t total = FIRST ? 0u : ldx<G>(&leaf_count[p]);
            active = ready = arrive_second<G>(&flags[p]);
            if (ready) {
                if (FIRST) total = join_children<G>(p, ch, node_lo, node_hi, leaf_count);
                big = total >= (uint32_t)TL_LEAVES;
                if (!big) {
                    const float c = ldx<G>(&cost[ch.x]) + ldx<G>(&cost[ch.y]);
                    cost[p] = node_cost(half_area(ldx<G>(&node_lo[p]), ldx<G>(&node_hi[p])), total, c, leaf_max);
                }
            }
        }
        __syncwarp();
        unsigned m = __ballot_sync(0xFFFFFFFFu, big);
        while (m) {
            const int l = __ffs(m) - 1;
            m &= m - 1;
            const int root = __shfl_sync(0xFFFFFFFFu, p, l);
            const int2 rc = make_int2(__shfl_sync(0xFFFFFFFFu, ch.x, l), __shfl_sync(0xFFFFFFFFu, ch.y, l));
            treelet_optimise<G>(root, rc, nl, children, parent, node_lo, node_hi, leaf_count, cost, T, mine, leaf_max);
        }
        if (ready) {
            p = up;
            active = p >= 0;
        }
        if (!__any_sync(0xFFFFFFFFu, active)) break;
    }
}

template <bool FIRST>
__global__ void __launch_bounds__(BLK, 4) k_treelet_pass(int n, const uint32_t* __restrict__ sorted,
                                                      const float4* __restrict__ plo, const float4* __restrict__ phi,
                                                      int2* children, int* parent, int* flags, float4* node_lo,
                                                      float4* node_hi, uint32_t* leaf_count, float* cost,
                                                      uint32_t leaf_max) {
    __shared__ TreeletSmem smem[TL_WARPS];
    const int j = blockIdx.x * BLK + threadIdx.x;
    if (FIRST && j < n) init_leaf(n + j, sorted[j], plo, phi, node_lo, node_hi, leaf_count);
    treelet_climb<true, FIRST>(j, n, n, children, parent, flags, node_lo, node_hi, leaf_count, cost,
                               smem[threadIdx.x >> 5], leaf_max);
}

// smallest power-of-two exponent (biased) with 2^(e-127) >= x; at least 1
__device__ __forceinline__ uint32_t ceil_exp_biased(float x) {
    uint32_t b = __float_as_uint(x);
    uint32_t e = (b >> 23) & 0xFFu;
    if (e == 0) return 1u;
    if (b & 0x7FFFFFu) e += 1;
    return e > 254u ? 254u : e;
}

// 8-bit child-box quantisation of a wide node: a power-of-two scale per axis
// (the smallest with 255 steps covering the parent box, rounded up) and child
// planes rounded outwards by at least QUANT_PAD of a step, which covers the rounding of
// the traversal's plane offsets (box_hits); the decoded boxes contain the exact ones.
// The grid starts 1/16 of a step (of the unpadded grid) below the box, rounded down,
// so that the lowest planes have their pad too: where the subtraction is exact the
// step is at most doubled by it, where it is not the origin moves by an ulp u of the
// box's corner, and the step, at most 2 (255 x 16 u + u) / 254.75, stays below 64 u.
constexpr float QUANT_PAD = 1.0f / 64.0f;
constexpr uint32_t QUANT_EXP_BIAS = 15;   // the stored exponents carry the traversal's 2^15
struct QuantFrame {
    float p[3], inv_scale[3];
    uint32_t eb[3];   // stored exponent bytes
};
__device__ __forceinline__ QuantFrame quant_frame(float4 plo, float4 phi) {
    QuantFrame F;
    const float lo[3] = {plo.x, plo.y, plo.z}, hi[3] = {phi.x, phi.y, phi.z};
    for (int a = 0; a < 3; a++) {
        const uint32_t e0 = ceil_exp_biased(__fdiv_ru(__fsub_ru(hi[a], lo[a]), 255.0f));
        F.p[a] = __fsub_rd(lo[a], __uint_as_float(e0 << 23) * 0.0625f);
        const uint32_t e1 = ceil_exp_biased(__fdiv_ru(__fsub_ru(hi[a], F.p[a]), 254.75f));
        const uint32_t e = min(max(e0, e1), 254u - QUANT_EXP_BIAS);
        F.eb[a] = e + QUANT_EXP_BIAS;
        F.inv_scale[a] = __uint_as_float((254u - e) << 23);   // 2^(127 - e)
    }
    return F;
}
__device__ __forceinline__ void quant_child(const QuantFrame& F, float4 a4, float4 z4, WideNode& node, int s) {
    const float clo[3] = {a4.x, a4.y, a4.z}, chi[3] = {z4.x, z4.y, z4.z};
    for (int a = 0; a < 3; a++) {
        const float ql = floorf(__fadd_rd(__fmul_rd(__fsub_rd(clo[a], F.p[a]), F.inv_scale[a]), -QUANT_PAD));
        const float qh = ceilf(__fadd_ru(__fmul_ru(__fsub_ru(chi[a], F.p[a]), F.inv_scale[a]), QUANT_PAD));
        node.qlo[a][s] = (uint8_t)fminf(fmaxf(ql, 0.0f), 255.0f);
        node.qhi[a][s] = (uint8_t)fminf(fmaxf(qh, 0.0f), 255.0f);
    }
}

// ---- SAH-optimal 8-wide collapse ------------------------------------------------
// Dynamic programming over the binary tree (Ylitie, Karras, Laine, HPG 2017): for
// every internal node x and every i in 1..8, D(x, i) is the least SAH cost of the
// subtree of x represented by at most i children of a wide node.  A child is x
// itself (a wide node of cost WIDE_CN A(x) plus the best distribution of x's
// subtree over 8 children, or a leaf of WIDE_CT A(x) per primitive when x holds at
// most leaf_pack primitives), or the children of a split of the i slots between
// x's two binary children.  wide_split[x] packs the argmins in 4-bit fields: field
// 0 the split of a wide node rooted at x (8 slots), field i - 1 (i = 2..8) the
// choice for D(x, i): 0 keeps x as one child, k > 0 gives k slots to the left child
// and i - k to the right one.
constexpr float WIDE_CN = 1.0f;   // one 8-wide node test
constexpr float WIDE_CT = 1.0f;   // one primitive test (0.3 and 0.6 gave the same trees on the test scenes)

template <bool G>
__device__ __forceinline__ void wide_costs(int c, int nl, const float4* node_lo, const float4* node_hi,
                                           const float* wide_cost, float d[8]) {
    if (c >= nl) {
        const float v = WIDE_CT * half_area(ldx<G>(&node_lo[c]), ldx<G>(&node_hi[c]));
#pragma unroll
        for (int i = 0; i < 8; i++) d[i] = v;
    } else {
        const float4* src = reinterpret_cast<const float4*>(wide_cost + 8 * (size_t)c);
        const float4 a = ldx<G>(src), b = ldx<G>(src + 1);
        d[0] = a.x; d[1] = a.y; d[2] = a.z; d[3] = a.w; d[4] = b.x; d[5] = b.y; d[6] = b.z; d[7] = b.w;
    }
}

// D(p, 1..8) and wide_split[p] of internal node p from its two children's entries
template <bool G>
__device__ __forceinline__ void wide_cost_node(int p, int nl, const int2* children, const float4* node_lo,
                                               const float4* node_hi, const uint32_t* leaf_count, float* wide_cost,
                                               uint32_t* wide_split, uint32_t leaf_max, uint32_t leaf_pack) {
    const int2 ch = ldx<G>(&children[p]);
    float a[8], b[8];
    wide_costs<G>(ch.x, nl, node_lo, node_hi, wide_cost, a);
    wide_costs<G>(ch.y, nl, node_lo, node_hi, wide_cost, b);
    float e[9];
    uint32_t ek[9];
#pragma unroll
    for (int i = 2; i <= 8; i++) {
        float best = a[0] + b[i - 2];
        uint32_t bk = 1;
#pragma unroll
        for (int k = 2; k < i; k++) {
            const float c = a[k - 1] + b[i - k - 1];
            if (c < best) { best = c; bk = (uint32_t)k; }
        }
        e[i] = best;
        ek[i] = bk;
    }
    const float area = half_area(ldx<G>(&node_lo[p]), ldx<G>(&node_hi[p]));
    const uint32_t cnt = ldx<G>(&leaf_count[p]);
    const float d1 = cnt <= leaf_pack ? WIDE_CT * area * (float)cnt : WIDE_CN * area + e[8];
    float d[8];
    uint32_t split = ek[8];
    d[0] = d1;
#pragma unroll
    for (int i = 2; i <= 8; i++) {
        const bool open = cnt > leaf_max && e[i] < d1;   // subtrees of at most leaf_max primitives stay leaves
        d[i - 1] = open ? e[i] : d1;
        split |= (open ? ek[i] : 0u) << (4 * (i - 1));
    }
    float4* dst = reinterpret_cast<float4*>(wide_cost + 8 * (size_t)p);
    dst[0] = make_float4(d[0], d[1], d[2], d[3]);
    dst[1] = make_float4(d[4], d[5], d[6], d[7]);
    wide_split[p] = split;
}

// bottom-up from leaf j (the second thread to arrive at a node completes it; FIRST: with
// its box and count)
template <bool G, bool FIRST>
__device__ void wide_cost_climb(int j, int nl, const int2* children, const int* parent, int* flags,
                                float4* node_lo, float4* node_hi, uint32_t* leaf_count,
                                float* wide_cost, uint32_t* wide_split, uint32_t leaf_max, uint32_t leaf_pack) {
    for (int p = parent[nl + j]; p >= 0; p = parent[p]) {
        if (!arrive_second<G>(&flags[p])) return;
        if (FIRST) join_children<G>(p, ldx<G>(&children[p]), node_lo, node_hi, leaf_count);
        wide_cost_node<G>(p, nl, children, node_lo, node_hi, leaf_count, wide_cost, wide_split, leaf_max, leaf_pack);
    }
}

template <bool FIRST>
__global__ void k_collapse_cost(int n, const uint32_t* __restrict__ sorted, const float4* __restrict__ plo,
                                const float4* __restrict__ phi, const int2* __restrict__ children,
                                const int* __restrict__ parent, int* flags, float4* node_lo, float4* node_hi,
                                uint32_t* leaf_count, float* wide_cost, uint32_t* wide_split, uint32_t leaf_max,
                                uint32_t leaf_pack) {
    const int j = blockIdx.x * BLK + threadIdx.x;
    if (j >= n) return;
    if (FIRST) init_leaf(n + j, sorted[j], plo, phi, node_lo, node_hi, leaf_count);
    wide_cost_climb<true, FIRST>(j, n, children, parent, flags, node_lo, node_hi, leaf_count, wide_cost, wide_split,
                                 leaf_max, leaf_pack);
}

// The children of the wide node rooted at internal node b chosen by wide_split (the
// least-SAH distribution of b's subtree over 8 slots), one per lane in the tree's
// order; returns their number.  All open items expand in one round of loads (lane k
// holds item k: a binary node and the slots it may fill; item: 8 entries of this
// warp's shared memory).
__device__ __forceinline__ int wide_children(int b, int nl, const int2* children, const uint32_t* wide_split,
                                             int2* item, int* child) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const int2 ch = children[b];
    const int k8 = (int)(wide_split[b] & 15u);
    int y = lane == 0 ? ch.x : ch.y, slots = lane == 0 ? k8 : 8 - k8, count = 2;
    for (int round = 0; round < 7; round++) {
        int k = 0;
        int2 cy = make_int2(0, 0);
        if (lane < count && y < nl && slots > 1) {
            k = (int)((wide_split[y] >> (4 * (slots - 1))) & 15u);
            cy = children[y];
            if (k >= slots) k = 0;
        }
        const unsigned open = __ballot_sync(FULL, k > 0);
        if (open == 0u) break;
        const int total = count + __popc(open);
        if (total > 8) return -1;   // (never with a consistent table)
        if (lane < count) {
            const int pos = lane + __popc(open & ((1u << lane) - 1u));
            item[pos] = k > 0 ? make_int2(cy.x, k) : make_int2(y, slots);
            if (k > 0) item[pos + 1] = make_int2(cy.y, slots - k);
        }
        count = total;
        __syncwarp();
        if (lane < count) { y = item[lane].x; slots = item[lane].y; }
        __syncwarp();
    }
    *child = lane < count ? y : -1;
    return count;
}

// ---- single-CTA agglomerative builder for small primitive sets -----------------
// The per-frame instance BVH (<= 1024 instances): one block of 1024 threads, every
// array in shared memory, one launch, no host synchronisation.  Locally-ordered
// clustering (PLOC, Meister & Bittner, TVCG 2018): clusters start as the
// primitives in Morton order; every round, each cluster finds the neighbour
// within PLOC_RADIUS positions whose merged box has the least surface area (ties:
// the lower position), mutual nearest neighbours merge into a new binary node, and
// the cluster list is compacted in order.  The globally closest pair is always
// mutual, so every round merges at least once.  Large boxes (a ground plane that
// spans the scene) are nobody's nearest neighbour and end up near the root.
// Internal node ids count down from n-2 as merges happen (the last merge is the
// root, node 0); leaves are n-1 + their Morton position, so the 8-wide collapse
// above applies unchanged.
constexpr int SMALL_THREADS = 1024;
constexpr int PLOC_RADIUS = 16;
static_assert(SMALL_BUILD_MAX == SMALL_THREADS, "one cluster per thread");

struct SmallSmem {
    unsigned long long keys[SMALL_BUILD_MAX];
    uint32_t vals[SMALL_BUILD_MAX];            // primitive at Morton position k
    int clusters[2][SMALL_BUILD_MAX];          // node ids of the live clusters, in order
    int2 children[SMALL_BUILD_MAX];
    float4 node_lo[2 * SMALL_BUILD_MAX], node_hi[2 * SMALL_BUILD_MAX];
    uint32_t leaf_count[2 * SMALL_BUILD_MAX];
    uint32_t tasks[2 * SMALL_BUILD_MAX];       // clustering: nearest neighbours; collapse: wide node l's binary node
    int parent[2 * SMALL_BUILD_MAX];           // treelet passes
    int flags[SMALL_BUILD_MAX];
    float cost[2 * SMALL_BUILD_MAX];
    uint32_t warp_sums[32];
    uint32_t counters[8];
    unsigned cb[6];
    union {
        TreeletSmem tl[SMALL_THREADS / 32];    // treelet passes
        struct {                               // then the least-SAH collapse table
            float wide_cost[8 * SMALL_BUILD_MAX];
            uint32_t wide_split[SMALL_BUILD_MAX];
        } dp;
    };
    WideNode stage[SMALL_THREADS / 32];        // per-warp staging of collapsed nodes
};
static_assert(sizeof(SmallSmem) <= 227 * 1024, "single-CTA builder exceeds shared memory");

__device__ __forceinline__ float4 f4min(float4 a, float4 b) {
    return make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z), 0.0f);
}
__device__ __forceinline__ float4 f4max(float4 a, float4 b) {
    return make_float4(fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z), 0.0f);
}

// inclusive block-wide sum of v (all SMALL_THREADS threads); *total = block sum
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* warp_sums, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += t;
    }
    if (lane == 31) warp_sums[warp] = v;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = warp_sums[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, w, o);
            if (lane >= o) w += t;
        }
        warp_sums[lane] = w;
    }
    __syncthreads();
    const uint32_t r = v + (warp ? warp_sums[warp - 1] : 0u);
    *total = warp_sums[31];
    __syncthreads();
    return r;
}

// float -> unsigned with the same order (for warp max reductions)
__device__ __forceinline__ unsigned order_f(float f) {
    const unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// Wide node `local` of the build, made of binary node b, by a whole warp (every lane
// passes the same).  counters: [2] wide nodes, [3] primitive slots, [4] capacity error
// bits.  Its internal children are nodes local' whose binary nodes go to tasks[local'];
// next_level (may be null) counts them.  cap: primitives of the build, cap_nodes: wide
// nodes it may write; internal binary nodes have ids below nl.  root_lo, root_hi (not
// null): returns (lane 0) the node's part of the SAH cost, its children's areas over the
// root's, one traversal step per internal child and one test per primitive.
// A level of the collapse is as long as one node's chain of loads: counts and leaf
// primitives are fetched with the boxes, the root's box before it is needed, the task
// before the level's size is known, and a child's task is found by its node's number
// (five rounds of loads and an atomic fewer in the chain: loading a 131,072-triangle
// terrain 1.678 -> 1.662 ms).  One launch whose warps wait for their node's parent instead
// of a launch per level was no faster (1.676 ms; 4,297 instances 264 -> 288 us).
// Lane k < nc holds candidate child k while the node is opened; the 64 (child,
// slot) pairs p = 8k + s of the slot assignment are spread two per lane; lane s
// < 8 then builds slot s.  Ties go to the lowest child / pair index, as in the
// sequential loops.  stage: this warp's 80-byte staging node in shared memory.
__device__ double collapse_task_warp(int b, uint32_t local, uint32_t* counters, uint32_t* next_level, uint32_t* tasks,
                                     uint32_t cap, uint32_t cap_nodes, int nl, const int2* children,
                                     const float4* node_lo, const float4* node_hi, const uint32_t* leaf_count,
                                     const uint32_t* sorted, WideNode* nodes, WideNode* stage, uint32_t node_base,
                                     uint32_t prim_base, uint32_t* prim_order, uint32_t leaf_max, uint32_t leaf_pack,
                                     const uint32_t* wide_split, const float4* root_lo, const float4* root_hi) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const uint32_t w = node_base + local;
    float4 rlo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), rhi = rlo;
    if (root_lo) { rlo = *root_lo; rhi = *root_hi; }
    int c = -1, nc;
    if (b >= nl) {
        nc = 1;
        if (lane == 0) c = b;
    } else if (wide_split) {
        nc = wide_children(b, nl, children, wide_split, reinterpret_cast<int2*>(stage), &c);
        if (nc < 0) {
            if (lane == 0) atomicOr(&counters[4], 8u);
            return 0.0;
        }
    } else {
        const int2 ch = children[b];
        nc = 2;
        c = lane == 0 ? ch.x : (lane == 1 ? ch.y : -1);
    }
    // greedy: open the largest internal candidate (more than leaf_max primitives) until 8 children
    while (!wide_split && nc < 8) {
        const bool elig = lane < nc && c < nl && leaf_count[c] > leaf_max;
        const unsigned key = elig ? __float_as_uint(half_area(node_lo[c], node_hi[c])) + 1u : 0u;   // areas >= 0
        const unsigned mx = __reduce_max_sync(FULL, key);
        if (mx == 0u) break;
        const int best = __ffs(__ballot_sync(FULL, key == mx)) - 1;
        const int cb = __shfl_sync(FULL, c, best);
        const int2 ch = children[cb];
        if (lane == best) c = ch.x;
        if (lane == nc) c = ch.y;
        nc++;
    }
    // parent box (min / max are exact, so the reduction order does not matter)
    float4 lo = make_float4(3.4e38f, 3.4e38f, 3.4e38f, 0.0f), hi = make_float4(-3.4e38f, -3.4e38f, -3.4e38f, 0.0f);
    float4 clo = lo, chi = hi;
    uint32_t c_count = 0, c_prim = 0;
    if (lane < nc) {
        clo = node_lo[c];
        chi = node_hi[c];
        c_count = leaf_count[c];
        if (c >= nl) c_prim = sorted[c - nl];
        lo = clo;
        hi = chi;
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        lo.x = fminf(lo.x, __shfl_xor_sync(FULL, lo.x, o)); lo.y = fminf(lo.y, __shfl_xor_sync(FULL, lo.y, o));
        lo.z = fminf(lo.z, __shfl_xor_sync(FULL, lo.z, o));
        hi.x = fmaxf(hi.x, __shfl_xor_sync(FULL, hi.x, o)); hi.y = fmaxf(hi.y, __shfl_xor_sync(FULL, hi.y, o));
        hi.z = fmaxf(hi.z, __shfl_xor_sync(FULL, hi.z, o));
    }
    const float4 plo = make_float4(__shfl_sync(FULL, lo.x, 0), __shfl_sync(FULL, lo.y, 0), __shfl_sync(FULL, lo.z, 0), 0.0f);
    const float4 phi = make_float4(__shfl_sync(FULL, hi.x, 0), __shfl_sync(FULL, hi.y, 0), __shfl_sync(FULL, hi.z, 0), 0.0f);
    const float pcx = 0.5f * (plo.x + phi.x), pcy = 0.5f * (plo.y + phi.y), pcz = 0.5f * (plo.z + phi.z);
    const float cx = 0.5f * (clo.x + chi.x) - pcx, cy = 0.5f * (clo.y + chi.y) - pcy, cz = 0.5f * (clo.z + chi.z) - pcz;
    // greedy slot assignment over the pairs p0 = lane, p1 = lane + 32 (child p >> 3, slot p & 7)
    const int s_ = lane & 7, k0 = lane >> 3, k1 = 4 + (lane >> 3);
    float sc[2];
    {
        const float x0 = __shfl_sync(FULL, cx, k0), y0 = __shfl_sync(FULL, cy, k0), z0 = __shfl_sync(FULL, cz, k0);
        const float x1 = __shfl_sync(FULL, cx, k1), y1 = __shfl_sync(FULL, cy, k1), z1 = __shfl_sync(FULL, cz, k1);
        sc[0] = ((s_ & 1) ? x0 : -x0) + ((s_ & 2) ? y0 : -y0) + ((s_ & 4) ? z0 : -z0);
        sc[1] = ((s_ & 1) ? x1 : -x1) + ((s_ & 2) ? y1 : -y1) + ((s_ & 4) ? z1 : -z1);
    }
    uint32_t used_c = 0, used_s = 0;
    int slot_k = -1;   // lane s < 8: the child in slot s
    for (int it = 0; it < nc; it++) {
        const bool v0 = k0 < nc && !((used_c >> k0) & 1u) && !((used_s >> s_) & 1u);
        const bool v1 = k1 < nc && !((used_c >> k1) & 1u) && !((used_s >> s_) & 1u);
        const bool take1 = v1 && (!v0 || sc[1] > sc[0]);
        const bool has = v0 || v1;
        const unsigned key = has ? order_f(take1 ? sc[1] : sc[0]) : 0u;
        const uint32_t p = take1 ? (uint32_t)lane + 32u : (uint32_t)lane;
        const unsigned mx = __reduce_max_sync(FULL, key);
        const uint32_t pm = __reduce_min_sync(FULL, (has && key == mx) ? p : 0xFFFFFFFFu);
        const int bk = (int)(pm >> 3), bs = (int)(pm & 7u);
        used_c |= 1u << bk;
        used_s |= 1u << bs;
        if (lane == bs) slot_k = bk;
    }
    const int from = slot_k < 0 ? 0 : slot_k;
    const int slot_c = __shfl_sync(FULL, c, from);
    const uint32_t slot_count = __shfl_sync(FULL, c_count, from), slot_prim = __shfl_sync(FULL, c_prim, from);
    // classify and allocate
    const bool mine = lane < 8 && slot_k >= 0;
    const bool is_int = mine && slot_c < nl && slot_count > leaf_pack;
    const uint32_t cnt = (mine && !is_int) ? slot_count : 0u;
    const unsigned int_mask = __ballot_sync(FULL, is_int);
    const uint32_t n_int = (uint32_t)__popc(int_mask);
    uint32_t off = cnt;   // inclusive scan of the leaf counts over the slots, then exclusive
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        const uint32_t t = __shfl_up_sync(FULL, off, o);
        if (lane >= o) off += t;
    }
    const uint32_t n_prims = __shfl_sync(FULL, off, 7);
    off -= cnt;
    uint32_t child_local = 0, prim_local = 0;
    if (lane == 0) {
        child_local = n_int ? atomicAdd(&counters[2], n_int) : 0u;
        prim_local = n_prims ? atomicAdd(&counters[3], n_prims) : 0u;
    }
    child_local = __shfl_sync(FULL, child_local, 0);
    prim_local = __shfl_sync(FULL, prim_local, 0);
    // capacity checks (never exceeded by a correct tree; a violation is recorded,
    // the node is not written and none of its children is made)
    if (child_local + n_int > cap_nodes || prim_local + n_prims > cap || local >= cap_nodes) {
        if (lane == 0) atomicOr(&counters[4], 1u);
        return 0.0;
    }
    if (next_level && lane == 0 && n_int) atomicAdd(next_level, n_int);
    const QuantFrame F = quant_frame(plo, phi);
    if (lane == 0) {
        stage->px = F.p[0]; stage->py = F.p[1]; stage->pz = F.p[2];
        stage->ex = (uint8_t)F.eb[0]; stage->ey = (uint8_t)F.eb[1]; stage->ez = (uint8_t)F.eb[2];
        stage->imask = (uint8_t)(int_mask & 0xFFu);
        stage->child_base = node_base + child_local;
        stage->prim_base = prim_base + prim_local;
    }
    if (lane < 8) {
        const int s = lane;
        if (!mine) {
            stage->meta[s] = 0;
            for (int a = 0; a < 3; a++) { stage->qlo[a][s] = 0; stage->qhi[a][s] = 0; }
        } else {
            quant_child(F, node_lo[slot_c], node_hi[slot_c], *stage, s);
            if (is_int) {
                const uint32_t rank = (uint32_t)__popc(int_mask & ((1u << s) - 1u));
                stage->meta[s] = (uint8_t)META_INTERNAL;
                tasks[child_local + rank] = (uint32_t)slot_c;
            } else if (slot_c >= nl) {
                stage->meta[s] = (uint8_t)((1u << 5) | off);
                prim_order[prim_local + off] = slot_prim;
            } else {
                stage->meta[s] = (uint8_t)((cnt << 5) | off);
                // the (<= leaf_pack) leaves of subtree slot_c, in order
                int stk[8];
                int sp = 0;
                stk[sp++] = slot_c;
                uint32_t k = 0;
                while (sp > 0) {
                    const int x = stk[--sp];
                    if (x >= nl) {
                        if (k < cnt) prim_order[prim_local + off + k] = sorted[x - nl];
                        k++;
                    } else if (sp < 7) {
                        const int2 ch = children[x];
                        stk[sp++] = ch.y;
                        stk[sp++] = ch.x;
                    } else {
                        atomicOr(&counters[4], 4u);
                    }
                }
            }
        }
    }
    __syncwarp();
    if (lane < 5) reinterpret_cast<uint4*>(nodes + w)[lane] = reinterpret_cast<const uint4*>(stage)[lane];
    __syncwarp();
    double sah = 0.0;
    if (root_lo) {
        const float area = half_area(rlo, rhi), inv_root = area > 0.0f ? 1.0f / area : 1.0f;
        if (mine) sah = (double)(half_area(node_lo[slot_c], node_hi[slot_c]) * inv_root) * (is_int ? 1.0 : (double)cnt);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) sah += __shfl_xor_sync(FULL, sah, o);
    }
    return sah;
}

__global__ void __launch_bounds__(SMALL_THREADS, 1)
k_build_small(const float4* __restrict__ plo, const float4* __restrict__ phi, int n, int passes, WideNode* nodes,
              uint32_t node_base, uint32_t prim_base, uint32_t* prim_order, SmallBuildOut* out, unsigned* err_word,
              float4* wide_box, uint32_t* wide_depth, uint32_t leaf_max, bool sah_collapse) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SmallSmem& S = *reinterpret_cast<SmallSmem*>(smem_raw);
    const int tid = threadIdx.x, nt = blockDim.x;
    // 1. centroid bounds
    if (tid < 6) S.cb[tid] = tid < 3 ? 0xFFFFFFFFu : 0u;
    __syncthreads();
    {
        unsigned mn[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, mx[3] = {0u, 0u, 0u};
        if (tid < n) {
            const float4 a = plo[tid], b = phi[tid];
            const float c[3] = {0.5f * (a.x + b.x), 0.5f * (a.y + b.y), 0.5f * (a.z + b.z)};
            for (int k = 0; k < 3; k++) { mn[k] = enc_f(c[k]); mx[k] = mn[k]; }
        }
        for (int k = 0; k < 3; k++) {
            const unsigned a = __reduce_min_sync(0xFFFFFFFFu, mn[k]), b = __reduce_max_sync(0xFFFFFFFFu, mx[k]);
            if ((tid & 31) == 0) { atomicMin(&S.cb[k], a); atomicMax(&S.cb[3 + k], b); }
        }
    }
    __syncthreads();
    // 2. Morton codes, padded to a power of two with keys that sort last
    int n2 = 1;
    while (n2 < n) n2 <<= 1;
    for (int i = tid; i < n2; i += nt) {
        S.keys[i] = i < n ? morton_of(plo[i], phi[i], S.cb) : ~0ull;
        S.vals[i] = (uint32_t)i;
    }
    __syncthreads();
    // 3. bitonic sort by (code, index): the order of a stable radix sort
    for (int k = 2; k <= n2; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = tid; i < n2; i += nt) {
                const int ixj = i ^ j;
                if (ixj > i) {
                    const unsigned long long ka = S.keys[i], kb = S.keys[ixj];
                    const uint32_t va = S.vals[i], vb = S.vals[ixj];
                    const bool gt = ka > kb || (ka == kb && va > vb);
                    if (gt == ((i & k) == 0)) {
                        S.keys[i] = kb; S.keys[ixj] = ka;
                        S.vals[i] = vb; S.vals[ixj] = va;
                    }
                }
            }
            __syncthreads();
        }
    }
    // 4. leaves and the initial cluster list
    const int nl = n - 1;
    if (tid < n) {
        const uint32_t p = S.vals[tid];
        S.node_lo[nl + tid] = plo[p];
        S.node_hi[nl + tid] = phi[p];
        S.leaf_count[nl + tid] = 1;
        S.clusters[0][tid] = nl + tid;
    }
    if (tid == 0) { S.counters[5] = (uint32_t)n; S.counters[6] = 0u; }
    __syncthreads();
    // 5. clustering rounds (thread i owns cluster position i) while more than 32
    // clusters remain; the last 32 finish inside warp 0 (every cluster sees every
    // other one, rounds synchronise through shuffles instead of block barriers)
    int cur = 0, rounds = 0;
    uint32_t m = (uint32_t)n;
    uint32_t next_id = n > 1 ? (uint32_t)(n - 2) : 0u;
    while (m > 32 && rounds < SMALL_BUILD_MAX) {
        // nearest neighbour of every position within PLOC_RADIUS: a group of tpc
        // threads per position splits the 2 * PLOC_RADIUS candidates, then takes
        // the minimum of (area, position), so ties keep the lower position
        {
            int tpc = 2 * PLOC_RADIUS;
            while (tpc > 1 && (uint32_t)tpc * m > (uint32_t)SMALL_THREADS) tpc >>= 1;
            const int g = tid / tpc, sub = tid % tpc;
            float best = 3.4e38f;
            uint32_t nn = 0xFFFFFFFFu;
            if (g < (int)m) {
                const int cg = S.clusters[cur][g];
                const float4 glo = S.node_lo[cg], ghi = S.node_hi[cg];
                for (int u = sub; u < 2 * PLOC_RADIUS; u += tpc) {
                    const int j = g + (u < PLOC_RADIUS ? u - PLOC_RADIUS : u - PLOC_RADIUS + 1);
                    if (j < 0 || j >= (int)m) continue;
                    const int cj = S.clusters[cur][j];
                    const float a = half_area(f4min(glo, S.node_lo[cj]), f4max(ghi, S.node_hi[cj]));
                    if (a < best) { best = a; nn = (uint32_t)j; }   // increasing j within the thread
                }
            }
            for (int o = 1; o < tpc; o <<= 1) {
                const float ob = __shfl_xor_sync(0xFFFFFFFFu, best, o);
                const uint32_t on = __shfl_xor_sync(0xFFFFFFFFu, nn, o);
                if (ob < best || (ob == best && on < nn)) { best = ob; nn = on; }
            }
            if (sub == 0 && g < (int)m) S.tasks[g] = nn;   // scratch: nearest neighbour per position
        }
        __syncthreads();
        const int i = tid;
        int nn = -1;
        float4 mylo = make_float4(0.f, 0.f, 0.f, 0.f), myhi = mylo;
        if (i < (int)m) {
            const int ci = S.clusters[cur][i];
            mylo = S.node_lo[ci];
            myhi = S.node_hi[ci];
            nn = (int)S.tasks[i];
        }
        bool merge = false, keep = false;
        if (i < (int)m) {
            const bool mutual = nn >= 0 && (int)S.tasks[nn] == i;
            merge = mutual && i < nn;
            keep = !mutual || i < nn;
        }
        // one scan of both counts: kept clusters in the low half, merges in the high half
        uint32_t totals;
        const uint32_t v = (keep ? 1u : 0u) | (merge ? 0x10000u : 0u);
        const uint32_t incl = block_scan(v, S.warp_sums, &totals);
        const uint32_t kpos = (incl & 0xFFFFu) - (keep ? 1u : 0u), mrank = (incl >> 16) - (merge ? 1u : 0u);
        const uint32_t total_keep = totals & 0xFFFFu, total_merge = totals >> 16;
        if (keep) {
            int id = S.clusters[cur][i];
            if (merge) {
                const int cj = S.clusters[cur][nn];
                id = (int)(next_id - mrank);
                S.children[id] = make_int2(S.clusters[cur][i], cj);
                S.node_lo[id] = f4min(mylo, S.node_lo[cj]);
                S.node_hi[id] = f4max(myhi, S.node_hi[cj]);
                S.leaf_count[id] = S.leaf_count[S.clusters[cur][i]] + S.leaf_count[cj];
            }
            S.clusters[cur ^ 1][kpos] = id;
        }
        if (total_merge == 0 && tid == 0) S.counters[6] |= 16u;   // no progress (cannot happen)
        next_id -= total_merge;
        m = total_keep;
        cur ^= 1;
        rounds++;
        __syncthreads();
        if (total_merge == 0) break;
    }
    if (tid < 32 && m > 1 && m <= 32) {
        const int lane = tid;
        const bool live0 = lane < (int)m;
        int id = live0 ? S.clusters[cur][lane] : -1;
        float4 lo = live0 ? S.node_lo[id] : make_float4(0.f, 0.f, 0.f, 0.f);
        float4 hi = live0 ? S.node_hi[id] : lo;
        uint32_t cnt = live0 ? S.leaf_count[id] : 0u;
        for (int r = 0; m > 1 && r < 64; r++) {
            const bool live = lane < (int)m;
            float best = 3.4e38f;
            int nn = -1;
            // every live cluster's box is stored at its node id (merges write it before
            // the __syncwarp that ends a round)
            for (int j = 0; j < (int)m; j++) {
                const int idj = __shfl_sync(0xFFFFFFFFu, id, j);
                if (j == lane || !live) continue;
                const float a = half_area(f4min(lo, S.node_lo[idj]), f4max(hi, S.node_hi[idj]));
                if (a < best) { best = a; nn = j; }
            }
            const int nn_of_nn = __shfl_sync(0xFFFFFFFFu, nn, nn < 0 ? lane : nn);
            const bool mutual = live && nn >= 0 && nn_of_nn == lane;
            const bool merge = mutual && lane < nn;
            const bool keep = live && (!mutual || lane < nn);
            const unsigned mm = __ballot_sync(0xFFFFFFFFu, merge), km = __ballot_sync(0xFFFFFFFFu, keep);
            const unsigned below = (1u << lane) - 1u;
            // partner data (for the merging lane)
            const int pid = __shfl_sync(0xFFFFFFFFu, id, nn < 0 ? lane : nn);
            const float4 pl = make_float4(__shfl_sync(0xFFFFFFFFu, lo.x, nn < 0 ? lane : nn),
                                          __shfl_sync(0xFFFFFFFFu, lo.y, nn < 0 ? lane : nn),
                                          __shfl_sync(0xFFFFFFFFu, lo.z, nn < 0 ? lane : nn), 0.0f);
            const float4 ph = make_float4(__shfl_sync(0xFFFFFFFFu, hi.x, nn < 0 ? lane : nn),
                                          __shfl_sync(0xFFFFFFFFu, hi.y, nn < 0 ? lane : nn),
                                          __shfl_sync(0xFFFFFFFFu, hi.z, nn < 0 ? lane : nn), 0.0f);
            const uint32_t pc = __shfl_sync(0xFFFFFFFFu, cnt, nn < 0 ? lane : nn);
            if (merge) {
                const int nid = (int)(next_id - (uint32_t)__popc(mm & below));
                S.children[nid] = make_int2(id, pid);
                lo = f4min(lo, pl);
                hi = f4max(hi, ph);
                cnt += pc;
                S.node_lo[nid] = lo;
                S.node_hi[nid] = hi;
                S.leaf_count[nid] = cnt;
                id = nid;
            }
            if (mm == 0u) { if (lane == 0) S.counters[6] |= 16u; break; }
            next_id -= (uint32_t)__popc(mm);
            // compact: lane k takes the k-th kept cluster
            const int k = lane < __popc(km) ? (int)__fns(km, 0, lane + 1) : lane;
            id = __shfl_sync(0xFFFFFFFFu, id, k);
            lo = make_float4(__shfl_sync(0xFFFFFFFFu, lo.x, k), __shfl_sync(0xFFFFFFFFu, lo.y, k),
                             __shfl_sync(0xFFFFFFFFu, lo.z, k), 0.0f);
            hi = make_float4(__shfl_sync(0xFFFFFFFFu, hi.x, k), __shfl_sync(0xFFFFFFFFu, hi.y, k),
                             __shfl_sync(0xFFFFFFFFu, hi.z, k), 0.0f);
            cnt = __shfl_sync(0xFFFFFFFFu, cnt, k);
            m = (uint32_t)__popc(km);
            __syncwarp();
        }
        if (lane == 0) S.clusters[cur][0] = id;
        if (lane == 0 && m != 1u) S.counters[6] |= 16u;
        __syncwarp();
    }
    __syncthreads();
    if (tid == 0 && n > 1 && (next_id != 0xFFFFFFFFu || S.clusters[cur][0] != 0)) S.counters[6] |= 16u;
    __syncthreads();
    // 5b. optional treelet restructuring of the clustered tree (leaves dealt
    // round-robin over the 32 warps so that treelets that become ready together
    // run in different warps)
    if (passes > 0 && n >= TL_LEAVES + 1 && S.counters[6] == 0u) {
        if (tid == 0) S.parent[0] = -1;
        if (tid < n - 1) {
            const int2 ch = S.children[tid];
            S.parent[ch.x] = tid;
            S.parent[ch.y] = tid;
        }
        for (int pass = 0; pass < passes; pass++) {
            if (tid < n) S.flags[tid] = 0;
            __syncthreads();
            treelet_climb<false, false>((tid & 31) * 32 + (tid >> 5), n, nl, S.children, S.parent, S.flags, S.node_lo,
                                        S.node_hi, S.leaf_count, S.cost, S.tl[tid >> 5], leaf_max);
            __syncthreads();
        }
    }
    // 5c. least-SAH choice of every wide node's children (bottom-up, in shared memory)
    const bool dp = sah_collapse && n > 1 && S.counters[6] == 0u;
    if (dp) {
        if (tid == 0) S.parent[0] = -1;
        if (tid < n - 1) {
            const int2 ch = S.children[tid];
            S.parent[ch.x] = tid;
            S.parent[ch.y] = tid;
        }
        if (tid < n) S.flags[tid] = 0;
        __syncthreads();
        if (tid < n)
            wide_cost_climb<false, false>(tid, nl, S.children, S.parent, S.flags, S.node_lo, S.node_hi, S.leaf_count,
                                          S.dp.wide_cost, S.dp.wide_split, leaf_max, leaf_max);
        __syncthreads();
    }
    // 6. collapse, level by level
    const float4 rlo = S.node_lo[0], rhi = S.node_hi[0];
    float rha = half_area(rlo, rhi);
    if (!(rha > 0.0f)) rha = 1.0f;
    if (tid == 0) {
        S.tasks[0] = 0u;
        S.counters[2] = 1u; S.counters[3] = 0u; S.counters[4] = 0u;
    }
    __syncthreads();
    // (a level's nodes are the ones that the level above has allocated: a run of numbers)
    uint32_t begin = 0, end = 1;
    int level = 0;
    for (; level < 4096; level++) {
        if (begin == end || S.counters[4] != 0u) break;   // done, or a capacity error
        // one warp per wide node (no SAH statistic: the per-frame build skips it)
        for (uint32_t local = begin + (uint32_t)(tid >> 5); local < end; local += (uint32_t)(nt >> 5)) {
            const int b = (int)S.tasks[local];
            // refit data: exact box and depth of every wide node
            if ((tid & 31) == 0) {
                wide_box[2 * local] = S.node_lo[b];
                wide_box[2 * local + 1] = S.node_hi[b];
                wide_depth[local] = (uint32_t)level;
            }
            collapse_task_warp(b, local, S.counters, nullptr, S.tasks, (uint32_t)n, (uint32_t)n + 1u, nl, S.children,
                               S.node_lo, S.node_hi, S.leaf_count, S.vals, nodes, &S.stage[tid >> 5], node_base,
                               prim_base, prim_order, leaf_max, leaf_max, dp ? S.dp.wide_split : nullptr, nullptr,
                               nullptr);
        }
        __syncthreads();
        begin = end;
        end = min(S.counters[2], (uint32_t)n + 1u);
        __syncthreads();
    }
    if (tid == 0) {
        uint32_t e = S.counters[4] | S.counters[6];
        if (S.counters[3] != (uint32_t)n) e |= 4u;
        if (level >= 4096) e |= 8u;
        out->num_nodes = S.counters[2];
        out->prims = S.counters[3];
        out->error = e;
        out->max_depth = level > 0 ? (uint32_t)(level - 1) : 0u;
        out->sah = 0.0;
        out->lo[0] = rlo.x; out->lo[1] = rlo.y; out->lo[2] = rlo.z; out->lo[3] = 0.0f;
        out->hi[0] = rhi.x; out->hi[1] = rhi.y; out->hi[2] = rhi.z; out->hi[3] = 0.0f;
        if (e && err_word) atomicOr(err_word, 8u);
    }
}

// ---- collapse without host round trips -----------------------------------------
// level_tasks[l] counts the wide nodes of level l, whose numbers follow those of the
// level above; tasks[number] is the binary node one is made of.  counters: [2] wide
// nodes, [3] primitive slots, [4] capacity error bits.  A few launches of k_collapse_level take the
// usual depths with every SM; k_collapse_finish takes whatever is left in one
// block, so no level count has to come back to the host.
constexpr int COLLAPSE_MAX_LEVELS = 128;
constexpr int COLLAPSE_FAST_LEVELS = 12;
constexpr int LEVEL_WARPS = 8;

// what the collapse reads and writes
struct CollapseArgs {
    BuildTrees B;
    uint32_t *tasks, *level_tasks, *counters;
    const int2* children;
    const float4 *node_lo, *node_hi;
    const uint32_t *leaf_count, *sorted, *wide_split;
    WideNode* nodes;
    uint32_t node_base, prim_base;
    uint32_t* prim_order;
    uint32_t leaf_max, leaf_pack;
    uint32_t* wide_depth;   // may be null
    double* sah;            // sum over the trees of primitives x SAH cost below the root; may be null
};

// the root of every tree: wide nodes node_base + t
__global__ void k_collapse_init(CollapseArgs A) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t <= (uint32_t)COLLAPSE_MAX_LEVELS) A.level_tasks[t] = t == 0u ? A.B.count : 0u;
    if (t < A.B.count) {
        const uint32_t first = tree_begin(A.B, t);
        const bool single = tree_end(A.B, t) - first == 1u;
        A.tasks[t] = single ? A.B.total + first : first;
    }
    if (t == 0u) {
        A.counters[2] = A.B.count;
        A.counters[3] = 0u;
        A.counters[4] = 0u;
        if (A.sah) *A.sah = 0.0;
    }
}

// Nodes begin + t0, begin + t0 + step, ... of the `count` of a level by this warp; returns
// their part of the SAH sum.  first_task: tasks[begin + t0], when that is in the array.
__device__ __forceinline__ double collapse_level(const CollapseArgs& A, int level, uint32_t begin, uint32_t count,
                                                 uint32_t t0, uint32_t step, uint32_t first_task, WideNode* stage) {
    const int lane = threadIdx.x & 31;
    const uint32_t n = A.B.total, cap_nodes = n + A.B.count;
    double sum = 0.0;
    for (uint32_t t = t0; t < count; t += step) {
        const uint32_t local = begin + t;
        if (local >= cap_nodes) break;   // (the task array holds cap_nodes entries)
        const uint32_t b = t == t0 ? first_task : A.tasks[local];
        if (A.wide_depth && lane == 0) A.wide_depth[local] = (uint32_t)level;   // (for a later refit)
        uint32_t prims = 0, root = 0;
        if (A.sah) {
            const uint32_t tree = tree_of(A.B, b >= n ? b - n : b);
            const uint32_t first = tree_begin(A.B, tree);
            prims = tree_end(A.B, tree) - first;
            root = prims == 1u ? n + first : first;
        }
        const double s = collapse_task_warp((int)b, local, A.counters, &A.level_tasks[level + 1], A.tasks, n, cap_nodes,
                                            (int)n, A.children, A.node_lo, A.node_hi, A.leaf_count, A.sorted, A.nodes,
                                            stage, A.node_base, A.prim_base, A.prim_order, A.leaf_max, A.leaf_pack,
                                            A.wide_split, A.sah ? A.node_lo + root : nullptr,
                                            A.sah ? A.node_hi + root : nullptr);
        sum += s * (double)prims;
    }
    return sum;
}

// adds the warps' sums (lane 0) to *out, one atomic per block; all threads call this
__device__ __forceinline__ void block_add(double sum, double* warp_sums, double* out) {
    const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if ((threadIdx.x & 31) == 0) warp_sums[w] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int k = 0; k < nw; k++) s += warp_sums[k];
        if (s != 0.0) atomicAdd(out, s);
    }
}

__global__ void __launch_bounds__(32 * LEVEL_WARPS) k_collapse_level(CollapseArgs A, int level) {
    __shared__ WideNode stage[LEVEL_WARPS];
    __shared__ double warp_sums[LEVEL_WARPS];
    const uint32_t w = threadIdx.x >> 5, t0 = blockIdx.x * LEVEL_WARPS + w;
    uint32_t begin = 0;
#pragma unroll
    for (int l = 0; l < COLLAPSE_FAST_LEVELS; l++) begin += l < level ? A.level_tasks[l] : 0u;
    uint32_t count = A.level_tasks[level];   // (final)
    const uint32_t bad = A.counters[4];
    if (blockIdx.x * LEVEL_WARPS >= count) return;
    if (bad != 0u) count = 0;                // (a capacity error: nothing more is written)
    const uint32_t task = begin + t0 < A.B.total + A.B.count ? A.tasks[begin + t0] : 0u;
    const double sum = collapse_level(A, level, begin, count, t0, gridDim.x * LEVEL_WARPS, task, &stage[w]);
    if (A.sah) block_add(sum, warp_sums, A.sah);
}

__global__ void __launch_bounds__(1024) k_collapse_finish(CollapseArgs A, int first_level, unsigned* err_word,
                                                          SmallBuildOut* out) {
    __shared__ WideNode stage[32];
    __shared__ double warp_sums[32];
    __shared__ uint32_t size;
    const uint32_t w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t begin = 0;
    for (int l = 0; l < first_level; l++) begin += A.level_tasks[l];
    int level = first_level;
    double sum = 0.0;
    for (; level < COLLAPSE_MAX_LEVELS; level++) {
        if (threadIdx.x == 0) size = A.counters[4] != 0u ? 0u : A.level_tasks[level];
        __syncthreads();
        const uint32_t count = size;
        if (count == 0u) break;
        const uint32_t task = begin + w < A.B.total + A.B.count ? A.tasks[begin + w] : 0u;
        sum += collapse_level(A, level, begin, count, w, nw, task, &stage[w]);
        begin += count;
        __syncthreads();   // this level's child tasks and their count are complete
    }
    if (A.sah) block_add(sum, warp_sums, A.sah);
    if (threadIdx.x == 0) {
        const bool unfinished = level >= COLLAPSE_MAX_LEVELS && A.level_tasks[COLLAPSE_MAX_LEVELS] != 0u;
        const bool bad = A.counters[4] != 0u || unfinished || A.counters[3] != A.B.total;
        if (bad && err_word) atomicOr(err_word, 8u);
        if (out) {   // what a refit and the host read: node count, deepest level, SAH sum
            uint32_t deepest = 0;
            for (int l = 0; l < COLLAPSE_MAX_LEVELS; l++)
                if (A.level_tasks[l] != 0u) deepest = (uint32_t)l;
            out->num_nodes = A.counters[2];
            out->prims = A.counters[3];
            out->error = bad ? 8u : 0u;
            out->max_depth = deepest;
            out->sah = A.sah ? atomicAdd(A.sah, 0.0) : 0.0;
        }
    }
}

// Refit of a per-frame wide BVH (made by k_build_small or by the device-driven
// multi-launch build) for moved primitives: the topology (child and primitive
// slots) stays, every node's exact box and quantised child planes are
// recomputed, deepest level first (one block, a barrier per level; the tree of
// n primitives has at most n + 1 nodes, each visited once per refit).
__global__ void __launch_bounds__(SMALL_THREADS, 1)
k_refit_small(WideNode* nodes, uint32_t node_base, uint32_t prim_base, const SmallBuildOut* info,
              float4* wide_box, const uint32_t* wide_depth, const uint32_t* prim_order,
              const float4* __restrict__ plo, const float4* __restrict__ phi, int n, unsigned* err_word) {
    const uint32_t nn = info->num_nodes;
    if (info->error || nn == 0 || nn > (uint32_t)n + 1u) return;
    const int max_depth = (int)min(info->max_depth, 4095u);
    for (int level = max_depth; level >= 0; level--) {
        for (uint32_t k = threadIdx.x; k < nn; k += blockDim.x) {
            if (wide_depth[k] != (uint32_t)level) continue;
            WideNode node;
            const uint4* src = reinterpret_cast<const uint4*>(nodes + node_base + k);
            uint4* dst4 = reinterpret_cast<uint4*>(&node);
            for (int q = 0; q < 5; q++) dst4[q] = src[q];
            float4 clo[8], chi[8];
            float4 lo = make_float4(3.4e38f, 3.4e38f, 3.4e38f, 0.0f), hi = make_float4(-3.4e38f, -3.4e38f, -3.4e38f, 0.0f);
            bool bad = false;
            for (int s = 0; s < 8; s++) {
                const uint32_t meta = node.meta[s];
                clo[s] = make_float4(3.4e38f, 3.4e38f, 3.4e38f, 0.0f);
                chi[s] = make_float4(-3.4e38f, -3.4e38f, -3.4e38f, 0.0f);
                if (meta == 0u) continue;
                if (meta == META_INTERNAL) {
                    const uint32_t child = node.child_base + (uint32_t)__popc(node.imask & ((1u << s) - 1u)) - node_base;
                    if (child >= nn) { bad = true; continue; }
                    clo[s] = wide_box[2 * child];
                    chi[s] = wide_box[2 * child + 1];
                } else {
                    const uint32_t cnt = meta >> 5, off = meta & 31u;
                    for (uint32_t j = 0; j < cnt; j++) {
                        const uint32_t slot = node.prim_base + off + j - prim_base;
                        if (slot >= (uint32_t)n) { bad = true; continue; }
                        const uint32_t li = prim_order[slot];
                        if (li >= (uint32_t)n) { bad = true; continue; }
                        clo[s] = f4min(clo[s], plo[li]);
                        chi[s] = f4max(chi[s], phi[li]);
                    }
                }
                lo = f4min(lo, clo[s]);
                hi = f4max(hi, chi[s]);
            }
            if (bad) { atomicOr(err_word, 8u); continue; }
            const QuantFrame F = quant_frame(lo, hi);
            node.px = F.p[0]; node.py = F.p[1]; node.pz = F.p[2];
            node.ex = (uint8_t)F.eb[0]; node.ey = (uint8_t)F.eb[1]; node.ez = (uint8_t)F.eb[2];
            for (int s = 0; s < 8; s++) {
                if (node.meta[s] == 0u) continue;
                quant_child(F, clo[s], chi[s], node, s);
            }
            uint4* out4 = reinterpret_cast<uint4*>(nodes + node_base + k);
            for (int q = 0; q < 5; q++) out4[q] = dst4[q];
            wide_box[2 * k] = lo;
            wide_box[2 * k + 1] = hi;
        }
        __syncthreads();
    }
}

// the 13 axes of a mesh's extents (MeshExtents): x y z, x+y x-y, x+z x-z, y+z y-z, then
// x+y+z x+y-z x-y+z x-y-z
__device__ __forceinline__ void extent_axes(const float* q, float* d) {
    d[0] = q[0]; d[1] = q[1]; d[2] = q[2];
    d[3] = q[0] + q[1]; d[4] = q[0] - q[1];
    d[5] = q[0] + q[2]; d[6] = q[0] - q[2];
    d[7] = q[1] + q[2]; d[8] = q[1] - q[2];
    d[9] = d[3] + q[2]; d[10] = d[3] - q[2]; d[11] = d[4] + q[2]; d[12] = d[4] - q[2];
}

// primitive i of the concatenated meshes (BuildTrees over the meshes that have
// triangles, tree_mesh[t] their indices): padded box of its triangle, and its part of
// the mesh's extents (zero at the start)
__global__ void __launch_bounds__(BLK) k_triangle_boxes(const float* __restrict__ pos, const uint32_t* __restrict__ idx,
                                                        BuildTrees B, const uint32_t* __restrict__ tree_mesh,
                                                        const MeshInfo* __restrict__ meshes, MeshExtents* extents,
                                                        float4* lo, float4* hi) {
    __shared__ unsigned red[BLK / 32][26];
    const uint32_t i = blockIdx.x * BLK + threadIdx.x;
    const bool valid = i < B.total;
    const uint32_t tree = tree_of(B, valid ? i : B.total - 1u), first = tree_begin(B, tree), t = i - first;
    const uint32_t mesh = __ldg(tree_mesh + tree);
    const MeshInfo& M = meshes[mesh];
    float l[3] = {3.4e38f, 3.4e38f, 3.4e38f}, h[3] = {-3.4e38f, -3.4e38f, -3.4e38f};
    unsigned ext26[26];   // order-preserving codes: largest along each axis, complements of the smallest
    for (int k = 0; k < 26; k++) ext26[k] = 0u;
    if (valid) {
        const float* c = pos + 3ull * (M.vertex_offset + idx[M.index_offset]);   // the mesh's reference point
        for (int k = 0; k < 3; k++) {
            const float* p = pos + 3ull * (M.vertex_offset + idx[M.index_offset + 3ull * t + k]);
            for (int a = 0; a < 3; a++) { l[a] = fminf(l[a], p[a]); h[a] = fmaxf(h[a], p[a]); }
            const float q[3] = {p[0] - c[0], p[1] - c[1], p[2] - c[2]};
            float d[13];
            extent_axes(q, d);
#pragma unroll
            for (int a = 0; a < 13; a++) {
                const unsigned e = enc_f(d[a]);
                ext26[a] = max(ext26[a], e);
                ext26[13 + a] = max(ext26[13 + a], ~e);
            }
        }
        if (t == 0u)
            for (int a = 0; a < 3; a++) extents[mesh].ref[a] = c[a];
    }
    {   // one atomic per axis and block (or warp, where the block holds several meshes)
        const uint32_t b0 = blockIdx.x * BLK, w0 = i & ~31u;
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const bool block_one = min(b0 + BLK, B.total) <= tree_end(B, tree_of(B, b0));
        const bool warp_one = __all_sync(0xFFFFFFFFu, !valid || w0 >= first);
        unsigned mine = 0u;
#pragma unroll
        for (int k = 0; k < 26; k++) {
            const unsigned m = __reduce_max_sync(0xFFFFFFFFu, ext26[k]);
            if (lane == k) mine = m;
        }
        unsigned* dst = extents[mesh].code;
        if (block_one) {
            if (lane < 26) red[warp][lane] = mine;
            __syncthreads();
            if (threadIdx.x < 26) {
                unsigned m = 0u;
                for (int w = 0; w < BLK / 32; w++) m = max(m, red[w][threadIdx.x]);
                atomicMax(&dst[threadIdx.x], m);
            }
        } else if (warp_one) {
            if (lane < 26 && w0 < B.total) atomicMax(&dst[lane], mine);
        } else if (valid) {
#pragma unroll
            for (int k = 0; k < 26; k++) atomicMax(&dst[k], ext26[k]);
        }
    }
    if (!valid) return;
    float ext = fmaxf(fmaxf(h[0] - l[0], h[1] - l[1]), h[2] - l[2]);
    for (int a = 0; a < 3; a++) {
        float pad = 1e-5f * (ext + fabsf(l[a]) + fabsf(h[a])) + 1e-7f;
        l[a] -= pad;
        h[a] += pad;
    }
    lo[i] = make_float4(l[0], l[1], l[2], 0.0f);
    hi[i] = make_float4(h[0], h[1], h[2], 0.0f);
}

// triangle records in the build's primitive order, and every mesh's root node and
// bounds (its tree's root box)
__global__ void k_fill_triangles(const uint32_t* __restrict__ order, BuildTrees B, const uint32_t* __restrict__ tree_mesh,
                                 uint32_t node_base, MeshInfo* meshes, const float* __restrict__ pos, const uint32_t* __restrict__ idx,
                                 const float4* __restrict__ node_lo, const float4* __restrict__ node_hi, TriRecord* out) {
    const uint32_t i = blockIdx.x * BLK + threadIdx.x;
    if (i >= B.total) return;
    const uint32_t prim = order[i], tree = tree_of(B, prim), first = tree_begin(B, tree), t = prim - first;
    MeshInfo& M = meshes[__ldg(tree_mesh + tree)];
    TriRecord r;
    float* v[3] = {r.v0, r.v1, r.v2};
    for (int k = 0; k < 3; k++) {
        const float* p = pos + 3ull * (M.vertex_offset + idx[M.index_offset + 3ull * t + k]);
        v[k][0] = p[0]; v[k][1] = p[1]; v[k][2] = p[2]; v[k][3] = 0.0f;
    }
    r.v0[3] = __uint_as_float(t);
    out[i] = r;
    if (t == 0u) {
        const uint32_t root = tree_end(B, tree) - first == 1u ? B.total + first : first;
        const float4 a = node_lo[root], z = node_hi[root];
        M.blas_root = node_base + tree;
        M.lo[0] = a.x; M.lo[1] = a.y; M.lo[2] = a.z;
        M.hi[0] = z.x; M.hi[1] = z.y; M.hi[2] = z.z;
    }
}

// How far a mesh reaches from its reference point along direction n, at most: with
// |n| sorted as p >= q >= r, n = (p - q) axis + (q - r) edge + r corner of the cube's
// directions, and what a shape reaches along a sum of directions is at most the sum of
// what it reaches along each.
__device__ __forceinline__ float reach(const MeshExtents& E, const float* n) {
    const float a[3] = {fabsf(n[0]), fabsf(n[1]), fabsf(n[2])};
    const bool neg[3] = {n[0] < 0.0f, n[1] < 0.0f, n[2] < 0.0f};
    auto along = [&](int axis, bool minus) {   // along +axis or -axis
        return minus ? -dec_f(~E.code[13 + axis]) : dec_f(E.code[axis]);
    };
    int p = 0, r = 0;
    if (a[1] > a[p]) p = 1;
    if (a[2] > a[p]) p = 2;
    if (a[1] <= a[r]) r = 1;
    if (a[2] <= a[r]) r = 2;
    if (p == r) { p = 0; r = 2; }   // (all alike)
    const int q = 3 - p - r, lo = min(p, q), hi = max(p, q);
    const int edge = (lo == 0 ? (hi == 1 ? 3 : 5) : 7) + (neg[lo] != neg[hi] ? 1 : 0);
    const int corner = 9 + (neg[1] != neg[0] ? 2 : 0) + (neg[2] != neg[0] ? 1 : 0);
    return (a[p] - a[q]) * along(p, neg[p]) + (a[q] - a[r]) * along(edge, neg[lo]) + a[r] * along(corner, neg[0]);
}

// World box of an instance: the box of its mesh's box corners, cut to what the mesh
// reaches along the box's own directions (26 object-space extents: a rotated mesh that
// does not fill its box gets a box of its own size, not of the box's corners; a
// sphere's is 1.1 to 1.2 instead of up to 1.7 times its diameter), with 1 % of the extent
// and 1e-5 of the mesh's coordinates to spare for the roundings of the object-space ray
// (0.1 % of the extent to spare gave 0.3 % more on the terrain, 5 % to spare took 1 %
// back).  A ray that enters an instance and leaves it
// without a hit costs its transform and a walk from the mesh's root: over 4,097 turned
// spheres, a 1920x1080 path-traced frame 1.997 -> 1.918 ms, one with reservoirs 16.98 ->
// 16.40 ms, 2^20 device rays 370 -> 347 us; the eight-view terrain (19.2 Mpx) 2.3 % less
// over eight seeds.  The extents cost the mesh build 12 us at 132,000 triangles
// (k_triangle_boxes 3 -> 7 us and a memset).
__global__ void k_instance_boxes(const uint32_t* __restrict__ list, uint32_t n, const InstShade* __restrict__ inst,
                                 const MeshInfo* __restrict__ meshes, const MeshExtents* __restrict__ extents,
                                 float4* lo, float4* hi) {
    uint32_t i = blockIdx.x * BLK + threadIdx.x;
    if (i >= n) return;
    const InstShade& I = inst[list[i]];
    const MeshInfo& M = meshes[I.mesh_id];
    const MeshExtents& E = extents[I.mesh_id];
    float l[3] = {3.4e38f, 3.4e38f, 3.4e38f}, h[3] = {-3.4e38f, -3.4e38f, -3.4e38f};
    for (int c = 0; c < 8; c++) {
        V3 p = v3((c & 1) ? M.hi[0] : M.lo[0], (c & 2) ? M.hi[1] : M.lo[1], (c & 4) ? M.hi[2] : M.lo[2]);
        V3 q = xform_point(I.m, p);
        l[0] = fminf(l[0], q.x); l[1] = fminf(l[1], q.y); l[2] = fminf(l[2], q.z);
        h[0] = fmaxf(h[0], q.x); h[1] = fmaxf(h[1], q.y); h[2] = fmaxf(h[2], q.z);
    }
    const V3 ref = xform_point(I.m, v3(E.ref[0], E.ref[1], E.ref[2]));
    const float r[3] = {ref.x, ref.y, ref.z};
    for (int a = 0; a < 3; a++) {
        const float up[3] = {I.m[4 * a], I.m[4 * a + 1], I.m[4 * a + 2]}, down[3] = {-up[0], -up[1], -up[2]};
        const float zl = r[a] - reach(E, down), zh = r[a] + reach(E, up);
        // the extent's share, and what the object-space ray may be off by: its roundings (and
        // ref's) are some ten of 2^-24 of the mesh's coordinates, which the world box need not
        // show when the translation takes them back; 1e-5 of them, as the triangles' boxes have
        // that the corners' box is made of
        float at = 0.0f;
        for (int k = 0; k < 3; k++) at += fabsf(up[k]) * fmaxf(fabsf(M.lo[k]), fabsf(M.hi[k]));
        const float spare = 0.01f * (zh - zl) + 1e-5f * at;
        if (zl - spare > l[a]) l[a] = zl - spare;   // (false for a NaN: the corners' box stays)
        if (zh + spare < h[a]) h[a] = zh + spare;
    }
    float ext = fmaxf(fmaxf(h[0] - l[0], h[1] - l[1]), h[2] - l[2]);
    for (int a = 0; a < 3; a++) {
        float pad = 1e-5f * (ext + fabsf(l[a]) + fabsf(h[a])) + 1e-6f;
        l[a] -= pad;
        h[a] += pad;
    }
    lo[i] = make_float4(l[0], l[1], l[2], 0.0f);
    hi[i] = make_float4(h[0], h[1], h[2], 0.0f);
}

__global__ void k_map_prims(const uint32_t* __restrict__ order, const uint32_t* __restrict__ list, uint32_t n,
                            uint32_t* out) {
    uint32_t i = blockIdx.x * BLK + threadIdx.x;
    if (i < n) out[i] = list[order[i]];
}

inline unsigned grid_for(uint32_t n) { return (n + BLK - 1) / BLK; }

}  // namespace

namespace {
// Morton codes of the build's primitives, sorted by (tree, code) stably; *keys / *sorted:
// the codes and primitives in order (either buffer pair)
Status sort_prims(BuildScratch& sc, const BuildTrees& B, const float4* prim_lo, const float4* prim_hi, cudaStream_t st,
                  const unsigned long long** keys, const uint32_t** sorted) {
    const uint32_t n = B.total, g = grid_for(n);
    *keys = sc.keys.p;
    *sorted = sc.vals.p;
    if (B.count == 1 && n <= SORT_BITONIC_MAX) {
        k_morton<<<g, BLK, 0, st>>>(prim_lo, prim_hi, B, sc.cbounds.p, sc.keys.p, sc.vals.p, nullptr, 0u);
        uint32_t N = 2;
        while (N < n) N <<= 1;
        k_sort_bitonic<<<1, SORT_THREADS, N * (sizeof(unsigned long long) + sizeof(uint32_t)), st>>>(sc.keys.p,
                                                                                                  sc.vals.p, n);
        SNK_TRY_CUDA(cudaGetLastError());
        return Status::Ok();
    }
    int passes = SORT_CODE_PASSES;
    for (uint32_t t = B.count - 1u; t; t >>= 8) passes++;
    uint32_t shift = 10;   // tiles of 1024 (one element per thread), or more when that would make over SORT_TILES
    while (((uint64_t)n + (1ull << shift) - 1) >> shift > SORT_TILES) shift++;
    const uint32_t tiles = (uint32_t)(((uint64_t)n + (1ull << shift) - 1) >> shift);
    const size_t rows = (size_t)SORT_RADIX * tiles;
    SNK_TRY_CUDA(sc.sort_hist.reserve(rows * passes));
    SNK_TRY_CUDA(cudaMemsetAsync(sc.sort_hist.p, 0, rows * passes * sizeof(uint32_t), st));
    k_morton<<<g, BLK, 0, st>>>(prim_lo, prim_hi, B, sc.cbounds.p, sc.keys.p, sc.vals.p, sc.sort_hist.p, shift);
    unsigned long long *sk = sc.keys.p, *dk = sc.keys_alt.p;
    uint32_t *sv = sc.vals.p, *dv = sc.vals_alt.p;
    for (int pass = 0; pass < passes; pass++) {
        k_sort_pass<<<tiles, SORT_THREADS, 0, st>>>(sk, sv, B, pass, shift, sc.sort_hist.p + rows * pass,
                                                    pass + 1 < passes ? sc.sort_hist.p + rows * (pass + 1) : nullptr, dk,
                                                    dv);
        std::swap(sk, dk);
        std::swap(sv, dv);
    }
    SNK_TRY_CUDA(cudaGetLastError());
    *keys = sk;
    *sorted = sv;
    return Status::Ok();
}
}  // namespace

Status build_wide_bvhs(BuildScratch& sc, const float4* prim_lo, const float4* prim_hi, const BuildTrees& B,
                       uint32_t max_n, WideNode* nodes, uint32_t node_base, uint32_t prim_base, uint32_t* prim_order,
                       unsigned* err_word, cudaStream_t st, int treelet_passes, uint32_t leaf_max, uint32_t leaf_pack,
                       SmallBuildOut* out, uint32_t* wide_depth, bool sah_collapse, bool sah_cost) {
    const uint32_t n = B.total;
    if (leaf_max < 1 || leaf_max > LEAF_MAX_LIMIT || leaf_pack < leaf_max || leaf_pack > LEAF_MAX_LIMIT)
        return Status::Err(1, "build_wide_bvhs: leaf size out of range");
    if (n == 0 || B.count == 0) return Status::Err(1, "build_wide_bvhs: no primitives");
    if (n > (1u << 30)) return Status::Err(1, "build_wide_bvhs: too many primitives");
    SNK_TRY_CUDA(sc.keys.reserve(n));
    SNK_TRY_CUDA(sc.keys_alt.reserve(n));
    SNK_TRY_CUDA(sc.vals.reserve(n));
    SNK_TRY_CUDA(sc.vals_alt.reserve(n));
    SNK_TRY_CUDA(sc.children.reserve(n));
    SNK_TRY_CUDA(sc.parent.reserve(2 * (size_t)n));
    SNK_TRY_CUDA(sc.flags.reserve(n));
    SNK_TRY_CUDA(sc.node_lo.reserve(2 * (size_t)n));
    SNK_TRY_CUDA(sc.node_hi.reserve(2 * (size_t)n));
    SNK_TRY_CUDA(sc.leaf_count.reserve(2 * (size_t)n));
    SNK_TRY_CUDA(sc.cost.reserve(2 * (size_t)n));
    SNK_TRY_CUDA(sc.tasks.reserve((size_t)n + B.count));
    SNK_TRY_CUDA(sc.counters.reserve(5));
    SNK_TRY_CUDA(sc.cbounds.reserve(6 * (size_t)B.count));
    SNK_TRY_CUDA(sc.sah.reserve(1));
    SNK_TRY_CUDA(sc.level_tasks.reserve(COLLAPSE_MAX_LEVELS + 1));

    const unsigned g = grid_for(n);
    SNK_TRY_CUDA(cudaMemsetAsync(sc.cbounds.p, 0, 6 * (size_t)B.count * sizeof(unsigned), st));
    SNK_TRY_CUDA(cudaMemsetAsync(sc.flags.p, 0, sizeof(int) * n, st));
    k_centroid_bounds<<<g, BLK, 0, st>>>(prim_lo, prim_hi, B, sc.cbounds.p);
    const unsigned long long* keys = nullptr;
    const uint32_t* sorted = nullptr;
    SNK_TRY(sort_prims(sc, B, prim_lo, prim_hi, st, &keys, &sorted));
    k_karras<<<g, BLK, 0, st>>>(keys, B, sc.children.p, sc.parent.p);
    bool boxes = false;   // the tree's boxes and counts are in place
    if (max_n >= (uint32_t)TL_LEAVES + 1) {
        for (int pass = 0; pass < treelet_passes; pass++) {
            if (boxes)
                k_treelet_pass<false><<<g, BLK, 0, st>>>((int)n, sorted, prim_lo, prim_hi, sc.children.p, sc.parent.p,
                                                         sc.flags.p, sc.node_lo.p, sc.node_hi.p, sc.leaf_count.p,
                                                         sc.cost.p, leaf_max);
            else
                k_treelet_pass<true><<<g, BLK, 0, st>>>((int)n, sorted, prim_lo, prim_hi, sc.children.p, sc.parent.p,
                                                        sc.flags.p, sc.node_lo.p, sc.node_hi.p, sc.leaf_count.p,
                                                        sc.cost.p, leaf_max);
            boxes = true;
        }
    }
    const uint32_t* wide_split = nullptr;
    if (sah_collapse) {   // SAH-optimal choice of each wide node's children over the final binary trees
        if (sc.wide_cost.reserve(std::max(8 * (size_t)n, SCRATCH_BYTES / sizeof(float))) != cudaSuccess) {
            cudaGetLastError();
            SNK_TRY_CUDA(sc.wide_cost.reserve(8 * (size_t)n));
        }
        SNK_TRY_CUDA(sc.wide_split.reserve(n));
        if (boxes)
            k_collapse_cost<false><<<g, BLK, 0, st>>>((int)n, sorted, prim_lo, prim_hi, sc.children.p, sc.parent.p,
                                                      sc.flags.p, sc.node_lo.p, sc.node_hi.p, sc.leaf_count.p,
                                                      sc.wide_cost.p, sc.wide_split.p, leaf_max, leaf_pack);
        else
            k_collapse_cost<true><<<g, BLK, 0, st>>>((int)n, sorted, prim_lo, prim_hi, sc.children.p, sc.parent.p,
                                                     sc.flags.p, sc.node_lo.p, sc.node_hi.p, sc.leaf_count.p,
                                                     sc.wide_cost.p, sc.wide_split.p, leaf_max, leaf_pack);
        wide_split = sc.wide_split.p;
    } else if (!boxes) {
        k_bottom_up<<<g, BLK, 0, st>>>(sorted, prim_lo, prim_hi, (int)n, sc.children.p, sc.parent.p, sc.flags.p,
                                       sc.node_lo.p, sc.node_hi.p, sc.leaf_count.p);
    }
    SNK_TRY_CUDA(cudaGetLastError());
    CollapseArgs A;
    A.B = B;
    A.tasks = sc.tasks.p;
    A.level_tasks = sc.level_tasks.p; A.counters = sc.counters.p;
    A.children = sc.children.p; A.node_lo = sc.node_lo.p; A.node_hi = sc.node_hi.p;
    A.leaf_count = sc.leaf_count.p; A.sorted = sorted; A.wide_split = wide_split;
    A.nodes = nodes; A.node_base = node_base; A.prim_base = prim_base; A.prim_order = prim_order;
    A.leaf_max = leaf_max; A.leaf_pack = leaf_pack; A.wide_depth = wide_depth;
    A.sah = sah_cost ? sc.sah.p : nullptr;
    k_collapse_init<<<(std::max(B.count, (uint32_t)COLLAPSE_MAX_LEVELS + 1u) + 255u) / 256u, 256, 0, st>>>(A);
    // enough warps for the widest level of a typical tree, at most 1024 blocks
    uint32_t grid = (n + 8u * LEVEL_WARPS - 1u) / (8u * LEVEL_WARPS);
    grid = grid < 1u ? 1u : (grid > 1024u ? 1024u : grid);
    // multi-block launches for about the depth of a balanced 8-wide tree; deeper
    // levels (unbalanced trees) go to the single-block finish
    int fast = 1;
    for (uint64_t cap = 8; cap < max_n && fast < COLLAPSE_FAST_LEVELS; cap *= 8) fast++;
    fast = fast + 2 < COLLAPSE_FAST_LEVELS ? fast + 2 : COLLAPSE_FAST_LEVELS;
    for (int level = 0; level < fast; level++) k_collapse_level<<<grid, 32 * LEVEL_WARPS, 0, st>>>(A, level);
    k_collapse_finish<<<1, 1024, 0, st>>>(A, fast, err_word, out);
    SNK_TRY_CUDA(cudaGetLastError());
    return Status::Ok();
}

Status build_wide_bvh_small(const float4* prim_lo, const float4* prim_hi, uint32_t n, WideNode* nodes,
                            uint32_t node_base, uint32_t prim_base, uint32_t* prim_order, int treelet_passes,
                            SmallBuildOut* out, unsigned* err_word, float4* wide_box, uint32_t* wide_depth,
                            cudaStream_t st, uint32_t leaf_max, bool sah_collapse) {
    if (n == 0 || n > (uint32_t)SMALL_BUILD_MAX) return Status::Err(1, "build_wide_bvh_small: bad primitive count");
    if (leaf_max < 1 || leaf_max > LEAF_MAX_LIMIT) return Status::Err(1, "build_wide_bvh_small: leaf size out of range");
    SNK_TRY_CUDA(cudaFuncSetAttribute(k_build_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)sizeof(SmallSmem)));
    k_build_small<<<1, SMALL_THREADS, sizeof(SmallSmem), st>>>(prim_lo, prim_hi, (int)n, treelet_passes, nodes,
                                                                node_base, prim_base, prim_order, out, err_word,
                                                                wide_box, wide_depth, leaf_max, sah_collapse);
    SNK_TRY_CUDA(cudaGetLastError());
    return Status::Ok();
}

Status refit_wide_bvh(const float4* prim_lo, const float4* prim_hi, uint32_t n, WideNode* nodes, uint32_t node_base,
                      uint32_t prim_base, const uint32_t* prim_order, const SmallBuildOut* info, float4* wide_box,
                      const uint32_t* wide_depth, unsigned* err_word, cudaStream_t st) {
    if (n == 0 || n > (1u << 30)) return Status::Err(1, "refit_wide_bvh: bad primitive count");
    k_refit_small<<<1, SMALL_THREADS, 0, st>>>(nodes, node_base, prim_base, info, wide_box, wide_depth, prim_order,
                                               prim_lo, prim_hi, (int)n, err_word);
    SNK_TRY_CUDA(cudaGetLastError());
    return Status::Ok();
}

Status launch_triangle_boxes(const float* positions, const uint32_t* indices, const BuildTrees& B,
                             const uint32_t* tree_mesh, const MeshInfo* meshes, MeshExtents* extents, float4* lo,
                             float4* hi, cudaStream_t s) {
    if (B.total)
        k_triangle_boxes<<<grid_for(B.total), BLK, 0, s>>>(positions, indices, B, tree_mesh, meshes, extents, lo, hi);
    SNK_TRY_CUDA(cudaGetLastError());
    return Status::Ok();
}

Status launch_fill_triangles(const BuildScratch& sc, const uint32_t* order, const BuildTrees& B,
                             const uint32_t* tree_mesh, uint32_t node_base, MeshInfo* meshes, const float* positions,
                             const uint32_t* indices, TriRecord* out, cudaStream_t s) {
    if (B.total)
        k_fill_triangles<<<grid_for(B.total), BLK, 0, s>>>(order, B, tree_mesh, node_base, meshes, positions, indices,
                                                           sc.node_lo.p, sc.node_hi.p, out);
    SNK_TRY_CUDA(cudaGetLastError());
    return Status::Ok();
}

Status launch_instance_boxes(const uint32_t* list, uint32_t n, const InstShade* inst, const MeshInfo* meshes,
                             const MeshExtents* extents, float4* lo, float4* hi, cudaStream_t s) {
    if (n) k_instance_boxes<<<grid_for(n), BLK, 0, s>>>(list, n, inst, meshes, extents, lo, hi);
    SNK_TRY_CUDA(cudaGetLastError());
    return Status::Ok();
}

Status launch_map_prims(const uint32_t* order, const uint32_t* list, uint32_t n, uint32_t* out, cudaStream_t s) {
    if (n) k_map_prims<<<grid_for(n), BLK, 0, s>>>(order, list, n, out);
    SNK_TRY_CUDA(cudaGetLastError());
    return Status::Ok();
}

}  // namespace snk

// snk_host.h -- host-side helpers shared by the library's translation units.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <string>
#include <utility>

#include "snk_device.cuh"
#include "snk_pt.h"

namespace snk {

// Owning device allocation (cudaMalloc/cudaFree); grows, never shrinks.
template <class T>
struct DBuf {
    T* p = nullptr;
    size_t n = 0;
    DBuf() = default;
    DBuf(const DBuf&) = delete;
    DBuf& operator=(const DBuf&) = delete;
    DBuf(DBuf&& o) noexcept : p(o.p), n(o.n) { o.p = nullptr; o.n = 0; }
    DBuf& operator=(DBuf&& o) noexcept { std::swap(p, o.p); std::swap(n, o.n); return *this; }
    ~DBuf() { release(); }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
    cudaError_t reserve(size_t count) {
        if (count <= n && p) return cudaSuccess;
        release();
        if (count == 0) count = 1;
        cudaError_t e = cudaMalloc(&p, count * sizeof(T));
        if (e != cudaSuccess) { p = nullptr; return e; }
        n = count;
        return cudaSuccess;
    }
    T* get() const { return p; }
};

// Error carrying a status code of snk_pt.h and a message.
struct Status {
    int code = 0;
    std::string msg;
    bool ok() const { return code == 0; }
    static Status Ok() { return Status(); }
    static Status Err(int c, std::string m) { Status s; s.code = c; s.msg = std::move(m); return s; }
};

#define SNK_TRY_CUDA(call)                                                                            \
    do {                                                                                              \
        cudaError_t e_ = (call);                                                                      \
        if (e_ != cudaSuccess)                                                                        \
            return ::snk::Status::Err(e_ == cudaErrorMemoryAllocation ? 3 : 2,                        \
                                      std::string(#call) + ": " + cudaGetErrorString(e_));           \
    } while (0)

#define SNK_TRY(expr)              \
    do {                           \
        ::snk::Status s_ = (expr); \
        if (!s_.ok()) return s_;   \
    } while (0)

// ---- BVH builder ---------------------------------------------------------------
// Least size of BuildScratch::wide_cost: what a part of a contact query needs.  (An
// allocation of 59 MB takes no longer than one of 4.)
constexpr size_t SCRATCH_BYTES = 56ull << 20;
struct BuildScratch {
    DBuf<unsigned long long> keys, keys_alt;
    DBuf<uint32_t> vals, vals_alt;
    DBuf<int2> children;
    DBuf<int> parent, flags;
    DBuf<float4> node_lo, node_hi;
    DBuf<uint32_t> leaf_count;
    DBuf<float> cost;             // binary-tree SAH cost per node (treelet restructuring)
    DBuf<uint32_t> tasks;         // per wide node: the binary node it is made of
    DBuf<uint32_t> counters;      // [2] wide nodes, [3] prims, [4] error bits
    DBuf<unsigned> cbounds;       // centroid bounds per tree, order-preserving encoded
    DBuf<uint32_t> sort_hist;     // per-tile digit counts of the radix sort, every digit
    DBuf<double> sah;             // SAH accumulator
    DBuf<uint32_t> level_tasks;   // task count per wide level
    DBuf<float> wide_cost;        // 8 per binary internal node: SAH cost of its subtree in 1..8 wide children;
                                  // between builds the scratch of the contact queries (SCRATCH_BYTES)
    DBuf<uint32_t> wide_split;    // per binary internal node: the split of those children (4-bit fields)
};

// How far a mesh reaches from one of its vertices (ref) along 13 axes: order-preserving
// codes of the largest distances, then the complements of the codes of the smallest
// (made by atomic maxima, so zero is the start).
struct MeshExtents {
    unsigned code[26];
    float ref[3];
    unsigned pad[3];
};

// The trees of one build: tree t's primitives are [first[t], first[t + 1]) of the
// concatenated boxes (device array of count + 1, each tree at least one primitive;
// not read for a single tree)
struct BuildTrees {
    const uint32_t* first;
    uint32_t count, total;
};

struct SmallBuildOut;
// Builds the 8-wide compressed BVHs of B's trees over their primitive boxes
// (prim_lo/prim_hi, xyz used) without host round trips.  Tree t's root is
// nodes[node_base + t], the other nodes follow with absolute child indices, at most
// total + count nodes in all; primitive slots are [prim_base, prim_base + total) and
// prim_order[k] receives the primitive (index of its box) stored in slot prim_base + k.
// max_n: the largest tree's primitives.  A build error (never seen for a correct tree)
// sets bit 8 of *err_word (when given) and out->error.  out (may be null) receives the
// node count, the deepest level and, with sah_cost, the sum over the trees of
// primitives x SAH cost below the root (internal 1, primitive 1, area relative to the
// root); wide_depth (total + 1 entries, may be null) every node's depth: with it a
// single tree can be refitted.
Status build_wide_bvhs(BuildScratch& sc, const float4* prim_lo, const float4* prim_hi, const BuildTrees& B,
                       uint32_t max_n, WideNode* nodes, uint32_t node_base, uint32_t prim_base, uint32_t* prim_order,
                       unsigned* err_word, cudaStream_t stream, int treelet_passes, uint32_t leaf_max,
                       uint32_t leaf_pack, SmallBuildOut* out, uint32_t* wide_depth, bool sah_collapse, bool sah_cost);

// Single-launch build for n <= SMALL_BUILD_MAX primitives (one CTA, shared
// memory, no host synchronisation); same collapse and output layout as
// build_wide_bvhs.  The result record stays on the device.  A build error (never
// seen for a correct tree) sets out->error and bit 8 of *err_word.
constexpr int SMALL_BUILD_MAX = 1024;
struct SmallBuildOut {
    uint32_t num_nodes, prims, error, max_depth;
    double sah;   // not computed by the per-frame builds (0)
    float lo[4], hi[4];
};
// wide_box (2 x (n + 1) float4: exact lo, hi per wide node) and wide_depth
// (n + 1) receive what a later refit needs.
Status build_wide_bvh_small(const float4* prim_lo, const float4* prim_hi, uint32_t n, WideNode* nodes,
                            uint32_t node_base, uint32_t prim_base, uint32_t* prim_order, int treelet_passes,
                            SmallBuildOut* out, unsigned* err_word, float4* wide_box, uint32_t* wide_depth,
                            cudaStream_t stream, uint32_t leaf_max, bool sah_collapse = true);
// Refit of a tree made by build_wide_bvh_small or build_wide_bvhs (one tree, with its
// record and depths) for the same n primitives in new boxes (prim_order as that
// build wrote it; wide_box: 2 x (n + 1) float4 of scratch that receives every
// node's exact box; everything stays on the device).
Status refit_wide_bvh(const float4* prim_lo, const float4* prim_hi, uint32_t n, WideNode* nodes, uint32_t node_base,
                      uint32_t prim_base, const uint32_t* prim_order, const SmallBuildOut* info, float4* wide_box,
                      const uint32_t* wide_depth, unsigned* err_word, cudaStream_t stream);

// Padded object-space boxes of the triangles of B's meshes (tree t is mesh tree_mesh[t]),
// and the meshes' extents (zeroed by the caller).
Status launch_triangle_boxes(const float* positions, const uint32_t* indices, const BuildTrees& B,
                             const uint32_t* tree_mesh, const MeshInfo* meshes, MeshExtents* extents, float4* lo,
                             float4* hi, cudaStream_t s);
// Triangle records from the build's primitive order, and the meshes' root nodes
// (node_base + t) and bounds (after the build that left its trees in sc).
Status launch_fill_triangles(const BuildScratch& sc, const uint32_t* prim_order, const BuildTrees& B,
                             const uint32_t* tree_mesh, uint32_t node_base, MeshInfo* meshes, const float* positions,
                             const uint32_t* indices, TriRecord* out, cudaStream_t s);
// World boxes of the listed instances (from the mesh bounds and extents) for the instance BVH.
Status launch_instance_boxes(const uint32_t* inst_list, uint32_t n, const InstShade* inst, const MeshInfo* meshes,
                             const MeshExtents* extents, float4* lo, float4* hi, cudaStream_t s);
// ---- per-frame scene tables (scene_tables.cu) ---------------------------------
struct LightCdfScratch {
    DBuf<unsigned long long> acc, wmax, tile_sums, q;   // prefix sums, max weight, tile sums, quantised weights
};
// traversal and shading records of n instances from their raw records
Status launch_instance_records(const snk_instance* raw, uint32_t n, const MeshInfo* meshes, InstTrace* it,
                               InstShade* is, cudaStream_t st);
// ReSTIR candidate records of the emissive instances em_list[0..n_em) (after their instance records)
Status launch_emissive_records(const uint32_t* em_list, uint32_t n_em, const InstShade* is, const MeshInfo* meshes,
                               const MaterialDev* mats, EmissiveRec* recs, cudaStream_t st);
// NEE records and weights of the n_tri triangles of the emissive instances em_list[0..n_em)
// (em_first: prefix sums of their triangle counts)
Status launch_emissive_lights(const snk_instance* raw, const uint32_t* em_list, const uint32_t* em_first, uint32_t n_em,
                              uint32_t n_tri, const MeshInfo* meshes, const float* pos, const uint32_t* idx,
                              const MaterialDev* mats, LocalLight* lights, double* w, cudaStream_t st);
// light-selection CDF and PMF of n weights (quantised to integers, exact prefix sums)
Status launch_light_cdf(const double* w, uint32_t n, LightCdfScratch& sc, float* cdf, float* pmf, cudaStream_t st);
// the same table computed on the host (for tables whose weights are all known there)
void light_cdf_host(const double* w, uint32_t n, float* cdf, float* pmf);

// tlas_prims[k] = inst_list[prim_order[k]]
Status launch_map_prims(const uint32_t* prim_order, const uint32_t* inst_list, uint32_t n, uint32_t* out,
                        cudaStream_t s);

}  // namespace snk

// Locator block of a tetrahedral-mesh field (jt_mesh.cuh): the table that
// stands for the first moves of the octree descent, and the tetrahedron
// records in element-list order.
#include <math_constants.h>
#include <stdint.h>

#include "jt_internal.h"
#include "jt_kernels.cuh"
#include "jt_mesh.cuh"

namespace jt {

// Header and the cells' {lower, upper} faces, one thread per axis and cell.
__global__ void __launch_bounds__(kBlock) k_locator_faces(const float* __restrict__ splits, int depth, float* header,
                                                          float2* faces) {
    const int n = 1 << depth, i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 3 * n) return;
    const int a = i >> depth, c = i & (n - 1);
    const float* s = splits + a * (n + 1);
    faces[i] = make_float2(c == 0 ? CUDART_NAN_F : s[c], c == n - 1 ? CUDART_NAN_F : s[c + 1]);
    if (c == 0) {
        const float w = s[n] - s[0];
        header[a] = s[0];
        header[3 + a] = w > 0.0f ? (float)n / w : 0.0f;
    }
}

// One thread per cell walks the moves its path takes, comparing every centre
// with the face the cells are cut at; a difference is reported in *mismatch.
__global__ void __launch_bounds__(kBlock) k_locator_table(const int4* __restrict__ desc, const int2* __restrict__ dtab,
                                                          const float* __restrict__ splits, int depth, int max_depth,
                                                          int2* __restrict__ table, int32_t* mismatch) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 1 << (3 * depth)) return;
    const int n = 1 << depth, cell[3] = {i >> (2 * depth), (i >> depth) & (n - 1), i & (n - 1)};
    int node = 0;
    bool below = true;  // the descent goes on below `node`
    for (int d = 0; d < depth; ++d) {
        const int4 h = __ldg(desc + node);
        const unsigned w = (unsigned)h.w, m = w & 0xffu;
        if (m == 0u) { below = false; break; }
        const int c[3] = {h.x, h.y, h.z}, low = depth - 1 - d;
        int oct = 0;
        bool same = true;
        for (int a = 0; a < 3; ++a) {
            const int half = ((cell[a] >> (low + 1)) * 2 + 1) << low;  // first cell of the upper half
            same &= __float_as_int(splits[a * (n + 1) + half]) == c[a];
            oct |= ((cell[a] >> low) & 1) << a;
        }
        if (!same) atomicExch(mismatch, 1);
        if (!((m >> oct) & 1u)) { below = false; break; }
        node = (int)(w >> 8) + __popc(m & ((1u << oct) - 1u));
    }
    table[i] = below && depth < max_depth ? make_int2(node, -1) : __ldg(dtab + node);
}

// Geometry and filter records of the element lists, one warp per list and one
// lane per slot.  Lists longer than kAloneMost get no JT_TET_ALONE (the check
// compares every pair of a list).
constexpr int kAloneMost = 96;

__global__ void __launch_bounds__(kBlock) k_locator_slots(const int2* __restrict__ dtab, int n_nodes,
                                                          const int32_t* __restrict__ elems,
                                                          const float* __restrict__ tet_box,
                                                          const float* __restrict__ geom, int n_entries,
                                                          uint4* __restrict__ slots, uint4* __restrict__ filters) {
    const int node = (blockIdx.x * kBlock + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (node >= n_nodes) return;
    const int2 oc = __ldg(dtab + node);
    for (int s = lane; s < oc.y && oc.x + s < n_entries; s += 32) {
        const int64_t slot = oc.x + s, t = __ldg(elems + slot);
        const uint4* g4 = reinterpret_cast<const uint4*>(geom) + 4 * t;
        float g[12], b[8];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint4 r = __ldg(g4 + k);
            slots[4 * slot + k] = r;
            if (k < 3) {
                g[4 * k] = __uint_as_float(r.x);
                g[4 * k + 1] = __uint_as_float(r.y);
                g[4 * k + 2] = __uint_as_float(r.z);
                g[4 * k + 3] = __uint_as_float(r.w);
            }
        }
        for (int k = 0; k < 8; ++k) b[k] = __ldg(tet_box + 8 * t + k);
        uint32_t flags = shape_ratio(g) <= kWellShaped ? JT_TET_SHAPED : 0;
        if (flags && oc.y <= kAloneMost) {
            bool alone = true;
            for (int r = 0; r < s && alone; ++r) {
                const int64_t o = __ldg(elems + oc.x + r);
                float ge[12], be[8];
                for (int k = 0; k < 12; ++k) ge[k] = __ldg(geom + 16 * o + k);
                for (int k = 0; k < 8; ++k) be[k] = __ldg(tet_box + 8 * o + k);
                alone = tets_apart(ge, be, g, b);
            }
            if (alone) flags |= JT_TET_ALONE;
        }
        uint32_t w[8];
        make_filter(g, b, flags, w);
        filters[2 * slot] = make_uint4(w[0], w[1], w[2], w[3]);
        filters[2 * slot + 1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
}

}  // namespace jt

using namespace jt;

extern "C" size_t jt_mesh_locator_bytes(int32_t n_nodes, int32_t n_tets, int32_t depth) {
    if (n_nodes < 1 || n_tets < 1 || depth < 1 || depth > JT_MESH_LOCATOR_MAX_DEPTH) return 0;
    return locator_layout(n_nodes, n_tets, depth).bytes;
}

extern "C" int jt_mesh_locator_build(const jt_mesh_field* m, int32_t depth, const float* splits,
                                     int32_t* locator_out, void* stream) {
    if (m == nullptr || splits == nullptr || locator_out == nullptr)
        return set_error(JT_ERR_INVALID, "mesh, splits and locator_out are required");
    *locator_out = 0;
    if (m->desc == nullptr || m->dtab == nullptr || m->elems == nullptr || m->tet_geom == nullptr ||
        m->tet_box == nullptr)
        return set_error(JT_ERR_INVALID, "the locator needs desc, dtab, elems, tet_box and tet_geom");
    if (((uintptr_t)m->dtab & 63u) != 0) return set_error(JT_ERR_INVALID, "dtab must be 64-byte aligned");
    if (m->n_nodes < 1 || m->n_tets < 1) return set_error(JT_ERR_INVALID, "n_nodes and n_tets must be positive");
    if ((int64_t)m->n_nodes > (int64_t)1 << 26) return set_error(JT_ERR_UNSUPPORTED, "too many nodes for a locator");
    if (depth < 1 || depth > JT_MESH_LOCATOR_MAX_DEPTH || depth > m->max_depth)
        return set_error(JT_ERR_INVALID, "locator depth %d must be 1..%d and at most max_depth", depth,
                         JT_MESH_LOCATOR_MAX_DEPTH);
    const LocatorLayout o = locator_layout(m->n_nodes, m->n_tets, depth);
    char* base = reinterpret_cast<char*>(const_cast<int32_t*>(m->dtab));
    float* header = reinterpret_cast<float*>(base + o.header);
    int32_t* mismatch = reinterpret_cast<int32_t*>(header) + 7;
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t err = cudaMemsetAsync(header, 0, 64, s);
    if (err != cudaSuccess) return cuda_status(err, "mesh locator memset");
    k_locator_faces<<<grid_blocks((int64_t)3 << depth), kBlock, 0, s>>>(splits, depth, header,
                                                                       reinterpret_cast<float2*>(base + o.faces));
    k_locator_table<<<grid_blocks((int64_t)1 << (3 * depth)), kBlock, 0, s>>>(
        reinterpret_cast<const int4*>(m->desc), reinterpret_cast<const int2*>(m->dtab), splits, depth, m->max_depth,
        reinterpret_cast<int2*>(base + o.table), mismatch);
    k_locator_slots<<<grid_blocks(32 * (int64_t)m->n_nodes), kBlock, 0, s>>>(
        reinterpret_cast<const int2*>(m->dtab), m->n_nodes, m->elems, m->tet_box, m->tet_geom, m->n_tets,
        reinterpret_cast<uint4*>(base + o.slots), reinterpret_cast<uint4*>(base + o.filters));
    int32_t bad = 0;
    err = cudaGetLastError();
    if (err == cudaSuccess) err = cudaMemcpyAsync(&bad, mismatch, sizeof(bad), cudaMemcpyDeviceToHost, s);
    if (err == cudaSuccess) err = cudaStreamSynchronize(s);
    if (err != cudaSuccess) return cuda_status(err, "mesh locator build");
    if (bad == 0) *locator_out = kLocatorMagic | depth;
    return JT_OK;
}

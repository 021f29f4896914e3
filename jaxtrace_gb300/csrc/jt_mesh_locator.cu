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

// A tetrahedron's record into its list slot, 16 B per thread.
__global__ void __launch_bounds__(kBlock) k_locator_slots(const int32_t* __restrict__ elems,
                                                          const float* __restrict__ geom, int64_t n,
                                                          uint4* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 4 * n) return;
    const float* g = geom + 16 * (int64_t)__ldg(elems + (i >> 2));
    uint4 r = __ldg(reinterpret_cast<const uint4*>(g) + (i & 3));
    if ((i & 3) == 3 && well_shaped(g)) r.x |= 0x80000000u;
    out[i] = r;
}

}  // namespace jt

using namespace jt;

extern "C" size_t jt_mesh_locator_bytes(int32_t n_nodes, int32_t n_entries, int32_t depth) {
    if (n_nodes < 1 || n_entries < 0 || depth < 1 || depth > JT_MESH_LOCATOR_MAX_DEPTH) return 0;
    return locator_layout(n_nodes, n_entries, depth).bytes;
}

extern "C" int jt_mesh_locator_build(const jt_mesh_field* m, int32_t n_entries, int32_t depth, const float* splits,
                                     int32_t* locator_out, void* stream) {
    if (m == nullptr || splits == nullptr || locator_out == nullptr)
        return set_error(JT_ERR_INVALID, "mesh, splits and locator_out are required");
    *locator_out = 0;
    if (m->desc == nullptr || m->dtab == nullptr || m->elems == nullptr || m->tet_geom == nullptr)
        return set_error(JT_ERR_INVALID, "the locator needs desc, dtab, elems and tet_geom");
    if (((uintptr_t)m->dtab & 63u) != 0) return set_error(JT_ERR_INVALID, "dtab must be 64-byte aligned");
    if (m->n_nodes < 1 || n_entries < 0) return set_error(JT_ERR_INVALID, "n_nodes and n_entries must be positive");
    if (depth < 1 || depth > JT_MESH_LOCATOR_MAX_DEPTH || depth > m->max_depth)
        return set_error(JT_ERR_INVALID, "locator depth %d must be 1..%d and at most max_depth", depth,
                         JT_MESH_LOCATOR_MAX_DEPTH);
    const LocatorLayout o = locator_layout(m->n_nodes, n_entries, depth);
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
    if (n_entries > 0)
        k_locator_slots<<<grid_blocks(4 * (int64_t)n_entries), kBlock, 0, s>>>(
            m->elems, m->tet_geom, n_entries, reinterpret_cast<uint4*>(base + o.slots));
    int32_t bad = 0;
    err = cudaGetLastError();
    if (err == cudaSuccess) err = cudaMemcpyAsync(&bad, mismatch, sizeof(bad), cudaMemcpyDeviceToHost, s);
    if (err == cudaSuccess) err = cudaStreamSynchronize(s);
    if (err != cudaSuccess) return cuda_status(err, "mesh locator build");
    if (bad == 0) *locator_out = kLocatorMagic | depth;
    return JT_OK;
}

// Filter records of a hash-grid FEM field (jt_mesh.cuh), one per tetrahedron.
//
// JT_TET_ALONE here: no tetrahedron with a smaller number accepts a query well
// inside this one, and this one is on the list of every cell such a query
// looks in.  The first is checked against the elements of the hash cells this
// one's box meets, where every element whose box meets it is listed.  For the
// second, a query well inside lies kInsideTrue of the box's extent or more from
// the box's faces; the lists' cell range and the query's cell round by less
// than 16 * 2^-24 of the grid, which has to be less than that.
#include <stdint.h>

#include "jt_fem.cuh"
#include "jt_internal.h"
#include "jt_kernels.cuh"

namespace jt {

constexpr int kFemAloneMost = 4096;  // listed elements compared per tetrahedron

// The records, without JT_TET_ALONE: their float64 gradients take a thread per
// tetrahedron (in the warp-per-tetrahedron kernel below they and float64 cell
// ranges were most of its 30 ms).
__global__ void __launch_bounds__(kBlock) k_fem_filters(jt_fem_field F, uint4* __restrict__ out) {
    const int t = blockIdx.x * kBlock + threadIdx.x;
    if (t >= F.n_tets) return;
    float g[12], b[8];
    for (int k = 0; k < 12; ++k) g[k] = __ldg(F.tet_geom + 16 * (int64_t)t + k);
    for (int k = 0; k < 8; ++k) b[k] = __ldg(F.tet_box + 8 * (int64_t)t + k);
    uint32_t w[8];
    make_filter(g, b, shape_ratio(g) <= kWellShaped ? JT_TET_SHAPED : 0, w);
    out[2 * (int64_t)t] = make_uint4(w[0], w[1], w[2], w[3]);
    out[2 * (int64_t)t + 1] = make_uint4(w[4], w[5], w[6], w[7]);
}

// JT_TET_ALONE, one warp per tetrahedron, the lanes over the elements of its
// cells.  Those whose boxes meet this one's are gathered 32 at a time before
// tets_apart runs: one lane in ten has one.
__global__ void __launch_bounds__(kBlock) k_fem_alone(jt_fem_field F, uint32_t* __restrict__ filters) {
    __shared__ int32_t queue[kBlock / 32][64];
    const int t = (blockIdx.x * kBlock + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (t >= F.n_tets) return;
    int32_t* mine = queue[threadIdx.x >> 5];
    float g[12], b[8];
    for (int k = 0; k < 12; ++k) g[k] = __ldg(F.tet_geom + 16 * (int64_t)t + k);
    for (int k = 0; k < 8; ++k) b[k] = __ldg(F.tet_box + 8 * (int64_t)t + k);
    bool alone = shape_ratio(g) <= kWellShaped;
    int lo[3], hi[3];
    for (int a = 0; a < 3; ++a) {
        const float cs = F.cell_size[a], n = (float)F.grid_size[a];
        if (cs > 0.0f) {
            // the cells the box meets, widened by more than the lists' rounding
            // and this one's (at most 4 * 2^-24 of 4096 cells)
            const float l = (b[a] - F.grid_min[a]) / cs, h = (b[4 + a] - F.grid_min[a]) / cs;
            alone = alone && n <= 4096.0f && kInsideTrue * (h - l) >= 16.0f / 16777216.0f * (n + 1.0f);
            lo[a] = (int)fminf(fmaxf(floorf(l - 4e-3f), 0.0f), n - 1.0f);
            hi[a] = (int)fminf(fmaxf(floorf(h + 4e-3f), 0.0f), n - 1.0f);
        } else {
            alone = false;
            lo[a] = hi[a] = 0;
        }
    }
    const auto apart = [&](int e) {
        float ge[12], be[8];
        const auto load = [](float* v, const float* p) {
            const float4 r = __ldg(reinterpret_cast<const float4*>(p));
            v[0] = r.x; v[1] = r.y; v[2] = r.z; v[3] = r.w;
        };
#pragma unroll
        for (int k = 0; k < 3; ++k) load(ge + 4 * k, F.tet_geom + 16 * (int64_t)e + 4 * k);
#pragma unroll
        for (int k = 0; k < 2; ++k) load(be + 4 * k, F.tet_box + 8 * (int64_t)e + 4 * k);
        return tets_apart(ge, be, g, b);
    };
    int visits = 0, queued = 0;
    const int ny = hi[1] - lo[1] + 1, nz = hi[2] - lo[2] + 1, cells = (hi[0] - lo[0] + 1) * ny * nz;
    alone = alone && cells <= kFemAloneMost;
    for (int c = 0; c < cells && alone; ++c) {
        const int i = lo[0] + c / (ny * nz), j = lo[1] + (c / nz) % ny, k = lo[2] + c % nz;
        const int64_t cell = ((int64_t)i * F.grid_size[1] + j) * F.grid_size[2] + k;
        // an element that reaches well into the previous cell of an axis, which
        // this box meets too, is on that cell's list and was seen there
        const float fx = i > lo[0] ? F.grid_min[0] + ((float)i - 0.01f) * F.cell_size[0] : -3.4e38f;
        const float fy = j > lo[1] ? F.grid_min[1] + ((float)j - 0.01f) * F.cell_size[1] : -3.4e38f;
        const float fz = k > lo[2] ? F.grid_min[2] + ((float)k - 0.01f) * F.cell_size[2] : -3.4e38f;
        const int s0 = __ldg(F.cell_start + cell), s1 = __ldg(F.cell_start + cell + 1);
        visits += s1 - s0;
        alone = visits <= kFemAloneMost;
        for (int s = s0; s < s1 && alone; s += 32) {
            const int e = s + lane < s1 ? __ldg(F.cell_elems + s + lane) : t;
            if (__shfl_sync(0xffffffffu, e, 0) >= t) break;  // ascending lists
            bool meets = false;
            if (e < t) {
                const float4 mn = __ldg(reinterpret_cast<const float4*>(F.tet_box) + 2 * (int64_t)e);
                const float4 mx = __ldg(reinterpret_cast<const float4*>(F.tet_box) + 2 * (int64_t)e + 1);
                meets = !(mn.x > b[4] || mx.x < b[0] || mn.y > b[5] || mx.y < b[1] || mn.z > b[6] || mx.z < b[2]) &&
                        !(mn.x < fx || mn.y < fy || mn.z < fz);
            }
            const unsigned m = __ballot_sync(0xffffffffu, meets);
            if (meets) mine[queued + __popc(m & ((1u << lane) - 1u))] = e;
            queued += __popc(m);
            __syncwarp();
            if (queued >= 32) {
                alone = __all_sync(0xffffffffu, apart(mine[lane]));
                queued -= 32;
                const int rest = lane < queued ? mine[32 + lane] : 0;
                __syncwarp();
                mine[lane] = rest;
                __syncwarp();
            }
        }
    }
    if (alone && queued > 0) alone = __all_sync(0xffffffffu, lane >= queued || apart(mine[lane]));
    if (lane == 0 && alone) filters[8 * (int64_t)t + 7] |= (uint32_t)JT_TET_ALONE << 16;
}

// ---------------------------------------------------------------------------
// Pruned sub-cell lists: the sub-cell lists hold every element whose box meets
// the sub-cell, about 12.6 on a jittered hexahedral split where the elements
// themselves meet 3.6.  An element stays unless one of its filtered barycentrics
// is below -slack everywhere in the sub-cell (widened by eps, as the lists are):
// the filter then rejects each of its queries, so the first hits are the same.
// The float16 gradients' rounding beyond the element's box, up to the cell's
// half-width h, adds 2^-11 h |g| a component.
// ---------------------------------------------------------------------------
struct SubBox {
    float c[3], h[3];
};

__device__ __forceinline__ bool filter_misses(const uint32_t (&w)[8], const SubBox& s) {
    const auto h2 = [&w](int i) { return __half22float2(*reinterpret_cast<const __half2*>(&w[i])); };
    const float2 a = h2(3), b = h2(4), c = h2(5), d = h2(6), e = h2(7);
    const float g[3][3] = {{a.x, a.y, b.x}, {b.y, c.x, c.y}, {d.x, d.y, e.x}};
    const float p[3] = {s.c[0] - __uint_as_float(w[0]), s.c[1] - __uint_as_float(w[1]), s.c[2] - __uint_as_float(w[2])};
    float b0 = 1.0f, reach0 = 0.0f, spread = 0.0f;
    bool miss = false;
    for (int i = 0; i < 3; ++i) {
        const float v = p[0] * g[i][0] + p[1] * g[i][1] + p[2] * g[i][2];
        const float reach = s.h[0] * fabsf(g[i][0]) + s.h[1] * fabsf(g[i][1]) + s.h[2] * fabsf(g[i][2]);
        miss = miss || v + 1.001f * reach < -e.y;
        b0 -= v;
        spread += reach;
    }
    for (int k = 0; k < 3; ++k) reach0 += s.h[k] * fabsf(g[0][k] + g[1][k] + g[2][k]);
    return miss || b0 + reach0 + 1e-3f * spread < -e.y;
}

// One thread per sub-cell.  FILL 0: counts[sc] = entries kept; FILL 1: writes
// them at start[sc], in their order.
template <int FILL>
__global__ void __launch_bounds__(kBlock) k_fem_prune(jt_fem_field F, float3 eps, int64_t n_sub,
                                                      uint32_t* __restrict__ counts, const uint32_t* __restrict__ start,
                                                      int32_t* __restrict__ out) {
    const int64_t sc = (int64_t)blockIdx.x * kBlock + threadIdx.x;
    if (sc >= n_sub) return;
    const int S = F.sub_div & ~JT_FEM_FILTERS, S3 = S * S * S;
    const int64_t cell = sc / S3;
    const int sub = (int)(sc - cell * S3);
    const int cc[3] = {(int)(cell / ((int64_t)F.grid_size[1] * F.grid_size[2])),
                       (int)((cell / F.grid_size[2]) % F.grid_size[1]), (int)(cell % F.grid_size[2])};
    const int ss[3] = {sub / (S * S), (sub / S) % S, sub % S};
    const float ep[3] = {eps.x, eps.y, eps.z};
    SubBox box;
    for (int a = 0; a < 3; ++a) {
        const double w = (double)F.cell_size[a] / S;
        box.c[a] = (float)((double)F.grid_min[a] + (double)cc[a] * (double)F.cell_size[a] + (ss[a] + 0.5) * w);
        box.h[a] = (float)(0.5 * w) + ep[a];
    }
    const int b = __ldg(F.sub_start + sc), en = __ldg(F.sub_start + sc + 1);
    const char* filters = reinterpret_cast<const char*>(F.tet_geom) + (int64_t)F.n_tets * 64;
    uint32_t n = FILL ? start[sc] : 0u;
    const uint32_t end = FILL ? start[sc + 1] : 0u;
    for (int s = b; s < en; ++s) {
        const int t = __ldg(F.sub_elems + s);
        uint32_t w[8];
        ldg256(filters + (int64_t)t * 32, w);
        if (filter_misses(w, box)) continue;
        if (FILL && n < end) out[n] = t;
        ++n;
    }
    if (!FILL) counts[sc] = n;
}

static int64_t sub_cells(const jt_fem_field& f) {
    const int64_t S = f.sub_div & ~JT_FEM_FILTERS;
    return (int64_t)f.grid_size[0] * f.grid_size[1] * f.grid_size[2] * S * S * S;
}

static int check_prune(const jt_fem_field* f, const float* eps) {
    if (f == nullptr || eps == nullptr || f->sub_start == nullptr || f->sub_elems == nullptr || f->tet_geom == nullptr)
        return set_error(JT_ERR_INVALID, "pruning needs a field with sub-cell lists, and eps");
    const int S = f->sub_div & ~JT_FEM_FILTERS;
    if (!(f->sub_div & JT_FEM_FILTERS) || S < 1 || S > 16)
        return set_error(JT_ERR_INVALID, "pruning needs sub_div 1..16 with JT_FEM_FILTERS");
    if (sub_cells(*f) + 1 > scan_capacity()) return set_error(JT_ERR_UNSUPPORTED, "too many sub-cells");
    return JT_OK;
}

}  // namespace jt

using namespace jt;

extern "C" int jt_fem_prune_count(const jt_fem_field* f, const float* eps, uint32_t* start, int64_t* total,
                                  void* stream) {
    if (int rc = check_prune(f, eps)) return rc;
    if (start == nullptr || total == nullptr) return set_error(JT_ERR_INVALID, "start and total are required");
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t n = sub_cells(*f), p1 = scan_partials(n + 1), p2 = scan_partials2(n + 1);
    uint32_t* sums = nullptr;
    cudaError_t e = dev_alloc((void**)&sums, (size_t)(p1 + p2) * 4, s);
    if (e != cudaSuccess) return cuda_status(e, "prune scan scratch");
    e = cudaMemsetAsync(start + n, 0, 4, s);
    if (e == cudaSuccess) {
        k_fem_prune<0><<<grid_blocks(n), kBlock, 0, s>>>(*f, make_float3(eps[0], eps[1], eps[2]), n, start, nullptr,
                                                        nullptr);
        e = cudaGetLastError();
    }
    const int rc = e == cudaSuccess ? exclusive_scan_u32(start, n + 1, sums, sums + p1, s) : JT_OK;
    uint32_t last = 0;
    if (e == cudaSuccess && rc == JT_OK) e = cudaMemcpyAsync(&last, start + n, 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess && rc == JT_OK) e = cudaStreamSynchronize(s);
    dev_free(sums, s);
    if (e != cudaSuccess) return cuda_status(e, "prune count");
    *total = last;
    return rc;
}

extern "C" int jt_fem_prune_fill(const jt_fem_field* f, const float* eps, const uint32_t* start, int32_t* elems,
                                 void* stream) {
    if (int rc = check_prune(f, eps)) return rc;
    if (start == nullptr || elems == nullptr) return set_error(JT_ERR_INVALID, "start and elems are required");
    const int64_t n = sub_cells(*f);
    k_fem_prune<1><<<grid_blocks(n), kBlock, 0, (cudaStream_t)stream>>>(*f, make_float3(eps[0], eps[1], eps[2]), n,
                                                                       nullptr, start, elems);
    return cuda_status(cudaGetLastError(), "prune fill");
}

extern "C" size_t jt_fem_filters_bytes(int32_t n_tets) { return n_tets < 1 ? 0 : (size_t)n_tets * 96; }

extern "C" int jt_fem_filters_build(const jt_fem_field* f, void* stream) {
    if (f == nullptr || f->n_tets < 1 || f->tet_box == nullptr || f->tet_geom == nullptr || f->cell_start == nullptr ||
        f->cell_elems == nullptr)
        return set_error(JT_ERR_INVALID, "the filter records need tetrahedra, boxes, geometry and cell lists");
    for (int a = 0; a < 3; ++a)
        if (f->grid_size[a] < 1) return set_error(JT_ERR_INVALID, "grid_size must be positive");
    if (((uintptr_t)f->tet_geom & 31u) != 0)
        return set_error(JT_ERR_INVALID, "filter records need tet_geom on a 32-byte boundary");
    if (f->n_tets > 1 << 26) return set_error(JT_ERR_UNSUPPORTED, "too many tetrahedra for filter records");
    char* out = reinterpret_cast<char*>(const_cast<float*>(f->tet_geom)) + (int64_t)f->n_tets * 64;
    cudaStream_t s = (cudaStream_t)stream;
    k_fem_filters<<<grid_blocks(f->n_tets), kBlock, 0, s>>>(*f, reinterpret_cast<uint4*>(out));
    k_fem_alone<<<grid_blocks(32 * (int64_t)f->n_tets), kBlock, 0, s>>>(*f, reinterpret_cast<uint32_t*>(out));
    return cuda_status(cudaGetLastError(), "filter records");
}

// Build of the nearest-node candidate lists (jt_nearest.cuh).
//
// Node p is on a cell's list unless j0, the node nearest to the cell's centre,
// is nearer to every point of the cell: |x - p|^2 - |x - j0|^2 is linear in x,
// so its least value over the cell is that at one corner, and p is left out
// where that exceeds kListMargin times the largest |x - j0|^2 in the cell: a
// float32 squared distance is off by less than 4 * 2^-24 of itself, so the
// argmin of a query in the cell cannot be p, nor tie with it.  Cells are grown
// by 1e-3 of their edge, above the float32 rounding of a query's cell.
#include <stdint.h>

#include "jt_internal.h"
#include "jt_kernels.cuh"
#include "jt_nearest.cuh"

namespace jt {

// A cell whose surroundings are too sparse or too crowded for a short list gets
// an empty one; its queries are searched through the cell list as before.  The
// limits keep the build linear in the cells whatever the nodes' spread.
constexpr float kListMargin = 1e-5f;
constexpr int kListCube = 3;      // cell-list cells around the centre's searched for j0
constexpr int kListRows = 144;    // rows of cells and
constexpr int kListVisits = 2048; // nodes looked at
constexpr int kListMost = 48;     // nodes listed

// One thread per cell.  FILL 0: counts[cell] = length of its list; FILL 1:
// writes the records at start[cell] and sorts them by id.
template <int FILL>
__global__ void __launch_bounds__(kBlock) k_nearest_lists(jt_nearest_field F, NearestLists g,
                                                          uint32_t* __restrict__ counts,
                                                          const uint32_t* __restrict__ start, float4* __restrict__ rec) {
    const int64_t cell = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (cell >= g.cells) return;
    const int i[3] = {(int)(cell % g.n[0]), (int)((cell / g.n[0]) % g.n[1]), (int)(cell / ((int64_t)g.n[0] * g.n[1]))};
    double c[3];
    float h[3], diag = 0.0f;
    for (int a = 0; a < 3; ++a) {
        const double e = 1.0 / (double)g.inv[a];
        c[a] = (double)g.org[a] + ((double)i[a] + 0.5) * e;
        h[a] = (float)(0.501 * e);
        diag += h[a] * h[a];
    }
    diag = sqrtf(diag) * 1.0001f;
    const float4* pts = reinterpret_cast<const float4*>(F.points);
    const auto cell_of = [&F](double x, float w, int a) {
        const float f = (float)(x - (double)F.origin[a]) * F.inv_cell[a] + w;
        return (int)fminf(fmaxf(floorf(f), 0.0f), (float)(F.cells[a] - 1));
    };
    // j0: the node nearest to the centre within the smallest cube of cells that
    // has one (any node near the centre would do)
    int near = -1;
    float dn = __int_as_float(0x7f800000);
    for (int r = 0; r <= kListCube && near < 0; ++r)
        for (int z = max(cell_of(c[2], 0.0f, 2) - r, 0); z <= min(cell_of(c[2], 0.0f, 2) + r, F.cells[2] - 1); ++z)
            for (int y = max(cell_of(c[1], 0.0f, 1) - r, 0); y <= min(cell_of(c[1], 0.0f, 1) + r, F.cells[1] - 1); ++y) {
                const int row = (z * F.cells[1] + y) * F.cells[0], x = cell_of(c[0], 0.0f, 0);
                const int b = __ldg(F.cell_start + row + max(x - r, 0));
                const int en = min(__ldg(F.cell_start + row + min(x + r, F.cells[0] - 1) + 1), b + kListVisits);
                for (int s = b; s < en; ++s) {
                    const float4 q = __ldg(pts + s);
                    const float p[3] = {(float)((double)q.x - c[0]), (float)((double)q.y - c[1]),
                                        (float)((double)q.z - c[2])};
                    const float d = p[0] * p[0] + p[1] * p[1] + p[2] * p[2];
                    if (d < dn) { dn = d; near = s; }
                }
            }
    if (near < 0) {
        if (!FILL) counts[cell] = 0;
        return;
    }
    const float4 pj = __ldg(pts + near);
    const float j[3] = {(float)((double)pj.x - c[0]), (float)((double)pj.y - c[1]), (float)((double)pj.z - c[2])};
    const float jj = j[0] * j[0] + j[1] * j[1] + j[2] * j[2], dj = sqrtf(jj);
    const float reach = kListMargin * (dj + diag) * (dj + diag);
    // a listed node is nearer than j0 somewhere in the cell: within dj + 2 diag
    const float r = (dj + 2.0f * diag) * 1.001f;
    int lo[3], hi[3];
    for (int a = 0; a < 3; ++a) {
        const float w = r * F.inv_cell[a] + 1e-2f;
        lo[a] = cell_of(c[a], -w, a);
        hi[a] = cell_of(c[a], w, a);
    }
    bool fits = (int64_t)(hi[1] - lo[1] + 1) * (hi[2] - lo[2] + 1) <= kListRows;
    int visits = 0;
    const uint32_t out = FILL ? start[cell] : 0u, room = FILL ? start[cell + 1] - out : 0u;
    if (FILL && room == 0) return;
    uint32_t n = 0;
    for (int z = lo[2]; z <= hi[2] && fits; ++z)
        for (int y = lo[1]; y <= hi[1] && fits; ++y) {
            const int row = (z * F.cells[1] + y) * F.cells[0];
            const int b = __ldg(F.cell_start + row + lo[0]), en = __ldg(F.cell_start + row + hi[0] + 1);
            visits += en - b;
            fits = visits <= kListVisits;
            for (int s = b; s < en && fits; ++s) {
                const float4 q = __ldg(pts + s);
                const float p[3] = {(float)((double)q.x - c[0]), (float)((double)q.y - c[1]),
                                    (float)((double)q.z - c[2])};
                const float pp = p[0] * p[0] + p[1] * p[1] + p[2] * p[2];
                const float low = pp - jj - 2.0f * (h[0] * fabsf(j[0] - p[0]) + h[1] * fabsf(j[1] - p[1]) +
                                                    h[2] * fabsf(j[2] - p[2]));
                // the sums' own rounding: a few 2^-24 of their terms
                if (s != near && low > reach + 1e-6f * (pp + jj)) continue;
                if (FILL && n < room) {
                    const int id = __ldg(F.point_ids + s);
                    uint32_t k = n;  // insertion by id
                    for (; k > 0; --k) {
                        const float4 o = rec[out + k - 1];
                        if (__float_as_int(o.w) < id) break;
                        rec[out + k] = o;
                    }
                    rec[out + k] = make_float4(q.x, q.y, q.z, __int_as_float(id));
                }
                ++n;
                fits = n <= kListMost;
            }
        }
    if (!FILL) counts[cell] = fits ? n : 0;
}

static int check_lists(const jt_nearest_field* f, const NearestLists& g) {
    if (f->n_points < 1 || f->points == nullptr || f->point_ids == nullptr || f->cell_start == nullptr)
        return set_error(JT_ERR_INVALID, "nearest field needs points and a cell list");
    if (g.cells < 1) return set_error(JT_ERR_UNSUPPORTED, "this nearest field gets no candidate lists");
    return JT_OK;
}

}  // namespace jt

using namespace jt;

extern "C" int64_t jt_nearest_lists_cells(const jt_nearest_field* f) {
    return f == nullptr ? 0 : nearest_lists(*f).cells;
}

extern "C" int jt_nearest_lists_count(const jt_nearest_field* f, uint32_t* start, int64_t* total, void* stream) {
    if (f == nullptr || start == nullptr || total == nullptr)
        return set_error(JT_ERR_INVALID, "field, start and total are required");
    const NearestLists g = nearest_lists(*f);
    if (int rc = check_lists(f, g)) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    uint32_t* sums = nullptr;
    const int64_t n = g.cells + 1, p1 = scan_partials(n), p2 = scan_partials2(n);
    cudaError_t e = dev_alloc((void**)&sums, (size_t)(p1 + p2) * 4, s);
    if (e != cudaSuccess) return cuda_status(e, "candidate list scan scratch");
    e = cudaMemsetAsync(start + g.cells, 0, 4, s);
    if (e == cudaSuccess) {
        k_nearest_lists<0><<<grid_blocks(g.cells), kBlock, 0, s>>>(*f, g, start, nullptr, nullptr);
        e = cudaGetLastError();
    }
    int rc = e == cudaSuccess ? exclusive_scan_u32(start, n, sums, sums + p1, s) : JT_OK;
    uint32_t last = 0;
    if (e == cudaSuccess && rc == JT_OK) e = cudaMemcpyAsync(&last, start + g.cells, 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess && rc == JT_OK) e = cudaStreamSynchronize(s);
    dev_free(sums, s);
    if (e != cudaSuccess) return cuda_status(e, "candidate list count");
    *total = last;
    return rc;
}

extern "C" size_t jt_nearest_lists_bytes(const jt_nearest_field* f, int64_t total) {
    if (f == nullptr || total < 0) return 0;
    const NearestLists g = nearest_lists(*f);
    return g.cells > 0 ? g.rec + (size_t)total * 16 : 0;
}

extern "C" int jt_nearest_lists_fill(const jt_nearest_field* f, const uint32_t* start, void* stream) {
    if (f == nullptr || start == nullptr) return set_error(JT_ERR_INVALID, "field and start are required");
    const NearestLists g = nearest_lists(*f);
    if (int rc = check_lists(f, g)) return rc;
    if (((uintptr_t)f->points & 63u) != 0)
        return set_error(JT_ERR_INVALID, "candidate lists need points on a 64-byte boundary");
    cudaStream_t s = (cudaStream_t)stream;
    char* base = reinterpret_cast<char*>(const_cast<float*>(f->points));
    const cudaError_t e = cudaMemcpyAsync(base + g.start, start, (size_t)(g.cells + 1) * 4, cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return cuda_status(e, "candidate list offsets");
    k_nearest_lists<1><<<grid_blocks(g.cells), kBlock, 0, s>>>(*f, g, nullptr, start,
                                                              reinterpret_cast<float4*>(base + g.rec));
    return cuda_status(cudaGetLastError(), "candidate list fill");
}

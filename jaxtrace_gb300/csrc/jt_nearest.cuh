// Scattered-node field: nearest-node sampling of TimeSeriesField
// (fields/time_series.py:249-259 and :391-412).  The reference takes the
// argmin over all nodes of the float32 squared distance, the lowest index on
// ties.  Here a query reads the candidate list of its cell (jt_nearest_lists_fill);
// outside the lists' grid, and for fields without lists, a uniform cell list
// limits the search to rings of cells around the query, and the ring loop stops
// once no unvisited cell can hold a point at or below the best squared distance.
#pragma once

#include "jt_common.cuh"

namespace jt {

// Nodes [b, en) of the sorted node array against the best so far: argmin of
// the float32 squared distance, lowest id on ties.  The id is read only for
// a distance at or below the best (a new best or a tie).
template <bool EXACT>
__device__ __forceinline__ void nearest_scan(const jt_nearest_field& F, const V3& q, int b, int en, float& best,
                                             int& best_id) {
    typedef Ar<EXACT> A;
    for (int s = b; s < en; ++s) {
        const float4 p = __ldg(reinterpret_cast<const float4*>(F.points) + s);
        const float ddx = A::sub(q.x, p.x), ddy = A::sub(q.y, p.y), ddz = A::sub(q.z, p.z);
        const float d = A::add(A::add(A::mul(ddx, ddx), A::mul(ddy, ddy)), A::mul(ddz, ddz));
        if (d <= best) {
            const int id = __ldg(F.point_ids + s);
            if (d < best || id < best_id) { best = d; best_id = id; }
        }
    }
}

// Lower bound of the distance from the query to a neighbouring row of cells
// along one axis, in cell units: 0 for its own row, else the gap from its
// continuous cell coordinate f to the shared cell face, less 1e-3 of a cell
// for the float32 rounding of f and of the nodes' own cell coordinates.
__device__ __forceinline__ float row_gap(int d, float frac) {
    const float g = d < 0 ? frac : (d > 0 ? 1.0f - frac : 0.0f);
    return fmaxf(g - 1e-3f, 0.0f);
}

// Index of the node nearest to q (argmin of the float32 squared distance,
// lowest index on ties; 0 for a NaN query, whose distances are all NaN).
// h_min: the smallest cell edge, scaled down slightly (ring-stop bound).
// Cells are walked in rows along x: a row's cells are consecutive in the
// cell list, so their nodes are one range of the sorted node array.  In the
// first ring a row whose gap from the query already exceeds the best
// distance (with a 1e-4 relative margin) is skipped; no node in it can reach
// the best or tie with it.
template <bool EXACT>
__device__ __forceinline__ int nearest_id(const jt_nearest_field& F, float h_min, const V3& q) {
    if (q.x != q.x || q.y != q.y || q.z != q.z) return 0;
    const float qq[3] = {q.x, q.y, q.z};
    int c[3];
    float frac[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float fc = (qq[a] - F.origin[a]) * F.inv_cell[a];
        const float f = floorf(fc);
        int ci = (f != f) ? 0 : (f < 0.0f ? 0 : (f >= (float)F.cells[a] ? F.cells[a] - 1 : (int)f));
        c[a] = ci;
        // the query's position inside its cell (clamped cells: the nearer face)
        frac[a] = fminf(fmaxf(fc - (float)ci, 0.0f), 1.0f);
    }
    const int nx = F.cells[0], ny = F.cells[1], nz = F.cells[2];
    const float hy = 1.0f / F.inv_cell[1], hz = 1.0f / F.inv_cell[2];
    float best = __int_as_float(0x7f800000);
    int best_id = 0x7fffffff;
    const int rmax = max(nx, max(ny, nz));
    for (int r = 0; r <= rmax; ++r) {
        if (r >= 2) {
            const float lb = (float)(r - 1) * h_min;
            if (lb * lb > best * 1.00001f) break;
        }
        for (int dz = -r; dz <= r; ++dz) {
            const int cz = c[2] + dz;
            if (cz < 0 || cz >= nz) continue;
            for (int dy = -r; dy <= r; ++dy) {
                const int cy = c[1] + dy;
                if (cy < 0 || cy >= ny) continue;
                if (r == 1 && (dy != 0 || dz != 0) && F.inv_cell[1] > 0.0f && F.inv_cell[2] > 0.0f) {
                    const float gy = row_gap(dy, frac[1]) * hy, gz = row_gap(dz, frac[2]) * hz;
                    if ((gy * gy + gz * gz) * 0.9999f > best) continue;
                }
                const int row = (cz * ny + cy) * nx;
                const bool face = (dz == -r || dz == r || dy == -r || dy == r);
                if (face) {  // the whole row [c - r, c + r] as one node range
                    const int x0 = max(c[0] - r, 0), x1 = min(c[0] + r, nx - 1);
                    nearest_scan<EXACT>(F, q, __ldg(F.cell_start + row + x0), __ldg(F.cell_start + row + x1 + 1),
                                        best, best_id);
                } else {     // the two end cells of an inner row
                    if (c[0] - r >= 0) {
                        const int cell = row + c[0] - r;
                        nearest_scan<EXACT>(F, q, __ldg(F.cell_start + cell), __ldg(F.cell_start + cell + 1),
                                            best, best_id);
                    }
                    if (c[0] + r < nx) {
                        const int cell = row + c[0] + r;
                        nearest_scan<EXACT>(F, q, __ldg(F.cell_start + cell), __ldg(F.cell_start + cell + 1),
                                            best, best_id);
                    }
                }
            }
        }
    }
    return best_id == 0x7fffffff ? 0 : best_id;
}

// ---------------------------------------------------------------------------
// Candidate lists: behind the sorted nodes, 64-byte aligned, the lists' offsets
// (cells + 1) and then {x, y, z, id} records, ascending ids per list.
// ---------------------------------------------------------------------------
struct NearestLists {
    float org[3], inv[3];  // grid of the lists; a flat axis has one cell
    int n[3];
    size_t start, rec;     // offsets from points
    int64_t cells;         // 0: no lists
};

__host__ inline NearestLists nearest_lists(const jt_nearest_field& F) {
    NearestLists g{};
    float widest = 0.0f;  // the rim of a flat axis is that of the widest live one
    for (int a = 0; a < 3; ++a)
        if (F.cells[a] > 1 && F.inv_cell[a] > 0.0f) widest = fmaxf(widest, 0.5f / F.inv_cell[a]);
    // the margin of the lists, 1e-5 of a squared distance of that size, has to lie
    // far above the rounding of squares next to float32's smallest (2^-150)
    if (!(widest >= 1e-15f) || !isfinite(widest)) return g;
    int64_t cells = 1;
    for (int a = 0; a < 3; ++a) {
        if (F.inv_cell[a] > 0.0f) {
            g.n[a] = 2 * F.cells[a] + 2 * JT_NEAREST_RIM;
            g.inv[a] = 2.0f * F.inv_cell[a];
            g.org[a] = F.origin[a] - (float)JT_NEAREST_RIM / g.inv[a];
        } else {
            g.n[a] = 1;
            g.inv[a] = 0.5f / ((float)JT_NEAREST_RIM * widest);
            g.org[a] = F.origin[a] - (float)JT_NEAREST_RIM * widest;
        }
        if (!isfinite(g.inv[a]) || !isfinite(g.org[a]) || F.cells[a] > 4096) return g;
        cells *= g.n[a];
    }
    auto al = [](size_t b) { return (b + 63) & ~(size_t)63; };
    g.start = al((size_t)F.n_points * 16);
    if (cells > (int64_t)1 << 26) return g;
    g.cells = cells;
    g.rec = al(g.start + (size_t)(cells + 1) * 4);
    return g;
}

// Cell of q in the lists' grid, -1 outside it and for NaN.
__device__ __forceinline__ int nearest_list_cell(const NearestLists& g, const V3& q) {
    const float fx = (q.x - g.org[0]) * g.inv[0], fy = (q.y - g.org[1]) * g.inv[1], fz = (q.z - g.org[2]) * g.inv[2];
    if (!(fx >= 0.0f && fy >= 0.0f && fz >= 0.0f && fx < (float)g.n[0] && fy < (float)g.n[1] && fz < (float)g.n[2]))
        return -1;
    return ((int)fz * g.n[1] + (int)fy) * g.n[0] + (int)fx;
}

// nearest_id through the candidate lists; 0x7fffffff where they have no answer
// (no lists, a query outside their grid, a cell without a list).  One loop of a few
// contiguous 16-byte records per lane: the rings visit about 27 cells in rows
// of their own lengths (54 nodes), a ball around a first guess fewer but with
// per-lane trip counts in three nested loops, which left 5 of 32 lanes active
// and was slower than the rings.  200,003 particles x 50 RK4 steps over 35,937
// nodes: 9.3 -> 1.6 ms, 460 warp instructions per evaluation of a warp, 20 of
// 32 lanes active, bound by the L1 (79 %) on particles in no particular order.
template <bool EXACT>
__device__ __forceinline__ int nearest_listed(const jt_nearest_field& F, const NearestLists& g, const V3& q) {
    typedef Ar<EXACT> A;
    const int c = g.cells > 0 ? nearest_list_cell(g, q) : -1;
    if (c < 0) return 0x7fffffff;
    const char* base = reinterpret_cast<const char*>(F.points);
    const uint32_t* st = reinterpret_cast<const uint32_t*>(base + g.start) + c;
    const uint32_t b = __ldg(st), en = __ldg(st + 1);
    const float4* rec = reinterpret_cast<const float4*>(base + g.rec);
    float best = __int_as_float(0x7f800000);
    int id = 0x7fffffff;
    for (uint32_t s = b; s < en; ++s) {
        const float4 p = __ldg(rec + s);
        const float dx = A::sub(q.x, p.x), dy = A::sub(q.y, p.y), dz = A::sub(q.z, p.z);
        const float d = A::add(A::add(A::mul(dx, dx), A::mul(dy, dy)), A::mul(dz, dz));
        if (d < best) {  // ascending ids: the first of a tie stays
            best = d;
            id = __float_as_int(p.w);
        }
    }
    return id;
}

template <bool EXACT, int STORE>
struct NearestField {
    jt_nearest_field F;
    float h_min;  // smallest cell edge
    NearestLists lists;

    static NearestField create(const jt_nearest_field& d, float h) {
        NearestField f{d, h, NearestLists{}};
        if (d.storage & JT_NEAREST_LISTS) f.lists = nearest_lists(d);
        return f;
    }

    __device__ __forceinline__ V3 operator()(const V3& q, const jt_blend& e, int& flags) const {
        const int64_t base = (int64_t)min(max(e.pair, 0), F.n_pairs - 1) * F.pair_stride;
        int id = nearest_listed<EXACT>(F, lists, q);
        if (id == 0x7fffffff) id = nearest_id<EXACT>(F, h_min, q);
        return blend<EXACT, STORE>(load_pair<STORE>(F.pairs, base + id), e);
    }
};

}  // namespace jt

// Tetrahedral-mesh field with the hash-grid point location of
// FEMTimeSeriesField (fields/fem_time_series.py:16-110) and
// interpolate_in_mesh (fields/fem_interpolator.py:210-328): the query's cell
// of a uniform grid over the node bounding box, that cell's elements in
// ascending order, the first whose box and barycentric test hold the query
// gives P1; with none, the value of the nearest node of the whole mesh.  The
// time blend is the float32 one of TimeSeriesField's JAX path
// (fem_time_series.py:104).
#pragma once

#include "jt_mesh.cuh"
#include "jt_nearest.cuh"

namespace jt {

// 4 blocks of 256 (64 registers, some spills) against 3 (80): 8.0 and 8.5 ms for
// 1M particles x 32 steps on 1,572,864 tetrahedra
#ifndef JT_FEM_MIN_BLOCKS
#define JT_FEM_MIN_BLOCKS 4
#endif

// NEAR as in MeshFieldT
template <bool EXACT, int STORE, bool NEAR = false>
struct FemFieldT {
    static constexpr int kMinBlocks = JT_FEM_MIN_BLOCKS;
    static constexpr bool kHinted = true;
    jt_fem_field F;
    float h_min;  // smallest nearest-node cell edge (ring-stop bound)
    NearestLists lists;
    const char* filters;  // filter records by tetrahedron (jt_mesh.cuh), or NULL
    float mesh_hi[3];     // above the node bounding box's maximum

    static FemFieldT create(const jt_fem_field& d, float h) {
        FemFieldT f{d, h, NearestLists{}, nullptr, {0.0f, 0.0f, 0.0f}};
        if (d.nearest.storage & JT_NEAREST_LISTS) f.lists = nearest_lists(d.nearest);
        if (d.sub_div & JT_FEM_FILTERS) f.filters = reinterpret_cast<const char*>(d.tet_geom) + (int64_t)d.n_tets * 64;
        f.F.sub_div = d.sub_div & ~JT_FEM_FILTERS;
        for (int a = 0; a < 3; ++a) {
            const double w = (double)d.grid_size[a] * (double)d.cell_size[a];
            f.mesh_hi[a] = (float)((double)d.grid_min[a] + w + 1e-5 * w + 1e-6 * fabs((double)d.grid_min[a]));
        }
        return f;
    }

    __device__ __forceinline__ V3 node_value(int node, const jt_blend& e) const {
        const int64_t base = (int64_t)min(max(e.pair, 0), F.nearest.n_pairs - 1) * F.nearest.pair_stride;
        return blend<EXACT, STORE>(load_pair<STORE>(F.nearest.pairs, base + node), e);
    }

    // floor((q - grid_min) / cell_size).astype(int32) clipped to [0, n-1]
    // (fem_interpolator.py:262-263); the float clamp before the conversion
    // is XLA's saturating float->int (NaN lands on 0).
    __device__ __forceinline__ int cell_coord(float q, float lo, float cs, int n) const {
        typedef Ar<EXACT> A;
        const float f = floorf(A::div(A::sub(q, lo), cs));
        return (int)fminf(fmaxf(f, 0.0f), (float)(n - 1));
    }

    // sub-cell of coordinate q inside hash cell c: floor((q - (lo + c*cs)) /
    // (cs/S)) clipped to [0, S-1]; the host lists widen the sub-cells enough
    // to absorb the rounding of this float32 arithmetic
    __device__ __forceinline__ int sub_coord(float q, float lo, float cs, int c, int S) const {
        const float cell_lo = lo + (float)c * cs;
        const float f = floorf((q - cell_lo) * ((float)S / cs));
        return (int)fminf(fmaxf(f, 0.0f), (float)(S - 1));
    }

    // The query's candidates: entries [b0, b1) of the list returned.
    __device__ __forceinline__ const int32_t* candidates(const V3& q, int& b0, int& b1) const {
        const int cx = cell_coord(q.x, F.grid_min[0], F.cell_size[0], F.grid_size[0]);
        const int cy = cell_coord(q.y, F.grid_min[1], F.cell_size[1], F.grid_size[1]);
        const int cz = cell_coord(q.z, F.grid_min[2], F.cell_size[2], F.grid_size[2]);
        const int cell = (cx * F.grid_size[1] + cy) * F.grid_size[2] + cz;
        if (F.sub_div > 0) {
            // the query's sub-cell, clamped into its hash cell
            const int S = F.sub_div;
            const int sx = sub_coord(q.x, F.grid_min[0], F.cell_size[0], cx, S);
            const int sy = sub_coord(q.y, F.grid_min[1], F.cell_size[1], cy, S);
            const int sz = sub_coord(q.z, F.grid_min[2], F.cell_size[2], cz, S);
            const int64_t sc = (int64_t)cell * (S * S * S) + (sx * S + sy) * S + sz;
            b0 = __ldg(F.sub_start + sc);
            b1 = __ldg(F.sub_start + sc + 1);
            return F.sub_elems;
        }
        b0 = __ldg(F.cell_start + cell);
        b1 = __ldg(F.cell_start + cell + 1);
        return F.cell_elems;
    }

    // First candidate that holds the query (lax.scan keeps the first hit,
    // :280-305), through the filter records: as MeshFieldT::find_slot, with
    // the hint a tetrahedron, found without any list.  A query outside the
    // node bounding box lies in no element's box, so its list is left out.
    // The scan was the field's cost: 12.6 candidates a list, each a box and
    // often four determinants, and 8 lanes of 32 active.  1M particles x 32 steps on
    // 1,572,864 tetrahedra: 18.5 ms without filters, 15.2 ms with them, 8.0 ms
    // with the lists pruned to the 4.3 that can hold a query of the sub-cell.
    __device__ __forceinline__ bool find_filtered(const V3& q, int& hint, float4& b, int4& cn) const {
        uint32_t w[8];
        float slack;
        int s = 0, end = 0, first = 0, t = hint;
        const int32_t* list = nullptr;
        bool certain = false;
        if (hint >= 0) {
            ldg256(filters + (int64_t)hint * 32, w);
            certain = filter_bary(q, w, slack) >= slack + kInside;
        }
        if (!certain) {
            hint = -1;
            if (q.x < F.grid_min[0] || q.y < F.grid_min[1] || q.z < F.grid_min[2] || q.x > mesh_hi[0] ||
                q.y > mesh_hi[1] || q.z > mesh_hi[2])
                return false;
            list = candidates(q, s, end);
            first = end;
            int tn = 0;
            if (s < end) {
                t = __ldg(list + s);
                tn = __ldg(list + min(s + 1, end - 1));
                ldg256(filters + (int64_t)t * 32, w);
            }
            while (s < end) {
                // the next record and the id after it are on their way while this one is judged
                uint32_t nx[8];
                ldg256(filters + (int64_t)tn * 32, nx);
                const int tnn = __ldg(list + min(s + 2, end - 1));
                const float m = filter_bary(q, w, slack);
                if (m >= -slack) {
                    if (first == end) first = s;
                    if ((filter_flags(w) & JT_TET_ALONE) && m >= slack + kInside) {
                        certain = true;
                        hint = t;
                        break;
                    }
                }
                ++s;
                t = tn;
                tn = tnn;
#pragma unroll
                for (int k = 0; k < 8; ++k) w[k] = nx[k];
            }
        }
        for (s = first; certain || s < end; ++s) {
            if (!certain) {
                t = __ldg(list + s);
                if (s != first) {
                    ldg256(filters + (int64_t)t * 32, w);
                    if (filter_bary(q, w, slack) < -slack) continue;
                }
            }
            const float* rec = F.tet_geom + 16 * (int64_t)t;
            uint32_t g0[8], g1[8];
            ldg256(rec, g0);
            ldg256(rec + 8, g1);
            if (!slot_bary<EXACT>(q, g0, g1, b)) {
                if (certain) break;
                continue;
            }
            if (!certain || (NEAR && !EXACT)) {
                const float4* bx = reinterpret_cast<const float4*>(F.tet_box) + 2 * (int64_t)t;
                const float4 mn = __ldg(bx), mx = __ldg(bx + 1);
                if (!certain && !(q.x >= mn.x && q.y >= mn.y && q.z >= mn.z && q.x <= mx.x && q.y <= mx.y && q.z <= mx.z))
                    continue;
                if (NEAR && !EXACT && mn.w != 0.0f) b = bary_f64(q, F.tet_geom, t);
            }
            cn = make_int4((int)g1[4], (int)g1[5], (int)g1[6], (int)g1[7]);
            return true;
        }
        return false;
    }

    __device__ __forceinline__ V3 operator()(const V3& q, const jt_blend& e, int& flags) const {
        int hint = -1;
        return at(q, e, flags, hint);
    }

    // hint: the tetrahedron of the thread's last certain hit, or -1
    __device__ __forceinline__ V3 at(const V3& q, const jt_blend& e, int& flags, int& hint) const {
        float4 b;
        int4 cn;
        bool found = false;
        if (filters != nullptr) {
            found = find_filtered(q, hint, b, cn);
        } else {
            int s, b1;
            const int32_t* list = candidates(q, s, b1);
            for (; s < b1 && !found; ++s) {
                bool near;
                const int t = __ldg(list + s);
                found = tet_bary<EXACT>(q, F.tet_box, F.tet_geom, t, b, cn, near);
                if (NEAR && !EXACT && found && near) b = bary_f64(q, F.tet_geom, t);
            }
        }
        if (found)
            return p1_combine<EXACT>(b, node_value(cn.x, e), node_value(cn.y, e), node_value(cn.z, e),
                                     node_value(cn.w, e));
        // global nearest node (:311-316)
        flags |= JT_STATUS_OCTREE_FALLBACK;
        int id = nearest_listed<EXACT>(F.nearest, lists, q);
        if (id == 0x7fffffff) id = nearest_id<EXACT>(F.nearest, h_min, q);
        return node_value(id, e);
    }
};

template <bool EXACT, int STORE>
using FemField = FemFieldT<EXACT, STORE, false>;
template <bool EXACT, int STORE>
using FemFieldNear = FemFieldT<EXACT, STORE, true>;

}  // namespace jt

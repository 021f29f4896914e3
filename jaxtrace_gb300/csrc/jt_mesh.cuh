// Tetrahedral-mesh field: octree point location and P1 interpolation with
// the semantics of fields/octree_fem_interpolator_optimized.py:253-380 and
// the float32 time blend of fields/time_series.py:175-184 (JAX path, which
// that field always uses: octree_fem_time_series_optimized.py:108).
#pragma once

#include "jt_common.cuh"

namespace jt {

// 3x3 determinant of the matrix whose COLUMNS are c0, c1, c2, expanded as
// JAX evaluates jnp.linalg.det for 3x3 inputs (six triple products summed
// left to right).  Used by point_in_tetrahedron_fast (…optimized.py:231-242).
template <bool EXACT>
__device__ __forceinline__ float det3(const V3& c0, const V3& c1, const V3& c2) {
    typedef Ar<EXACT> A;
    const float a00 = c0.x, a01 = c1.x, a02 = c2.x;
    const float a10 = c0.y, a11 = c1.y, a12 = c2.y;
    const float a20 = c0.z, a21 = c1.z, a22 = c2.z;
    const float t1 = A::mul(A::mul(a00, a11), a22);
    const float t2 = A::mul(A::mul(a01, a12), a20);
    const float t3 = A::mul(A::mul(a02, a10), a21);
    const float t4 = A::mul(A::mul(a02, a11), a20);
    const float t5 = A::mul(A::mul(a00, a12), a21);
    const float t6 = A::mul(A::mul(a01, a10), a22);
    return A::sub(A::sub(A::sub(A::add(A::add(t1, t2), t3), t4), t5), t6);
}

// float64 determinant of three float32 columns (same expansion as det3)
__device__ __forceinline__ double det3_f64(double a00, double a10, double a20, double a01, double a11, double a21,
                                           double a02, double a12, double a22) {
    return a00 * a11 * a22 + a01 * a12 * a20 + a02 * a10 * a21 - a02 * a11 * a20 - a00 * a12 * a21 -
           a01 * a10 * a22;
}

// Near-degenerate tetrahedra: |det| below this fraction of
// |v1-v0| |v2-v0| |v3-v0| (about 0.7 for a regular tetrahedron) loses float32
// digits in cancellation.  jt_mark_near_degenerate flags them in the pad slot
// after the box minimum (tet_box[8t+3] = 1); in the compensated arithmetic the
// float32 solve still decides which tetrahedron holds the query (the
// reference's decision) and the weights of a flagged one are solved again in
// float64.
constexpr float kNearDegenerate = 1e-2f;

__device__ __forceinline__ bool near_degenerate(const float* g12) {
    const V3 v01{g12[3], g12[4], g12[5]}, v02{g12[6], g12[7], g12[8]}, v03{g12[9], g12[10], g12[11]};
    const float det = det3<true>(v01, v02, v03);
    const float l1 = __fadd_rn(__fadd_rn(__fmul_rn(v01.x, v01.x), __fmul_rn(v01.y, v01.y)), __fmul_rn(v01.z, v01.z));
    const float l2 = __fadd_rn(__fadd_rn(__fmul_rn(v02.x, v02.x), __fmul_rn(v02.y, v02.y)), __fmul_rn(v02.z, v02.z));
    const float l3 = __fadd_rn(__fadd_rn(__fmul_rn(v03.x, v03.x), __fmul_rn(v03.y, v03.y)), __fmul_rn(v03.z, v03.z));
    return __fmul_rn(det, det) < __fmul_rn(kNearDegenerate * kNearDegenerate, __fmul_rn(__fmul_rn(l1, l2), l3));
}

// Barycentrics (b1, b2, b3 in y, z, w; b0 in x) of tetrahedron t in float64
// from its stored float32 geometry, rounded once to float32; |det| < 1e-10
// gives det = 1 as in the float32 solve.
static __device__ __noinline__ float4 bary_f64(const V3 q, const float* tet_geom, int t) {
    const float4* g = reinterpret_cast<const float4*>(tet_geom) + 4 * (int64_t)t;
    const float4 g0 = __ldg(g), g1 = __ldg(g + 1), g2 = __ldg(g + 2);
    const V3 v0{g0.x, g0.y, g0.z};
    const V3 a{g0.w, g1.x, g1.y}, b{g1.z, g1.w, g2.x}, c{g2.y, g2.z, g2.w};
    const double px = (double)q.x - (double)v0.x, py = (double)q.y - (double)v0.y, pz = (double)q.z - (double)v0.z;
    double det = det3_f64(a.x, a.y, a.z, b.x, b.y, b.z, c.x, c.y, c.z);
    if (fabs(det) < 1e-10) det = 1.0;
    const double y = det3_f64(px, py, pz, b.x, b.y, b.z, c.x, c.y, c.z) / det;
    const double z = det3_f64(a.x, a.y, a.z, px, py, pz, c.x, c.y, c.z) / det;
    const double w = det3_f64(a.x, a.y, a.z, b.x, b.y, b.z, px, py, pz) / det;
    return make_float4((float)(1.0 - y - z - w), (float)y, (float)z, (float)w);
}

// Barycentric test of tetrahedron t (point_in_tetrahedron_fast,
// …optimized.py:218-250, and point_in_tetrahedron, fem_interpolator.py:146-207,
// which compute the same thing): true when the query's box test and the
// tolerance test pass; b receives (b0, b1, b2, b3) as (x, y, z, w) and cn
// the vertex ids.
template <bool EXACT>
__device__ __forceinline__ bool tet_bary(const V3& q, const float* tet_box, const float* tet_geom, int t,
                                         float4& b, int4& cn, bool& near) {
    typedef Ar<EXACT> A;
    const float4* bx = reinterpret_cast<const float4*>(tet_box) + 2 * (int64_t)t;
    const float4 mn = __ldg(bx), mx = __ldg(bx + 1);
    if (!(q.x >= mn.x && q.y >= mn.y && q.z >= mn.z && q.x <= mx.x && q.y <= mx.y && q.z <= mx.z)) return false;
    const float4* g = reinterpret_cast<const float4*>(tet_geom) + 4 * (int64_t)t;
    const float4 g0 = __ldg(g), g1 = __ldg(g + 1), g2 = __ldg(g + 2);
    const V3 v0{g0.x, g0.y, g0.z};
    const V3 v01{g0.w, g1.x, g1.y}, v02{g1.z, g1.w, g2.x}, v03{g2.y, g2.z, g2.w};
    const V3 v0p{A::sub(q.x, v0.x), A::sub(q.y, v0.y), A::sub(q.z, v0.z)};
    float det = det3<EXACT>(v01, v02, v03);
    near = !EXACT && mn.w != 0.0f;
    if (fabsf(det) < 1e-10f) det = 1.0f;
    b.y = A::div(det3<EXACT>(v0p, v02, v03), det);
    b.z = A::div(det3<EXACT>(v01, v0p, v03), det);
    b.w = A::div(det3<EXACT>(v01, v02, v0p), det);
    b.x = A::sub(A::sub(A::sub(1.0f, b.y), b.z), b.w);
    const float lo = -1e-6f, hi = 0.999999f;  // tol and 1 + tol as float32
    if (!(b.x >= lo && b.y >= lo && b.z >= lo && b.w >= lo && b.x <= hi && b.y <= hi && b.z <= hi && b.w <= hi))
        return false;
    cn = __ldg(reinterpret_cast<const int4*>(g + 3));
    return true;
}

// ---------------------------------------------------------------------------
// Locator block (jt_mesh_locator_build), behind the dtab rows:
//   header  8 floats: origin xyz, cells per unit xyz, 0, mismatch flag (build)
//   faces   per axis 2^D {lower, upper} faces of its cells, the outer ones
//           NaN (nothing is below or above them)
//   table   8^D {elem_offset, elem_count} of the node that D moves reach, or
//           {breadth-first node, -1} where the descent goes on below it
//   slots   64 B per element-list slot: the tetrahedron's tet_geom record
//   filters 32 B per element-list slot: the tetrahedron's filter record
// All offsets are multiples of 64 B from the 64-aligned end of dtab's rows.
//
// Why: the evaluation was held by the L1 (93 % busy) on 34 gathers per query,
// seven of them the levels of the descent and six per candidate (list entry,
// two halves of the box, three quarters of the geometry).  The table takes the
// descent to four independent loads and one dependent one, and the slot order
// the candidate to two 256-bit loads of one line.  1M particles x 64 steps on
// 1,572,864 tetrahedra (64^3 hexahedra): tracking kernel 15.6 -> 12.8 ms;
// 24 ensembles x 50 steps 7.1 -> 5.6 ms; same bits.
// ---------------------------------------------------------------------------
constexpr int32_t kLocatorMagic = 0x4a544c00;  // jt_mesh_field.locator = magic | depth

struct LocatorLayout {
    size_t header, faces, table, slots, filters, bytes;
};

__host__ __device__ inline LocatorLayout locator_layout(int64_t n_nodes, int64_t n_entries, int depth) {
    auto al = [](size_t b) { return (b + 63) & ~(size_t)63; };
    LocatorLayout o;
    o.header = al((size_t)n_nodes * 8);
    o.faces = o.header + 64;
    o.table = al(o.faces + ((size_t)3 << depth) * 8);
    o.slots = al(o.table + ((size_t)8 << (3 * depth)));
    o.filters = o.slots + (size_t)n_entries * 64;
    o.bytes = al(o.filters + (size_t)n_entries * 32);
    return o;
}

__host__ __device__ inline int locator_depth(const jt_mesh_field& F) {
    const int d = F.locator & 0xff;
    return (F.locator & ~0xff) == kLocatorMagic && d >= 1 && d <= JT_MESH_LOCATOR_MAX_DEPTH ? d : 0;
}

// ---------------------------------------------------------------------------
// Filter records.  A candidate is judged on 32 bytes and nine FMAs instead of
// its box, its 64-byte geometry and four determinants: words 0-2 hold v0 in
// float32, words 3-7 the gradients of the barycentrics b1, b2, b3 as nine
// float16 values (x, y, z of each); the last half-word is the record's slack
// as a float16, its two low bits the JT_TET_* flags.
//
// A query is rejected where a filtered barycentric is below -slack.  That never
// loses a candidate the full test accepts: such a query lies in the
// tetrahedron's box, so rounding the gradients to float16 (2^-11 relative, 2^-25
// absolute) changes no barycentric by more than 2^-11 times the spread, the sum
// over b1, b2, b3 and the axes of the box's extent times the gradient (and the
// absolute part), and the full test's own float32 barycentrics are off by at
// most kShapeError times the shape ratio; slack is above the two together.
// Where slack would exceed kSlackMost, or the tetrahedron is not well shaped,
// the gradients are zero: nothing is rejected.
//
// A tetrahedron is well shaped when its shape ratio, the cube of its longest
// edge over |det|, is at most kWellShaped: each numerator of the solve is six
// triple products of components no longer than that edge, three roundings each
// and five in the sum, in all less than 64 * 2^-24 times the ratio of the
// determinant.  A query whose computed barycentrics are all at least kInside
// then lies inside it, kInsideTrue of its box's extent or more away from each
// face of the box, and the box test, whose faces are the vertices' own floats,
// cannot fail.
//
// JT_TET_ALONE: well shaped, and no tetrahedron before this one in the list
// accepts a query whose computed barycentrics here are all at least kInside
// (checked at build by tets_apart).  Then this tetrahedron is the first hit of
// every such query, whatever the order they are tried in; one whose filtered
// barycentrics are all at least slack + kInside is such a query.
// ---------------------------------------------------------------------------
constexpr float kWellShaped = 128.0f;
constexpr float kShapeError = 64.0f / 16777216.0f;
constexpr float kInside = 1e-3f;
constexpr float kInsideTrue = kInside - kWellShaped * kShapeError;
constexpr float kSlackMost = 0.05f;
enum { JT_TET_SHAPED = 1, JT_TET_ALONE = 2 };

// Longest edge cubed over |det| of a geometry record; above kWellShaped for a
// tetrahedron that is not well shaped (a |det| the solve replaces by 1 included).
__device__ __forceinline__ float shape_ratio(const float* g12, float* longest = nullptr) {
    const V3 a{g12[3], g12[4], g12[5]}, b{g12[6], g12[7], g12[8]}, c{g12[9], g12[10], g12[11]};
    const float det = fabsf(det3<true>(a, b, c));
    auto len2 = [](float x, float y, float z) { return x * x + y * y + z * z; };
    const float l = sqrtf(fmaxf(fmaxf(fmaxf(len2(a.x, a.y, a.z), len2(b.x, b.y, b.z)), len2(c.x, c.y, c.z)),
                                fmaxf(fmaxf(len2(a.x - b.x, a.y - b.y, a.z - b.z), len2(a.x - c.x, a.y - c.y, a.z - c.z)),
                                      len2(b.x - c.x, b.y - c.y, b.z - c.z))));
    const float r = l * l * l / det;
    if (longest != nullptr) *longest = l;
    return det >= 1e-10f && r <= kWellShaped ? r : 2.0f * kWellShaped;
}

// Gradients of b1, b2, b3 (the rows of the inverse edge matrix).
template <class T>
__device__ __forceinline__ void bary_gradients(const float* g12, T (&g)[3][3]) {
    const T a[3] = {g12[3], g12[4], g12[5]}, b[3] = {g12[6], g12[7], g12[8]}, c[3] = {g12[9], g12[10], g12[11]};
    auto cross = [](const T (&u)[3], const T (&v)[3], T (&o)[3]) {
        o[0] = u[1] * v[2] - u[2] * v[1];
        o[1] = u[2] * v[0] - u[0] * v[2];
        o[2] = u[0] * v[1] - u[1] * v[0];
    };
    cross(b, c, g[0]);
    cross(c, a, g[1]);
    cross(a, b, g[2]);
    const T det = a[0] * g[0][0] + a[1] * g[0][1] + a[2] * g[0][2];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k) g[i][k] = g[i][k] / det;
}

// Smallest filtered barycentric of q, and the record's slack.
__device__ __forceinline__ float filter_bary(const V3& q, const uint32_t (&w)[8], float& slack) {
    const auto h2 = [&w](int i) { return __half22float2(*reinterpret_cast<const __half2*>(&w[i])); };
    const float px = q.x - __uint_as_float(w[0]), py = q.y - __uint_as_float(w[1]), pz = q.z - __uint_as_float(w[2]);
    const float2 a = h2(3), b = h2(4), c = h2(5), d = h2(6), e = h2(7);
    const float b1 = fmaf(px, a.x, fmaf(py, a.y, pz * b.x));
    const float b2 = fmaf(px, b.y, fmaf(py, c.x, pz * c.y));
    const float b3 = fmaf(px, d.x, fmaf(py, d.y, pz * e.x));
    slack = e.y;
    // NaN for a NaN query, which `>= -slack` rejects, as the full test would; a single
    // NaN, from a query at infinity, is passed over: the full test decides
    return fminf(fminf(1.0f - (b1 + b2 + b3), b1), fminf(b2, b3));
}

__device__ __forceinline__ uint32_t filter_flags(const uint32_t (&w)[8]) { return (w[7] >> 16) & 3u; }

// Filter record of a geometry record (g12) with the box b8.
__device__ __forceinline__ void make_filter(const float* g12, const float* b8, uint32_t flags, uint32_t (&w)[8]) {
    w[0] = __float_as_uint(g12[0]);
    w[1] = __float_as_uint(g12[1]);
    w[2] = __float_as_uint(g12[2]);
    uint32_t h[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, flags};
    if (flags & JT_TET_SHAPED) {
        double g[3][3], spread = 0.0;
        bary_gradients(g12, g);
        bool fits = true;
        for (int i = 0; i < 3; ++i)
            for (int k = 0; k < 3; ++k) {
                spread += ((double)b8[4 + k] - (double)b8[k]) * (fabs(g[i][k]) + 0x1p-14);
                fits &= fabs(g[i][k]) < 65000.0;
            }
        const double need = spread * 0x1p-11 + kShapeError * shape_ratio(g12) + 2e-5;
        if (fits && need <= kSlackMost) {
            for (int i = 0; i < 9; ++i) h[i] = __half_as_ushort(__double2half(g[i / 3][i % 3]));
            // one float16 step up and the two low bits cleared again above that
            h[9] = ((__half_as_ushort(__float2half_ru((float)need)) + 4u) & ~3u) | flags;
        }
    }
    for (int i = 0; i < 5; ++i) w[3 + i] = h[2 * i] | (h[2 * i + 1] << 16);
}

// Whether tetrahedron e (geometry ge, box be) accepts no query whose computed
// barycentrics in the well-shaped t (gt, bt) are all at least kInside: boxes
// apart (a query passes both box tests or neither answer matters), or t shrunken
// to barycentrics of kInsideTrue disjoint from e grown by what its own test is
// off (-1e-6 and kShapeError times its shape ratio).  Two disjoint tetrahedra
// are apart along a face normal of one or the cross product of an edge of each;
// neighbours that share an edge or a vertex often only along the latter: with
// the faces of e alone 14 % of a jittered hexahedral split passed.  A
// projection is off by less than 16 * 2^-24 |n|_1 P, P the largest coordinate
// beside t's v0, whichever way n itself is rounded.
__device__ __forceinline__ bool tets_apart(const float (&ge)[12], const float (&be)[8], const float (&gt)[12],
                                           const float (&bt)[8]) {
    for (int k = 0; k < 3; ++k)
        if (be[k] > bt[4 + k] || be[4 + k] < bt[k]) return true;
    const float r = shape_ratio(ge);
    if (!(r <= kWellShaped)) return false;
    const float grow = 4e-6f + r * kShapeError, m = kInsideTrue;
    V3 a[4], c[4];  // t shrunken, e grown, beside t's v0
    float far = 0.0f;
#pragma unroll
    for (int side = 0; side < 2; ++side) {
        const float* g = side ? ge : gt;
        V3* v = side ? c : a;
        const float w = side ? -grow : m;
        V3 sum{0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            v[j] = V3{g[0] - gt[0], g[1] - gt[1], g[2] - gt[2]};
            if (j > 0) v[j] = V3{v[j].x + g[3 * j], v[j].y + g[3 * j + 1], v[j].z + g[3 * j + 2]};
            sum = V3{sum.x + v[j].x, sum.y + v[j].y, sum.z + v[j].z};
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float f = 1.0f - 4.0f * w;
            v[j] = V3{f * v[j].x + w * sum.x, f * v[j].y + w * sum.y, f * v[j].z + w * sum.z};
            far = fmaxf(far, fmaxf(fmaxf(fabsf(v[j].x), fabsf(v[j].y)), fabsf(v[j].z)));
        }
    }
    const auto apart_by = [&](const V3& n) {
        const auto at = [&n](const V3& p) { return n.x * p.x + n.y * p.y + n.z * p.z; };
        const float a0 = at(a[0]), a1 = at(a[1]), a2 = at(a[2]), a3 = at(a[3]);
        const float c0 = at(c[0]), c1 = at(c[1]), c2 = at(c[2]), c3 = at(c[3]);
        const float alo = fminf(fminf(a0, a1), fminf(a2, a3)), ahi = fmaxf(fmaxf(a0, a1), fmaxf(a2, a3));
        const float clo = fminf(fminf(c0, c1), fminf(c2, c3)), chi = fmaxf(fmaxf(c0, c1), fmaxf(c2, c3));
        const float tol = 32.0f / 16777216.0f * (fabsf(n.x) + fabsf(n.y) + fabsf(n.z)) * far;
        return clo - ahi > tol || alo - chi > tol;
    };
    const auto apart_along = [&](const V3& u, const V3& v) {
        return apart_by(V3{u.y * v.z - u.z * v.y, u.z * v.x - u.x * v.z, u.x * v.y - u.y * v.x});
    };
    const auto edge = [](const V3* v, int k) {  // 01 02 03 12 13 23
        const int i = k < 3 ? 0 : (k < 5 ? 1 : 2), j = k < 3 ? k + 1 : (k < 5 ? k - 1 : 3);
        return V3{v[j].x - v[i].x, v[j].y - v[i].y, v[j].z - v[i].z};
    };
#pragma unroll
    for (int side = 0; side < 2; ++side) {
        const V3* v = side ? a : c;
        if (apart_along(edge(v, 0), edge(v, 1)) || apart_along(edge(v, 0), edge(v, 2)) ||
            apart_along(edge(v, 1), edge(v, 2)) || apart_along(edge(v, 3), edge(v, 4)))
            return true;
    }
#pragma unroll
    for (int k = 0; k < 36; ++k)
        if (apart_along(edge(a, k / 6), edge(c, k % 6))) return true;
    return false;
}

// The barycentric test of one 64-byte record (tet_bary without the box test).
// A candidate that is clearly outside is rejected on the numerators, before
// the three divisions: b = numerator / det is below -1.9e-6 or above 1.00001
// there, well past the -1e-6 and 0.999999 it is compared with, so the answer
// is that of the divided values.  Comparisons with NaN reject nothing and
// leave the decision to the full test.
template <bool EXACT>
__device__ __forceinline__ bool slot_bary(const V3& q, const uint32_t (&g0)[8], const uint32_t (&g1)[8], float4& b) {
    typedef Ar<EXACT> A;
    const auto f = [](uint32_t w) { return __uint_as_float(w); };
    const V3 v01{f(g0[3]), f(g0[4]), f(g0[5])}, v02{f(g0[6]), f(g0[7]), f(g1[0])}, v03{f(g1[1]), f(g1[2]), f(g1[3])};
    const V3 p{A::sub(q.x, f(g0[0])), A::sub(q.y, f(g0[1])), A::sub(q.z, f(g0[2]))};
    float det = det3<EXACT>(v01, v02, v03);
    if (fabsf(det) < 1e-10f) det = 1.0f;
    const float ad = fabsf(det), lo = -2e-6f * ad, hi = 1.00001f * ad;
    const uint32_t sg = __float_as_uint(det) & 0x80000000u;
    const auto signed_by = [sg](float v) { return __uint_as_float(__float_as_uint(v) ^ sg); };
    const float ny = det3<EXACT>(p, v02, v03);
    const float sy = signed_by(ny);
    if (sy < lo || sy > hi) return false;
    const float nz = det3<EXACT>(v01, p, v03);
    const float sz = signed_by(nz);
    if (sz < lo || sy + sz > hi) return false;
    const float nw = det3<EXACT>(v01, v02, p);
    const float sw = signed_by(nw);
    if (sw < lo || sy + sz + sw > hi) return false;
    b.y = A::div(ny, det);
    b.z = A::div(nz, det);
    b.w = A::div(nw, det);
    b.x = A::sub(A::sub(A::sub(1.0f, b.y), b.z), b.w);
    const float l = -1e-6f, h = 0.999999f;  // tol and 1 + tol as float32
    return b.x >= l && b.y >= l && b.z >= l && b.w >= l && b.x <= h && b.y <= h && b.z <= h && b.w <= h;
}

// jnp.dot(bary, node_values): terms accumulated in vertex order.
template <bool EXACT>
__device__ __forceinline__ V3 p1_combine(const float4& b, const V3& n0, const V3& n1, const V3& n2, const V3& n3) {
    typedef Ar<EXACT> A;
    return V3{A::add(A::add(A::add(A::mul(b.x, n0.x), A::mul(b.y, n1.x)), A::mul(b.z, n2.x)), A::mul(b.w, n3.x)),
              A::add(A::add(A::add(A::mul(b.x, n0.y), A::mul(b.y, n1.y)), A::mul(b.z, n2.y)), A::mul(b.w, n3.y)),
              A::add(A::add(A::add(A::mul(b.x, n0.z), A::mul(b.y, n1.z)), A::mul(b.z, n2.z)), A::mul(b.w, n3.z))};
}

#ifndef JT_MESH_MIN_BLOCKS
#define JT_MESH_MIN_BLOCKS 4
#endif

// NEAR: re-solve flagged near-degenerate tetrahedra in float64 (compensated
// arithmetic only); launched only for fields that have flagged ones, so the
// out-of-line call costs nothing elsewhere.
template <bool EXACT, int STORE, bool NEAR = false>
struct MeshFieldT {
    // the dependent gather chain is latency-bound: 4 blocks of 256 (64
    // registers, no spills) keep more warps in flight than the default 3
    static constexpr int kMinBlocks = JT_MESH_MIN_BLOCKS;
    static constexpr bool kHinted = true;
    jt_mesh_field F;
    const char* loc;      // locator block's header, or NULL
    int depth;            // its depth
    uint32_t faces, table, slots;  // offsets from the header
    const char* filters;

    static MeshFieldT create(const jt_mesh_field& d, int) {
        MeshFieldT m{d, nullptr, locator_depth(d), 0, 0, 0, nullptr};
        if (m.depth > 0) {
            const LocatorLayout o = locator_layout(d.n_nodes, d.n_tets, m.depth);
            m.loc = reinterpret_cast<const char*>(d.dtab) + o.header;
            m.faces = (uint32_t)(o.faces - o.header);
            m.table = (uint32_t)(o.table - o.header);
            m.slots = (uint32_t)(o.slots - o.header);
            m.filters = m.loc + (o.filters - o.header);
        }
        return m;
    }

    // Cell of coordinate x among the 2^depth cells of axis a: the number of
    // split centres at or below x, which is what the descent's comparisons
    // x >= centre add up to.  The guess is off by one only within rounding
    // of a face; NaN stays in cell 0, as every comparison of the descent fails.
    __device__ __forceinline__ int face_cell(float x, float org, float inv, int a) const {
        const int n = 1 << depth;
        int g = (int)fminf(fmaxf((x - org) * inv, 0.0f), (float)(n - 1));
        const float2* f = reinterpret_cast<const float2*>(loc + faces) + (a << depth);
        float2 b = __ldg(f + g);
        while (x < b.x) b = __ldg(f + --g);   // ends at the NaN of cell 0
        while (x >= b.y) b = __ldg(f + ++g);  // ends at the NaN of the last cell
        return g;
    }

    // The leaf (or dead end) of the descent, {elem_offset, elem_count}.
    __device__ __forceinline__ int2 locate(const V3& q) const {
        const float4 h0 = __ldg(reinterpret_cast<const float4*>(loc));
        const float2 h1 = __ldg(reinterpret_cast<const float2*>(loc) + 2);
        const int ix = face_cell(q.x, h0.x, h0.w, 0), iy = face_cell(q.y, h0.y, h1.x, 1);
        const int iz = face_cell(q.z, h0.z, h1.y, 2);
        const int2 oc = __ldg(reinterpret_cast<const int2*>(loc + table) + ((((ix << depth) | iy) << depth) | iz));
        return oc.y >= 0 ? oc : descend(q, oc.x, depth);
    }

    // Descent on the breadth-first copy from `node`, which `d` moves reached:
    // a child's index is the node's first child plus the present octants below
    // its own.
    __device__ __forceinline__ int2 descend(const V3& q, int node, int d) const {
        const int4* D = reinterpret_cast<const int4*>(F.desc);
        for (; d < F.max_depth; ++d) {
            const int4 h = __ldg(D + node);
            const unsigned w = (unsigned)h.w, m = w & 0xffu;
            if (m == 0u) break;  // a leaf (or a node without children)
            const int oct = (q.x >= __int_as_float(h.x) ? 1 : 0) + (q.y >= __int_as_float(h.y) ? 2 : 0) +
                            (q.z >= __int_as_float(h.z) ? 4 : 0);
            if (!((m >> oct) & 1u)) break;
            node = (int)(w >> 8) + __popc(m & ((1u << oct) - 1u));
        }
        return __ldg(reinterpret_cast<const int2*>(F.dtab) + node);
    }

    // First candidate of the list oc that holds the query (…optimized.py:309-360).
    // The filters are read until one is certainly the first hit; the full
    // test then runs on that candidate, or in list order on those that pass.
    // hint: the slot of the thread's last certain hit, tried before the list.
    // Filtering to the end before the full test keeps the warp together: with
    // the test inside the filter loop 10 lanes of 32 were active and the pass
    // took 16.8 ms; so, with the hint's record and the next one loaded ahead,
    // 11.5 ms, against 13.4 ms with the full test on every candidate (1M
    // particles x 64 steps, 1,572,864 tetrahedra).  Bound by latency and issue
    // together: L1 71 %, issue 60 %, 15 lanes of 32 active.
    // w: the hint's filter record, loaded before the leaf was known.
    __device__ __forceinline__ bool find_slot(const V3& q, int2 oc, int& hint, uint32_t (&w)[8], float4& b,
                                              int4& cn) const {
        const int end = oc.x + oc.y;
        int first = end, s = oc.x;
        bool certain = false;
        float slack;
        if ((unsigned)(hint - oc.x) < (unsigned)oc.y) {
            certain = filter_bary(q, w, slack) >= slack + kInside;
            if (certain) first = hint;
        }
        if (!certain) {
            hint = -1;
            if (s < end) ldg256(filters + (int64_t)s * 32, w);
            while (s < end) {
                // the next record is on its way while this one is judged
                uint32_t nx[8];
                ldg256(filters + (int64_t)min(s + 1, end - 1) * 32, nx);
                const float m = filter_bary(q, w, slack);
                const bool alone = filter_flags(w) & JT_TET_ALONE;
                if (m >= -slack) {
                    if (first == end) first = s;
                    if (alone && m >= slack + kInside) {
                        certain = true;
                        first = hint = s;
                        break;
                    }
                }
                ++s;
#pragma unroll
                for (int k = 0; k < 8; ++k) w[k] = nx[k];
            }
        }
        for (s = first; s < end; ++s) {
            if (!certain && s != first) {
                ldg256(filters + (int64_t)s * 32, w);
                if (filter_bary(q, w, slack) < -slack) continue;
            }
            const char* rec = loc + slots + (int64_t)s * 64;
            uint32_t g0[8], g1[8];
            ldg256(rec, g0);
            ldg256(rec + 32, g1);
            if (!slot_bary<EXACT>(q, g0, g1, b)) continue;
            if (!certain || (NEAR && !EXACT)) {
                const int t = __ldg(F.elems + s);
                const float4* bx = reinterpret_cast<const float4*>(F.tet_box) + 2 * (int64_t)t;
                const float4 mn = __ldg(bx), mx = __ldg(bx + 1);
                if (!(q.x >= mn.x && q.y >= mn.y && q.z >= mn.z && q.x <= mx.x && q.y <= mx.y && q.z <= mx.z)) continue;
                if (NEAR && !EXACT && mn.w != 0.0f) b = bary_f64(q, F.tet_geom, t);
            }
            cn = make_int4((int)g1[4], (int)g1[5], (int)g1[6], (int)g1[7]);
            return true;
        }
        return false;
    }

    __device__ __forceinline__ V3 node_value(int node, const jt_blend& e) const {
        const int64_t base = (int64_t)min(max(e.pair, 0), F.n_pairs - 1) * F.pair_stride;
        return blend<EXACT, STORE>(load_pair<STORE>(F.pairs, base + node), e);
    }

    __device__ __forceinline__ V3 operator()(const V3& q, const jt_blend& e, int& flags) const {
        int hint = -1;
        return at(q, e, flags, hint);
    }

    // The value at q; hint as find_slot keeps it from one evaluation of a
    // thread to the next (start with -1).
    __device__ __forceinline__ V3 at(const V3& q, const jt_blend& e, int& flags, int& hint) const {
        typedef Ar<EXACT> A;
        // fixed-depth descent (…optimized.py:278-302): at most max_depth moves,
        // stopping at a leaf or where the query's octant has no child; then
        // the candidate scan (…optimized.py:309-360): first candidate whose box
        // holds the query and whose barycentrics pass the tolerance test
        int2 oc;
        if (loc != nullptr) {
            uint32_t w[8];
            ldg256(filters + (int64_t)max(hint, 0) * 32, w);
            oc = locate(q);
            float4 b;
            int4 cn;
            if (find_slot(q, oc, hint, w, b, cn))
                return p1_combine<EXACT>(b, node_value(cn.x, e), node_value(cn.y, e), node_value(cn.z, e),
                                         node_value(cn.w, e));
        } else {
            if (F.desc != nullptr) {
                oc = descend(q, 0, 0);
            } else {
                int node = 0;
                for (int d = 0; d < F.max_depth; ++d) {
                    const int4 h = __ldg(reinterpret_cast<const int4*>(F.nodes + node));
                    if (h.w) break;  // is_leaf
                    const int oct = (q.x >= __int_as_float(h.x) ? 1 : 0) + (q.y >= __int_as_float(h.y) ? 2 : 0) +
                                    (q.z >= __int_as_float(h.z) ? 4 : 0);
                    const int ch = __ldg(&F.nodes[node].children[oct]);
                    if (ch < 0) break;
                    node = ch;
                }
                oc = __ldg(reinterpret_cast<const int2*>(&F.nodes[node].elem_offset));
            }
            for (int s = 0; s < oc.y; ++s) {
                float4 b;
                int4 cn;
                bool near;
                const int t = __ldg(F.elems + oc.x + s);
                if (!tet_bary<EXACT>(q, F.tet_box, F.tet_geom, t, b, cn, near)) continue;
                if (NEAR && !EXACT && near) b = bary_f64(q, F.tet_geom, t);
                return p1_combine<EXACT>(b, node_value(cn.x, e), node_value(cn.y, e), node_value(cn.z, e),
                                         node_value(cn.w, e));
            }
        }
        // cheap fallback (…optimized.py:364-376): nearest of the four vertices
        // of the first candidate; an empty list reads slot -1, which indexes
        // the last tetrahedron
        flags |= JT_STATUS_OCTREE_FALLBACK;
        int4 cn;
        if (loc != nullptr && oc.y > 0) {
            cn = __ldg(reinterpret_cast<const int4*>(loc + slots) + 4 * (int64_t)oc.x + 3);
        } else {
            int first = oc.y > 0 ? __ldg(F.elems + oc.x) : -1;
            if (first < 0) first += F.n_tets;
            cn = __ldg(reinterpret_cast<const int4*>(F.tet_geom) + 4 * (int64_t)first + 3);
        }
        const int ids[4] = {cn.x, cn.y, cn.z, cn.w};
        int best = ids[0];
        float bd = 0.0f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float4 pk = __ldg(reinterpret_cast<const float4*>(F.points) + ids[k]);
            const float dx = A::sub(pk.x, q.x), dy = A::sub(pk.y, q.y), dz = A::sub(pk.z, q.z);
            const float d = A::add(A::add(A::mul(dx, dx), A::mul(dy, dy)), A::mul(dz, dz));
            if (k == 0 || d < bd) { bd = d; best = ids[k]; }
        }
        return node_value(best, e);
    }
};

template <bool EXACT, int STORE>
using MeshField = MeshFieldT<EXACT, STORE, false>;
template <bool EXACT, int STORE>
using MeshFieldNear = MeshFieldT<EXACT, STORE, true>;

}  // namespace jt

// tess_clip_lean.cu -- the FP32 clipping: one Voronoi cell per warp, with one
// candidate plane per lane (Cell::compute_voronoi_cell, interface.rs:257-313).
//
// Positions, planes and classification are FP32, with a rigorous bound on each
// plane test's error (see plane_test).  A test inside its bound is undecided:
// the plain pass hands the cell on, the careful pass settles the test in FP64.
// The bins around the site come as rows (see the walk), a window of 32
// candidates is worked off as follows:
//
//   - The cell's vertices live in shared memory only.  When a window is
//     loaded, every lane tests its own candidate's bisector against every live
//     vertex and keeps the touched ones (Outside or undecided) as a 64-bit mask
//     over the slots.
//   - Candidates whose mask is empty can never cut (the cell only shrinks) and
//     cost nothing more.  The nearest candidate with a live touched vertex is
//     taken by one warp minimum; its mask is the cut's Outside set.
//   - After a cut every lane tests its candidate against the new vertices
//     alone (about four).
//   - A vertex inside a candidate's guard band counts as touched; when its
//     turn comes, the touched vertices are tested again, and one still inside
//     the band hands the cell over (every such vertex is touched).
//   - A window with few candidates within reach spreads the vertices of each
//     test over several lanes.
//
// A test of one candidate at a time against one vertex per lane, as in
// tess_clip_impl.cuh, takes 49 serial tests per cell, of which 32 cut nothing.
//
// What bounds it: instruction issue.  1,000,000 uniform points: 16.4 ms that
// way with the vertices in registers (12.9 k warp instructions per cell, 16
// warps per SM), 11.9 ms with a candidate per lane, 10.6 ms with the bins taken
// as rows (three batches a cell instead of five) and the undecided vertices
// found at the cut instead of in every test, 9.9 ms as it stands (9.6 k warp
// instructions a cell, 78% of the issue slots).  The code has to stay small: past
// about 40 KB of it the warps, each at another place, wait for instructions.
//
// With the FP64 finish (MIXED and the FP64 form) the faces' planes, vertices,
// areas and the volume are computed in FP64 from the FP64 positions; only the
// decisions which planes meet where are taken in FP32, each beyond its error
// bound.  For the FP64 form the band is wider by the reference's tolerance, so
// that every decision is the one its test takes in FP64.  250,007 uniform
// points in that form: 12.6 -> 3.6 ms; the FP64 clipping it replaces spent
// about 655 FP64 instructions on a cell, this finish about 130.
#include <climits>

#include "tess_clip_impl.cuh"

namespace tess {
namespace cliplean {

using namespace clipk;

constexpr int kSlots = 64;     // vertex slots
constexpr int kPlanes = 96;    // planes, walls included
constexpr int kNearZ = 2;      // the first three batches take the bins up to this offset along z

// Instances of the pass:
//   kPlain    over every cell; a cell with an undecided test or a crowded own
//             bin goes on to the careful pass
//   kCount    the same with work counters (they cost registers)
//   kDense    over the cells of crowded bins: seeded, points gathered
//   kCareful  as kDense, and undecided tests are settled in FP64 in place: over
//             the cells the others handed on, or over every cell of a small
//             input.  Always with the FP64 finish.  (An instance of its own: the
//             settling makes the code half as large again, and the dense pass
//             waits for instructions.)
//   kGeo      one cell with its geometry (single-cell queries): careful, the
//             site may be any position and the container any box
enum Mode : int { kPlain = 0, kCount = 1, kDense = 2, kCareful = 3, kGeo = 4 };

struct Lean {
    float4 vtx[kSlots];             // vertex position, error bound
    // x: planes a | b << 8 | c << 16; y: for the edges (a,b), (b,c), (c,a) the
    // vertex across, slot | k << 6, where k is the edge's index there
    uint2 topo[kSlots];
    uint32_t psrc[kPlanes + 1];     // sorted index of the point that made the plane
    // new-vertex ring map: of each plane, the new vertex that has it first (low
    // half) and second (high half), each tag of the cut << 8 | slot; tags run on
    // from cell to cell (the map is cleared when they wrap)
    uint32_t map[kPlanes];
    union {
        struct {                            // walk
            float4 pl[kPlanes + 1];         // plane: normal, offset
            float pn[kPlanes + 1];          // |normal|
            float vr[kSlots];               // (|v| + e_v)^2
            float4 cand[32];                // a window's candidates within reach: plane ...
            float candn[32];                // ... |normal| ...
            uint32_t candj[32];             // ... and (careful) sorted index
            float4 nv[32];                  // the new vertices of a cut, in order ...
            alignas(4) uint8_t nvs[32];     // ... and their slots
            uint32_t boff[32];              // batch: start - prefix of the k-th bin that holds points
            uint16_t items[32];             // boundary edges of a cut with more than 32 edges
            uint8_t fl[kSlots + kSlots];    // free-slot stack (top = lowest free slot)
        };
        struct {                            // finalize, FP32
            float4 q[kPlanes];              // face plane n.x = h as FP32 pairs: high parts ...
            float4 ql[kPlanes];             // ... and low parts
            float4 dv[kSlots];              // Newton corrections
            float dist[kPlanes];            // distance of the face plane from the site
            float area[kPlanes];
            alignas(16) int32_t ids[kPlanes + 4];   // ids of the cell's faces, in plane order
            uint8_t fsta[kPlanes];          // a vertex of each face: slot | plane's place << 6 (0xFF: none)
            uint8_t face[kPlanes];          // planes that have a face
            uint8_t rank[kPlanes];          // position of the face in id order
        } s;
        struct {                            // finalize, FP64
            double2 qa[kPlanes], qb[kPlanes];   // face plane n.x = h: {n.x, n.y}, {n.z, h}
            double rx[kSlots], ry[kSlots], rz[kSlots];   // refined positions
            double area[kPlanes];
            alignas(16) int32_t ids[kPlanes + 4];
            uint8_t fsta[kPlanes];
            uint8_t face[kPlanes];
            uint8_t rank[kPlanes];
        } d;
    };
};

__device__ __forceinline__ int byte_of(uint32_t t, int i) { return (int)__byte_perm(t, 0u, 0x4440u | (unsigned)i); }

// Hardware approximations without the subnormal handling of rsqrtf and
// __fdividef.  A subnormal squared length gives an infinite norm, a subnormal
// determinant an infinite vertex; both end in the guard band.
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rcp_ftz(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// Upper bound of sqrt(x), x >= 0: rsqrt is within 2 ulp and the product adds
// half an ulp, so the 2^-20 inflation keeps it above the exact root.  0 gives
// 0, +inf and NaN +inf.
__device__ __forceinline__ float norm_up(float x) {
    const float r = x * rsqrt_ftz(x) * 1.00000095367431640625f;
    return x == 0.f ? 0.f : (x < INFINITY ? r : INFINITY);
}
__device__ __forceinline__ float vertex_r2(float x, float y, float z, float e) {
    const float r = norm_up(x * x + y * y + z * z) + e;
    return r * r;
}

// Signed distance of a vertex and the half-width of its guard band for the
// bisector n = r, off = r.r / 2 of the site and a point at r, rn = |r|:
//   band = rn e + c0,  c0 = rn (guard_rel rn + tol) + eC,
// where e is the vertex's error bound e_v, to which guard_rel |v|_1 is added at
// its creation, and eC covers the hi/lo split of the positions.  A test with
// |sd| <= band is undecided.  The bound, with u = 2^-24, r~ the FP32 offset
// (|r~ - r| <= 2u |r|) and v~ the FP32 vertex (|v~ - v| <= e_v):
//   fma chain rounding       3u (rn |v~|_1 + off)
//   plane normal, vertex     2u rn |v|  +  rn e_v
//   offset r.r / 2           3u rn^2
// <= rn (e_v + 5u |v~|_1 + 4.5u rn), about rn (e_v + 3e-7 (|v~|_1 + rn)); the
// default guard_rel 4e-7 leaves a third in hand.  eC: per component the offset
// r~ = (hi_p - hi_s) + (lo_p - lo_s) is off by at most 2u |r| plus eta =
// 6.1 u^2 (|site|_inf + R) (the lo parts' rounding, the hi subtraction's share
// of it, the FP64 centring), which moves n.v - off by at most
// eta (|v|_1 + 1.8 rn) <= 5.4 eta R.  R only shrinks, so the initial radius
// bounds it for the whole cell.  Candidates nearer than 4 eta / u (plane error
// above u / 4 relative, beyond the vertex error model) send the cell to FP64.
__device__ __forceinline__ void plane_test(const float4& v, float nx, float ny, float nz, float off, float rn,
                                           float c0, float& sd, float& band) {
    sd = sdist(nx, ny, nz, off, v.x, v.y, v.z);
    band = fmaf(rn, v.w, c0);
}
// Outside, or undecided in FP32.
__device__ __forceinline__ bool touched(const float4& v, float nx, float ny, float nz, float off, float rn, float c0) {
    float sd, band;
    plane_test(v, nx, ny, nz, off, rn, c0, sd, band);
    return sd >= -band;
}

// The rows of bins (fixed x and y offset, running in z) in the order they are
// walked, packed per lane: byte 0/1 the x/y offset in the first batch, byte
// 2/3 in the second.
//   first batch: lanes 2r, 2r + 1 the part of central row r below and above
//     the 27 bins around the site's; lanes 18..29 the twelve rows at x or
//     y offset +-2 beside them
//   second batch: the corners (+-2, +-2), then the 24 rows of ring 3
// The nine central rows, nearest first: the site's own, the four beside it, the
// four at the corners.  (500,000 clustered points: 17.9 ms of dense, careful and
// FP64 passes in row-major order, 14.9 so; 3,614 cells beyond 96 planes, 29 so.
// Uniform points 1% faster.)
__device__ __forceinline__ int row_i(int r) { return (int)(0x28161ULL >> (2 * r) & 3u) - 1; }
__device__ __forceinline__ int row_j(int r) { return (int)(0x22215ULL >> (2 * r) & 3u) - 1; }
__device__ uint32_t row_plan(int lane) {
    int ia = 0, ja = 0, ib = 0, jb = 0;
    if (lane < 18) {
        ia = row_i(lane >> 1);
        ja = row_j(lane >> 1);
    } else if (lane < 30) {
        const int q = lane - 18, e = q % 3 - 1, f = (q / 3) & 1 ? 2 : -2;
        ia = q < 6 ? f : e;
        ja = q < 6 ? e : f;
    }
    if (lane < 4) {
        ib = lane & 1 ? 2 : -2;
        jb = lane & 2 ? 2 : -2;
    } else if (lane < 28) {
        const int q = lane - 4;
        if (q < 14) {
            ib = q < 7 ? -3 : 3;
            jb = q % 7 - 3;
        } else {
            ib = (q - 14) % 5 - 2;
            jb = q < 19 ? -3 : 3;
        }
    }
    return (uint32_t)(ia & 0xFF) | (uint32_t)(ja & 0xFF) << 8 | (uint32_t)(ib & 0xFF) << 16 | (uint32_t)(jb & 0xFF) << 24;
}
// Row r of batch 3 (both ends, two lanes each, of the rows up to ring 3) or of
// the 8 m rows of ring m > 3 (rows with max(|i|, |j|) = m).  Packed offsets,
// -1 past the last row.  Out of line: sparse regions and thin boxes.
__device__ __noinline__ int far_row(int m, int r) {
    int i, j;
    if (m == 3) {
        r >>= 1;
        if (r >= 49) return -1;
        i = r / 7 - 3;
        j = r % 7 - 3;
    } else {
        if (r >= 8 * m) return -1;
        const int side = 2 * m + 1;
        if (r < 2 * side) {
            i = r < side ? -m : m;
            j = r % side - m;
        } else {
            r -= 2 * side;
            i = r % (side - 2) - (m - 1);
            j = r < side - 2 ? -m : m;
        }
    }
    return (i + 2048) << 12 | (j + 2048);
}

// Coordinate a of the site in FP64 (a single-cell query may give a position),
// and of the container's corners.
__device__ __forceinline__ double site_coord(const ClipParams& P, uint32_t gs, int a) {
    if (P.at_point) return P.point[a];
    return a == 0 ? P.spx[gs] : (a == 1 ? P.spy[gs] : P.spz[gs]);
}
__device__ __forceinline__ double box_lo(const ClipParams& P, const DiagDesc& D, int a) {
    return P.box_override ? P.box[a] : D.blo[a];
}
__device__ __forceinline__ double box_hi(const ClipParams& P, const DiagDesc& D, int a) {
    return P.box_override ? P.box[3 + a] : D.bhi[a];
}

// A search radius (rare, out of line): the site's exact bin, and the end of
// the bins of a row whose search-order key stays within it (the key grows
// with the distance along the row).
__device__ __noinline__ int exact_bin(const ClipParams& P, const DiagDesc& D, uint32_t gs, int a) {
    return axis_index(site_coord(P, gs, a), D.glo[a], D.ghi[a], D.inv[a], D.cpd);
}
__device__ __noinline__ int radius_reach(const DiagDesc& D, double radius, int i, int j, int k) {
    const int step = k > 0 ? -1 : 1;
    while (k != 0 && gap_key(D.size, i, j, k) > radius) k += step;
    return (k == 0 && gap_key(D.size, i, j, 0) > radius) ? INT_MAX : k;
}

// The bins kl .. kh of row (i, j) whose key is within the radius (none: an empty
// range).  The row's least and greatest key in FP32 (four roundings) first: only a
// row near the radius takes FP64.
__device__ __noinline__ int2 radius_row(const DiagDesc& D, double radius, int i, int j, int kl, int kh, int cbz) {
    const float r = (float)radius;
    const int ni = max(abs(i) - 1, 0), nj = max(abs(j) - 1, 0), nk = max(max(cbz - kl, kh - cbz) - 1, 0);
    const float gx = (float)ni * D.size_f[0], gy = (float)nj * D.size_f[1], gz = (float)nk * D.size_f[2];
    const float least = gx * gx + gy * gy, most = least + gz * gz;
    if (least > r * 1.0001f + 1e-30f) return make_int2(1, 0);
    if ((ni | nj | nk) && !(r > 1e-30f && most < r * 0.9999f)) {
        const int a = radius_reach(D, radius, i, j, min(kl - cbz, 0)), b = radius_reach(D, radius, i, j, max(kh - cbz, 0));
        if (a == INT_MAX) return make_int2(1, 0);
        kl = max(kl, cbz + a);
        kh = min(kh, cbz + b);
    }
    return make_int2(kl, kh);
}
// The next batch or ring from m >= 2 on that has bins within the radius (none:
// INT_MAX): rows at an x or y offset of +-m or more, or (batch 3) ends beyond kNearZ.
__device__ __noinline__ int radius_next(const DiagDesc& D, double radius, int m) {
    auto rows_beyond = [&](int o) { return gap_key(D.size, o, 0, 0) > radius && gap_key(D.size, 0, o, 0) > radius; };
    if (m == 2 && rows_beyond(2)) m = 3;
    if (m == 3 && gap_key(D.size, 0, 0, kNearZ + 1) > radius) m = 4;
    return m >= 4 && rows_beyond(m) ? INT_MAX : m;
}

// A wall's distance from the site in FP64 (only cells that touch the box).
__device__ __noinline__ double wall_distance(const ClipParams& P, const DiagDesc& D, uint32_t gs, int p) {
    const int a = p >> 1;
    const double s = site_coord(P, gs, a);
    return (p & 1) ? box_hi(P, D, a) - s : s - box_lo(P, D, a);
}

// The vertex of planes a, b, c in FP64, by Cramer's rule on the walls and the
// bisectors of the FP64 positions; cond = |n_a| |n_b| |n_c| / |det|, +inf when
// the planes are singular.
struct Vertex64 {
    double x, y, z;
    float cond;
};
__device__ __forceinline__ Vertex64 vertex_fp64(const Lean& S, const ClipParams& P, const DiagDesc& D, uint32_t gs,
                                             uint32_t planes) {
    const double sx = site_coord(P, gs, 0), sy = site_coord(P, gs, 1), sz = site_coord(P, gs, 2);
    double n[3][3], h[3];
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        const int p = byte_of(planes, e);
        if (p < 6) {
            const int a = p >> 1;
            const double sg = (p & 1) ? 1.0 : -1.0;
            n[e][0] = a == 0 ? sg : 0.0;
            n[e][1] = a == 1 ? sg : 0.0;
            n[e][2] = a == 2 ? sg : 0.0;
            const double s = a == 0 ? sx : (a == 1 ? sy : sz);
            h[e] = (p & 1) ? box_hi(P, D, a) - s : s - box_lo(P, D, a);
        } else {
            const uint32_t j = tess_chk(S.psrc[p], P.npts, P.check, CK_POINT);
            n[e][0] = P.spx[j] - sx;
            n[e][1] = P.spy[j] - sy;
            n[e][2] = P.spz[j] - sz;
            h[e] = 0.5 * (n[e][0] * n[e][0] + n[e][1] * n[e][1] + n[e][2] * n[e][2]);
        }
    }
    const double bc0 = n[1][1] * n[2][2] - n[1][2] * n[2][1], bc1 = n[1][2] * n[2][0] - n[1][0] * n[2][2],
                 bc2 = n[1][0] * n[2][1] - n[1][1] * n[2][0];
    const double ca0 = n[2][1] * n[0][2] - n[2][2] * n[0][1], ca1 = n[2][2] * n[0][0] - n[2][0] * n[0][2],
                 ca2 = n[2][0] * n[0][1] - n[2][1] * n[0][0];
    const double ab0 = n[0][1] * n[1][2] - n[0][2] * n[1][1], ab1 = n[0][2] * n[1][0] - n[0][0] * n[1][2],
                 ab2 = n[0][0] * n[1][1] - n[0][1] * n[1][0];
    const double det = n[0][0] * bc0 + n[0][1] * bc1 + n[0][2] * bc2;
    const double inv = recip_nr(det);
    Vertex64 v;
    v.x = (h[0] * bc0 + h[1] * ca0 + h[2] * ab0) * inv;
    v.y = (h[0] * bc1 + h[1] * ca1 + h[2] * ab1) * inv;
    v.z = (h[0] * bc2 + h[1] * ca2 + h[2] * ab2) * inv;
    // one refinement step
    const double r0 = h[0] - (n[0][0] * v.x + n[0][1] * v.y + n[0][2] * v.z);
    const double r1 = h[1] - (n[1][0] * v.x + n[1][1] * v.y + n[1][2] * v.z);
    const double r2 = h[2] - (n[2][0] * v.x + n[2][1] * v.y + n[2][2] * v.z);
    v.x += (r0 * bc0 + r1 * ca0 + r2 * ab0) * inv;
    v.y += (r0 * bc1 + r1 * ca1 + r2 * ab1) * inv;
    v.z += (r0 * bc2 + r1 * ca2 + r2 * ab2) * inv;
    auto norm = [](const double (&u)[3]) {
        const float x = (float)u[0], y = (float)u[1], z = (float)u[2];
        return norm_up(x * x + y * y + z * z);
    };
    v.cond = fabsf((float)inv) * norm(n[0]) * norm(n[1]) * norm(n[2]);
    if (!(fabs(det) > 0.0)) v.cond = INFINITY;
    return v;
}

// Side of the vertex of `planes` relative to the bisector of the site and
// point j, decided in FP64 with the reference's test (vector3.rs:170-239,
// tolerance 1e-12): 1 Outside, 0 not, -1 when the planes are singular.  Out of
// line: few vertices need it.
__device__ __noinline__ int side_fp64(const Lean& S, const ClipParams& P, const DiagDesc& D, uint32_t gs, uint32_t planes,
                                      uint32_t j) {
    const Vertex64 v = vertex_fp64(S, P, D, gs, planes);
    if (!(v.cond < 1e12f)) return -1;
    const double qx = P.spx[j] - site_coord(P, gs, 0), qy = P.spy[j] - site_coord(P, gs, 1),
                 qz = P.spz[j] - site_coord(P, gs, 2);
    const double q2 = qx * qx + qy * qy + qz * qz;
    return (qx * v.x + qy * v.y + qz * v.z - 0.5 * q2) / sqrt(q2) > kTolerance ? 1 : 0;
}

template <bool EXACT, int MODE>
__device__ __forceinline__ void run_lean(const ClipParams& P, Lean& S, uint32_t gs, const DiagDesc& D, uint32_t plan, uint32_t& gen, Work& W,
                                         int lane) {
    const unsigned lt = (1u << lane) - 1u;
    const uint32_t pt_base = D.pt_base;
    constexpr bool COUNT = MODE != kPlain, SEED = MODE >= kDense, CAREFUL = MODE >= kCareful, GEO = MODE == kGeo;
    static_assert(EXACT || !CAREFUL, "cells with undecided tests finish in FP64");
    // a coordinate relative to the centre of the points as an FP32 pair
    auto pair = [&](double x, int a, float& h, float& l) {
        const double u = x - D.ctr[a];
        h = (float)u;
        l = (float)(u - (double)h);
    };
    float4 site_h, site_l;
    if (GEO && P.at_point) {
        pair(P.point[0], 0, site_h.x, site_l.x);
        pair(P.point[1], 1, site_h.y, site_l.y);
        pair(P.point[2], 2, site_h.z, site_l.z);
        site_h.w = __uint_as_float(0u);
    } else {
        site_h = P.phi[gs];
        site_l = P.plo[gs];
    }
    const float shx = site_h.x, shy = site_h.y, shz = site_h.z;
    const float slx = site_l.x, sly = site_l.y, slz = site_l.z;
    const uint32_t orig = tess_chk(__float_as_uint(site_h.w), P.npts, P.check, CK_POINT);
    const float gr = P.guard_rel, tol = P.tol;

    // ---- the container box, translated by -site (polyhedron.rs:268-392) ----
    // Offsets from the FP32 pairs of the box and the site relative to the
    // centre, one rounding each side of the sum (<= 2^-23 relative).
    auto wall = [&](int a, bool mx) {
        const float sh_a = a == 0 ? shx : (a == 1 ? shy : shz);
        const float sl_a = a == 0 ? slx : (a == 1 ? sly : slz);
        if (GEO && P.box_override) {
            float h, l;
            pair(P.box[mx ? 3 + a : a], a, h, l);
            return (h - sh_a) + (l - sl_a);
        }
        return mx ? (D.bhi_hi[a] - sh_a) + (D.bhi_lo[a] - sl_a) : (D.blo_hi[a] - sh_a) + (D.blo_lo[a] - sl_a);
    };
    if (lane < 6) {
        const int a = lane >> 1;
        const bool mx = lane & 1;
        const float sg = mx ? 1.f : -1.f, off = sg * wall(a, mx);
        S.pl[lane] = make_float4(a == 0 ? sg : 0.f, a == 1 ? sg : 0.f, a == 2 ? sg : 0.f, off);
        S.pn[lane] = 1.f;
    }
    float r2l = 0.f;
    if (lane < 8) {
        const int bx = lane & 1, by = (lane >> 1) & 1, bz = (lane >> 2) & 1;
        const float vx = wall(0, bx), vy = wall(1, by), vz = wall(2, bz);
        // 2^-23 relative per component (doubled), and the vertex's share of a
        // plane test's rounding
        const float ve = (2.5e-7f + gr) * (fabsf(vx) + fabsf(vy) + fabsf(vz));
        S.vtx[lane] = make_float4(vx, vy, vz, ve);
        r2l = vertex_r2(vx, vy, vz, ve);
        S.vr[lane] = r2l;
        const int pX = bx, pY = 2 + by, pZ = 4 + bz;
        const bool pos = ((bx + by + bz) & 1) != 0;     // sign of the corner's octant
        const int t0 = pX, t1 = pos ? pY : pZ, t2 = pos ? pZ : pY;
        auto flip = [](int p) { return p < 2 ? 1 : (p < 4 ? 2 : 4); };
        const int n0 = lane ^ flip(t2), n1 = lane ^ flip(t0), n2 = lane ^ flip(t1);
        // the corner across an edge has the opposite orientation: edges 0, 1, 2
        // are its edges 2, 1, 0
        S.topo[lane] = make_uint2((uint32_t)t0 | ((uint32_t)t1 << 8) | ((uint32_t)t2 << 16),
                                  (uint32_t)(n0 | 2 << 6) | ((uint32_t)(n1 | 1 << 6) << 8) | ((uint32_t)n2 << 16));
    }
    // free-slot stack: slots 8 .. 63, lowest on top
    S.fl[lane] = (uint8_t)(kSlots - 1 - lane);
    if (lane < kSlots - 8 - 32) S.fl[32 + lane] = (uint8_t)(kSlots - 1 - 32 - lane);
    int nfree = kSlots - 8;
    uint32_t l0 = 0xFFu, l1 = 0u;      // live slots
    int np = 6;
    float R2 = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(r2l)));
    // the hi/lo split's share of a plane test's error, and the distance below
    // which a candidate is handed to FP64 (see plane_test)
    float eC, dup2;
    {
        const float sa = fmaxf(fabsf(shx), fmaxf(fabsf(shy), fabsf(shz))) * 1.001f;
        const float R = norm_up(R2) * 1.001f;
        eC = 1.3e-13f * (sa + R) * R;
        const float d = 1.5e-6f * (sa + R);
        dup2 = d * d;
    }
    int status = ST_OK;

    // ---- the walk: bins around the site, nearest rows first ----
    // (ExpandingSearch, celery.rs:865-1075, visits single bins in key order;
    // any order that covers the bins within twice the cell radius gives the
    // same cell).  Bins of one x and y are contiguous in the sorted order along
    // z, so a lane takes a whole row of them as one range:
    //   batch 0   the 27 bins around the site's, no test
    //   batch 1   the rest of those nine rows and the twelve rows beside them
    //   batch 2   the four corner rows and ring 3
    //   then      ring by ring (sparse regions)
    // Rows and their ends beyond twice the current cell radius are left out.
    const int cpd = D.cpd;
    float feps = D.frac_eps;
    // the site in bin units (within feps), its bin and its place in it
    const float inx = D.inv_s[0], iny = D.inv_s[1], inz = D.inv_s[2];
    float px = ((shx - D.glo_hi[0]) + (slx - D.glo_lo[0])) * inx, py = ((shy - D.glo_hi[1]) + (sly - D.glo_lo[1])) * iny,
          pz = ((shz - D.glo_hi[2]) + (slz - D.glo_lo[2])) * inz;
    int cbx = min(max((int)px, 0), cpd - 1), cby = min(max((int)py, 0), cpd - 1), cbz = min(max((int)pz, 0), cpd - 1);
    // an axis without extent has all its points in the last bin
    if (inx == 0.f) px = cbx = cpd - 1;
    if (iny == 0.f) py = cby = cpd - 1;
    if (inz == 0.f) pz = cbz = cpd - 1;
    if constexpr (GEO) {
        // outside the container or far off the grid: the FP64 form; a little off
        // the grid: the bin position's error grows with it
        bool in = true;
        for (int a = 0; a < 3; ++a) in = in && site_coord(P, gs, a) > box_lo(P, D, a) && site_coord(P, gs, a) < box_hi(P, D, a);
        const float away = fabsf(px) + fabsf(py) + fabsf(pz);
        if (!in || !(away < 1e6f) || (P.at_point && (inx == 0.f || iny == 0.f || inz == 0.f))) status = ST_GUARD;
        feps += 1e-6f * away;
    }
    if (P.has_radius) {
        cbx = exact_bin(P, D, gs, 0);
        cby = exact_bin(P, D, gs, 1);
        cbz = exact_bin(P, D, gs, 2);
    }
    const float fx = fminf(fmaxf(px - (float)cbx, 0.f), 1.f), fy = fminf(fmaxf(py - (float)cby, 0.f), 1.f);
    const float fz = fminf(fmaxf(pz - (float)cbz, 0.f), 1.f);
    // Dense and careful: when the own bin is crowded, it and the crowded bins around it
    // are seeded first, nearest first: each lane takes the nearest point of its
    // stride of the bin, and the 32 are cut as one window.  Otherwise windows
    // in storage order meet the nearest points late, after many cuts by farther
    // ones (clustered inputs: 62 cuts a cell instead of 23).
    uint32_t nbeg = 0, ncnt = 0;
    float nd = INFINITY;
    unsigned pending = 0;
    bool undec = false;              // careful: a test was settled in FP64 ...
    int settled = 0;                 // ... in so many cuts
    if constexpr (SEED) {
        const int ti = lane / 9 - 1, tj = (lane / 3) % 3 - 1, tk = lane % 3 - 1;
        const int x = cbx + ti, y = cby + tj, z = cbz + tk;
        if (lane < 27 && x >= 0 && x < cpd && y >= 0 && y < cpd && z >= 0 && z < cpd) {
            const uint64_t lb = tess_chk(D.bin_base + ((uint64_t)x * cpd + y) * cpd + z, P.nbins, P.check, CK_BIN);
            nbeg = P.delims[lb];
            ncnt = P.delims[lb + 1] - nbeg;
            const float dx = fmaxf((ti > 0 ? 1.f - fx : (ti < 0 ? fx : 0.f)) - feps, 0.f) * D.size_f[0];
            const float dy = fmaxf((tj > 0 ? 1.f - fy : (tj < 0 ? fy : 0.f)) - feps, 0.f) * D.size_f[1];
            const float dz = fmaxf((tk > 0 ? 1.f - fz : (tk < 0 ? fz : 0.f)) - feps, 0.f) * D.size_f[2];
            nd = (dx * dx + dy * dy + dz * dz) * (1.0f - 1e-4f);
        }
        const unsigned many = __ballot_sync(FULL, ncnt >= P.seed_min);
        if (__shfl_sync(FULL, ncnt, 13) >= P.seed_min) pending = many;
    }
    const bool crowded = SEED && pending != 0;
    uint32_t pend = 0;               // batch 0: where my row's points that were not taken start
    int m = 0, ring0 = 0;            // batch (0, 1, 2) or ring (4 on); first row of a ring's batch
    // bin sides or a cell radius outside FP32's normal range
    if (!D.lean_ok) status = SEED ? ST_GUARD : ST_DENSE;
    if (!(R2 >= FLT_MIN)) status = ST_GUARD;
    if (GEO && !(R2 < 1e30f)) status = ST_GUARD;
    while (status == ST_OK) {
        float sx_ = 0.f, sy_ = 0.f, sz_ = 0.f, s2_ = INFINITY;   // my seed
        uint32_t sj_ = 0;
        unsigned total, pref = 0;
        uint32_t bbeg = 0, bcnt = 0;
        const bool direct = SEED && pending != 0;
        if (direct) {
            // ---- the seeds of the nearest crowded bin left ----
            const unsigned best = __reduce_min_sync(
                FULL, ((pending >> lane) & 1u) ? ((__float_as_uint(nd) & ~31u) | (unsigned)lane) : 0xFFFFFFFFu);
            const int cb = (int)(best & 31u);
            pending &= ~(1u << cb);
            // (beyond half a radius a bin's nearest points seldom cut, and its seeds
            // would be a whole window: 2,097,152 clustered points, passes after the
            // first: 51.0 ms when all bins within twice the radius are seeded, 47.1
            // up to 0.7 or 0.4 radii, 47.0 up to 0.55, 48.6 up to 0.17, 80.8 with
            // the own bin's seeds alone)
            if (cb != 13 && __shfl_sync(FULL, nd, cb) >= 0.3f * R2) {
                pending = 0;     // the others are farther
                continue;
            }
            const uint32_t sbeg = __shfl_sync(FULL, nbeg, cb), scnt = __shfl_sync(FULL, ncnt, cb);
            bool near = false;
#pragma unroll 1
            for (uint32_t q = lane; q < scnt; q += 32) {
                const uint32_t j = tess_chk(sbeg + q, P.npts, P.check, CK_POINT);
                const float4 h = P.phi[j], l = P.plo[j];
                const float rx = (h.x - shx) + (l.x - slx), ry = (h.y - shy) + (l.y - sly), rz = (h.z - shz) + (l.z - slz);
                const float r2 = rx * rx + ry * ry + rz * rz;
                near |= j != gs && !(r2 > dup2);
                bool take = j != gs && r2 > dup2 && r2 < s2_;
                if (take && P.target_group >= 0) take = (int64_t)(P.sgroup ? P.sgroup[j] : 0u) == P.target_group;
                if (take) {
                    sx_ = rx;
                    sy_ = ry;
                    sz_ = rz;
                    s2_ = r2;
                    sj_ = j;
                }
            }
            if (__any_sync(FULL, near)) {
                status = ST_NEAR;
                break;
            }
            total = 32;
        } else {
        // ---- the next batch: one row of bins per lane ----
        int i = 0, j = 0;
        bool have;
        if (m == 0) {
            have = lane < 10;
            if (lane < 9) {
                i = row_i(lane);
                j = row_j(lane);
            }
        } else {
            if (m >= 2) {
                // the farthest bin offsets within reach
                const float rc = 2.f * norm_up(R2) * 1.0001f;
                const float rx_ = rc * inx + feps, ry_ = rc * iny + feps, rz_ = rc * inz + feps;
                const float far = fmaxf(fmaxf(rx_ + fx, rx_ + 1.f - fx), fmaxf(ry_ + fy, ry_ + 1.f - fy));
                if (m == 2 && !(far >= 2.f)) m = 3;
                // (batch 3 goes on once begun, while the ends are in reach: a point of it
                // that cuts leaves a face at half its distance, so twice the radius
                // reaches the ends still; ring 4 begins at its first row in any case)
                if (m == 3 && !(fmaxf(rz_ + fz, rz_ + 1.f - fz) >= (float)(kNearZ + 1))) {
                    m = 4;
                    ring0 = 0;
                }
                // a cell that a search radius leaves open reaches far: its rings end
                // with the radius (50,000 points, radius 0: 3.1 -> 0.6 ms)
                if (P.has_radius) m = radius_next(D, P.search_radius, m);
                if (m >= 4 && (!(far >= (float)m) || m >= cpd)) break;
            }
            if (m <= 2) {
                have = lane < (m == 1 ? 30 : 28);
                const uint32_t w = m == 1 ? plan : plan >> 16;
                i = (int8_t)w;
                j = (int8_t)(w >> 8);
            } else {
                const int w = far_row(m, ring0 + lane);
                have = w >= 0;
                i = (w >> 12) - 2048;
                j = (w & 4095) - 2048;
            }
        }
        const uint32_t from = __shfl_sync(FULL, pend, lane >> 1);
        const int x = cbx + i, y = cby + j;
        if (have && x >= 0 && x < cpd && y >= 0 && y < cpd) {
            int kl = cbz, kh = cbz;
            bool on = true;
            if (!SEED && m == 0) {
                if (lane < 9) {
                    kl = max(cbz - 1, 0);
                    kh = min(cbz + 1, cpd - 1);
                }
            } else {
                // distance to the row, each gap shortened by the in-bin
                // position's error bound, and what is left of the reach along z
                const float dx = fmaxf((i > 0 ? (float)i - fx : (i < 0 ? (float)(-i - 1) + fx : 0.f)) - feps, 0.f) * D.size_f[0];
                const float dy = fmaxf((j > 0 ? (float)j - fy : (j < 0 ? (float)(-j - 1) + fy : 0.f)) - feps, 0.f) * D.size_f[1];
                const float rem = 4.f * R2 * 1.0003f - (dx * dx + dy * dy);
                on = rem > 0.f;
                const float zr = fminf(norm_up(rem) * inz * 1.0001f + 2.f * feps, GEO ? 4e6f : 4096.f);
                kl = max((int)floorf(pz - zr), 0);
                kh = min((int)floorf(pz + zr), cpd - 1);
            }
            if (m == 1 || m == 2) {
                kl = max(kl, cbz - kNearZ);
                kh = min(kh, cbz + kNearZ);
            } else if (m == 3) {
                if (lane & 1) kl = max(kl, cbz + kNearZ + 1);
                else kh = min(kh, cbz - kNearZ - 1);
            }
            if (P.has_radius) {
                const int2 z = radius_row(D, P.search_radius, i, j, kl, kh, cbz);
                kl = z.x;
                kh = z.y;
            }
            if (SEED && m == 0) {
                kl = max(kl, cbz - 1);
                kh = min(kh, cbz + 1);
            }
            const bool central = m == 1 && lane < 18;
            if (central && !(lane & 1)) kh = min(kh, cbz - 2);            // below the 27 bins
            if (central && (lane & 1)) {                                  // above them, and the points not taken
                kl = min(cbz + 1, cpd - 1);
                kh = max(kh, kl);
            }
            if (on && kl <= kh) {
                const uint64_t row = D.bin_base + ((uint64_t)x * cpd + y) * cpd;
                bbeg = P.delims[tess_chk(row + kl, P.nbins, P.check, CK_BIN)];
                const uint32_t end = P.delims[tess_chk(row + kh, P.nbins, P.check, CK_BIN) + 1];
                if (central && (lane & 1) && from != 0xFFFFFFFFu) bbeg = from;
                bcnt = end > bbeg ? end - bbeg : 0u;
            }
        }
        if (m == 0) {
            // a crowded own bin sends the cell to the seeded pass
            if (!SEED && P.list_dense && __shfl_sync(FULL, bcnt, 9) >= P.seed_min) {
                status = ST_DENSE;
                break;
            }
            if (lane == 9) bcnt = 0;
        }
        // ---- its points as one stream, 32 per window ----
        const unsigned inc = warp_incl_scan_u(bcnt, lane);
        total = __shfl_sync(FULL, inc, 31);
        pref = inc - bcnt;
        if (m == 0) {
            // whole windows only; the rest joins the next batch
            if (total > 32) total &= ~31u;
            pend = bcnt ? bbeg + min(max((int)(total - pref), 0), (int)bcnt) : (SEED ? 0xFFFFFFFFu : bbeg);
        }
        // A cell with a long batch lies beside a cluster that it mostly does not
        // reach: the seeded pass leaves its points out by their support.  500,000
        // clustered points: plain pass 2.98 -> 1.28 ms, the others 15.4 -> 14.6.
        // (From 512 on, cells of two-species inputs go as well, and lose 2%;
        // uniform points have 125 a batch.)
        if (!SEED && P.list_dense && total >= 1024) {
            status = ST_DENSE;
            break;
        }
        // the batch after this one
        if (m < 3) {
            ++m;
        } else {
            ring0 += 32;
            if (ring0 >= (m == 3 ? 98 : 8 * m)) {
                ++m;
                ring0 = 0;
            }
        }
        if (total == 0) continue;
        if constexpr (COUNT) ++W.batches;
        {
            const unsigned nz = __ballot_sync(FULL, bcnt > 0);
            __syncwarp();                         // the last batch's offsets are read
            if (bcnt) S.boff[__popc(nz & lt)] = bbeg - pref;
        }
        }
        __syncwarp();
        unsigned before = 0;      // ranges that began in earlier windows
        // (a long batch: the cell lies beside a cluster)
        const bool bounded = SEED && (crowded || total >= 256);
        unsigned w0 = 0;
        do {
            __syncwarp();                         // the last window's candidates are read
            float rx, ry, rz, r2;
            uint32_t jp;
            bool keep, near;
            float lim = 4.f * R2 * (float)kStopMargin;
            // Seeded: the bounds of the cell's vertices and of their errors.  In
            // clusters most points within twice the radius lie where the cell
            // does not reach: a bisector beyond the box's support cannot touch
            // a vertex (clustered inputs: 260 points a cell are within twice
            // the radius, of which 22 cut).
            float bl0 = 0.f, bl1 = 0.f, bl2 = 0.f, bh0 = 0.f, bh1 = 0.f, bh2 = 0.f, be = 0.f;
            if constexpr (SEED) {
                if (bounded && !direct) {
                    float4 v = S.vtx[lane];
                    bool lv = (l0 >> lane) & 1u;
                    bl0 = bh0 = lv ? v.x : 0.f;      // the site is inside its bounds
                    bl1 = bh1 = lv ? v.y : 0.f;
                    bl2 = bh2 = lv ? v.z : 0.f;
                    be = lv ? v.w : 0.f;
                    if ((l1 >> lane) & 1u) {
                        v = S.vtx[32 + lane];
                        bl0 = fminf(bl0, v.x);
                        bh0 = fmaxf(bh0, v.x);
                        bl1 = fminf(bl1, v.y);
                        bh1 = fmaxf(bh1, v.y);
                        bl2 = fminf(bl2, v.z);
                        bh2 = fmaxf(bh2, v.z);
                        be = fmaxf(be, v.w);
                    }
                    // non-negative floats order like their bits
                    auto top = [](float x) { return __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(fmaxf(x, 0.f)))); };
                    bl0 = -top(-bl0);
                    bl1 = -top(-bl1);
                    bl2 = -top(-bl2);
                    bh0 = top(bh0);
                    bh1 = top(bh1);
                    bh2 = top(bh2);
                    be = top(be) + 1e-6f * norm_up(R2);   // and the support's own rounding
                }
            }
            auto reaches = [&](float x, float y, float z, float q2) {
                const float h = fmaxf(x * bl0, x * bh0) + fmaxf(y * bl1, y * bh1) + fmaxf(z * bl2, z * bh2);
                const float n = norm_up(q2);
                return h + fmaf(n, be + fmaf(gr, n, tol), eC) >= 0.5f * q2;
            };
            // 32 points of the stream, one per lane
            auto load = [&]() {
                const unsigned rel = pref - w0;
                const unsigned heads = __reduce_or_sync(FULL, (bcnt && rel < 32u) ? 1u << rel : 0u);
                const unsigned c = w0 + lane;
                keep = near = false;
                rx = ry = rz = r2 = 0.f;
                jp = 0;
                if (c < total) {
                    jp = tess_chk(S.boff[before + __popc(heads & (lt | (1u << lane))) - 1] + c, P.npts, P.check, CK_POINT);
                    const float4 h = P.phi[jp], l = P.plo[jp];
                    rx = (h.x - shx) + (l.x - slx);
                    ry = (h.y - shy) + (l.y - sly);
                    rz = (h.z - shz) + (l.z - slz);
                    r2 = rx * rx + ry * ry + rz * rz;
                    keep = jp != gs && r2 > dup2 && r2 < lim;
                    near = jp != gs && !(r2 > dup2);
                    if (keep && P.target_group >= 0) keep = (int64_t)(P.sgroup ? P.sgroup[jp] : 0u) == P.target_group;
                    if constexpr (SEED && MODE != kDense) keep = keep && (!bounded || reaches(rx, ry, rz, r2));
                }
                // (few of a crowded bin's 32 are within twice the radius, often none:
                // 2,097,152 clustered points, passes after the first: 47.0 -> 45.3
                // ms with this and the early end below; 44.1 with ranges read one
                // after the other, but inputs of 100,000 points 3% slower)
                if constexpr (MODE == kDense) {
                    if (bounded && __any_sync(FULL, keep)) keep = keep && reaches(rx, ry, rz, r2);
                }
                return heads;
            };
            if (direct) {
                rx = sx_;
                ry = sy_;
                rz = sz_;
                r2 = s2_;
                jp = sj_;
                keep = s2_ < lim;
                near = false;
                w0 += 32;
            } else if constexpr (SEED) {
                // gather the points within reach until the window is full
                // (crowded bins hold hundreds that are not)
                unsigned nk = 0;
                bool anynear = false;
                do {
                    const unsigned heads = load();
                    const unsigned kk = __ballot_sync(FULL, keep);
                    anynear |= near;
                    if (MODE == kDense && !kk) {
                        before += __popc(heads);
                        w0 += 32;
                        continue;
                    }
                    if (nk + __popc(kk) > 32u) break;
                    if (keep) {
                        const unsigned at = nk + __popc(kk & lt);
                        S.cand[at] = make_float4(rx, ry, rz, r2);
                        S.candj[at] = jp;
                    }
                    nk += __popc(kk);
                    before += __popc(heads);
                    w0 += 32;
                } while (w0 < total && nk < 24u);
                __syncwarp();
                near = anynear;
                keep = (unsigned)lane < nk;
                const float4 own = S.cand[lane];
                rx = own.x;
                ry = own.y;
                rz = own.z;
                r2 = own.w;
                jp = S.candj[lane];
                // (a seed that cut is a plane already)
                if (crowded)
#pragma unroll 1
                    for (int p = 6; p < np; ++p) keep = keep && S.psrc[p] != jp;
                __syncwarp();
            } else {
                before += __popc(load());
                w0 += 32;
            }
            // (near-)coincident points are decided in FP64
            if (__any_sync(FULL, near)) {
                status = ST_NEAR;
                break;
            }
            unsigned km = __ballot_sync(FULL, keep);      // candidates within reach
            if constexpr (COUNT) {
                ++W.windows;
                W.tested += (unsigned)__popc(km);
            }
            if (!km) continue;
            const float rn = norm_up(r2), off = 0.5f * r2;
            const float c0 = fmaf(rn, fmaf(gr, rn, tol), eC);
            uint32_t t0, t1 = 0;                          // my candidate's touched slots
            {
                // 2^sh lanes per candidate, each testing every 2^sh-th slot
                const int rk = __popc(km & lt);
                if (keep) {
                    S.cand[rk] = make_float4(rx, ry, rz, off);
                    S.candn[rk] = rn;
                }
                __syncwarp();
                const int sh = __clz(__popc(km) - 1) - 27;
                const float4 n = S.cand[lane >> sh];
                const float nn = S.candn[lane >> sh];
                const float cc = fmaf(nn, fmaf(gr, nn, tol), eC);
                const int g = 1 << sh, v0 = lane & (g - 1);
                // (two slots per turn; the one past the last is masked off, and
                // v0 + g * turn stays below 64)
                const int turns = (32 - __clz(l0) + g - 1) >> sh;
                const float4* vp = S.vtx + v0;
                uint32_t u0 = 0, bit = 1u << v0;
#pragma unroll 1
                for (int k = 0; k < turns; k += 2) {
                    const float4 va = vp[0], vb = vp[g];
                    if (touched(va, n.x, n.y, n.z, n.w, nn, cc)) u0 |= bit;
                    bit = g < 32 ? bit << g : 0u;
                    if (touched(vb, n.x, n.y, n.z, n.w, nn, cc)) u0 |= bit;
                    bit = g < 32 ? bit << g : 0u;
                    vp += 2 * g;
                }
#pragma unroll 1
                for (int o = 1; o < g; o <<= 1) u0 |= __shfl_xor_sync(FULL, u0, o);
                t0 = __shfl_sync(FULL, u0, rk << sh);
                if (l1) {
                    uint32_t u1 = 0;
#pragma unroll 1
                    for (int v = v0; v < 32; v += g)
                        if (touched(S.vtx[32 + v], n.x, n.y, n.z, n.w, nn, cc)) u1 |= 1u << v;
#pragma unroll 1
                    for (int o = 1; o < g; o <<= 1) u1 |= __shfl_xor_sync(FULL, u1, o);
                    t1 = __shfl_sync(FULL, u1, rk << sh);
                }
            }
            // Nearest first: the closest candidate that may cut, by a warp
            // minimum of its distance (top 27 bits of r2, ties by lane).
            int decided = -1;        // careful: a candidate whose undecided tests were settled
            const unsigned mykey = (__float_as_uint(r2) & ~31u) | (unsigned)lane;
            for (;;) {
                const bool act = keep && r2 < lim && ((t0 & l0) | (t1 & l1)) != 0;
                const unsigned best = __reduce_min_sync(FULL, act ? mykey : 0xFFFFFFFFu);
                if (best == 0xFFFFFFFFu) break;
                const int src = (int)(best & 31u);
                int f = np;
                if constexpr (SEED) {
                    if (f >= kPlanes) {
                        // the table is full: an id that no live vertex has any
                        // more (planes cut away entirely leave them behind)
                        __syncwarp();             // the last cut's vertices are written
                        uint32_t u0 = 0x3Fu, u1 = 0, u2 = 0;       // the walls stay
#pragma unroll 1
                        for (int k = 0; k < 2; ++k)
                            if (((k ? l1 : l0) >> lane) & 1u) {
                                const uint32_t tt = S.topo[32 * k + lane].x;
#pragma unroll 1
                                for (int e = 0; e < 3; ++e) {
                                    const int p = byte_of(tt, e);
                                    if (p < 32) u0 |= 1u << p;
                                    else if (p < 64) u1 |= 1u << (p - 32);
                                    else u2 |= 1u << (p - 64);
                                }
                            }
                        u0 = ~__reduce_or_sync(FULL, u0);
                        u1 = ~__reduce_or_sync(FULL, u1);
                        u2 = ~__reduce_or_sync(FULL, u2);
                        f = u0 ? __ffs(u0) - 1 : (u1 ? 31 + __ffs(u1) : (u2 ? 63 + __ffs(u2) : kPlanes));
                    }
                }
                if (lane == src) {
                    S.pl[f] = make_float4(rx, ry, rz, off);
                    S.pn[f] = rn;
                    S.psrc[f] = jp;
                    keep = false;
                }
                km &= ~(1u << src);
                const uint32_t o0 = __shfl_sync(FULL, t0, src) & l0, o1 = __shfl_sync(FULL, t1, src) & l1;
                // ---- cut by plane f: the Outside slots are o0, o1 ----
                if (f >= kPlanes) {
                    status = ST_PCAP;
                    break;
                }
                gen = (gen + 1) & 0xFFu;
                if (gen == 0) {
                    __syncwarp();                 // the last cut's ring is read
#pragma unroll 1
                    for (int i = lane; i < kPlanes; i += 32) S.map[i] = 0;
                    gen = 1;
                }
                // the Outside slots go onto the free-slot stack; the new
                // vertices pop theirs from its top
                const int base = nfree;
                const int R0 = __popc(o0), R = R0 + __popc(o1);
                if ((o0 >> lane) & 1u) S.fl[base + __popc(o0 & lt)] = (uint8_t)lane;
                if ((o1 >> lane) & 1u) S.fl[base + R0 + __popc(o1 & lt)] = (uint8_t)(32 + lane);
                __syncwarp();
                const float4 pf = S.pl[f];
                const float nf = S.pn[f], cf = fmaf(nf, fmaf(gr, nf, tol), eC);
                // an edge of an Outside vertex whose neighbour is not Outside
                // gets a new vertex: one lane per edge, or (large cuts) one
                // lane per listed boundary edge
                int a = 0, b = 0, y = 0, q = 0, B;      // y: the neighbour's slot | edge index << 6
                bool bnd = false, und = false;           // und: a touched vertex in the guard band
                auto edge = [&](int x, int e) {
                    const uint2 tp = S.topo[x];
                    a = byte_of(tp.x, e);
                    b = byte_of(tp.x, e == 2 ? 0 : e + 1);
                    y = byte_of(tp.y, e);
                    return !(((y & 32 ? o1 : o0) >> (y & 31)) & 1u);
                };
                if (3 * R <= 32) {
                    if (lane < 3 * R) {
                        const int xi = (lane * 11) >> 5;          // lane / 3 for lane < 32
                        const int x = S.fl[base + xi];
                        bnd = edge(x, lane - 3 * xi);
                        float sd, band;
                        plane_test(S.vtx[x], pf.x, pf.y, pf.z, pf.w, nf, cf, sd, band);
                        und = sd <= band && (!CAREFUL || src != decided);
                    }
                    const unsigned bm = __ballot_sync(FULL, bnd);
                    B = __popc(bm);
                    q = __popc(bm & lt);
                } else {
                    B = 0;
#pragma unroll 1
                    for (int r0 = 0; r0 < 3 * R; r0 += 32) {
                        const int ei = r0 + lane;
                        bool bd = false;
                        int x = 0, e = 0;
                        if (ei < 3 * R) {
                            x = S.fl[base + ei / 3];
                            e = ei % 3;
                            bd = edge(x, e);
                            float sd, band;
                            plane_test(S.vtx[x], pf.x, pf.y, pf.z, pf.w, nf, cf, sd, band);
                            und |= sd <= band && (!CAREFUL || src != decided);
                        }
                        const unsigned bm = __ballot_sync(FULL, bd);
                        const int at = B + __popc(bm & lt);
                        if (bd && at < 32) S.items[at] = (uint16_t)(x | (e << 8));
                        B += __popc(bm);
                    }
                    __syncwarp();
                    bnd = lane < B;
                    q = lane;
                    if (bnd && B <= 32) {
                        const int it = S.items[lane];
                        edge(it & 0xFF, it >> 8);
                    }
                }
                if (__any_sync(FULL, und)) {
                    if constexpr (!CAREFUL) {
                        status = ST_GUARD;
                        break;
                    }
                    undec = true;
                    if (!GEO && ++settled > P.settle_most) {
                        status = ST_GUARD;
                        break;
                    }
                    // settle the touched vertices in FP64, one lane each, and
                    // choose again
                    uint32_t d0 = 0, d1 = 0;
                    bool fail = false;
                    for (int r0 = 0; r0 < R; r0 += 32) {
                        if (r0 + lane < R) {
                            const int x = S.fl[base + r0 + lane];
                            float sd, band;
                            plane_test(S.vtx[x], pf.x, pf.y, pf.z, pf.w, nf, cf, sd, band);
                            int side = 1;
                            if (sd <= band) side = side_fp64(S, P, D, gs, S.topo[x].x, tess_chk(S.psrc[f], P.npts, P.check, CK_POINT));
                            fail |= side < 0;
                            if (side > 0 && x < 32) d0 |= 1u << x;
                            if (side > 0 && x >= 32) d1 |= 1u << (x - 32);
                        }
                    }
                    if (__any_sync(FULL, fail)) {
                        status = ST_GUARD;
                        break;
                    }
                    d0 = __reduce_or_sync(FULL, d0);
                    d1 = __reduce_or_sync(FULL, d1);
                    if (lane == src) {
                        t0 = d0;
                        t1 = d1;
                        keep = true;
                    }
                    km |= 1u << src;
                    decided = src;
                    __syncwarp();
                    continue;
                }
                decided = -1;
                if constexpr (COUNT) {
                    ++W.cuts;
                    W.newv += (unsigned)B;
                }
                // more vertices than lanes or free slots: the larger forms
                if (B > 32 || B > base + R) {
                    status = ST_VCAP;
                    break;
                }
                int slot = 0;
                bool bad = false;
                const uint32_t tag = gen << 8;
                uint32_t n0 = 0, n1 = 0;
                if (bnd) {
                    // the vertex of planes (a, b, f) by Cramer's rule; its error
                    // depends on its own conditioning only
                    const float4 pa = S.pl[a], pb = S.pl[b];
                    const float bfx = pb.y * pf.z - pb.z * pf.y, bfy = pb.z * pf.x - pb.x * pf.z, bfz = pb.x * pf.y - pb.y * pf.x;
                    const float fax = pf.y * pa.z - pf.z * pa.y, fay = pf.z * pa.x - pf.x * pa.z, faz = pf.x * pa.y - pf.y * pa.x;
                    const float abx = pa.y * pb.z - pa.z * pb.y, aby = pa.z * pb.x - pa.x * pb.z, abz = pa.x * pb.y - pa.y * pb.x;
                    const float det = pa.x * bfx + pa.y * bfy + pa.z * bfz;
                    const float inv = rcp_ftz(det);
                    const float px = (pa.w * bfx + pb.w * fax + pf.w * abx) * inv;
                    const float py = (pa.w * bfy + pb.w * fay + pf.w * aby) * inv;
                    const float pz = (pa.w * bfz + pb.w * faz + pf.w * abz) * inv;
                    const float x1 = fabsf(px) + fabsf(py) + fabsf(pz);
                    float pe = kVertexErr * x1 * (S.pn[a] * S.pn[b] * nf) * fabsf(inv);
                    // singular (or nearly): not a vertex to go on from
                    // (careful: beyond 0.03 the first-order bound is no bound)
                    bad = CAREFUL ? !(pe <= 0.03f * x1) : !(pe < 1e30f);
                    pe += gr * x1;
                    slot = tess_chk((int)S.fl[base + R - 1 - q], kSlots, P.check, CK_SLOT);
                    S.vtx[slot] = S.nv[q] = make_float4(px, py, pz, pe);
                    S.nvs[q] = (uint8_t)slot;
                    S.vr[slot] = vertex_r2(px, py, pz, pe);
                    // Y's edge back to X now leads to the new vertex's edge 0
                    reinterpret_cast<uint8_t*>(&S.topo[y & 63].y)[y >> 6] = (uint8_t)slot;
                    uint16_t* const mp = reinterpret_cast<uint16_t*>(S.map);
                    mp[2 * a] = (uint16_t)(tag | (uint32_t)slot);
                    mp[2 * b + 1] = (uint16_t)(tag | (uint32_t)slot);
                    if (slot & 32) n1 = 1u << (slot & 31);
                    else n0 = 1u << slot;
                }
                n0 = __reduce_or_sync(FULL, n0);
                n1 = ((l1 | o1) != 0 || __any_sync(FULL, n1 != 0)) ? __reduce_or_sync(FULL, n1) : 0u;
                __syncwarp();
                if (bnd) {
                    // the ring: across (b, f) lies the new vertex whose first
                    // plane is b (its edge 2), across (f, a) the one whose second
                    // plane is a (its edge 1); both from this cut, and the two
                    // planes know this vertex in turn
                    const uint32_t me = tag | (uint32_t)slot;
                    const uint32_t wb = S.map[b], wa = S.map[a];
                    bad |= ((wb ^ (me << 16 | tag)) & 0xFFFFFF00u) != 0 || ((wa ^ (tag << 16 | me)) & 0xFF00FFFFu) != 0;
                    S.topo[slot] = make_uint2((uint32_t)a | ((uint32_t)b << 8) | ((uint32_t)f << 16),
                                              (uint32_t)y | ((wb & 0x3Fu | 2u << 6) << 8) | (wa & 0x3F0000u) | 1u << 22);
                }
                l0 = (l0 & ~o0) | n0;
                l1 = (l1 & ~o1) | n1;
                nfree = base + R - B;
                np = SEED ? max(np, f + 1) : f + 1;
                // the smaller cell's radius, and the new vertices against the
                // waiting candidates
                float rr = ((l0 >> lane) & 1u) ? S.vr[lane] : 0.f;
                if ((l1 >> lane) & 1u) rr = fmaxf(rr, S.vr[32 + lane]);
                const float R2b = R2;
                R2 = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(rr)));
                // a cut moves no vertex beyond the cell: a radius that grew
                // means a wrong vertex
                if constexpr (CAREFUL) bad |= !(R2 <= R2b * 1.001f);
                if (km) {
                    t0 &= ~n0;
                    t1 &= ~n1;
                    if (!n1) {
#pragma unroll 1
                        for (int q0 = 0; q0 < B; q0 += 4) {
                            const uint32_t sl = *reinterpret_cast<const uint32_t*>(S.nvs + q0);
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                if (touched(S.nv[q0 + k], rx, ry, rz, off, rn, c0) && q0 + k < B) t0 |= 1u << byte_of(sl, k);
                        }
                    } else {
#pragma unroll 1
                        for (int k = 0; k < B; ++k) {
                            const int s = S.nvs[k];
                            const bool hit = touched(S.nv[k], rx, ry, rz, off, rn, c0);
                            if (hit && s < 32) t0 |= 1u << s;
                            if (hit && s >= 32) t1 |= 1u << (s - 32);
                        }
                    }
                }
                lim = 4.f * R2 * (float)kStopMargin;
                if (__any_sync(FULL, bad)) {
                    status = ST_DEGEN;
                    break;
                }
            }
            if (status != ST_OK) break;
        } while (w0 < total);
    }

    // ---- finalize: faces, areas, volume (polyhedron.rs:776-855) ----
    uint8_t* const fsta = EXACT ? S.d.fsta : S.s.fsta;
    uint8_t* const face = EXACT ? S.d.face : S.s.face;
    uint8_t* const rank = EXACT ? S.d.rank : S.s.rank;
    int32_t* const ids = EXACT ? S.d.ids : S.s.ids;
    const int nlive = __popc(l0) + __popc(l1);
    double vol = 0.0;
    int F = 0;
    if (status == ST_OK) {
        __syncwarp();
        if (lane < kPlanes / 4) reinterpret_cast<uint32_t*>(fsta)[lane] = 0xFFFFFFFFu;
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (((k ? l1 : l0) >> lane) & 1u) {
                const uint32_t tt = S.topo[32 * k + lane].x;
#pragma unroll
                for (int e = 0; e < 3; ++e) fsta[byte_of(tt, e)] = (uint8_t)(32 * k + lane + 64 * e);
            }
        }
        __syncwarp();
        // the planes that have a face, in plane order, and their equations:
        // the bisector of the site and point q has n = q = p_j - site and
        // h = q.q / 2 (vector3.rs:223-239 up to the scale of n).
#pragma unroll 1
        for (int p0 = 0; p0 < np; p0 += 32) {
            const int p = p0 + lane;
            const bool has = p < np && fsta[p] != 0xFFu;
            const unsigned m = __ballot_sync(FULL, has);
            if (has) {
                const int at = F + __popc(m & lt);
                face[at] = (uint8_t)p;
                int32_t id = -1 - p;   // -1 x_min, -2 x_max, -3 y_min, -4 y_max, -5 z_min, -6 z_max
                if constexpr (EXACT) {
                    double qx, qy, qz, qh;
                    if (p < 6) {
                        const int a = p >> 1;
                        const bool mx = p & 1;
                        qh = wall_distance(P, D, gs, p);
                        qx = a == 0 ? (mx ? 1.0 : -1.0) : 0.0;
                        qy = a == 1 ? (mx ? 1.0 : -1.0) : 0.0;
                        qz = a == 2 ? (mx ? 1.0 : -1.0) : 0.0;
                    } else {
                        const uint32_t j = tess_chk(S.psrc[p], P.npts, P.check, CK_POINT);
                        id = (int32_t)(__float_as_uint(P.phi[j].w) - pt_base);
                        qx = P.spx[j] - site_coord(P, gs, 0);
                        qy = P.spy[j] - site_coord(P, gs, 1);
                        qz = P.spz[j] - site_coord(P, gs, 2);
                        qh = 0.5 * (qx * qx + qy * qy + qz * qz);
                    }
                    S.d.qa[p] = make_double2(qx, qy);
                    S.d.qb[p] = make_double2(qz, qh);
                } else {
                    // as FP32 pairs without the FP64 pipe: q by a TwoSum of the
                    // points' high parts (error ~2^-46 of the distance from the
                    // centre), h in double-float.  Walls keep an FP64 distance.
                    float q0, q1, q2, e0 = 0.f, e1 = 0.f, e2 = 0.f, hh, hl, dist;
                    if (p < 6) {
                        const int a = p >> 1;
                        const bool mx = p & 1;
                        const double h = wall_distance(P, D, gs, p);
                        hh = (float)h;
                        hl = (float)(h - (double)hh);
                        q0 = a == 0 ? (mx ? 1.f : -1.f) : 0.f;
                        q1 = a == 1 ? (mx ? 1.f : -1.f) : 0.f;
                        q2 = a == 2 ? (mx ? 1.f : -1.f) : 0.f;
                        dist = hh;
                    } else {
                        const uint32_t j = tess_chk(S.psrc[p], P.npts, P.check, CK_POINT);
                        const float4 h = P.phi[j], l = P.plo[j];
                        id = (int32_t)(__float_as_uint(h.w) - pt_base);
                        float sh, se;
                        two_sum(h.x, -shx, sh, se);
                        two_sum(sh, (l.x - slx) + se, q0, e0);
                        two_sum(h.y, -shy, sh, se);
                        two_sum(sh, (l.y - sly) + se, q1, e1);
                        two_sum(h.z, -shz, sh, se);
                        two_sum(sh, (l.z - slz) + se, q2, e2);
                        float p0_, r0, p1, r1, p2, r2_, s01, t01, s2, t2;
                        two_prod(q0, q0, p0_, r0);
                        two_prod(q1, q1, p1, r1);
                        two_prod(q2, q2, p2, r2_);
                        two_sum(p0_, p1, s01, t01);
                        two_sum(s01, p2, s2, t2);
                        const float low = ((r0 + r1) + r2_) + (t01 + t2) + 2.f * (q0 * e0 + q1 * e1 + q2 * e2);
                        float H, HL;
                        two_sum(s2, low, H, HL);
                        hh = 0.5f * H;   // exact scalings
                        hl = 0.5f * HL;
                        dist = 0.5f * sqrtf(H);
                    }
                    S.s.q[p] = make_float4(q0, q1, q2, hh);
                    S.s.ql[p] = make_float4(e0, e1, e2, hl);
                    S.s.dist[p] = dist;
                }
                ids[at] = id;
            }
            F += __popc(m);
        }
        if (lane < 3) ids[F + lane] = 0x7FFFFFFF;   // the ranks read groups of four
        __syncwarp();
        // FP32: one Newton step per vertex, residuals of its three planes in
        // double-float, the correction solved in FP32 by Cramer's rule.  FP64
        // finish: the same step in FP64.  A vertex that moves beyond its error
        // bound was not trustworthy: the cell re-runs.
        auto resid = [&](const float4& h, const float4& l, float x, float y, float z) -> float {
            float p0, e0, p1, e1, p2, e2, s1, t1_, s2, t2, s3, t3;
            two_prod(h.x, x, p0, e0);
            two_prod(h.y, y, p1, e1);
            two_prod(h.z, z, p2, e2);
            two_sum(h.w, -p0, s1, t1_);
            two_sum(s1, -p1, s2, t2);
            two_sum(s2, -p2, s3, t3);
            const float low = ((l.w - e0) - e1) - e2 + ((t1_ + t2) + t3) - (l.x * x + l.y * y + l.z * z);
            return s3 + low;
        };
        const float vlim = P.verify_rel * sqrtf(R2);
        bool vbad = false;
#pragma unroll 1
        for (int k = 0; k < (l1 ? 2 : 1); ++k) {
            if (((k ? l1 : l0) >> lane) & 1u) {
                const int s = 32 * k + lane;
                const uint32_t tt = S.topo[s].x;
                const int a = byte_of(tt, 0), b = byte_of(tt, 1), c = byte_of(tt, 2);
                const float4 v = S.vtx[s];
                float ddx, ddy, ddz;
                if constexpr (EXACT) {
                    const double2 a0 = S.d.qa[a], a1 = S.d.qb[a], b0 = S.d.qa[b], b1 = S.d.qb[b], c0_ = S.d.qa[c], c1 = S.d.qb[c];
                    const double bcx = b0.y * c1.x - b1.x * c0_.y, bcy = b1.x * c0_.x - b0.x * c1.x, bcz = b0.x * c0_.y - b0.y * c0_.x;
                    const double cax = c0_.y * a1.x - c1.x * a0.y, cay = c1.x * a0.x - c0_.x * a1.x, caz = c0_.x * a0.y - c0_.y * a0.x;
                    const double abx = a0.y * b1.x - a1.x * b0.y, aby = a1.x * b0.x - a0.x * b1.x, abz = a0.x * b0.y - a0.y * b0.x;
                    const double inv = recip_nr(a0.x * bcx + a0.y * bcy + a1.x * bcz);
                    // the residuals at the FP32 vertex, and the step that removes
                    // them: its error is the residuals' rounding (solving for
                    // the vertex itself loses 1 / det of it: 2e-12 of a thin
                    // cell's volume against 1e-15)
                    const double vx = v.x, vy = v.y, vz = v.z;
                    const double ra = a1.y - (a0.x * vx + a0.y * vy + a1.x * vz);
                    const double rb = b1.y - (b0.x * vx + b0.y * vy + b1.x * vz);
                    const double rc = c1.y - (c0_.x * vx + c0_.y * vy + c1.x * vz);
                    const double ex = (ra * bcx + rb * cax + rc * abx) * inv;
                    const double ey = (ra * bcy + rb * cay + rc * aby) * inv;
                    const double ez = (ra * bcz + rb * caz + rc * abz) * inv;
                    S.d.rx[s] = vx + ex;
                    S.d.ry[s] = vy + ey;
                    S.d.rz[s] = vz + ez;
                    ddx = (float)ex;
                    ddy = (float)ey;
                    ddz = (float)ez;
                } else {
                    const float4 ha = S.s.q[a], hb = S.s.q[b], hc = S.s.q[c];
                    const float ra = resid(ha, S.s.ql[a], v.x, v.y, v.z);
                    const float rb = resid(hb, S.s.ql[b], v.x, v.y, v.z);
                    const float rc = resid(hc, S.s.ql[c], v.x, v.y, v.z);
                    const float bcx = hb.y * hc.z - hb.z * hc.y, bcy = hb.z * hc.x - hb.x * hc.z, bcz = hb.x * hc.y - hb.y * hc.x;
                    const float cax = hc.y * ha.z - hc.z * ha.y, cay = hc.z * ha.x - hc.x * ha.z, caz = hc.x * ha.y - hc.y * ha.x;
                    const float abx = ha.y * hb.z - ha.z * hb.y, aby = ha.z * hb.x - ha.x * hb.z, abz = ha.x * hb.y - ha.y * hb.x;
                    const float inv = rcp_ftz(ha.x * bcx + ha.y * bcy + ha.z * bcz);
                    ddx = (ra * bcx + rb * cax + rc * abx) * inv;
                    ddy = (ra * bcy + rb * cay + rc * aby) * inv;
                    ddz = (ra * bcz + rb * caz + rc * abz) * inv;
                    S.s.dv[s] = make_float4(ddx, ddy, ddz, 0.f);
                }
                const float vl = 2.0f * v.w + vlim;
                if (!(fabsf(ddx) <= vl && fabsf(ddy) <= vl && fabsf(ddz) <= vl)) vbad = true;
            }
        }
        __syncwarp();
        // each face: walk its vertices, rank its id
        bool bad = false;
        double vpart = 0.0;
        unsigned nsteps = 0;
#pragma unroll 1
        for (int i0 = 0; i0 < F; i0 += 32) {
            const int i = i0 + lane;
            if (i < F) {
                const int p = face[i];
                // walk: from a vertex with p at place e across its edge e; there
                // the edge is number k and p at place k + 1
                const int st = fsta[p];
                const int start = st & 63;
                int at = st, steps = 0;
                auto next = [&]() -> int {
                    const int w = byte_of(S.topo[at & 63].y, at >> 6);
                    at = w + 64 >= 192 ? w - 128 : w + 64;
                    return w & 63;
                };
                if constexpr (EXACT) {
                    // The area from the face's projection on the plane normal to
                    // the dominant axis m of its normal (shoelace): w_m = 2 A
                    // q_m / |q|; the pyramid from the site is qh w_m / (6 q_m).
                    const double2 qa = S.d.qa[p], qb = S.d.qb[p];
                    const double q0 = qa.x, q1 = qa.y, q2 = qb.x;
                    const int m = (fabs(q0) >= fabs(q1) && fabs(q0) >= fabs(q2)) ? 0 : (fabs(q1) >= fabs(q2) ? 1 : 2);
                    const double* X1 = m == 0 ? S.d.ry : (m == 1 ? S.d.rz : S.d.rx);
                    const double* X2 = m == 0 ? S.d.rz : (m == 1 ? S.d.rx : S.d.ry);
                    const double qm = m == 0 ? q0 : (m == 1 ? q1 : q2);
                    const double a1 = X1[start], a2 = X2[start];
                    double u1 = 0.0, u2 = 0.0, wm = 0.0;
#pragma unroll 1
                    do {
                        const int nx = next();
                        const double v1 = X1[nx] - a1, v2 = X2[nx] - a2;
                        if (steps > 0) wm += v1 * u2 - v2 * u1;
                        u1 = v1;
                        u2 = v2;
                        ++steps;
                    } while (at != st && steps <= kSlots);
                    const double inv_qm = 1.0 / qm;
                    S.d.area[i] = 0.5 * wm * inv_qm * sqrt(q0 * q0 + q1 * q1 + q2 * q2);
                    vpart += qb.y * wm * inv_qm * 0.5;
                } else {
                    // fan from the first vertex on refined positions:
                    // (x - anchor) = (x32 - a32) + (dx - da)
                    const float4 va = S.vtx[start], da = S.s.dv[start];
                    float ux = 0.f, uy = 0.f, uz = 0.f, wx = 0.f, wy = 0.f, wz = 0.f;
#pragma unroll 1
                    do {
                        const int nx = next();
                        const float4 v = S.vtx[nx], dd = S.s.dv[nx];
                        const float vx = (v.x - va.x) + (dd.x - da.x);
                        const float vy = (v.y - va.y) + (dd.y - da.y);
                        const float vz = (v.z - va.z) + (dd.z - da.z);
                        if (steps > 0) {
                            wx += uy * vz - uz * vy;
                            wy += uz * vx - ux * vz;
                            wz += ux * vy - uy * vx;
                        }
                        ux = vx;
                        uy = vy;
                        uz = vz;
                        ++steps;
                    } while (at != st && steps <= kSlots);
                    const float area = 0.5f * sqrtf(wx * wx + wy * wy + wz * wz);
                    S.s.area[i] = area;
                    vpart += (double)(area * S.s.dist[p]);
                }
                bad |= at != st || steps < 3;
                nsteps += (unsigned)steps;
                if constexpr (GEO) S.psrc[i] = (uint32_t)steps;
                const int32_t my = ids[i];
                int rk = 0;
#pragma unroll 1
                for (int o = 0; o < F; o += 4) {
                    const int4 v = *reinterpret_cast<const int4*>(ids + o);
                    rk += (v.x < my) + (v.y < my) + (v.z < my) + (v.w < my);
                }
                rank[i] = (uint8_t)rk;
            }
        }
        // every vertex lies on three faces, each walk closes, and V - E + F = 2
        nsteps = __reduce_add_sync(FULL, nsteps);
        vol = EXACT ? warp_sum_d(vpart) / 3.0 : warp_sum_d(vpart) * (1.0 / 3.0);
        if (nsteps != 3u * (unsigned)nlive || (nlive > 0 && F != nlive / 2 + 2)) bad = true;
        if (__any_sync(FULL, bad)) status = ST_DEGEN;
        else if (__any_sync(FULL, vbad)) status = ST_VERIFY;
    }

    // ---- outputs ----
    if constexpr (GEO) {
        GeoOut& G = *P.geo;
        if (lane == 0) {
            G.status = status;
            G.nv = nlive;
            G.nf = F;
            G.volume = vol;
            G.face_off[0] = 0;
        }
        if (status != ST_OK) return;
        __syncwarp();
        // vertices: the live slots in slot order
        auto number = [&](int s) { return s < 32 ? __popc(l0 & ((1u << s) - 1u)) : __popc(l0) + __popc(l1 & ((1u << (s - 32)) - 1u)); };
#pragma unroll 1
        for (int k = 0; k < 2; ++k)
            if (((k ? l1 : l0) >> lane) & 1u) {
                const int s = 32 * k + lane, v = tess_chk(number(s), 256, P.check, CK_SLOT);
                G.verts[3 * v] = S.d.rx[s];
                G.verts[3 * v + 1] = S.d.ry[s];
                G.verts[3 * v + 2] = S.d.rz[s];
            }
        // faces by id, a lane each; the reversed walk is counter-clockwise
        // seen from outside
#pragma unroll 1
        for (int i = lane; i < F; i += 32) {
            const int r = tess_chk((int)rank[i], 256, P.check, CK_FACE), deg = (int)S.psrc[i];
            int o = 0;
#pragma unroll 1
            for (int q = 0; q < F; ++q) o += rank[q] < r ? (int)S.psrc[q] : 0;
            G.face_nbr[r] = ids[i];
            G.face_area[r] = S.d.area[i];
            G.face_off[r + 1] = o + deg;
            int at = fsta[face[i]];
#pragma unroll 1
            for (int k = 0; k < deg; ++k) {
                G.face_vtx[tess_chk(o + (k ? deg - k : 0), 3 * 256, P.check, CK_FACE)] = number(at & 63);
                const int w = byte_of(S.topo[at & 63].y, at >> 6);
                at = w + 64 >= 192 ? w - 128 : w + 64;
            }
        }
        return;
    }
    if constexpr (CAREFUL) {
        // as the first pass, it counts what the plain pass would hand on
        if (lane == 0 && !P.work) {
            if (crowded) atomicAdd(P.list_dense_count, 1u);
            else if (undec || status == ST_GUARD || status == ST_NEAR || status == ST_DEGEN || status == ST_VERIFY) atomicAdd(P.flag_count, 1u);
        }
    }
    if (status != ST_OK) {
        if (lane == 0) {
            uint32_t* list = nullptr;
            unsigned* count = nullptr;
            if (P.reasons) atomicAdd(&P.reasons[status == ST_NEAR ? ST_GUARD : status], 1u);
            if (status == ST_GUARD || status == ST_DEGEN || status == ST_VERIFY) {
                list = P.list_fp64;
                count = P.list_fp64_count;
            } else if (status == ST_NEAR) {
                // the careful pass would meet the same point
                list = P.list_near;
                count = P.list_near_count;
                if (!CAREFUL) atomicAdd(P.flag_count, 1u);
            } else if (status == ST_DENSE) {
                list = P.list_dense;
                count = P.list_dense_count;
            } else {
                list = P.list_cap;
                count = P.list_cap_count;
            }
            if (list) {
                list[tess_chk(atomicAdd(count, 1u), P.npts, P.check, CK_LIST)] = gs;
                P.status[orig] = ST_PENDING;
            } else {
                P.status[orig] = (uint8_t)status;
                P.vol[orig] = 0.0;
                P.nface[orig] = 0;
                atomicAdd(P.fail_count, 1u);
            }
        }
        __syncwarp();
        return;
    }
    unsigned long long fbase = 0;
    if (lane == 0) fbase = atomicAdd(P.face_cursor, (unsigned long long)F);
    fbase = __shfl_sync(FULL, fbase, 0);
    if (fbase + F > P.face_cap) {
        if (lane == 0) {
            P.status[orig] = ST_POOL;
            P.nface[orig] = 0;
        }
        __syncwarp();
        return;   // the host sees the face cursor past the capacity and recomputes
    }
#pragma unroll 1
    for (int i = lane; i < F; i += 32) {
        const unsigned long long fi = tess_chk(fbase + rank[i], P.face_cap, P.check, CK_FACE);
        P.face_nbr[fi] = ids[i];
        P.face_area[fi] = EXACT ? S.d.area[i] : (double)S.s.area[i];
    }
    if (lane == 0) {
        P.vol[orig] = vol;
        P.nface[orig] = (uint32_t)F;
        P.fstart[orig] = fbase;
        P.status[orig] = ST_OK;
    }
    __syncwarp();
}

// 4 warps per block, five blocks per SM: 96 registers, no spills.  At
// 1,000,000 uniform points: 13.3 ms with 16 warps per SM, 11.9 with 20, 12.4
// with 24 (80 registers, 19% more instructions and the instruction cache full).
template <bool EXACT, int MODE>
__global__ void __launch_bounds__(128, MODE == kCareful ? 4 : 5) k_lean(ClipParams P) {
    after_previous();
    extern __shared__ __align__(16) unsigned char smraw[];
    Lean& S = reinterpret_cast<Lean*>(smraw)[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    if (P.grid_err && *P.grid_err == 1) return;   // non-finite input: nothing to clip
    for (int i = lane; i < kPlanes; i += 32) S.map[i] = 0;
    const uint32_t plan = row_plan(lane);
    uint32_t gen = 0;
    Work W;
    int d = 0;                                    // diagram of the last cell
    const unsigned total = P.work_count ? *P.work_count : P.total;
    if constexpr (MODE == kCareful) {
        // most cells undecided (lattices): all of them are the FP64 clipping's (a simple
        // cubic one of 125,000 points: 20.5 -> 4.8 ms; moved by 1e-4: 7.9 -> 6.4)
        if (P.work_count && total > P.work_most) {
            for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < ((total + 31u) & ~31u); i += gridDim.x * blockDim.x) {
                unsigned at = 0;
                if (lane == 0) at = atomicAdd(P.list_fp64_count, min(32u, total - i));
                at = __shfl_sync(FULL, at, 0) + lane;
                if (i < total) P.list_fp64[tess_chk(at, P.npts, P.check, CK_LIST)] = P.work[i];
            }
            return;
        }
    }
    // the next cell's number is fetched while a cell is worked on
    unsigned w = 0;
    if (lane == 0) w = atomicAdd(P.cursor, 1u);
    w = __shfl_sync(FULL, w, 0);
    while (w < total) {
        unsigned wn = 0;
        if (lane == 0) wn = atomicAdd(P.cursor, 1u);
        const uint32_t gs = P.work ? P.work[w] : w;
        if (P.ndiag > 1 && !(P.diags[d].pt_base <= gs && gs - P.diags[d].pt_base < P.diags[d].n)) {
            int lo = 0, hi = P.ndiag - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (P.diags[mid].pt_base <= gs) lo = mid;
                else hi = mid - 1;
            }
            d = lo;
        }
        run_lean<EXACT, MODE>(P, S, gs, P.diags[d], plan, gen, W, lane);
        w = __shfl_sync(FULL, wn, 0);
    }
    if constexpr (MODE != kPlain) {
        if (lane == 0 && P.work_ctr) {
            atomicAdd(&P.work_ctr[0], (unsigned long long)W.tested);
            atomicAdd(&P.work_ctr[1], (unsigned long long)W.cuts);
            atomicAdd(&P.work_ctr[2], (unsigned long long)W.newv);
            atomicAdd(&P.work_ctr[3], (unsigned long long)W.windows);
            atomicAdd(&P.work_ctr[4], (unsigned long long)W.batches);
        }
    }
}

// One cell with its geometry, one warp, for every precision.  What bounds it is
// the chain of dependent steps of the one warp.  A query of one cell of 1,000
// points through it, with the results written straight into host memory: 68 us
// from Python; through the FP64 clipping, copied back, 160 us.
__global__ void __launch_bounds__(32) k_lean_cell(ClipParams P) {
    extern __shared__ __align__(16) unsigned char smraw[];
    Lean& S = *reinterpret_cast<Lean*>(smraw);
    const int lane = threadIdx.x & 31;
    if (P.grid_err && *P.grid_err == 1) {         // non-finite input: nothing to clip
        if (lane == 0) P.geo->status = ST_GUARD;
        return;
    }
    for (int i = lane; i < kPlanes; i += 32) S.map[i] = 0;
    uint32_t gen = 0;
    Work W;
    run_lean<true, kGeo>(P, S, P.at_point ? 0xFFFFFFFFu : tess_chk(*P.work, P.npts, P.check, CK_POINT), P.diags[0], row_plan(lane), gen, W,
                         lane);
}

template <bool EXACT, int MODE>
cudaError_t configure(size_t bytes) {
    static std::mutex mu;
    static size_t configured[kMaxDevices] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    size_t* slot = (dev >= 0 && dev < kMaxDevices) ? &configured[dev] : nullptr;
    if (slot && bytes <= *slot) return cudaSuccess;
    e = cudaFuncSetAttribute(k_lean<EXACT, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess && slot) *slot = bytes;
    return e;
}

template <bool EXACT, int MODE>
cudaError_t launch(const ClipParams& p, int wpb, int blocks, cudaStream_t s) {
    const size_t sm = sizeof(Lean) * (size_t)wpb;
    cudaError_t e = configure<EXACT, MODE>(sm);
    if (e != cudaSuccess) return e;
    return launch_after(k_lean<EXACT, MODE>, blocks, 32 * wpb, sm, s, p);
}

template <bool EXACT, int MODE>
int blocks_for(int wpb, int device) {
    const size_t sm = sizeof(Lean) * (size_t)wpb;
    int per = 0, nsm = 0;
    if (configure<EXACT, MODE>(sm) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_lean<EXACT, MODE>, 32 * wpb, sm) != cudaSuccess)
        per = 1;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
    cudaGetLastError();   // leave no sticky error behind a failed query
    if (per < 1) per = 1;
    return per * (nsm > 0 ? nsm : 1);
}

}  // namespace cliplean

// form: kFormLean (the plain pass; with TESS_FLAG_COUNTERS its counting
// instance, the results are the same) or kFormDense, with kFormExact for the FP64
// finish, or kFormCareful | kFormExact.
cudaError_t launch_clip_lean(const ClipParams& p, int form, int wpb, int blocks, cudaStream_t s) {
    using namespace cliplean;
    const bool x = form & kFormExact;
    switch (form & 3) {
        case kFormCareful: return launch<true, kCareful>(p, wpb, blocks, s);
        case kFormDense: return x ? launch<true, kDense>(p, wpb, blocks, s) : launch<false, kDense>(p, wpb, blocks, s);
        default: break;
    }
    if (p.work_ctr) return x ? launch<true, kCount>(p, wpb, blocks, s) : launch<false, kCount>(p, wpb, blocks, s);
    return x ? launch<true, kPlain>(p, wpb, blocks, s) : launch<false, kPlain>(p, wpb, blocks, s);
}

cudaError_t launch_cell_lean(const ClipParams& p, cudaStream_t s) {
    static_assert(sizeof(cliplean::Lean) <= 48 * 1024, "launched without a shared memory attribute");
    cliplean::k_lean_cell<<<1, 32, sizeof(cliplean::Lean), s>>>(p);
    return cudaGetLastError();
}

int clip_blocks_lean(int form, int wpb, int device) {
    using namespace cliplean;
    const bool x = form & kFormExact;
    switch (form & 3) {
        case kFormCareful: return blocks_for<true, kCareful>(wpb, device);
        case kFormDense: return x ? blocks_for<true, kDense>(wpb, device) : blocks_for<false, kDense>(wpb, device);
        default: return x ? blocks_for<true, kPlain>(wpb, device) : blocks_for<false, kPlain>(wpb, device);
    }
}

}  // namespace tess

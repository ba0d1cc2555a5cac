// tess_clip_impl.cuh -- the FP64 clipping kernel: one Voronoi cell per warp, for
// the cells that the FP32 passes (tess_clip_lean.cu) do not settle, single-cell
// geometry included.
//
// The GPU form of Cell::compute_voronoi_cell (interface.rs:257-313) with
// Polyhedron::cut_with_plane (polyhedron.rs:438-642), ExpandingSearch
// (celery.rs:865-1075) and the cell outputs (polyhedron.rs:776-935).
//
// Cell representation (per warp).  The polyhedron starts as the container
// box translated by -site (polyhedron.rs:268-392, interface.rs:266).  Every
// vertex is the meeting point of three face planes and is stored as
//   - its position: in lane registers (slot s lives in lane s % 32, register
//     set s / 32) with a mirror in shared memory,
//   - its plane triple (a, b, c), ordered counter-clockwise seen from outside,
//   - its three neighbours: adj[i] is the vertex across the edge (t[i], t[i+1]).
// The half-edge pools of the reference (pool.rs) become these fixed-capacity
// slot arrays; a cell that outgrows them is listed for a larger capacity.
//
// Cutting by a bisector (vector3.rs:223-239):
//   1. every lane classifies its vertices, sd = n.v - offset, Outside when
//      sd > 1e-12 (vector3.rs:170-193, polyhedron.rs:221); one ballot per
//      register set gives the Outside mask.  No Outside vertex: no cut.
//   2. an edge of an Outside vertex X whose neighbour Y is not Outside is a
//      boundary edge; it gets a new vertex at the reference's intersection
//      X + (Y - X) * sd_X / (sd_X - sd_Y) (vector3.rs:213-219) with the
//      triple (a, b, new plane).  An Incident Y (|sd| <= tol) yields a
//      vertex at Y's position, as the reference duplicates Incident vertices
//      (polyhedron.rs:554-565).
//   3. the new vertices link into a ring through two small maps
//      (first plane -> vertex, second plane -> vertex), Outside slots are
//      freed and reused (clean_up_vertices / clean_up_edges, polyhedron.rs:645-730).
//
// Candidates come bin by bin in shell order (get_search_order,
// celery.rs:418-679) and the walk stops once the next bin's gap distance is
// at least twice the largest vertex distance: no farther point can cut
// (the security radius; the reference walks every point instead,
// celery.rs:971-1018, with the same result).
//
// Areas and volumes are accumulated in FP64 (weighted normals and volume / 6,
// polyhedron.rs:776-855).
//
// Crowded bins: a cell whose own bin holds many points is first cut by the
// nearest point of each lane's stride of that bin (32 seeds, nearest first),
// which shrinks it to about its final size before the shell walk.
#pragma once
#include <cfloat>
#include <cmath>
#include <mutex>

#include "tess_internal.cuh"

namespace tess {
namespace clipk {

constexpr unsigned FULL = 0xffffffffu;
// FP32 form: relative error constant of a vertex solved from its three planes
// (a few FP32 roundings of the plane data and of Cramer's rule).
constexpr float kVertexErr = 1.5e-6f;
// Pre-test a window's candidates against the live vertices when at least
// this many are within twice the cell radius.
constexpr int kPretestMin = 2;
// A site whose own bin holds at least ClipParams::seed_min points (12 by
// default, autotuned per input) is seeded before the shell walk: every lane
// takes the nearest point of its stride of that bin and the 32 seeds are cut
// nearest first.  In crowded bins the walk's 32-point windows otherwise meet
// the nearest points late, after many cuts by farther ones (plane capacity,
// larger radius, more guard-band tests).
template <int K>
struct Smem {
    static constexpr int V = 32 * K;                                 // vertex slots
    static constexpr int P = (32 * K + 32) < 254 ? (32 * K + 32) : 254;  // planes (< 0xFF)
    static constexpr int VUSE = V < 255 ? V : 255;                    // slot 255 is the map sentinel
    // live through the whole cell
    double vx[V], vy[V], vz[V];            // vertex mirror
    int32_t pid[P];                   // neighbour id (local original index) or wall code
    uint32_t tri[V];                  // planes a | b << 8 | c << 16
    uint32_t adj[V];                  // neighbours n0 | n1 << 8 | n2 << 16
    // The walk's working arrays and the finalize's share storage: no array
    // of one phase is read in the other, and every walk array is set up
    // again at the start of each cell.
    union {
        struct {                      // walk
            double px[P], py[P], pz[P], pd[P];     // plane: normal, offset (n.x = offset)
            double vsd[V];                         // signed distances of the current cut
            float vr[V];                      // (|v| + e_v)^2 of each slot (FP32), |v|^2 rounded up (FP64)
            double cbx[32], cby[32], cbz[32], cb2[32];   // kept candidates waiting for a full window ...
            uint32_t cbj[32];                 // ... their sorted indices
            int32_t cbid[32];                 // ... and local original ids
            uint32_t nbeg[32], ncnt[32];      // crowded bins: the 27 neighbour bins' ranges ...
            float nd[32];                     // ... and the squared distance to their nearest point
            float blo[3], bhi[3];             // bounds of the live vertices (long batches)
            uint32_t pending;                 // crowded bins still to handle (mask over the 27)
            double sdx[32], sdy[32], sdz[32], sd2[32];   // each lane's seed: offset, squared length ...
            uint32_t sdj[32];                 // ... sorted index (~0: none)
            int32_t sdcid[32];                // ... and local original id
            int32_t cbin;                     // the crowded bin being handled
            int32_t ring;                     // Chebyshev ring being walked ...
            uint32_t r0;                      // ... and the position in it
            uint32_t pused[(P + 31) / 32];    // plane recycling: planes referenced by live vertices
            uint16_t items[V + 32];           // boundary edges of a cut: slot | edge << 8
            uint8_t fl[V + 32];               // free-slot stack (top = lowest free slot)
            // new-vertex ring maps: gen << 8 | slot; entries with another
            // cut's tag are stale
            uint16_t mapf[P], maps[P];
            float fvx[V], fvy[V], fvz[V];     // the vertices rounded to FP32 (window pre-test)
        };
        struct {                      // finalize
            uint32_t fdeg[P];                 // live vertices per face
            int32_t flist[P];                 // compacted face ids
            uint8_t fsta[P];                  // one vertex of each face
            uint8_t rank2p[P];                // geometry output: rank -> plane
        };
    };
};

__device__ __forceinline__ unsigned warp_incl_scan_u(unsigned v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned t = __shfl_up_sync(FULL, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    return v;
}

// Position of the q-th (0-based) set bit of m; requires q < popc(m).
__device__ __forceinline__ int select32(uint32_t m, int q) {
    int pos = 0;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        const uint32_t low = (1u << (pos + s)) - 1u;
        if (__popc(m & low) <= q) pos += s;
    }
    return pos;
}

template <int K>
__device__ __forceinline__ int select_k(const uint32_t (&m)[K], int q) {
    int res = -1;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int c = __popc(m[k]);
        if (res < 0) {
            if (q < c) res = k * 32 + select32(m[k], q);
            else q -= c;
        }
    }
    return res;
}

template <int K>
__device__ __forceinline__ bool bit_k(const uint32_t (&m)[K], int s) {
    uint32_t w = m[0];
#pragma unroll
    for (int k = 1; k < K; ++k)
        if ((s >> 5) == k) w = m[k];
    return (w >> (s & 31)) & 1u;
}

template <int K>
__device__ __forceinline__ void set_k(uint32_t (&m)[K], int s) {
#pragma unroll
    for (int k = 0; k < K; ++k)
        if ((s >> 5) == k) m[k] |= 1u << (s & 31);
}

__device__ __forceinline__ int plane_of(uint32_t t, int i) { return (int)((t >> (8 * i)) & 0xFFu); }

// Error-free transforms (Knuth's TwoSum; the product's rounding error by one
// FMA): s + e == a + b and p + e == a * b exactly.  Explicit round-to-nearest
// intrinsics keep the compiler from contracting or reordering them.
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}
__device__ __forceinline__ void two_prod(float a, float b, float& p, float& e) {
    p = __fmul_rn(a, b);
    e = __fmaf_rn(a, b, -p);
}

// Signed distance n.v - offset.
__device__ __forceinline__ float sdist(float nx, float ny, float nz, float off, float x, float y, float z) {
    return fmaf(nx, x, fmaf(ny, y, fmaf(nz, z, -off)));
}
__device__ __forceinline__ double sdist(double nx, double ny, double nz, double off, double x, double y,
                                        double z) {
    return fma(nx, x, fma(ny, y, fma(nz, z, -off)));
}

// Bisector of the site (origin) and r (halfway_from_origin_to, vector3.rs:223-239),
// unnormalised: n = r, off = r.r / 2, with rn = r.r = |n|^2, so that the
// reference's test of the normalised signed distance against 1e-12
// (Plane::vector_location, vector3.rs:170-185) compares with one threshold
// (tol_of): no FP64 square root and no division per candidate.  A normalised
// plane cost ~27 FP64-pipe instructions per candidate.
__device__ __forceinline__ void bisector(double rx, double ry, double rz, double r2, double& nx,
                                         double& ny, double& nz, double& off, double& rn) {
    nx = rx;
    ny = ry;
    nz = rz;
    off = 0.5 * r2;
    rn = r2;
}

// 1/d for the FP64 form's edge interpolation, by Newton-Raphson: the FP32
// reciprocal, then two steps y' = y + y (1 - d y) in FP64, each of which
// squares the relative error (2^-23 -> 2^-46 -> the FP64 rounding, about 2
// ulp in all).  Outside FP32's normal range, the FP64 division.
__device__ __forceinline__ double recip_nr(double d) {
    const float df = (float)d;
    const float a = fabsf(df);
    if (!(a > 1e-36f && a < 1e36f)) return 1.0 / d;
    double y = (double)__frcp_rn(df);
    double e = fma(-d, y, 1.0);
    y = fma(y, e, y);
    e = fma(-d, y, 1.0);
    return fma(y, e, y);
}

// The FP64 form's tolerance for a plane with |n|^2 = n2: Outside is
// sd > 1e-12 |n|, Inside sd < -1e-12 |n| (the reference's test on the
// normalised distance).  |n| comes from the FP32 square root: off by ~1e-7 of
// 1e-12 |n|, far inside the FP64 rounding of a signed distance, and each test
// is one compare.  Planes beyond FP32's range take the FP64 root.
__device__ __forceinline__ double tol_of(double n2) {
    const float n2f = (float)n2;
    return n2f >= FLT_MIN && n2f < 1e37f ? (double)(1e-12f * sqrtf(n2f)) : kTolerance * sqrt(n2);
}

// A vertex's share of the cell radius: |v|^2 rounded up to FP32 (the radius only
// bounds the search, and FP32 keeps its warp maximum off the FP64 pipe).
__device__ __forceinline__ float vrad2(double x, double y, double z) {
    return __double2float_ru(x * x + y * y + z * z);
}

// Per-warp work counters (reported when ClipParams::work_ctr is set).
struct Work {
    unsigned tested = 0, cuts = 0, newv = 0, windows = 0, batches = 0;
};

template <int K>
struct CellRegs {
    double vx[K], vy[K], vz[K];
    uint32_t lm[K];   // live masks (warp-uniform)
    int np;           // planes used (warp-uniform)
    int nfree;        // entries on the free-slot stack (warp-uniform)
    uint32_t gen;     // tag of the current cut in the ring maps, 0..255 (warp-uniform)
};

// The general form of a cut (more than 32 edges leave the Outside
// vertices): owners loop over their edges; placement runs in rounds of 32.
// The plane table is full: find a plane id (not a wall) that no live vertex
// references any more, or -1.  Faces cut away entirely leave such ids
// behind; cells cut hundreds of times (next to dense clusters) need them.
template <int K>
__device__ __noinline__ int recycle_plane(Smem<K>& S, const CellRegs<K>& C, int lane) {
    using S_t = Smem<K>;
    constexpr int NW = (S_t::P + 31) / 32;
    for (int w = lane; w < NW; w += 32) S.pused[w] = 0;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if ((C.lm[k] >> lane) & 1u) {
            const uint32_t t = S.tri[k * 32 + lane];
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                const int p = plane_of(t, e);
                if (p < S_t::P) atomicOr(&S.pused[p >> 5], 1u << (p & 31));
            }
        }
    }
    __syncwarp();
    int res = -1;
    for (int w = 0; w < NW && res < 0; ++w) {
        uint32_t fr = ~S.pused[w];
        if (w == 0) fr &= ~0x3Fu;                                  // the walls stay
        if (w == NW - 1 && (S_t::P & 31)) fr &= (1u << (S_t::P & 31)) - 1u;
        if (fr) res = w * 32 + __ffs(fr) - 1;
    }
    __syncwarp();
    return res;
}

template <typename V, int K>
struct Regs {
    V v[K];
};

template <int K>
__device__ __forceinline__ int cut_general(Smem<K>& S, CellRegs<K>& C, const Regs<double, K> sdv,
                                        const Regs<uint32_t, K> omv, double nx, double ny, double nz, double off, double rn,
                                        int32_t id, int f, int lane, int* P_check) {
    using S_t = Smem<K>;
    const double(&sd)[K] = sdv.v;
    const uint32_t(&om)[K] = omv.v;

    // Signed distances of live vertices go to shared memory for the lanes
    // that place new vertices; my Outside vertices' triples and neighbours are
    // read before any slot is reused.
    uint32_t xt[K], xa[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int s = k * 32 + lane;
        if (((C.lm[k] >> lane) & 1u)) S.vsd[s] = sd[k];   // read by the FP64 interpolation
        xt[k] = 0;
        xa[k] = 0;
        if ((om[k] >> lane) & 1u) {
            xt[k] = S.tri[s];
            xa[k] = S.adj[s];
        }
    }
    // Every slot and plane id read below must be in range; a violation
    // (inconsistent topology) abandons the cell before anything is written.
    bool badref = false;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if ((om[k] >> lane) & 1u) {
#pragma unroll
            for (int e = 0; e < 3; ++e)
                badref |= plane_of(xt[k], e) >= C.np || plane_of(xa[k], e) >= S_t::V;
        }
    }
    if (__any_sync(FULL, badref)) return -ST_DEGEN;
    // Boundary edges: edges of Outside vertices whose neighbour is not Outside.
    unsigned bnd = 0;
    int cnt = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if ((om[k] >> lane) & 1u) {
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                const int nb = plane_of(xa[k], e);
                if (!bit_k<K>(om, nb)) {
                    bnd |= 1u << (3 * k + e);
                    ++cnt;
                }
            }
        }
    }
    const unsigned incl = warp_incl_scan_u((unsigned)cnt, lane);
    const int B = (int)__shfl_sync(FULL, incl, 31);
    const int q0 = (int)incl - cnt;
    int nlive = 0;
    uint32_t fm[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const uint32_t keep = C.lm[k] & ~om[k];
        nlive += __popc(keep);
        fm[k] = ~keep;
    }
    if (K == 8) fm[K - 1] &= 0x7FFFFFFFu;
    if (nlive + B > S_t::VUSE) return -ST_VCAP;
    const int rounds = (B + 31) >> 5;
    if (rounds > 1) {
        // More than 32 new vertices (a cut through a large cell): make sure
        // no Outside slot is reused before every round has read it.
        int nfree_clean = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) nfree_clean += __popc(fm[k] & ~om[k]);
        if (nfree_clean < B) return -ST_VCAP;
#pragma unroll
        for (int k = 0; k < K; ++k) fm[k] &= ~om[k];
    }
    // Owners list their boundary edges (slot | edge << 8) at their prefix
    // positions; lane l then places new vertex l (+ 32 per round).
    uint16_t* items = S.items;
    {
        int qq = q0;
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
            for (int e = 0; e < 3; ++e)
                if (bnd & (1u << (3 * k + e)))
                    items[tess_chk(qq++, S_t::V + 32, P_check, CK_SLOT)] = (uint16_t)((k * 32 + lane) | (e << 8));
    }
    __syncwarp();
    uint32_t newm[K];
#pragma unroll
    for (int k = 0; k < K; ++k) newm[k] = 0;
    bool bad = false;
    for (int r0 = 0; r0 < B; r0 += 32) {
        const int qi = r0 + lane;
        const bool act = qi < B;
        int y = 0, a = 0, b = 0, slot = 0;
        uint32_t ty = 0;
        double px = 0, py = 0, pz = 0;
        if (act) {
            const uint32_t it = items[qi];
            const int x = it & 0xFF, e = it >> 8;
            const uint32_t xt_ = S.tri[x], xa_ = S.adj[x];
            a = plane_of(xt_, e);
            b = plane_of(xt_, e == 2 ? 0 : e + 1);
            y = plane_of(xa_, e);
            const double xx = S.vx[x], xy = S.vy[x], xz = S.vz[x], xsd = S.vsd[x];
            const double yx = S.vx[y], yy = S.vy[y], yz = S.vz[y], ysd = S.vsd[y];
            ty = S.tri[y];
            // intersection(outside X, inside Y) (vector3.rs:213-219); an
            // Incident Y is kept as the new vertex (polyhedron.rs:554-565)
            const double den = xsd - ysd;
            const double t = ysd >= -(double)tol_of(rn) ? 1.0 : xsd * recip_nr(den);
            px = xx + (yx - xx) * t;
            py = xy + (yy - xy) * t;
            pz = xz + (yz - xz) * t;
            slot = tess_chk(select_k<K>(fm, qi), S_t::V, P_check, CK_SLOT);
        }
        __syncwarp();
        if (act) {
            S.vx[slot] = px;
            S.vy[slot] = py;
            S.vz[slot] = pz;
            // the FP32 copies (rounded to nearest) serve the
            // window pre-test and the cell radius: |v|^2 from them, times
            // 1 + 5 * 2^-23 (the copies' and the sum's rounding are at
            // most 2.5 * 2^-23), is an upper bound, off the FP64 pipe
            const float fx = (float)px, fy = (float)py, fz = (float)pz;
            S.fvx[slot] = fx;
            S.fvy[slot] = fy;
            S.fvz[slot] = fz;
            S.vr[slot] = fmaf(fx, fx, fmaf(fy, fy, fz * fz)) * 1.000000596f;
            S.tri[slot] = (uint32_t)a | ((uint32_t)b << 8) | ((uint32_t)f << 16);
            // Y's pointer back to X is the edge (b, a) of Y's triple.
            const int yi = (plane_of(ty, 0) == b && plane_of(ty, 1) == a)   ? 0
                           : (plane_of(ty, 1) == b && plane_of(ty, 2) == a) ? 1
                                                                            : 2;
            reinterpret_cast<uint8_t*>(S.adj)[4 * y + yi] = (uint8_t)slot;
            S.mapf[a] = (uint16_t)((C.gen << 8) | (uint32_t)slot);
            S.maps[b] = (uint16_t)((C.gen << 8) | (uint32_t)slot);
            S.adj[slot] = (uint32_t)y;
#pragma unroll
            for (int k = 0; k < K; ++k)
                if ((slot >> 5) == k) newm[k] |= 1u << (slot & 31);
        }
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < K; ++k) newm[k] = __reduce_or_sync(FULL, newm[k]);
    // Link the ring of new vertices (each by its owner lane): across (b, f)
    // lies the new vertex whose first plane is b, across (f, a) the one whose
    // second plane is a.
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if ((newm[k] >> lane) & 1u) {
            const int s = k * 32 + lane;
            const uint32_t tt = S.tri[s];
            const int a = plane_of(tt, 0), b = plane_of(tt, 1);
            const uint32_t tag = C.gen << 8;
            const uint32_t mb = S.mapf[b], ma = S.maps[a];
            const int n1 = (mb & 0xFF00u) == tag ? (int)(mb & 0xFFu) : 0xFF;
            const int n2 = (ma & 0xFF00u) == tag ? (int)(ma & 0xFFu) : 0xFF;
            bad |= (S.mapf[a] != (tag | (uint32_t)s)) || (S.maps[b] != (tag | (uint32_t)s)) || n1 == 0xFF || n2 == 0xFF;
            S.adj[s] = (S.adj[s] & 0xFFu) | ((uint32_t)n1 << 8) | ((uint32_t)n2 << 16);
        }
    }
    if (__any_sync(FULL, bad)) return -ST_DEGEN;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        C.lm[k] = (C.lm[k] & ~om[k]) | newm[k];
        if ((newm[k] >> lane) & 1u) {
            const int s = k * 32 + lane;
            C.vx[k] = S.vx[s];
            C.vy[k] = S.vy[s];
            C.vz[k] = S.vz[s];
        }
    }
    if (lane == 0) {
        S.px[f] = nx;
        S.py[f] = ny;
        S.pz[f] = nz;
        S.pd[f] = off;
        S.pid[f] = id;
    }
    if (f >= C.np) C.np = f + 1;
    // rebuild the free-slot stack from the live masks
    {
        int n = 0;
#pragma unroll
        for (int k = K - 1; k >= 0; --k) {
            uint32_t fr = ~C.lm[k];
            if (K == 8 && k == K - 1) fr &= 0x7FFFFFFFu;
            const int c = __popc(fr);
            // descending slot order, so the lowest free slot is on top
            if ((fr >> (31 - lane)) & 1u) {
                const uint32_t above = lane == 0 ? 0u : (fr >> (32 - lane));
                S.fl[n + __popc(above)] = (uint8_t)(k * 32 + 31 - lane);
            }
            n += c;
        }
        C.nfree = n;
    }
    __syncwarp();
    return B + 1;
}

// Clip the cell by the half-space {x : n.x - off <= 0} of a bisector (n = r,
// off = r.r / 2): a vertex is Outside when n.v - off > 1e-12 |n|
// (vector3.rs:170-193, polyhedron.rs:221).  Returns the new vertices + 1 when
// vertices were cut off, 0 when nothing was Outside, or -status.
template <int K>
__device__ int cut(Smem<K>& S, CellRegs<K>& C, double nx, double ny, double nz, double off, double rn, int32_t id, int lane,
                   const ClipParams& P) {
    using S_t = Smem<K>;
    double sd[K];
    uint32_t om[K];
    // the tolerance of the normalised test, rn = |n|^2 (see bisector)
    const double tolr = tol_of(rn);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        sd[k] = 0.0;
        om[k] = 0;
        // register sets without live vertices are skipped (the free-slot
        // stack hands out the lowest slots first, so the upper sets are
        // usually empty)
        if (C.lm[k] == 0) continue;
        const bool live = (C.lm[k] >> lane) & 1u;
        sd[k] = sdist(nx, ny, nz, off, C.vx[k], C.vy[k], C.vz[k]);
        bool out;
        out = live && sd[k] > tolr;
        om[k] = __ballot_sync(FULL, out);
    }
    uint32_t anyo = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) anyo |= om[k];
    if (!anyo) return 0;
    int f = C.np;
    if (f >= S_t::P) {
        // Only the largest capacity recycles plane ids: a call here costs the
        // smaller instantiations' hot path registers even when never taken,
        // and their cells re-run at the next capacity instead.
        if constexpr (K == 8) {
            f = recycle_plane<K>(S, C, lane);
            if (f < 0) return -ST_PCAP;
        } else {
            return -ST_PCAP;
        }
    }
    // a new tag for this cut's ring-map entries; every 256 cuts the maps are
    // cleared, so a stale entry never carries the current tag
    C.gen = (C.gen + 1) & 0xFFu;
    if (C.gen == 0) {
        for (int i = lane; i < S_t::P; i += 32) {
            S.mapf[i] = 0xFFFF;
            S.maps[i] = 0xFFFF;
        }
        __syncwarp();
    }
    int R = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) R += __popc(om[k]);
    if (3 * R <= 32) {
        // Fast path: one lane per edge of an Outside vertex.  The Outside
        // slots are pushed onto the free-slot stack; the new vertices pop
        // slots from its top (reusing freed slots first).
        const int base = C.nfree;
        int before = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int s = k * 32 + lane;
            if (((C.lm[k] >> lane) & 1u)) S.vsd[s] = sd[k];   // read by the FP64 interpolation
            if ((om[k] >> lane) & 1u)
                S.fl[tess_chk(base + before + __popc(om[k] & ((1u << lane) - 1u)), S_t::V + 32, P.check, CK_SLOT)] = (uint8_t)s;
            before += __popc(om[k]);
        }
        __syncwarp();
        const bool edge = lane < 3 * R;
        int x = 0, y = 0, a = 0, b = 0;
        bool bnd = false, bad = false;
        if (edge) {
            const int xi = (lane * 11) >> 5;          // lane / 3 for lane < 32
            const int e = lane - 3 * xi;
            x = tess_chk((int)S.fl[tess_chk(base + xi, S_t::V + 32, P.check, CK_SLOT)], S_t::V, P.check, CK_SLOT);
            const uint32_t xt_ = S.tri[x], xa_ = S.adj[x];
            a = plane_of(xt_, e);
            b = plane_of(xt_, e == 2 ? 0 : e + 1);
            y = plane_of(xa_, e);
            bad = a >= C.np || b >= C.np || y >= S_t::V;
            bnd = !bad && !bit_k<K>(om, y);
        }
        if (__any_sync(FULL, bad)) return -ST_DEGEN;
        const unsigned bm = __ballot_sync(FULL, bnd);
        const int B = __popc(bm);
        // capacity: the stack (with the pushed Outside slots) must hold B
        if (B > base + R) return -ST_VCAP;
        const int q = __popc(bm & ((1u << lane) - 1u));
        int slot = 0;
        uint32_t ty = 0;
        double px = 0, py = 0, pz = 0;
            if (bnd) {
            const double xx = S.vx[x], xy = S.vy[x], xz = S.vz[x], xsd = S.vsd[x];
            const double yx = S.vx[y], yy = S.vy[y], yz = S.vz[y], ysd = S.vsd[y];
            const double t = ysd >= -tolr ? 1.0 : xsd * recip_nr(xsd - ysd);
            px = xx + (yx - xx) * t;
            py = xy + (yy - xy) * t;
            pz = xz + (yz - xz) * t;
            ty = S.tri[y];
            slot = tess_chk((int)S.fl[tess_chk(base + R - 1 - q, S_t::V + 32, P.check, CK_SLOT)], S_t::V, P.check, CK_SLOT);
        }
        __syncwarp();
        if (bnd) {
            S.vx[slot] = px;
            S.vy[slot] = py;
            S.vz[slot] = pz;
            // the FP32 copies (rounded to nearest) serve the
            // window pre-test and the cell radius: |v|^2 from them, times
            // 1 + 5 * 2^-23 (the copies' and the sum's rounding are at
            // most 2.5 * 2^-23), is an upper bound, off the FP64 pipe
            const float fx = (float)px, fy = (float)py, fz = (float)pz;
            S.fvx[slot] = fx;
            S.fvy[slot] = fy;
            S.fvz[slot] = fz;
            S.vr[slot] = fmaf(fx, fx, fmaf(fy, fy, fz * fz)) * 1.000000596f;
            S.tri[slot] = (uint32_t)a | ((uint32_t)b << 8) | ((uint32_t)f << 16);
            // Y's pointer back to X is the edge (b, a) of Y's triple.
            const int yi = (plane_of(ty, 0) == b && plane_of(ty, 1) == a)   ? 0
                           : (plane_of(ty, 1) == b && plane_of(ty, 2) == a) ? 1
                                                                            : 2;
            reinterpret_cast<uint8_t*>(S.adj)[4 * y + yi] = (uint8_t)slot;
            S.mapf[a] = (uint16_t)((C.gen << 8) | (uint32_t)slot);
            S.maps[b] = (uint16_t)((C.gen << 8) | (uint32_t)slot);
        }
        __syncwarp();
        if (bnd) {
            // across (b, f): the new vertex whose first plane is b; across
            // (f, a): the one whose second plane is a (entries of this cut only)
            const uint32_t tag = C.gen << 8;
            const uint32_t mb = S.mapf[b], ma = S.maps[a];
            const int n1 = (mb & 0xFF00u) == tag ? (int)(mb & 0xFFu) : 0xFF;
            const int n2 = (ma & 0xFF00u) == tag ? (int)(ma & 0xFFu) : 0xFF;
            bad = (S.mapf[a] != (tag | (uint32_t)slot)) || (S.maps[b] != (tag | (uint32_t)slot)) || n1 == 0xFF ||
                  n2 == 0xFF;
            S.adj[slot] = (uint32_t)y | ((uint32_t)n1 << 8) | ((uint32_t)n2 << 16);
        }
        if (__any_sync(FULL, bad)) return -ST_DEGEN;
        C.nfree = base + R - B;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const uint32_t nm = __reduce_or_sync(FULL, (bnd && (slot >> 5) == k) ? (1u << (slot & 31)) : 0u);
            C.lm[k] = (C.lm[k] & ~om[k]) | nm;
            if ((nm >> lane) & 1u) {
                const int s = k * 32 + lane;
                C.vx[k] = S.vx[s];
                C.vy[k] = S.vy[s];
                C.vz[k] = S.vz[s];
            }
        }
        // the plane (predicated stores of one lane: no divergent branches)
        if (lane == 0) {
            S.px[f] = nx;
            S.py[f] = ny;
            S.pz[f] = nz;
            S.pd[f] = off;
            S.pid[f] = id;
        }
        if (f >= C.np) C.np = f + 1;
        __syncwarp();
        return B + 1;
    }
    Regs<double, K> sdv;
    Regs<uint32_t, K> omv;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        sdv.v[k] = sd[k];
        omv.v[k] = om[k];
    }
    return cut_general<K>(S, C, sdv, omv, nx, ny, nz, off, rn, id, f, lane, P.check);
}

// Squared radius of the cell about its site, an FP32 upper bound: the maximum
// over the live vertices of the terms (vrad2) written with them.
template <int K>
__device__ __forceinline__ float live_r2f(const Smem<K>& S, const CellRegs<K>& C, int lane) {
    float r2 = 0.f;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if (C.lm[k] == 0) continue;
        if ((C.lm[k] >> lane) & 1u) r2 = fmaxf(r2, S.vr[k * 32 + lane]);
    }
    // r2 >= 0 and never NaN (fmaxf drops NaN): its bits order like its value
    return __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(r2)));
}

__device__ __forceinline__ void ring_offset(int s, uint32_t r, int& i, int& j, int& k) {
    const uint32_t a = 2u * s + 1u, b = 2u * s - 1u;
    const uint32_t nx = 2u * a * a, ny = 2u * b * a;
    if (r < nx) {
        const uint32_t side = r / (a * a), rem = r % (a * a);
        i = side ? s : -s;
        j = (int)(rem / a) - s;
        k = (int)(rem % a) - s;
    } else if (r < nx + ny) {
        r -= nx;
        const uint32_t side = r / (b * a), rem = r % (b * a);
        j = side ? s : -s;
        i = (int)(rem / a) - (s - 1);
        k = (int)(rem % a) - s;
    } else {
        r -= nx + ny;
        const uint32_t side = r / (b * b), rem = r % (b * b);
        k = side ? s : -s;
        i = (int)(rem / b) - (s - 1);
        j = (int)(rem % b) - (s - 1);
    }
}

// The FP32 bounds of the live vertices (and the site), into shared memory.
template <int K>
struct Masks {
    uint32_t m[K];
};
template <int K>
__device__ __noinline__ void live_bounds(Smem<K>& S, Masks<K> live, int lane) {
    __syncwarp();
    // non-negative floats order like their bits (+0, not -0)
    auto top = [](float x) { return __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(fmaxf(x, 0.f)))); };
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float* v = a == 0 ? S.fvx : (a == 1 ? S.fvy : S.fvz);
        float lo = 0.f, hi = 0.f;
#pragma unroll
        for (int k = 0; k < K; ++k)
            if ((live.m[k] >> lane) & 1u) {
                lo = fminf(lo, v[k * 32 + lane]);
                hi = fmaxf(hi, v[k * 32 + lane]);
            }
        lo = -top(-lo);
        hi = top(hi);
        if (lane == 0) {
            S.blo[a] = lo;
            S.bhi[a] = hi;
        }
    }
    __syncwarp();
}

template <int K, bool GEO>
__device__ void run_cell(const ClipParams& P, Smem<K>& S, uint32_t gs, int lane, Work& W) {
    using S_t = Smem<K>;
    // ---- diagram of this cell ----
    int d = 0;
    if (P.ndiag > 1 && !P.at_point) {
        int lo = 0, hi = P.ndiag - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (P.diags[mid].pt_base <= gs) lo = mid;
            else hi = mid - 1;
        }
        d = lo;
    }
    const DiagDesc& D = P.diags[d];
    const uint32_t pt_base = D.pt_base;
    const uint64_t bin_base = D.bin_base;
    const uint32_t tab_len = D.tab_len;
    double sx, sy, sz;
    uint32_t self = 0xFFFFFFFFu, orig = 0;
    if (P.at_point) {
        sx = P.point[0];
        sy = P.point[1];
        sz = P.point[2];
    } else {
        sx = P.spx[gs];
        sy = P.spy[gs];
        sz = P.spz[gs];
        self = gs;
        orig = tess_chk(P.sorted[tess_chk(gs, P.npts, P.check, CK_POINT)], P.npts, P.check, CK_POINT);
    }
    // ---- the container box, translated by -site (polyhedron.rs:268-392) ----
    const double* blo = P.box_override ? P.box : D.blo;
    const double* bhi = P.box_override ? P.box + 3 : D.bhi;
    CellRegs<K> C;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        C.vx[k] = C.vy[k] = C.vz[k] = 0.0;
        C.lm[k] = 0;
    }
    C.lm[0] = 0xFFu;
    C.np = 6;
    if (lane < 6) {
        const int a = lane >> 1;
        const bool mx = lane & 1;
        const double s_a = a == 0 ? sx : (a == 1 ? sy : sz);
        const double offt = (double)(mx ? (bhi[a] - s_a) : (s_a - blo[a]));
        const double sg = mx ? 1.0 : -1.0;
        S.px[lane] = a == 0 ? sg : 0.0;
        S.py[lane] = a == 1 ? sg : 0.0;
        S.pz[lane] = a == 2 ? sg : 0.0;
        S.pd[lane] = offt;
        S.pid[lane] = -1 - lane;   // -1 x_min, -2 x_max, -3 y_min, -4 y_max, -5 z_min, -6 z_max
    }
    if (lane < 8) {
        const int bx = lane & 1, by = (lane >> 1) & 1, bz = (lane >> 2) & 1;
        C.vx[0] = (double)((bx ? bhi[0] : blo[0]) - sx);
        C.vy[0] = (double)((by ? bhi[1] : blo[1]) - sy);
        C.vz[0] = (double)((bz ? bhi[2] : blo[2]) - sz);
        S.vx[lane] = C.vx[0];
        S.vy[lane] = C.vy[0];
        S.vz[lane] = C.vz[0];
        S.fvx[lane] = (float)C.vx[0];
        S.fvy[lane] = (float)C.vy[0];
        S.fvz[lane] = (float)C.vz[0];
        S.vr[lane] = vrad2(C.vx[0], C.vy[0], C.vz[0]);
        const int pX = bx, pY = 2 + by, pZ = 4 + bz;
        const int sgn = (bx ? 1 : -1) * (by ? 1 : -1) * (bz ? 1 : -1);
        const int t0 = pX, t1 = sgn > 0 ? pY : pZ, t2 = sgn > 0 ? pZ : pY;
        S.tri[lane] = (uint32_t)t0 | ((uint32_t)t1 << 8) | ((uint32_t)t2 << 16);
        auto flip = [](int p) { return p < 2 ? 1 : (p < 4 ? 2 : 4); };
        const int n0 = lane ^ flip(t2), n1 = lane ^ flip(t0), n2 = lane ^ flip(t1);
        S.adj[lane] = (uint32_t)n0 | ((uint32_t)n1 << 8) | ((uint32_t)n2 << 16);
    }
    C.gen = 0;
    for (int i = lane; i < S_t::P; i += 32) {
        S.mapf[i] = 0xFFFF;
        S.maps[i] = 0xFFFF;
    }
    // free-slot stack: slots 8 .. VUSE-1, lowest on top
    C.nfree = S_t::VUSE - 8;
    for (int i = lane; i < C.nfree; i += 32) S.fl[i] = (uint8_t)(S_t::VUSE - 1 - i);
    __syncwarp();
    // the squared radius, and its value in FP32 for the search bounds, so that
    // they stay off the FP64 pipe
    float R2f = live_r2f(S, C, lane);
    double R2 = (double)R2f;
    int status = ST_OK;

    // ---- the walk over bins in shell order (celery.rs:1023-1075) ----
    const int cpd = D.cpd;
    // (an axis without extent has all its points in the last bin, and its offsets
    // count nothing in a key: a position beside it searches from there)
    auto bin_on = [&](double x, int a) {
        return D.ghi[a] > D.glo[a] ? axis_index(x, D.glo[a], D.ghi[a], D.inv[a], cpd) : cpd - 1;
    };
    const int cbx = bin_on(sx, 0), cby = bin_on(sy, 1), cbz = bin_on(sz, 2);
    const double radius = P.search_radius;
    const bool has_radius = radius >= 0.0;
    const int64_t tgroup = P.target_group;
    const TabEntry* tab = P.table + D.tab_base;

    // The offset p - site of sorted point j and its squared length.
    auto cand = [&](uint32_t j, double& rx, double& ry, double& rz, double& r2) {
        rx = (double)(P.spx[j] - sx);
        ry = (double)(P.spy[j] - sy);
        rz = (double)(P.spz[j] - sz);
        r2 = rx * rx + ry * ry + rz * rz;
    };
    // Sorted index of the lane's seed (none: ~0u); never a window candidate.
    uint32_t seedj = 0xFFFFFFFFu;

    // One window: up to one candidate per lane (keep), cut nearest first.
    auto run_window = [&](bool keep, double rx, double ry, double rz, double r2, uint32_t j, int32_t cid) -> int {
        unsigned km = __ballot_sync(FULL, keep);
        // Pre-test the window at once: each lane tests its own candidate's
        // bisector against every live vertex.  A bisector with no vertex
        // Outside cuts nothing now and nothing later (the cell only shrinks), so
        // only possible cutters go on to the serial nearest-first loop.
        if (__popc(km) >= kPretestMin) {
            bool maycut = false;
            if (keep) {
                // the test in FP32 on the vertices' FP32 copies,
                // kept unless the FP32 distance is below minus four times
                // its error bound (inputs rounded: 2u |r_i v_i|; FMA chain
                // and offset: 3u (sum |r_i v_i| + off) + u off; |v_i| <= R)
                const float fx = (float)rx, fy = (float)ry, fz = (float)rz, f2 = (float)r2;
                const float Rf = sqrtf((float)R2) * 1.0001f;
                const float margin = 2.4e-7f * (5.f * (fabsf(fx) + fabsf(fy) + fabsf(fz)) * Rf + 2.f * f2);
                const float foff = 0.5f * f2;
                bool out = false;
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    uint32_t m = C.lm[k];
                    while (m) {
                        const int sl = (k * 32 + __ffs(m) - 1);
                        m &= m - 1u;
                        const float sdf = fmaf(fx, S.fvx[sl], fmaf(fy, S.fvy[sl], fmaf(fz, S.fvz[sl], -foff)));
                        out |= !(sdf <= -margin);
                    }
                }
                maycut = out;
            }
            km = __ballot_sync(FULL, keep && maycut);
        }
        // Nearest first: repeatedly take the closest remaining candidate
        // (warp minimum of its distance, ties by lane), so the closest
        // bisectors shrink the cell before the farther ones are tested.
        // The key keeps the top 27 bits of r2 (a positive float orders
        // like its bits) and the lane in the low 5.
        const unsigned mykey = (__float_as_uint((float)r2) & ~31u) | (unsigned)lane;
        while (km) {
            const unsigned best = __reduce_min_sync(FULL, ((km >> lane) & 1u) ? mykey : 0xFFFFFFFFu);
            const int src = (int)(best & 31u);
            km &= ~(1u << src);
            const double cx = __shfl_sync(FULL, rx, src);
            const double cy = __shfl_sync(FULL, ry, src);
            const double cz = __shfl_sync(FULL, rz, src);
            const double c2 = __shfl_sync(FULL, r2, src);
            const uint32_t cj = __shfl_sync(FULL, j, src);
            const int32_t cidb = __shfl_sync(FULL, cid, src);
            // on the FP32 key (r2 rounded to FP32, truncated)
            // against the FP32 bound (margin 1e-5); a candidate beyond
            // reach that passes only costs a test (the cut decides exactly)
            const float k2 = __uint_as_float(best & ~31u), l2 = 4.f * R2f * (float)kStopMargin;
            if (!(k2 < l2)) {
                if (k2 > l2 * 1.001f) km = 0;
                continue;
            }
            double nx, ny, nz, off, rn;
            bisector(cx, cy, cz, c2, nx, ny, nz, off, rn);
            const int r = cut<K>(S, C, nx, ny, nz, off, rn, cidb, lane, P);
            ++W.tested;
            if (r < 0) return -r;
            if (r > 0) {
                ++W.cuts;
                W.newv += (unsigned)(r - 1);
                R2f = live_r2f(S, C, lane);
                R2 = (double)R2f;
            }
        }
        return ST_OK;
    };

    // Cut by every point of the lanes' bins, given as sorted ranges
    // [beg, beg + cnt), in lane order; or (direct) by one window of the
    // lanes' seeds of a crowded bin (S.sd*).
    auto process = [&](unsigned beg, unsigned cnt, bool direct) -> int {
        unsigned total = 32, pref = 0;
        if (!direct) {
            const unsigned inc = warp_incl_scan_u(cnt, lane);
            total = __shfl_sync(FULL, inc, 31);
            pref = inc - cnt;
        }
        // The windows' kept candidates are gathered in shared memory and cut 32
        // at a time, as each window's pre-test costs the same however few of its
        // candidates are kept (clustered 4M in FP64: 1,204 -> 1,070 ms).
        unsigned nbuf = 0;
        // A long batch (cells beside a cluster): a bisector beyond the support of
        // the vertices' bounds touches no vertex.  FP32 with a margin of 4e-6 of
        // the terms, several times their rounding.  500,000 clustered points, 41
        // cells here, the longest one's latency: 2.0 -> 1.0 ms.  (The bounds out
        // of line: inline, they cost 36,000 crystal cells 5%.)
        const bool bounded = !direct && total >= 256;
        auto bound = [&]() {
            Masks<K> live;
#pragma unroll
            for (int k = 0; k < K; ++k) live.m[k] = C.lm[k];
            live_bounds<K>(S, live, lane);
        };
        if (bounded) bound();
        for (unsigned w0 = 0;; w0 += 32) {
            const bool more = w0 < total;
            if (!more && (direct || nbuf == 0)) break;
            bool keep = false;
            double rx = 0, ry = 0, rz = 0, r2 = 0;
            uint32_t j = 0;
            int32_t cid = 0;
            if (!more) {
            } else if (direct) {
                j = S.sdj[lane];
                keep = j != 0xFFFFFFFFu;
                rx = S.sdx[lane];
                ry = S.sdy[lane];
                rz = S.sdz[lane];
                r2 = S.sd2[lane];
                cid = S.sdcid[lane];
            } else {
                ++W.windows;
                const unsigned c = w0 + lane;
                // the lane's bin: the last with prefix <= c (never an empty one)
                int lo = 0;
#pragma unroll
                for (int step = 16; step > 0; step >>= 1)
                    if (__shfl_sync(FULL, pref, lo + step) <= c) lo += step;
                const unsigned bbeg = __shfl_sync(FULL, beg, lo), bpref = __shfl_sync(FULL, pref, lo);
                if (c < total) {
                    j = tess_chk(bbeg + (c - bpref), P.npts, P.check, CK_POINT);
                    cand(j, rx, ry, rz, r2);
                    keep = (j != self) && r2 > 0.0 && (float)r2 < 4.f * R2f * (float)kStopMargin;
                    keep = keep && j != seedj;
                    if (bounded && keep) {
                        const float gx = (float)rx, gy = (float)ry, gz = (float)rz, off = 0.5f * (float)r2;
                        const float h = fmaxf(gx * S.blo[0], gx * S.bhi[0]) + fmaxf(gy * S.blo[1], gy * S.bhi[1]) +
                                        fmaxf(gz * S.blo[2], gz * S.bhi[2]);
                        keep = !(h * 1.000004f + 4e-6f * (fabsf(gx) + fabsf(gy) + fabsf(gz)) * sqrtf(R2f) < off * 0.999996f);
                    }
                    cid = (int32_t)(P.sorted[j] - pt_base);
                    if (keep && tgroup >= 0) keep = (int64_t)(P.sgroup ? P.sgroup[j] : 0u) == tgroup;
                }
            }
            if (!direct) {
                const unsigned km = __ballot_sync(FULL, keep);
                const unsigned nk = __popc(km);
                const unsigned pos = nbuf + __popc(km & ((1u << lane) - 1u));
                if (keep && pos < 32) {
                    S.cbx[pos] = rx;
                    S.cby[pos] = ry;
                    S.cbz[pos] = rz;
                    S.cb2[pos] = r2;
                    S.cbj[pos] = j;
                    S.cbid[pos] = cid;
                }
                if (more && nbuf + nk < 32) {
                    nbuf += nk;
                    continue;
                }
                // a full window (or the batch's last candidates) from the buffer
                __syncwarp();
                const unsigned cw = more ? 32u : nbuf;
                const bool kw = (unsigned)lane < cw;
                const double bx = S.cbx[lane], by = S.cby[lane], bz = S.cbz[lane], b2 = S.cb2[lane];
                const uint32_t bj = S.cbj[lane];
                const int32_t bid = S.cbid[lane];
                __syncwarp();
                // the candidates beyond the full window wait for the next one
                if (keep && pos >= 32) {
                    S.cbx[pos - 32] = rx;
                    S.cby[pos - 32] = ry;
                    S.cbz[pos - 32] = rz;
                    S.cb2[pos - 32] = r2;
                    S.cbj[pos - 32] = j;
                    S.cbid[pos - 32] = cid;
                }
                nbuf = more ? nbuf + nk - 32 : 0;
                keep = kw;
                rx = bx;
                ry = by;
                rz = bz;
                r2 = b2;
                j = bj;
                cid = bid;
            }
            const int st = run_window(keep, rx, ry, rz, r2, j, cid);
            if (st != ST_OK) return st;
            if (!more) break;
            if (bounded) bound();
        }
        __syncwarp();
        return ST_OK;
    };

    // The site's fractional position inside its bin, for a tighter per-bin
    // test than the gap key: a point of bin (b + o) lies at least
    // |o| - 1 + f (o < 0) or o - f (o > 0) bin sides from the site on each
    // axis.  Off-grid sites (cells of external points) skip the test.
    const float fx = (float)(__dmul_rn(sx - D.glo[0], D.inv[0]) - (double)cbx);
    const float fy = (float)(__dmul_rn(sy - D.glo[1], D.inv[1]) - (double)cby);
    const float fz = (float)(__dmul_rn(sz - D.glo[2], D.inv[2]) - (double)cbz);
    const bool near_ok = fx >= -1e-3f && fx <= 1.001f && fy >= -1e-3f && fy <= 1.001f && fz >= -1e-3f &&
                         fz <= 1.001f && D.has_extent;
    const float bsx = D.size_f[0], bsy = D.size_f[1], bsz = D.size_f[2];
    const float feps = D.frac_eps;
    // squared distance (bin units scaled by the bin sides) from the site to
    // the nearest point of the bin at offset (i, j, k), each gap shortened by
    // the in-bin position's error bound
    auto near2 = [&](int i, int j, int k) -> float {
        const float fxc = fminf(fmaxf(fx, 0.f), 1.f), fyc = fminf(fmaxf(fy, 0.f), 1.f),
                    fzc = fminf(fmaxf(fz, 0.f), 1.f);
        const float dx = i > 0 ? fmaxf((float)i - fxc - feps, 0.f) : (i < 0 ? fmaxf((float)(-i - 1) + fxc - feps, 0.f) : 0.f);
        const float dy = j > 0 ? fmaxf((float)j - fyc - feps, 0.f) : (j < 0 ? fmaxf((float)(-j - 1) + fyc - feps, 0.f) : 0.f);
        const float dz = k > 0 ? fmaxf((float)k - fzc - feps, 0.f) : (k < 0 ? fmaxf((float)(-k - 1) + fzc - feps, 0.f) : 0.f);
        const float ax = dx * bsx, ay = dy * bsy, az = dz * bsz;
        return ax * ax + ay * ay + az * az;
    };
    auto bin_of = [&](int i, int j, int k) -> long long {
        const int x = cbx + i, y = cby + j, z = cbz + k;
        if (x < 0 || x >= cpd || y < 0 || y >= cpd || z < 0 || z >= cpd) return -1;
        // no point of this bin can cut: it lies beyond twice the cell radius
        if (near_ok && near2(i, j, k) * (1.0f - 1e-4f) >= 4.f * R2f)
            return -1;
        return (long long)tess_chk(bin_base + ((uint64_t)x * cpd + y) * cpd + z, P.nbins, P.check, CK_BIN);
    };

    // Phases of the walk:
    //   0  crowded bins (when the site's own bin is crowded);
    //   1  the sorted shell table, 32 entries per batch (one per lane); the
    //      next batch's entries and bin ranges are loaded before the current
    //      batch is cut, so their latency overlaps the cutting;
    //   2  Chebyshev rings beyond the table (sparse regions).
    // They run as one loop with one call of process(), so the window and cut
    // code is inlined once: with a copy per phase, instruction fetch limited
    // the pass (crowded bins of the clustered 4M set: 238 -> 214 ms).
    uint32_t t = 0;
    // a batch entry: offsets, key and, after the bin test, the sorted range
    struct Ent {
        int i, j, k;
        float key;
        unsigned beg, cnt;
    };
    uint32_t done = 0;   // crowded bins already handled (see below)
    auto load_entry = [&](uint32_t idx, Ent& e) {
        e.i = e.j = e.k = 0;
        e.key = INFINITY;
        e.beg = e.cnt = 0;
        if (idx < tab_len) {
            const TabEntry te = tab[idx];
            e.i = te.i;
            e.j = te.j;
            e.k = te.k;
            e.key = te.key;
            if (has_radius && gap_key(D.size, e.i, e.j, e.k) > radius) e.key = INFINITY;
            long long lb = bin_of(e.i, e.j, e.k);
            if (done && abs(e.i) <= 1 && abs(e.j) <= 1 && abs(e.k) <= 1 &&
                ((done >> ((e.i + 1) * 9 + (e.j + 1) * 3 + (e.k + 1))) & 1u))
                lb = -1;   // handled among the crowded bins
            if (lb >= 0) {
                e.beg = P.delims[lb];
                e.cnt = P.delims[lb + 1] - e.beg;
            }
        }
    };
    int ph = 1;
    // ---- phase 0: crowded bins first ----
    // When the site's own bin is crowded, it and every crowded neighbour bin
    // still within reach are handled one at a time, nearest first, in two
    // steps each: the 32 seeds (the nearest point of each lane's stride of
    // the bin) are cut nearest first, then the bin's windows, each lane
    // skipping its own seed (window lane = position mod 32, the seed's
    // stride).  The shell walk skips the bins done here (27-bit mask `done`
    // over the offsets {-1,0,1}^3).
    // (their ranges and distances wait in shared memory: in registers they
    // would stay live through every later cut)
    bool seed_step = true;       // phase 0: the next step cuts a bin's seeds
    {
        const uint64_t sb = tess_chk(bin_base + ((uint64_t)cbx * cpd + cby) * cpd + cbz, P.nbins, P.check, CK_BIN);
        if (P.delims[sb + 1] - P.delims[sb] >= P.seed_min) {
            const int ti = lane / 9 - 1, tj = (lane / 3) % 3 - 1, tk = lane % 3 - 1;
            unsigned nb = 0, nc = 0;
            float dn = INFINITY;
            if (lane < 27) {
                const long long lb = bin_of(ti, tj, tk);
                if (lb >= 0 && !(has_radius && gap_key(D.size, ti, tj, tk) > radius)) {
                    nb = P.delims[lb];
                    nc = P.delims[lb + 1] - nb;
                }
                dn = lane == 13 ? 0.f : (near_ok ? near2(ti, tj, tk) : INFINITY);
            }
            S.nbeg[lane] = nb;
            S.ncnt[lane] = nc;
            S.nd[lane] = dn;
            S.pending = __ballot_sync(FULL, nc >= P.seed_min && dn < INFINITY);
            __syncwarp();
            ph = 0;
        }
    }
    Ent ea;
    bool loaded = false;                 // phase 1: the first batch is loaded
    S.ring = 1;
    S.r0 = 0;
    while (status == ST_OK) {
        unsigned ba = 0, ca = 0;
        bool direct = false;
        if (ph == 0) {
            if (seed_step) {
                const unsigned pending = S.pending;
                if (!pending) {
                    ph = 1;
                    continue;
                }
                const unsigned ndkey = (__float_as_uint(S.nd[lane]) & ~31u) | (unsigned)lane;
                const unsigned best = __reduce_min_sync(FULL, ((pending >> lane) & 1u) ? ndkey : 0xFFFFFFFFu);
                const int cbin = (int)(best & 31u);
                S.pending = pending & ~(1u << cbin);
                S.cbin = cbin;
                // still within reach of the (shrinking) cell?
                if (cbin != 13 && S.nd[cbin] * (1.0f - 1e-4f) >= 4.f * R2f)
                    continue;
                const unsigned sbeg = S.nbeg[cbin], scnt = S.ncnt[cbin];
                double drx = 0, dry = 0, drz = 0, dr2 = (double)INFINITY;
                seedj = 0xFFFFFFFFu;
                for (unsigned q = lane; q < scnt; q += 32) {
                    const uint32_t j = tess_chk(sbeg + q, P.npts, P.check, CK_POINT);
                    double rx, ry, rz, r2;
                    cand(j, rx, ry, rz, r2);
                    bool keep = (j != self) && r2 > 0.0 && r2 < dr2;
                    if (keep && tgroup >= 0) keep = (int64_t)(P.sgroup ? P.sgroup[j] : 0u) == tgroup;
                    if (keep) {
                        drx = rx;
                        dry = ry;
                        drz = rz;
                        dr2 = r2;
                        seedj = j;
                    }
                }
                S.sdx[lane] = drx;
                S.sdy[lane] = dry;
                S.sdz[lane] = drz;
                S.sd2[lane] = dr2;
                S.sdj[lane] = seedj;
                S.sdcid[lane] = seedj != 0xFFFFFFFFu ? (int32_t)(P.sorted[seedj] - pt_base) : 0;
                direct = true;
                seed_step = false;
            } else {
                // the bin as lane 0's range (window lane = position mod 32)
                ba = S.nbeg[S.cbin];
                ca = lane == 0 ? S.ncnt[S.cbin] : 0u;
                seed_step = true;
            }
        } else if (ph == 1) {
            if (!loaded) {
                load_entry(lane, ea);
                loaded = true;
            }
            // The table key is rounded toward zero and the threshold up, so
            // stopping on key >= thr never drops a bin that could hold a cutter.
            const float thr = 4.f * R2f * (float)kStopMargin;
            const unsigned ma = __ballot_sync(FULL, !(ea.key < thr));
            const int na = ma ? __ffs(ma) - 1 : 32;
            ba = ea.beg;
            ca = lane < na ? ea.cnt : 0u;
            // re-test the bins against the current (smaller) radius
            if (ca && near_ok &&
                near2(ea.i, ea.j, ea.k) * (1.0f - 1e-4f) >= 4.f * R2f)
                ca = 0;
            t += (uint32_t)na;
            if (ma) {
                ph = (t >= tab_len) && isfinite(D.tab_kmax) ? 2 : 3;
            } else {
                load_entry(t + lane, ea);
            }
            ++W.batches;
        } else if (ph == 2) {
            const int ring = S.ring;
            const uint32_t r0 = S.r0;
            if (r0 == 0) {
                // a new ring: stop when even its nearest bins are out of reach
                double lbk = (double)(ring - 1) * D.min_size;
                lbk = lbk * lbk;
                if (lbk < D.tab_kmax) lbk = D.tab_kmax;
                if (ring > cpd - 1 || lbk >= 4.0 * (double)R2 * kStopMargin || (radius >= 0.0 && lbk > radius)) {
                    ph = 3;
                    continue;
                }
            }
            const uint32_t rs = 24u * (uint32_t)ring * (uint32_t)ring + 2u;
            const double thr = 4.0 * (double)R2 * kStopMargin;
            long long lb = -1;
            const uint32_t r = r0 + lane;
            if (r < rs) {
                int i, j, k;
                ring_offset(ring, r, i, j, k);
                const double key = gap_key(D.size, i, j, k);
                if (key > D.tab_kmax && key < thr && !(radius >= 0.0 && key > radius)) lb = bin_of(i, j, k);
            }
            S.r0 = r0 + 32 < rs ? r0 + 32 : 0u;
            S.ring = r0 + 32 < rs ? ring : ring + 1;
            if (!__any_sync(FULL, lb >= 0)) continue;
            ++W.batches;
            if (lb >= 0) {
                ba = P.delims[lb];
                ca = P.delims[lb + 1] - ba;
            }
        } else {
            break;
        }
        status = process(ba, ca, direct);
        if (ph == 0 && seed_step) {
            // a crowded bin's windows are done
            seedj = 0xFFFFFFFFu;
            done |= 1u << S.cbin;
        }
    }

    // ---- finalize: faces, areas, volume in FP64 (polyhedron.rs:776-855) ----
    int nlive = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) nlive += __popc(C.lm[k]);
    double vol = 0.0;
    int F = 0;
    constexpr int R = (S_t::P + 31) / 32;
    double farea[R];
    int fdegr[R];
    if (status == ST_OK) {
        for (int i = lane; i < C.np; i += 32) S.fdeg[i] = 0;
        __syncwarp();
        bool fbad = false;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if ((C.lm[k] >> lane) & 1u) {
                const int s = k * 32 + lane;
                const uint32_t tt = S.tri[s];
#pragma unroll
                for (int e = 0; e < 3; ++e) {
                    const int p = plane_of(tt, e);
                    if (p < C.np) {
                        atomicAdd(&S.fdeg[p], 1u);
                        S.fsta[p] = (uint8_t)s;
                    } else {
                        fbad = true;
                    }
                }
            }
        }
        __syncwarp();
        bool bad = fbad;
        double vpart = 0.0;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int p = r * 32 + lane;
            farea[r] = 0.0;
            fdegr[r] = 0;
            if (p < C.np && S.fdeg[p] > 0) {
                const int start = tess_chk((int)S.fsta[p], S_t::V, P.check, CK_SLOT);
                int cur = start, steps = 0;
                double ax = 0.0, ay = 0.0, az = 0.0;
                do {
                    const uint32_t tt = S.tri[cur], aa = S.adj[cur];
                    const int i = plane_of(tt, 0) == p ? 0 : (plane_of(tt, 1) == p ? 1 : 2);
                    const int nx = plane_of(aa, i);
                    if (plane_of(tt, i) != p || nx >= S_t::V) {
                        bad = true;
                        break;
                    }
                    const double X0 = (double)S.vx[cur], X1 = (double)S.vy[cur], X2 = (double)S.vz[cur];
                    const double Y0 = (double)S.vx[nx], Y1 = (double)S.vy[nx], Y2 = (double)S.vz[nx];
                    // the walk runs clockwise seen from outside: Y x X is outward
                    ax += Y1 * X2 - Y2 * X1;
                    ay += Y2 * X0 - Y0 * X2;
                    az += Y0 * X1 - Y1 * X0;
                    cur = nx;
                    ++steps;
                } while (cur != start && steps <= S_t::V);
                const double A0 = (double)S.vx[start], A1 = (double)S.vy[start], A2 = (double)S.vz[start];
                vpart += (ax * A0 + ay * A1 + az * A2) * 0.5;
                farea[r] = 0.5 * sqrt(ax * ax + ay * ay + az * az);
                bad |= (cur != start) || (steps != (int)S.fdeg[p]) || steps < 3;
                fdegr[r] = steps;
            }
        }
        // volume: sum of pyramids from the site, area * height / 3
        // (compute_volume, polyhedron.rs:838-855)
        vol = warp_sum_d(vpart) / 3.0;
#pragma unroll
        for (int r = 0; r < R; ++r) F += __popc(__ballot_sync(FULL, fdegr[r] > 0));
        // Every vertex has three faces: V - E + F = 2 with E = 3V/2.
        if (nlive > 0 && F != nlive / 2 + 2) bad = true;
        if (__any_sync(FULL, bad)) status = ST_DEGEN;
    }

    // ---- outputs ----
    if (status != ST_OK) {
        if (GEO) {
            if (lane == 0) P.geo->status = status;
            return;
        }
        if (lane == 0) {
            if (P.reasons) atomicAdd(&P.reasons[status], 1u);
            if ((status == ST_VCAP || status == ST_PCAP) && P.list_cap) {
                P.list_cap[tess_chk(atomicAdd(P.list_cap_count, 1u), P.npts, P.check, CK_LIST)] = gs;
                P.status[orig] = ST_PENDING;
            } else {
                P.status[orig] = (uint8_t)status;
                P.vol[orig] = 0.0;
                P.nface[orig] = 0;
                atomicAdd(P.fail_count, 1u);
            }
        }
        return;
    }
    // compact live face ids, rank faces by id (faces are reported sorted)
    {
        int base = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int p = r * 32 + lane;
            const unsigned m = __ballot_sync(FULL, fdegr[r] > 0);
            if (fdegr[r] > 0) S.flist[base + __popc(m & ((1u << lane) - 1u))] = S.pid[p];
            base += __popc(m);
        }
        __syncwarp();
    }
    int rank[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        rank[r] = 0;
        if (fdegr[r] > 0) {
            const int32_t my = S.pid[r * 32 + lane];
            for (int q = 0; q < F; ++q) rank[r] += S.flist[q] < my;
        }
    }
    if (GEO) {
        GeoOut* G = P.geo;
        // vertices: live slots renumbered in slot order
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if ((C.lm[k] >> lane) & 1u) {
                int vi = __popc(C.lm[k] & ((1u << lane) - 1u));
#pragma unroll
                for (int kk = 0; kk < K; ++kk)
                    if (kk < k) vi += __popc(C.lm[kk]);
                const int s = k * 32 + lane;
                G->verts[3 * vi] = (double)S.vx[s];
                G->verts[3 * vi + 1] = (double)S.vy[s];
                G->verts[3 * vi + 2] = (double)S.vz[s];
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (fdegr[r] > 0) {
                S.rank2p[rank[r]] = (uint8_t)(r * 32 + lane);
                G->face_nbr[rank[r]] = S.pid[r * 32 + lane];
                G->face_area[rank[r]] = farea[r];
            }
        }
        __syncwarp();
        if (lane == 0) {
            int off = 0;
            for (int q = 0; q < F; ++q) {
                const int p = S.rank2p[q];
                G->face_off[q] = off;
                const int deg = (int)S.fdeg[p];
                const int start = tess_chk((int)S.fsta[p], S_t::V, P.check, CK_SLOT);
                int cur = start;
                // reversed walk: counter-clockwise seen from outside
                for (int st = 0; st < deg; ++st) {
                    int vi = 0;
                    for (int k = 0; k < K; ++k) {
                        if ((cur >> 5) == k) vi += __popc(C.lm[k] & ((1u << (cur & 31)) - 1u));
                        else if ((cur >> 5) > k) vi += __popc(C.lm[k]);
                    }
                    G->face_vtx[tess_chk(off + (deg - st) % deg, 3 * 256, P.check, CK_FACE)] = vi;
                    const uint32_t tt = S.tri[cur], aa = S.adj[cur];
                    const int i = plane_of(tt, 0) == p ? 0 : (plane_of(tt, 1) == p ? 1 : 2);
                    cur = plane_of(aa, i) % S_t::V;
                }
                off += deg;
            }
            G->face_off[F] = off;
            G->nv = nlive;
            G->nf = F;
            G->volume = vol;
            G->status = ST_OK;
        }
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
        return;   // the host sees the face cursor past the capacity and recomputes
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (fdegr[r] > 0) {
            const unsigned long long fi = tess_chk(fbase + rank[r], P.face_cap, P.check, CK_FACE);
            P.face_nbr[fi] = S.pid[r * 32 + lane];
            P.face_area[fi] = farea[r];
        }
    }
    if (lane == 0) {
        P.vol[orig] = vol;
        P.nface[orig] = (uint32_t)F;
        P.fstart[orig] = fbase;
        P.status[orig] = ST_OK;
    }
}

// K = 2: 8 warps per block, two blocks per SM (registers capped at 128).
template <int K, bool GEO>
__global__ void __launch_bounds__(K == 2 ? 256 : 128, K == 2 ? 2 : 1) k_clip(ClipParams P) {
    after_previous();
    extern __shared__ __align__(16) unsigned char smraw[];
    Smem<K>& S = reinterpret_cast<Smem<K>*>(smraw)[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const unsigned n1 = P.work_count ? *P.work_count : P.total, n2 = P.work2 ? *P.work2_count : 0u;
    unsigned total = (P.work_least && n1 <= P.work_least ? 0u : n1) + (n2 <= P.work2_most ? n2 : 0u);
    if (P.grid_err && *P.grid_err == 1) total = 0;   // non-finite input: nothing to clip
    Work W;
    while (total) {
        unsigned w = 0;
        if (lane == 0) w = atomicAdd(P.cursor, 1u);
        w = __shfl_sync(FULL, w, 0);
        if (w >= total) break;
        const uint32_t gs = w >= n1 ? P.work2[w - n1] : (P.work ? P.work[w] : w);
        run_cell<K, GEO>(P, S, gs, lane, W);
    }
    if (P.work_ctr && lane == 0) {
        atomicAdd(&P.work_ctr[0], (unsigned long long)W.tested);
        atomicAdd(&P.work_ctr[1], (unsigned long long)W.cuts);
        atomicAdd(&P.work_ctr[2], (unsigned long long)W.newv);
        atomicAdd(&P.work_ctr[3], (unsigned long long)W.windows);
        atomicAdd(&P.work_ctr[4], (unsigned long long)W.batches);
    }
}

// Raise the kernel's dynamic shared memory limit to what `bytes` needs, once
// per size and device: cudaFuncSetAttribute applies to the current device
// only, so the limit is remembered per device ordinal.  A mutex keeps two
// host threads from lowering each other's limit.  Kept out of stream capture
// by the host's warm-up calls.
constexpr int kMaxDevices = 64;
template <int K, bool GEO>
cudaError_t configure_smem(size_t bytes) {
    static std::mutex mu;
    static size_t configured[kMaxDevices] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    size_t* slot = (dev >= 0 && dev < kMaxDevices) ? &configured[dev] : nullptr;
    if (slot && bytes <= *slot) return cudaSuccess;
    e = cudaFuncSetAttribute(k_clip<K, GEO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess && slot) *slot = bytes;
    return e;
}

template <int K, bool GEO>
cudaError_t launch_t(const ClipParams& p, int wpb, int blocks, cudaStream_t s) {
    const size_t sm = sizeof(Smem<K>) * (size_t)wpb;
    cudaError_t e = configure_smem<K, GEO>(sm);
    if (e != cudaSuccess) return e;
    return launch_after(k_clip<K, GEO>, blocks, 32 * wpb, sm, s, p);
}

template <int K, bool GEO>
int blocks_t(int wpb, int device) {
    const size_t sm = sizeof(Smem<K>) * (size_t)wpb;
    int per = 0, nsm = 0;
    if (configure_smem<K, GEO>(sm) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_clip<K, GEO>, 32 * wpb, sm) != cudaSuccess)
        per = 1;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
    cudaGetLastError();   // leave no sticky error behind a failed query
    if (per < 1) per = 1;
    return per * (nsm > 0 ? nsm : 1);
}

}  // namespace clipk
}  // namespace tess

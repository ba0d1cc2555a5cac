// tess_radius.cu -- fixed-radius queries on the bin grid (sm_103a).
//
// Four query kinds share one kernel body:
//   RQ_CELLS        Celery::find_cells_in_radius (celery.rs:753-796): the bins
//                   of the box [q - r, q + r] (clamped to the point bounds)
//                   whose gap distance to q's bin is within r
//                   (check_cell_in_range, celery.rs:708-748), in i, j, k order.
//   RQ_CELL_RADIUS  find_neighbors_in_cell_radius (celery.rs:802-818): every
//                   point of those bins, bin by bin.
//   RQ_REAL_RADIUS  find_neighbors_in_real_radius (celery.rs:825-855): those
//                   points whose squared distance (celery.rs:700-702) is at
//                   most r * r.
//   RQ_CLOUD        Cell::compute_neighbor_cloud (interface.rs:348-365): the
//                   expanding search from the cell's position over the search
//                   order up to the first key above r (celery.rs:1023-1075),
//                   optionally filtered by group.
//
// Large batches of the two point queries take a lane per query (k_radius_lane,
// below); else one warp answers one query.  The warp takes 32 candidate bins at
// a time (box cells or search-order entries), keeps the ones in range, and then
// walks the kept bins' points as one concatenated stream, 32 points per step:
// a warp prefix sum of the bins' counts maps each lane to its bin.  Results
// stay in the reference's order (bins in query order, sorted_indices order
// within a bin, which is ascending point index here) because every step
// compacts with a ballot.  Each query runs twice: a count pass, then (after a
// scan of the counts into offsets) a fill pass that writes at the offsets.
// All FP64 arithmetic is correctly rounded with no contraction, so the bins
// and points found are the reference's exactly.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "tess_internal.cuh"

namespace tess {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr uint32_t kLongRun = 64;     // points of a row from which a warp shares them
constexpr int kLaneThreads = 128;     // threads of such a block
constexpr int kLaneRows = 16;         // rows listed at a time

__device__ __forceinline__ double sq_rn(double a) { return __dmul_rn(a, a); }

struct WarpOut {
    uint64_t pos;   // fill pass: next output slot of this query
    uint32_t cnt;   // results so far
};

// One query as the point test sees it: the FP64 position and radius of the
// reference's arithmetic, and an FP32 pre-filter.  The filter decides a
// candidate when its FP32 squared distance (from the points' FP32 high
// parts) is farther than `band` from r^2, where `band` bounds the FP32
// estimate's error against the exact squared distance; inside the band the
// exact FP64 test decides.  Either way the answer is the FP64 one.
struct QueryTest {
    double x, y, z, r2;
    float fx, fy, fz;
    float lo_thr, hi_thr;   // accept below, reject above (when on)
    bool on;
};

// Kept out of line: inlined, the compiler predicates these FP64 operations
// into every candidate step, and predicated-off FP64 instructions still take
// the (slow) FP64 pipe's issue slots.
__device__ __noinline__ bool exact_within(const RadiusParams& p, double x, double y, double z, double r2, uint32_t s) {
    // distance_squared(x, y, z, point), celery.rs:700-702
    const double dx = __dsub_rn(x, p.spx[s]);
    const double dy = __dsub_rn(y, p.spy[s]);
    const double dz = __dsub_rn(z, p.spz[s]);
    return __dadd_rn(__dadd_rn(sq_rn(dx), sq_rn(dy)), sq_rn(dz)) <= r2;
}

// Up to 32 runs (one per lane: first element `beg`, length `c`) as one
// stream in lane order.  The elements are sorted positions of points, or
// bin ids for RQ_CELLS.
template <int MODE, bool FILL>
__device__ __forceinline__ void emit_stream(const RadiusParams& p, uint32_t beg, uint32_t c, const QueryTest& qt,
                                            uint32_t pt_base, int lane, WarpOut& w) {
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += t;
    }
    const uint32_t tot = __shfl_sync(kFull, incl, 31);
    if (tot == 0) return;
    const bool test = MODE == RQ_REAL_RADIUS || (MODE == RQ_CLOUD && p.group >= 0);
    if (!test && !FILL) {
        w.cnt += tot;
        return;
    }
    if (MODE == RQ_CELLS) {
        const uint32_t ex = incl - c;
        for (uint32_t o = 0; o < tot; o += 32) {
            const uint32_t t = o + lane;
            int L = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const uint32_t v = __shfl_sync(kFull, incl, L + step - 1);
                if (v <= t) L += step;
            }
            const uint32_t e0 = __shfl_sync(kFull, ex, L);
            const uint32_t b0 = __shfl_sync(kFull, beg, L);
            if (t < tot) p.out[w.pos + t - o] = b0 + (t - e0);
            w.pos += min(32u, tot - o);
        }
        w.cnt += tot;
        return;
    }
    const uint32_t excl = incl - c;
    const unsigned lt = (1u << lane) - 1u;
    for (uint32_t o = 0; o < tot; o += 32) {
        const uint32_t t = o + lane;
        // owner lane: the first lane whose inclusive count exceeds t
        int L = 0;
#pragma unroll
        for (int step = 16; step > 0; step >>= 1) {
            const uint32_t v = __shfl_sync(kFull, incl, L + step - 1);
            if (v <= t) L += step;
        }
        const uint32_t ex = __shfl_sync(kFull, excl, L);
        const uint32_t b0 = __shfl_sync(kFull, beg, L);
        const bool valid = t < tot;
        bool ok = valid;
        const uint32_t s = b0 + (t - ex);
        if (MODE == RQ_REAL_RADIUS) {
            bool band = false;
            if (qt.on) {
                if (valid) {
                    const float4 h = p.phi[s];
                    const float dx = __fsub_rn(qt.fx, h.x);
                    const float dy = __fsub_rn(qt.fy, h.y);
                    const float dz = __fsub_rn(qt.fz, h.z);
                    const float d2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
                    ok = d2 < qt.lo_thr;
                    band = !ok && !(d2 > qt.hi_thr);      // NaN lands in the band
                }
            } else {
                band = valid;
                ok = false;
            }
            if (__any_sync(kFull, band) && band) ok = exact_within(p, qt.x, qt.y, qt.z, qt.r2, s);
        }
        if (MODE == RQ_CLOUD && ok && p.group >= 0) ok = (int64_t)(p.sgroup ? p.sgroup[s] : 0u) == p.group;
        const unsigned bal = __ballot_sync(kFull, ok);
        if (FILL && ok) p.out[w.pos + __popc(bal & lt)] = p.sorted[s] - pt_base;
        w.pos += __popc(bal);
        w.cnt += __popc(bal);
    }
}

// One batch of up to 32 candidate bins (one per lane).
template <int MODE, bool FILL>
__device__ __forceinline__ void emit_bins(const RadiusParams& p, bool keep, uint32_t bin, uint64_t bin_base,
                                          const QueryTest& qt, uint32_t pt_base, int lane, WarpOut& w) {
    uint32_t beg = 0, c = 0;
    if (keep) {
        beg = p.delims[bin_base + bin];
        c = p.delims[bin_base + bin + 1] - beg;
    }
    emit_stream<MODE, FILL>(p, beg, c, qt, pt_base, lane, w);
}

// A double to float, rounded toward zero, from the bit pattern alone (no
// FP64-pipe conversion): |result| <= |v| and |v - result| < 2^-23 |v| in the
// float range; below it 0 (error under 2^-126), above it (and NaN) +-inf.
__device__ __forceinline__ float f64_to_f32_rz(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const unsigned sign = (unsigned)(b >> 63) << 31;
    const int e = (int)((b >> 52) & 0x7FF) - 1023 + 127;
    if (e <= 0) return __uint_as_float(sign);
    if (e >= 255) return __uint_as_float(sign | 0x7F800000u);
    return __uint_as_float(sign | ((unsigned)e << 23) | (unsigned)((b >> 29) & 0x7FFFFFu));
}

__device__ __forceinline__ bool is_nan_bits(unsigned long long b) {
    return (b & 0x7FFFFFFFFFFFFFFFull) > 0x7FF0000000000000ull;
}

// axis_index(v) (celery.rs:269-314) without FP64 arithmetic: axis_index is
// monotone in v, so it is the number of bin boundaries at or below v, found by
// binary search over the order codes of the boundaries.  NaN gives 0, as
// axis_index does.
__device__ __forceinline__ int axis_index_table(unsigned long long vbits, const unsigned long long* b, int cpd,
                                                int top) {
    if (is_nan_bits(vbits)) return 0;
    const unsigned long long e = (vbits >> 63) ? ~vbits : (vbits | 0x8000000000000000ull);
    int i = 0;
    for (int step = top; step > 0; step >>= 1)
        if (i + step < cpd && __ldg(b + i + step) <= e) i += step;
    return i;
}

// Smallest double (as an order code) whose axis_index is >= i, by binary
// search over the order codes between -inf and +inf, evaluating the exact
// FP64 axis_index.
__global__ void k_axis_bounds(const DiagDesc* desc, int cpd, unsigned long long* bnd) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 3 * cpd) return;
    const int a = t / cpd, i = t % cpd;
    const DiagDesc& D = desc[0];
    if (i == 0) {
        bnd[t] = 0ull;
        return;
    }
    unsigned long long lo = ord_enc(-INFINITY), hi = ord_enc(INFINITY);   // axis_index(+inf) = cpd - 1 >= i
    while (lo < hi) {
        const unsigned long long mid = lo + (hi - lo) / 2;
        if (axis_index(ord_dec(mid), D.glo[a], D.ghi[a], D.inv[a], cpd) >= i)
            hi = mid;
        else
            lo = mid + 1;
    }
    bnd[t] = lo;
}

// check_cell_in_range's squared gap distance (celery.rs:708-748) in FP64;
// out of line for the same reason as exact_within.
__device__ __noinline__ double gap_ds(int gx, int gy, int gz, double sz0, double sz1, double sz2) {
    return __dadd_rn(__dadd_rn(sq_rn(__dmul_rn((double)gx, sz0)), sq_rn(__dmul_rn((double)gy, sz1))),
                     sq_rn(__dmul_rn((double)gz, sz2)));
}

template <int MODE, bool FILL>
__global__ void __launch_bounds__(256) k_radius(RadiusParams p) {
    const int lane = threadIdx.x & 31;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const DiagDesc& D = p.desc[0];
    const int cpd = D.cpd;
    const uint64_t bin_base = D.bin_base;
    const uint32_t pt_base = D.pt_base;
    const double sz0 = D.size[0], sz1 = D.size[1], sz2 = D.size[2];
    const double r = p.radius;
    const double r2 = p.radius2;
    // Per-lane axis for the spread evaluation of the query's bin indices:
    // lanes 0-2 the query's own bin (x, y, z), lanes 3-5 the box's low end,
    // lanes 6-8 its high end (celery.rs:753-778); other lanes repeat lane % 3.
    const int ax = lane % 3;
    const int kind = lane < 9 ? lane / 3 : 0;
    const unsigned long long* abnd = p.bnd + ax * cpd;
    // box ends clamp to the point bounds: max_float(c - r, min), min_float(c + r, max)
    const unsigned long long clamp_bits =
        (unsigned long long)__double_as_longlong(kind == 2 ? D.ghi[ax] : D.glo[ax]);
    const unsigned long long clamp_code = (clamp_bits >> 63) ? ~clamp_bits : (clamp_bits | 0x8000000000000000ull);
    // lanes 9-11 form the query relative to the diagram's centre (the frame
    // of the points' FP32 parts) in the same FP64 add
    const double delta = kind == 1 ? -r : (kind == 2 ? r : (lane >= 9 && lane < 12 ? -D.ctr[ax] : 0.0));
    int top = 1;
    while (2 * top < cpd) top *= 2;
    // magnitude bound of the point coordinates relative to the centre, and
    // the radius, for the FP32 filter's error band
    double gm = 0.0;
    for (int a = 0; a < 3; ++a) gm = fmax(gm, fmax(fabs(D.glo[a] - D.ctr[a]), fabs(D.ghi[a] - D.ctr[a])));
    const float gmag = (float)gm;
    const float fr = (float)r;
    const float r2f = (float)r2;

    for (uint32_t wq0 = warp; wq0 < p.nq; wq0 += nwarps) {
        const uint32_t wq = p.qorder ? p.qorder[wq0] : wq0;
        uint32_t q = wq;
        double x, y, z;
        if (p.qxyz) {
            x = p.qxyz[3 * (size_t)wq];
            y = p.qxyz[3 * (size_t)wq + 1];
            z = p.qxyz[3 * (size_t)wq + 2];
        } else if (p.qcell) {
            const uint32_t c = p.qcell[wq];
            if (c >= D.n) {                     // not a cell of this diagram: no results, flagged
                if (lane == 0) {
                    if (!FILL) p.count[q] = 0;
                    atomicExch(p.err, 1);
                }
                continue;
            }
            const size_t g = (size_t)pt_base + c;
            x = p.xyz[3 * g];
            y = p.xyz[3 * g + 1];
            z = p.xyz[3 * g + 2];
        } else {
            // every cell, walked in bin order so neighbouring warps share bins
            const uint32_t s = pt_base + wq;
            q = p.sorted[s] - pt_base;
            x = p.spx[s];
            y = p.spy[s];
            z = p.spz[s];
        }
        WarpOut w{FILL ? p.offs[q] : 0, 0};
        QueryTest qt;
        qt.x = x;
        qt.y = y;
        qt.z = z;
        qt.r2 = r2;
        qt.on = false;

        // the bin indices this query needs, one per lane, with exact FP64
        // arithmetic: get_{x,y,z}_cell_index of the coordinate, of
        // max_float(c - r, min) and of min_float(c + r, max)
        const double ca = ax == 0 ? x : (ax == 1 ? y : z);
        unsigned long long vb = (unsigned long long)__double_as_longlong(ca);
        if (MODE != RQ_CLOUD) {
            // c - r (exactly c + (-r)) or c + r, one FP64 add for all lanes
            vb = (unsigned long long)__double_as_longlong(__dadd_rn(ca, delta));
            if (kind != 0) {
                // max_float / min_float: v is kept only when strictly inside
                // the bound (NaN: the bound)
                const unsigned long long ve = (vb >> 63) ? ~vb : (vb | 0x8000000000000000ull);
                const bool inside = kind == 1 ? ve > clamp_code : ve < clamp_code;
                if (is_nan_bits(vb) || !inside) vb = clamp_bits;
            }
        }
        const int idx = axis_index_table(vb, abnd, cpd, top);
        const int xi = __shfl_sync(kFull, idx, 0);
        const int yi = __shfl_sync(kFull, idx, 1);
        const int zi = __shfl_sync(kFull, idx, 2);

        if (MODE == RQ_CLOUD) {
            // ExpandingSearch::new, celery.rs:882-902
            for (uint32_t base = 0; base < p.rtab_len; base += 32) {
                const uint32_t t = base + lane;
                bool keep = false;
                uint32_t bin = 0;
                if (t < p.rtab_len) {
                    const short4 e = p.rtab[t];
                    const int X = xi + e.x, Y = yi + e.y, Z = zi + e.z;
                    keep = X >= 0 && X < cpd && Y >= 0 && Y < cpd && Z >= 0 && Z < cpd;
                    if (keep) bin = ((uint32_t)X * (uint32_t)cpd + (uint32_t)Y) * (uint32_t)cpd + (uint32_t)Z;
                }
                emit_bins<MODE, FILL>(p, keep, bin, bin_base, qt, pt_base, lane, w);
            }
        } else {
            // find_cells_in_radius, celery.rs:753-796
            const int i0 = __shfl_sync(kFull, idx, 3), j0 = __shfl_sync(kFull, idx, 4);
            const int k0 = __shfl_sync(kFull, idx, 5), i1 = __shfl_sync(kFull, idx, 6);
            const int j1 = __shfl_sync(kFull, idx, 7), k1 = __shfl_sync(kFull, idx, 8);
            if (MODE == RQ_REAL_RADIUS && p.f32_filter) {
                // error band of the FP32 squared distance, q and p relative to
                // the diagram's centre (each FP64-rounded, 2^-53 |q|): per axis
                // the query's truncation to FP32 (2^-23 |q|), the point's
                // rounding (2^-24 |p|) and the subtraction's (2^-24 |dq|), at most
                // e = 6e-8 (3 m + 2.1 r); squared and summed near r^2 that is
                // 2 sqrt(3) 1.01 r e + 3 e^2, plus 4 roundings of the sum and
                // the FP64 side, doubled
                // integer ops, the centre-relative coordinates of lanes 9-11
                const float fa = f64_to_f32_rz(__longlong_as_double((long long)vb));
                qt.fx = __shfl_sync(kFull, fa, 9);
                qt.fy = __shfl_sync(kFull, fa, 10);
                qt.fz = __shfl_sync(kFull, fa, 11);
                const float qmag = fmaxf(fmaxf(fabsf(qt.fx), fabsf(qt.fy)), fabsf(qt.fz));
                const float m = fmaxf(gmag, qmag) * 1.0001f;
                const float e = 6.0e-8f * (3.0f * m + 2.1f * fr);
                const float band = 2.0f * (3.5f * fr * e + 3.0f * e * e) + 1.0e-6f * r2f;
                qt.lo_thr = r2f - band;
                qt.hi_thr = r2f + band;
                qt.on = m < 1.0e18f;
            }
            // The box's rows (i, j), i-major, one per lane.  Within a row the
            // kept bins are those whose gap gz = max(|zi - k| - 1, 0) is at
            // most the row's limit T (the gap distance grows with gz), i.e. one
            // contiguous k range around zi; its points are one contiguous run
            // of the sorted order (bins in k order, sorted order within).
            const int nx = i1 - i0 + 1, ny = j1 - j0 + 1;
            const int nrows = (nx > 0 && ny > 0 && k1 >= k0) ? nx * ny : 0;
            for (int base = 0; base < nrows; base += 32) {
                const int t = base + lane;
                uint32_t beg = 0, c = 0;
                if (t < nrows) {
                    const int i = i0 + t / ny, j = j0 + t % ny;
                    const int gx = max(abs(xi - i) - 1, 0), gy = max(abs(yi - j) - 1, 0);
                    const int gz_need = max(max(zi - k0, k1 - zi) - 1, 0);   // largest gap in the row
                    int T = -1;
                    int from = 0;
                    if (p.gtab && gx <= p.gtab_x && gy <= p.gtab_y) {
                        T = __ldg(p.gtab + gx * (p.gtab_y + 1) + gy);
                        from = T == p.gtab_z ? p.gtab_z + 1 : gz_need + 1;    // table ends at gtab_z
                    }
                    for (int gz = from; gz <= gz_need; ++gz) {                 // FP64 rows (rare)
                        if (!(gap_ds(gx, gy, gz, sz0, sz1, sz2) <= r2)) break;
                        T = gz;
                    }
                    if (T >= 0) {
                        const int kl = max(k0, zi - T - 1), kh = min(k1, zi + T + 1);
                        if (kl <= kh) {
                            const uint32_t row = ((uint32_t)i * (uint32_t)cpd + (uint32_t)j) * (uint32_t)cpd;
                            if (MODE == RQ_CELLS) {
                                beg = row + (uint32_t)kl;
                                c = (uint32_t)(kh - kl + 1);
                            } else {
                                beg = p.delims[bin_base + row + (uint32_t)kl];
                                c = p.delims[bin_base + row + (uint32_t)kh + 1] - beg;
                            }
                        }
                    }
                }
                emit_stream<MODE, FILL>(p, beg, c, qt, pt_base, lane, w);
            }
        }
        if (!FILL && lane == 0) p.count[q] = w.cnt;
    }
}

// The bin indices of k_radius_lane that FP32 leaves open, exactly: bit 3 a + e of
// `open` is axis a's e-th of the query's own bin, the box's low and its high end.
__device__ __noinline__ int exact_index(const RadiusParams& p, double c, int a, int e, int top) {
    const DiagDesc& D = p.desc[0];
    unsigned long long v = (unsigned long long)__double_as_longlong(e == 0 ? c : __dadd_rn(c, e == 2 ? p.radius : -p.radius));
    if (e != 0) {
        const unsigned long long clamp = (unsigned long long)__double_as_longlong(e == 2 ? D.ghi[a] : D.glo[a]);
        const unsigned long long cc = (clamp >> 63) ? ~clamp : (clamp | 0x8000000000000000ull);
        const unsigned long long ve = (v >> 63) ? ~v : (v | 0x8000000000000000ull);
        if (is_nan_bits(v) || !(e == 2 ? ve < cc : ve > cc)) v = clamp;
    }
    return axis_index_table(v, p.bnd + a * D.cpd, D.cpd, top);
}

// Square root to 2 ulp, of a positive number.
__device__ __forceinline__ float sqrt_near(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Whether point s is within the radius of query q, exactly (rare).
__device__ __noinline__ bool exact_query(const RadiusParams& p, uint32_t q, uint32_t s) {
    const double* c = p.qxyz + 3 * (size_t)q;
    return exact_within(p, c[0], c[1], c[2], p.radius2, s);
}

// RQ_REAL_RADIUS and RQ_CELL_RADIUS with one query per lane: the same rows and
// the same order of the results.  A warp per query spends its instructions on
// finding the query's bins and on mapping lanes to them (300 for 110 points); a
// lane per query does that once for 32 queries.  Further:
//   - The bins come from FP32 places; what is too near a boundary is looked up.
//   - Only bins that the ball reaches are read (85 points instead of 110 with a
//     radius of one bin).
//   - The rows are listed first; then each lane goes through its own points,
//     four at a time, whatever row the others are at.
//   - A counting pass of real radius queries also lists each query's first
//     p.stage_len results, so that only the queries with more of them are found
//     again by a second pass (542 -> 421 us).
//   - A long row of a few lanes (clusters) is taken by the whole warp.
// 1,000,000 queries with 16 results each among 1,000,000 points: the two passes
// 1,650 us by warps; this one 225 and k_radius_place 45.  Bound by the latency
// and the wavefronts of the scattered 16-byte reads (L1 63% busy, issue 55%):
// 24 warps per SM; 20 and 28 are no faster, nor is reading four points ahead.
template <int MODE, bool FILL>
__global__ void __launch_bounds__(kLaneThreads, 6) k_radius_lane(RadiusParams p) {
    static_assert(MODE == RQ_REAL_RADIUS || MODE == RQ_CELL_RADIUS, "other queries take a warp each");
    constexpr bool REAL = MODE == RQ_REAL_RADIUS;
    __shared__ uint2 rows[kLaneRows][kLaneThreads];
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const uint64_t at = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool have = at < p.nq;
    const uint32_t q = have ? (p.qorder ? p.qorder[at] : (uint32_t)at) : 0u;
    if (FILL && have && p.stage_len) have = p.count[q] > p.stage_len;   // (the others are listed)
    if (!__any_sync(kFull, have)) return;
    const DiagDesc& D = p.desc[0];
    const int cpd = D.cpd;
    const uint64_t bin_base = D.bin_base;
    const uint32_t pt_base = D.pt_base;
    const double x = p.qxyz[3 * (size_t)q], y = p.qxyz[3 * (size_t)q + 1], z = p.qxyz[3 * (size_t)q + 2];
    const float fr = (float)p.radius, r2f = (float)p.radius2;

    // The query in FP32, relative to the diagram's centre and in bins.  Its place
    // in bins is known within feps: 2^-23 of the position, 2^-24 of the corner
    // and three roundings, at most 6 2^-24 cpd on the grid (8 taken), in
    // proportion off it; the same for the radius; and the FP64 rounding of c - r.
    const float qx = f64_to_f32_rz(__dadd_rn(x, -D.ctr[0])), qy = f64_to_f32_rz(__dadd_rn(y, -D.ctr[1])),
                qz = f64_to_f32_rz(__dadd_rn(z, -D.ctr[2]));
    const float px = (qx - D.glo_hi[0]) * D.inv_s[0], py = (qy - D.glo_hi[1]) * D.inv_s[1], pz = (qz - D.glo_hi[2]) * D.inv_s[2];
    const float away = fabsf(px) + fabsf(py) + fabsf(pz);
    const float inv_most = fmaxf(D.inv_s[0], fmaxf(D.inv_s[1], D.inv_s[2]));
    const float glo_most = fmaxf(fabsf(D.glo_f[0]), fmaxf(fabsf(D.glo_f[1]), fabsf(D.glo_f[2])));
    const float feps = 8.0f * 5.9604645e-8f * (float)cpd + 1e-6f + 1e-6f * away + 4e-7f * fabsf(fr) * inv_most +
                       1e-15f * glo_most * inv_most;
    const bool grid = D.lean_ok && D.inv_s[0] > 0.f && D.inv_s[1] > 0.f && D.inv_s[2] > 0.f && away < 1e6f && feps < 0.25f;

    // the query's bin and the box's ends.  A place further than feps from the
    // bin boundaries between 1 and cpd - 1 has its index; the others are
    // looked up.
    unsigned open = 0;
    auto index = [&](float u, int bit) {
        const float f = floorf(u), fr_ = u - f;
        const bool inner = u > 1.f - feps && u < (float)(cpd - 1) + feps;
        if (!grid || !(u == u) || (inner && (fr_ < feps || fr_ > 1.f - feps))) open |= 1u << bit;
        return min(max((int)f, 0), cpd - 1);
    };
    const float rx = fr * D.inv_s[0], ry = fr * D.inv_s[1], rz = fr * D.inv_s[2];
    int xi = index(px, 0), i0 = index(px - rx, 1), i1 = index(px + rx, 2);
    int yi = index(py, 3), j0 = index(py - ry, 4), j1 = index(py + ry, 5);
    int zi = index(pz, 6), k0 = index(pz - rz, 7), k1 = index(pz + rz, 8);
    if (open) {
        int top = 1;
        while (2 * top < cpd) top *= 2;
#pragma unroll 1
        for (; open; open &= open - 1u) {
            const int bit = __ffs(open) - 1, a = bit / 3;
            const int v = exact_index(p, p.qxyz[3 * (size_t)q + a], a, bit - 3 * a, top);
            if (bit == 0) xi = v;
            if (bit == 1) i0 = v;
            if (bit == 2) i1 = v;
            if (bit == 3) yi = v;
            if (bit == 4) j0 = v;
            if (bit == 5) j1 = v;
            if (bit == 6) zi = v;
            if (bit == 7) k0 = v;
            if (bit == 8) k1 = v;
        }
    }

    // FP32 filter: the error band of k_radius (the distance is summed from
    // -r^2 up, the same roundings)
    float band = INFINITY;      // nothing decided in FP32
    bool filter = false;
    if (REAL && p.f32_filter) {
        float m = fmaxf(fmaxf(fabsf(qx), fabsf(qy)), fabsf(qz));
#pragma unroll
        for (int a = 0; a < 3; ++a) m = fmaxf(m, fmaxf(fabsf(D.glo_hi[a]), fabsf(D.glo_hi[a] + D.size_f[a] * (float)cpd)));
        m *= 1.0001f;
        const float e = 6.0e-8f * (3.0f * m + 2.1f * fr);
        filter = m < 1.0e18f;
        if (filter) band = 2.0f * (3.5f * fr * e + 3.0f * e * e) + 1.0e-6f * r2f;
    }
    // Real radius: of the box's bins only those that the ball may reach.
    const bool tight = REAL && filter && grid;
    // A bin whose gap distance is beyond the radius is beyond the ball, so the gap
    // test leaves nothing out that the ball does not, unless some gap distance
    // is the radius to within the ball's margin (in squares 5e-4 and 6 feps).
    const bool gaps = !tight || !p.gtab || p.gtab_tie || !(feps < 1e-3f);
    const float fx = fminf(fmaxf(px - (float)xi, 0.f), 1.f), fy = fminf(fmaxf(py - (float)yi, 0.f), 1.f);
    const float sx = D.size_f[0], sy = D.size_f[1], inz = D.inv_s[2];

    // the results' places: one after the other, or (listed) a warp's first
    // results, its second ones, ... side by side
    constexpr uint32_t kStep = FILL ? 1 : 32;
    using Place = std::conditional_t<FILL, uint64_t, uint32_t>;     // (the lists have at most 2^31 entries)
    Place out = 0, end = 0;
    uint32_t cnt = 0;
    if (FILL && have) out = p.offs[q];
    if (!FILL && have) {
        out = (uint32_t)(at - lane) * p.stage_len + lane;
        end = out + 32 * p.stage_len;
    }
    uint32_t* const results = FILL ? p.out : p.stage;
    const int ny = j1 - j0 + 1, nx = i1 - i0 + 1;
    const int nrows = have && nx > 0 && ny > 0 && k1 >= k0 ? nx * ny : 0;
    const int gz_need = max(max(zi - k0, k1 - zi) - 1, 0);
    int i = i0, j = j0;
    // the points of row (i, j) that the query has to look at; on to the next row
    auto row = [&](uint32_t& beg, uint32_t& c) {
        const int di = i - xi, dj = j - yi;
        const uint32_t first = ((uint32_t)i * (uint32_t)cpd + (uint32_t)j) * (uint32_t)cpd;
        if (++j > j1) {
            j = j0;
            ++i;
        }
        int kl = k0, kh = k1;
        if (tight) {
            const float dx = fmaxf((di > 0 ? (float)di - fx : (di < 0 ? (float)(-di - 1) + fx : 0.f)) - feps, 0.f) * sx;
            const float dy = fmaxf((dj > 0 ? (float)dj - fy : (dj < 0 ? (float)(-dj - 1) + fy : 0.f)) - feps, 0.f) * sy;
            const float rem = r2f * 1.0003f - (dx * dx + dy * dy);
            if (!(rem > 0.f)) return;
            const float zr = fminf(sqrt_near(rem) * inz * 1.0001f + 2.f * feps, 4e6f);
            kl = max(kl, (int)floorf(pz - zr));
            kh = min(kh, (int)floorf(pz + zr));
        }
        if (gaps) {
            const int gx = max(abs(di) - 1, 0), gy = max(abs(dj) - 1, 0);
            int T = -1, from = 0;
            if (p.gtab && gx <= p.gtab_x && gy <= p.gtab_y) {
                T = __ldg(p.gtab + gx * (p.gtab_y + 1) + gy);
                from = T == p.gtab_z ? p.gtab_z + 1 : gz_need + 1;
            }
            for (int gz = from; gz <= gz_need; ++gz) {
                if (!(gap_ds(gx, gy, gz, D.size[0], D.size[1], D.size[2]) <= p.radius2)) break;
                T = gz;
            }
            kl = max(kl, zi - T - 1);
            kh = min(kh, zi + T + 1);
            if (T < 0) return;
        }
        if (kl > kh) return;
        beg = p.delims[bin_base + first + (uint32_t)kl];
        c = p.delims[bin_base + first + (uint32_t)kh + 1] - beg;
    };
    // the first c points from s on, four at most: which are results.  (Reads all
    // four: the array has three entries more than points.)
    auto load = [&](uint32_t s, float4 (&h)[4]) {
#pragma unroll
        for (int k = 0; k < 4; ++k) h[k] = p.phi[s + k];
    };
    auto test = [&](uint32_t s, uint32_t c, const float4 (&h)[4]) {
        const unsigned all = c >= 4 ? 15u : (1u << c) - 1u;
        if (!REAL) return all;
        // t = d^2 - r^2; a result has t < 0, |t| within the band decides nothing
        unsigned in = 0;
        float t[4], least = filter ? INFINITY : 0.f;
#pragma unroll
        for (int k = 3; k >= 0; --k) {
            const float dx = __fsub_rn(qx, h[k].x), dy = __fsub_rn(qy, h[k].y), dz = __fsub_rn(qz, h[k].z);
            t[k] = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmaf_rn(dz, dz, -r2f)));
            in = __funnelshift_l(__float_as_uint(t[k]), in, 1);
            least = fminf(least, fabsf(t[k]));
        }
        in &= all;
        if (least <= band)
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (!(fabsf(t[k]) > band) && ((all >> k) & 1u))
                    in = (in & ~(1u << k)) | (exact_query(p, q, s + k) ? 1u << k : 0u);
        return in;
    };
    auto put = [&](unsigned ok, const float4 (&h)[4]) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (((ok >> u) & 1u) && (FILL || out < end)) {
                results[out] = __float_as_uint(h[u].w) - pt_base;
                out += kStep;
            }
        cnt += __popc(ok);
    };
    const int most = __reduce_max_sync(kFull, nrows);
#pragma unroll 1
    for (int t0 = 0; t0 < most; t0 += kLaneRows) {
        // ---- the next rows that hold points ----
        int n = 0;
        bool has_long = false;
#pragma unroll 1
        for (int t = t0; t < min(t0 + kLaneRows, nrows); ++t) {
            uint32_t beg = 0, c = 0;
            row(beg, c);
            if (!REAL && !FILL) {
                cnt += c;
            } else if (c) {
                rows[n++][threadIdx.x] = make_uint2(beg, c);
                has_long |= c >= kLongRun;
            }
        }
        if (!REAL && !FILL) continue;
        if (!__any_sync(kFull, has_long)) {
            // ---- each lane its own points, four at a time ----
            int k = 0;
            uint32_t s = 0, c = 0;
            uint2 e = k < n ? rows[k++][threadIdx.x] : make_uint2(0u, 0u);
            for (;;) {
                if (c == 0) {
                    s = e.x;
                    c = e.y;
                    if (c == 0) break;
                    e = k < n ? rows[k++][threadIdx.x] : make_uint2(0u, 0u);
                }
                float4 h[4];
                load(s, h);
                put(test(s, c, h), h);
                s += 4;
                c = c > 4 ? c - 4 : 0;
            }
            __syncwarp();
            continue;
        }
        // ---- row by row; a long row of a few lanes is taken by the warp ----
        const int rounds = __reduce_max_sync(kFull, n);
#pragma unroll 1
        for (int k = 0; k < rounds; ++k) {
            const uint2 e = k < n ? rows[k][threadIdx.x] : make_uint2(0, 0);
            uint32_t c = e.y;
            unsigned longs = __ballot_sync(kFull, c >= kLongRun);
            if (__popc(longs) <= 16) {
                if (c >= kLongRun) c = 0;
#pragma unroll 1
                for (; longs; longs &= longs - 1u) {
                    const int src = __ffs(longs) - 1;
                    const uint32_t sb = __shfl_sync(kFull, e.x, src), sc = __shfl_sync(kFull, e.y, src);
                    const uint32_t uq = __shfl_sync(kFull, q, src);
                    const float vx = __shfl_sync(kFull, qx, src), vy = __shfl_sync(kFull, qy, src), vz = __shfl_sync(kFull, qz, src);
                    const float vb = __shfl_sync(kFull, band, src);
                    const Place o = __shfl_sync(kFull, out, src), oe = __shfl_sync(kFull, end, src);
                    uint32_t found = 0;
#pragma unroll 1
                    for (uint32_t b = 0; b < sc; b += 32) {
                        const uint32_t s = sb + b + lane;
                        bool ok = b + lane < sc;
                        float4 h = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (ok) {
                            h = p.phi[s];
                            if (REAL) {
                                const float dx = __fsub_rn(vx, h.x), dy = __fsub_rn(vy, h.y), dz = __fsub_rn(vz, h.z);
                                const float t = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmaf_rn(dz, dz, -r2f)));
                                ok = fabsf(t) > vb ? t < 0.f : exact_query(p, uq, s);
                            }
                        }
                        const unsigned bal = __ballot_sync(kFull, ok);
                        const uint64_t to = o + (uint64_t)(found + __popc(bal & lt)) * kStep;
                        if (ok && (FILL || to < oe)) results[to] = __float_as_uint(h.w) - pt_base;
                        found += __popc(bal);
                    }
                    if (lane == src) {
                        out = FILL ? o + found : (Place)min((uint64_t)oe, o + (uint64_t)found * kStep);
                        cnt += found;
                    }
                }
            }
#pragma unroll 1
            for (uint32_t b = 0; b < c; b += 4) {
                float4 h[4];
                load(e.x + b, h);
                put(test(e.x + b, c - b, h), h);
            }
            __syncwarp();
        }
    }
    if (!FILL && have) {
        p.count[q] = cnt;
        if (p.stage_len && cnt > p.stage_len) p.err[1] = 1;     // left to a second pass
    }
}

// The listed results to their places: a warp takes the lists of a warp of
// k_radius_lane, 32 results of each at a time, through shared memory, so that
// both sides are read and written in runs.
__global__ void __launch_bounds__(kLaneThreads) k_radius_place(RadiusParams p) {
    __shared__ uint32_t tiles[kLaneThreads / 32][32][33];
    uint32_t(*tile)[33] = tiles[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const uint64_t at = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t c = 0;
    unsigned long long to = 0;
    if (at < p.nq) {
        const uint32_t q = p.qorder ? p.qorder[at] : (uint32_t)at;
        c = p.count[q];
        to = p.offs[q];
        if (c > p.stage_len) c = 0;
    }
    const uint32_t most = __reduce_max_sync(kFull, c);
    const uint32_t* from = p.stage + (at - lane) * p.stage_len + lane;
#pragma unroll 1
    for (uint32_t k0 = 0; k0 < most; k0 += 32) {
#pragma unroll 8
        for (uint32_t k = 0; k < 32; ++k)
            if (k0 + k < c) tile[k][lane] = from[(size_t)(k0 + k) * 32];
        __syncwarp();
        const uint32_t k = lane & 15;
#pragma unroll 4
        for (int j = 0; j < 32; j += 2) {
            const int src = j + (lane >> 4);
            const uint32_t n = __shfl_sync(kFull, c, src);
            uint32_t* const o = p.out + __shfl_sync(kFull, to, src) + k0;
            if (k0 + k < n) o[k] = tile[k][src];
            if (k0 + k + 16 < n) o[k + 16] = tile[k + 16][src];
        }
        __syncwarp();
    }
}

// Position of query wq (a given position, or the position of a given cell).
__device__ __forceinline__ bool query_position(const RadiusParams& p, uint32_t wq, double& x, double& y, double& z) {
    if (p.qxyz) {
        x = p.qxyz[3 * (size_t)wq];
        y = p.qxyz[3 * (size_t)wq + 1];
        z = p.qxyz[3 * (size_t)wq + 2];
        return true;
    }
    const uint32_t c = p.qcell[wq];
    if (c >= p.desc[0].n) return false;
    const size_t g = (size_t)p.desc[0].pt_base + c;
    x = p.xyz[3 * g];
    y = p.xyz[3 * g + 1];
    z = p.xyz[3 * g + 2];
    return true;
}

__global__ void __launch_bounds__(256) k_query_bin(RadiusParams p, QueryOrder o) {
    const DiagDesc& D = p.desc[0];
    const int shift = 1;
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < p.nq; q += gridDim.x * blockDim.x) {
        double x = 0.0, y = 0.0, z = 0.0;
        uint32_t c = 0;
        if (query_position(p, q, x, y, z)) {
            // (the order is for locality only: FP32 places)
            auto place = [&](double v, int a) {
                const float u = (f64_to_f32_rz(__dadd_rn(v, -D.ctr[a])) - D.glo_hi[a]) * D.inv_s[a];
                return (uint32_t)min(max((int)u, 0), D.cpd - 1) >> shift;
            };
            const uint32_t ix = place(x, 0), iy = place(y, 1), iz = place(z, 2);
            c = (ix * (uint32_t)o.cpdc + iy) * (uint32_t)o.cpdc + iz;
        }
        o.qbin[q] = c;
        o.qrank[q] = atomicAdd(&o.cnt[c], 1u);
    }
}

__global__ void __launch_bounds__(256) k_query_scatter(uint32_t nq, QueryOrder o) {
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += gridDim.x * blockDim.x)
        o.order[o.coff[o.qbin[q]] + o.qrank[q]] = q;
}

template <int MODE>
cudaError_t launch_mode(const RadiusParams& p, bool fill, int blocks, cudaStream_t s) {
    if constexpr (MODE == RQ_REAL_RADIUS || MODE == RQ_CELL_RADIUS) {
        if (p.lanes) {
            const unsigned nb = (unsigned)(((uint64_t)p.nq + kLaneThreads - 1) / kLaneThreads);
            if (fill && p.stage_len) {
                k_radius_place<<<nb, kLaneThreads, 0, s>>>(p);
                const cudaError_t e = cudaGetLastError();
                if (e != cudaSuccess || !p.unlisted) return e;
            }
            if (fill)
                k_radius_lane<MODE, true><<<nb, kLaneThreads, 0, s>>>(p);
            else
                k_radius_lane<MODE, false><<<nb, kLaneThreads, 0, s>>>(p);
            return cudaGetLastError();
        }
    }
    if (fill)
        k_radius<MODE, true><<<blocks, 256, 0, s>>>(p);
    else
        k_radius<MODE, false><<<blocks, 256, 0, s>>>(p);
    return cudaGetLastError();
}

// Host copy of the search-order key (celery.rs:423-427 on gap counts); the
// library's host code is compiled without FMA contraction, so this is the
// same correctly rounded FP64 arithmetic as the device's gap_key.
double host_gap_key(const double size[3], int i, int j, int k) {
    if (i == 0 && j == 0 && k == 0) return -1.0;
    const int gi = i < 0 ? -i - 1 : (i > 0 ? i - 1 : 0);
    const int gj = j < 0 ? -j - 1 : (j > 0 ? j - 1 : 0);
    const int gk = k < 0 ? -k - 1 : (k > 0 ? k - 1 : 0);
    const double a = (double)gi * size[0], b = (double)gj * size[1], c = (double)gk * size[2];
    return a * a + b * b + c * c;
}

// Largest offset along an axis that can still have key <= radius: offsets
// with gap g >= G satisfy (g * s)^2 > radius, so |offset| <= G suffices.
int axis_reach(double s, int cpd, double radius) {
    if (!(s > 0.0) || std::isnan(radius) || std::isinf(radius)) return cpd - 1;
    auto beyond = [&](long g) {
        const double a = (double)g * s;
        return a * a > radius;
    };
    long g = radius > 0.0 ? (long)std::min(std::floor(std::sqrt(radius) / s), (double)cpd) : 0;
    while (g > 0 && beyond(g - 1)) --g;
    while (g < cpd && !beyond(g)) ++g;
    return (int)std::min<long>(g, cpd - 1);
}

// check_cell_in_range's squared gap distance on the host (same operation
// order, no contraction).
double host_gap_ds(const double size[3], int gx, int gy, int gz) {
    const double a = (double)gx * size[0], b = (double)gy * size[1], c = (double)gz * size[2];
    return a * a + b * b + c * c;
}

struct RadiusEntry {
    double key;
    int i, j, k;
};

}  // namespace

// Queries from which a lane answers one.  Whole calls on an evenly filled grid, by
// warps and by lanes, 1,000,000 points and 16 results each: 4,000 queries 89 and 109
// us, 8,192 about 105 and 104, 16,384 137 and 120, 65,535 213 and 112; every point
// of the bins instead: 8,192 59 and 75, 16,384 74 and 78, 32,768 85 and 80.
// Where points crowd, a lane in the crowd keeps its warp waiting: 200,000 points, 90%
// of them in 64 clusters, 19 results each: 8,192 queries 153 and 468, 65,536 475 and
// 563, 131,072 805 and 923, 262,144 1,473 and 1,360, 600,000 3,146 and 1,925; 10%
// in the clusters 95 and 206, 223 and 222, 338 and 342, 565 and 478, 1,134 and 520;
// every point of the bins, 615 of them: 600,000 1,299 and 4,090.
constexpr uint32_t kLaneMin = 8192, kLaneMinCell = 16384, kLaneMinCrowded = 262144;
bool radius_lanes(int mode, uint32_t nq, uint32_t n, const DiagDesc& D) {
    const bool even = D.crowd <= n / 64;
    if (mode == RQ_REAL_RADIUS) return nq >= (even ? kLaneMin : kLaneMinCrowded);
    return mode == RQ_CELL_RADIUS && even && nq >= kLaneMinCell;
}

uint32_t radius_stage_len(int mode, uint32_t n, const DiagDesc& D, double radius) {
    if (mode != RQ_REAL_RADIUS) return 0;
    double mean = n * 4.1887902047863910 * radius * radius * radius;
    for (int a = 0; a < 3; ++a) mean /= D.size[a] * D.cpd;
    if (!(mean >= 0.0 && mean <= 200.0)) return 0;
    return ((uint32_t)std::ceil(mean + 6.0 * std::sqrt(mean)) + 7) / 8 * 8;
}

cudaError_t launch_radius(const RadiusParams& p, int mode, bool fill, int blocks, cudaStream_t s) {
    if (p.nq == 0) return cudaSuccess;
    switch (mode) {
        case RQ_CELLS: return launch_mode<RQ_CELLS>(p, fill, blocks, s);
        case RQ_CELL_RADIUS: return launch_mode<RQ_CELL_RADIUS>(p, fill, blocks, s);
        case RQ_REAL_RADIUS: return launch_mode<RQ_REAL_RADIUS>(p, fill, blocks, s);
        case RQ_CLOUD: return launch_mode<RQ_CLOUD>(p, fill, blocks, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_axis_bounds(const DiagDesc* desc, int cpd, unsigned long long* bnd, cudaStream_t s) {
    k_axis_bounds<<<(3 * cpd + 127) / 128, 128, 0, s>>>(desc, cpd, bnd);
    return cudaGetLastError();
}

cudaError_t launch_query_order(const RadiusParams& p, const QueryOrder& o, int blocks, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(o.cnt, 0, sizeof(uint32_t) * o.ncoarse, s);
    if (e != cudaSuccess) return e;
    k_query_bin<<<blocks, 256, 0, s>>>(p, o);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if ((e = launch_csr_offsets(o.cnt, o.ncoarse, o.coff, o.scan_tmp, s)) != cudaSuccess) return e;
    k_query_scatter<<<blocks, 256, 0, s>>>(p.nq, o);
    return cudaGetLastError();
}

// The prefix of the search order (celery.rs:418-679: every offset with
// |i|, |j|, |k| <= cpd - 1, sorted by key; ties broken by i, j, k) that
// expand_all_in_radius visits before its first key above the radius.
bool build_radius_table(const double size[3], int cpd, double radius, size_t max_entries,
                        std::vector<short4>& out) {
    out.clear();
    if (radius < -1.0) return true;                     // even the own bin (key -1) is beyond
    const int gx = axis_reach(size[0], cpd, radius);
    const int gy = axis_reach(size[1], cpd, radius);
    const int gz = axis_reach(size[2], cpd, radius);
    const double enumerate = (2.0 * gx + 1) * (2.0 * gy + 1) * (2.0 * gz + 1);
    if (enumerate > (double)max_entries) return false;
    std::vector<RadiusEntry> e;
    e.reserve((size_t)enumerate);
    for (int i = -gx; i <= gx; ++i)
        for (int j = -gy; j <= gy; ++j)
            for (int k = -gz; k <= gz; ++k) {
                const double key = host_gap_key(size, i, j, k);
                if (key > radius) continue;             // celery.rs:1037-1039
                e.push_back({key, i, j, k});
            }
    std::sort(e.begin(), e.end(), [](const RadiusEntry& a, const RadiusEntry& b) {
        if (a.key != b.key) return a.key < b.key;
        if (a.i != b.i) return a.i < b.i;
        if (a.j != b.j) return a.j < b.j;
        return a.k < b.k;
    });
    out.resize(e.size());
    for (size_t t = 0; t < e.size(); ++t)
        out[t] = make_short4((short)e[t].i, (short)e[t].j, (short)e[t].k, 0);
    return true;
}

bool build_gap_table(const double size[3], const double inv[3], int cpd, double radius, size_t max_entries,
                     std::vector<int16_t>& out, int* gx, int* gy, int* gz, bool* tie) {
    *tie = false;
    if (!(radius >= 0.0) || std::isinf(radius)) return false;
    // The box of find_cells_in_radius spans at most ceil(r * inv) + 1 bins on
    // either side of the query's bin, so gaps stay below ceil(r * inv) + 1.
    int g[3];
    for (int a = 0; a < 3; ++a) {
        const double reach = radius * inv[a];
        g[a] = (size[a] > 0.0 && reach < 1e6) ? std::min(cpd - 1, (int)std::ceil(reach) + 2) : cpd - 1;
        if (g[a] > 32767) return false;
    }
    if ((size_t)(g[0] + 1) * (size_t)(g[1] + 1) > max_entries) return false;
    const double r2 = radius * radius;
    out.assign((size_t)(g[0] + 1) * (size_t)(g[1] + 1), (int16_t)-1);
    for (int i = 0; i <= g[0]; ++i)
        for (int j = 0; j <= g[1]; ++j) {
            int best = -1;
            for (int k = 0; k <= g[2]; ++k) {           // the distance grows with k
                const double ds = host_gap_ds(size, i, j, k);
                if (!(ds <= r2)) {
                    *tie = *tie || !(ds > r2 * 1.01);
                    break;
                }
                best = k;
            }
            out[(size_t)i * (size_t)(g[1] + 1) + (size_t)j] = (int16_t)best;
        }
    *gx = g[0];
    *gy = g[1];
    *gz = g[2];
    return true;
}

}  // namespace tess

// tess_grid.cu -- the binning pass (the GPU form of Celery::reset,
// celery.rs:253-266): tight bounds, bin sizes, bin histogram, exclusive scan
// into delimiters, scatter into bin order, gather of sorted positions, and the
// per-diagram shell table.  All passes are HBM-bound streaming kernels; the
// integer outputs (bins, delimiters, sorted order) are bit-exact with the
// reference formulas.
#include <cfloat>
#include <cmath>

#include "tess_internal.cuh"

namespace tess {
namespace {

constexpr int kBoundsThreads = 256;

// The pass runs on the integer pipes: on this part an FP64 instruction costs
// dozens of issue slots' worth of pipe time, which made the FP64 forms of the
// bounds, the bin formula and the split bound the pass by the FP64 pipe.

__device__ __forceinline__ unsigned long long warp_min_u64(unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// CeleryCellInfo::new (celery.rs:153-181) from the bounds and the host's cpd.
// Four threads per diagram (t / 4), one per axis and one idle: the FP64
// divisions of the axes run side by side.  Whole warps.
__device__ __forceinline__ void grid_params(const GridBuffers& g, int t) {
    const int d = min(t >> 2, g.ndiag - 1), a = min(t & 3, 2);
    const bool mine = (t >> 2) < g.ndiag && (t & 3) < 3;
    DiagDesc& D = g.diags[d];
    const double c = (double)D.cpd;
    const double lo = ord_dec(__ldcg(&g.bounds[6 * d + a]));
    const double hi = ord_dec(__ldcg(&g.bounds[6 * d + 3 + a]));
    const double half = 0.5 * lo + 0.5 * hi;
    const double ctr = isfinite(half) ? half : 0.0;
    const double ext = __dsub_rn(hi, lo);
    const double size = __ddiv_rn(ext, c), inv = __ddiv_rn(c, ext);
    const float size_f = __double2float_rn(size), inv_f = __double2float_rn(inv);
    const bool ok_a = !(ext > 0.0) || (size_f >= FLT_MIN && size_f <= FLT_MAX && inv_f >= FLT_MIN && inv_f <= FLT_MAX);
    const unsigned quad = (__ballot_sync(0xffffffffu, ok_a) >> (threadIdx.x & 28)) & 7u;
    // the smallest nonzero bin side, through its order-preserving bits
    unsigned long long m = size > 0.0 ? (unsigned long long)__double_as_longlong(size) : ~0ull;
    m = min(m, __shfl_xor_sync(0xffffffffu, m, 1));
    m = min(m, __shfl_xor_sync(0xffffffffu, m, 2));
    if (t == 0 && g.host_flag) *g.host_flag = __ldcg(g.error_flag);
    if (!mine) return;
    D.glo[a] = lo;
    D.ghi[a] = hi;
    D.ctr[a] = ctr;
    D.size[a] = size;
    D.inv[a] = inv;
    // FP32 forms for the FP32 clipping pass: offsets from the centre as
    // FP32 pairs (48 bits), the bin sides and their inverses
    const double gl = lo - ctr, bl = D.blo[a] - ctr, bh = D.bhi[a] - ctr;
    const float glf = __double2float_rn(gl), blf = __double2float_rn(bl), bhf = __double2float_rn(bh);
    D.glo_hi[a] = glf;
    D.glo_lo[a] = __double2float_rn(gl - (double)glf);
    D.blo_hi[a] = blf;
    D.blo_lo[a] = __double2float_rn(bl - (double)blf);
    D.bhi_hi[a] = bhf;
    D.bhi_lo[a] = __double2float_rn(bh - (double)bhf);
    D.inv_f[a] = inv_f;
    D.glo_f[a] = __double2float_rn(lo);
    D.size_f[a] = size_f;
    D.inv_s[a] = ext > 0.0 ? inv_f : 0.f;
    if (a != 0) return;
    D.lean_ok = quad == 7u;
    D.crowd = 0;
    // (x - glo) * inv from the FP32 pairs: one rounding of the difference, one
    // of inv, one of the product (u = 2^-24 each, relative to the result, at
    // most cpd bins), with a factor 4 in hand
    D.frac_eps = 4.0f * 5.9604645e-8f * (float)D.cpd + 1e-6f;
    // Table extent: every offset whose key is <= (gaps * m)^2 has all gap
    // counts <= gaps, hence |offset| <= gaps + 1 on every axis.
    int cheb = g.table_gaps + 1;
    if (cheb > D.cpd - 1) cheb = D.cpd - 1;
    if (cheb < 0) cheb = 0;
    D.cheb = cheb;
    // The table holds every offset of the grid when that fits; otherwise the
    // offsets with key <= kmax, and the walk continues ring by ring.
    const bool complete = cheb == D.cpd - 1 && (2 * cheb + 1) * (2 * cheb + 1) * (2 * cheb + 1) <= kMaxTable;
    D.has_extent = m != ~0ull;
    if (m == ~0ull) {            // every point identical: only the own bin holds points
        D.min_size = 0.0;
        D.tab_kmax = INFINITY;
        D.cheb = 0;
    } else {
        const double ms = __longlong_as_double((long long)m);
        D.min_size = ms;
        const int gaps = cheb - 1;
        D.tab_kmax = complete ? (double)INFINITY
                              : __dmul_rn(__dmul_rn((double)gaps, ms), __dmul_rn((double)gaps, ms));
    }
}

__global__ void __launch_bounds__(128) k_grid_params(GridBuffers g) {
    grid_params(g, (int)(blockIdx.x * blockDim.x + threadIdx.x));
}

// True in every thread of the last block of a grid to get here: what the other
// blocks wrote before is visible (through L2).
__device__ bool last_block(unsigned* ticket) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    __threadfence();
    return last;
}

// CeleryBounds::new (celery.rs:81-125): per-chunk min/max of the coordinates'
// order-preserving integer codes (ord_enc: the same order as the doubles),
// merged with 64-bit atomics.  Non-finite inputs (exponent all ones) raise
// error_flag.  A single diagram's grid parameters are computed by the last
// block (a launch of their own takes 5 us, 2% of a 1,000-point pass).
__global__ void __launch_bounds__(kBoundsThreads) k_bounds(GridBuffers g) {
    after_previous();
    __shared__ unsigned long long red[6][kBoundsThreads / 32];
    for (uint32_t c = blockIdx.x; c < g.nchunks; c += gridDim.x) {
        const uint32_t d = g.chunk_diag[c];
        const uint32_t beg = g.chunk_start[c];
        const DiagDesc& D = g.diags[d];
        const uint32_t end = min(beg + g.chunk, D.pt_base + D.n);
        unsigned long long mn[3] = {~0ull, ~0ull, ~0ull};
        unsigned long long mx[3] = {0ull, 0ull, 0ull};
        bool bad = false;
        const double* const in = g.src ? g.src : g.xyz;
        for (uint32_t i = beg + threadIdx.x; i < end; i += blockDim.x) {
            for (int a = 0; a < 3; ++a) {
                const double v = in[3ull * i + a];
                if (g.src) g.xyz[3ull * i + a] = v;
                const unsigned long long b = (unsigned long long)__double_as_longlong(v);
                bad |= ((b >> 52) & 0x7FFull) == 0x7FFull;
                const unsigned long long e = (b >> 63) ? ~b : (b | 0x8000000000000000ull);
                mn[a] = min(mn[a], e);
                mx[a] = max(mx[a], e);
            }
        }
        if (__syncthreads_or(bad) && threadIdx.x == 0) atomicExch(g.error_flag, 1);
        const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
        for (int a = 0; a < 3; ++a) {
            const unsigned long long lo = warp_min_u64(mn[a]), hi = warp_max_u64(mx[a]);
            if (l == 0) { red[a][w] = lo; red[3 + a][w] = hi; }
        }
        __syncthreads();
        if (threadIdx.x < 6) {
            const int a = threadIdx.x;
            unsigned long long v = red[a][0];
            for (int k = 1; k < kBoundsThreads / 32; ++k) v = a < 3 ? min(v, red[a][k]) : max(v, red[a][k]);
            if (a < 3) atomicMin(&g.bounds[6 * d + a], v);
            else atomicMax(&g.bounds[6 * d + a], v);
        }
        __syncthreads();
    }
    if (g.ndiag == 1 && last_block(&g.tickets[0]) && threadIdx.x < 32) grid_params(g, threadIdx.x);
}

// x rounded toward zero to FP32 by integer operations (within 2^-23 |x|).
// False for zeros, subnormals, non-finite values and magnitudes outside
// FP32's normal range: those take the exact FP64 formula.
__device__ __forceinline__ bool f32_trunc(double x, float& f) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const uint32_t hi = (uint32_t)(b >> 32);
    const int e = (int)((hi >> 20) & 0x7FFu);
    const int fe = e - 1023 + 127;
    if (e == 0 || e == 0x7FF || fe < 1 || fe > 254) return false;
    f = __uint_as_float((hi & 0x80000000u) | ((uint32_t)fe << 23) | (uint32_t)((b >> 29) & 0x7FFFFFull));
    return true;
}

// axis_index (celery.rs:269-314) without the FP64 pipe for nearly every point:
// x >= max is decided on the order-preserving codes (exact), and
// v = (x - min) * inv by an FP32 estimate t with a bound E on |t - v|:
//   x to FP32 by truncation (2^-23 |x|), min and inv rounded (2^-24 each),
//   the difference and the product rounded (2^-24 each), and v's own two
//   FP64 roundings (2^-52 each), so
//   |t - v| <= inv (2^-23 |x| + 2^-24 |min|) + 3.1 * 2^-24 |t|,
// which E = inv (|x| + |min|) 2^-22 + |t| 2^-21 covers twice over.  When
// [t - E, t + E] holds no integer (nor 0, nor cpd - 1) the bin is the one
// the FP64 formula gives; otherwise (a point within E of a bin boundary,
// about 2 * 10^-4 of a bin for the unit cube at cpd = 238) ok is false and
// the caller uses the FP64 formula.
__device__ __forceinline__ int axis_index_fast(double x, const DiagDesc& D, int a, int cpd, bool& ok) {
    const unsigned long long xb = (unsigned long long)__double_as_longlong(x);
    float xf;
    if (!f32_trunc(x, xf)) {
        ok = false;
        return 0;
    }
    const unsigned long long hb = (unsigned long long)__double_as_longlong(D.ghi[a]);
    const unsigned long long xe = (xb >> 63) ? ~xb : (xb | 0x8000000000000000ull);
    const unsigned long long he = (hb >> 63) ? ~hb : (hb | 0x8000000000000000ull);
    if (xe >= he) return cpd - 1;
    const float lf = D.glo_f[a], inv = D.inv_f[a];
    const float t = (xf - lf) * inv;
    const float E = inv * (fabsf(xf) + fabsf(lf)) * 2.3841858e-7f + fabsf(t) * 4.7683716e-7f;
    const float up = t + E;
    if (up < 1.0f) return 0;                      // v < 1: 0 (v <= 0 gives 0 too)
    const float dn = t - E;
    if (dn >= (float)(cpd - 1)) return cpd - 1;   // v >= cpd - 1
    const float fl = floorf(dn);
    if (dn > 0.f && fl == floorf(up)) return (int)fl;
    ok = false;
    return 0;
}

// ---- exclusive scan of the bin counts -> delimiters (celery.rs:372-414) ----
__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
    const int l = threadIdx.x & 31;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (l >= o) v += t;
    }
    return v;
}

// Block-wide exclusive scan of kScanThreads values; returns the block total.
__device__ uint32_t block_excl_scan(uint32_t v, uint32_t* out, uint32_t* sh) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    uint32_t inc = warp_incl_scan(v);
    if (l == 31) sh[w] = inc;
    __syncthreads();
    if (w == 0) {
        uint32_t s = (l < (int)(blockDim.x >> 5)) ? sh[l] : 0;
        uint32_t si = warp_incl_scan(s);
        sh[l] = si - s;
        if (l == 31) sh[32] = si;
    }
    __syncthreads();
    *out = inc - v + sh[w];
    uint32_t total = sh[32];
    __syncthreads();
    return total;
}

// The whole scan by one block (of any size): carry by carry.
__device__ void scan_by_block(uint32_t* data, uint32_t n, uint32_t* sh) {
    uint32_t carry = 0;
    for (uint32_t base0 = 0; base0 < n; base0 += blockDim.x * kScanItems) {
        const uint32_t base = base0 + threadIdx.x * kScanItems;
        uint32_t v[kScanItems];
        uint32_t s = 0;
        for (int k = 0; k < kScanItems; ++k) {
            v[k] = base + k < n ? __ldcg(&data[base + k]) : 0u;
            s += v[k];
        }
        uint32_t ex;
        const uint32_t tot = block_excl_scan(s, &ex, sh);
        uint32_t run = carry + ex;
        for (int k = 0; k < kScanItems; ++k) {
            if (base + k < n) data[base + k] = run;
            run += v[k];
        }
        carry += tot;
    }
}
// Grids of few bins: up to kScanLastMax the last block of the histogram scans
// them, up to kScanOneMax one block in a launch of its own, three launches
// beyond.
constexpr uint64_t kScanLastMax = 4096, kScanOneMax = 16384;

// get_cells (celery.rs:342-354) + histogram.  rank = arrival order in the bin.
__global__ void __launch_bounds__(256) k_bin_count(GridBuffers g) {
    after_previous();
    for (uint32_t c = blockIdx.x; c < g.nchunks; c += gridDim.x) {
        const uint32_t d = g.chunk_diag[c];
        const uint32_t beg = g.chunk_start[c];
        const DiagDesc& D = g.diags[d];
        const uint32_t end = min(beg + g.chunk, D.pt_base + D.n);
        const int cpd = D.cpd;
        for (uint32_t i = beg + threadIdx.x; i < end; i += blockDim.x) {
            const double x = g.xyz[3ull * i], y = g.xyz[3ull * i + 1], z = g.xyz[3ull * i + 2];
            bool okx = true, oky = true, okz = true;
            int bx = axis_index_fast(x, D, 0, cpd, okx);
            int by = axis_index_fast(y, D, 1, cpd, oky);
            int bz = axis_index_fast(z, D, 2, cpd, okz);
            // the exact FP64 formula for the few coordinates near a boundary
            if (!okx) bx = axis_index(x, D.glo[0], D.ghi[0], D.inv[0], cpd);
            if (!oky) by = axis_index(y, D.glo[1], D.ghi[1], D.inv[1], cpd);
            if (!okz) bz = axis_index(z, D.glo[2], D.ghi[2], D.inv[2], cpd);
            // get_cell_from_indices, celery.rs:317-325
            const uint64_t b = tess_chk(D.bin_base + ((uint64_t)bx * cpd + by) * cpd + bz, g.total_bins, g.check, CK_GRID);
            g.bin[i] = (uint32_t)b;
            g.rank[i] = atomicAdd(&g.delims[b], 1u);
        }
    }
    if (g.total_bins + 1 <= kScanLastMax) {
        __shared__ uint32_t sh[33];
        if (last_block(&g.tickets[1])) scan_by_block(g.delims, (uint32_t)g.total_bins + 1, sh);
    }
}

__global__ void __launch_bounds__(kScanThreads) k_scan_partial(uint32_t* data, uint64_t n, uint32_t* sums) {
    after_previous();
    __shared__ uint32_t sh[33];
    const uint64_t base = (uint64_t)blockIdx.x * kScanThreads * kScanItems + (uint64_t)threadIdx.x * kScanItems;
    uint32_t s = 0;
    for (int k = 0; k < kScanItems; ++k) s += (base + k < n) ? data[base + k] : 0u;
    uint32_t ex;
    uint32_t tot = block_excl_scan(s, &ex, sh);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_sums(uint32_t* sums, uint32_t nblocks) {
    after_previous();
    __shared__ uint32_t sh[33];
    uint32_t carry = 0;
    for (uint32_t b0 = 0; b0 < nblocks; b0 += kScanThreads) {
        const uint32_t b = b0 + threadIdx.x;
        uint32_t v = b < nblocks ? sums[b] : 0u;
        uint32_t ex;
        uint32_t tot = block_excl_scan(v, &ex, sh);
        if (b < nblocks) sums[b] = carry + ex;
        carry += tot;
    }
}

__global__ void __launch_bounds__(kScanThreads) k_scan_final(uint32_t* data, uint64_t n, const uint32_t* sums) {
    after_previous();
    __shared__ uint32_t sh[33];
    const uint64_t base = (uint64_t)blockIdx.x * kScanThreads * kScanItems + (uint64_t)threadIdx.x * kScanItems;
    uint32_t v[kScanItems];
    uint32_t s = 0;
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = (base + k < n) ? data[base + k] : 0u;
        s += v[k];
    }
    uint32_t ex;
    block_excl_scan(s, &ex, sh);
    uint32_t run = sums[blockIdx.x] + ex;
    for (int k = 0; k < kScanItems; ++k) {
        if (base + k < n) data[base + k] = run;
        run += v[k];
    }
}

__global__ void __launch_bounds__(kScanThreads) k_scan_one(uint32_t* data, uint32_t n) {
    after_previous();
    __shared__ uint32_t sh[33];
    scan_by_block(data, n, sh);
}

// get_sorted_indices (celery.rs:357-369): counting-sort scatter.
__global__ void k_scatter(GridBuffers g) {
    after_previous();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.total) return;
    const uint32_t b = tess_chk(g.bin[i], g.total_bins, g.check, CK_GRID);
    g.sorted[tess_chk(g.delims[b] + g.rank[i], g.total, g.check, CK_GRID)] = i;
}

// Ascending sort of a[0, n) by one block: a bitonic network in the form whose
// comparators all point the same way (the first step of each merge compares
// mirrored positions), over n rounded up to a power of two.  Positions >= n
// stand for +inf: a comparator with one of them never swaps, so they are
// simply skipped and never stored.  a is shared or global memory; the block's
// barriers order the steps either way.
// I is the index type: 32-bit in shared memory, 64-bit for a bin that may
// approach 2^32 points.
template <typename I>
__device__ void block_bitonic_sort(uint32_t* a, I n) {
    I np = 1;
    while (np < n) np <<= 1;
    const I half = np >> 1;
    auto cmpswap = [&](I lo, I hi) {
        if (hi < n) {
            const uint32_t x = a[lo], y = a[hi];
            if (x > y) {
                a[lo] = y;
                a[hi] = x;
            }
        }
    };
    for (I k = 2; k <= np; k <<= 1) {
        const I hk = k >> 1;
        for (I i = threadIdx.x; i < half; i += blockDim.x) {
            const I base = (i / hk) * k, off = i % hk;
            cmpswap(base + off, base + k - 1 - off);
        }
        __syncthreads();
        for (I j = hk >> 1; j > 0; j >>= 1) {
            for (I i = threadIdx.x; i < half; i += blockDim.x) {
                const I lo = (i / j) * 2 * j + i % j;
                cmpswap(lo, lo + j);
            }
            __syncthreads();
        }
    }
}

// Within-bin order ascending by input index (deterministic; the reference's
// sort_unstable_by leaves it unspecified).  Bins hold ~1.25 points on
// average: a thread per bin sorts the small ones by insertion; bins of more
// than 32 points (crowded regions) are sorted afterwards by the whole block,
// in shared memory up to kSortSmem points, in place beyond.
constexpr uint32_t kSortSmem = 4096;
__global__ void __launch_bounds__(256) k_bin_order(GridBuffers g) {
    after_previous();
    __shared__ uint32_t big[256];
    __shared__ uint32_t nbig;
    __shared__ uint32_t buf[kSortSmem];
    if (threadIdx.x == 0) nbig = 0;
    __syncthreads();
    const uint64_t b0 = (uint64_t)blockIdx.x * blockDim.x;
    const uint64_t b = b0 + threadIdx.x;
    uint32_t crowd = 0;
    if (b < g.total_bins) {
        const uint32_t beg = g.delims[b], end = g.delims[b + 1];
        if (end - beg > g.crowded) crowd = end - beg;
        if (end - beg > 32) {
            big[atomicAdd(&nbig, 1u)] = threadIdx.x;
        } else if (end - beg >= 2) {
            for (uint32_t s = beg + 1; s < end; ++s) {
                uint32_t v = g.sorted[s];
                uint32_t t = s;
                while (t > beg && g.sorted[t - 1] > v) {
                    g.sorted[t] = g.sorted[t - 1];
                    --t;
                }
                g.sorted[t] = v;
            }
        }
    }
    // how evenly the points fill the grid (radius queries, of one diagram)
    crowd = __reduce_add_sync(0xffffffffu, crowd);
    if (crowd && g.ndiag == 1 && (threadIdx.x & 31) == 0) atomicAdd(&g.diags[0].crowd, crowd);
    __syncthreads();
    const uint32_t nb = nbig;
    for (uint32_t q = 0; q < nb; ++q) {
        const uint64_t bb = b0 + big[q];
        const uint32_t beg = g.delims[bb], n = g.delims[bb + 1] - beg;
        if (n <= kSortSmem) {
            for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) buf[i] = g.sorted[beg + i];
            __syncthreads();
            block_bitonic_sort<uint32_t>(buf, n);
            for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) g.sorted[beg + i] = buf[i];
        } else {
            block_bitonic_sort<uint64_t>(g.sorted + beg, (uint64_t)n);
        }
        __syncthreads();
    }
}

// hi = u rounded to FP32 (to nearest, ties to even) and lo = u - hi rounded to
// FP32, by integer operations on u's bits: the same values as
// __double2float_rn(u) and __double2float_rn(u - (double)hi).  u - hi is
// exact in units of 2^(E - 52) (at most 29 bits), so one integer-to-FP32
// rounding and an exact power-of-two scale give lo.  False (the FP64 form
// then runs) when lo would be subnormal or hi leaves FP32's normal range.
__device__ __forceinline__ bool split_rn_int(double u, float& hi, float& lo) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(u);
    const uint32_t sign = (uint32_t)(b >> 32) & 0x80000000u;
    const int e = (int)((b >> 52) & 0x7FFull);
    if (e == 0) {
        if ((b << 1) != 0) return false;          // subnormal
        hi = __uint_as_float(sign);               // +-0: lo = +0 as u - hi is +0
        lo = 0.f;
        return true;
    }
    if (e == 0x7FF) return false;
    const unsigned long long m = (b & 0xFFFFFFFFFFFFFull) | (1ull << 52);
    unsigned long long q = m >> 29;
    const unsigned long long rem = m & ((1ull << 29) - 1);
    if (rem > (1ull << 28) || (rem == (1ull << 28) && (q & 1ull))) q += 1;
    const long long diff = (long long)m - (long long)(q << 29);
    int ehi = e;
    if (q == (1ull << 24)) {
        q >>= 1;
        ehi += 1;
    }
    const int fe = ehi - 1023 + 127;
    const int pe = e - 1023 - 52 + 127;
    if (fe < 1 || fe > 254 || (diff != 0 && pe < 1)) return false;
    hi = __uint_as_float(sign | ((uint32_t)fe << 23) | ((uint32_t)q & 0x7FFFFFu));
    lo = diff == 0 ? 0.f : __ll2float_rn(sign ? -diff : diff) * __uint_as_float((uint32_t)pe << 23);
    return true;
}

// Positions (and groups) in sorted order, SoA for coalesced candidate loads.
// The FP32 pair (hi, lo) splits the position relative to its diagram's
// centre: the split keeps 48 bits of that offset, so its error scales with
// the diagram's extent rather than with the coordinates' distance from 0.
__global__ void k_gather(GridBuffers g) {
    after_previous();
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= g.total) return;
    const uint32_t i = tess_chk(g.sorted[s], g.total, g.check, CK_GRID);
    if (g.inv) g.inv[i] = s;
    const double x = g.xyz[3ull * i], y = g.xyz[3ull * i + 1], z = g.xyz[3ull * i + 2];
    g.spx[s] = x;
    g.spy[s] = y;
    g.spz[s] = z;
    int lo = 0, hi = g.ndiag - 1;     // the diagram holding sorted position s
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (g.diags[mid].pt_base <= s) lo = mid;
        else hi = mid - 1;
    }
    const DiagDesc& D = g.diags[lo];
    const double u[3] = {x - D.ctr[0], y - D.ctr[1], z - D.ctr[2]};
    float hi4[3], lo4[3];
    for (int a = 0; a < 3; ++a) {
        float h, l;
        if (!split_rn_int(u[a], h, l)) {
            h = __double2float_rn(u[a]);
            l = __double2float_rn(u[a] - (double)h);
        }
        hi4[a] = h;
        lo4[a] = l;
    }
    g.phi[s] = make_float4(hi4[0], hi4[1], hi4[2], __uint_as_float(i));
    g.plo[s] = make_float4(lo4[0], lo4[1], lo4[2], 0.f);
    if (g.sgroup) g.sgroup[s] = g.groups[i];
}

// The inverse permutation, point -> sorted position, for the queries that
// start from a point's original index (radius queries by cell, single-cell
// computes).  Built on first use after a binning pass rather than in it: its
// 4-byte scatter writes cost a partial DRAM sector per point.
__global__ void k_inverse(const uint32_t* sorted, uint32_t* inv, uint32_t n, int* check) {
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x)
        inv[tess_chk(sorted[s], n, check, CK_GRID)] = s;
}

// ---- shell table (get_search_order, celery.rs:418-679) ----
// One block per diagram: every offset within Chebyshev radius `cheb` whose key
// is <= tab_kmax, sorted by (key, i, j, k).  An offset's key depends on its gap
// counts alone (0 for -1, 0 and 1, else |o| - 1), so only the at most 9^3 gap
// triples are sorted, one per thread (the short steps of the network by
// shuffles).  Each triple's offsets then take their place by the prefix sum of
// the triples' sizes, and the offsets of equal keys order themselves by
// counting.  Sorting all offsets in shared memory, with an FP64 key each, took
// 97 us a block; this takes 13.
//
// On an axis without extent every offset has the key of its other two, so a
// plane of points (5,000 offsets) or a line (6,900) has more than kMaxTable
// entries.  The table then ends with the last key whose offsets all fit, and
// tab_kmax says so: the walk goes on ring by ring beyond it.
constexpr int kTabThreads = 1024;
constexpr int kTabGaps = 9;          // gap counts per axis: 0 .. table_gaps (at most 8)
__global__ void __launch_bounds__(kTabThreads) k_table(GridBuffers g) {
    __shared__ double sq[3][kTabGaps];
    __shared__ unsigned long long skey[kTabThreads];
    __shared__ uint16_t sid[kTabThreads];
    __shared__ uint32_t wsum[kTabThreads / 32 + 1];
    __shared__ uint32_t start[kTabThreads];      // first entry of the r-th triple
    __shared__ uint16_t code[kMaxTable];         // an entry's offset, lexicographic
    __shared__ uint16_t rank[kMaxTable];         // ... and the place of its triple
    __shared__ int ends;                         // more than fit: the triple where the table ends
    const int d = blockIdx.x, t = threadIdx.x, lane = t & 31;
    DiagDesc& D = g.diags[d];
    const int c = D.cheb, side = 2 * c + 1;
    const int ng = c > 0 ? c : 1;                // gap counts 0 .. ng - 1
    if (t < 3 * ng) {
        const double v = __dmul_rn((double)(t % ng), D.size[t / ng]);
        sq[t / ng][t % ng] = __dmul_rn(v, v);
    }
    __syncthreads();
    // the triple's key as ordered bits (gap_key's operations); ~0: not kept
    unsigned long long key = ~0ull;
    int id = t;
    if (t < ng * ng * ng) {
        const double k = __dadd_rn(__dadd_rn(sq[0][t / (ng * ng)], sq[1][(t / ng) % ng]), sq[2][t % ng]);
        if (k <= D.tab_kmax) key = (unsigned long long)__double_as_longlong(k);
    }
    // bitonic sort of (key, id), ascending, one pair per thread
    for (int k2 = 2; k2 <= kTabThreads; k2 <<= 1) {
        for (int j2 = k2 >> 1; j2 > 0; j2 >>= 1) {
            unsigned long long ok;
            int oi;
            if (j2 >= 32) {
                skey[t] = key;
                sid[t] = (uint16_t)id;
                __syncthreads();
                ok = skey[t ^ j2];
                oi = sid[t ^ j2];
                __syncthreads();
            } else {
                ok = __shfl_xor_sync(0xffffffffu, key, j2);
                oi = __shfl_xor_sync(0xffffffffu, id, j2);
            }
            const bool less = ok < key || (ok == key && oi < id);      // the partner's pair is smaller
            const bool low = (t & j2) == 0, up = (t & k2) == 0;
            if (less == (low == up)) {
                key = ok;
                id = oi;
            }
        }
    }
    // the triple's offsets: {-1, 0, 1} for a gap of 0 (0 alone when the grid has
    // one bin), {-g - 1, g + 1} otherwise
    auto width = [&](int gap) { return gap ? 2u : (c > 0 ? 3u : 1u); };
    auto pick = [&](int gap, uint32_t q) { return gap ? (q ? gap + 1 : -gap - 1) : (c > 0 ? (int)q - 1 : 0); };
    const bool kept = key != ~0ull;
    const int gi = id / (ng * ng), gj = (id / ng) % ng, gk = id % ng;
    const uint32_t w0 = width(gi), w1 = width(gj), w2 = width(gk);
    const uint32_t cnt = kept ? w0 * w1 * w2 : 0u;
    uint32_t inc = cnt;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
    }
    if (lane == 31) wsum[t >> 5] = inc;
    skey[t] = key;
    __syncthreads();
    if (t < 32) {
        const uint32_t v = wsum[t];
        uint32_t i2 = v;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, i2, o);
            if (lane >= o) i2 += u;
        }
        wsum[t] = i2 - v;
        if (t == 31) wsum[32] = i2;
    }
    __syncthreads();
    const uint32_t beg = wsum[t >> 5] + inc - cnt;
    start[t] = beg;
    const uint32_t total = wsum[32], cap = min((uint32_t)kMaxTable, D.tab_cap);
    uint32_t m = total;
    if (total > cap) {
        if (t == 0) ends = 0;
        __syncthreads();
        if (kept && beg <= cap && t > 0 && skey[t - 1] != key) atomicMax(&ends, t);
        __syncthreads();
        m = start[ends];
        if (t == 0) D.tab_kmax = ends ? __longlong_as_double((long long)skey[ends - 1]) : -1.0;
    }
    // (not even the first key's, sides below 1e-162, or no key is a number, sides
    // beyond FP64's range: the own bin alone)
    if (t == 0 && m == 0) g.table[D.tab_base] = TabEntry{-1.0f, 0, 0, 0, 0};
    for (uint32_t q = 0; q < cnt; ++q) {
        if (beg + q >= m) break;
        const int i = pick(gi, q / (w1 * w2)), j = pick(gj, (q / w2) % w1), k = pick(gk, q % w2);
        code[beg + q] = (uint16_t)(((i + c) * side + (j + c)) * side + (k + c));
        rank[beg + q] = (uint16_t)t;
    }
    __syncthreads();
    const uint32_t self = (uint32_t)((c * side + c) * side + c);
    for (uint32_t e = t; e < m; e += blockDim.x) {
        // the entries of the same key: those of the triples around this one
        int r0 = rank[e], r1 = r0;
        const unsigned long long mine = skey[r0];
        while (r0 > 0 && skey[r0 - 1] == mine) --r0;
        while (r1 + 1 < kTabThreads && skey[r1 + 1] == mine) ++r1;
        const uint32_t b = start[r0], n = r1 + 1 < kTabThreads ? min(start[r1 + 1], m) : m;
        const uint32_t cd = code[e];
        // (the own bin comes first: its key is -1)
        uint32_t at = b;
        if (cd != self)
            for (uint32_t o = b; o < n; ++o) at += (code[o] < cd || code[o] == self) ? 1u : 0u;
        TabEntry te;
        te.key = cd == self ? -1.0f : __double2float_rz(__longlong_as_double((long long)mine));
        te.i = (int8_t)((int)(cd / (side * side)) - c);
        te.j = (int8_t)((int)((cd / side) % side) - c);
        te.k = (int8_t)((int)(cd % side) - c);
        te.pad = 0;
        g.table[D.tab_base + at] = te;
    }
    if (t == 0) D.tab_len = max(m, 1u);
    if (t == 0 && d == 0) *g.table_len = max(m, 1u);
}

}  // namespace

size_t scan_tmp_words(uint64_t nitems) {
    const uint64_t per = (uint64_t)kScanThreads * kScanItems;
    return (size_t)((nitems + per - 1) / per) + 1;
}

namespace {
// Bin occupancy for the autotuner: out[0] = most points in one bin, out[1] =
// points in bins of at least `crowd` points.  One atomic per warp.
__global__ void k_occupancy(const uint32_t* delims, uint64_t nbins, uint32_t crowd, unsigned long long* out) {
    unsigned long long mx = 0, crowded = 0;
    for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; b < nbins; b += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t c = delims[b + 1] - delims[b];
        mx = c > mx ? c : mx;
        if (c >= crowd) crowded += c;
    }
    for (int o = 16; o > 0; o >>= 1) {
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        crowded += __shfl_xor_sync(0xffffffffu, crowded, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&out[0], mx);
        atomicAdd(&out[1], crowded);
    }
}

// Start values of a binning pass: bounds, histogram, error flag.
__global__ void __launch_bounds__(256) k_grid_clear(GridBuffers g) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
    if (t == 0) *g.error_flag = 0;
    if (t < 2) g.tickets[t] = 0u;
    for (uint64_t i = t; i < 6ull * g.ndiag; i += stride) g.bounds[i] = (i % 6) < 3 ? ~0ull : 0ull;
    for (uint64_t i = t; i <= g.total_bins; i += stride) g.delims[i] = 0u;
}
}  // namespace

cudaError_t launch_inverse(const uint32_t* sorted, uint32_t* inv, uint32_t n, int* check, cudaStream_t s) {
    const uint32_t blocks = std::min<uint32_t>((n + 255) / 256, 152u * 16u);
    if (blocks) k_inverse<<<blocks, 256, 0, s>>>(sorted, inv, n, check);
    return cudaGetLastError();
}

// Bulk copy by the SMs: 16-byte loads and stores, grid-stride, then the tail
// byte by byte.  Either side may be pinned host memory (its device address):
// the SMs then move the bytes over the host link themselves.
__global__ void k_copy_bytes(const uint8_t* src, uint8_t* dst, size_t n) {
    after_previous();
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const size_t i0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    const size_t n16 = n / 16;
    const uint4* s16 = reinterpret_cast<const uint4*>(src);
    uint4* d16 = reinterpret_cast<uint4*>(dst);
    for (size_t i = i0; i < n16; i += stride) d16[i] = s16[i];
    for (size_t i = 16 * n16 + i0; i < n; i += stride) dst[i] = src[i];
}

cudaError_t launch_copy_bytes(void* dst, const void* src, size_t n, int sms, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    // 4 blocks of 256 threads per SM keep enough 16-byte requests in flight
    // to fill the host link (≈ 192 GB/s measured either way)
    const size_t want = (n / 16 + 255) / 256;
    const int blocks = (int)std::max<size_t>(1, std::min<size_t>(want, (size_t)4 * (sms > 0 ? sms : 152)));
    return launch_after(k_copy_bytes, blocks, 256, 0, s, static_cast<const uint8_t*>(src), static_cast<uint8_t*>(dst), n);
}

cudaError_t launch_occupancy(const uint32_t* delims, uint64_t nbins, uint32_t crowd, unsigned long long* out,
                             int blocks, cudaStream_t s) {
    cudaMemsetAsync(out, 0, 2 * sizeof(unsigned long long), s);
    k_occupancy<<<blocks, 256, 0, s>>>(delims, nbins, crowd, out);
    return cudaGetLastError();
}

uint64_t grid_launches(uint64_t total_bins, size_t ndiag) {
    return 7 + (ndiag > 1 ? 1 : 0) + (total_bins + 1 <= kScanLastMax ? 0 : (total_bins + 1 <= kScanOneMax ? 1 : 3));
}

// Binning pass: bounds -> grid parameters -> shell tables -> histogram ->
// scan -> scatter -> within-bin order -> gather.  A fixed launch sequence
// (no host synchronisation), so it can be captured in a CUDA graph.
cudaError_t launch_grid_build(const GridBuffers& g, cudaStream_t s, cudaStream_t side, cudaEvent_t fork,
                              cudaEvent_t join, cudaEvent_t bounds_done) {
    const int ndiag = g.ndiag;
    const uint64_t nclear = std::max<uint64_t>(6ull * ndiag, g.total_bins + 1);
    k_grid_clear<<<(unsigned)std::min<uint64_t>((nclear + 1023) / 1024, 152u * 8u), 256, 0, s>>>(g);
    const int cblocks = (int)(g.nchunks < 4096u ? g.nchunks : 4096u);
    launch_after(k_bounds, cblocks, kBoundsThreads, 0, s, g);
    if (ndiag > 1) k_grid_params<<<(4 * ndiag + 127) / 128, 128, 0, s>>>(g);   // else by k_bounds
    if (bounds_done) cudaEventRecord(bounds_done, s);
    // the shell tables need only the grid parameters: build them beside the
    // histogram, scan and scatter when a side stream is given
    const bool forked = side && fork && join;
    if (forked) {
        cudaEventRecord(fork, s);
        cudaStreamWaitEvent(side, fork, 0);
        k_table<<<ndiag, kTabThreads, 0, side>>>(g);
        cudaEventRecord(join, side);
    } else {
        k_table<<<ndiag, kTabThreads, 0, s>>>(g);
    }
    launch_after(k_bin_count, cblocks, 256, 0, s, g);
    const uint64_t nscan = g.total_bins + 1;
    const uint64_t per = (uint64_t)kScanThreads * kScanItems;
    const uint32_t nblk = (uint32_t)((nscan + per - 1) / per);
    if (nscan <= kScanLastMax) {
        // by k_bin_count
    } else if (nscan <= kScanOneMax) {
        launch_after(k_scan_one, 1, kScanThreads, 0, s, g.delims, (uint32_t)nscan);
    } else {
        launch_after(k_scan_partial, nblk, kScanThreads, 0, s, g.delims, nscan, g.scan_tmp);
        launch_after(k_scan_sums, 1, kScanThreads, 0, s, g.scan_tmp, nblk);
        launch_after(k_scan_final, nblk, kScanThreads, 0, s, g.delims, nscan, g.scan_tmp);
    }
    launch_after(k_scatter, (g.total + 255) / 256, 256, 0, s, g);
    launch_after(k_bin_order, (unsigned)((g.total_bins + 255) / 256), 256, 0, s, g);
    launch_after(k_gather, (g.total + 255) / 256, 256, 0, s, g);
    if (forked) cudaStreamWaitEvent(s, join, 0);
    return cudaGetLastError();
}

}  // namespace tess

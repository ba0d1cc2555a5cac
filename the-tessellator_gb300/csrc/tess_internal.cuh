// tess_internal.cuh -- device data layout shared by the binning pass, the
// clipping kernels and the host driver of libtessgpu.so (sm_103a).
//
// HBM layout of one set of diagrams (a single Diagram is a set of one):
//   points   xyz[3 * total]            FP64 AoS, concatenated diagram by diagram
//   bins     bin[total], rank[total]    global bin id and arrival rank per point
//   grid     delims[total_bins + 1]     CSR offsets of the bin-sorted order
//   sorted   sorted[total]              sorted position -> point (concatenated index)
//            spx/spy/spz[total]         FP64 positions in sorted order (SoA)
//            phi/plo[total]             FP32 pair of the sorted positions, 16 bytes each, the
//                                       point's index in the high part's fourth word
//            sgroup[total]              group ids in sorted order (optional)
//   table    tab[...]                   per-diagram shell table (sorted offsets)
//   results  vol[total], nface[total], fstart[total], status[total]  (point order)
//            face_nbr[cap], face_area[cap]   face pool, filled by atomic allocation
#pragma once

#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

namespace tess {

constexpr double kTolerance = 1e-12;        // polyhedron.rs:221-223
constexpr double kStopMargin = 1.0 + 1e-5;  // slack on the security-radius test
constexpr int kMaxTable = 4096;             // shell-table entries per diagram (sort capacity)

// Per-cell status codes written by the clipping kernels.
enum CellStatus : uint8_t {
    ST_OK = 0,
    ST_GUARD = 1,       // plane-side test inside the guard band (plain, dense) -> careful
                        // pass; not to be settled there -> FP64 clipping
    ST_VCAP = 2,        // vertex capacity exceeded -> FP64 clipping, larger
    ST_PCAP = 3,        // face (plane) capacity exceeded -> FP64 clipping, larger
    ST_DEGEN = 4,       // inconsistent topology -> as ST_GUARD; FP64 clipping: error
    ST_POOL = 5,        // face pool full -> host grows the pool
    ST_VERIFY = 6,      // FP32 vertex failed the FP64 check -> as ST_GUARD
    ST_DENSE = 7,       // crowded own bin or long batch (plain pass) -> seeded pass
    ST_NEAR = 8,        // a (near-)coincident point (FP32 passes) -> FP64 clipping
    ST_PENDING = 255    // not computed yet
};

// The checked build (compiled with TESS_CHECKED=1, libtessgpu_checked.so): the
// binning and clipping kernels test every data-dependent index into a device
// array before use.  An index outside [0, n) sets bit `site` of the handle's
// check word and is replaced by 0, so the access stays in bounds; the host
// then fails the call with TESS_E_CHECK.  The regular build compiles no test.
#ifndef TESS_CHECKED
#define TESS_CHECKED 0
#endif
enum CheckSite : int {
    CK_POINT = 0,   // a point (sorted or original index)
    CK_BIN = 1,     // a bin of the grid
    CK_SLOT = 2,    // a vertex slot or free-slot stack entry of a cell
    CK_PLANE = 3,   // a plane of a cell
    CK_LIST = 4,    // an entry of a work list
    CK_FACE = 5,    // a face of the face pool
    CK_GRID = 6     // a position of the binning pass's sort
};
template <typename I, typename N>
__device__ __forceinline__ I tess_chk(I i, N n, int* check, int site) {
#if TESS_CHECKED
    if (!((unsigned long long)(long long)i < (unsigned long long)n)) {
        if (check) atomicOr(check, 1 << site);
        return (I)0;
    }
#else
    (void)n;
    (void)check;
    (void)site;
#endif
    return i;
}

// One diagram as the kernels see it.  Filled partly by the host (counts,
// bases, box) and partly on the device (bounds, bin sizes, table length).
struct DiagDesc {
    double glo[3], ghi[3];   // CeleryBounds (celery.rs:81-125), tight point bounds
    double ctr[3];           // centre of those bounds: the FP32 hi/lo positions are split relative to it
    double size[3];          // x/y/z_cell_size (celery.rs:165-167)
    double inv[3];           // x/y/z_inverse_cell_size (celery.rs:169-171)
    double blo[3], bhi[3];   // container box (walls)
    double tab_kmax;         // every offset with key <= tab_kmax is in the table
    double min_size;         // smallest nonzero bin side
    uint64_t bin_base;       // first global bin of this diagram
    uint64_t tab_base;       // first table entry of this diagram
    uint32_t pt_base;        // first point (concatenated order == sorted order base)
    uint32_t n;              // points
    uint32_t tab_len;        // table entries (device-written)
    uint32_t tab_cap;        // table capacity reserved by the host
    int32_t cpd;             // cells_per_dimension (host, glibc cbrt)
    int32_t cheb;            // Chebyshev radius enumerated into the table
    // FP32 forms of the grid and the box for the FP32 clipping pass (device-
    // written with the grid): offsets from ctr as FP32 pairs (hi + lo), so the
    // site's place in its bin and the box corners come out of FP32 arithmetic
    float glo_hi[3], glo_lo[3];          // point bounds' low corner - ctr
    float blo_hi[3], blo_lo[3];          // container box low corner - ctr
    float bhi_hi[3], bhi_lo[3];          // container box high corner - ctr
    float inv_f[3];                      // inverse bin sides
    float glo_f[3];                      // point bounds' low corner, rounded to FP32
    float size_f[3];                     // bin sides
    float inv_s[3];                      // inverse bin sides, 0 on an axis without extent
    float frac_eps;                      // bound on the FP32 in-bin position's error, in bins
    int32_t has_extent;                  // some bin side is nonzero (min_size > 0)
    uint32_t crowd;                      // points in bins of more than GridBuffers::crowded (a single diagram's)
    int32_t lean_ok;                     // inv_s and size_f are in FP32's normal range (or 0)
};

// Shell-table entry: a bin offset and its search-order key (celery.rs:423-427)
// rounded toward zero to FP32 so the stop test stays conservative.
struct TabEntry {
    float key;
    int8_t i, j, k, pad;
};

// Output of one cell's full geometry (single-cell queries); the leading
// fields mirror tess_cell_geometry of the C ABI.
struct GeoOut {
    double volume;
    int32_t nv, nf;
    double verts[3 * 256];          // site-relative vertex positions
    int32_t face_nbr[256];
    double face_area[256];
    int32_t face_off[257];          // offsets into face_vtx
    int32_t face_vtx[3 * 256];      // vertex indices, CCW seen from outside
    int32_t status;
};

// Programmatic dependent launch: a kernel launched with launch_after() may be
// brought onto the SMs while the kernel before it in the stream runs out.  Such
// a kernel begins with after_previous(), in every thread and before any access
// to memory: it lets its own successor in, then waits until the kernel before
// it is complete and its writes are visible (so none of its pointers may be
// __restrict__, whose loads could be moved before the wait).  Launched the
// ordinary way, it does not wait.  A pass over 1,000 points in FP32, 8 such
// launches: 224 -> 218 us; 10,000 in FP64, 11: 419 -> 395.
__device__ __forceinline__ void after_previous() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <typename... Params, typename... Args>
cudaError_t launch_after(void (*kernel)(Params...), unsigned blocks, unsigned threads, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

// Order-preserving map of doubles onto uint64 (for atomicMin/atomicMax).
__device__ __forceinline__ unsigned long long ord_enc(double v) {
    unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double ord_dec(unsigned long long e) {
    unsigned long long b = (e >> 63) ? (e & 0x7FFFFFFFFFFFFFFFull) : ~e;
    return __longlong_as_double((long long)b);
}

// get_{x,y,z}_cell_index (celery.rs:269-314): x >= max -> cpd-1, else
// min(trunc((x - min) * inv), cpd-1), with `as usize` saturating at 0 for
// negative and NaN values.  Exact FP64 multiply, no FMA.
__device__ __forceinline__ int axis_index(double x, double lo, double hi, double inv, int cpd) {
    if (x >= hi) return cpd - 1;
    double v = __dmul_rn(__dsub_rn(x, lo), inv);
    if (!(v > 0.0)) return 0;
    if (v >= (double)(cpd - 1)) return cpd - 1;
    return (int)v;
}

// Search-order key of a bin offset (celery.rs:423-427 on the gap counts,
// celery.rs:447-639), self = -1 (celery.rs:438-443).  Exact FP64, no FMA.
__device__ __forceinline__ double gap_key(const double size[3], int i, int j, int k) {
    if (i == 0 && j == 0 && k == 0) return -1.0;
    int gi = i < 0 ? -i - 1 : (i > 0 ? i - 1 : 0);
    int gj = j < 0 ? -j - 1 : (j > 0 ? j - 1 : 0);
    int gk = k < 0 ? -k - 1 : (k > 0 ? k - 1 : 0);
    double a = __dmul_rn((double)gi, size[0]);
    double b = __dmul_rn((double)gj, size[1]);
    double c = __dmul_rn((double)gk, size[2]);
    return __dadd_rn(__dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b)), __dmul_rn(c, c));
}

// ---- launchers (tess_grid.cu) ----
struct GridBuffers {
    double* xyz;                // concatenated points, AoS
    const double* src;          // device memory to take the points from (copied to xyz on the way), or null
    const uint32_t* groups;     // point groups or null
    DiagDesc* diags;
    int ndiag;
    uint32_t total;             // total points
    uint64_t total_bins;
    uint32_t chunk;             // chunk_points(total)
    const uint32_t* chunk_diag; // per chunk: diagram id
    const uint32_t* chunk_start;
    uint32_t nchunks;
    unsigned long long* bounds; // 6 per diagram (encoded)
    unsigned* tickets;          // 2: blocks done, for the work of a last block
    uint32_t* bin;
    uint32_t* rank;
    uint32_t* delims;           // total_bins + 1
    uint32_t* scan_tmp;         // block sums
    uint32_t* sorted;
    uint32_t* inv;              // point -> sorted position, or null (built on demand)
    double* spx;
    double* spy;
    double* spz;
    // FP32 split of the sorted positions relative to the centre, x = hi + lo:
    // phi = {hi, point index}, plo = {lo, 0}
    float4* phi;
    float4* plo;
    uint32_t* sgroup;           // null when groups is null
    TabEntry* table;
    int table_gaps;
    int* error_flag;            // set when an input coordinate is not finite
    unsigned* table_len;        // entries of the first diagram's shell table
    uint32_t crowded;           // a bin's points that evenly spread points do not reach
    int* host_flag;             // its value after the bounds, in mapped host memory, or null
    int* check;                 // checked build: the check word
};
// Points per block of the bounds and histogram kernels: one per thread up to
// 131,072 points (512 blocks), where a block's rounds are the kernels' time
// (1,000 points: 17 us in both with 2,048); 2,048 beyond.
constexpr uint32_t kChunkSmall = 256, kChunkLarge = 2048;
constexpr uint32_t chunk_points(uint64_t total) { return total <= 131072 ? kChunkSmall : kChunkLarge; }
constexpr int kScanItems = 8;       // items per thread in the scan
constexpr int kScanThreads = 1024;

// side/fork/join (optional): a second stream and two events; the shell
// table is then built on the side stream while the histogram, scan and
// scatter run (fork after the grid parameters, join before returning).
// bounds_done (optional) is recorded when the input is read and host_flag is
// written.
cudaError_t launch_grid_build(const GridBuffers& g, cudaStream_t s, cudaStream_t side = nullptr,
                              cudaEvent_t fork = nullptr, cudaEvent_t join = nullptr,
                              cudaEvent_t bounds_done = nullptr);
// Kernels launched by one binning pass.
uint64_t grid_launches(uint64_t total_bins, size_t ndiag);
// inv[sorted[s]] = s for s < n (the point -> sorted position map, on demand).
cudaError_t launch_inverse(const uint32_t* sorted, uint32_t* inv, uint32_t n, int* check, cudaStream_t s);
// n bytes from src to dst by the SMs (16-byte aligned pointers; either may be
// the device address of pinned host memory).
cudaError_t launch_copy_bytes(void* dst, const void* src, size_t n, int sms, cudaStream_t s);
// out[0] = most points in one bin, out[1] = points in bins of >= crowd points
// (every bin of every diagram of the set)
cudaError_t launch_occupancy(const uint32_t* delims, uint64_t nbins, uint32_t crowd, unsigned long long* out,
                             int blocks, cudaStream_t s);
size_t scan_tmp_words(uint64_t nitems);

// ---- radius queries (tess_radius.cu) ----
// Query kinds: find_cells_in_radius (celery.rs:753-796), the points of those
// bins (find_neighbors_in_cell_radius, celery.rs:802-818), those within the
// radius (find_neighbors_in_real_radius, celery.rs:825-855), and the
// expanding-search neighbour cloud of a cell (interface.rs:348-365).
enum RadiusMode { RQ_CELLS = 0, RQ_CELL_RADIUS = 1, RQ_REAL_RADIUS = 2, RQ_CLOUD = 3 };

struct RadiusParams {
    const DiagDesc* desc;       // the diagram (a set of one)
    const uint32_t* delims;
    const uint32_t* sorted;
    const double* spx;          // FP64 positions in sorted order
    const double* spy;
    const double* spz;
    const uint32_t* sgroup;     // groups in sorted order, or null (all 0)
    const double* xyz;          // points, AoS, original order
    const double* qxyz;         // query positions (AoS), or null: queries are cells
    const uint32_t* qcell;      // cloud query cells (original index), or null: every cell
    uint32_t nq;
    double radius, radius2;     // and its square
    int64_t group;              // cloud only: < 0 keeps every group
    const short4* rtab;         // cloud only: bin offsets with key <= radius, search order
    uint32_t rtab_len;
    uint32_t* count;            // count pass: results per query
    const uint64_t* offs;       // fill pass: CSR offsets per query
    uint32_t* out;              // fill pass: bin ids or original point indices
    int* err;                   // [0] set to 1 when a query cell is out of range, [1] by a query with more than stage_len results
    const uint32_t* qorder;     // processing order of the queries (spatially sorted), or null
    const float4* phi;          // FP32 high parts of the sorted positions (see GridBuffers), for the FP32 filter
    int f32_filter;             // real radius: pre-filter candidates in FP32 (radius in range)
    // check_cell_in_range as a table: for gaps gx <= gtab_x, gy <= gtab_y, the
    // largest gz <= gtab_z whose squared gap distance is within radius^2
    // (-1: none); null: the FP64 formula per bin
    const int16_t* gtab;
    int gtab_x, gtab_y, gtab_z;
    // counting pass, one query per lane: result k < stage_len of the query at
    // place i of the processing order, at stage[(i / 32 * stage_len + k) * 32 + i % 32]
    uint32_t* stage;
    uint32_t stage_len;
    int lanes;                  // a lane per query
    int unlisted;               // fill pass: some query has more results than are listed
    int gtab_tie;               // some squared gap distance is at most 1% above radius^2
    // bin boundaries per axis: bnd[a * cpd + i] (1 <= i < cpd) is the order
    // code (ord_enc) of the smallest double whose axis_index is >= i
    const unsigned long long* bnd;
};

// RadiusParams::stage_len for a batch of nq queries of a diagram of n points: six
// standard deviations above the results that a uniform density gives a query; 0:
// nothing is listed.
uint32_t radius_stage_len(int mode, uint32_t n, const DiagDesc& D, double radius);
// Whether a batch of nq queries takes a lane per query (else a warp).
bool radius_lanes(int mode, uint32_t nq, uint32_t n, const DiagDesc& D);

// Fills RadiusParams::bnd for diagram 0 (3 * cpd entries).
cudaError_t launch_axis_bounds(const DiagDesc* desc, int cpd, unsigned long long* bnd, cudaStream_t s);

// Spatial processing order for large query batches: a counting sort of the
// queries by the coarse bin (2 x 2 x 2 grid bins) holding their position.
struct QueryOrder {
    uint32_t* qbin;             // [nq] coarse bin of each query
    uint32_t* qrank;            // [nq] arrival rank within its coarse bin
    uint32_t* cnt;              // [ncoarse] queries per coarse bin
    uint64_t* coff;             // [ncoarse + 1] offsets
    uint64_t* scan_tmp;         // csr_tmp_words(ncoarse)
    uint32_t* order;            // [nq] the result
    uint32_t ncoarse;
    int cpdc;                   // coarse bins per dimension
};
cudaError_t launch_query_order(const RadiusParams& p, const QueryOrder& o, int blocks, cudaStream_t s);

cudaError_t launch_radius(const RadiusParams& p, int mode, bool fill, int blocks, cudaStream_t s);
// Bin offsets of the search order (celery.rs:418-679) whose key is at most
// `radius`, sorted by (key, i, j, k), for a grid of cpd bins per axis with
// the given bin sizes.  Returns false if more than max_entries would be kept
// or enumerated.
bool build_radius_table(const double size[3], int cpd, double radius, size_t max_entries,
                        std::vector<short4>& out);
// The gap table of RadiusParams::gtab for this radius; false if the radius is
// not finite and non-negative or the table would exceed max_entries.
bool build_gap_table(const double size[3], const double inv[3], int cpd, double radius, size_t max_entries,
                     std::vector<int16_t>& out, int* gx, int* gy, int* gz, bool* tie);

// ---- launchers (tess_clip.cu) ----
struct ClipParams {
    const DiagDesc* diags;
    int ndiag;
    const double* spx;
    const double* spy;
    const double* spz;
    const float4* phi;              // FP32 split of the sorted positions, point index (see GridBuffers)
    const float4* plo;
    const uint32_t* sorted;
    const uint32_t* delims;
    const uint32_t* sgroup;
    const TabEntry* table;
    // work: sorted positions to process
    const uint32_t* work;          // null: 0 .. total-1
    const uint32_t* work_count;    // null: total
    // FP64 clipping: a list not longer than work_least is left to the next pass, which
    // takes it as its second one (work2) when it is not longer than work2_most
    unsigned work_least;
    const uint32_t* work2;
    const uint32_t* work2_count;
    unsigned work2_most;
    uint32_t total;
    unsigned int* cursor;          // work cursor (zeroed before launch)
    // results, indexed by point (concatenated original order)
    double* vol;
    uint32_t* nface;
    uint64_t* fstart;
    uint8_t* status;
    int32_t* face_nbr;
    double* face_area;
    unsigned long long* face_cursor;
    uint64_t face_cap;
    // routing of failed cells
    uint32_t* list_fp64;          // FP32 passes: guard, degenerate and verify cells
    unsigned int* list_fp64_count;
    uint32_t* list_near;          // cells with a (near-)coincident point
    unsigned int* list_near_count;
    unsigned work_most;           // careful pass over a list longer than this: it hands all of it on
    int settle_most;              // careful pass: a cell with more such cuts is handed on
    uint32_t* list_cap;           // capacity overflow cells or null
    unsigned int* list_cap_count;
    uint32_t* list_dense;         // plain pass: cells of crowded bins, or null
    unsigned int* list_dense_count;
    unsigned int* flag_count;     // careful pass over every cell: cells with an undecided FP32 test
    unsigned int* fail_count;     // cells left with an error status
    unsigned int* reasons;        // per status code: cells routed or failed for it
    unsigned long long* work_ctr; // optional work counters (tested, cuts, new vertices, windows, batches)
    // options
    double search_radius;         // < 0: none
    int has_radius;               // search_radius >= 0
    int64_t target_group;         // < 0: none
    float guard_rel;
    float verify_rel;
    float tol;                    // FP32 first pass: plane tests nearer than this are undecided (FP64 form)
    uint32_t seed_min;            // own-bin count from which a cell is seeded (crowded bins)
    // single-cell geometry output (queries); null for bulk runs
    GeoOut* geo;
    int at_point;                 // 1: site = point[] below, not a diagram point
    double point[3];
    int box_override;             // 1: walls from box[] instead of the diagram's box
    double box[6];                // lo xyz, hi xyz
    // the binning pass's error flag: when it reports non-finite input (1),
    // the clipping kernels return at once (the batch graph runs every pass
    // without a host check in between)
    const int* grid_err;
    // checked build: the check word, the points and the bins of the set
    int* check;
    uint32_t npts;
    uint64_t nbins;
};

// Forms of the clipping:
//   kFormLean     the FP32 first pass (tess_clip_lean.cu: 64 slots, a candidate
//                 plane per lane);
//   kFormDense    the same over the cells of crowded bins, seeded;
//   kFormCareful  the same over the cells those hand on (and over every cell of
//                 a small input), with undecided plane tests settled in FP64;
//   kFormStd      FP64 clipping (tess_clip_f64.cu), for what neither settles
//                 and for single cells;
//   kFormExact    a flag on the first three: faces, vertices, areas and volume
//                 computed in FP64 (the MIXED and FP64 forms, and always the careful
//                 pass)
enum ClipForm : int { kFormLean = 0, kFormStd = 1, kFormDense = 2, kFormCareful = 3, kFormExact = 4 };
cudaError_t launch_clip_lean(const ClipParams& p, int form, int wpb, int blocks, cudaStream_t s);
// One cell with its geometry into p.geo (readable by the host once the stream
// is done): point *p.work of the single diagram, or the site p.point.  Any
// status but ST_OK means the FP64 form has to take it.
cudaError_t launch_cell_lean(const ClipParams& p, cudaStream_t s);
int clip_blocks_lean(int form, int wpb, int device);
cudaError_t launch_clip_f64(const ClipParams& p, int slots, int wpb, int blocks, cudaStream_t s);
int clip_blocks_f64(int slots, int wpb, int device);
// slots (kFormStd): vertex slots per lane, 2, 4 or 8.
cudaError_t launch_clip(const ClipParams& p, int slots, int form, int warps_per_block, int blocks, cudaStream_t s);
int clip_blocks_for(int slots, int form, int warps_per_block, int device);
// CSR offsets (3 launches) and the gather into them (1 launch).
cudaError_t launch_csr_offsets(const uint32_t* nface, uint32_t n, uint64_t* offs, uint64_t* scan_tmp,
                               cudaStream_t s);
cudaError_t launch_csr_gather(const uint32_t* nface, const uint64_t* fstart, const int32_t* face_nbr,
                              const double* face_area, uint32_t n, const uint64_t* offs, int32_t* nbr_out,
                              double* area_out, cudaStream_t s);
size_t csr_tmp_words(uint32_t n);
uint64_t csr_offset_launches(uint32_t n);   // kernels of launch_csr_offsets

// Sets the calling thread's last error message (printf format).
void set_error(const char* fmt, ...);

}  // namespace tess

// Internal declarations shared by the host planner (gbn_plan.cu) and the
// device kernels (gbn_gather.cu, gbn_visit.cuh, gbn_spread.cu, gbn_padcrop.cu, gbn_grad.cu,
// gbn_fftpass.cu, ...).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace gbn {

// Kernel width limit of the register-resident coefficient arrays.
constexpr int JMAX = 8;

// Spread register blocks: a warp sums SB0 x SB1 x SB2 cells of its tile at a
// time (16 accumulators per lane); a tile has at most 8 of them.
template <int NDIM> struct SpreadBlock;
template <> struct SpreadBlock<1> { static constexpr int B0 = 16, B1 = 1, B2 = 1; };
template <> struct SpreadBlock<2> { static constexpr int B0 = 4, B1 = 4, B2 = 1; };
template <> struct SpreadBlock<3> { static constexpr int B0 = 4, B1 = 4, B2 = 1; };
// Spread items are counted by size: level q holds those of more entries than
// SPREAD_SHARE_ENTRIES << q.  A launch shares the items of one level among the
// warps of a CTA each.
constexpr int SPREAD_SHARE_ENTRIES = 32, SPREAD_HEAVY_LEVELS = 6;

template <typename R> struct Cx;
template <> struct Cx<float> { typedef float2 T; };
template <> struct Cx<double> { typedef double2 T; };

// Geometry in memory-axis order (axis 0 fastest) with the tiling of the
// list being processed.
template <typename R>
struct Geom {
    int ndim;
    int N[3], K[3], J[3], T[3], nt[3];
    int L;
    int ncenter[3];          // floor(J*L/2): table index of t = 0
    const R* hr[3];          // device tables (shifted past their zero padding)
    const R* hi[3];          // imaginary tables, nullptr for a real kernel
    int64_t Kprod, Nprod;
    // Grid layout: cell (k0, k1, k2) of coil c of frame f at f * gsf + c * gsp +
    // k0 * gs0 + k1 * gs1 + k2 * gs2.  Plane-major ([frame][coil][K...]), for
    // transforms on the library's own FFT passes coil-minor
    // ([frame][K...][coil]), around cuFFT's passes in 2-D row-interleaved
    // ([K1][frame][coil][K0]), the layout their pruning needs.
    int64_t gsf, gsp, gs0, gs1, gs2;
    R pbc[3];                // phase_before coefficient per memory axis
    int pbo[3];              // summation order of the per-axis phases
    const typename Cx<R>::T* ptab;   // phase_before per cell [K...], or nullptr: computed
    // Checked builds (GBN_CHECKED): the plan's status word and the extents
    // (complex elements) of the grid and sample buffers of the call
    unsigned* check;
    int64_t grid_elems, sample_elems;
};

// Status bits of a checked build: which kind of index failed its bound.
constexpr unsigned CHK_GRID_READ = 1u, CHK_GRID_WRITE = 2u, CHK_SAMPLE_READ = 4u, CHK_SAMPLE_WRITE = 8u,
                   CHK_SCRATCH = 16u, CHK_LIST = 32u, CHK_IMAGE = 64u;

// Coil-lane layout of a CTA: LS lanes per sample (power of two <= 32),
// SW = 32 / LS samples per warp.  Staged grid values for one cell occupy
// LSP complex slots (LS + 1 for LS > 1: conflict-free transposed staging).
struct Lanes {
    int LS, lsh, LSP;
};

// Sorted sample list (one per direction).
template <typename R>
struct SampleList {
    const R* t[3];                  // coordinate per memory axis, list order
    const int* idx;                 // sample index within its frame
    const typename Cx<R>::T* ph;    // per-sample phase (list order) or nullptr
    const short4* ls;               // spread list: window start in tile coordinates
    // Gather list: coefficients precomputed in list order, or nullptr (the
    // kernels then interpolate the tables): entry e holds, from cr + e * cstride
    // on, the J_0 taps of axis 0, then the J_1 taps of axis 1, ...; ci the
    // imaginary parts for a complex kernel.
    const R* cr;
    const R* ci;
    int cstride;
    const R* rec;                   // real single precision: records of cstride values, {cell of the
                                    // window's start in the staged tile, sample index, phase} and
                                    // the coefficients padded with zeros to 16 bytes
    int64_t len;                    // entries in the list
};

// Fill the gather list's precomputed coefficients: from the tables (bitwise
// the values the kernels would interpolate) or, in sparse-matrix mode, from
// per-sample weights wr[d] / wi[d] ([M_total][J_d], sample order = frame
// offset + index).
template <typename R>
struct CoefParams {
    Geom<R> g;
    SampleList<R> s;
    const int64_t* foff;
    int F;
    const R* wr[3];
    const R* wi[3];
    R* out;
    int off, stride;                // an entry's coefficients lie from out + e * stride + off on
    int jsum;
    int cx;
    int* place;                     // [samples] list position of each sample; nullptr: the coefficients
                                    // alone, of sample m (all frames) at out + m * stride + off
};

template <typename R>
struct GatherParams {
    Geom<R> g;
    Lanes ln;
    SampleList<R> s;
    const int4* items;              // {frame, tile, start, count}
    int nitems;
    int coils;
    const int64_t* foff;            // device frame offsets [F+1]
    const typename Cx<R>::T* grid;  // [F][coils][Kprod]
    typename Cx<R>::T* y;           // samples
    int apply_pb;                   // multiply staged cells by phase_before
    R grid_scale;                   // divide staged cells by this (ortho)
    int apply_ph;                   // multiply outputs by the sample phase
    int* tickets;                   // work counter pair of the persistent (3-D) launch, zero
                                    // between launches; the 1-D and 2-D kernels ignore it
    int chunks;                     // coil chunks of LS lanes
};

// Visit lists (gbn_visit.cuh): per (work item, register block) the samples
// whose window touches the block, and their coefficients clipped to it.
template <typename R>
struct VisitBuildParams {
    Geom<R> g;
    SampleList<R> s;
    const int4* items;              // {frame, tile, start, count}
    int nitems, nblk;               // register blocks per tile
    const int64_t* foff;
    const R* rec;                   // the gather's coefficients, at rec + place[sample] * stride
    const int* place;
    int64_t samples, nvisits;       // extents: of place and the records, of vidx and vco
    int stride, jsum;
    int cx;
    int* count;                     // [nitems * nblk], multiples of four
    const long long* start;         // exclusive scan of the counts, [nitems * nblk + 1]
    int* vidx;                      // [nvisits] sample index within its frame (without vco: list
                                    // position), -1 for padding
    R* vco;                         // [nvisits][coefficients], or nullptr: computed in the spread
};

// Sample values of a call, coil-minor and times conj(sample phase).
template <typename R>
struct ValuesParams {
    const typename Cx<R>::T* y;     // samples [frame][coil][m]
    const typename Cx<R>::T* ph;    // sample phase, sample order, or nullptr
    typename Cx<R>::T* out;         // [frame][m][coil]
    const int64_t* foff;
    int F, coils, row;              // row: values per sample of out, from one to the next
    int first, n;                   // the coils laid out
    int64_t M;                      // samples of all frames
    unsigned* check;
    int64_t out_elems;
};

// Coil lanes of a spread that copies the samples as they lie.  1024 x 1024 with
// 1.2 million radial samples, 32 coils, single precision: 1035 us in four chunks of
// 8 lanes, 1926 with 32 lanes.  Double, whose values fill half a sector each: 3.9 ms
// for one chunk of 8, 9.5 with 32 lanes for all.
template <typename R> constexpr int inplace_lanes() { return sizeof(R) == 4 ? 8 : 32; }

template <typename R>
struct VisitParams {
    Geom<R> g;
    SampleList<R> s;                // the entries, where the coefficients are computed on the way
    const long long* start;
    const int* vidx;
    const R* vco;                   // or nullptr: from the tables
    int64_t nvisits;
    const int4* items;
    const int2* parts;              // {scratch slot or -1, nparts}
    int nitems, nblk;
    int nheavy[SPREAD_HEAVY_LEVELS];   // leading items of more entries than 32 << level
    // set by the launcher, per block of a tile: origin, and its offset in the
    // grid, in a scratch tile and in the phase table
    short4 borg[8];
    int64_t boff[8], bcell[8];
    int bscr[8];
    int nshared, nwhole;            // set by the launcher: leading items shared by a CTA's warps, in equal
                                    // runs, and further on a block to each
    int coils, LS, chunks, row;
    int nchunk;                     // coil chunks of the launch (chunks: of the scratch's layout)
    const int64_t* foff;
    const typename Cx<R>::T* vals;  // [frame][m][row] (launch_values), or nullptr: read y in place
    int rec;                        // without vco: place in a row of vals, in reals, of the sample's
                                    // coefficients (launch_coef), or 0: from the tables
    const typename Cx<R>::T* y;
    const typename Cx<R>::T* ph;    // with y: sample phase, sample order, or nullptr
    typename Cx<R>::T* grid;
    typename Cx<R>::T* scratch;     // [slot][chunk][tile cells][LS] partial sums
    int64_t tile_cells, scratch_elems;
    int apply_pb;
};

template <typename R>
struct ReduceParams {
    Geom<R> g;
    Lanes ln;
    const int4* tiles;              // {frame, tile, first slot, nparts}
    int ntiles;
    int coils;
    const typename Cx<R>::T* scratch;
    typename Cx<R>::T* grid;
    int64_t tile_cells;
    int64_t scratch_elems;
    int apply_pb;
};

template <typename R>
struct PadParams {
    int ndim;
    int N[3], K[3];
    int64_t Nprod, Kprod;
    int64_t gsp, gs1, gs2;          // layout of the padded grid: plane (frame * coils + coil), rows, z-planes
    int planes;
    const typename Cx<R>::T* x;
    const R* sn;
    typename Cx<R>::T* out;
    // coil-sensitivity fusion: x is one image per frame [F][N] and plane
    // f * coils + c receives sn * maps[c] * x[f]; nullptr for the plain pad
    const typename Cx<R>::T* maps;
    int coils;
    unsigned* check;                // checked builds: status word
    int64_t x_elems, out_elems;     // extents of x and out
};

template <typename R>
struct CropParams {
    int ndim;
    int N[3], K[3];
    int64_t Nprod, Kprod;
    int64_t gsp, gs1, gs2;          // layout of the grid read: plane (frame * coils + coil), rows, z-planes
    int planes;
    const typename Cx<R>::T* grid;
    const R* sn;
    R scale;
    typename Cx<R>::T* x;
    // coil combination: x[f] = sum_c conj(maps[c]) * (cropped plane f * coils
    // + c), one image per frame; nullptr for the plain crop
    const typename Cx<R>::T* maps;
    int coils;
    unsigned* check;                // checked builds: status word
    int64_t grid_elems, x_elems;    // extents of grid and x
};

template <typename R>
struct GradParams {
    Geom<R> g;
    const R* t[3];                  // coordinates, gather-list order
    const int* idx;                 // sample index of each list entry
    const R* dh[3];                 // derivative tables (shifted like hr)
    const typename Cx<R>::T* ph;    // sample phase, list order, or nullptr
    R phase_shift[3];               // s_d * gamma_d: d(phase)/d(tm_d) / i
    int64_t M;                      // list length (single frame)
    int coils;
    int apply_pb;
    R grid_scale;
    const int* phased;              // the grid holds phase_before and the scale already (or nullptr: it does not)
    const typename Cx<R>::T* grid;  // as the forward left it
    const typename Cx<R>::T* gy;    // [coils][M] incoming gradient
    R* gtm;                         // [M][ndim] out
};

// Device binning (gbn_bin.cu): per-sample pass over coordinates tm
// ([M][ndim], plan precision, device) for the plan's tilings.
template <typename R>
struct BinParams {
    int ndim, F;
    int K[3], J[3], Tg[3], ntg[3], Ts[3], nts[3];
    int ntiles_g, ntiles_s;        // per frame
    double tm_limit;               // |tm| bound (larger or non-finite: err)
    int64_t M;
    const R* tm;
    const int64_t* foff;           // device frame offsets [F+1]
    int* err;                      // set to 1 on an invalid coordinate
    unsigned* gkey;                // [M] gather bin (frame * ntiles_g + tile)
    unsigned* gval;                // [M] sample index (sort payload)
    int* ecount;                   // [M] spread entries of each sample
    const int* eoff;               // [M] exclusive scan of ecount (emit pass)
    int B[3];                      // register block edges
    unsigned long long* nvisits;   // sum over samples of the register blocks their windows touch
    unsigned* skey;                // [entries] spread bin
    unsigned* sval;                // [entries] entry index (sort payload)
    int* em;                       // [entries] sample index
    short4* els;                   // [entries] window start in tile coordinates
};

// Work items from per-bin counts (starts = exclusive scans of the counts).
struct ItemParams {
    int nbins_g, nbins_s, ntiles_g, ntiles_s;
    int gchunk, schunk;
    const unsigned* gkeys;         // sorted bins of the lists' entries
    const unsigned* skeys;
    int glen, slen;
    int* gcnt;                     // parts pass: entries per bin, and the first
    int* gstart;
    int* scnt;
    int* sstart;
    int* gparts;                   // parts pass: gather items per bin
    int* sparts;                   //   spread items per bin
    int* rslots;                   //   scratch slots per bin (parts of split tiles)
    int* rflag;                    //   1 for a split tile
    const int* goff;               // items pass: scans of the above
    const int* soff;
    const int* slotoff;
    const int* roff;
    int4* gitems;
    unsigned* gsize;               // sort key: chunk - count (heaviest first)
    unsigned* gorder;
    int4* sitems;
    int2* sslot;
    unsigned* ssize;
    unsigned* sorder;
    int4* rtiles;
    int* nheavy;                   // parts pass: spread items of more than 32 << level entries
};

// List packing: position i of a sorted list takes sample em[order[i]] (or
// order[i] itself when em is null, the gather list).
template <typename R>
struct PackParams {
    int ndim, F;
    int64_t len;
    const unsigned* order;
    const int* em;
    const short4* els;
    const R* tm;
    const typename Cx<R>::T* ph;
    const int64_t* foff;
    short4* ls_out;
    typename Cx<R>::T* ph_out;
    R* t_out[3];
    int* idx_out;
};

template <typename R> cudaError_t launch_bin_count(const BinParams<R>& p, cudaStream_t s);
template <typename R> cudaError_t launch_bin_emit(const BinParams<R>& p, cudaStream_t s);
cudaError_t launch_bin_parts(const ItemParams& p, cudaStream_t s);
cudaError_t launch_bin_items(const ItemParams& p, cudaStream_t s);
cudaError_t launch_item_order(const ItemParams& p, int n_g, int n_s, int4* gout, int4* sout, int2* slot_out,
                              cudaStream_t s);
template <typename R>
cudaError_t launch_bin_pack(const PackParams<R>& gather, const PackParams<R>& spread, cudaStream_t s);

// Pruned FFT pass along one axis (gbn_fftpass.cu), of length L.
//   Plain (sn null): ncols columns; column j = array j / S, place j % S, its
//   element n at in[(j / S) psi + j % S + n S], at out[(j / S) pso + j % S + n S];
//   elements >= nin are read as zero, elements >= nout are not written.
//   Image (sn set): forward, image [frames][coils][nin][Sxy] times sn
//   [nin][Sxy] (with maps: one image [frames][nin][Sxy] times maps
//   [coils][nin][Sxy]) to arrays [frames (pso)][L][Sxy][coils], S = Sxy coils;
//   inverse, arrays [frames (psi)][L][Sxy][coils] to the image's nout elements
//   times scale sn.
struct FftPassParams {
    const float2* in;
    float2* out;
    const float2* tw;               // exp(-2 pi i m / L), m < L
    int L, nin, nout;
    int64_t ncols, S, psi, pso;
    const float* sn;
    const float2* maps;
    float scale;                    // image, inverse
    int frames, coils, Sxy;
    int cwsh, nct, nxt;             // set by the launcher: coils per CTA (log2), CTAs over coils and places
    // Forward, plain: outputs times phase[(array % prows) L + k] (or nullptr),
    // divided by div, the orthonormal scale.
    const float2* phase;
    int prows;
    float div;
    int* state;                     // receives whether they were (or nullptr)
    unsigned* check;                // checked builds: status word and extents
    int64_t in_elems, out_elems;
};
bool fftpass_supported(int L);
// sign -1: forward (exp(-2 pi i nk / L)), +1: inverse (unnormalised)
cudaError_t launch_fftpass(const FftPassParams& p, int sign, cudaStream_t s);

template <typename R> cudaError_t launch_gather(const GatherParams<R>& p, cudaStream_t s);
template <typename R> cudaError_t launch_visit_count(const VisitBuildParams<R>& p, cudaStream_t s);
template <typename R> cudaError_t launch_visit_fill(const VisitBuildParams<R>& p, cudaStream_t s);
template <typename R> cudaError_t launch_values(const ValuesParams<R>& p, cudaStream_t s);
template <typename R> cudaError_t launch_spread_visits(const VisitParams<R>& p, cudaStream_t s);
template <typename R> cudaError_t launch_reduce(const ReduceParams<R>& p, cudaStream_t s);
template <typename R> cudaError_t launch_pad(const PadParams<R>& p, cudaStream_t s);
template <typename R> cudaError_t launch_crop(const CropParams<R>& p, cudaStream_t s);
// x[f] = sum_c conj(maps[c]) * images[f][c], in coil order; n values per image.
cudaError_t launch_combine(const float2* images, const float2* maps, float2* x, int frames, int coils, int64_t n,
                           cudaStream_t s);
template <typename R> cudaError_t launch_grad(const GradParams<R>& p, cudaStream_t s);
template <typename R> cudaError_t launch_coef(const CoefParams<R>& p, cudaStream_t s);
// phase_before of every grid cell, [K_{ndim-1}]...[K_0].
template <typename R> cudaError_t launch_phase_table(const Geom<R>& g, typename Cx<R>::T* out, cudaStream_t s);
// The gather on a coil-minor grid (gbn_gather_cm.cu), and whether it takes a launch.
bool gather_cm_supported(const GatherParams<float>& p);
cudaError_t launch_gather_cm(const GatherParams<float>& p, cudaStream_t s);

// Shared-memory bytes needed by the gather kernel for a lane layout.
template <typename R> size_t gather_smem(const Geom<R>& g, const Lanes& ln);
// 32 x the register blocks of a spread tile.
int spread_threads(int ndim, const int* T);

// Raise a kernel's dynamic shared-memory limit to at least `bytes` on the
// current device.  The attribute is set once per (kernel, device) and size
// (later launches needing no more skip the call), so launches recorded in a
// CUDA graph after a warm-up call make no attribute call.
cudaError_t ensure_dynamic_smem(const void* kernel, size_t bytes);

// CTAs of `kernel` (with this block size and dynamic shared memory) that fit
// on the current device at once: the grid of a persistent launch.  Cached
// per (kernel, device, threads, smem); 0 if the query fails.
int resident_ctas(const void* kernel, int threads, size_t smem);

// Address and size of the fixed no-alloc scratch array on the current device
// (gbn_noalloc.cu); looked up on every request.
cudaError_t noalloc_scratch(void** ptr, size_t* bytes);

cudaError_t launch_dtft(bool adjoint, int ndim, const int* Nd, const double* n_shift,
                        const double* omega, int64_t M, const double2* in, double2* out,
                        int reps, cudaStream_t s);

}  // namespace gbn

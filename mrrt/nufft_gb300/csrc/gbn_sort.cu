// Device-side scan and stable radix sort used by the sample binning
// (gbn_bin.cu).  Written for this project (no CUB): exclusive scans and an
// LSD radix sort with 8-bit digits whose scatter ranks equal keys in input
// order, so the sort is stable and its output is the same in every run.
//
// Binning some 10^5 samples is a chain of small launches, each shorter than
// the gap to the next, so what counts is their number: several scans, and
// the passes of two sorts, share a launch (blockIdx.y is the job), a scan of
// up to SCAN_FLAT tiles takes two launches (one for a single tile), and its
// total comes with it.
#include <cuda_runtime.h>

#include <algorithm>
#include <utility>

#include "gbn_sort.cuh"

namespace gbn {

namespace {

constexpr int SCAN_THREADS = 512;
constexpr int SCAN_PER_THREAD = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_PER_THREAD;   // 2048 elements per CTA

constexpr int RADIX_THREADS = 256;
constexpr int RADIX_WARPS = RADIX_THREADS / 32;
constexpr int RADIX_BUCKETS = 256;
// Items per lane: 16 (4096 items per CTA) for large sorts; 2 (512 per CTA)
// below RADIX_SMALL items, where 4096-item tiles would leave most SMs idle.
constexpr int RADIX_ROUNDS_LARGE = 16, RADIX_ROUNDS_SMALL = 2;
constexpr int64_t RADIX_SMALL = 1 << 20;
inline int radix_rounds(int64_t n) { return n < RADIX_SMALL ? RADIX_ROUNDS_SMALL : RADIX_ROUNDS_LARGE; }

inline size_t round256(size_t v) { return (v + 255) & ~(size_t)255; }

// Exclusive scan of a CTA's values held one per thread; *out_total gets the
// CTA total.
template <typename T>
__device__ __forceinline__ T block_exclusive_scan(T v, T* warp_sums, T* out_total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        T w = lane < nw ? warp_sums[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const T y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < nw) warp_sums[lane] = w;   // inclusive
    }
    __syncthreads();
    const T before = warp > 0 ? warp_sums[warp - 1] : 0;
    *out_total = warp_sums[(blockDim.x >> 5) - 1];
    return before + x - v;
}

template <typename TI, typename TO>
struct ScanSet {
    const TI* in[SCAN_JOBS];
    TO* out[SCAN_JOBS];
    TO* total[SCAN_JOBS];
    TO* bsum[SCAN_JOBS];      // sums of the tiles (null for one tile)
    const TO* boff[SCAN_JOBS];   // their scan, where it was made by another launch
    int64_t n[SCAN_JOBS];
};

template <typename TI, typename TO>
__device__ __forceinline__ TO load_tile(const TI* in, int64_t n, TO (&v)[SCAN_PER_THREAD]) {
    const int64_t base = (int64_t)blockIdx.x * SCAN_TILE + (int64_t)threadIdx.x * SCAN_PER_THREAD;
    TO s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_PER_THREAD; ++k) {
        v[k] = base + k < n ? in[base + k] : 0;
        s += v[k];
    }
    return s;
}

// Sums of the tiles of jobs of more than one.
template <typename TI, typename TO>
__global__ void __launch_bounds__(SCAN_THREADS) scan_sums_kernel(const ScanSet<TI, TO> p) {
    __shared__ TO ws[32];
    const int j = blockIdx.y;
    if (p.n[j] <= (int64_t)blockIdx.x * SCAN_TILE || !p.bsum[j]) return;   // the whole CTA
    TO v[SCAN_PER_THREAD], total;
    block_exclusive_scan(load_tile<TI, TO>(p.in[j], p.n[j], v), ws, &total);
    if (threadIdx.x == 0) p.bsum[j][blockIdx.x] = total;
}

// The scans.  A tile's offset is the sum of the tiles before it, which each
// CTA adds up for itself from their sums (at most SCAN_FLAT of them), or
// reads where those were scanned before.
template <typename TI, typename TO>
__global__ void __launch_bounds__(SCAN_THREADS) scan_kernel(const ScanSet<TI, TO> p) {
    __shared__ TO ws[32], before;
    const int j = blockIdx.y;
    const int64_t n = p.n[j];
    if (n <= (int64_t)blockIdx.x * SCAN_TILE && blockIdx.x > 0) return;   // the whole CTA
    TO total;
    if (threadIdx.x == 0) before = p.boff[j] ? p.boff[j][blockIdx.x] : (TO)0;
    if (p.bsum[j] && !p.boff[j]) {
        TO s = 0;
        for (int b = threadIdx.x; b < (int)blockIdx.x; b += SCAN_THREADS) s += p.bsum[j][b];
        block_exclusive_scan(s, ws, &total);
        if (threadIdx.x == 0) before = total;
    }
    __syncthreads();
    TO v[SCAN_PER_THREAD];
    const TO s = load_tile<TI, TO>(p.in[j], n, v);
    TO run = before + block_exclusive_scan(s, ws, &total);
    const int64_t base = (int64_t)blockIdx.x * SCAN_TILE + (int64_t)threadIdx.x * SCAN_PER_THREAD;
#pragma unroll
    for (int k = 0; k < SCAN_PER_THREAD; ++k) {
        if (base + k < n) p.out[j][base + k] = run;
        run += v[k];
    }
    // the last tile's end
    if (threadIdx.x == 0 && p.total[j] && (int64_t)(blockIdx.x + 1) * SCAN_TILE >= n) *p.total[j] = before + total;
}

__device__ __forceinline__ int digit_of(unsigned key, int shift) { return (int)((key >> shift) & 0xffu); }

// One digit of the sorts (a job without CTAs has no pass left).
struct SortPass {
    const unsigned *keys[SORT_JOBS], *vals[SORT_JOBS];
    unsigned *keys_out[SORT_JOBS], *vals_out[SORT_JOBS];
    int *hist[SORT_JOBS], *offs[SORT_JOBS];
    int64_t n[SORT_JOBS];
    int nblk[SORT_JOBS];
    int shift;
};

template <int RADIX_ROUNDS>
__global__ void __launch_bounds__(RADIX_THREADS) radix_hist_kernel(const SortPass p) {
    const int j = blockIdx.y, nblk = p.nblk[j], shift = p.shift;
    if ((int)blockIdx.x >= nblk) return;   // the whole CTA
    const int64_t n = p.n[j];
    const unsigned* keys = p.keys[j];
    int* hist = p.hist[j];
    constexpr int RADIX_TILE = RADIX_THREADS * RADIX_ROUNDS;
    __shared__ int h[RADIX_BUCKETS];
    for (int q = threadIdx.x; q < RADIX_BUCKETS; q += blockDim.x) h[q] = 0;
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t base = (int64_t)blockIdx.x * RADIX_TILE + (int64_t)warp * (32 * RADIX_ROUNDS) + lane;
#pragma unroll 4
    for (int r = 0; r < RADIX_ROUNDS; ++r) {
        const int64_t i = base + r * 32;
        if (i < n) atomicAdd(&h[digit_of(keys[i], shift)], 1);
    }
    __syncthreads();
    // digit-major: the scan of hist gives, for digit d and CTA b, the output
    // position of the CTA's first item with digit d
    for (int q = threadIdx.x; q < RADIX_BUCKETS; q += blockDim.x) hist[(int64_t)q * nblk + blockIdx.x] = h[q];
}

// Items of a CTA in index order are (warp, round, lane); each lands after
// every earlier item with the same digit, so the pass is stable.
template <int RADIX_ROUNDS>
__global__ void __launch_bounds__(RADIX_THREADS) radix_scatter_kernel(const SortPass p) {
    const int j = blockIdx.y, nblk = p.nblk[j], shift = p.shift;
    if ((int)blockIdx.x >= nblk) return;   // the whole CTA
    const int64_t n = p.n[j];
    const unsigned *keys = p.keys[j], *vals = p.vals[j];
    const int* offs = p.offs[j];
    unsigned *keys_out = p.keys_out[j], *vals_out = p.vals_out[j];
    constexpr int RADIX_TILE = RADIX_THREADS * RADIX_ROUNDS;
    __shared__ int wh[RADIX_WARPS][RADIX_BUCKETS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int q = lane; q < RADIX_BUCKETS; q += 32) wh[warp][q] = 0;
    __syncwarp();
    const int64_t base = (int64_t)blockIdx.x * RADIX_TILE + (int64_t)warp * (32 * RADIX_ROUNDS) + lane;
    const unsigned lt = (1u << lane) - 1u;
    unsigned k[RADIX_ROUNDS], v[RADIX_ROUNDS];
    // sweep 1: digit counts of this warp's items
#pragma unroll
    for (int r = 0; r < RADIX_ROUNDS; ++r) {
        const int64_t i = base + r * 32;
        const bool ok = i < n;
        k[r] = ok ? keys[i] : 0u;
        v[r] = ok ? vals[i] : 0u;
        const int d = ok ? digit_of(k[r], shift) : RADIX_BUCKETS + lane;   // out of range: matches no one
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        if (ok && (peers & lt) == 0) wh[warp][d] += __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // warp offsets within the CTA, per digit, in warp order
    for (int d = threadIdx.x; d < RADIX_BUCKETS; d += blockDim.x) {
        int acc = offs[(int64_t)d * nblk + blockIdx.x];
        for (int w = 0; w < RADIX_WARPS; ++w) {
            const int c = wh[w][d];
            wh[w][d] = acc;
            acc += c;
        }
    }
    __syncthreads();
    // sweep 2: scatter
#pragma unroll
    for (int r = 0; r < RADIX_ROUNDS; ++r) {
        const int64_t i = base + r * 32;
        const bool ok = i < n;
        const int d = ok ? digit_of(k[r], shift) : RADIX_BUCKETS + lane;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        if (ok) {
            const int pos = wh[warp][d] + __popc(peers & lt);
            keys_out[pos] = k[r];
            vals_out[pos] = v[r];
        }
        __syncwarp();
        if (ok && (peers & lt) == 0) wh[warp][d] += __popc(peers);
        __syncwarp();
    }
}

// Tiles up to which each CTA adds up the sums before its own: two loads a
// thread.  Beyond, the sums are scanned by a launch of their own.
constexpr int64_t SCAN_FLAT = 1024;

template <typename TI, typename TO>
cudaError_t scan_set(ScanSet<TI, TO>& p, int count, void* temp, cudaStream_t s) {
    int64_t most = 1;
    for (int j = 0; j < count; ++j) most = std::max(most, (p.n[j] + SCAN_TILE - 1) / SCAN_TILE);
    if (most > SCAN_FLAT && count > 1) {   // one by one, sharing temp
        for (int j = 0; j < count; ++j) {
            ScanSet<TI, TO> one = {};
            one.in[0] = p.in[j];
            one.out[0] = p.out[j];
            one.total[0] = p.total[j];
            one.n[0] = p.n[j];
            cudaError_t e = scan_set(one, 1, temp, s);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
    char* t = reinterpret_cast<char*>(temp);
    const size_t part = round256((size_t)most * sizeof(long long));
    for (int j = 0; j < count; ++j) {
        p.boff[j] = nullptr;
        p.bsum[j] = p.n[j] > SCAN_TILE ? reinterpret_cast<TO*>(t + j * part) : nullptr;
    }
    const dim3 grid((unsigned)most, (unsigned)count);
    if (most > 1) scan_sums_kernel<TI, TO><<<grid, SCAN_THREADS, 0, s>>>(p);
    if (most > SCAN_FLAT) {
        ScanSet<TO, TO> sums = {};
        sums.in[0] = p.bsum[0];
        sums.out[0] = reinterpret_cast<TO*>(t + part);
        sums.n[0] = most;
        cudaError_t e = scan_set(sums, 1, t + 2 * part, s);
        if (e != cudaSuccess) return e;
        p.boff[0] = sums.out[0];
    }
    scan_kernel<TI, TO><<<grid, SCAN_THREADS, 0, s>>>(p);
    return cudaGetLastError();
}

}  // namespace

size_t scan_temp_bytes(int64_t n) {
    size_t bytes = 0;
    const int64_t flat = std::min((n + SCAN_TILE - 1) / SCAN_TILE, SCAN_FLAT);
    while (n > SCAN_TILE) {
        const int64_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
        bytes += 2 * round256((size_t)nb * sizeof(long long));
        n = nb;
    }
    return std::max(bytes, SCAN_JOBS * round256((size_t)flat * sizeof(long long))) + 256;
}

cudaError_t exclusive_scans(const ScanJob* jobs, int count, void* temp, cudaStream_t s) {
    if (count < 1 || count > SCAN_JOBS) return cudaErrorInvalidValue;
    ScanSet<int, int> p = {};
    for (int j = 0; j < count; ++j) {
        p.in[j] = jobs[j].in;
        p.out[j] = jobs[j].out;
        p.n[j] = jobs[j].n;
        p.total[j] = jobs[j].total;
    }
    return scan_set(p, count, temp, s);
}

cudaError_t exclusive_scan64(const int* in, long long* out, int64_t n, long long* total, void* temp, cudaStream_t s) {
    ScanSet<int, long long> p = {};
    p.in[0] = in;
    p.out[0] = out;
    p.n[0] = n;
    p.total[0] = total;
    return scan_set(p, 1, temp, s);
}

// temp layout: keys and values of the other ping-pong side, the digit
// histogram, its scan, the scans' own temporaries (each 256-byte aligned)
size_t radix_temp_bytes(int64_t n) {
    // the larger of the two tilings' histograms (either may run for a
    // smaller sort sharing this workspace)
    const int64_t nblk = (n + RADIX_THREADS * RADIX_ROUNDS_SMALL - 1) / (RADIX_THREADS * RADIX_ROUNDS_SMALL);
    const int64_t nh = nblk * RADIX_BUCKETS;
    return 2 * round256((size_t)n * sizeof(unsigned)) + 2 * round256((size_t)nh * sizeof(int)) +
           scan_temp_bytes(nh);
}

cudaError_t radix_sort_pairs(SortJob (&jobs)[SORT_JOBS], void* const (&temp)[SORT_JOBS], cudaStream_t s) {
    int64_t most = 0;
    int bits = 0;
    for (const SortJob& q : jobs)
        if (q.n > 1) {
            most = std::max(most, q.n);
            bits = std::max(bits, q.bits);
        }
    const int rounds = radix_rounds(most);
    const int tile = RADIX_THREADS * rounds;
    SortPass p = {};
    unsigned *k2[SORT_JOBS], *v2[SORT_JOBS];
    int longest = 0;
    void* scan_tmp = nullptr;   // the longest job's serve both
    for (int j = 0; j < SORT_JOBS; ++j) {
        const int64_t n = std::max<int64_t>(jobs[j].n, 0);
        const int64_t nh = (n + tile - 1) / tile * RADIX_BUCKETS;
        char* t = reinterpret_cast<char*>(temp[j]);
        k2[j] = reinterpret_cast<unsigned*>(t);
        t += round256((size_t)n * sizeof(unsigned));
        v2[j] = reinterpret_cast<unsigned*>(t);
        t += round256((size_t)n * sizeof(unsigned));
        p.hist[j] = reinterpret_cast<int*>(t);
        t += round256((size_t)nh * sizeof(int));
        p.offs[j] = reinterpret_cast<int*>(t);
        t += round256((size_t)nh * sizeof(int));
        if (jobs[j].n >= jobs[longest].n) longest = j;
        if (longest == j) scan_tmp = t;
        p.n[j] = n;
    }
    for (p.shift = 0; p.shift < bits; p.shift += 8) {
        ScanJob scans[SORT_JOBS];
        int widest = 0;
        for (int j = 0; j < SORT_JOBS; ++j) {
            const bool on = jobs[j].n > 1 && p.shift < jobs[j].bits;
            p.nblk[j] = on ? (int)((jobs[j].n + tile - 1) / tile) : 0;
            p.keys[j] = jobs[j].keys;
            p.vals[j] = jobs[j].vals;
            p.keys_out[j] = k2[j];
            p.vals_out[j] = v2[j];
            widest = std::max(widest, p.nblk[j]);
            scans[j] = ScanJob{p.hist[j], p.offs[j], (int64_t)p.nblk[j] * RADIX_BUCKETS, nullptr};
            if (on) {
                std::swap(jobs[j].keys, k2[j]);
                std::swap(jobs[j].vals, v2[j]);
            }
        }
        const dim3 grid((unsigned)widest, SORT_JOBS);
        if (rounds == RADIX_ROUNDS_SMALL) radix_hist_kernel<RADIX_ROUNDS_SMALL><<<grid, RADIX_THREADS, 0, s>>>(p);
        else radix_hist_kernel<RADIX_ROUNDS_LARGE><<<grid, RADIX_THREADS, 0, s>>>(p);
        cudaError_t e = exclusive_scans(scans, SORT_JOBS, scan_tmp, s);
        if (e != cudaSuccess) return e;
        if (rounds == RADIX_ROUNDS_SMALL) radix_scatter_kernel<RADIX_ROUNDS_SMALL><<<grid, RADIX_THREADS, 0, s>>>(p);
        else radix_scatter_kernel<RADIX_ROUNDS_LARGE><<<grid, RADIX_THREADS, 0, s>>>(p);
    }
    return cudaGetLastError();
}

}  // namespace gbn

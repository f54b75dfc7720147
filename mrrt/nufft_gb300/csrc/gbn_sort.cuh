// Device scan and stable radix sort (gbn_sort.cu).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace gbn {

// Exclusive scans, several in one launch: out[i] = in[0] + ... + in[i-1]
// (in and out may not alias); total (device, optional) receives the sum of
// all n.  Each is asynchronous on s.
struct ScanJob {
    const int* in;
    int* out;
    int64_t n;
    int* total;
};
constexpr int SCAN_JOBS = 4;
// Bytes of device temporaries for scans of at most n elements each.
size_t scan_temp_bytes(int64_t n);
cudaError_t exclusive_scans(const ScanJob* jobs, int count, void* temp, cudaStream_t s);
// One scan with 64-bit sums.
cudaError_t exclusive_scan64(const int* in, long long* out, int64_t n, long long* total, void* temp, cudaStream_t s);

// A stable sort of (keys, vals) by the low `bits` bits of keys.
struct SortJob {
    unsigned* keys;
    unsigned* vals;
    int64_t n;
    int bits;
};
constexpr int SORT_JOBS = 2;
// Bytes of device temporaries for a sort of n pairs.
size_t radix_temp_bytes(int64_t n);
// Sorts both jobs, pass by pass in shared launches.  Asynchronous on s; the
// result is the same in every run, and lies where the job's keys and vals
// point on return (its own arrays or its temporaries).
cudaError_t radix_sort_pairs(SortJob (&jobs)[SORT_JOBS], void* const (&temp)[SORT_JOBS], cudaStream_t s);

}  // namespace gbn

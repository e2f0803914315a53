// Internal device-side helpers shared by the CUDA translation units of libsge.
#pragma once
#include <cuda_runtime.h>

#include "common.hpp"

namespace sge {

// Restores the caller's current device when an entry point returns, so that
// a call which selects the graph's (or scorer's) device does not move a
// multi-GPU caller's later allocations and launches to that device.
struct DeviceGuard {
    int prev = -1;
    DeviceGuard() {
        if (cudaGetDevice(&prev) != cudaSuccess) {
            prev = -1;
            cudaGetLastError();
        }
    }
    ~DeviceGuard() {
        if (prev >= 0) cudaSetDevice(prev);
    }
    DeviceGuard(const DeviceGuard &) = delete;
    DeviceGuard &operator=(const DeviceGuard &) = delete;
};

// Exclusive prefix sum of n uint32 values in device memory (out may be
// `in` itself), ordered on stream s; temporary space is allocated here.
sge_status device_exclusive_scan(const uint32_t *in, uint32_t *out, uint64_t n, cudaStream_t s);

// Sorts n 64-bit keys of `bits` bits in device memory on stream s (tmp: as
// many); the result is in `keys`, which may have changed places with tmp.
sge_status device_sort_keys(unsigned long long *&keys, unsigned long long *&tmp, uint64_t n, uint32_t bits,
                            cudaStream_t s);

// sge_enumerate; any_representative = true may write another member of each
// automorphism class than the plan's restrictions keep.
sge_status enumerate_rows(sge_graph *g, const sge_plan *p, uint32_t *d_out, uint64_t capacity, uint64_t *n_matches,
                          bool any_representative);

// Wraps a CSR already in device memory on `device` (d_off: n+1 offsets,
// d_adj: nnz neighbours; symmetric, lists strictly increasing, no
// self-loops) as a graph, which takes ownership of both arrays (also on
// failure).  The root-edge list and the wedge sample are built on the device;
// the degree statistics on the host, from h_off when the caller has the CSR in
// host memory, else from a copy of the offsets.  planner_stats = false leaves
// out what only the planner reads.
sge_status graph_adopt(uint32_t *d_off, uint32_t *d_adj, uint32_t n, uint64_t nnz, int device, sge_graph **out,
                       const uint32_t *h_off = nullptr, const uint32_t *h_adj = nullptr, bool planner_stats = true);

}  // namespace sge

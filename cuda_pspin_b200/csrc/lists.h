// lists.h -- device construction of a dense sample's site lists, quartet table and
// neighbour masks (lists.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "internal.h"

namespace pspin {

// plan() (masked) or plan_fc() (every quartet active in channel 0, or !tiles) finds
// the sizes and whether tiles pay; write() puts everything in place:
// the entries at `out` (entry `entry0` of the engine's), its chunk starts (chunk
// `chunk0`), site-chunk table, quartets and neighbour masks.  g4 and mask stay
// the caller's until then.  A plan fails where device memory is short, or (invalid
// value) where a sample's entries are not counted in 31 bits: the host lays it out.
struct DeviceLists {
    bool tiles = false;
    int64_t nominal = 0, entries = 0, chunks = 0, quartets = 0;
    double flops = 0.0;
    size_t held = 0;         // bytes of device memory until destroyed

    DeviceLists() = default;
    DeviceLists(const DeviceLists&) = delete;
    DeviceLists& operator=(const DeviceLists&) = delete;
    ~DeviceLists();
    cudaError_t plan(int N, const double* g4, const uint8_t* mask, const double* g2_host, cudaStream_t st);
    cudaError_t plan_fc(int N, const double* g4, const uint8_t* mask, const double* g2_host, cudaStream_t st);
    cudaError_t write(int64_t entry0, int64_t chunk0, int2* out, int64_t* chunk_start, int* site_chunks, Q64* q, uint32_t* nb,
                      cudaStream_t st) const;

private:
    int N = 0;
    bool fc = false;
    const double* d_g4 = nullptr;
    const uint8_t* d_mask = nullptr;
    double* d_g2 = nullptr;
    void* slab = nullptr;
    void* groups_slab = nullptr;
    int2 *d_totals = nullptr, *d_sizes = nullptr;
    int* d_gbase = nullptr;
    unsigned long long* d_sums = nullptr;
    uint32_t* d_nb = nullptr;
    int64_t* d_qoff = nullptr;
    int4* d_groups = nullptr;
    uint8_t* d_width = nullptr;
};

}  // namespace pspin

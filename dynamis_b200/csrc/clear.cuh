// Ranges of memory set to a byte, as one launch of a chain.
#pragma once

#include <algorithm>

#include "common.cuh"

namespace dynb {

struct ClearRange { void* at; int64_t bytes; uint32_t byte; };
constexpr int CLEAR_RANGES = 4;
struct ClearRanges { ClearRange range[CLEAR_RANGES]; };

static __global__ void __launch_bounds__(256)
clear_ranges_kernel(const ClearRanges c)
{
    chain_begin();
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
#pragma unroll
    for (int k = 0; k < CLEAR_RANGES; k++) {
        unsigned char* const at = static_cast<unsigned char*>(c.range[k].at);
        const int64_t bytes = c.range[k].bytes;
        if (bytes <= 0) continue;
        const uint32_t word = (c.range[k].byte & 255u) * 0x01010101u;
        // single bytes up to the first multiple of 16 and behind the last one
        const int64_t head = min((int64_t)((0u - (uint32_t)reinterpret_cast<uintptr_t>(at)) & 15u), bytes);
        const int64_t body = (bytes - head) / 16, tail = bytes - head - 16 * body;
        uint4* const wide = reinterpret_cast<uint4*>(at + head);
        for (int64_t i = i0; i < body; i += stride) wide[i] = make_uint4(word, word, word, word);
        if (i0 < head) at[i0] = (unsigned char)word;
        if (i0 < tail) at[bytes - tail + i0] = (unsigned char)word;
    }
}

// A memset between two kernels is a full wait on both sides of it: rebuild of 1 M atoms 403 us with them and 397 without, refresh 648 and 631.
static inline cudaError_t clear_ranges(cudaStream_t stream, ClearRange a, ClearRange b = {}, ClearRange c = {}, ClearRange d = {})
{
    const ClearRanges ranges = {{a, b, c, d}};
    int64_t most = 0;
    for (const ClearRange& r : ranges.range) most = std::max(most, r.bytes);
    if (most == 0) return cudaSuccess;
    const int64_t blocks = std::min<int64_t>((most + 4095) / 4096, (int64_t)sm_count_cached() * 4);
    return launch_chained(clear_ranges_kernel, (unsigned)blocks, 256, 0, stream, ranges);
}

}  // namespace dynb

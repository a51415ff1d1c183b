// Device helpers shared by the count pass (sj_join.cu) and the emission pass
// (sj_emit.cu): the warp bit-matrix transpose and the candidate-validity masks
// of a block of 32 stream positions.  Both passes must agree bit for bit.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace sjdev {

// 32x32 bit-matrix transpose over a warp: lane i holds row i; afterwards lane j
// holds column j.  The usual five exchange steps; the halves of a step's result
// are merged by one byte permute (distances 16 and 8), or by a rotation and one
// three-input select (4, 2, 1), with the selectors, rotations and masks that
// depend on the lane made once: 13 instructions a transpose, half of the
// shift-and-mask form.
struct Transpose {
    uint32_t sel16, sel8, rot4, rot2, rot1, keep4, keep2, keep1;

    __device__ __forceinline__ explicit Transpose(uint32_t lane)
    {
        sel16 = (lane & 16u) ? 0x3276u : 0x5410u;
        sel8 = (lane & 8u) ? 0x3715u : 0x6240u;
        rot4 = (lane & 4u) ? 28u : 4u;
        rot2 = (lane & 2u) ? 30u : 2u;
        rot1 = (lane & 1u) ? 31u : 1u;
        keep4 = (lane & 4u) ? 0xf0f0f0f0u : 0x0f0f0f0fu;
        keep2 = (lane & 2u) ? 0xccccccccu : 0x33333333u;
        keep1 = (lane & 1u) ? 0xaaaaaaaau : 0x55555555u;
    }

    __device__ __forceinline__ uint32_t operator()(uint32_t x) const
    {
        x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 16), sel16);
        x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 8), sel8);
        uint32_t y = __shfl_xor_sync(0xffffffffu, x, 4);
        x = (x & keep4) | (__funnelshift_l(y, y, rot4) & ~keep4);
        y = __shfl_xor_sync(0xffffffffu, x, 2);
        x = (x & keep2) | (__funnelshift_l(y, y, rot2) & ~keep2);
        y = __shfl_xor_sync(0xffffffffu, x, 1);
        return (x & keep1) | (__funnelshift_l(y, y, rot1) & ~keep1);
    }
};

// Candidate-validity masks of a block of 32 stream positions starting at blk.
// Inside a symmetric home segment (stream positions < homeEnd are the home
// cell's points from the query tile's first point on) a query keeps candidates
// at or after itself; the mirrored direction drops the query itself.
__device__ __forceinline__ uint32_t home_bits(uint32_t blk, uint32_t homeEnd, bool sym)
{
    if (!sym || blk >= homeEnd) return 0u;
    const uint32_t hn = homeEnd - blk;
    return hn >= 32 ? 0xffffffffu : ((1u << hn) - 1u);
}

__device__ __forceinline__ uint32_t row_keep(uint32_t qi, uint32_t blk, uint32_t hb)
{
    const int lo = (int)qi - (int)blk;   // home candidate index >= query index
    const uint32_t ge = lo <= 0 ? 0xffffffffu : (lo >= 32 ? 0u : (0xffffffffu << lo));
    return ~hb | (hb & ge);
}

__device__ __forceinline__ uint32_t mir_keep(uint32_t qi, uint32_t blk, uint32_t hb)
{
    const int lo = (int)qi - (int)blk;
    return (lo >= 0 && lo < 32) ? ~(hb & (1u << lo)) : 0xffffffffu;
}

}  // namespace sjdev

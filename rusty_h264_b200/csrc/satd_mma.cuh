// satd_mma.cuh -- 4x4 Hadamard SATD (Σ|H·(p−s)·Hᵀ|, satd_4x4_sum,
// crates/rusty_h264-common/src/transform.rs:701) on the tensor cores.
//
// The 2D Hadamard of a 4x4 block is a 16x16 matrix of ±1 applied to its 16
// pixels, so eight blocks' coefficients of the residual are one
// mma.m16n8k32 (s8 x u8, s32 accumulators, exact): A = [H | −H], a B column
// the 16 predicted and then the 16 source pixels of a block, D = H·p − H·s.
// A lane's B registers are one 4-pixel row word of the prediction and the
// same row of the source: lane l serves column l / 4, row l % 4, straight
// from the packed bytes it loaded, with no unpacking and no subtraction.  One mma and
// six integer instructions (four |.|, two three-input adds) then price eight
// 4x4 blocks per warp, where the butterflies of satd4x4_packed take about 100
// instructions for 32.  mma.sync, not tcgen05: a search round prices a few
// candidates and waits for them, and the register-to-register mma answers in
// about 20 cycles (8 cycles apart on one sub-core, measured), while a tcgen05
// product would go through shared memory, tensor memory and a commit.
#pragma once

#include "h264a_device.cuh"

namespace h264a {

// The lane's A fragment of [H | −H]: rows g = lane / 4 and g + 8, k = 4q..4q+3
// (q = lane % 4) and 16 + those.  Row m = 4u + v is the product of the signs
// (−1)^popc(u & r) over pixel row r and (−1)^popc(v & c) over column c; the
// sum of absolute values does not depend on the rows' order or signs.
struct HadFrag {
    uint32_t a[4];
};
__device__ __forceinline__ HadFrag had_frag(int lane) {
    const int g = lane >> 2, q = lane & 3;
    HadFrag h;
#pragma unroll
    for (int half = 0; half < 2; half++) {
        const int m = g + 8 * half, u = m >> 2, v = m & 3;
        uint32_t pos = 0, neg = 0;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const bool minus = (__popc(u & q) + __popc(v & c)) & 1;
            pos |= (minus ? 0xffu : 0x01u) << (8 * c);
            neg |= (minus ? 0x01u : 0xffu) << (8 * c);
        }
        h.a[half] = pos;
        h.a[2 + half] = neg;
    }
    return h;
}

// Adds Σ|coefficients| of the blocks in columns 2q and 2q+1 (rows g and g+8,
// this lane's share) to s0 and s1.  p: the lane's predicted row word, s: the
// same row of the source.
__device__ __forceinline__ void had_mma(const HadFrag& h, uint32_t p, uint32_t s, int& s0, int& s1) {
    int d0, d1, d2, d3;
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%10, %10, %10, %10};"
        : "=r"(d0), "=r"(d1), "=r"(d2), "=r"(d3)
        : "r"(h.a[0]), "r"(h.a[1]), "r"(h.a[2]), "r"(h.a[3]), "r"(p), "r"(s), "r"(0));
    s0 += abs(d0) + abs(d2);
    s1 += abs(d1) + abs(d3);
}

}  // namespace h264a

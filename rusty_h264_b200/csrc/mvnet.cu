// mvnet.cu -- the learned motion-vector proposal network: training and
// inference kernels (bf16 tensor-core products, fp32 accumulation) and the
// C ABI around them.
//
// The network has no counterpart in the reference encoder: rusty_h264 runs
// motion_search (crates/rusty_h264-encoder/src/mb16.rs:2433) on every MB.
// Here a small conv net looks at an MB's co-located 48x48 regions of the
// current and reference frames plus three neighbour MVs and proposes the 8
// most likely full-pel MVs; h264a_me_frames_learned prices them with the
// search's exact integer cost and refines the best one with the reference's
// own sub-pel refinement (motion_search with a start vector).
//
// Network (per MB):  X0 48x48x2 -> conv1 3x3/2 -> 24x24x16 -> conv2 3x3/2 ->
// 12x12x32 -> conv3 3x3/2 -> 6x6x32 -> [1152 features | 6 MV features | 10
// zeros] = 1168 -> FC1 -> 256 -> head -> 296 logits (289 classes: full-pel
// offsets dx, dy in -8..8, class (dy+8)*17 + dx+8).  ReLU after every layer
// but the head.  Activations are stored as bf16 (NHWC), every product runs on
// the tensor cores (tcgen05.mma, bf16 operands, fp32 accumulators in tensor
// memory).
//
// Every layer is one implicit GEMM: C[M][N] = sum_k A[m][k] B[k][n], with A
// and B gathered on the fly by a functor (im2col of a stride-2 3x3 window, a
// transposed view of a weight or activation tensor, ...) and an epilogue
// functor (bias + ReLU + bf16 store, ReLU-mask + bf16 store, or an fp32
// atomic add for weight gradients, whose K dimension -- the batch times the
// output positions -- is split over CTAs).  Every gather moves 16 bytes: the
// weight gradients' operands are staged as they lie in memory, M- and N-major
// (the tensor core transposes), and the data gradients read weights that
// prep_kernel has transposed.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "h264a_device.cuh"
#include "h264accel_internal.h"

namespace h264a {
namespace mvnet {

// ---- shapes and the flat parameter vector --------------------------------
constexpr int NCLS = 289, HEAD_N = 296, FEAT = 1168, HID = 256, CONVF = 1152;
constexpr int O_W1 = 0, N_W1 = 16 * 9 * 2;
constexpr int O_B1 = O_W1 + N_W1;
constexpr int O_W2 = O_B1 + 16, N_W2 = 32 * 9 * 16;
constexpr int O_B2 = O_W2 + N_W2;
constexpr int O_W3 = O_B2 + 32, N_W3 = 32 * 9 * 32;
constexpr int O_B3 = O_W3 + N_W3;
constexpr int O_W4 = O_B3 + 32, N_W4 = HID * FEAT;
constexpr int O_B4 = O_W4 + N_W4;
constexpr int O_W5 = O_B4 + HID, N_W5 = HEAD_N * HID;
constexpr int O_B5 = O_W5 + N_W5;
constexpr int NPARAMS = O_B5 + HEAD_N;
static_assert(NPARAMS == H264A_MVNET_NPARAMS, "parameter count");
static_assert((O_W1 | O_W2 | O_W3 | O_W4 | O_W5) % 2 == 0, "weights start on bf16 pairs");

typedef uint16_t bf16_t;  // raw bf16 bits

__device__ __forceinline__ bf16_t f2bf(float f) {  // round to nearest even
    uint32_t u = __float_as_uint(f);
    u += 0x7fffu + ((u >> 16) & 1u);
    return bf16_t(u >> 16);
}
__device__ __forceinline__ float bf2f(bf16_t b) { return __uint_as_float(uint32_t(b) << 16); }
__device__ __forceinline__ uint32_t pack2(bf16_t lo, bf16_t hi) { return uint32_t(lo) | (uint32_t(hi) << 16); }
__device__ __forceinline__ uint32_t ld_pair(const bf16_t* p) { return *reinterpret_cast<const uint32_t*>(p); }
__device__ __forceinline__ uint4 ld8(const bf16_t* p) { return *reinterpret_cast<const uint4*>(p); }
// 8 values (bias added, ReLU) rounded to bf16 and stored as one 16-byte word
__device__ __forceinline__ void st8_relu(bf16_t* dst, const float* v, const bf16_t* bias) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; i++)
        w[i] = pack2(f2bf(fmaxf(v[2 * i] + bf2f(bias[2 * i]), 0.f)), f2bf(fmaxf(v[2 * i + 1] + bf2f(bias[2 * i + 1]), 0.f)));
    *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
}

// ---- a batch: frame pairs of one geometry, every MB a sample ---------------
// Trunk maps (NHWC bf16): A1 (ch/2)x(cw/2)x16, A2 (ch/4)x(cw/4)x32, A3
// (ch/8)x(cw/8)x32 per pair; samples are the pairs' MBs, pair-major, raster
// order within a pair.
struct Geo {
    const h264a_mvnet_pair* pairs;
    int P, cw, ch;
    int H1, W1, H2, W2, H3, W3;
    int mb_w, mb_h, nmb;
    const int16_t* nmv;     // 6 per sample
    const int16_t* labels;  // 1 per sample (training)
};

// X0 pair (reference, current) at pixel (iy, ix) of pair b; zero outside the
// frame (the conv's padding).
__device__ __forceinline__ uint32_t x0_pair(const Geo& g, int b, int iy, int ix) {
    if (iy < 0 || iy >= g.ch || ix < 0 || ix >= g.cw) return 0u;
    const h264a_mvnet_pair p = g.pairs[b];
    const long long o = (long long)iy * g.cw + ix;
    const float r = (float(p.d_ref[o]) - 128.f) * (1.f / 64.f), c = (float(p.d_cur[o]) - 128.f) * (1.f / 64.f);
    return pack2(f2bf(r), f2bf(c));  // exact: k/64 with |k| <= 128
}
__device__ __forceinline__ bf16_t mv_feat(const Geo& g, int m, int i) {
    const int v = min(max(int(g.nmv[6LL * m + i]), -128), 128);
    return f2bf(float(v) * (1.f / 64.f));  // exact
}

// ---- the tcgen05 GEMM: 128 x BN tiles, accumulators in tensor memory --------
// The GEMM of every forward layer and data gradient, C[M][N] = sum_k A[m][k]
// B[k][n], on the sm_100 tensor cores: per 64-wide K step all 256 threads
// gather the A (128 x 64) and B (BN x 64) tiles into one of two shared-memory
// stages, one thread issues four tcgen05.mma (M 128, N BN, K 16, bf16 in, fp32
// accumulated in tensor memory) and commits them to the stage's mbarrier, and
// the gathers of the next step overlap them.  The epilogue reads the accumulator rows with
// tcgen05.ld: warp w may read tensor-memory lanes 32(w % 4) .. +31 (its tile
// rows), warps w and w + 4 taking half of the columns each.
constexpr int TC_BM = 128, TC_BK = 64, TC_THREADS = 256;

template <int BN>
constexpr int tc_cols() {
    return BN <= 32 ? 32 : (BN <= 64 ? 64 : (BN <= 128 ? 128 : 256));
}

// A K-major operand tile of R rows x 64 k (bf16) in the canonical
// no-swizzle UMMA layout: 8x8 core matrices of 128 contiguous bytes (8 rows
// of 16 bytes), the eight k-chunks of an 8-row group 128 bytes apart (the
// leading byte offset) and the groups 1024 bytes apart (the stride byte
// offset).  Byte offset of (row, k-chunk):
__device__ __forceinline__ uint32_t tc_off(int row, int chunk) {
    return uint32_t(((row >> 3) * 8 + chunk) * 128 + (row & 7) * 16);
}
// The shared-memory matrix descriptor of such a tile from shared address a:
// start >> 4 (bits 0-13), leading byte offset 128 >> 4 (16-29), stride byte
// offset 1024 >> 4 (32-45), descriptor version 1 (46-47), base offset 0,
// layout SWIZZLE_NONE (61-63).
__device__ __forceinline__ uint64_t tc_sdesc(uint32_t a) {
    return uint64_t((a >> 4) & 0x3fffu) | (uint64_t(128 >> 4) << 16) | (uint64_t(1024 >> 4) << 32) | (1ull << 46);
}
// The instruction descriptor of kind::f16: fp32 accumulator (bits 4-5 = 1),
// A and B bf16 (7-9 = 1, 10-12 = 1), both K-major (15, 16 = 0), N >> 3
// (17-22), M >> 4 (24-28).
template <int BN>
constexpr uint32_t tc_idesc() {
    return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(BN >> 3) << 17) | (uint32_t(TC_BM >> 4) << 24);
}

__device__ __forceinline__ uint32_t tc_smem_u32(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }

// Waits (bounded) for phase `parity` of an mbarrier; on timeout records 4 in
// status and keeps waiting up to twice as long, so that no tensor-core work
// is left reading a stage or writing tensor memory.
__device__ __forceinline__ void tc_wait(uint32_t bar, uint32_t parity, int* status) {
    constexpr int kLimit = 1 << 22;
    for (int it = 0; !mbar_try_wait(bar, parity); it++) {
        if (it == kLimit && status != nullptr) atomicCAS(status, 0, 4);
        if (it >= 2 * kLimit) break;
    }
}

// An Op gathers 8 consecutive k at once (op.a8(row, k), op.b8(k, n): 16 bytes,
// k a multiple of 8, zero past its tensor) and stores 8 consecutive n
// (op.store8(row, m, n, v)).  Its `Row` is what its gathers need of output row
// m (sample, position, base offset), made once per CTA row by op.row(m), so
// the per-chunk gathers divide by no runtime size.  K and N are multiples of 8.
template <int BN, class Op>
__global__ void __launch_bounds__(TC_THREADS) gemm_tc_kernel(const Op op, int M, int N, int K, int* status) {
    static_assert(BN % 16 == 0 && BN >= 16 && BN <= 256, "tcgen05 N for M = 128");
    constexpr int A_BYTES = TC_BM * TC_BK * 2, B_BYTES = BN * TC_BK * 2, STAGE = A_BYTES + B_BYTES;
    constexpr int NCOL = tc_cols<BN>();
    constexpr uint32_t IDESC = tc_idesc<BN>();
    extern __shared__ __align__(128) uint8_t tc_smem[];
    __shared__ __align__(8) unsigned long long tc_bar[2];
    __shared__ uint32_t tc_tmem;
    __shared__ typename Op::Row tc_rows[TC_BM];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * TC_BM, n0 = blockIdx.y * BN;
    for (int i = tid; i < TC_BM; i += TC_THREADS) tc_rows[i] = op.row(min(m0 + i, M - 1));  // read after the __syncthreads below
    const int kb = 0, ke = K;
    const uint32_t sbase = tc_smem_u32(tc_smem), bar0 = tc_smem_u32(&tc_bar[0]);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(&tc_tmem)),
                     "r"(NCOL));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        mbar_init(bar0, 1);
        mbar_init(bar0 + 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tc_tmem;
    const int nk = ke > kb ? (ke - kb + TC_BK - 1) / TC_BK : 0;
    for (int it = 0; it < nk; it++) {
        const int st = it & 1;
        const int k0 = kb + it * TC_BK;
        const uint32_t sa = sbase + uint32_t(st * STAGE), sb = sa + A_BYTES;
        // consecutive threads fill consecutive 16-byte rows of a core
        // matrix, so a warp's stores meet no bank twice
        {
            // the step's gathers are issued before waiting for the stage, so
            // they overlap the MMAs still reading it
            constexpr int AQ = TC_BM * 8 / TC_THREADS, BQ = (BN * 8 + TC_THREADS - 1) / TC_THREADS;
            uint4 va[AQ], vb[BQ];
#pragma unroll
            for (int j = 0; j < AQ; j++) {
                const int q = tid + j * TC_THREADS;
                const int row = ((q >> 6) << 3) | (q & 7), c = (q >> 3) & 7, m = m0 + row, k = k0 + 8 * c;
                va[j] = (m < M && k < ke) ? op.a8(tc_rows[row], k) : make_uint4(0u, 0u, 0u, 0u);
            }
#pragma unroll
            for (int j = 0; j < BQ; j++) {
                const int q = tid + j * TC_THREADS;
                const int row = ((q >> 6) << 3) | (q & 7), c = (q >> 3) & 7, n = n0 + row, k = k0 + 8 * c;
                vb[j] = (q < BN * 8 && n < N && k < ke) ? op.b8(k, n) : make_uint4(0u, 0u, 0u, 0u);
            }
            // the stage's previous MMAs (step it - 2) have read it
            if (it >= 2) tc_wait(bar0 + 8 * st, uint32_t((it - 2) >> 1) & 1u, status);
#pragma unroll
            for (int j = 0; j < AQ; j++) {
                const int q = tid + j * TC_THREADS, row = ((q >> 6) << 3) | (q & 7), c = (q >> 3) & 7;
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sa + tc_off(row, c)), "r"(va[j].x),
                             "r"(va[j].y), "r"(va[j].z), "r"(va[j].w)
                             : "memory");
            }
#pragma unroll
            for (int j = 0; j < BQ; j++) {
                const int q = tid + j * TC_THREADS, row = ((q >> 6) << 3) | (q & 7), c = (q >> 3) & 7;
                if (q < BN * 8)
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sb + tc_off(row, c)), "r"(vb[j].x),
                                 "r"(vb[j].y), "r"(vb[j].z), "r"(vb[j].w)
                                 : "memory");
            }
        }
        // the tiles' generic-proxy writes, visible to the tensor cores
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int j = 0; j < TC_BK / 16; j++) {
                const uint64_t da = tc_sdesc(sa + 256u * j), db = tc_sdesc(sb + 256u * j);
                const uint32_t acc = (it > 0 || j > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(tmem),
                    "l"(da), "l"(db), "r"(IDESC), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar0 +
                                                                                                          8 * st)
                         : "memory");
        }
    }
    if (nk > 0) {
        // the last step's commit completes after every earlier MMA
        tc_wait(bar0 + 8 * ((nk - 1) & 1), uint32_t((nk - 1) >> 1) & 1u, status);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int row = m0 + (warp & 3) * 32 + lane;
        const uint32_t taddr = tmem + (uint32_t((warp & 3) * 32) << 16);
        const int cb = (warp >> 2) * (BN / 2);
#pragma unroll 1
        for (int c0 = cb; c0 < cb + BN / 2; c0 += 8) {
            uint32_t r[8];
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                         : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                           "=r"(r[7])
                         : "r"(taddr + uint32_t(c0)));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (row < M && n0 + c0 < N) {
                float f[8];
#pragma unroll
                for (int i = 0; i < 8; i++) f[i] = __uint_as_float(r[i]);
                op.store8(tc_rows[row - m0], row, n0 + c0, f);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NCOL));
}

// ---- the layers as GEMM operands --------------------------------------------
struct Bufs {
    const bf16_t* w;  // bf16 parameters
    float* grad;      // fp32 parameter gradients (accumulated)
    bf16_t *a1, *a2, *a3, *h, *dl, *dh, *df, *da3, *da2, *da1;
    const bf16_t *w4t, *w5t, *wd3, *wd2;  // prep_kernel's rearranged weights
    float* logits;
};

// conv1 forward: M = P*H1*W1, N = 16, K = 18 (padded to 32)
struct Conv1Fwd {
    Geo g; Bufs z;
    __device__ uint32_t b(int k, int n) const { return k < 18 ? ld_pair(z.w + O_W1 + n * 18 + k) : 0u; }
    struct Row {
        int b, y0, x0;  // pair, top-left input pixel of the 3x3 window
    };
    __device__ Row row(int m) const {
        const int OHW = g.H1 * g.W1;
        const int b = m / OHW, r = m - b * OHW, oy = r / g.W1, ox = r - oy * g.W1;
        return Row{b, 2 * oy - 1, 2 * ox - 1};
    }
    __device__ uint4 a8(const Row& w, int k) const {
        uint32_t v[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int tap = (k >> 1) + i, ky = (tap * 11) >> 5, kx = tap - ky * 3;  // ky = tap / 3 for tap < 9
            v[i] = tap < 9 ? x0_pair(g, w.b, w.y0 + ky, w.x0 + kx) : 0u;
        }
        return make_uint4(v[0], v[1], v[2], v[3]);
    }
    __device__ uint4 b8(int k, int n) const {
        uint32_t v[4];
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = b(k + 2 * i, n);
        return make_uint4(v[0], v[1], v[2], v[3]);
    }
    __device__ void store8(const Row&, int m, int n, const float* v) const { st8_relu(z.a1 + (long long)m * 16 + n, v, z.w + O_B1 + n); }
};
// conv2 / conv3 forward: im2col of the previous map
template <int C, int OW, int OB, int WHICH>
struct ConvFwd {
    Geo g; Bufs z;
    // k a multiple of 8 (C = 16 or 32): the chunk is 8 channels of one tap,
    // 16 contiguous bytes of the NHWC map
    struct Row {
        long long base;  // element offset of input pixel (y0, x0), channel 0 (may lie outside the map)
        int y0, x0;
    };
    __device__ Row row(int m) const {
        const int H = WHICH == 2 ? g.H1 : g.H2, W = WHICH == 2 ? g.W1 : g.W2;
        const int ow = W >> 1, ohw = (H >> 1) * ow;
        const int b = m / ohw, r = m - b * ohw, oy = r / ow, ox = r - oy * ow;
        return Row{((long long)(b * H + 2 * oy - 1) * W + 2 * ox - 1) * C, 2 * oy - 1, 2 * ox - 1};
    }
    __device__ uint4 a8(const Row& w, int k) const {
        const int H = WHICH == 2 ? g.H1 : g.H2, W = WHICH == 2 ? g.W1 : g.W2;
        const int tap = k / C, ci = k - tap * C, ky = (tap * 11) >> 5, kx = tap - ky * 3;
        const int iy = w.y0 + ky, ix = w.x0 + kx;
        if (iy < 0 || iy >= H || ix < 0 || ix >= W) return make_uint4(0u, 0u, 0u, 0u);
        return ld8((WHICH == 2 ? z.a1 : z.a2) + w.base + (long long)(ky * W + kx) * C + ci);
    }
    __device__ uint4 b8(int k, int n) const { return ld8(z.w + OW + n * 9 * C + k); }
    __device__ void store8(const Row&, int m, int n, const float* v) const {
        st8_relu((WHICH == 2 ? z.a2 : z.a3) + (long long)m * 32 + n, v, z.w + OB + n);
    }
};
using Conv2Fwd = ConvFwd<16, O_W2, O_B2, 2>;
using Conv3Fwd = ConvFwd<32, O_W3, O_B3, 3>;

struct Fc1Fwd {
    Geo g; Bufs z;
    // k < 1152, a multiple of 8: 8 channels of one crop cell, 16 contiguous
    // bytes of A3 (its MB's 6x6-cell crop, zero outside the map); then the 6
    // neighbour-MV features and zeros
    struct Row {
        long long base;  // element offset of the crop's top-left cell (y0, x0), channel 0
        int m, y0, x0;
    };
    __device__ Row row(int m) const {
        const int b = m / g.nmb, r = m - b * g.nmb, mby = r / g.mb_w, mbx = r - mby * g.mb_w;
        const int y0 = 2 * mby - 2, x0 = 2 * mbx - 2;
        return Row{((long long)(b * g.H3 + y0) * g.W3 + x0) * 32, m, y0, x0};
    }
    __device__ uint4 a8(const Row& w, int k) const {
        if (k < CONVF) {
            const int cy = k / 192, rem = k - cy * 192, cx = rem >> 5, c = rem & 31;
            const int y = w.y0 + cy, x = w.x0 + cx;
            if (y < 0 || y >= g.H3 || x < 0 || x >= g.W3) return make_uint4(0u, 0u, 0u, 0u);
            return ld8(z.a3 + w.base + (long long)(cy * g.W3 + cx) * 32 + c);
        }
        if (k == CONVF)
            return make_uint4(pack2(mv_feat(g, w.m, 0), mv_feat(g, w.m, 1)), pack2(mv_feat(g, w.m, 2), mv_feat(g, w.m, 3)),
                              pack2(mv_feat(g, w.m, 4), mv_feat(g, w.m, 5)), 0u);
        return make_uint4(0u, 0u, 0u, 0u);
    }
    __device__ uint4 b8(int k, int n) const { return ld8(z.w + O_W4 + (long long)n * FEAT + k); }
    __device__ void store8(const Row&, int m, int n, const float* v) const { st8_relu(z.h + (long long)m * HID + n, v, z.w + O_B4 + n); }
};
struct HeadFwd {
    Bufs z;
    using Row = int;
    __device__ Row row(int m) const { return m; }
    __device__ uint4 a8(Row m, int k) const { return ld8(z.h + (long long)m * HID + k); }
    __device__ uint4 b8(int k, int n) const { return ld8(z.w + O_W5 + n * HID + k); }
    __device__ void store8(const Row&, int m, int n, const float* v) const {
        float4* d = reinterpret_cast<float4*>(z.logits + (long long)m * HEAD_N + n);
        const bf16_t* bias = z.w + O_B5 + n;
        d[0] = make_float4(v[0] + bf2f(bias[0]), v[1] + bf2f(bias[1]), v[2] + bf2f(bias[2]), v[3] + bf2f(bias[3]));
        d[1] = make_float4(v[4] + bf2f(bias[4]), v[5] + bf2f(bias[5]), v[6] + bf2f(bias[6]), v[7] + bf2f(bias[7]));
    }
};

// ---- data gradients ---------------------------------------------------------
// The weights as the data gradients' GEMMs read them, K contiguous: w5t
// [256][296] and w4t [1152][256] transposed; wd3 [128][128] and wd2 [64][128]
// the stride-2 transposed convolutions over a 2x2 block of input pixels: row
// n = (2 py + px) * C + ci of input pixel (2a + py, 2b + px), column k =
// (2 ny + nx) * 32 + co of output position (a + ny, b + nx), the tap
// (py + 1 - 2 ny, px + 1 - 2 nx) or zero.  (A GEMM over input pixels and all
// nine taps reads four times as much and multiplies mostly zeros: 970 us
// against 83 for conv2's on four 1080p pairs.)
constexpr int N_W4T = CONVF * HID, N_W5T = HID * HEAD_N, N_WD3 = 128 * 128, N_WD2 = 64 * 128;
constexpr int N_PREP = N_W4T + N_W5T + N_WD3 + N_WD2;
__device__ __forceinline__ bf16_t wd_at(const bf16_t* w, int C, int i) {  // w [32][9][C]
    const int n = i >> 7, k = i & 127, par = n / C, ci = n - par * C, nb = k >> 5, co = k & 31;
    const int ky = (par >> 1) + 1 - 2 * (nb >> 1), kx = (par & 1) + 1 - 2 * (nb & 1);
    return ky < 0 || kx < 0 ? bf16_t(0) : w[(co * 9 + ky * 3 + kx) * C + ci];
}
__global__ void prep_kernel(const bf16_t* __restrict__ w, bf16_t* __restrict__ out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < N_W4T) {
        out[i] = w[O_W4 + (i % HID) * FEAT + i / HID];
        return;
    }
    i -= N_W4T;
    if (i < N_W5T) {
        out[N_W4T + i] = w[O_W5 + (i % HEAD_N) * HID + i / HEAD_N];
        return;
    }
    i -= N_W5T;
    if (i < N_WD3) {
        out[N_W4T + N_W5T + i] = wd_at(w + O_W3, 32, i);
        return;
    }
    i -= N_WD3;
    if (i < N_WD2) out[N_W4T + N_W5T + N_WD3 + i] = wd_at(w + O_W2, 16, i);
}

__device__ __forceinline__ uint32_t mask_pair(uint32_t act, uint32_t v) {  // bf16 pair v where the activation is not zero
    return v & ((act & 0xffffu ? 0xffffu : 0u) | (act & 0xffff0000u ? 0xffff0000u : 0u));
}
// 8 values rounded to bf16, stored as one 16-byte word; with act, zero where
// the activation there is (ReLU's gradient)
__device__ __forceinline__ void st8_mask(bf16_t* dst, const float* v, const bf16_t* act) {
    uint4 w = make_uint4(pack2(f2bf(v[0]), f2bf(v[1])), pack2(f2bf(v[2]), f2bf(v[3])), pack2(f2bf(v[4]), f2bf(v[5])),
                         pack2(f2bf(v[6]), f2bf(v[7])));
    if (act != nullptr) {
        const uint4 a = ld8(act);
        w = make_uint4(mask_pair(a.x, w.x), mask_pair(a.y, w.y), mask_pair(a.z, w.z), mask_pair(a.w, w.w));
    }
    *reinterpret_cast<uint4*>(dst) = w;
}

struct HeadBwdData {  // dh = relu'(h) * (dl W5): M = B, N = 256, K = 296
    Bufs z;
    using Row = int;
    __device__ Row row(int m) const { return m; }
    __device__ uint4 a8(Row m, int k) const { return ld8(z.dl + (long long)m * HEAD_N + k); }
    __device__ uint4 b8(int k, int n) const { return ld8(z.w5t + n * HEAD_N + k); }
    __device__ void store8(const Row&, int m, int n, const float* v) const {
        const long long o = (long long)m * HID + n;
        st8_mask(z.dh + o, v, z.h + o);
    }
};
struct Fc1BwdData {  // df = (dh W4)[:, :1152]: M = B, N = 1152, K = 256
    Bufs z;
    using Row = int;
    __device__ Row row(int m) const { return m; }
    __device__ uint4 a8(Row m, int k) const { return ld8(z.dh + (long long)m * HID + k); }
    __device__ uint4 b8(int k, int n) const { return ld8(z.w4t + n * HID + k); }
    __device__ void store8(const Row&, int m, int n, const float* v) const { st8_mask(z.df + (long long)m * CONVF + n, v, nullptr); }
};
// conv input gradient: M = pairs x output positions (2x2 input blocks),
// N = 4 C, K = 4 x 32 (see prep_kernel); WHICH 3: da3 -> da2, 2: da2 -> da1
template <int C, int WHICH>
struct ConvBwdData {
    Geo g; Bufs z;
    struct Row {
        long long in, out;  // element offsets of dy position (a, b) and of input pixel (2a, 2b)
        bool down, right;   // (a + 1, .) and (., b + 1) lie inside the map
    };
    __device__ Row row(int m) const {
        const int OH = WHICH == 3 ? g.H3 : g.H2, OW = WHICH == 3 ? g.W3 : g.W2;
        const int ohw = OH * OW, b = m / ohw, r = m - b * ohw, a = r / OW, x = r - a * OW;
        return Row{(long long)m * 32, ((long long)(b * 2 * OH + 2 * a) * (2 * OW) + 2 * x) * C, a + 1 < OH, x + 1 < OW};
    }
    __device__ uint4 a8(const Row& w, int k) const {
        const int nb = k >> 5, OW = WHICH == 3 ? g.W3 : g.W2;
        if (((nb & 2) && !w.down) || ((nb & 1) && !w.right)) return make_uint4(0u, 0u, 0u, 0u);
        return ld8((WHICH == 3 ? z.da3 : z.da2) + w.in + ((nb & 2) ? OW * 32 : 0) + ((nb & 1) ? 32 : 0) + (k & 31));
    }
    __device__ uint4 b8(int k, int n) const { return ld8((WHICH == 3 ? z.wd3 : z.wd2) + n * 128 + k); }
    __device__ void store8(const Row& w, int, int n, const float* v) const {
        const int par = n / C, ci = n - par * C, W = WHICH == 3 ? g.W2 : g.W1;
        const long long o = w.out + ((par & 2) ? W * C : 0) + ((par & 1) ? C : 0) + ci;
        st8_mask((WHICH == 3 ? z.da2 : z.da1) + o, v, (WHICH == 3 ? z.a2 : z.a1) + o);
    }
};

// ---- weight gradients ---------------------------------------------------------
// dW[i][j] = sum_m dy[m][i] x[m][j] over the rows m (samples, or the pairs'
// map positions), split over CTAs: M = output channels, N = input columns,
// K = rows.  Both operands lie row by row in memory, that is M- and N-major:
// each thread moves 16-byte chunks (8 columns of one row) as they are into the
// M/N-major no-swizzle layout -- 8 (M or N) x 8 (K) core matrices of 128 bytes,
// a row of K each 16 bytes, the KS/8 K-blocks of an 8-column block 128 bytes
// apart (the leading byte offset) and the blocks KS * 16 apart (the stride byte
// offset) -- and the tensor core transposes.  (Gathering K-major tiles took
// two 2-byte loads per pair: 791 us for FC1's gradient on four 1080p pairs,
// 32,640 samples, against 112 this way; 577 against 58 for conv2's.)  A tile holds only the M - m0 columns there are: the MMA's
// further rows read whatever follows in shared memory into accumulator rows
// that nothing reads.  The bias gradient is the sum of dy's chunks as the
// threads of the first N tile pass them on.
//   Op: rows K; RowW row(m); uint4 a8(row, i), b8(row, j); grad offsets out
// (with leading dimension ld) and bias; n_real columns are stored.
template <int KS>
constexpr uint64_t wg_sdesc_hi() {
    return (uint64_t(128 >> 4) << 16) | (uint64_t((KS * 16) >> 4) << 32) | (1ull << 46);
}
__device__ __forceinline__ void red_add_v4(float* p, const float* v) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3])
                 : "memory");
}

template <int BN, int KS, int AQ, class Op>  // AQ: 8-column chunks of A per thread and step
__global__ void __launch_bounds__(TC_THREADS) wgrad_tc_kernel(const Op op, int M, int N, int K, int kchunk, int* status) {
    static_assert(BN % 16 == 0 && BN >= 16 && BN <= 256 && KS % 16 == 0 && TC_THREADS % KS == 0, "tile shape");
    constexpr int GR = TC_THREADS / KS;          // threads per row
    constexpr int BLK = KS * 16;                 // bytes of one 8-column block of a tile
    constexpr int BQ = (BN / 8 + GR - 1) / GR, A_BYTES = AQ * GR * BLK, STAGE = A_BYTES + (BN / 8) * BLK;
    constexpr int NCOL = tc_cols<BN>();
    constexpr uint32_t IDESC = tc_idesc<BN>() | (1u << 15) | (1u << 16);  // A and B transposed (M/N-major)
    extern __shared__ __align__(128) uint8_t tc_smem[];
    __shared__ __align__(8) unsigned long long tc_bar[2];
    __shared__ uint32_t tc_tmem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * TC_BM, n0 = blockIdx.y * BN;
    const int mblk = min(TC_BM, M - m0) / 8, nblk = min(BN, N - n0) / 8;
    const int kb = blockIdx.z * kchunk, ke = min(K, kb + kchunk);
    const uint32_t sbase = tc_smem_u32(tc_smem), bar0 = tc_smem_u32(&tc_bar[0]);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(&tc_tmem)),
                     "r"(NCOL));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        mbar_init(bar0, 1);
        mbar_init(bar0 + 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tc_tmem;
    const int p = tid % KS, c0 = tid / KS;  // the thread's row of a step and its first chunk
    const uint32_t off = uint32_t((p >> 3) * 128 + (p & 7) * 16);
    const bool with_bias = blockIdx.y == 0;
    float bias[AQ][8];
#pragma unroll
    for (int j = 0; j < AQ; j++)
#pragma unroll
        for (int i = 0; i < 8; i++) bias[j][i] = 0.f;
    const int nk = ke > kb ? (ke - kb + KS - 1) / KS : 0;
    for (int it = 0; it < nk; it++) {
        const int st = it & 1, m = kb + it * KS + p;
        const uint32_t sa = sbase + uint32_t(st * STAGE), sb = sa + A_BYTES;
        const bool live = m < ke;
        const typename Op::Row row = op.row(live ? m : ke - 1);
        uint4 va[AQ], vb[BQ];
#pragma unroll
        for (int j = 0; j < AQ; j++) {
            const int c = c0 + j * GR;
            va[j] = live && c < mblk ? op.a8(row, m0 + 8 * c) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int j = 0; j < BQ; j++) {
            const int c = c0 + j * GR;
            vb[j] = live && c < nblk ? op.b8(row, n0 + 8 * c) : make_uint4(0u, 0u, 0u, 0u);
        }
        if (with_bias) {
#pragma unroll
            for (int j = 0; j < AQ; j++) {
                const uint32_t w[4] = {va[j].x, va[j].y, va[j].z, va[j].w};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    bias[j][2 * i] += bf2f(bf16_t(w[i] & 0xffffu));
                    bias[j][2 * i + 1] += bf2f(bf16_t(w[i] >> 16));
                }
            }
        }
        // the stage's previous MMAs (step it - 2) have read it
        if (it >= 2) tc_wait(bar0 + 8 * st, uint32_t((it - 2) >> 1) & 1u, status);
#pragma unroll
        for (int j = 0; j < AQ; j++)
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sa + uint32_t((c0 + j * GR) * BLK) + off), "r"(va[j].x),
                         "r"(va[j].y), "r"(va[j].z), "r"(va[j].w)
                         : "memory");
#pragma unroll
        for (int j = 0; j < BQ; j++)
            if (c0 + j * GR < BN / 8)
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sb + uint32_t((c0 + j * GR) * BLK) + off),
                             "r"(vb[j].x), "r"(vb[j].y), "r"(vb[j].z), "r"(vb[j].w)
                             : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int j = 0; j < KS / 16; j++) {
                const uint64_t da = uint64_t(((sa + 256u * j) >> 4) & 0x3fffu) | wg_sdesc_hi<KS>();
                const uint64_t db = uint64_t(((sb + 256u * j) >> 4) & 0x3fffu) | wg_sdesc_hi<KS>();
                const uint32_t acc = (it > 0 || j > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(tmem),
                    "l"(da), "l"(db), "r"(IDESC), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar0 + 8 * st)
                         : "memory");
        }
    }
    if (nk > 0) {
        tc_wait(bar0 + 8 * ((nk - 1) & 1), uint32_t((nk - 1) >> 1) & 1u, status);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int row = m0 + (warp & 3) * 32 + lane;
        const uint32_t taddr = tmem + (uint32_t((warp & 3) * 32) << 16);
        const int nc = min(BN, op.n_real - n0);
        if (m0 + (warp & 3) * 32 < M) {
#pragma unroll 1
            for (int c = (warp >> 2) * 8; c < nc; c += 16) {
                uint32_t r[8];
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                               "=r"(r[7])
                             : "r"(taddr + uint32_t(c)));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (row < M) {
                    float f[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) f[i] = __uint_as_float(r[i]);
                    float* d = op.z.grad + op.out + (long long)row * op.ld + n0 + c;
                    if (op.ld % 4 == 0 && op.out % 4 == 0) {  // every column chunk is whole then
                        red_add_v4(d, f);
                        red_add_v4(d + 4, f + 4);
                    } else {
#pragma unroll
                        for (int i = 0; i < 8; i++)
                            if (c + i < nc) atomicAdd(d + i, f[i]);
                    }
                }
            }
        }
        if (with_bias) {
#pragma unroll
            for (int j = 0; j < AQ; j++)
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    float v = bias[j][i];
                    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                    if (lane == 0 && c0 + j * GR < mblk) atomicAdd(op.z.grad + op.bias + m0 + 8 * (c0 + j * GR) + i, v);
                }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NCOL));
}

struct HeadBwdW {  // M = 296, N = 256, K = B
    Bufs z;
    static constexpr int out = O_W5, ld = HID, bias = O_B5, n_real = HID;
    using Row = int;
    __device__ Row row(int m) const { return m; }
    __device__ uint4 a8(Row m, int i) const { return ld8(z.dl + (long long)m * HEAD_N + i); }
    __device__ uint4 b8(Row m, int j) const { return ld8(z.h + (long long)m * HID + j); }
};
struct Fc1BwdW {  // M = 256, N = 1168, K = B
    Geo g; Bufs z;
    static constexpr int out = O_W4, ld = FEAT, bias = O_B4, n_real = FEAT;
    using Row = Fc1Fwd::Row;
    __device__ Row row(int m) const { return Fc1Fwd{g, z}.row(m); }
    __device__ uint4 a8(const Row& w, int i) const { return ld8(z.dh + (long long)w.m * HID + i); }
    __device__ uint4 b8(const Row& w, int j) const { return Fc1Fwd{g, z}.a8(w, j); }
};
// conv weight gradient: M = CO, N = 9 C, K = pairs x output positions
template <class Fwd, int C, int CO, int OW, int OB, int WHICH>
struct ConvBwdW {
    Geo g; Bufs z;
    static constexpr int out = OW, ld = 9 * C, bias = OB, n_real = 9 * C;
    struct Row {
        typename Fwd::Row r;
        int m;
    };
    __device__ Row row(int m) const { return Row{Fwd{g, z}.row(m), m}; }
    __device__ uint4 a8(const Row& w, int i) const {
        return ld8((WHICH == 1 ? z.da1 : (WHICH == 2 ? z.da2 : z.da3)) + (long long)w.m * CO + i);
    }
    __device__ uint4 b8(const Row& w, int j) const { return Fwd{g, z}.a8(w.r, j); }
};
using Conv1BwdW = ConvBwdW<Conv1Fwd, 2, 16, O_W1, O_B1, 1>;
using Conv2BwdW = ConvBwdW<Conv2Fwd, 16, 32, O_W2, O_B2, 2>;
using Conv3BwdW = ConvBwdW<Conv3Fwd, 32, 32, O_W3, O_B3, 3>;

// da3 = relu'(a3) * (sum of the crop gradients of the up to 9 MBs whose 6x6
// crop holds the cell): one thread per (pair, cell, 8 channels).
__global__ void uncrop_kernel(const Geo g, const bf16_t* __restrict__ df, const bf16_t* __restrict__ a3,
                              bf16_t* __restrict__ da3) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long total = (long long)g.P * g.H3 * g.W3 * 4;
    if (i >= total) return;
    const int c = int(i & 3) * 8;
    const int cell = int(i >> 2), hw = g.H3 * g.W3;
    const int b = cell / hw, r = cell - b * hw, y = r / g.W3, x = r - y * g.W3;
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const int ylo = max(0, (y - 2) >> 1), yhi = min(g.mb_h - 1, (y + 2) >> 1);
    const int xlo = max(0, (x - 2) >> 1), xhi = min(g.mb_w - 1, (x + 2) >> 1);
    for (int mby = ylo; mby <= yhi; mby++) {
        const int cy = y - 2 * mby + 2;
        if (cy < 0 || cy >= 6) continue;
        for (int mbx = xlo; mbx <= xhi; mbx++) {
            const int cx = x - 2 * mbx + 2;
            if (cx < 0 || cx >= 6) continue;
            const long long m = (long long)b * g.nmb + mby * g.mb_w + mbx;
            const uint4 v = ld8(df + m * CONVF + cy * 192 + cx * 32 + c);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                s[2 * k] += bf2f(bf16_t(w[k] & 0xffffu));
                s[2 * k + 1] += bf2f(bf16_t(w[k] >> 16));
            }
        }
    }
    const long long o = (long long)cell * 32 + c;
    st8_mask(da3 + o, s, a3 + o);
}

// ---- loss, proposals, optimiser -------------------------------------------------
// One warp per sample: softmax over the 289 classes, the sample's share of the
// mean cross-entropy (atomically summed into *loss) and dl = (p - onehot) / B
// in bf16 (zero for the 7 padding logits).
// The row stays in registers (HEAD_N = 296: ten values a lane).
__global__ void loss_kernel(const float* __restrict__ logits, const int16_t* __restrict__ labels, int B,
                            bf16_t* __restrict__ dl, float* __restrict__ loss) {
    __shared__ float part[8];
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    float mine = 0.f;
    if (w < B) {
        const float* z = logits + (long long)w * HEAD_N;
        float v[10], mx = -INFINITY;
#pragma unroll
        for (int i = 0; i < 10; i++) {
            const int c = lane + 32 * i;
            v[i] = c < NCLS ? z[c] : -INFINITY;
            mx = fmaxf(mx, v[i]);
        }
        for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const int label = min(max(int(labels[w]), 0), NCLS - 1);
        const float zl = z[label];
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < 10; i++) {
            v[i] = lane + 32 * i < NCLS ? expf(v[i] - mx) : 0.f;
            s += v[i];
        }
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const float inv = 1.f / s, scale = 1.f / float(B);
#pragma unroll
        for (int i = 0; i < 10; i++) {
            const int c = lane + 32 * i;
            if (c < HEAD_N) dl[(long long)w * HEAD_N + c] = f2bf(c < NCLS ? (v[i] * inv - (c == label ? 1.f : 0.f)) * scale : 0.f);
        }
        mine = (logf(s) + mx - zl) * scale;
    }
    if (lane == 0) part[threadIdx.x >> 5] = mine;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int i = 0; i < int(blockDim.x >> 5); i++) t += part[i];
        atomicAdd(loss, t);
    }
}

// One warp per sample: the 8 largest logits (ties to the lower class) as
// quarter-pel MVs, 16 i32 per sample; sample i of a batch is MB mb0 + i of
// the frame whose proposals out points to.
// A frame of a propose batch: its guide MVs (may be null) and its proposals.
struct PropFrame {
    const int32_t* guide;
    int32_t* props;
};

__device__ __forceinline__ void top8_one(const float* __restrict__ z, int32_t* __restrict__ o);

// top8 of every MB of P frames of nmb MBs each, into each frame's proposals
__global__ void top8_frames_kernel(const float* __restrict__ logits, int P, int nmb, const PropFrame* __restrict__ fr) {
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= (long long)P * nmb) return;
    const int k = int(w / nmb), m = int(w - (long long)k * nmb);
    top8_one(logits + w * HEAD_N, fr[k].props + 16LL * m);
}

__device__ __forceinline__ void top8_one(const float* __restrict__ z, int32_t* __restrict__ o) {
    const int lane = threadIdx.x & 31;
    float v[10];
#pragma unroll
    for (int i = 0; i < 10; i++) {
        const int c = lane + 32 * i;
        v[i] = c < NCLS ? z[c] : -INFINITY;
    }
    for (int r = 0; r < 8; r++) {
        float bv = -INFINITY;
        int bc = 1 << 30;
#pragma unroll
        for (int i = 0; i < 10; i++)
            if (v[i] > bv) { bv = v[i]; bc = lane + 32 * i; }
        for (int s = 16; s; s >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, s);
            const int oc = __shfl_xor_sync(0xffffffffu, bc, s);
            if (ov > bv || (ov == bv && oc < bc)) { bv = ov; bc = oc; }
        }
        if ((bc & 31) == lane) {
#pragma unroll
            for (int i = 0; i < 10; i++)
                if (lane + 32 * i == bc) v[i] = -INFINITY;
        }
        if (lane == 0) {
            o[2 * r] = 4 * (bc % 17 - 8);
            o[2 * r + 1] = 4 * (bc / 17 - 8);
        }
    }
}

__global__ void adam_kernel(float* __restrict__ master, bf16_t* __restrict__ w, const float* __restrict__ grad,
                            float* __restrict__ m1, float* __restrict__ m2, int n, float lr, float b1, float b2,
                            float c1, float c2, float eps) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float g = grad[i];
    const float a = b1 * m1[i] + (1.f - b1) * g, b = b2 * m2[i] + (1.f - b2) * g * g;
    m1[i] = a;
    m2[i] = b;
    const float nw = master[i] - lr * (a * c1) / (sqrtf(b * c2) + eps);
    master[i] = nw;
    w[i] = f2bf(nw);
}

__global__ void to_bf16_kernel(const float* __restrict__ src, bf16_t* __restrict__ dst, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = f2bf(src[i]);
}

// The neighbour MV features of every MB of the P frames of a propose batch
// (frame k's MBs at samples k * nmb ..) from their guide MVs (2 i32 per MB):
// left, top, top-right MB, zero outside the frame or when the frame has no
// guide MVs.
__global__ void guide_frames_kernel(const PropFrame* __restrict__ fr, int P, int mb_w, int mb_h,
                                    int16_t* __restrict__ nmv) {
    const int nmb = mb_w * mb_h;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)P * nmb) return;
    const int k = int(t / nmb), m = int(t - (long long)k * nmb);
    const int32_t* guide = fr[k].guide;
    const int mbx = m % mb_w, mby = m / mb_w;
    const int nb[3] = {mbx > 0 ? m - 1 : -1, mby > 0 ? m - mb_w : -1, (mby > 0 && mbx + 1 < mb_w) ? m - mb_w + 1 : -1};
    int16_t* o = nmv + 6 * t;
    for (int j = 0; j < 3; j++) {
        int vx = 0, vy = 0;
        if (guide && nb[j] >= 0) {
            vx = guide[2 * nb[j]];
            vy = guide[2 * nb[j] + 1];
        }
        o[2 * j] = int16_t(min(max(vx, -32768), 32767));
        o[2 * j + 1] = int16_t(min(max(vy, -32768), 32767));
    }
}

template <int BN, class Op>
static void gemm(const Op& op, int M, int N, int K, cudaStream_t st) {
    constexpr int smem = 2 * (TC_BM * TC_BK * 2 + BN * TC_BK * 2);
    static const bool attr_ok = [] {  // once per instantiation (the dynamic shared memory above 48 KB)
        return cudaFuncSetAttribute(gemm_tc_kernel<BN, Op>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) ==
               cudaSuccess;
    }();
    (void)attr_ok;
    dim3 grid((M + TC_BM - 1) / TC_BM, (N + BN - 1) / BN);
    gemm_tc_kernel<BN, Op><<<grid, TC_THREADS, smem, st>>>(op, M, N, K, nullptr);
}

// Weight-gradient GEMM: K split over about two CTAs per SM (what its shared
// and tensor memory hold), at least four steps each.
template <int BN, int KS, int AQ, class Op>
static void wgrad(const Op& op, int M, int N, int K, int sms, cudaStream_t st) {
    constexpr int GR = TC_THREADS / KS, BLK = KS * 16, A_BYTES = AQ * GR * BLK, STAGE = A_BYTES + (BN / 8) * BLK;
    // the MMA reads 16 blocks of A whatever there are: 16 * BLK from the last stage's start
    constexpr int smem = STAGE + (STAGE > 16 * BLK ? STAGE : 16 * BLK);
    static const bool attr_ok = [] {
        return cudaFuncSetAttribute(wgrad_tc_kernel<BN, KS, AQ, Op>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) ==
               cudaSuccess;
    }();
    (void)attr_ok;
    const int tiles = ((M + TC_BM - 1) / TC_BM) * ((N + BN - 1) / BN);
    int splits = (2 * sms + tiles - 1) / tiles;
    splits = std::max(1, std::min(splits, (K + 4 * KS - 1) / (4 * KS)));
    int kchunk = (K + splits - 1) / splits;
    kchunk = (kchunk + KS - 1) / KS * KS;
    dim3 grid((M + TC_BM - 1) / TC_BM, (N + BN - 1) / BN, (K + kchunk - 1) / kchunk);
    wgrad_tc_kernel<BN, KS, AQ, Op><<<grid, TC_THREADS, smem, st>>>(op, M, N, K, kchunk, nullptr);
}

}  // namespace mvnet
}  // namespace h264a

using namespace h264a;
using namespace h264a::mvnet;

constexpr long long MAXPIX = H264A_MVNET_MAX_PIXELS;
constexpr long long MAXS = MAXPIX / 256;  // samples (MBs) per batch

struct h264a_mvnet {
    int device = 0, sms = 0;
    float* master = nullptr;  // fp32 parameters
    bf16_t* w = nullptr;      // their bf16 copy (what the kernels read)
    float *grad = nullptr, *m1 = nullptr, *m2 = nullptr;
    long long step = 0;
    // maps, activations and gradients of one batch
    bf16_t *a1 = nullptr, *a2 = nullptr, *a3 = nullptr, *h = nullptr, *dl = nullptr, *dh = nullptr, *df = nullptr;
    bf16_t *da3 = nullptr, *da2 = nullptr, *da1 = nullptr;
    bf16_t *wprep = nullptr;  // the weights as the data gradients read them
    float* logits = nullptr;
    float* loss = nullptr;
    // inference: the batch's pair table and neighbour features
    h264a_mvnet_pair* ipairs = nullptr;
    PropFrame* iprop = nullptr;  // a propose batch's frames: guide MVs and proposals
    int16_t* inmv = nullptr;
};

namespace {

template <class T>
int dmalloc(T** p, size_t n) {
    if (cudaMalloc(reinterpret_cast<void**>(p), n * sizeof(T)) != cudaSuccess) {
        cudaGetLastError();
        return fail(H264A_E_NOMEM, "mvnet: cudaMalloc failed");
    }
    return H264A_OK;
}

void free_net(h264a_mvnet* n) {
    void* ps[] = {n->master, n->w, n->grad, n->m1, n->m2, n->a1, n->a2, n->a3, n->h, n->dl, n->dh, n->df,
                  n->da3, n->da2, n->da1, n->wprep, n->logits, n->loss, n->ipairs, n->inmv, n->iprop};
    for (void* p : ps)
        if (p) cudaFree(p);
    delete n;
}

uint64_t splitmix(uint64_t& s) {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// He-normal weights (Box-Muller over splitmix64), zero biases, and zero rows /
// columns that only pad (FC1 inputs 1158..1167, head rows 289..295).
void init_params(std::vector<float>& p, uint64_t seed) {
    uint64_t s = seed;
    auto normal = [&]() {
        const double u1 = (double(splitmix(s) >> 11) + 1.0) * (1.0 / 9007199254740992.0);
        const double u2 = double(splitmix(s) >> 11) * (1.0 / 9007199254740992.0);
        return std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2);
    };
    p.assign(NPARAMS, 0.f);
    auto fill = [&](int off, int n, int fan_in) {
        const double sd = std::sqrt(2.0 / fan_in);
        for (int i = 0; i < n; i++) p[off + i] = float(normal() * sd);
    };
    fill(O_W1, N_W1, 18);
    fill(O_W2, N_W2, 144);
    fill(O_W3, N_W3, 288);
    fill(O_W4, N_W4, CONVF + 6);
    fill(O_W5, N_W5, HID);
    for (int o = 0; o < HID; o++)
        for (int k = CONVF + 6; k < FEAT; k++) p[O_W4 + o * FEAT + k] = 0.f;
    for (int r = NCLS; r < HEAD_N; r++)
        for (int k = 0; k < HID; k++) p[O_W5 + r * HID + k] = 0.f;
}

int upload_params(h264a_mvnet* n, const float* h) {
    H264A_CUDA(cudaMemcpy(n->master, h, sizeof(float) * NPARAMS, cudaMemcpyHostToDevice));
    to_bf16_kernel<<<(NPARAMS + 255) / 256, 256>>>(n->master, n->w, NPARAMS);
    H264A_CUDA(cudaGetLastError());
    H264A_CUDA(cudaDeviceSynchronize());
    return H264A_OK;
}

Bufs bufs(h264a_mvnet* n) {
    Bufs z;
    z.w = n->w; z.grad = n->grad;
    z.a1 = n->a1; z.a2 = n->a2; z.a3 = n->a3; z.h = n->h; z.dl = n->dl; z.dh = n->dh; z.df = n->df;
    z.da3 = n->da3; z.da2 = n->da2; z.da1 = n->da1;
    z.w4t = n->wprep;
    z.w5t = z.w4t + N_W4T;
    z.wd3 = z.w5t + N_W5T;
    z.wd2 = z.wd3 + N_WD3;
    z.logits = n->logits;
    return z;
}

Geo make_geo(const h264a_mvnet_pair* pairs, int P, int cw, int ch, const int16_t* nmv, const int16_t* labels) {
    Geo g;
    g.pairs = pairs; g.P = P; g.cw = cw; g.ch = ch;
    g.H1 = ch / 2; g.W1 = cw / 2; g.H2 = ch / 4; g.W2 = cw / 4; g.H3 = ch / 8; g.W3 = cw / 8;
    g.mb_w = cw / 16; g.mb_h = ch / 16; g.nmb = g.mb_w * g.mb_h;
    g.nmv = nmv; g.labels = labels;
    return g;
}

int check_geo(const h264a_mvnet* n, const h264a_mvnet_pair* d_pairs, int P, int cw, int ch, const void* nmv) {
    if (!n || !d_pairs || !nmv) return fail(H264A_E_ARG, "mvnet: null pointer");
    if (P < 1 || cw < 16 || ch < 16 || cw % 16 || ch % 16 || cw > 8192 || ch > 8192)
        return fail(H264A_E_ARG, "mvnet: frames must be MB-aligned, 16 to 8192 pixels a side, at least one pair");
    if ((long long)P * cw * ch > MAXPIX)
        return fail(H264A_E_ARG, "mvnet: a batch holds at most " + std::to_string(MAXPIX) + " luma pixels");
    return H264A_OK;
}

void trunk_forward(h264a_mvnet* n, const Geo& g, cudaStream_t st) {
    const Bufs z = bufs(n);
    gemm<16>(Conv1Fwd{g, z}, g.P * g.H1 * g.W1, 16, 32, st);
    gemm<32>(Conv2Fwd{g, z}, g.P * g.H2 * g.W2, 32, 144, st);
    gemm<32>(Conv3Fwd{g, z}, g.P * g.H3 * g.W3, 32, 288, st);
}

void head_forward(h264a_mvnet* n, const Geo& g, float* logits, cudaStream_t st) {
    Bufs z = bufs(n);
    z.logits = logits;
    const int B = g.P * g.nmb;
    gemm<256>(Fc1Fwd{g, z}, B, HID, FEAT, st);
    gemm<160>(HeadFwd{z}, B, HEAD_N, HID, st);
}

void backward(h264a_mvnet* n, const Geo& g, cudaStream_t st) {
    const Bufs z = bufs(n);
    const int B = g.P * g.nmb, S = n->sms;
    const int K3 = g.P * g.H3 * g.W3, K2 = g.P * g.H2 * g.W2, K1 = g.P * g.H1 * g.W1;
    prep_kernel<<<(N_PREP + 255) / 256, 256, 0, st>>>(n->w, n->wprep);
    wgrad<256, 64, 4>(HeadBwdW{z}, HEAD_N, HID, B, S, st);
    gemm<256>(HeadBwdData{z}, B, HID, HEAD_N, st);
    wgrad<256, 64, 4>(Fc1BwdW{g, z}, HID, FEAT, B, S, st);
    gemm<192>(Fc1BwdData{z}, B, CONVF, HID, st);
    const long long cells = (long long)K3 * 4;
    uncrop_kernel<<<unsigned((cells + 255) / 256), 256, 0, st>>>(g, n->df, n->a3, n->da3);
    wgrad<144, 64, 1>(Conv3BwdW{g, z}, 32, 288, K3, S, st);
    gemm<128>(ConvBwdData<32, 3>{g, z}, K3, 128, 128, st);
    wgrad<144, 128, 2>(Conv2BwdW{g, z}, 32, 144, K2, S, st);
    gemm<64>(ConvBwdData<16, 2>{g, z}, K2, 64, 128, st);
    wgrad<32, 128, 1>(Conv1BwdW{g, z}, 16, 24, K1, S, st);
}

}  // namespace

extern "C" int h264a_mvnet_create(int device, uint64_t seed, h264a_mvnet** out) {
    if (!out) return fail(H264A_E_ARG, "mvnet_create: null out");
    *out = nullptr;
    H264A_CUDA(cudaSetDevice(device));
    h264a_mvnet* n = new h264a_mvnet();
    n->device = device;
    cudaDeviceGetAttribute(&n->sms, cudaDevAttrMultiProcessorCount, device);
    int rc = H264A_OK;
    if (!rc) rc = dmalloc(&n->master, NPARAMS);
    if (!rc) rc = dmalloc(&n->w, NPARAMS);
    if (!rc) rc = dmalloc(&n->grad, NPARAMS);
    if (!rc) rc = dmalloc(&n->m1, NPARAMS);
    if (!rc) rc = dmalloc(&n->m2, NPARAMS);
    if (!rc) rc = dmalloc(&n->a1, size_t(MAXPIX / 4 * 16));
    if (!rc) rc = dmalloc(&n->da1, size_t(MAXPIX / 4 * 16));
    if (!rc) rc = dmalloc(&n->a2, size_t(MAXPIX / 16 * 32));
    if (!rc) rc = dmalloc(&n->da2, size_t(MAXPIX / 16 * 32));
    if (!rc) rc = dmalloc(&n->a3, size_t(MAXPIX / 64 * 32));
    if (!rc) rc = dmalloc(&n->da3, size_t(MAXPIX / 64 * 32));
    if (!rc) rc = dmalloc(&n->h, size_t(MAXS * HID));
    if (!rc) rc = dmalloc(&n->dh, size_t(MAXS * HID));
    if (!rc) rc = dmalloc(&n->dl, size_t(MAXS * HEAD_N));
    if (!rc) rc = dmalloc(&n->df, size_t(MAXS * CONVF));
    if (!rc) rc = dmalloc(&n->logits, size_t(MAXS * HEAD_N));
    if (!rc) rc = dmalloc(&n->wprep, size_t(N_PREP));
    if (!rc) rc = dmalloc(&n->loss, 1);
    if (!rc) rc = dmalloc(&n->inmv, size_t(MAXS * 6));
    if (!rc) rc = dmalloc(&n->ipairs, size_t(MAXPIX / 256));
    if (!rc) rc = dmalloc(&n->iprop, size_t(MAXPIX / 256));
    if (rc) {
        free_net(n);
        return rc;
    }
    std::vector<float> p;
    init_params(p, seed);
    rc = upload_params(n, p.data());
    if (!rc && cudaMemset(n->m1, 0, sizeof(float) * NPARAMS) != cudaSuccess) rc = fail(H264A_E_CUDA, "mvnet: memset");
    if (!rc && cudaMemset(n->m2, 0, sizeof(float) * NPARAMS) != cudaSuccess) rc = fail(H264A_E_CUDA, "mvnet: memset");
    if (rc) {
        free_net(n);
        return rc;
    }
    *out = n;
    return H264A_OK;
}

extern "C" int h264a_mvnet_destroy(h264a_mvnet* n) {
    if (!n) return H264A_OK;
    cudaSetDevice(n->device);
    cudaDeviceSynchronize();
    free_net(n);
    return H264A_OK;
}

extern "C" int h264a_mvnet_set_params(h264a_mvnet* n, const float* h_params) {
    if (!n || !h_params) return fail(H264A_E_ARG, "mvnet_set_params: null pointer");
    H264A_CUDA(cudaSetDevice(n->device));
    const int rc = upload_params(n, h_params);
    if (rc) return rc;
    H264A_CUDA(cudaMemset(n->m1, 0, sizeof(float) * NPARAMS));
    H264A_CUDA(cudaMemset(n->m2, 0, sizeof(float) * NPARAMS));
    n->step = 0;
    return H264A_OK;
}

extern "C" int h264a_mvnet_get_params(h264a_mvnet* n, float* h_params) {
    if (!n || !h_params) return fail(H264A_E_ARG, "mvnet_get_params: null pointer");
    H264A_CUDA(cudaSetDevice(n->device));
    H264A_CUDA(cudaDeviceSynchronize());
    H264A_CUDA(cudaMemcpy(h_params, n->master, sizeof(float) * NPARAMS, cudaMemcpyDeviceToHost));
    return H264A_OK;
}

extern "C" int h264a_mvnet_forward(h264a_mvnet* n, const h264a_mvnet_pair* d_pairs, int npairs, int cw, int ch,
                                   const int16_t* d_nmv, float* d_logits, void* stream) {
    int rc = check_geo(n, d_pairs, npairs, cw, ch, d_nmv);
    if (rc) return rc;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const Geo g = make_geo(d_pairs, npairs, cw, ch, d_nmv, nullptr);
    trunk_forward(n, g, st);
    // straight into the caller's buffer when the epilogue's 16-byte stores can
    const bool direct = d_logits != nullptr && (reinterpret_cast<uintptr_t>(d_logits) & 15) == 0;
    head_forward(n, g, direct ? d_logits : n->logits, st);
    if (d_logits && !direct)
        H264A_CUDA(cudaMemcpyAsync(d_logits, n->logits, sizeof(float) * HEAD_N * npairs * g.nmb,
                                   cudaMemcpyDeviceToDevice, st));
    return check_launch("mvnet forward");
}

extern "C" int h264a_mvnet_grads(h264a_mvnet* n, const h264a_mvnet_pair* d_pairs, int npairs, int cw, int ch,
                                 const int16_t* d_nmv, const int16_t* d_labels, float* d_grads, float* d_loss,
                                 void* stream) {
    int rc = check_geo(n, d_pairs, npairs, cw, ch, d_nmv);
    if (rc) return rc;
    if (!d_labels) return fail(H264A_E_ARG, "mvnet_grads: null labels");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const Geo g = make_geo(d_pairs, npairs, cw, ch, d_nmv, d_labels);
    const int B = npairs * g.nmb;
    H264A_CUDA(cudaMemsetAsync(n->grad, 0, sizeof(float) * NPARAMS, st));
    H264A_CUDA(cudaMemsetAsync(n->loss, 0, sizeof(float), st));
    trunk_forward(n, g, st);
    head_forward(n, g, n->logits, st);
    loss_kernel<<<(B * 32 + 255) / 256, 256, 0, st>>>(n->logits, d_labels, B, n->dl, n->loss);
    backward(n, g, st);
    if (d_grads) H264A_CUDA(cudaMemcpyAsync(d_grads, n->grad, sizeof(float) * NPARAMS, cudaMemcpyDeviceToDevice, st));
    if (d_loss) H264A_CUDA(cudaMemcpyAsync(d_loss, n->loss, sizeof(float), cudaMemcpyDeviceToDevice, st));
    return check_launch("mvnet grads");
}

extern "C" int h264a_mvnet_train_step(h264a_mvnet* n, const h264a_mvnet_pair* d_pairs, int npairs, int cw, int ch,
                                      const int16_t* d_nmv, const int16_t* d_labels, float lr, float* d_loss,
                                      void* stream) {
    if (!(lr > 0.f)) return fail(H264A_E_ARG, "mvnet_train_step: lr must be positive");
    int rc = h264a_mvnet_grads(n, d_pairs, npairs, cw, ch, d_nmv, d_labels, nullptr, d_loss, stream);
    if (rc) return rc;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    n->step++;
    const double b1 = 0.9, b2 = 0.999;
    const float c1 = float(1.0 / (1.0 - std::pow(b1, double(n->step))));
    const float c2 = float(1.0 / (1.0 - std::pow(b2, double(n->step))));
    adam_kernel<<<(NPARAMS + 255) / 256, 256, 0, st>>>(n->master, n->w, n->grad, n->m1, n->m2, NPARAMS, lr, float(b1),
                                                       float(b2), c1, c2, 1e-8f);
    return check_launch("mvnet adam");
}

extern "C" int h264a_mvnet_propose(h264a_mvnet* n, const h264a_mvnet_frame* h_frames, int nframes, void* stream) {
    if (!n || !h_frames) return fail(H264A_E_ARG, "mvnet_propose: null pointer");
    if (nframes < 1) return fail(H264A_E_ARG, "mvnet_propose: need at least one frame");
    for (int i = 0; i < nframes; i++) {
        const h264a_mvnet_frame& f = h_frames[i];
        if (!f.d_cur || !f.d_ref || !f.d_props) return fail(H264A_E_ARG, "mvnet_propose: null frame pointer");
        if (f.cw < 16 || f.ch < 16 || f.cw % 16 || f.ch % 16 || f.cw > 8192 || f.ch > 8192 ||
            (long long)f.cw * f.ch > MAXPIX)
            return fail(H264A_E_ARG, "mvnet_propose: frames must be MB-aligned, at most 8192 pixels a side");
    }
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    // consecutive frames of one geometry, up to MAXPIX pixels, form a batch:
    // their trunk maps in one pass, then FC1 + head over their MBs, then each
    // frame's top-8 into its own d_props
    std::vector<h264a_mvnet_pair> pr;
    std::vector<PropFrame> pf;
    int i = 0;
    while (i < nframes) {
        const int cw = h_frames[i].cw, ch = h_frames[i].ch;
        int j = i;
        pr.clear();
        pf.clear();
        while (j < nframes && h_frames[j].cw == cw && h_frames[j].ch == ch && (long long)(j - i + 1) * cw * ch <= MAXPIX) {
            pr.push_back(h264a_mvnet_pair{h_frames[j].d_cur, h_frames[j].d_ref});
            pf.push_back(PropFrame{h_frames[j].d_guide_mvs, h_frames[j].d_props});
            j++;
        }
        const int P = j - i;
        // the previous batch's kernels read the tables on this stream, so the
        // uploads are stream-ordered after them (pageable sources: the copies
        // are staged before the call returns)
        H264A_CUDA(cudaMemcpyAsync(n->ipairs, pr.data(), sizeof(h264a_mvnet_pair) * P, cudaMemcpyHostToDevice, st));
        H264A_CUDA(cudaMemcpyAsync(n->iprop, pf.data(), sizeof(PropFrame) * P, cudaMemcpyHostToDevice, st));
        const Geo g = make_geo(n->ipairs, P, cw, ch, n->inmv, nullptr);
        const long long samples = (long long)P * g.nmb;
        guide_frames_kernel<<<unsigned((samples + 255) / 256), 256, 0, st>>>(n->iprop, P, g.mb_w, g.mb_h, n->inmv);
        trunk_forward(n, g, st);
        head_forward(n, g, n->logits, st);
        top8_frames_kernel<<<unsigned((samples * 32 + 255) / 256), 256, 0, st>>>(n->logits, P, g.nmb, n->iprop);
        i = j;
    }
    return check_launch("mvnet propose");
}

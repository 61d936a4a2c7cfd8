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
static_assert((O_W1 | O_W2 | O_W3 | O_W4 | O_W5 | O_B2 | O_B3 | O_B4 | O_B5) % 8 == 0, "16-byte weight and bias chunks");

// The GEMMs' weights lie WREP times in memory, CTA x reading copy x % WREP:
// every CTA of a layer reads the same few hundred lines at nearly the same
// time, and one copy's lines sit in few of the L2's slices.  conv2 on four
// 1080p pairs: 100 us from one copy, 69 from three, 66 from eight; conv3's
// data gradient 45, 39 and 37.
constexpr int WREP = 8, WSTRIDE = (NPARAMS + 7) / 8 * 8;

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
__device__ __forceinline__ void st8(bf16_t* p, const uint4& v) { *reinterpret_cast<uint4*>(p) = v; }
// 8 bf16 values as floats
__device__ __forceinline__ void unpack8(const uint4& w, float* f) {
    const uint32_t a[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        f[2 * i] = bf2f(bf16_t(a[i] & 0xffffu));
        f[2 * i + 1] = bf2f(bf16_t(a[i] >> 16));
    }
}
__device__ __forceinline__ uint4 pack8(const float* v) {  // rounded to bf16
    return make_uint4(pack2(f2bf(v[0]), f2bf(v[1])), pack2(f2bf(v[2]), f2bf(v[3])), pack2(f2bf(v[4]), f2bf(v[5])),
                      pack2(f2bf(v[6]), f2bf(v[7])));
}
// 8 values, bias added, ReLU
__device__ __forceinline__ uint4 relu8(const float* v, const bf16_t* bias) {
    float b[8], r[8];
    unpack8(ld8(bias), b);
#pragma unroll
    for (int i = 0; i < 8; i++) r[i] = fmaxf(v[i] + b[i], 0.f);
    return pack8(r);
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

// The bf16 pair (reference, current) of two pixels, (v - 128) / 64 each: k/64
// with |k| <= 128, so float and bf16 hold it exactly and its upper half is the
// bf16.  The byte is the mantissa of 2^23 + v; the multiply-add takes 2^23 / 64
// + 2 away again.
__device__ __forceinline__ uint32_t x0_word(uint32_t r, uint32_t c) {
    const float a = fmaf(__uint_as_float(0x4b000000u | r), 1.f / 64.f, -131074.f);
    const float b = fmaf(__uint_as_float(0x4b000000u | c), 1.f / 64.f, -131074.f);
    return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}
__device__ __forceinline__ bf16_t mv_feat(const Geo& g, int m, int i) {
    const int v = min(max(int(g.nmv[6LL * m + i]), -128), 128);
    return f2bf(float(v) * (1.f / 64.f));  // exact
}

// ---- the tcgen05 GEMM: 128 x BN tiles, accumulators in tensor memory --------
// The GEMM of FC1, the head and their data gradients, C[M][N] = sum_k A[m][k]
// B[k][n], on the sm_100 tensor cores: per 64-wide K step all 256
// threads copy the A (MT x 128 x 64) and B (BN x 64) tiles by 16-byte cp.async
// into one of ST shared-memory stages (steps it + 1 .. it + ST - 1 are in flight
// while step it multiplies), one thread issues four tcgen05.mma (M 128, N BN,
// K 16, bf16 in, fp32 accumulated in tensor memory) and commits them to the
// stage's mbarrier.  The epilogue reads the accumulator rows with tcgen05.ld
// (warp w may read tensor-memory lanes 32(w % 4) .. +31, its tile rows; warps w
// and w + 4 take half of the columns each), puts the packed results where the
// stages were and writes whole rows from there: stored row by row from the
// registers, 32 rows a request, it took longer than the products (head 27,000
// of a CTA's 45,000 cycles).  Bound by the operands' way through the L2 (five
// or so TB/s over both dies).  Four 1080p pairs, before (operands through
// registers) and now: FC1 85 -> 61 us, head 48 -> 32, FC1's data gradient
// 128 -> 89.
constexpr int TC_BM = 128, TC_BK = 64, TC_THREADS = 256;

template <int BN>
constexpr int tc_cols() {
    return BN <= 32 ? 32 : (BN <= 64 ? 64 : (BN <= 128 ? 128 : (BN <= 256 ? 256 : 512)));
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
// status (the net's host word, see check_waits) and keeps waiting up to twice
// as long, so that no tensor-core work is left reading a stage or writing
// tensor memory.
__device__ __forceinline__ void tc_wait(uint32_t bar, uint32_t parity, int* status) {
    constexpr int kLimit = 1 << 22;
    for (int it = 0; !mbar_try_wait(bar, parity); it++) {
        if (it == kLimit) *reinterpret_cast<volatile int*>(status) = 4;
        if (it >= 2 * kLimit) break;
    }
}

// 16 accumulator columns of the lane's row
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float* f) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) f[i] = __uint_as_float(r[i]);
}
// 16 bytes global -> shared, zeros where not ok (`any`: an address to name then)
__device__ __forceinline__ void cp16z(uint32_t dst, const bf16_t* p, bool ok, const bf16_t* any) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(ok ? p : any), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void st16s(uint32_t dst, const uint4& v) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

__device__ __forceinline__ uint4 ld16s(uint32_t src) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(src) : "memory");
    return v;
}

// An Op names the 16 bytes of 8 consecutive k of A as op.a8(row, step, p):
// their address in p, false for zeros.  Row is what output row m gives
// (op.row(m): base address, position) and Step what chunk k gives (op.step(k),
// k a multiple of 8: offset, window cell).  A thread of the GEMM below keeps
// its rows and makes one Step per K step, one of the weight gradients its
// Steps and one row per K step, so a copy costs an add and two compares.
// Where kCalc, op.calc(step) chunks are op.make(row, step) instead.  B is
// op.b(copy) with op.ldb columns per row n.  op.pack(n, v) makes 8 results
// (n ..) the 16 bytes (32 where kF32) that op.store(o, n, w) puts at n .. of a
// row with output offset o = op.out_at(m).  K and N are multiples of 8.
template <class Op>
__device__ __forceinline__ void stage_a8(const Op& op, uint32_t dst, const typename Op::Row& row, const typename Op::Step& s,
                                         bool live) {
    if constexpr (Op::kCalc) {
        if (live && op.calc(s)) {
            st16s(dst, op.make(row, s));
            return;
        }
    }
    const bf16_t* p = op.z.w;
    live = op.a8(row, s, p) && live;
    cp16z(dst, p, live, op.z.w);
}

template <int BN, int MT, int ST, class Op>
__global__ void __launch_bounds__(TC_THREADS) gemm_tc_kernel(const Op op, int M, int N, int K, int* status) {
    static_assert(BN % 32 == 0 && BN <= 256 && ST >= 2, "tcgen05 N for M = 128, halves of 16 columns");
    constexpr int ROWS = MT * TC_BM, A_TILE = TC_BM * TC_BK * 2, A_BYTES = MT * A_TILE, STAGE = A_BYTES + BN * TC_BK * 2;
    constexpr int NCOL = tc_cols<BN * MT>();
    constexpr uint32_t IDESC = tc_idesc<BN>();
    extern __shared__ __align__(128) uint8_t tc_smem[];
    __shared__ __align__(8) unsigned long long tc_bar[ST];
    __shared__ uint32_t tc_tmem;
    __shared__ typename Op::Row tc_rows[ROWS];
    __shared__ long long tc_out[ROWS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * ROWS, n0 = blockIdx.y * BN;
    // read after the __syncthreads below; rows past M repeat the last and are not stored
    for (int i = tid; i < 2 * ROWS; i += TC_THREADS) {
        const int m = min(m0 + i % ROWS, M - 1);
        if (i < ROWS)
            tc_rows[i] = op.row(m);
        else
            tc_out[i - ROWS] = op.out_at(m);
    }
    const uint32_t sbase = tc_smem_u32(tc_smem), bar0 = tc_smem_u32(&tc_bar[0]);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(&tc_tmem)),
                     "r"(NCOL));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
#pragma unroll
        for (int s = 0; s < ST; s++) mbar_init(bar0 + 8 * s, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tc_tmem;
    const int nk = (K + TC_BK - 1) / TC_BK;
    // consecutive threads fill consecutive 16-byte rows of a core matrix, so
    // a warp's stores meet no bank twice; a thread keeps one chunk column and
    // every 32nd row
    constexpr int AQ = ROWS * 8 / TC_THREADS, BQ = BN * 8 / TC_THREADS;
    static_assert(AQ * TC_THREADS == ROWS * 8 && BQ * TC_THREADS == BN * 8, "whole passes");
    const int c = (tid >> 3) & 7, r0 = ((tid >> 6) << 3) | (tid & 7);
    typename Op::Row rows[AQ];
#pragma unroll
    for (int j = 0; j < AQ; j++) rows[j] = tc_rows[r0 + 32 * j];
    const bf16_t* bp = op.b(blockIdx.x % WREP) + (long long)(n0 + r0) * Op::ldb + 8 * c;
    const uint32_t off0 = tc_off(r0, c);
    auto load = [&](int it) {
        const uint32_t sa = sbase + uint32_t((it % ST) * STAGE) + off0, sb = sa + A_BYTES;
        const bool kin = it * TC_BK + 8 * c < K;
        const typename Op::Step s = op.step(it * TC_BK + 8 * c);
#pragma unroll
        for (int j = 0; j < AQ; j++) stage_a8(op, sa + 4096u * j, rows[j], s, kin);
#pragma unroll
        for (int j = 0; j < BQ; j++)
            cp16z(sb + 4096u * j, bp + it * TC_BK + 32 * j * Op::ldb, kin && n0 + r0 + 32 * j < N, op.z.w);
    };
#pragma unroll
    for (int s = 0; s < ST - 1; s++) {
        if (s < nk) load(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int it = 0; it < nk; it++) {
        const uint32_t sa = sbase + uint32_t((it % ST) * STAGE), sb = sa + A_BYTES;
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
        // the tiles' generic-proxy writes, visible to the tensor cores
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int j = 0; j < TC_BK / 16; j++) {
                const uint64_t db = tc_sdesc(sb + 256u * j);
                const uint32_t acc = (it > 0 || j > 0) ? 1u : 0u;
#pragma unroll
                for (int t = 0; t < MT; t++)
                    asm volatile(
                        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(tmem + uint32_t(t * BN)),
                        "l"(tc_sdesc(sa + uint32_t(t * A_TILE) + 256u * j)), "l"(db), "r"(IDESC), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
                        : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar0 + 8 * (it % ST))
                         : "memory");
        }
        if (it + ST - 1 < nk) {
            // the stage's previous MMAs (step it - 1) have read it
            if (it >= 1) tc_wait(bar0 + 8 * ((it - 1) % ST), uint32_t((it - 1) / ST) & 1u, status);
            load(it + ST - 1);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // the last step's commit completes after every earlier MMA
    tc_wait(bar0 + 8 * ((nk - 1) % ST), uint32_t((nk - 1) / ST) & 1u, status);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    {
        constexpr int ES = Op::kF32 ? 4 : 2, PITCH = BN * ES + 16, CH = BN * ES / 16;
        static_assert(MT * TC_BM * PITCH <= ST * STAGE, "the results take the stages' place");
        const int cb = (warp >> 2) * (BN / 2);
#pragma unroll 1
        for (int t = 0; t < MT; t++) {
            const uint32_t so = sbase + uint32_t((t * TC_BM + (warp & 3) * 32 + lane) * PITCH);
            const uint32_t taddr = tmem + uint32_t(t * BN) + (uint32_t((warp & 3) * 32) << 16);
#pragma unroll 1
            for (int c0 = cb; c0 < cb + BN / 2; c0 += 16) {
                float f[16];
                tc_ld16(taddr + uint32_t(c0), f);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int n = min(n0 + c0 + 8 * h, N - 8);  // columns past N are not stored
                    if constexpr (Op::kF32) {
                        uint4 w[2];
                        op.pack(n, f + 8 * h, w);
                        st16s(so + uint32_t(c0 + 8 * h) * 4, w[0]);
                        st16s(so + uint32_t(c0 + 8 * h) * 4 + 16, w[1]);
                    } else {
                        st16s(so + uint32_t(c0 + 8 * h) * 2, op.pack(n, f + 8 * h));
                    }
                }
            }
        }
        __syncthreads();
#pragma unroll 4
        for (int i = tid; i < ROWS * CH; i += TC_THREADS) {
            const int row = i / CH, ch = i - row * CH, n = n0 + ch * (16 / ES);
            if (m0 + row < M && n < N) op.store(tc_out[row], n, ld16s(sbase + uint32_t(row * PITCH + ch * 16)));
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NCOL));
}

// The GEMMs of few columns and a short K (conv2, conv3 and their data
// gradients: N <= 128, at most KT = 2 .. 5 steps), persistent: a CTA keeps the
// whole B in shared memory and walks row tiles, its ring of ST stages of A
// running on from one tile into the next and its accumulators in two sets, so
// a tile's loads, products and results overlap its neighbours'.  (A CTA per
// tile spent most of its time on its own start: row table, tensor memory,
// first loads, then results with nothing behind them.)  Bound by the 16-byte
// gathers (conv2 reads each input cell 2.25 times).  Four 1080p pairs, a CTA
// per tile and persistent: conv2 67 -> 57 us, conv3 30 -> 29, conv3's data
// gradient 37 -> 32, conv2's 83 -> 84.
template <int BN, int KT, int ST>
constexpr int conv_smem() {
    return KT * BN * TC_BK * 2 + ST * TC_BM * TC_BK * 2 + TC_BM * (BN * 2 + 16);
}
template <int BN, int KT, int ST, class Op>
__global__ void __launch_bounds__(TC_THREADS) conv_tc_kernel(const Op op, int M, int K, int* status) {
    static_assert(BN % 32 == 0 && BN <= 128 && ST >= 2 && !Op::kCalc && !Op::kF32, "tile shape");
    constexpr int A_BYTES = TC_BM * TC_BK * 2, B_STEP = BN * TC_BK * 2, NCOL = tc_cols<2 * BN>();
    constexpr uint32_t IDESC = tc_idesc<BN>();
    extern __shared__ __align__(128) uint8_t tc_smem[];
    __shared__ __align__(8) unsigned long long tc_bar[ST + 2];  // stages, accumulator sets
    __shared__ uint32_t tc_tmem;
    __shared__ long long tc_out[2][TC_BM];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t sw = tc_smem_u32(tc_smem), sbase = sw + KT * B_STEP, sres = sbase + ST * A_BYTES;
    const uint32_t bar0 = tc_smem_u32(&tc_bar[0]), tbar = bar0 + 8 * ST;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(&tc_tmem)),
                     "r"(NCOL));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
#pragma unroll
        for (int s = 0; s < ST + 2; s++) mbar_init(bar0 + 8 * s, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tc_tmem;
    const int tiles = (M + TC_BM - 1) / TC_BM;
    const int nt = (tiles - int(blockIdx.x) + int(gridDim.x) - 1) / int(gridDim.x), steps = nt * KT;  // grid <= tiles: nt >= 1
    auto tile_m0 = [&](int i) { return (int(blockIdx.x) + i * int(gridDim.x)) * TC_BM; };
    constexpr int AQ = TC_BM * 8 / TC_THREADS;
    const int c = (tid >> 3) & 7, r0 = ((tid >> 6) << 3) | (tid & 7);
    const uint32_t off0 = tc_off(r0, c);
    {
        const bf16_t* bp = op.b(blockIdx.x % WREP);
        for (int i = tid; i < BN * 8 * KT; i += TC_THREADS) {
            const int n = ((i >> 6) << 3 | (i & 7)) % BN, ks = i / (BN * 8), ch = (i >> 3) & 7, k = ks * TC_BK + 8 * ch;
            cp16z(sw + uint32_t(ks * B_STEP) + tc_off(n, ch), bp + n * Op::ldb + k, k < K, op.z.w);
        }
    }
    typename Op::Row rows[AQ];
    auto load = [&](int g) {  // in order of g
        const int ks = g % KT;
        if (ks == 0) {
            const int m0 = tile_m0(g / KT);
#pragma unroll
            for (int j = 0; j < AQ; j++) rows[j] = op.row(min(m0 + r0 + 32 * j, M - 1));
        }
        const uint32_t sa = sbase + uint32_t((g % ST) * A_BYTES) + off0;
        const int k = ks * TC_BK + 8 * c;
        const typename Op::Step s = op.step(k);
#pragma unroll
        for (int j = 0; j < AQ; j++) stage_a8(op, sa + 4096u * j, rows[j], s, k < K);
    };
    auto results = [&](int i) {  // of the CTA's tile i, whose products are committed
        constexpr int PITCH = BN * 2 + 16, CH = BN / 8;
        tc_wait(tbar + 8 * (i & 1), uint32_t(i >> 1) & 1u, status);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t so = sres + uint32_t(((warp & 3) * 32 + lane) * PITCH);
        const uint32_t taddr = tmem + uint32_t((i & 1) * BN) + (uint32_t((warp & 3) * 32) << 16);
        const int cb = (warp >> 2) * (BN / 2);
#pragma unroll 1
        for (int c0 = cb; c0 < cb + BN / 2; c0 += 16) {
            float f[16];
            tc_ld16(taddr + uint32_t(c0), f);
            st16s(so + uint32_t(c0) * 2, op.pack(c0, f));
            st16s(so + uint32_t(c0) * 2 + 16, op.pack(c0 + 8, f + 8));
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        const int m0 = tile_m0(i);
#pragma unroll 4
        for (int j = tid; j < TC_BM * CH; j += TC_THREADS) {
            const int row = j / CH, ch = j - row * CH;
            if (m0 + row < M) op.store(tc_out[i & 1][row], 8 * ch, ld16s(sres + uint32_t(row * PITCH + ch * 16)));
        }
    };
#pragma unroll
    for (int s = 0; s < ST - 1; s++) {
        if (s < steps) load(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int i = 0, g = 0; i < nt; i++) {
        for (int ks = 0; ks < KT; ks++, g++) {
            const uint32_t sa = sbase + uint32_t((g % ST) * A_BYTES), sb = sw + uint32_t(ks * B_STEP);
            asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();  // also: everyone has read tile i - 2's accumulators and results
            if (tid == 0) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int j = 0; j < TC_BK / 16; j++)
                    asm volatile(
                        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(
                            tmem + uint32_t((i & 1) * BN)),
                        "l"(tc_sdesc(sa + 256u * j)), "l"(tc_sdesc(sb + 256u * j)), "r"(IDESC), "r"((ks > 0 || j > 0) ? 1u : 0u),
                        "r"(0u), "r"(0u), "r"(0u), "r"(0u)
                        : "memory");
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar0 + 8 * (g % ST))
                             : "memory");
                if (ks == KT - 1)
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tbar + 8 * (i & 1))
                                 : "memory");
            }
            if (ks == 0 && tid < TC_BM) tc_out[i & 1][tid] = op.out_at(min(tile_m0(i) + tid, M - 1));
            if (g + ST - 1 < steps) {
                // the stage's previous MMAs (step g - 1) have read it
                if (g >= 1) tc_wait(bar0 + 8 * ((g - 1) % ST), uint32_t((g - 1) / ST) & 1u, status);
                load(g + ST - 1);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        if (i > 0) results(i - 1);
    }
    __syncthreads();  // the last tile's row offsets, where KT = 1
    results(nt - 1);
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
    int* status;  // the net's status word
};

// conv1's window of output position m: the pair's planes at its top-left pixel
// (oy = 0 and ox = 0 reach one row and column outside the frame)
struct Conv1Row {
    const uint8_t *r, *c;
    bool top, left;  // the window's first row / column lies outside
};
__device__ __forceinline__ Conv1Row conv1_row(const Geo& g, int m) {
    const int OHW = g.H1 * g.W1;
    const int b = m / OHW, q = m - b * OHW, oy = q / g.W1, ox = q - oy * g.W1;
    const h264a_mvnet_pair p = g.pairs[b];
    const long long o = (long long)(2 * oy - 1) * g.cw + 2 * ox - 1;
    return Conv1Row{p.d_ref + o, p.d_cur + o, oy == 0, ox == 0};
}
// the input pair of tap (ky, kx), zero outside the frame (the conv's padding)
__device__ __forceinline__ uint32_t conv1_tap(const Conv1Row& w, int cw, int ky, int kx) {
    if ((w.top && ky == 0) || (w.left && kx == 0)) return 0u;
    const int o = ky * cw + kx;
    return x0_word(w.r[o], w.c[o]);
}

// conv1 forward: M = P*H1*W1, N = 16, K = 18 in two K 16 steps (the rest
// zeros).  Persistent: a thread gathers its row's nine taps (18 byte loads)
// into the 128 x 32 A tile while the tensor core multiplies the tile before.
// Bound by those loads' issue; 64-wide K steps of generic gathers, a CTA per
// tile, took 165 us on four 1080p pairs, this 38.
constexpr int C1_CTAS = 8;  // per SM
__global__ void __launch_bounds__(128, C1_CTAS) conv1_kernel(const Geo g, const Bufs z, int M, int* status) {
    constexpr int STAGE = 128 * 64;  // bytes: 16 row groups x 4 k-chunks x 128
    constexpr uint64_t DESC_HI = (uint64_t(128 >> 4) << 16) | (uint64_t(512 >> 4) << 32) | (1ull << 46);
    __shared__ __align__(128) uint8_t smem[2 * STAGE + 16 * 64];
    __shared__ __align__(8) unsigned long long bar[2];
    __shared__ uint32_t tmem_s;
    const int tid = threadIdx.x, warp = tid >> 5;
    const uint32_t sbase = tc_smem_u32(smem), sw = sbase + 2 * STAGE, bar0 = tc_smem_u32(bar);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(&tmem_s)), "r"(32));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        mbar_init(bar0, 1);
        mbar_init(bar0 + 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // element offset of (row, k-chunk) of a 32-wide tile, in bytes
    auto off = [](int row, int chunk) { return uint32_t(((row >> 3) * 4 + chunk) * 128 + (row & 7) * 16); };
    if (tid < 64) {  // weights: 16 rows of 18, zero to 32
        const int n = tid >> 2, ch = tid & 3;
        uint32_t v[4];
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = 8 * ch + 2 * i < 18 ? ld_pair(z.w + O_W1 + n * 18 + 8 * ch + 2 * i) : 0u;
        st16s(sw + off(n, ch), make_uint4(v[0], v[1], v[2], v[3]));
    }
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    st16s(sbase + off(tid, 3), zero);  // k 24..31 of both stages
    st16s(sbase + STAGE + off(tid, 3), zero);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_s;
    float bias[16];
#pragma unroll
    for (int i = 0; i < 16; i++) bias[i] = bf2f(z.w[O_B1 + i]);
    const int tiles = (M + 127) / 128;
    int prev = -1, it = 0;  // the tile whose accumulators are to be read
    for (int t = blockIdx.x;; t += gridDim.x, it++) {
        const int st = it & 1;
        if (t < tiles) {
            const Conv1Row w = conv1_row(g, min(t * 128 + tid, M - 1));
            uint32_t v[9];
#pragma unroll
            for (int k = 0; k < 9; k++) v[k] = conv1_tap(w, g.cw, k / 3, k % 3);
            const uint32_t sa = sbase + uint32_t(st * STAGE);
            st16s(sa + off(tid, 0), make_uint4(v[0], v[1], v[2], v[3]));
            st16s(sa + off(tid, 1), make_uint4(v[4], v[5], v[6], v[7]));
            st16s(sa + off(tid, 2), make_uint4(v[8], 0u, 0u, 0u));
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");  // the reads of tile it - 2's accumulators
            __syncthreads();
            if (tid == 0) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const uint64_t da = uint64_t(((sa + 256u * j) >> 4) & 0x3fffu) | DESC_HI;
                    const uint64_t db = uint64_t(((sw + 256u * j) >> 4) & 0x3fffu) | DESC_HI;
                    const uint32_t acc = j > 0 ? 1u : 0u;
                    asm volatile(
                        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(tmem + 16u * st),
                        "l"(da), "l"(db), "r"(tc_idesc<16>()), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
                        : "memory");
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar0 + 8 * st)
                             : "memory");
            }
        }
        if (prev >= 0) {
            tc_wait(bar0 + 8 * (st ^ 1), uint32_t((it - 1) >> 1) & 1u, status);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float f[16];
            tc_ld16(tmem + 16u * (st ^ 1) + (uint32_t(warp * 32) << 16), f);
            const int m = prev * 128 + tid;
            if (m < M) {
                uint32_t o[8];
#pragma unroll
                for (int i = 0; i < 8; i++)
                    o[i] = pack2(f2bf(fmaxf(f[2 * i] + bias[2 * i], 0.f)), f2bf(fmaxf(f[2 * i + 1] + bias[2 * i + 1], 0.f)));
                uint4* d = reinterpret_cast<uint4*>(z.a1 + (long long)m * 16);
                d[0] = make_uint4(o[0], o[1], o[2], o[3]);
                d[1] = make_uint4(o[4], o[5], o[6], o[7]);
            }
        }
        if (t >= tiles) break;
        prev = t;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(32));
}
// A row of a window over an NHWC map: its top-left cell (which may lie outside)
struct WinRow {
    const bf16_t* p;
    int y0, x0;
};
struct WinStep {
    int off, dy, dx;  // element offset and cell of the chunk in the window
};
__device__ __forceinline__ bool win_a8(const WinRow& w, const WinStep& s, int H, int W, const bf16_t*& p) {
    p = w.p + s.off;
    return unsigned(w.y0 + s.dy) < unsigned(H) && unsigned(w.x0 + s.dx) < unsigned(W);
}
// A row of a plain matrix; its step is the column
struct MatRow {
    const bf16_t* p;
};
__device__ __forceinline__ bool mat_a8(const MatRow& w, int k, const bf16_t*& p) {
    p = w.p + k;
    return true;
}

// conv2 / conv3 forward: im2col of the previous map; a chunk is 8 channels of
// one tap, 16 contiguous bytes
template <int C, int OW, int OB, int WHICH>
struct ConvFwd {
    Geo g; Bufs z;
    using Row = WinRow;
    using Step = WinStep;
    static constexpr bool kCalc = false;
    static constexpr int ldb = 9 * C;
    __device__ Row row(int m) const {
        const int H = WHICH == 2 ? g.H1 : g.H2, W = WHICH == 2 ? g.W1 : g.W2;
        const int ow = W >> 1, ohw = (H >> 1) * ow;
        const int b = m / ohw, r = m - b * ohw, oy = r / ow, ox = r - oy * ow;
        return Row{(WHICH == 2 ? z.a1 : z.a2) + ((long long)(b * H + 2 * oy - 1) * W + 2 * ox - 1) * C, 2 * oy - 1, 2 * ox - 1};
    }
    __device__ Step step(int k) const {
        const int tap = k / C, ci = k - tap * C, ky = (tap * 11) >> 5, kx = tap - ky * 3;  // ky = tap / 3 for tap < 16
        return Step{(ky * (WHICH == 2 ? g.W1 : g.W2) + kx) * C + ci, ky, kx};
    }
    __device__ bool a8(const Row& w, const Step& s, const bf16_t*& p) const {
        return win_a8(w, s, WHICH == 2 ? g.H1 : g.H2, WHICH == 2 ? g.W1 : g.W2, p);
    }
    __device__ const bf16_t* b(int copy) const { return z.w + OW + copy * WSTRIDE; }
    __device__ long long out_at(int m) const { return (long long)m * 32; }
    static constexpr bool kF32 = false;
    __device__ uint4 pack(int n, const float* v) const { return relu8(v, z.w + OB + n); }
    __device__ void store(long long o, int n, const uint4& w) const { st8((WHICH == 2 ? z.a2 : z.a3) + o + n, w); }
};
using Conv2Fwd = ConvFwd<16, O_W2, O_B2, 2>;
using Conv3Fwd = ConvFwd<32, O_W3, O_B3, 3>;

// FC1: k < 1152 are the channels of the MB's 6x6-cell crop of A3 (zero outside
// the map), then the 6 neighbour-MV features (one chunk) and zeros
struct Fc1Fwd {
    Geo g; Bufs z;
    struct Row {
        WinRow w;
        int m;
    };
    struct Step {
        WinStep s;
        int k;
    };
    static constexpr bool kCalc = true;
    static constexpr int ldb = FEAT;
    __device__ Row row(int m) const {
        const int b = m / g.nmb, r = m - b * g.nmb, mby = r / g.mb_w, mbx = r - mby * g.mb_w;
        const int y0 = 2 * mby - 2, x0 = 2 * mbx - 2;
        return Row{WinRow{z.a3 + ((long long)(b * g.H3 + y0) * g.W3 + x0) * 32, y0, x0}, m};
    }
    __device__ Step step(int k) const {
        const int cy = k / 192, rem = k - cy * 192, cx = rem >> 5;
        return Step{WinStep{(cy * g.W3 + cx) * 32 + (rem & 31), cy, cx}, k};
    }
    __device__ bool calc(const Step& s) const { return s.k == CONVF; }
    __device__ uint4 make(const Row& w, const Step&) const {
        return make_uint4(pack2(mv_feat(g, w.m, 0), mv_feat(g, w.m, 1)), pack2(mv_feat(g, w.m, 2), mv_feat(g, w.m, 3)),
                          pack2(mv_feat(g, w.m, 4), mv_feat(g, w.m, 5)), 0u);
    }
    __device__ bool a8(const Row& w, const Step& s, const bf16_t*& p) const {
        return win_a8(w.w, s.s, g.H3, g.W3, p) && s.k < CONVF;
    }
    __device__ const bf16_t* b(int copy) const { return z.w + O_W4 + copy * WSTRIDE; }
    __device__ long long out_at(int m) const { return (long long)m * HID; }
    static constexpr bool kF32 = false;
    __device__ uint4 pack(int n, const float* v) const { return relu8(v, z.w + O_B4 + n); }
    __device__ void store(long long o, int n, const uint4& w) const { st8(z.h + o + n, w); }
};
struct HeadFwd {
    Bufs z;
    using Row = MatRow;
    using Step = int;
    static constexpr bool kCalc = false;
    static constexpr int ldb = HID;
    __device__ Row row(int m) const { return Row{z.h + (long long)m * HID}; }
    __device__ Step step(int k) const { return k; }
    __device__ bool a8(const Row& w, Step k, const bf16_t*& p) const { return mat_a8(w, k, p); }
    __device__ const bf16_t* b(int copy) const { return z.w + O_W5 + copy * WSTRIDE; }
    __device__ long long out_at(int m) const { return (long long)m * HEAD_N; }
    static constexpr bool kF32 = true;
    __device__ void pack(int n, const float* v, uint4* w) const {
        float b[8];
        unpack8(ld8(z.w + O_B5 + n), b);
#pragma unroll
        for (int i = 0; i < 8; i++) b[i] += v[i];
        w[0] = make_uint4(__float_as_uint(b[0]), __float_as_uint(b[1]), __float_as_uint(b[2]), __float_as_uint(b[3]));
        w[1] = make_uint4(__float_as_uint(b[4]), __float_as_uint(b[5]), __float_as_uint(b[6]), __float_as_uint(b[7]));
    }
    __device__ void store(long long o, int n, const uint4& w) const { *reinterpret_cast<uint4*>(z.logits + o + n) = w; }
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
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N_PREP) return;
    bf16_t v;
    if (i < N_W4T)
        v = w[O_W4 + (i % HID) * FEAT + i / HID];
    else if (i < N_W4T + N_W5T)
        v = w[O_W5 + ((i - N_W4T) % HEAD_N) * HID + (i - N_W4T) / HEAD_N];
    else if (i < N_W4T + N_W5T + N_WD3)
        v = wd_at(w + O_W3, 32, i - N_W4T - N_W5T);
    else
        v = wd_at(w + O_W2, 16, i - N_W4T - N_W5T - N_WD3);
    for (int r = 0; r < WREP; r++) out[i + r * N_PREP] = v;
}

__device__ __forceinline__ uint32_t mask_pair(uint32_t act, uint32_t v) {  // bf16 pair v where the activation is not zero
    return v & ((act & 0xffffu ? 0xffffu : 0u) | (act & 0xffff0000u ? 0xffff0000u : 0u));
}
// 8 bf16 values, zero where the activation there is (ReLU's gradient)
__device__ __forceinline__ uint4 mask8(const uint4& a, const uint4& w) {
    return make_uint4(mask_pair(a.x, w.x), mask_pair(a.y, w.y), mask_pair(a.z, w.z), mask_pair(a.w, w.w));
}

struct HeadBwdData {  // dh = relu'(h) * (dl W5): M = B, N = 256, K = 296
    Bufs z;
    using Row = MatRow;
    using Step = int;
    static constexpr bool kCalc = false;
    static constexpr int ldb = HEAD_N;
    __device__ Row row(int m) const { return Row{z.dl + (long long)m * HEAD_N}; }
    __device__ Step step(int k) const { return k; }
    __device__ bool a8(const Row& w, Step k, const bf16_t*& p) const { return mat_a8(w, k, p); }
    __device__ const bf16_t* b(int copy) const { return z.w5t + copy * N_PREP; }
    __device__ long long out_at(int m) const { return (long long)m * HID; }
    static constexpr bool kF32 = false;
    __device__ uint4 pack(int, const float* v) const { return pack8(v); }
    __device__ void store(long long o, int n, const uint4& w) const { st8(z.dh + o + n, mask8(ld8(z.h + o + n), w)); }
};
struct Fc1BwdData {  // df = (dh W4)[:, :1152]: M = B, N = 1152, K = 256
    Bufs z;
    using Row = MatRow;
    using Step = int;
    static constexpr bool kCalc = false;
    static constexpr int ldb = HID;
    __device__ Row row(int m) const { return Row{z.dh + (long long)m * HID}; }
    __device__ Step step(int k) const { return k; }
    __device__ bool a8(const Row& w, Step k, const bf16_t*& p) const { return mat_a8(w, k, p); }
    __device__ const bf16_t* b(int copy) const { return z.w4t + copy * N_PREP; }
    __device__ long long out_at(int m) const { return (long long)m * CONVF; }
    static constexpr bool kF32 = false;
    __device__ uint4 pack(int, const float* v) const { return pack8(v); }
    __device__ void store(long long o, int n, const uint4& w) const { st8(z.df + o + n, w); }
};
// conv input gradient: M = pairs x output positions (2x2 input blocks),
// N = 4 C, K = 4 x 32 (see prep_kernel); WHICH 3: da3 -> da2, 2: da2 -> da1
template <int C, int WHICH>
struct ConvBwdData {
    Geo g; Bufs z;
    using Row = WinRow;  // of dy position (a, b); steps lead to (a + ny, b + nx)
    using Step = WinStep;
    static constexpr bool kCalc = false;
    static constexpr int ldb = 128;
    __device__ Row row(int m) const {
        const int OW = WHICH == 3 ? g.W3 : g.W2, ohw = (WHICH == 3 ? g.H3 : g.H2) * OW;
        const int r = m % ohw, a = r / OW;
        return Row{(WHICH == 3 ? z.da3 : z.da2) + (long long)m * 32, a, r - a * OW};
    }
    __device__ Step step(int k) const {
        const int nb = k >> 5;
        return Step{((nb >> 1) * (WHICH == 3 ? g.W3 : g.W2) + (nb & 1)) * 32 + (k & 31), nb >> 1, nb & 1};
    }
    __device__ bool a8(const Row& w, const Step& s, const bf16_t*& p) const {
        return win_a8(w, s, WHICH == 3 ? g.H3 : g.H2, WHICH == 3 ? g.W3 : g.W2, p);
    }
    __device__ const bf16_t* b(int copy) const { return (WHICH == 3 ? z.wd3 : z.wd2) + copy * N_PREP; }
    __device__ long long out_at(int m) const {  // input pixel (2a, 2b)
        const int OW = WHICH == 3 ? g.W3 : g.W2;
        const int y = m / OW, x = m - y * OW;  // y: pair * OH + a
        return ((long long)(2 * y) * (2 * OW) + 2 * x) * C;
    }
    static constexpr bool kF32 = false;
    __device__ uint4 pack(int, const float* v) const { return pack8(v); }
    __device__ void store(long long o, int n, const uint4& w) const {
        const int par = n / C, ci = n - par * C, W = WHICH == 3 ? g.W2 : g.W1;
        o += ((par & 2) ? W * C : 0) + ((par & 1) ? C : 0) + ci;
        st8((WHICH == 3 ? z.da2 : z.da1) + o, mask8(ld8((WHICH == 3 ? z.a2 : z.a1) + o), w));
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
// that nothing reads.  The bias gradient is the sum of dy's chunks, which
// the threads of the first N tile read back.
//   Op: dy() with lddy columns per row m; rows and steps of x as above; grad
// offsets out (with leading dimension ld) and bias; n_real columns are stored.
template <int KS>
constexpr uint64_t wg_sdesc_hi() {
    return (uint64_t(128 >> 4) << 16) | (uint64_t((KS * 16) >> 4) << 32) | (1ull << 46);
}
__device__ __forceinline__ void red_add_v4(float* p, const float* v) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3])
                 : "memory");
}

template <int BN, int KS, int AQ, int ST, class Op>  // AQ: 8-column chunks of dy per thread and step
__global__ void __launch_bounds__(TC_THREADS) wgrad_tc_kernel(const Op op, int M, int N, int K, int kchunk, int* status) {
    static_assert(BN % 16 == 0 && BN >= 16 && BN <= 256 && KS % 16 == 0 && TC_THREADS % KS == 0, "tile shape");
    constexpr int GR = TC_THREADS / KS;          // threads per row
    constexpr int BLK = KS * 16;                 // bytes of one 8-column block of a tile
    constexpr int BQ = (BN / 8 + GR - 1) / GR, A_BYTES = AQ * GR * BLK, STAGE = A_BYTES + (BN / 8) * BLK;
    constexpr int NCOL = tc_cols<BN>();
    constexpr uint32_t IDESC = tc_idesc<BN>() | (1u << 15) | (1u << 16);  // A and B transposed (M/N-major)
    extern __shared__ __align__(128) uint8_t tc_smem[];
    __shared__ __align__(8) unsigned long long tc_bar[ST];
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
#pragma unroll
        for (int s = 0; s < ST; s++) mbar_init(bar0 + 8 * s, 1);
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
    typename Op::Step steps[BQ];
#pragma unroll
    for (int j = 0; j < BQ; j++) steps[j] = op.step(n0 + 8 * (c0 + j * GR));
    const bf16_t* dyp = op.dy() + m0 + 8 * c0;
    auto load = [&](int it) {
        const int m = kb + it * KS + p;
        const uint32_t sa = sbase + uint32_t((it % ST) * STAGE + c0 * BLK) + off, sb = sa + A_BYTES;
        const bool live = m < ke;
        const int mr = live ? m : ke - 1;
        const typename Op::Row row = op.row(mr);
        const bf16_t* d = dyp + (long long)mr * Op::lddy;
#pragma unroll
        for (int j = 0; j < AQ; j++) cp16z(sa + uint32_t(j * GR * BLK), d + 8 * j * GR, live && c0 + j * GR < mblk, op.z.w);
#pragma unroll
        for (int j = 0; j < BQ; j++) {
            const int c = c0 + j * GR;
            if (c < BN / 8) stage_a8(op, sb + uint32_t(j * GR * BLK), row, steps[j], live && c < nblk);
        }
    };
#pragma unroll
    for (int s = 0; s < ST - 1; s++) {
        if (s < nk) load(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int it = 0; it < nk; it++) {
        const uint32_t sa = sbase + uint32_t((it % ST) * STAGE), sb = sa + A_BYTES;
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
        if (with_bias) {
#pragma unroll
            for (int j = 0; j < AQ; j++) {
                uint32_t w[4];
                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                             : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
                             : "r"(sa + uint32_t((c0 + j * GR) * BLK) + off)
                             : "memory");
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    bias[j][2 * i] += bf2f(bf16_t(w[i] & 0xffffu));
                    bias[j][2 * i + 1] += bf2f(bf16_t(w[i] >> 16));
                }
            }
        }
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
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar0 + 8 * (it % ST))
                         : "memory");
        }
        if (it + ST - 1 < nk) {
            // the stage's previous MMAs (step it - 1) have read it
            if (it >= 1) tc_wait(bar0 + 8 * ((it - 1) % ST), uint32_t((it - 1) / ST) & 1u, status);
            load(it + ST - 1);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (nk > 0) {
        tc_wait(bar0 + 8 * ((nk - 1) % ST), uint32_t((nk - 1) / ST) & 1u, status);
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

struct HeadBwdW : HeadFwd {  // M = 296, N = 256, K = B
    static constexpr int out = O_W5, ld = HID, bias = O_B5, n_real = HID, lddy = HEAD_N;
    __device__ const bf16_t* dy() const { return z.dl; }
};
struct Fc1BwdW : Fc1Fwd {  // M = 256, N = 1168, K = B
    static constexpr int out = O_W4, ld = FEAT, bias = O_B4, n_real = FEAT, lddy = HID;
    __device__ const bf16_t* dy() const { return z.dh; }
};
// conv weight gradient: M = 32, N = 9 C, K = pairs x output positions
template <class Fwd, int C, int OW, int OB>
struct ConvBwdW : Fwd {
    static constexpr int out = OW, ld = 9 * C, bias = OB, n_real = 9 * C, lddy = 32;
    __device__ const bf16_t* dy() const { return C == 16 ? this->z.da2 : this->z.da3; }
};
using Conv2BwdW = ConvBwdW<Conv2Fwd, 16, O_W2, O_B2>;
using Conv3BwdW = ConvBwdW<Conv3Fwd, 32, O_W3, O_B3>;
struct Conv1BwdW {  // M = 16, N = 18 (24 staged)
    Geo g; Bufs z;
    static constexpr int out = O_W1, ld = 18, bias = O_B1, n_real = 18, lddy = 16;
    using Row = Conv1Row;
    using Step = int;
    static constexpr bool kCalc = true;
    __device__ Row row(int m) const { return conv1_row(g, m); }
    __device__ Step step(int k) const { return k; }
    __device__ bool calc(Step) const { return true; }
    __device__ uint4 make(const Row& w, Step j) const {
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (j == 0)
            v = make_uint4(conv1_tap(w, g.cw, 0, 0), conv1_tap(w, g.cw, 0, 1), conv1_tap(w, g.cw, 0, 2), conv1_tap(w, g.cw, 1, 0));
        else if (j == 8)
            v = make_uint4(conv1_tap(w, g.cw, 1, 1), conv1_tap(w, g.cw, 1, 2), conv1_tap(w, g.cw, 2, 0), conv1_tap(w, g.cw, 2, 1));
        else
            v.x = conv1_tap(w, g.cw, 2, 2);
        return v;
    }
    __device__ bool a8(const Row&, Step, const bf16_t*&) const { return false; }
    __device__ const bf16_t* dy() const { return z.da1; }
};

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
    st8(da3 + o, mask8(ld8(a3 + o), pack8(s)));
}

// ---- loss, proposals, optimiser -------------------------------------------------
// One warp per sample: softmax over the 289 classes, the sample's share of the
// mean cross-entropy (atomically summed into *loss, in 64 bits) and dl = (p - onehot) / B
// in bf16 (zero for the 7 padding logits).
// The row stays in registers (HEAD_N = 296: ten values a lane).
__global__ void loss_kernel(const float* __restrict__ logits, const int16_t* __restrict__ labels, int B,
                            bf16_t* __restrict__ dl, double* __restrict__ loss) {
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
        double t = 0.0;
        for (int i = 0; i < int(blockDim.x >> 5); i++) t += double(part[i]);
        atomicAdd(loss, t);
    }
}
__global__ void loss_out_kernel(const double* __restrict__ loss, float* __restrict__ out) { *out = float(*loss); }

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

// Logits as integers of the same order (0: never chosen, as NaN and -inf are
// not), so that a round is two warp reductions, and only the lane that lost
// its largest looks for its next.  23 learned 720p pairs: 120 us with
// shuffle trees over (value, class), 93 now.
__device__ __forceinline__ void top8_one(const float* __restrict__ z, int32_t* __restrict__ o) {
    const int lane = threadIdx.x & 31;
    uint32_t v[10];
#pragma unroll
    for (int i = 0; i < 10; i++) {
        const int c = lane + 32 * i;
        const float f = c < NCLS ? z[c] + 0.f : -INFINITY;  // -0 counts as 0
        const uint32_t u = __float_as_uint(f);
        v[i] = f > -INFINITY ? ((u >> 31) ? ~u : u | 0x80000000u) : 0u;
    }
    uint32_t bv;
    int bc, mine = 1 << 30;
    auto largest = [&]() {
        bv = 0u;
        bc = 1 << 30;
#pragma unroll
        for (int i = 0; i < 10; i++)
            if (v[i] > bv) { bv = v[i]; bc = lane + 32 * i; }
    };
    largest();
    for (int r = 0; r < 8; r++) {
        const uint32_t m = __reduce_max_sync(0xffffffffu, bv);
        const int c = int(__reduce_min_sync(0xffffffffu, bv == m ? unsigned(bc) : unsigned(1 << 30)));
        if (c == bc) {
#pragma unroll
            for (int i = 0; i < 10; i++)
                if (lane + 32 * i == c) v[i] = 0u;
            largest();
        }
        __syncwarp();
        if (lane == r) mine = c;
    }
    if (lane < 8) {
        o[2 * lane] = 4 * (mine % 17 - 8);
        o[2 * lane + 1] = 4 * (mine / 17 - 8);
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
    for (int r = 0; r < WREP; r++) w[i + r * WSTRIDE] = f2bf(nw);
}

__global__ void to_bf16_kernel(const float* __restrict__ src, bf16_t* __restrict__ dst, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        for (int r = 0; r < WREP; r++) dst[i + r * WSTRIDE] = f2bf(src[i]);
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

// Each launcher has its kernel's opt-in to dynamic shared memory above 48 KB, an
// attribute of the current device (opt_in_kernels).
template <int BN, int MT, int ST>
constexpr int gemm_smem() {
    return ST * (MT * TC_BM + BN) * TC_BK * 2;
}
template <int BN, int MT, int ST, class Op>
static cudaError_t gemm_opt_in() {
    return cudaFuncSetAttribute(gemm_tc_kernel<BN, MT, ST, Op>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                gemm_smem<BN, MT, ST>());
}
template <int BN, int MT, int ST, class Op>
static void gemm(const Op& op, int M, int N, int K, cudaStream_t st) {
    constexpr int smem = gemm_smem<BN, MT, ST>();
    dim3 grid((M + MT * TC_BM - 1) / (MT * TC_BM), (N + BN - 1) / BN);
    gemm_tc_kernel<BN, MT, ST, Op><<<grid, TC_THREADS, smem, st>>>(op, M, N, K, op.z.status);
}

template <int BN, int KT, int ST, class Op>
static cudaError_t conv_gemm_opt_in() {
    return cudaFuncSetAttribute(conv_tc_kernel<BN, KT, ST, Op>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                conv_smem<BN, KT, ST>());
}
template <int BN, int KT, int ST, class Op>
static void conv_gemm(const Op& op, int M, int K, int sms, cudaStream_t st) {
    constexpr int smem = conv_smem<BN, KT, ST>(), fit = 226 * 1024 / (smem + 4096), per_sm = fit < 4 ? fit : 4;
    static_assert(per_sm >= 1 && per_sm * tc_cols<2 * BN>() <= 512, "shared and tensor memory");
    const int tiles = (M + TC_BM - 1) / TC_BM;
    conv_tc_kernel<BN, KT, ST, Op><<<std::min(tiles, per_sm * sms), TC_THREADS, smem, st>>>(op, M, K, op.z.status);
}

// Weight-gradient GEMM: K split over the CTAs that shared and tensor memory
// and the threads let stay resident, at least four steps each.
template <int BN, int KS, int AQ, int ST>
constexpr int wgrad_smem() {
    constexpr int GR = TC_THREADS / KS, BLK = KS * 16, A_BYTES = AQ * GR * BLK, STAGE = A_BYTES + (BN / 8) * BLK;
    // the MMA reads 16 blocks of A whatever there are: 16 * BLK from the last stage's start
    return (ST - 1) * STAGE + (STAGE > 16 * BLK ? STAGE : 16 * BLK);
}
template <int BN, int KS, int AQ, int ST, class Op>
static cudaError_t wgrad_opt_in() {
    return cudaFuncSetAttribute(wgrad_tc_kernel<BN, KS, AQ, ST, Op>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                wgrad_smem<BN, KS, AQ, ST>());
}
template <int BN, int KS, int AQ, int ST, class Op>
static void wgrad(const Op& op, int M, int N, int K, int sms, cudaStream_t st) {
    constexpr int smem = wgrad_smem<BN, KS, AQ, ST>();
    constexpr int by_smem = 224 * 1024 / (smem + 2048), by_tmem = 512 / tc_cols<BN>();
    constexpr int resident = by_smem < by_tmem ? (by_smem < 4 ? by_smem : 4) : (by_tmem < 4 ? by_tmem : 4);
    static_assert(resident >= 1, "shared memory");
    const int tiles = ((M + TC_BM - 1) / TC_BM) * ((N + BN - 1) / BN);
    int splits = resident * sms / tiles;
    splits = std::max(1, std::min(splits, (K + 4 * KS - 1) / (4 * KS)));
    int kchunk = (K + splits - 1) / splits;
    kchunk = (kchunk + KS - 1) / KS * KS;
    dim3 grid((M + TC_BM - 1) / TC_BM, (N + BN - 1) / BN, (K + kchunk - 1) / kchunk);
    wgrad_tc_kernel<BN, KS, AQ, ST, Op><<<grid, TC_THREADS, smem, st>>>(op, M, N, K, kchunk, op.z.status);
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
    double* loss = nullptr;
    int* status = nullptr;  // mapped host word: non-zero once a kernel's wait has run out
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
    if (n->status) cudaFreeHost(n->status);
    delete n;
}

// An earlier batch's kernel may have given up a wait: its results are not to be
// used, and the net says so at the next call (no synchronisation here).
// h264a_mvnet_set_params starts afresh.
int check_waits(const h264a_mvnet* n) {
    if (n && *const_cast<const volatile int*>(n->status) != 0)
        return fail(H264A_E_TIMEOUT, "mvnet: a wait of an earlier batch ran out (status 4); its results are not valid");
    return H264A_OK;
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
    z.status = n->status;  // mapped: one address on host and device
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
    const int m1 = g.P * g.H1 * g.W1;
    conv1_kernel<<<std::min((m1 + 127) / 128, n->sms * C1_CTAS), 128, 0, st>>>(g, z, m1, z.status);
    conv_gemm<32, 3, 3>(Conv2Fwd{g, z}, g.P * g.H2 * g.W2, 144, n->sms, st);
    conv_gemm<32, 5, 3>(Conv3Fwd{g, z}, g.P * g.H3 * g.W3, 288, n->sms, st);
}

void head_forward(h264a_mvnet* n, const Geo& g, float* logits, cudaStream_t st) {
    Bufs z = bufs(n);
    z.logits = logits;
    const int B = g.P * g.nmb;
    // FC1's weights (600 KB) cross the L2 once per row tile: 256-row tiles halve
    // that, and keep every SM busy from two 128-row tiles per SM on (four 1080p
    // pairs, 32,640 samples: 76 us with 128 rows, 61 with 256; below, the
    // smaller tile spreads the samples over more SMs)
    if (B > TC_BM * n->sms)
        gemm<256, 2, 3>(Fc1Fwd{g, z}, B, HID, FEAT, st);
    else
        gemm<256, 1, 2>(Fc1Fwd{g, z}, B, HID, FEAT, st);
    gemm<160, 1, 3>(HeadFwd{z}, B, HEAD_N, HID, st);
}

void backward(h264a_mvnet* n, const Geo& g, cudaStream_t st) {
    const Bufs z = bufs(n);
    const int B = g.P * g.nmb, S = n->sms;
    const int K3 = g.P * g.H3 * g.W3, K2 = g.P * g.H2 * g.W2, K1 = g.P * g.H1 * g.W1;
    prep_kernel<<<(N_PREP + 255) / 256, 256, 0, st>>>(n->w, n->wprep);
    wgrad<256, 64, 4, 2>(HeadBwdW{{z}}, HEAD_N, HID, B, S, st);
    gemm<256, 1, 2>(HeadBwdData{z}, B, HID, HEAD_N, st);
    wgrad<256, 64, 4, 2>(Fc1BwdW{{g, z}}, HID, FEAT, B, S, st);
    gemm<192, 1, 2>(Fc1BwdData{z}, B, CONVF, HID, st);
    const long long cells = (long long)K3 * 4;
    uncrop_kernel<<<unsigned((cells + 255) / 256), 256, 0, st>>>(g, n->df, n->a3, n->da3);
    wgrad<144, 64, 1, 3>(Conv3BwdW{{g, z}}, 32, 288, K3, S, st);
    conv_gemm<128, 2, 2>(ConvBwdData<32, 3>{g, z}, K3, 128, S, st);
    wgrad<144, 128, 2, 2>(Conv2BwdW{{g, z}}, 32, 144, K2, S, st);
    conv_gemm<64, 2, 3>(ConvBwdData<16, 2>{g, z}, K2, 128, S, st);
    wgrad<32, 128, 1, 2>(Conv1BwdW{g, z}, 16, 24, K1, S, st);
}

// Every instantiation launched above, on the current device.
static int opt_in_kernels() {
    H264A_CUDA((conv_gemm_opt_in<32, 3, 3, Conv2Fwd>()));
    H264A_CUDA((conv_gemm_opt_in<32, 5, 3, Conv3Fwd>()));
    H264A_CUDA((gemm_opt_in<256, 2, 3, Fc1Fwd>()));
    H264A_CUDA((gemm_opt_in<256, 1, 2, Fc1Fwd>()));
    H264A_CUDA((gemm_opt_in<160, 1, 3, HeadFwd>()));
    H264A_CUDA((wgrad_opt_in<256, 64, 4, 2, HeadBwdW>()));
    H264A_CUDA((gemm_opt_in<256, 1, 2, HeadBwdData>()));
    H264A_CUDA((wgrad_opt_in<256, 64, 4, 2, Fc1BwdW>()));
    H264A_CUDA((gemm_opt_in<192, 1, 2, Fc1BwdData>()));
    H264A_CUDA((wgrad_opt_in<144, 64, 1, 3, Conv3BwdW>()));
    H264A_CUDA((conv_gemm_opt_in<128, 2, 2, ConvBwdData<32, 3>>()));
    H264A_CUDA((wgrad_opt_in<144, 128, 2, 2, Conv2BwdW>()));
    H264A_CUDA((conv_gemm_opt_in<64, 2, 3, ConvBwdData<16, 2>>()));
    H264A_CUDA((wgrad_opt_in<32, 128, 1, 2, Conv1BwdW>()));
    return H264A_OK;
}

}  // namespace

extern "C" int h264a_mvnet_create(int device, uint64_t seed, h264a_mvnet** out) {
    if (!out) return fail(H264A_E_ARG, "mvnet_create: null out");
    *out = nullptr;
    H264A_CUDA(cudaSetDevice(device));
    int rc = opt_in_kernels();
    if (rc) return rc;
    h264a_mvnet* n = new h264a_mvnet();
    n->device = device;
    cudaDeviceGetAttribute(&n->sms, cudaDevAttrMultiProcessorCount, device);
    if (!rc) rc = dmalloc(&n->master, NPARAMS);
    if (!rc) rc = dmalloc(&n->w, size_t(WREP) * WSTRIDE);
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
    if (!rc) rc = dmalloc(&n->wprep, size_t(WREP) * N_PREP);
    if (!rc) rc = dmalloc(&n->loss, 1);
    if (!rc && cudaHostAlloc(reinterpret_cast<void**>(&n->status), sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        rc = fail(H264A_E_NOMEM, "mvnet: cudaHostAlloc failed");
    }
    if (!rc) *n->status = 0;
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
    *n->status = 0;  // the device is idle here
    H264A_CUDA(cudaMemset(n->m1, 0, sizeof(float) * NPARAMS));
    H264A_CUDA(cudaMemset(n->m2, 0, sizeof(float) * NPARAMS));
    n->step = 0;
    return H264A_OK;
}

extern "C" int h264a_mvnet_get_params(h264a_mvnet* n, float* h_params) {
    if (!n || !h_params) return fail(H264A_E_ARG, "mvnet_get_params: null pointer");
    H264A_CUDA(cudaSetDevice(n->device));
    H264A_CUDA(cudaDeviceSynchronize());
    const int rc = check_waits(n);
    if (rc) return rc;
    H264A_CUDA(cudaMemcpy(h_params, n->master, sizeof(float) * NPARAMS, cudaMemcpyDeviceToHost));
    return H264A_OK;
}

extern "C" int h264a_mvnet_forward(h264a_mvnet* n, const h264a_mvnet_pair* d_pairs, int npairs, int cw, int ch,
                                   const int16_t* d_nmv, float* d_logits, void* stream) {
    int rc = check_geo(n, d_pairs, npairs, cw, ch, d_nmv);
    if (!rc) rc = check_waits(n);
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
    rc = check_waits(n);
    if (rc) return rc;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const Geo g = make_geo(d_pairs, npairs, cw, ch, d_nmv, d_labels);
    const int B = npairs * g.nmb;
    H264A_CUDA(cudaMemsetAsync(n->grad, 0, sizeof(float) * NPARAMS, st));
    H264A_CUDA(cudaMemsetAsync(n->loss, 0, sizeof(double), st));
    trunk_forward(n, g, st);
    head_forward(n, g, n->logits, st);
    loss_kernel<<<(B * 32 + 255) / 256, 256, 0, st>>>(n->logits, d_labels, B, n->dl, n->loss);
    backward(n, g, st);
    if (d_grads) H264A_CUDA(cudaMemcpyAsync(d_grads, n->grad, sizeof(float) * NPARAMS, cudaMemcpyDeviceToDevice, st));
    if (d_loss) loss_out_kernel<<<1, 1, 0, st>>>(n->loss, d_loss);
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
    const int wrc = check_waits(n);
    if (wrc) return wrc;
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

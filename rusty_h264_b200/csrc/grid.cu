// grid.cu -- exhaustive full-pel cost grids: 16x16 SAD and SATD of every
// integer offset within ±R of each MB's centre, the distortions the ME cost
// functions return at full-pel MVs (mc_sad_hp / mc_satd_hp,
// crates/rusty_h264-encoder/src/mb16.rs:1930-2074), and the per-MB argmin of
// dist + (λ·bits(mv − pmv)) in raster order with first-wins ties, the order of
// the exhaustive probe in motion_search (mb16.rs:2889-2900).
//
// The (16+2R)² search window of an MB (edge reads clamped, i.e. read from the
// padded F plane with clamping) is staged once in shared memory.
//  * SAD (fullpel_sad_kernel): a work item is one column offset and a run of
//    GRID_K row offsets; every window row is loaded and byte-aligned once and
//    feeds the GRID_K candidates it overlaps with one packed __vsadu4 per 4
//    pixels, the source MB in registers.  A CTA takes `mbs` consecutive MBs,
//    chosen on the host so that their items fill whole rounds of its threads
//    (3 at R = 32: 975 items in four rounds of 256).  The argmin skips the
//    lambda*rate of a candidate whose distortion alone cannot beat the
//    thread's best (exact: a thread meets its candidates in scan order).
//  * SATD (fullpel_satd_kernel): one CTA per MB.  The Hadamard transform is
//    linear, so the predictions' 4x4 blocks are transformed once per window
//    position (77^2 at R = 32) instead of once per candidate and block
//    (16 * 65^2); a candidate's SATD is then 16 packed maxima a block.
#include <algorithm>

#include "h264a_device.cuh"

namespace h264a {

constexpr int GRID_K = 13;      // row offsets per SAD work item
constexpr int GRID_THREADS = 256;

struct GridArgs {
    Planes P;
    const uint8_t* src;
    int cw, ch, mb_w, R;
    const int32_t* centers;
    const int32_t* pmv;
    int metric, kind;
    const uint16_t* tab;
    double lambda;
    int32_t* sad_grid;
    int32_t* satd_grid;
    int32_t* best;
};

__device__ __forceinline__ uint32_t win_word(const uint8_t* row, int x) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(row + (x & ~3));
    const uint32_t sh = uint32_t(x & 3) * 8u;
    return sh ? __funnelshift_r(w[0], w[1], sh) : w[0];
}

// Stages the clamped window of MB (lx, ly) with full-pel centre (cxf, cyf):
// window (x, y) = picture (lx+cxf-R+x, ly+cyf-R+y), rows `ws` .. `wrows`-1
// and columns past `ws` zero (the reads of the last partial chunk and the
// fifth word of an unaligned read land there).  Row per warp, lanes along it.
__device__ __forceinline__ void stage_grid_window(uint8_t* win, const Planes& P, int lx, int ly, int cxf, int cyf,
                                                  int R, int ws, int pitch, int wrows, int row0, int rstep) {
    const int ox = lx + cxf - R + P.pad, oy = ly + cyf - R + P.pad;
    for (int y = row0; y < wrows; y += rstep) {
        const uint8_t* prow = P.base + (long long)clampi(oy + y, 0, P.ph - 1) * P.pw;
        for (int x = threadIdx.x & 31; x < pitch; x += 32)
            win[y * pitch + x] = (y < ws && x < ws) ? __ldg(prow + clampi(ox + x, 0, P.pw - 1)) : uint8_t(0);
    }
}

__device__ __forceinline__ long long grid_cost(const GridArgs& a, int dist, int mvx, int mvy, int pmx, int pmy) {
    return dist + lam_cost(a.lambda, mvbits(a.kind, a.tab, mvx - pmx) + mvbits(a.kind, a.tab, mvy - pmy));
}

// The argmin record of MB mb from its best key (cost << 32 | scan index).
__device__ __forceinline__ void grid_store_best(const GridArgs& a, int mb, long long key, int cxf, int cyf, int pmx,
                                                int pmy) {
    const int n = 2 * a.R + 1;
    const int idx = int(key & 0xffffffffLL);
    const long long cost = key >> 32;
    const int dyi = idx / n, dxi = idx % n;
    const int mvx = (cxf + dxi - a.R) * 4, mvy = (cyf + dyi - a.R) * 4;
    const long long rc = lam_cost(a.lambda, mvbits(a.kind, a.tab, mvx - pmx) + mvbits(a.kind, a.tab, mvy - pmy));
    a.best[4 * mb + 0] = mvx;
    a.best[4 * mb + 1] = mvy;
    a.best[4 * mb + 2] = int32_t(cost > 0x7fffffffLL ? 0x7fffffffLL : cost);
    a.best[4 * mb + 3] = int32_t(cost - rc);
}

__device__ __forceinline__ void grid_center(const GridArgs& a, int mb, int& cxf, int& cyf, int& pmx, int& pmy) {
    cxf = cyf = 0;
    if (a.centers) {
        cxf = (a.centers[2 * mb] + 2) >> 2;  // snapped like motion_search's integer snap
        cyf = (a.centers[2 * mb + 1] + 2) >> 2;
    }
    pmx = a.pmv ? a.pmv[2 * mb] : 0;
    pmy = a.pmv ? a.pmv[2 * mb + 1] : 0;
}

constexpr int SAD_MAX_MBS = 8;

// SAD grid and argmin of MBs mbs*blockIdx.x .. +mbs-1 (of nmb); dynamic
// shared memory: mbs windows of win_bytes.
__global__ void __launch_bounds__(GRID_THREADS, 2) fullpel_sad_kernel(GridArgs a, int mbs, int nmb, int win_bytes) {
    extern __shared__ __align__(16) uint8_t wins[];
    __shared__ __align__(16) uint32_t src_s[SAD_MAX_MBS][16][4];
    __shared__ unsigned long long best_s[SAD_MAX_MBS];
    const int R = a.R, n = 2 * R + 1;
    const int ws = 16 + 2 * R, pitch = (ws + 4 + 3) & ~3, wrows = ws + GRID_K;
    const int mb0 = blockIdx.x * mbs;
    const int nm = nmb - mb0 < mbs ? nmb - mb0 : mbs;
    const int nwarps = blockDim.x >> 5;
    for (int q = 0; q < nm; q++) {
        const int mb = mb0 + q;
        int cxf, cyf, pmx, pmy;
        grid_center(a, mb, cxf, cyf, pmx, pmy);
        stage_grid_window(wins + q * win_bytes, a.P, (mb % a.mb_w) * 16, (mb / a.mb_w) * 16, cxf, cyf, R, ws, pitch,
                          wrows, threadIdx.x >> 5, nwarps);
    }
    for (int t = threadIdx.x; t < nm * 64; t += blockDim.x) {
        const int q = t >> 6, r = (t >> 2) & 15, c = t & 3, mb = mb0 + q;
        src_s[q][r][c] = ld4u(a.src + (long long)((mb / a.mb_w) * 16 + r) * a.cw + (mb % a.mb_w) * 16 + 4 * c);
    }
    if (threadIdx.x < SAD_MAX_MBS) best_s[threadIdx.x] = ULLONG_MAX;
    __syncthreads();
    const bool argmin = a.metric == 0;
    const int chunks = (n + GRID_K - 1) / GRID_K, per_mb = n * chunks;
    for (int item = threadIdx.x; item < nm * per_mb; item += blockDim.x) {
        const int q = item / per_mb, it = item - q * per_mb;
        const int mb = mb0 + q;
        const int dxi = it % n, dy0 = (it / n) * GRID_K;
        const uint32_t sh = uint32_t(dxi & 3) * 8u;
        const uint8_t* win = wins + q * win_bytes;
        uint32_t s[16][4];
#pragma unroll
        for (int r = 0; r < 16; r++) {
            const uint4 v = *reinterpret_cast<const uint4*>(&src_s[q][r][0]);
            s[r][0] = v.x; s[r][1] = v.y; s[r][2] = v.z; s[r][3] = v.w;
        }
        int acc[GRID_K];
#pragma unroll
        for (int k = 0; k < GRID_K; k++) acc[k] = 0;
#pragma unroll
        for (int i = 0; i < GRID_K + 15; i++) {
            // the row's 16 bytes at dxi: five aligned words and funnel shifts
            const uint32_t* rw = reinterpret_cast<const uint32_t*>(win + (dy0 + i) * pitch + (dxi & ~3));
            uint32_t a5[5];
#pragma unroll
            for (int c = 0; c < 5; c++) a5[c] = rw[c];
            uint32_t w[4];
#pragma unroll
            for (int c = 0; c < 4; c++) w[c] = __funnelshift_r(a5[c], a5[c + 1], sh);
#pragma unroll
            for (int k = 0; k < GRID_K; k++) {
                const int r = i - k;
                if (r >= 0 && r < 16)
                    acc[k] += int(__vsadu4(s[r][0], w[0]) + __vsadu4(s[r][1], w[1]) + __vsadu4(s[r][2], w[2]) +
                                  __vsadu4(s[r][3], w[3]));
            }
        }
        int cxf, cyf, pmx, pmy;
        grid_center(a, mb, cxf, cyf, pmx, pmy);
        long long best_key = LLONG_MAX;  // this item's (cost << 32 | scan index) minimum
#pragma unroll
        for (int k = 0; k < GRID_K; k++) {
            const int dyi = dy0 + k;
            if (dyi < n) {
                const int idx = dyi * n + dxi;
                if (a.sad_grid) a.sad_grid[(long long)mb * n * n + idx] = acc[k];
                if (argmin && acc[k] < int(best_key >> 32)) {  // lambda*rate >= 0: a larger distortion cannot win
                    const long long key = (grid_cost(a, acc[k], (cxf + dxi - R) * 4, (cyf + dyi - R) * 4, pmx, pmy)
                                           << 32) | (long long)idx;
                    best_key = key < best_key ? key : best_key;
                }
            }
        }
        if (argmin && best_key != LLONG_MAX) atomicMin(&best_s[q], (unsigned long long)best_key);
    }
    __syncthreads();
    if (argmin && a.best && threadIdx.x < nm) {
        const int mb = mb0 + threadIdx.x;
        int cxf, cyf, pmx, pmy;
        grid_center(a, mb, cxf, cyf, pmx, pmy);
        grid_store_best(a, mb, (long long)best_s[threadIdx.x], cxf, cyf, pmx, pmy);
    }
}

// The 4x4 Hadamard coefficients of a block (4 row words) as eight words of two
// 16-bit halves, SATD_BIAS added to each: |coefficient| <= 8 * 255 but for the
// sum of all pixels, so every half is 0 .. 6120.  Two columns' worth per 32-bit
// integer (lo + 65536 * hi): the vertical butterflies are plain adds, and the
// bias on row 0 reaches every output.
constexpr int SATD_BIAS = 2040;
__device__ __forceinline__ int dot4_us(uint32_t pix, uint32_t coef, int acc) {  // unsigned bytes x signed bytes
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(pix), "r"(coef), "r"(acc));
    return d;
}
__device__ __forceinline__ void had_words(const uint32_t w[4], uint32_t o[8]) {
    int x[4], y[4];
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const int b = r == 0 ? SATD_BIAS : 0;
        x[r] = dot4_us(w[r], 0x01010101u, b) + dot4_us(w[r], 0xffff0101u, b) * 65536;
        y[r] = dot4_us(w[r], 0x01ffff01u, b) + dot4_us(w[r], 0xff01ff01u, b) * 65536;
    }
    const int a = x[0] + x[1], b = x[0] - x[1], c = x[2] + x[3], d = x[2] - x[3];
    o[0] = uint32_t(a + c), o[1] = uint32_t(a - c), o[2] = uint32_t(b + d), o[3] = uint32_t(b - d);
    const int e = y[0] + y[1], f = y[0] - y[1], g = y[2] + y[3], h = y[2] - y[3];
    o[4] = uint32_t(e + g), o[5] = uint32_t(e - g), o[6] = uint32_t(f + h), o[7] = uint32_t(f - h);
}

// SATD grid and argmin, one CTA per MB.
//
// With the biased coefficients P of a prediction block and S of a source
// block, sum |P - S| = 2 sum max(P, S) - sum P - sum S, and sum P = 16 times
// the block's first pixel + 16 * SATD_BIAS (a Hadamard matrix's rows sum to
// its first column).  Per (candidate, block) that is eight packed maxima, four
// three-operand adds (a half's sum stays below 2^16; the ninth addend is the
// first pixel's share, SATD_BIAS - 8 * pixel >= 0) and one dp2a.
//
// Offsets with row dy = ph (mod 4) use window rows ph (mod 4) only: a stage
// transforms the rows of `ps` such phases and `g` runs of SATD_J candidates
// down (4 rows apart) into shared memory, then a thread takes one column
// offset and one run: SATD_J + 3 positions per block column, each met by up to
// four candidates, with the column's four source blocks in registers.  Bound
// by the integer pipes: 4 million packed operations a MB at R = 32.  3,600
// MBs, R = 32: 1,833 us transforming every candidate's blocks, 463 now (the
// integer pipe 60% busy, barriers between the stages most of the rest; runs of
// 9 candidates 531).
//
// Dynamic shared memory: the window, then per stage position two uint4 of
// coefficients and one word.
constexpr int SATD_J = 6;
__host__ __device__ constexpr int satd_rows(int ps, int g) { return ps * (SATD_J * g + 3); }
__global__ void __launch_bounds__(GRID_THREADS) fullpel_satd_kernel(GridArgs a, int ps, int g) {
    extern __shared__ __align__(16) uint8_t win[];
    __shared__ long long red_key[GRID_THREADS / 32];
    __shared__ __align__(16) uint32_t hs[16][8];  // source blocks [4 * by + bx]
    __shared__ int ksum;
    const int mb = blockIdx.x;
    const int lx = (mb % a.mb_w) * 16, ly = (mb / a.mb_w) * 16;
    const int R = a.R, n = 2 * R + 1;
    int cxf, cyf, pmx, pmy;
    grid_center(a, mb, cxf, cyf, pmx, pmy);
    const int ws = 16 + 2 * R, pitch = (ws + 4 + 3) & ~3;
    stage_grid_window(win, a.P, lx, ly, cxf, cyf, R, ws, pitch, ws, threadIdx.x >> 5, blockDim.x >> 5);
    if (threadIdx.x < 32) {
        const int b = threadIdx.x & 15;
        uint32_t w[4], o[8];
#pragma unroll
        for (int r = 0; r < 4; r++) w[r] = ld4u(a.src + (long long)(ly + 4 * (b >> 2) + r) * a.cw + lx + 4 * (b & 3));
        had_words(w, o);
#pragma unroll
        for (int i = 0; i < 8; i++) hs[b][i] = o[i];
        int s = int(w[0] & 0xffu);
#pragma unroll
        for (int i = 8; i > 0; i >>= 1) s += __shfl_xor_sync(0xffffffffu, s, i);
        if (threadIdx.x == 0) ksum = 8 * s + 16 * (SATD_BIAS + 16 * SATD_BIAS);
    }
    const int wx = n + 12, prows = SATD_J * g + 3, npos = satd_rows(ps, g) * wx;
    uint4* h0 = reinterpret_cast<uint4*>(win + ((size_t(ws) * pitch + 15) & ~size_t(15)));
    uint4* h1 = h0 + npos;
    uint32_t* ex = reinterpret_cast<uint32_t*>(h1 + npos);
    __syncthreads();
    const int k_mb = ksum;

    long long best_key = LLONG_MAX;  // (cost << 32) | scan index; min = first-wins argmin
    const long long grid_base = (long long)mb * n * n;
    // rates are below 2^17: up to this lambda a cost is its distortion and a
    // product >= 0, and fits 31 bits
    const bool argmin = a.metric == 1, rate_pos = a.lambda >= 0.0 && a.lambda <= 8192.0;
    for (int ph0 = 0; ph0 < 4; ph0 += ps)
        for (int j0 = 0; ph0 + 4 * j0 < n; j0 += SATD_J * g) {
            for (int i = threadIdx.x; i < npos; i += blockDim.x) {
                const int row = i / wx, x = i - row * wx, p = row / prows;
                const int y0 = ph0 + p + 4 * (j0 + row - p * prows);
                uint32_t w[4], o[8];
#pragma unroll
                for (int r = 0; r < 4; r++) w[r] = win_word(win + min(y0 + r, ws - 1) * pitch, x);  // past the window: unused
                had_words(w, o);
                h0[i] = make_uint4(o[0], o[1], o[2], o[3]);
                h1[i] = make_uint4(o[4], o[5], o[6], o[7]);
                ex[i] = uint32_t(SATD_BIAS) - 8u * (w[0] & 0xffu);
            }
            __syncthreads();
            for (int item = threadIdx.x; item < ps * g * n; item += blockDim.x) {
                const int u = item / n, dxi = item - u * n, p = u / g, c = u - p * g;
                uint32_t acc[SATD_J];
#pragma unroll
                for (int j = 0; j < SATD_J; j++) acc[j] = 0;
#pragma unroll 1
                for (int bx = 0; bx < 4; bx++) {
                    uint4 s0[4], s1[4];
#pragma unroll
                    for (int by = 0; by < 4; by++) {
                        s0[by] = *reinterpret_cast<const uint4*>(&hs[4 * by + bx][0]);
                        s1[by] = *reinterpret_cast<const uint4*>(&hs[4 * by + bx][4]);
                    }
                    const int at = (p * prows + c * SATD_J) * wx + dxi + 4 * bx;
#pragma unroll
                    for (int k = 0; k < SATD_J + 3; k++) {
                        const uint4 v0 = h0[at + k * wx], v1 = h1[at + k * wx];
                        const uint32_t e = ex[at + k * wx];
#pragma unroll
                        for (int by = 0; by < 4; by++) {
                            const int j = k - by;
                            if (j < 0 || j >= SATD_J) continue;
                            const uint32_t t = e + __vmaxu2(v0.x, s0[by].x) + __vmaxu2(v0.y, s0[by].y) +
                                               __vmaxu2(v0.z, s0[by].z) + __vmaxu2(v0.w, s0[by].w) +
                                               __vmaxu2(v1.x, s1[by].x) + __vmaxu2(v1.y, s1[by].y) +
                                               __vmaxu2(v1.z, s1[by].z) + __vmaxu2(v1.w, s1[by].w);
                            acc[j] = __dp2a_lo(t, 0x0101u, acc[j]);
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j < SATD_J; j++) {
                    const int dyi = ph0 + p + 4 * (j0 + c * SATD_J + j);
                    if (dyi >= n) continue;
                    const int idx = dyi * n + dxi, dist = 2 * (int(acc[j]) - k_mb);
                    if (a.satd_grid) a.satd_grid[grid_base + idx] = dist;
                    // a larger distortion than the best cost cannot win then
                    if (argmin && (!rate_pos || (long long)dist <= (best_key >> 32))) {
                        const long long key =
                            (grid_cost(a, dist, (cxf + dxi - R) * 4, (cyf + dyi - R) * 4, pmx, pmy) << 32) | (long long)idx;
                        best_key = key < best_key ? key : best_key;
                    }
                }
            }
            __syncthreads();
        }
    if (!argmin) return;
    // ---- argmin over the CTA ----
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const long long other = __shfl_xor_sync(0xffffffffu, best_key, o);
        best_key = other < best_key ? other : best_key;
    }
    if ((threadIdx.x & 31) == 0) red_key[threadIdx.x >> 5] = best_key;
    __syncthreads();
    if (threadIdx.x == 0 && a.best) {
        long long k = red_key[0];
        for (int i = 1; i < int(blockDim.x >> 5); i++) k = red_key[i] < k ? red_key[i] : k;
        grid_store_best(a, mb, k, cxf, cyf, pmx, pmy);
    }
}

}  // namespace h264a

using namespace h264a;

extern "C" int h264a_fullpel_grid(h264a_ctx* ctx, const h264a_picture* h_pic, int R, const int32_t* d_centers,
                                  const int32_t* d_pmv, int metric, int mv_cost_kind, const uint16_t* d_mv_cost_tab,
                                  double lambda, int32_t* d_sad_grid, int32_t* d_satd_grid, int32_t* d_best,
                                  void* stream) {
    if (!ctx || !h_pic || !h_pic->d_src || !h_pic->d_planes) return fail(H264A_E_ARG, "fullpel_grid: null pointer");
    if (R < 1 || R > 64) return fail(H264A_E_ARG, "fullpel_grid: 1 <= R <= 64");
    if (metric != 0 && metric != 1) return fail(H264A_E_ARG, "fullpel_grid: metric 0 (SAD) or 1 (SATD)");
    if ((mv_cost_kind == 1 || mv_cost_kind == 2) && !d_mv_cost_tab)
        return fail(H264A_E_ARG, "fullpel_grid: mv cost kinds 1 and 2 need a table");
    const h264a_picture& pc = *h_pic;
    if (pc.cw < 16 || pc.ch < 16 || pc.cw % 16 || pc.ch % 16 || pc.pad < 3 || pc.pad > 128)
        return fail(H264A_E_ARG, "fullpel_grid: MB-aligned picture with 3 <= pad <= 128");
    GridArgs a;
    a.P.base = pc.d_planes;
    a.P.pad = pc.pad;
    a.P.pw = pc.cw + 2 * pc.pad;
    a.P.ph = pc.ch + 2 * pc.pad;
    a.P.ps = (long long)a.P.pw * a.P.ph;
    a.src = pc.d_src;
    a.cw = pc.cw;
    a.ch = pc.ch;
    a.mb_w = pc.cw / 16;
    a.R = R;
    a.centers = d_centers;
    a.pmv = d_pmv;
    a.metric = metric;
    a.kind = mv_cost_kind;
    a.tab = d_mv_cost_tab;
    a.lambda = lambda;
    a.sad_grid = d_sad_grid;
    a.satd_grid = d_satd_grid;
    a.best = d_best;
    const int ws = 16 + 2 * R;
    const int pitch = (ws + 4 + 3) & ~3;
    const size_t smem = (size_t)(ws + GRID_K) * pitch;  // one window
    const int nmb = (pc.cw / 16) * (pc.ch / 16);
    cudaStream_t st = pick_stream(ctx, stream);
    // one launch per metric wanted (its grid, or the argmin's metric)
    if (d_sad_grid || metric == 0) {
        // MBs per CTA: the most even fill of whole rounds of GRID_THREADS
        // items, at most SAD_MAX_MBS windows and SAD_SMEM (two CTAs per SM)
        constexpr size_t SAD_SMEM = 100 * 1024;
        const int n = 2 * R + 1, per_mb = n * ((n + GRID_K - 1) / GRID_K);
        const int win_bytes = int((smem + 15) & ~size_t(15));
        int mbs = 1;
        double best_fill = 0.0;
        for (int m = 1; m <= SAD_MAX_MBS && size_t(m) * win_bytes <= SAD_SMEM; m++) {
            const int rounds = (m * per_mb + GRID_THREADS - 1) / GRID_THREADS;
            const double fill = double(m * per_mb) / double(rounds * GRID_THREADS);
            if (fill > best_fill + 1e-9) {
                best_fill = fill;
                mbs = m;
            }
        }
        const size_t sm = size_t(mbs) * win_bytes;
        if (sm > 48 * 1024)
            H264A_CUDA(cudaFuncSetAttribute(fullpel_sad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(SAD_SMEM)));
        fullpel_sad_kernel<<<unsigned((nmb + mbs - 1) / mbs), GRID_THREADS, sm, st>>>(a, mbs, nmb, win_bytes);
        const int rc = check_launch("fullpel_sad_kernel");
        if (rc) return rc;
    }
    if (d_satd_grid || metric == 1) {
        // runs of SATD_J candidates and phases per stage: as many as give a
        // thread each up to a CTA's threads and fit SATD_SMEM (R = 32: one
        // phase's three runs, 195 threads, three CTAs per SM)
        constexpr size_t SATD_SMEM = 72 * 1024;
        const int n = 2 * R + 1, nj = (n + 3) / 4, runs = (nj + SATD_J - 1) / SATD_J;
        const size_t wbytes = (size_t(ws) * pitch + 15) & ~size_t(15);
        auto need = [&](int ps, int g) { return wbytes + size_t(satd_rows(ps, g)) * (n + 12) * 36; };
        int ps = 1, g = 1;
        while (g < runs && (g + 1) * n <= GRID_THREADS && need(1, g + 1) <= SATD_SMEM) g++;
        while (g == runs && ps < 4 && 2 * ps * g * n <= GRID_THREADS && need(2 * ps, g) <= SATD_SMEM) ps *= 2;
        const size_t sm = need(ps, g);
        if (sm > 48 * 1024)
            H264A_CUDA(cudaFuncSetAttribute(fullpel_satd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(SATD_SMEM)));
        const int threads = std::min(GRID_THREADS, (ps * g * n + 31) / 32 * 32);
        fullpel_satd_kernel<<<nmb, threads, sm, st>>>(a, ps, g);
        const int rc = check_launch("fullpel_satd_kernel");
        if (rc) return rc;
    }
    return H264A_OK;
}

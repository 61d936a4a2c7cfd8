// lookahead.cu -- a16-a19: the mb-tree lookahead's per-frame costs
// (crates/rusty_h264-encoder/src/mbtree.rs:61-263).
//
//  * downsample2x: one thread per 4 x 4 output pixels, 8-byte loads.
//  * intra_cost: one lane per 4x4 sub-block, Σ|Hadamard AC| reduced per MB.
//  * inter_cost + frame_costs: the seeded full-pel diamond.  The seed chain
//    (left MV, else top MV; mbtree.rs:225-231) makes every row a sequential
//    chain that starts from column 0, and column 0 a chain down the frame.
//    Frames are independent (source domain, f against f-1).  One persistent
//    kernel deals the column-0 chains first (publishing each MB's flag as it
//    finishes), then the rows in row order across frames: a row waits (bounded)
//    only for its own column-0 MB, so rows start while column 0 is still
//    walking down the frame.  Inside a search the ring points of the cascading
//    diamond are priced together and the first improvement taken, the rest of
//    the ring priced again around the moved centre (the reference's evaluation
//    order).
//    HalfRes mode (the default) has a kernel of its own, one chain per warp:
//    see la_half_kernel.  FullRes and Hybrid walk two chains per warp.
#include <cstring>
#include <vector>

#include "h264a_device.cuh"
#include "satd_mma.cuh"

namespace h264a {

// Eight pixels of two rows -> four averages: adjacent pixels summed in 16-bit
// halves, each (sum + 2) / 4.
__device__ __forceinline__ uint32_t ds_avg(uint32_t a, uint32_t b) {  // two outputs, in bytes 0 and 2
    const uint32_t m = 0x00ff00ffu;
    return (((a & m) + ((a >> 8) & m) + (b & m) + ((b >> 8) & m) + 0x00020002u) >> 2) & m;
}
// DS_ROWS output rows a thread (hh is a multiple of 8), all their loads in
// flight together.  Bound by DRAM: 60 1080p frames, 155 MB, 44 us with one row
// a thread, 26 now.
constexpr int DS_ROWS = 4;
__global__ void __launch_bounds__(256) downsample2x_kernel(const uint8_t* __restrict__ in, int cw, int ch, size_t fstride,
                                                           uint8_t* __restrict__ out) {
    const int hw = cw / 2, hh = ch / 2;
    const int f = blockIdx.z;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;  // group of 4 x DS_ROWS outputs
    const int groups_per_row = hw / 4;
    const int jb = t / groups_per_row, j = jb * DS_ROWS, i4 = (t - jb * groups_per_row) * 4;
    if (j >= hh) return;
    const uint8_t* a = in + fstride * f + (long long)(2 * j) * cw + 2 * i4;
    uint2 r[2 * DS_ROWS];
#pragma unroll
    for (int k = 0; k < 2 * DS_ROWS; k++) r[k] = __ldg(reinterpret_cast<const uint2*>(a + (long long)k * cw));
    uint8_t* o = out + (size_t)hw * hh * f + (long long)j * hw + i4;
#pragma unroll
    for (int k = 0; k < DS_ROWS; k++)
        *reinterpret_cast<uint32_t*>(o + (long long)k * hw) =
            __byte_perm(ds_avg(r[2 * k].x, r[2 * k + 1].x), ds_avg(r[2 * k].y, r[2 * k + 1].y), 0x6420);
}

// Scoring-resolution geometry of one lookahead mode.
struct LaGeom {
    int bs;        // block size at the scoring resolution (8 HalfRes, 16 otherwise)
    int sw, sh;    // scoring picture size
};

// intra_cost (mbtree.rs:78-93) of every MB of every frame; frame 0 (IDR) also
// gets inter = intra, mv = 0 (mbtree.rs:257).
__global__ void la_intra_kernel(const uint8_t* __restrict__ pics, size_t fstride, LaGeom g, int mb_w, int mb_h, int n,
                                int32_t* __restrict__ intra, int32_t* __restrict__ inter, int32_t* __restrict__ mvs) {
    const int lg = g.bs == 16 ? 4 : 2;  // sub-blocks per MB: 16 or 4
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long gm = t >> lg;  // global MB index
    const long long nmb = (long long)mb_w * mb_h;
    const int sb = int(t & ((1 << lg) - 1));
    int v = 0;
    const bool live = gm < nmb * n;
    if (live) {
        const int f = int(gm / nmb), m = int(gm % nmb);
        const int mbx = m % mb_w, mby = m / mb_w;
        const int nbx = g.bs / 4;
        const int x = mbx * g.bs + (sb % nbx) * 4, y = mby * g.bs + (sb / nbx) * 4;
        const uint8_t* p = pics + fstride * f + (long long)y * g.sw + x;
        uint32_t s[4];
        const uint32_t z[4] = {0, 0, 0, 0};
#pragma unroll
        for (int r = 0; r < 4; r++) s[r] = ld4u(p + (long long)r * g.sw);
        const int dc = int(__vsadu4(s[0], 0) + __vsadu4(s[1], 0) + __vsadu4(s[2], 0) + __vsadu4(s[3], 0));
        v = satd4x4_rows(s, z) - dc;  // Σ|AC|: the DC coefficient is the (non-negative) block sum
    }
    v = warp_seg_sum(v, 1 << lg);
    if (live && sb == 0) {
        const int c = v < 1 ? 1 : v;
        intra[gm] = c;
        if (gm < nmb) {  // frame 0: the IDR, no reference
            inter[gm] = c;
            mvs[2 * gm] = 0;
            mvs[2 * gm + 1] = 0;
        }
    }
}

// One lane's view of the SATD search of a bs x bs block.  The warp holds two
// searches, lane group g = lane / 16 (slots 16g.. of the candidate and
// distortion arrays), each walking its own row chain; a group prices
// 16 / (bs/4)^2 candidates per pass (four 8x8 or one 16x16).
struct LaSearch {
    const uint8_t* cur;
    const uint8_t* ref;
    int w, h, bs, lg_nb, gl, gb, bxo, byo, x0, y0;
    uint32_t spa[4], spb[4];  // the source rows split into column pairs (split_pairs)
    int2* cand;
    int* dist;

    __device__ void init(const uint8_t* c, const uint8_t* r, int pw, int ph, int b, int bx0, int by0, int2* cs,
                         int* ds) {
        cur = c; ref = r; w = pw; h = ph; bs = b; x0 = bx0; y0 = by0; cand = cs; dist = ds;
        const int lane = threadIdx.x & 31;
        gl = lane & 15;
        gb = lane & 16;
        lg_nb = b == 16 ? 4 : 2;
        const int nbx = b / 4;
        const int sb = gl & ((1 << lg_nb) - 1);
        bxo = (sb % nbx) * 4;
        byo = (sb / nbx) * 4;
        {
            uint32_t srow[4];
#pragma unroll
            for (int r = 0; r < 4; r++) srow[r] = ld4u(cur + (long long)(y0 + byo + r) * w + x0 + bxo);
            split_pairs(srow, spa, spb);
        }
    }

    // SATD of each group's cand[gb..gb+n) (full-pel MVs, quarter-pel units)
    // added into dist (zeroed by the caller) by shared-memory atomics of the
    // lanes' 4x4 blocks; passes run to the larger group's need.
    template <bool FULLPEL>  // FULLPEL: every candidate is a full-pel MV (FullRes)
    __device__ void eval(int n) {
        const int cps = 4 - lg_nb;  // log2 candidates per pass of a group
        const int npass = __reduce_max_sync(0xffffffffu, (n + (1 << cps) - 1) >> cps);
        for (int k = 0; k < npass; k++) {
            const int c = (k << cps) + (gl >> lg_nb);
            int d = 0;
            if (c < n) {
                const int2 mv = cand[gb + c];
                uint32_t p[4];
                if (FULLPEL || ((mv.x | mv.y) & 3) == 0)
                    fullpel_rows_clamped(ref, w, h, x0 + bxo + (mv.x >> 2), y0 + byo + (mv.y >> 2), p);
                else  // a sub-pel seed (Hybrid mode halves a full-res MV): mc_luma on the plain picture
                    subpel_rows_clamped(ref, w, h, x0 + bxo + (mv.x >> 2), y0 + byo + (mv.y >> 2), mv.x & 3, mv.y & 3, p);
                d = satd4x4_packed(spa, spb, p);
            }
            if (c < n) atomicAdd(&dist[gb + c], d);  // the candidate's blocks, summed in shared memory
        }
        __syncwarp();
    }
};

// The four-point diamond in the order mbtree.rs:181 walks it:
// right, left, down, up.
__device__ __forceinline__ int la_ring_dx(int k) { return k == 0 ? 1 : (k == 1 ? -1 : 0); }
__device__ __forceinline__ int la_ring_dy(int k) { return k == 2 ? 1 : (k == 3 ? -1 : 0); }

// inter_cost (mbtree.rs:154-197) of each group's block: (0,0) and the seed,
// then the cascading four-point diamond at steps max_step .. 1 full pixels
// (first improvement moves the centre, the rest of the ring is priced around
// it; a ring that moved is walked again at the same step), stopping at once
// when (0,0) costs nothing.  `active` false: the group takes no part.
template <bool FULLPEL>
__device__ void la_inter_cost(LaSearch& s, bool active, int seedx, int seedy, int max_step, int& cost, int& mvx,
                              int& mvy) {
    const int gl = s.gl, gb = s.gb;
    int phase = active ? 0 : 2;  // 0 seeds, 1 rings, 2 done
    int step = max_step, ri = 0, guard = 0;
    bool moved = false;
    long long best = 0;
    int bx = 0, by = 0;
    for (;;) {
        int n = 0;
        if (phase == 0) {
            if (gl == 0) {
                s.cand[gb] = make_int2(0, 0);
                s.cand[gb + 1] = make_int2(seedx, seedy);
            }
            n = 2;
        } else if (phase == 1) {
            n = 4 - ri;
            if (gl < n)
                s.cand[gb + gl] = make_int2(bx + la_ring_dx(ri + gl) * step * 4, by + la_ring_dy(ri + gl) * step * 4);
        }
        if (__all_sync(0xffffffffu, phase == 2)) break;
        if (gl < n) s.dist[gb + gl] = 0;  // eval adds each lane's block into its candidate's slot
        __syncwarp();
        s.eval<FULLPEL>(n);
        const int d = gl < n ? s.dist[gb + gl] : 0;
        const unsigned hit = (__ballot_sync(0xffffffffu, gl < n && (long long)d < best) >> gb) & 0xffffu;
        const int j = hit ? __ffs(hit) - 1 : 0;
        const int dj = __shfl_sync(0xffffffffu, d, gb + j);
        const int d0 = __shfl_sync(0xffffffffu, d, gb), d1 = __shfl_sync(0xffffffffu, d, gb + 1);
        if (phase == 0) {
            best = d0;
            if (best == 0) {
                phase = 2;
            } else {
                if ((seedx != 0 || seedy != 0) && (long long)d1 < best) {
                    best = d1;
                    bx = seedx;
                    by = seedy;
                }
                phase = 1;
            }
        } else if (phase == 1) {
            bool ring_end;
            if (hit) {
                best = dj;
                bx = s.cand[gb + j].x;
                by = s.cand[gb + j].y;
                moved = true;
                ri += j + 1;
                ring_end = ri >= 4;
            } else {
                ring_end = true;
            }
            if (ring_end) {
                if (moved && ++guard < (1 << 20)) {
                    ri = 0;  // walk the ring again at this step
                } else {
                    step >>= 1;
                    ri = 0;
                    guard = 0;
                    if (step == 0) phase = 2;
                }
                moved = false;
            }
        }
        __syncwarp();
    }
    cost = best > 0x7fffffffLL ? 0x7fffffff : int(best);
    mvx = bx;
    mvy = by;
}

struct LaBufs {
    CUtensorMap hmap;     // HalfRes: the half-res frames as (cw/2, ch/2, n), box LA_WIN_W x LA_WIN_H x 1
    int hmap_ok;          // HalfRes with a valid map: searches read windows
    const uint8_t* full;  // n frames cw x ch
    const uint8_t* half;  // n frames cw/2 x ch/2 (modes 1, 2)
    int cw, ch, mb_w, mb_h, n, mode;
    int32_t* intra;
    int32_t* inter;
    int32_t* mvs;
};

// frame_costs for MB (mbx, mby) of frame f >= 1 given the full-res seed
// (MODE 0 FullRes, 1 Hybrid).
template <int MODE>
__device__ void la_mb(const LaBufs& b, bool active, int f, int mbx, int mby, int sfx, int sfy, int2* cs, int* ds,
                      int& outx, int& outy) {
    const long long nmb = (long long)b.mb_w * b.mb_h;
    const long long gm = nmb * f + (long long)mby * b.mb_w + mbx;
    const int cwh = b.cw / 2, chh = b.ch / 2;
    const size_t fs = (size_t)b.cw * b.ch, hs = (size_t)cwh * chh;
    LaSearch s;
    int cost, mx, my;
    // an input (la_intra_kernel's output): read before the search, used after it
    const int ic = active && (threadIdx.x & 15) == 0 ? __ldg(b.intra + gm) : 0;
    if (MODE == 0) {  // FullRes
        s.init(b.full + fs * f, b.full + fs * (f - 1), b.cw, b.ch, 16, mbx * 16, mby * 16, cs, ds);
        la_inter_cost<true>(s, active, sfx, sfy, 8, cost, mx, my);
    } else {
        s.init(b.half + hs * f, b.half + hs * (f - 1), cwh, chh, 8, mbx * 8, mby * 8, cs, ds);
        int hx, hy;
        la_inter_cost<false>(s, active, sfx / 2, sfy / 2, 8, cost, hx, hy);
        // refine at full-res from the coarse MV
        s.init(b.full + fs * f, b.full + fs * (f - 1), b.cw, b.ch, 16, mbx * 16, mby * 16, cs, ds);
        la_inter_cost<true>(s, active, hx * 2, hy * 2, 2, cost, mx, my);
    }
    if (active && s.gl == 0) {
        b.inter[gm] = cost < ic ? cost : ic;
        b.mvs[2 * gm] = mx;
        b.mvs[2 * gm + 1] = my;
    }
    outx = mx;
    outy = my;
}

constexpr int LA_WARPS = 4;

// Column-0 chains and row chains in one persistent launch, two chains per
// warp (lane group g = lane / 16 walks the second).  Tickets 0 .. ceil(nf/2)-1
// walk column 0 of frames 1+2t+g and publish flag (f-1)*mb_h + y after MB
// (0, y); later tickets take rows 2p and 2p+1 of the row order (rows in
// order, frames interleaved), each group waiting for its own column-0 flag
// and walking columns 1.. seeded by the left neighbour.
// Several streams' lookaheads in one launch: stream s's column tickets are
// col0[s] .. col0[s+1]-1, all of them before any stream's row tickets
// (rowt0[s] .. rowt0[s+1]-1 after col0[ns]), so a row ticket's column chain
// was taken earlier, by a warp that waits for nothing; stream s's flags start
// at flag0[s].
constexpr int LA_MAXS = 24;
struct LaMulti {
    LaBufs b[LA_MAXS];
    int col0[LA_MAXS + 1];
    long long rowt0[LA_MAXS + 1];
    long long flag0[LA_MAXS];
    int ns;
};

template <int MODE>  // b.mode, as a constant
__global__ void __launch_bounds__(32 * LA_WARPS, 4) la_chains_kernel(const __grid_constant__ LaMulti lm,
                                                                 int* __restrict__ counter, int* __restrict__ flags0,
                                                                 int epoch, int* __restrict__ status, int spin_limit) {
    __shared__ int2 cs[LA_WARPS][32];
    __shared__ int ds[LA_WARPS][32];
    const int w = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int grp = lane >> 4, gl = lane & 15;
    const int ns = lm.ns;
    for (;;) {
        int t = 0;
        if (lane == 0) t = atomicAdd(counter, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t < lm.col0[ns]) {
            int sidx = 0;
            while (sidx + 1 < ns && lm.col0[sidx + 1] <= t) sidx++;
            const LaBufs& b = lm.b[sidx];
            int* flags = flags0 + lm.flag0[sidx];
            const int nf = b.n - 1;
            const int f = 1 + 2 * (t - lm.col0[sidx]) + grp;
            const bool active = f <= nf;
            int sx = 0, sy = 0;
            for (int mby = 0; mby < b.mb_h; mby++) {
                int mx, my;
                la_mb<MODE>(b, active, active ? f : 1, 0, mby, sx, sy, cs[w], ds[w], mx, my);
                sx = mx;
                sy = my;
                if (active && gl == 0) st_release(flags + (f - 1) * b.mb_h + mby, epoch);  // after the lane's MV store
                __syncwarp();
            }
            continue;
        }
        const long long tr = (long long)t - lm.col0[ns];
        if (tr >= lm.rowt0[ns]) return;
        int sidx = 0;
        while (sidx + 1 < ns && lm.rowt0[sidx + 1] <= tr) sidx++;
        const LaBufs& b = lm.b[sidx];
        int* flags = flags0 + lm.flag0[sidx];
        const int nf = b.n - 1;
        const long long nrows = (long long)nf * b.mb_h;
        const long long r = 2 * (tr - lm.rowt0[sidx]) + grp;
        const bool active = r < nrows;
        const int mby = active ? int(r / nf) : 0, f = active ? 1 + int(r % nf) : 1;
        if (active && gl == 0) wait_flag(flags + (f - 1) * b.mb_h + mby, epoch, status, 1, spin_limit);
        __syncwarp();
        const long long gm0 = (long long)b.mb_w * b.mb_h * f + (long long)mby * b.mb_w;
        int sx = active ? __ldcg(b.mvs + 2 * gm0) : 0, sy = active ? __ldcg(b.mvs + 2 * gm0 + 1) : 0;
        for (int mbx = 1; mbx < b.mb_w; mbx++) {
            int mx, my;
            la_mb<MODE>(b, active, f, mbx, mby, sx, sy, cs[w], ds[w], mx, my);
            sx = mx;
            sy = my;
            __syncwarp();
        }
    }
}

// ---- HalfRes ------------------------------------------------------------------
// The search of an 8x8 half-res block by a whole warp, eight candidates a
// round on the tensor cores (satd_mma.cuh): candidate c is column c of four
// mmas, one per 4x4 block, lane l holding row l % 4 of candidate l / 4's
// blocks; a candidate's sum (<= 65,280) is half a word, so three shuffles
// reduce two candidates at once.
//
// The diamond evaluates its points one after the other and moves at the first
// improvement, so the points that follow while nothing improves are known:
// a round prices the next eight of that list (the rest of the ring, then the
// following steps' rings), takes its first improvement and forgets what came
// after it.  The first round is (0,0), the seed and the first six points
// around the seed.  A block that keeps its seed takes three rounds.
//
// Bound by a chain's serial latency (a 1080p frame: 68 blocks down column 0,
// then 119 along the last row), so everything else stays off it: the next
// block's source and intra cost are loaded a block ahead, the reference
// windows two copies ahead (TMA; along a row two blocks share a window).  60
// 1080p frames: 1,216 us with 16 lanes a chain through shared-memory slots,
// one ring a round; 451 this way (five CTAs an SM; eight, with 64 registers a
// thread, 631: every row resident, most of them waiting).
//
// Windows: LA_BUFS buffers a chain of LA_WIN_H rows of LA_WIN_W bytes, the
// block +-16 rows, and 48 columns from the 16-byte boundary at or left of the
// block's x - 16.  A candidate outside the picture reads clamped coordinates;
// one whose clamped rows or columns lie outside the window reads the picture.
constexpr int LA_HWARPS = 4, LA_BUFS = 3;
constexpr int LA_WIN_W = 48, LA_WIN_H = 40, LA_WIN_BYTES = LA_WIN_W * LA_WIN_H;
constexpr int LA_WIN_BUF = 2048;  // buffer stride: 128-byte aligned, with room for a row read's further words
extern __shared__ __align__(128) uint8_t la_win[];

__device__ __noinline__ uint32_t la_clamped_word(const uint8_t* ref, int w, int h, int x, int y) {
    const uint8_t* row = ref + (long long)clampi(y, 0, h - 1) * w;
    uint32_t v = 0;
#pragma unroll
    for (int c = 0; c < 4; c++) v |= uint32_t(__ldg(row + clampi(x + c, 0, w - 1))) << (8 * c);
    return v;
}

// Point `pos` (0 .. 10) of the list that follows while nothing improves, from
// ring point 0 of the ring at `step` on: its step (0 past the end).  `moved`:
// that ring is walked again at its step.
__device__ __forceinline__ int la_list_step(int step, bool moved, int pos) {
    const int ring = pos >> 2;
    return step >> (moved && ring > 0 ? ring - 1 : ring);
}
// Adds ring point k at step st
__device__ __forceinline__ void la_ring_add(int k, int st, int& x, int& y) {
    const int s = (k & 1) ? -st : st;
    x += (k & 2) ? 0 : s;
    y += (k & 2) ? s : 0;
}

struct LaBlock {
    const uint8_t* ref;
    int w, h, x0, y0;
    const uint8_t* win;  // null: none
    int wx0, wy0;
    int mode;  // 0 no window, 1 the window reaches outside the picture, 2 it does not
    uint32_t src[4];
};

// SATD of the lane's candidate column (full-pel offset dx, dy): candidates 2q
// (low half) and 2q + 1 (high half) of lane q = lane % 4, in every lane
__device__ __forceinline__ uint32_t la_price(const HadFrag& hf, const LaBlock& b, int dx, int dy) {
    const int x = b.x0 + dx, y = b.y0 + dy + int(threadIdx.x & 3);
    uint32_t p[4];
    bool ok = false;
    if (b.mode != 0) {
        if (b.mode == 2) {
            const int cx = x - b.wx0, cy = y - b.wy0;
            ok = unsigned(cx) <= unsigned(LA_WIN_W - 8) && unsigned(cy) < unsigned(LA_WIN_H - 4);
            if (ok) {
                const int a = cy * LA_WIN_W + cx;
                const uint32_t* w0 = reinterpret_cast<const uint32_t*>(b.win + (a & ~3));
                const uint32_t* w1 = w0 + LA_WIN_W;  // four rows down
                const uint32_t sh = uint32_t(a & 3) * 8u;
                const uint32_t m0 = w0[1], m1 = w1[1];
                p[0] = __funnelshift_r(w0[0], m0, sh);
                p[1] = __funnelshift_r(m0, w0[2], sh);
                p[2] = __funnelshift_r(w1[0], m1, sh);
                p[3] = __funnelshift_r(m1, w1[2], sh);
            }
        } else {
            const int xa = clampi(x, 0, b.w - 4), xb = clampi(x + 4, 0, b.w - 4);
            const int ya = clampi(y, 0, b.h - 1) - b.wy0, yb = clampi(y + 4, 0, b.h - 1) - b.wy0;
            ok = unsigned(xa - b.wx0) <= unsigned(LA_WIN_W - 4) && unsigned(xb - b.wx0) <= unsigned(LA_WIN_W - 4) &&
                 unsigned(ya) < unsigned(LA_WIN_H) && unsigned(yb) < unsigned(LA_WIN_H);
            if (ok) {
                // byte i of a clamped word is byte clamp(i + x - xa, 0, 3) of the word at xa
                const uint32_t sa = __funnelshift_r(0x33210000u, 0x33u, uint32_t(4 * (clampi(x - xa, -3, 3) + 3)));
                const uint32_t sb = __funnelshift_r(0x33210000u, 0x33u, uint32_t(4 * (clampi(x + 4 - xb, -3, 3) + 3)));
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int a = ((i & 2) ? yb : ya) * LA_WIN_W + ((i & 1) ? xb : xa) - b.wx0;
                    const uint32_t* wp = reinterpret_cast<const uint32_t*>(b.win + (a & ~3));
                    p[i] = __byte_perm(__funnelshift_r(wp[0], wp[1], uint32_t(a & 3) * 8u), 0u, (i & 1) ? sb : sa);
                }
            }
        }
    }
    if (!ok) {
#pragma unroll 1
        for (int i = 0; i < 4; i++) {
            const uint32_t v = la_clamped_word(b.ref, b.w, b.h, x + 4 * (i & 1), y + 4 * (i >> 1));
            p[0] = i == 0 ? v : p[0];
            p[1] = i == 1 ? v : p[1];
            p[2] = i == 2 ? v : p[2];
            p[3] = i == 3 ? v : p[3];
        }
    }
    __syncwarp();
    int s0 = 0, s1 = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) had_mma(hf, p[i], b.src[i], s0, s1);
    uint32_t v = uint32_t(s0) | uint32_t(s1) << 16;
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Takes the first improvement of a round's list, whose point 0 is candidate
// `base`, or goes past it.  (Candidates before `base` and past the list's end
// cost no less than `best`: they are what `best` is the least of, and the
// centre again.)
__device__ __forceinline__ void la_take(uint32_t v, int qa, int base, int& bx, int& by, int& step, int& ri, bool& moved,
                                        uint32_t& best) {
    const unsigned mine = (v & 0xffffu) < best ? unsigned(qa) : ((v >> 16) < best ? unsigned(qa + 1) : 8u);
    const int hit = int(__reduce_min_sync(0xffffffffu, mine));
    const int pos = ri + hit - base;
    step = la_list_step(step, moved, pos);
    moved = moved && pos < 4;
    ri = pos & 3;
    if (hit < 8) {
        const uint32_t d = __shfl_sync(0xffffffffu, v, hit >> 1);
        best = (hit & 1) ? d >> 16 : d & 0xffffu;
        la_ring_add(ri, step, bx, by);
        moved = ri != 3;  // after its last point the ring is walked again
        ri = (ri + 1) & 3;
    }
}

// inter_cost (mbtree.rs:154-197), as la_inter_cost above; seed and result in
// full pixels.  (The reference's bound on walks of one ring cannot be reached:
// each follows an improvement of a cost below 2^16.)
__device__ __forceinline__ void la_half_search(const HadFrag& hf, const LaBlock& b, int seedx, int seedy, int& cost,
                                               int& mvx, int& mvy) {
    const int lane = threadIdx.x & 31, c = lane >> 2, qa = 2 * (lane & 3);
    int bx = seedx, by = seedy, step = 8, ri = 0;
    bool moved = false;
    uint32_t best = 0;
    {
        const int pos = max(c - 2, 0);
        int dx = c == 0 ? 0 : bx, dy = c == 0 ? 0 : by;
        la_ring_add(pos & 3, c < 2 ? 0 : 8 >> (pos >> 2), dx, dy);
        const uint32_t v = la_price(hf, b, dx, dy);
        const uint32_t v0 = __shfl_sync(0xffffffffu, v, 0);
        best = v0 & 0xffffu;
        if (best == 0) {
            cost = mvx = mvy = 0;
            return;
        }
        if ((bx | by) == 0 || (v0 >> 16) < best) {
            best = min(best, v0 >> 16);
            la_take(v, qa, 2, bx, by, step, ri, moved, best);
        } else {
            bx = by = 0;  // the points around the seed do not count
        }
    }
    while (step > 0) {
        const int pos = ri + c;
        int dx = bx, dy = by;
        la_ring_add(pos & 3, la_list_step(step, moved, pos), dx, dy);
        la_take(la_price(hf, b, dx, dy), qa, 0, bx, by, step, ri, moved, best);
    }
    cost = int(best);
    mvx = bx;
    mvy = by;
}

// Column-0 chains and row chains in one persistent launch, one per warp:
// tickets as la_chains_kernel's, chain by chain.
__global__ void __launch_bounds__(32 * LA_HWARPS, 5) la_half_kernel(const __grid_constant__ LaMulti lm, int* __restrict__ counter,
                                                                    int* __restrict__ flags0, int epoch,
                                                                    int* __restrict__ status, int spin_limit) {
    __shared__ __align__(8) unsigned long long la_bar[LA_HWARPS][LA_BUFS];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    uint8_t* win = la_win + wp * LA_BUFS * LA_WIN_BUF;
    const uint32_t win0 = uint32_t(__cvta_generic_to_shared(win));
    const uint32_t bar0 = uint32_t(__cvta_generic_to_shared(&la_bar[wp][0]));
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < LA_BUFS; i++) mbar_init(bar0 + 8 * i, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    const HadFrag hf = had_frag(lane);
    uint32_t parity = 0;  // bit k: the phase buffer k completes next
    const int ns = lm.ns;
    for (;;) {
        int t = 0;
        if (lane == 0) t = atomicAdd(counter, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        const bool col = t < lm.col0[ns];
        const long long tr = (long long)t - lm.col0[ns];
        if (!col && tr >= lm.rowt0[ns]) return;
        int sidx = 0;
        if (col)
            while (sidx + 1 < ns && lm.col0[sidx + 1] <= t) sidx++;
        else
            while (sidx + 1 < ns && lm.rowt0[sidx + 1] <= tr) sidx++;
        const LaBufs& b = lm.b[sidx];
        int* flags = flags0 + lm.flag0[sidx];
        const int nf = b.n - 1, mbw = b.mb_w, mbh = b.mb_h;
        const int r = col ? 0 : int(tr - lm.rowt0[sidx]);
        const int f = col ? 1 + t - lm.col0[sidx] : 1 + r % nf, row = col ? 0 : r / nf;
        // the chain's blocks: (0, i), or (i, row) from i = 1 on; its windows:
        // one per block, or one per two columns
        const int i0 = col ? 0 : 1, ni = col ? mbh : mbw, wshift = col ? 0 : 1, nw = (ni + wshift) >> wshift;
        if (i0 >= ni) continue;
        LaBlock blk;
        blk.w = b.cw / 2;
        blk.h = b.ch / 2;
        const size_t hs = size_t(blk.w) * blk.h;
        const uint8_t* cur = b.half + hs * f;
        blk.ref = cur - hs;
        const bool uw = b.hmap_ok != 0;
        auto issue = [&](int wn) {  // window wn into its buffer, whose earlier reads are complete
            __syncwarp();
            if (lane == 0) {
                const uint32_t bar = bar0 + 8 * (wn % LA_BUFS);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                mbar_expect_tx(bar, uint32_t(LA_WIN_BYTES));
                tma_load_3d(win0 + uint32_t(wn % LA_BUFS * LA_WIN_BUF), &b.hmap, col ? -16 : 16 * wn - 16,
                            (col ? 8 * wn : 8 * row) - 16, f - 1, bar);
            }
        };
        if (uw)
            for (int k = 0; k < LA_BUFS - 1 && k < nw; k++) issue(k);
        const int q = lane & 3;
        const uint8_t* sp = cur + (long long)(col ? 0 : 8 * row + 0) * blk.w + (col ? 0 : 8 * i0) + (long long)q * blk.w;
        const long long sstep = col ? 8LL * blk.w : 8;
        uint32_t nsrc[4];
#pragma unroll
        for (int i = 0; i < 4; i++) nsrc[i] = ld4u(sp + (long long)(4 * (i >> 1)) * blk.w + 4 * (i & 1));
        const long long gm0 = (long long)mbw * mbh * f + (long long)row * mbw;
        int nic = __ldg(b.intra + gm0 + i0);
        int sx = 0, sy = 0;
        if (!col) {
            if (lane == 0) wait_flag(flags + (f - 1) * mbh + row, epoch, status, 1, spin_limit);
            __syncwarp();
            sx = __ldcg(b.mvs + 2 * gm0) / 8;
            sy = __ldcg(b.mvs + 2 * gm0 + 1) / 8;
        }
        int wn = -1;
        for (int i = i0; i < ni; i++) {
            const int ic = nic;
#pragma unroll
            for (int k = 0; k < 4; k++) blk.src[k] = nsrc[k];
            const long long gm = col ? gm0 + (long long)i * mbw : gm0 + i;
            if (i + 1 < ni) {
                sp += sstep;
#pragma unroll
                for (int k = 0; k < 4; k++) nsrc[k] = ld4u(sp + (long long)(4 * (k >> 1)) * blk.w + 4 * (k & 1));
                nic = __ldg(b.intra + gm + (col ? mbw : 1));
            }
            blk.x0 = col ? 0 : 8 * i;
            blk.y0 = col ? 8 * i : 8 * row;
            if ((i >> wshift) != wn) {
                wn = i >> wshift;
                blk.wx0 = col ? -16 : 16 * wn - 16;
                blk.wy0 = blk.y0 - 16;
                blk.mode = !uw ? 0
                           : blk.wx0 < 0 || blk.wy0 < 0 || blk.wx0 + LA_WIN_W > blk.w || blk.wy0 + LA_WIN_H > blk.h ? 1 : 2;
                blk.win = win + wn % LA_BUFS * LA_WIN_BUF;
                if (uw) {
                    if (wn + LA_BUFS - 1 < nw) issue(wn + LA_BUFS - 1);
                    wait_window(bar0 + 8 * (wn % LA_BUFS), (parity >> (wn % LA_BUFS)) & 1u, status, 3, spin_limit);
                    parity ^= 1u << (wn % LA_BUFS);
                    __syncwarp();
                }
            }
            int cost, mx, my;
            la_half_search(hf, blk, sx, sy, cost, mx, my);
            sx = mx;
            sy = my;
            if (lane == 0) {
                b.inter[gm] = cost < ic ? cost : ic;
                b.mvs[2 * gm] = mx * 8;
                b.mvs[2 * gm + 1] = my * 8;
                if (col) st_release(flags + (f - 1) * mbh + i, epoch);  // after the lane's MV store
            }
            __syncwarp();
        }
    }
}

}  // namespace h264a

using namespace h264a;

extern "C" int h264a_downsample2x(h264a_ctx* ctx, const uint8_t* d_frames, int cw, int ch, int n, size_t frame_stride,
                                  uint8_t* d_half, void* stream) {
    if (!ctx || !d_frames || !d_half) return fail(H264A_E_ARG, "downsample2x: null pointer");
    if (cw < 16 || ch < 16 || cw % 16 || ch % 16 || n < 1 || n > 65535)
        return fail(H264A_E_ARG, "downsample2x: frames must be MB-aligned, 1 <= n <= 65535");
    if (frame_stride % 8 || (n > 1 && frame_stride < (size_t)cw * ch) ||
        (reinterpret_cast<uintptr_t>(d_frames) & 7) || (reinterpret_cast<uintptr_t>(d_half) & 3))
        return fail(H264A_E_ARG, "downsample2x: misaligned frames");
    const long long groups = (long long)(cw / 8) * (ch / 2 / DS_ROWS);
    dim3 grid(unsigned((groups + 255) / 256), 1, n);
    downsample2x_kernel<<<grid, 256, 0, pick_stream(ctx, stream)>>>(d_frames, cw, ch, frame_stride, d_half);
    return check_launch("downsample2x_kernel");
}

namespace {

// Validates one stream's lookahead and fills its LaBufs (no launch).
int la_prepare(const h264a_la_stream& q, int mode, LaBufs& b) {
    if (!q.d_full || !q.d_intra || !q.d_inter || !q.d_mvs) return fail(H264A_E_ARG, "lookahead_costs: null pointer");
    if (mode != 0 && !q.d_half) return fail(H264A_E_ARG, "lookahead_costs: modes 1 and 2 need the half-res frames");
    if (q.cw < 16 || q.ch < 16 || q.cw % 16 || q.ch % 16 || q.n < 1)
        return fail(H264A_E_ARG, "lookahead_costs: bad geometry");
    if ((long long)(q.n - 1) * (q.ch / 16) > (1 << 24)) return fail(H264A_E_ARG, "lookahead_costs: too many rows");
    memset(&b, 0, sizeof b);
    b.full = q.d_full; b.half = q.d_half; b.cw = q.cw; b.ch = q.ch; b.mb_w = q.cw / 16; b.mb_h = q.ch / 16; b.n = q.n;
    b.mode = mode;
    b.intra = q.d_intra; b.inter = q.d_inter; b.mvs = q.d_mvs;
    b.hmap_ok = mode == 2 ? encode_u8_map_3d(&b.hmap, q.d_half, q.cw / 2, q.ch / 2, q.n, LA_WIN_W, LA_WIN_H, 1) : 0;
    return H264A_OK;
}

// intra costs of every stream, then their chains in persistent launches of
// up to LA_MAXS streams each (the queue is the context's lookahead queue).
int la_run(h264a_ctx* ctx, const h264a_la_stream* qs, int nq, int mode, cudaStream_t st) {
    if (mode < 0 || mode > 2) return fail(H264A_E_ARG, "lookahead_costs: mode must be 0 (full), 1 (hybrid) or 2 (half)");
    std::vector<LaBufs> bufs(nq);
    for (int i = 0; i < nq; i++) {
        const int rc = la_prepare(qs[i], mode, bufs[i]);
        if (rc) return rc;
    }
    for (int i = 0; i < nq; i++) {
        const h264a_la_stream& q = qs[i];
        const int cw = q.cw, ch = q.ch, n = q.n;
        const LaGeom g = mode == 2 ? LaGeom{8, cw / 2, ch / 2} : LaGeom{16, cw, ch};
        const size_t fstride = mode == 2 ? (size_t)(cw / 2) * (ch / 2) : (size_t)cw * ch;
        const long long nmb = (long long)(cw / 16) * (ch / 16);
        const long long threads = nmb * n * (g.bs == 16 ? 16 : 4);
        la_intra_kernel<<<unsigned((threads + 255) / 256), 256, 0, st>>>(mode == 2 ? q.d_half : q.d_full, fstride, g,
                                                                        cw / 16, ch / 16, n, q.d_intra, q.d_inter,
                                                                        q.d_mvs);
        const int rc = check_launch("la_intra_kernel");
        if (rc) return rc;
    }
    const int smem = mode == 2 ? LA_HWARPS * LA_BUFS * LA_WIN_BUF : 0;
    const int wpc = mode == 2 ? LA_HWARPS : LA_WARPS, cpw = mode == 2 ? 1 : 2;  // warps per CTA, chains per warp
    auto kern = mode == 0 ? la_chains_kernel<0> : (mode == 1 ? la_chains_kernel<1> : la_half_kernel);
    for (int s0 = 0; s0 < nq; s0 += LA_MAXS) {
        LaMulti* lm = new LaMulti;
        memset(lm, 0, sizeof *lm);
        long long flags = 0;
        for (int i = s0; i < nq && lm->ns < LA_MAXS; i++) {
            if (qs[i].n < 2) continue;  // intra only
            const int k = lm->ns++;
            const int nf = qs[i].n - 1;
            const long long nrows = (long long)nf * (qs[i].ch / 16);
            lm->b[k] = bufs[i];
            lm->col0[k + 1] = lm->col0[k] + (nf + cpw - 1) / cpw;
            lm->rowt0[k + 1] = lm->rowt0[k] + (nrows + cpw - 1) / cpw;
            lm->flag0[k] = flags;
            flags += nrows;
        }
        if (lm->ns == 0) {
            delete lm;
            continue;
        }
        const long long chains = lm->col0[lm->ns] + lm->rowt0[lm->ns];  // tickets
        int rc = flags > (1LL << 30) ? fail(H264A_E_ARG, "lookahead_costs: too many rows") : H264A_OK;
        if (!rc) rc = ensure_me_scratch(ctx, size_t(flags), Q_LOOKAHEAD);
        if (!rc && cudaMemsetAsync(ctx->q[Q_LOOKAHEAD].d_counter, 0, sizeof(int32_t), st) != cudaSuccess)
            rc = cuda_fail(cudaGetLastError(), "lookahead_costs: counter reset");
        const int epoch = rc ? -1 : next_epoch(ctx, st, Q_LOOKAHEAD);
        if (!rc && epoch < 0) rc = H264A_E_CUDA;
        int per_sm = 0;
        if (!rc && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * wpc, smem) != cudaSuccess)
            rc = cuda_fail(cudaGetLastError(), "lookahead_costs: occupancy");
        if (!rc) {
            long long blocks = (long long)ctx->num_sms * (per_sm > 0 ? per_sm : 1);
            const long long need = (chains + wpc - 1) / wpc;
            if (blocks > need) blocks = need;
            kern<<<unsigned(blocks), 32 * wpc, smem, st>>>(*lm, ctx->q[Q_LOOKAHEAD].d_counter,
                                                                ctx->q[Q_LOOKAHEAD].d_flags, epoch, ctx->d_status,
                                                                SPIN_LIMIT);
            rc = check_launch("la_chains_kernel");
        }
        delete lm;
        if (rc) return rc;
    }
    return H264A_OK;
}

}  // namespace

extern "C" int h264a_lookahead_costs(h264a_ctx* ctx, const uint8_t* d_full, const uint8_t* d_half, int cw, int ch, int n,
                                     int mode, int32_t* d_intra, int32_t* d_inter, int32_t* d_mvs, void* stream) {
    if (!ctx) return fail(H264A_E_ARG, "lookahead_costs: null pointer");
    const h264a_la_stream q{d_full, d_half, cw, ch, n, d_intra, d_inter, d_mvs};
    return la_run(ctx, &q, 1, mode, pick_stream(ctx, stream));
}

extern "C" int h264a_lookahead_streams(h264a_ctx* ctx, const h264a_la_stream* streams, int nstreams, int mode,
                                       void* stream) {
    if (!ctx || !streams) return fail(H264A_E_ARG, "lookahead_streams: null pointer");
    if (nstreams < 1) return fail(H264A_E_ARG, "lookahead_streams: need at least one stream");
    return la_run(ctx, streams, nstreams, mode, pick_stream(ctx, stream));
}

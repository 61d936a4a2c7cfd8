// mb_search.cuh -- the searches of one macroblock (motion_search,
// crates/rusty_h264-encoder/src/mb16.rs:2433-3302, as best_part runs them,
// :4921) by one warp: the 16x16, then the four 16x8 / 8x16 partitions side by
// side, every candidate priced on the tensor cores (satd_mma.cuh).
//
// A round prices up to eight candidate slots per group of eight lanes.  Mode 0
// (16x16): the four groups hold identical state and the warp's eight mma
// columns are the eight slots, 16 blocks each.  Mode 1: group g searches
// partition g (0 16x8 top, 1 16x8 bottom, 2 8x16 left, 3 8x16 right; they
// share the seeds [pmv, mv16], the mvd centre and λ, mb16.rs:8869-8913, so
// they are independent), and an mma's columns are two slots of each group.
// Either way 16 mma are one pass: "tile A" and "tile B" of eight blocks,
// the upper and lower half of the 16x16 candidate, or slots c and c + 2 of
// the partitions.  A pass costs the same for one candidate as for eight
// (mode 0) or four per partition (mode 1), so rings are priced whole, and the
// spare columns of a fixed-centre ring of four price the next rung's ring
// around the same centre, which the walk needs next whenever the ring does not
// improve.  Neither changes a decision: only the points the reference evaluates are
// folded, in its order, and only they are counted.
//
// The bound is the wavefront's latency: each MB's rounds depend on one
// another, and a round is a chain of shared-memory reads, mma and shuffles.
// Measured with Balanced inside the closed loop's launch (and in the step's): a
// 16x16 round takes 1,230 (1,160) cycles, where the butterflies on 32 lanes
// (satd4x4_packed, two 16x16 candidates or one per partition a pass, four warps
// a MB) took about 3,000, and a partition round 1,980 (1,510); an MB has about
// 6.5 to 7.8 and 11 to 12 of them.  59 1080p P frames of the closed loop: 46.6 ms
// before, 24.9 now; 15 P frames of five mixed streams (one launch): 8.3 and 3.8.
#pragma once

#include <cstddef>

#include "satd_mma.cuh"

namespace h264a {

// The reference picture's readiness in the pipelined closed loop: its planes
// are built segment by segment (16 picture rows by segw picture columns;
// segment (b, s)'s flag == epoch means every segment up and left of it is
// complete), and a search waits (bounded) for the segment of every pixel it
// reads.
struct BandWait {
    const int* flags;  // nbands x nseg readiness flags, band-major
    int nbands, nseg, segw, epoch, limit;
    int* status;
};

// Waits until the reference's planes (and reconstruction) are final at
// picture pixel (row, col), clamped into the picture: the flag of the band
// (16 rows) and column segment (segw columns) holding it.  Segment (b, s) is
// published after (b-1, s) and (b, s-1), so it stands for every segment up
// and left of it.  `ready` caches a segment seen ready, packed b << 12 | s
// (-1: none); any value stored there was seen ready, so a torn update between
// lanes only loses a shortcut.  Nothing when the search has no BandWait.
// Out of line: it is called from several places, mostly to find a segment
// seen ready.
__device__ __noinline__ void band_wait_at(const BandWait* bw, int* ready, int row, int col) {
    const int b = min(max(row, 0) >> 4, bw->nbands - 1);
    const int sg = min(max(col, 0) / bw->segw, bw->nseg - 1);
    const int c = *reinterpret_cast<volatile int*>(ready);
    if (c >= 0 && b <= (c >> 12) && sg <= (c & 4095)) return;
    wait_flag(bw->flags + b * bw->nseg + sg, bw->epoch, bw->status, 1, bw->limit);
    if (c < 0 || (b >= (c >> 12) && sg >= (c & 4095))) *reinterpret_cast<volatile int*>(ready) = (b << 12) | sg;
}

__device__ __forceinline__ void band_wait_px(const BandWait* bw, int* ready, int row, int col) {
    if (bw != nullptr) band_wait_at(bw, ready, row, col);
}

// Per-warp shared state of an MB's searches (read rarely, or by one lane).
struct MbScratch {
    const uint8_t* base;  // the reference's F|H|V|C planes
    const uint8_t* src;   // the source luma
    const BandWait* bw;   // the reference's segment readiness, or nullptr (complete)
    int pw, ph, pad, cw, ch;
    int wx0, wy0;         // the window's origin in padded-plane coordinates
    int bready;           // a reference segment seen complete (band_wait_px)
};

// ---------------------------------------------------------------------------
// Per-MB reference window in shared memory
// ---------------------------------------------------------------------------
// The F|H|V|C planes around the MB's predicted position, copied once per MB by
// the bulk-copy (TMA) engine: WIN_H rows of WIN_W bytes per plane, every
// search of the MB (16x16 and its partitions) then reads its candidates from
// shared memory.  Candidates whose reads leave the window take the plane path
// (pred_word), which gives the same bytes.  Rows are WIN_STRIDE = 80 bytes
// (20 banks) apart, so eight consecutive rows start four banks apart and the
// row words a ring's candidates read together rarely share a bank.
constexpr int WIN_W = 64, WIN_H = 42, WIN_STRIDE = 80;
constexpr int WIN_PLANE = WIN_H * WIN_STRIDE;  // bytes per plane (a multiple of 16)
constexpr int WIN_BYTES = 4 * WIN_PLANE;
constexpr int WIN_R = 12;  // the window starts this far up/left of the predicted position
constexpr int WIN_OFF = -(1 << 30);  // window offset of a search without one: below -2^29 for any MV, so every read misses

// Rows of the 4x4 block at window position (wx, wy) (full-pel part of the MV
// applied) at phase (fx, fy): the same operand table and averaging as
// pred_rows, read from the staged window at shared address `win`.
__device__ __forceinline__ void win_rows(uint32_t win, int wx, int wy, int fx, int fy, uint32_t out[4]) {
    const uint32_t pb = phase_bits(fx, fy);
    const int pa = int(pb & 3), pbb = int((pb >> 2) & 3);
    const int xa = wx + int((pb >> 4) & 1), ya = wy + int((pb >> 5) & 1);
    const uint32_t a = win + uint32_t(pa * WIN_PLANE + ya * WIN_STRIDE + (xa & ~3));
    const uint32_t sha = uint32_t(xa & 3) * 8u;
#pragma unroll
    for (int r = 0; r < 4; r++) out[r] = __funnelshift_r(lds_u32(a + r * WIN_STRIDE), lds_u32(a + r * WIN_STRIDE + 4), sha);
    if (pbb != 0) {
        const int xb = wx + int((pb >> 6) & 1), yb = wy + int((pb >> 7) & 1);
        const uint32_t b = win + uint32_t(pbb * WIN_PLANE + yb * WIN_STRIDE + (xb & ~3));
        const uint32_t shb = uint32_t(xb & 3) * 8u;
#pragma unroll
        for (int r = 0; r < 4; r++)
            out[r] = avg_up4(out[r], __funnelshift_r(lds_u32(b + r * WIN_STRIDE), lds_u32(b + r * WIN_STRIDE + 4), shb));
    }
}

// Both operands of a 4x4 block at window position (wx, wy) lie inside the
// window: x reads cover the aligned words from (wx + dx) & ~3 to +8, rows
// wy + dy .. wy + dy + 3, with dx, dy <= 1.
__device__ __forceinline__ bool win_covers(int wx, int wy) {
    return wx >= 0 && ((wx + 1) & ~3) <= WIN_W - 8 && wy >= 0 && wy + 5 <= WIN_H;
}

// ---------------------------------------------------------------------------
// Pricing
// ---------------------------------------------------------------------------

// A lane's view of the MB's searches.  px, py, rw, rh: its group's partition;
// wox, woy: that partition's origin in window coordinates (WIN_OFF: no
// window); src: the source words of row lane % 4 of the pass's sixteen blocks.
struct MbLane {
    int lane, gl, gb;
    int px, py, rw, rh, wox, woy, gather;
    uint32_t winq;
    HadFrag had;
    uint32_t src[16];
};

// The lane's share of the source MB (row lane % 4 of each block row, 16 bytes).
__device__ __forceinline__ void mb_load_src(MbLane& s, const uint8_t* src, int cw, int lx, int ly) {
    const int q = threadIdx.x & 3;
    const uint8_t* p = src + (long long)(ly + q) * cw + lx;
    if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {  // cw is a multiple of 16
#pragma unroll
        for (int b = 0; b < 4; b++) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(p + (long long)(4 * b) * cw));
            s.src[4 * b] = v.x; s.src[4 * b + 1] = v.y; s.src[4 * b + 2] = v.z; s.src[4 * b + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 16; i++) s.src[i] = ld4u(p + (long long)(4 * (i >> 2)) * cw + 4 * (i & 3));
    }
}

// The partition's place in the staged window (ws.wx0, ws.wy0), or no window.
__device__ __forceinline__ void mb_lane_window(MbLane& s, const MbScratch& ws, bool win_ok) {
    s.wox = win_ok ? s.px + ws.pad - ws.wx0 : WIN_OFF;
    s.woy = win_ok ? s.py + ws.pad - ws.wy0 : WIN_OFF;
}

// Mode 0: the 16x16 search (source words loaded by mb_load_src).
__device__ __forceinline__ void mb_lane_16x16(MbLane& s, int lx, int ly, uint32_t win) {
    const int lane = threadIdx.x & 31;
    s.lane = lane;
    s.gl = lane & 7;
    s.gb = lane & 24;
    s.px = lx; s.py = ly; s.rw = 16; s.rh = 16;
    s.winq = win + uint32_t((lane & 3) * WIN_STRIDE);
    s.gather = (s.gl >> 1) + 16 * (s.gl & 1);
    s.had = had_frag(lane);
}

// Mode 1 after mode 0: the lane's group's partition of the same MB.
__device__ __forceinline__ void mb_lane_parts(MbLane& s) {
    const int g = s.lane >> 3;
    const bool tall = g >= 2;  // 8x16
    const int ox = g == 3 ? 8 : 0, oy = g == 1 ? 8 : 0;
    s.px += ox; s.py += oy;
    s.wox += ox; s.woy += oy;
    s.rw = tall ? 8 : 16;
    s.rh = tall ? 16 : 8;
    s.gather = g + 8 * ((s.gl >> 1) & 1) + 16 * (s.gl & 1);
    uint32_t t[8];
#pragma unroll
    for (int b = 0; b < 4; b++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const uint32_t wide = g == 1 ? s.src[8 + 2 * b + i] : s.src[2 * b + i];
            const uint32_t high = g == 3 ? s.src[4 * b + 2 + i] : s.src[4 * b + i];
            t[2 * b + i] = tall ? high : wide;
        }
#pragma unroll
    for (int i = 0; i < 8; i++) s.src[i] = t[i];
}

// Where candidates are read: the MB's window in shared memory, the reference's
// planes in global memory through L1 (launch shapes without a window), or
// through L2 (passes that leave the window: the planes may be written during
// the launch).
constexpr int REF_WINDOW = 1, REF_PLANES = 0, REF_PLANES_L2 = 2;
template <int REF>
struct RefSrc;
template <>
struct RefSrc<REF_WINDOW> {
    using Addr = uint32_t;
    static __device__ __forceinline__ uint32_t ld(Addr a) { return lds_u32(a); }
    static __device__ __forceinline__ uint32_t stride(const MbScratch&) { return WIN_STRIDE; }
};
template <>
struct RefSrc<REF_PLANES> {
    using Addr = const uint8_t*;
    static __device__ __forceinline__ uint32_t ld(Addr a) { return __ldg(reinterpret_cast<const uint32_t*>(a)); }
    static __device__ __forceinline__ uint32_t stride(const MbScratch& ws) { return uint32_t(ws.pw); }
};
template <>
struct RefSrc<REF_PLANES_L2> {
    using Addr = const uint8_t*;
    static __device__ __forceinline__ uint32_t ld(Addr a) { return __ldcg(reinterpret_cast<const unsigned int*>(a)); }
    static __device__ __forceinline__ uint32_t stride(const MbScratch& ws) { return uint32_t(ws.pw); }
};
__device__ __forceinline__ uint32_t align4(uint32_t a) { return a & ~3u; }
__device__ __forceinline__ const uint8_t* align4(const uint8_t* a) {
    return reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(a) & ~uintptr_t(3));
}
__device__ __forceinline__ uint32_t shift8(uint32_t a) { return a * 8u; }  // the funnel shift takes it modulo 32
__device__ __forceinline__ uint32_t shift8(const uint8_t* a) { return uint32_t(reinterpret_cast<uintptr_t>(a)) * 8u; }

// A candidate's operands: byte addresses a (and b, equal to a at one-plane
// phases) of the lane's row of the partition's first block; a safe address
// when the reads are not covered (the window, or the planes, do not hold them).
template <int REF>
struct CandAddr {
    typename RefSrc<REF>::Addr a, b;
    bool covered;
};
template <int REF>
__device__ __forceinline__ CandAddr<REF> cand_addr(const MbLane& s, const MbScratch& ws, uint32_t lut, int mvx, int mvy) {
    CandAddr<REF> t;
    if constexpr (REF == REF_WINDOW) {
        uint2 ent;
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(ent.x), "=r"(ent.y) : "r"(lut + uint32_t(((mvx & 3) * 4 + (mvy & 3)) * 8)));
        const int wx = s.wox + (mvx >> 2), wy = s.woy + (mvy >> 2);
        t.covered = unsigned(wx) <= unsigned(WIN_W - 5 - s.rw) && unsigned(wy) <= unsigned(WIN_H - 1 - s.rh);
        const uint32_t base = t.covered ? s.winq + uint32_t(wy * WIN_STRIDE + wx) : s.winq;
        t.a = base + ent.x;
        t.b = base + ent.y;
    } else {
        const uint32_t pb = phase_bits(mvx & 3, mvy & 3);
        const long long ps = (long long)ws.pw * ws.ph;
        const int x = s.px + ws.pad + (mvx >> 2), y = s.py + ws.pad + (mvy >> 2);
        t.covered = x >= 0 && y >= 0 && x + s.rw + 5 <= ws.pw && y + s.rh + 1 <= ws.ph;
        const uint8_t* base = ws.base + (long long)(s.lane & 3) * ws.pw + (t.covered ? (long long)y * ws.pw + x : 0);
        t.a = base + ps * (pb & 3u) + ((pb & 32u) ? ws.pw : 0) + ((pb >> 4) & 1u);
        t.b = ((pb >> 2) & 3u) ? base + ps * ((pb >> 2) & 3u) + ((pb & 128u) ? ws.pw : 0) + ((pb >> 6) & 1u) : t.a;
    }
    return t;
}

// One word (4 pixels of a row) of the prediction at picture position (x, y)
// for MV (mvx, mvy), from the planes with every coordinate clamped where it
// leaves them: pred_rows for one row.
__device__ __noinline__ static uint32_t plane_word(const MbScratch& ws, int x, int y, int mvx, int mvy) {
    const int fx = mvx & 3, fy = mvy & 3, px = x + (mvx >> 2) + ws.pad, py = y + (mvy >> 2) + ws.pad;
    const int pw = ws.pw, ph = ws.ph;
    const long long ps = (long long)pw * ph;
    const bool cg = ws.bw != nullptr;
    const uint32_t pb = phase_bits(fx, fy);
    const int pa = int(pb & 3), pbb = int((pb >> 2) & 3);
    uint32_t out[2];
#pragma unroll 1
    for (int k = 0; k < 2; k++) {
        const uint8_t* P = ws.base + ps * (k ? pbb : pa);
        const int xo = px + int((pb >> (k ? 6 : 4)) & 1), yo = py + int((pb >> (k ? 7 : 5)) & 1);
        const uint8_t* row = P + (long long)clampi(yo, 0, ph - 1) * pw;
        uint32_t w = 0;
        if (xo >= 0 && xo + 8 <= pw) {
            const uintptr_t ad = reinterpret_cast<uintptr_t>(row + xo);
            const uint32_t* p = reinterpret_cast<const uint32_t*>(ad & ~uintptr_t(3));
            w = __funnelshift_r(ldw(p, cg), ldw(p + 1, cg), uint32_t(ad & 3) * 8u);
        } else {
#pragma unroll 1
            for (int c = 0; c < 4; c++) w |= uint32_t(ldb(row + clampi(xo + c, 0, pw - 1), cg)) << (8 * c);
        }
        out[k] = w;
        if (pbb == 0) return w;
    }
    return avg_up4(out[0], out[1]);
}

// Rows of the 4x4 block at (x, y) under an MV from the planes (pred_rows), for
// the MB in a hundred whose pick its window does not cover.
__device__ __noinline__ static uint4 plane_rows(const MbScratch* ws, int x, int y, int mvx, int mvy) {
    uint4 r;
    r.x = plane_word(*ws, x, y, mvx, mvy);
    r.y = plane_word(*ws, x, y + 1, mvx, mvy);
    r.z = plane_word(*ws, x, y + 2, mvx, mvy);
    r.w = plane_word(*ws, x, y + 3, mvx, mvy);
    return r;
}

// The sixteen words of a pass: mode 0 the candidate's (four block rows of
// five aligned words), mode 1 tile A's and tile B's eight (four pairs of
// adjacent blocks, three words each).
template <int MODE, int REF>
__device__ __forceinline__ void pass_words(const MbLane& s, const MbScratch& ws, typename RefSrc<REF>::Addr a0,
                                           typename RefSrc<REF>::Addr b0, uint32_t p[16]) {
    using R = RefSrc<REF>;
    const auto a = align4(a0);
    const uint32_t sa = shift8(a0);
    if constexpr (MODE == 0) {
#pragma unroll
        for (int r = 0; r < 4; r++) {
            uint32_t w[5];
#pragma unroll
            for (int i = 0; i < 5; i++) w[i] = R::ld(a + (r * 4 * R::stride(ws) + 4 * i));
#pragma unroll
            for (int i = 0; i < 4; i++) p[4 * r + i] = __funnelshift_r(w[i], w[i + 1], sa);
        }
    } else {
        const auto b = align4(b0);
        const uint32_t sb = shift8(b0);
        const uint32_t o1 = s.rw == 8 ? 4 * R::stride(ws) : 8u, o2 = (s.rw == 8 ? 8 : 4) * R::stride(ws);
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const auto ad = (k < 4 ? a : b) + ((k & 1) ? o1 : 0u) + ((k & 2) ? o2 : 0u);
            const uint32_t w0 = R::ld(ad), w1 = R::ld(ad + 4), w2 = R::ld(ad + 8);
            p[2 * k] = __funnelshift_r(w0, w1, k < 4 ? sa : sb);
            p[2 * k + 1] = __funnelshift_r(w1, w2, k < 4 ? sa : sb);
        }
    }
}

// The columns of a pass whose candidates' reads the window does not cover
// (`miss`: the lane's), from the planes; ax, ay / bx, by: the column's MVs in
// tiles A and B (mode 0: A) of the rw-wide partition at (px, py).  Returns the
// shares of the column sums as a0 | a1 << 16, b0 | b1 << 16 (each below 2^16:
// 8 blocks of at most 2 x 4,080), and the row SADs of both tiles, put in their
// places among the other columns' in `part`.  Out of line, with nothing of the search's state
// in memory: between one pass in a hundred and one in ten needs it (at the
// edges of fast objects; one in four with 16-pixel steps), and the wavefront
// may wait for it, so only the missing columns are read, the second plane only
// where a phase has one, and all loads are in flight together unless a read
// leaves the planes.  (A pass that read every column from both operands through
// L2, and the source beside them, took 3,900 cycles, 5,400 for the partitions;
// this one 2,600 and 2,800.)  Inlined for the presets other than Balanced, whose
// steps leave the window more often and whose kernels have the registers: `own`
// the lane's source words then.
template <int MODE, bool CG>
__device__ __forceinline__ int4 slow_columns(MbScratch* ws, const HadFrag& had, const uint32_t* own, int px, int py, int rw, int ax, int ay,
                                             int bx, int by, bool miss, int4 part) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int REF = CG ? REF_PLANES_L2 : REF_PLANES;
    const int lane = threadIdx.x & 31, rh = MODE == 0 ? 16 : 24 - rw;
    if (CG && miss) band_wait_px(ws->bw, &ws->bready, py + (max(ay, by) >> 2) + rh + 1, px + (max(ax, bx) >> 2) + rw + 1);
    __syncwarp();
    MbLane s;
    s.lane = lane;
    s.px = px; s.py = py; s.rw = rw; s.rh = rh;
    // block k of the pass: 16 wide, four a row; 8 wide, two
    const bool wide = MODE == 0 || rw == 16;
    const uint8_t* const src = ws->src + (long long)(py + (lane & 3)) * ws->cw + px;
    const long long sstep = 4LL * ws->cw;
    const CandAddr<REF> ta = cand_addr<REF>(s, *ws, 0u, ax, ay), tb = cand_addr<REF>(s, *ws, 0u, bx, by);
    int a0 = 0, a1 = 0, b0 = 0, b1 = 0, sa = 0, sb = 0;
    if (__all_sync(FULL, !miss || (ta.covered && tb.covered))) {
        uint32_t p[16];
#pragma unroll
        for (int i = 0; i < 16; i++) p[i] = 0;
        if (__any_sync(FULL, miss && ((ax | ay | bx | by) & 1))) {  // quarter phases have two operands
            if (miss) {
                uint32_t r[16];
                pass_words<MODE, REF>(s, *ws, ta.a, tb.a, p);
                pass_words<MODE, REF>(s, *ws, ta.b, tb.b, r);
#pragma unroll
                for (int i = 0; i < 16; i++) p[i] = avg_up4(p[i], r[i]);
            }
        } else if (miss) {
            pass_words<MODE, REF>(s, *ws, ta.a, tb.a, p);
        }
        __syncwarp();
        uint32_t sw[MODE == 0 ? 16 : 8];
#pragma unroll
        for (int k = 0; k < (MODE == 0 ? 16 : 8); k++)
            sw[k] = own != nullptr ? own[k] : ld4u(src + (wide ? k >> 2 : k >> 1) * sstep + 4 * (wide ? k & 3 : k & 1));  // (from L1)
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t va = sw[i], vb = sw[MODE == 0 ? 8 + i : i];
            had_mma(had, p[i], va, a0, a1);
            had_mma(had, p[8 + i], vb, b0, b1);
            sa += int(__vsadu4(p[i], va));
            sb += int(__vsadu4(p[8 + i], vb));
        }
    } else {
#pragma unroll 1
        for (int j = 0; j < 16; j++) {
            const bool second = MODE == 1 && j >= 8;
            const int k = MODE == 0 ? j : j & 7;
            const int xo = wide ? 4 * (k & 3) : 4 * (k & 1), yo = wide ? 4 * (k >> 2) : 4 * (k >> 1);
            const uint32_t sw = ld4u(src + (wide ? k >> 2 : k >> 1) * sstep + xo);
            uint32_t pw = 0;
            if (miss) pw = plane_word(*ws, px + xo, py + yo + (lane & 3), second ? bx : ax, second ? by : ay);
            __syncwarp();
            int t0 = 0, t1 = 0;
            had_mma(had, pw, sw, t0, t1);
            const int sd = int(__vsadu4(pw, sw));
            if (j >= 8) { b0 += t0; b1 += t1; sb += sd; }
            else { a0 += t0; a1 += t1; sa += sd; }
        }
    }
    // columns 2q and 2q + 1 (four lanes each) and the lane's own, as they missed
    const unsigned m = __ballot_sync(FULL, miss) >> (8 * (lane & 3));
    const int keep = ((m & 1u) ? 0 : 0xffff) | ((m & 16u) ? 0 : int(0xffff0000u));
    part.x = (part.x & keep) | ((a0 | (a1 << 16)) & ~keep);
    part.y = (part.y & keep) | ((b0 | (b1 << 16)) & ~keep);
    if (miss) { part.z = sa; part.w = sb; }
    return part;
}
template <int MODE, bool CG>
__device__ __noinline__ int4 slow_pass(MbScratch* ws, int px, int py, int rw, int ax, int ay, int bx, int by, bool miss, int4 part) {
    return slow_columns<MODE, CG>(ws, had_frag(threadIdx.x & 31), nullptr, px, py, rw, ax, ay, bx, by, miss, part);
}

// One pass: the lane's column's candidates at ta (tile A) and, mode 1, tb
// (tile B) -- MVs ax, ay and bx, by -- give the lane's shares of
// the column sums in a0, a1 (columns 2q, 2q+1 of tile A; mode 0: of the whole
// candidate) and b0, b1 (tile B), and the lane's row SADs in sa, sb; of these
// what `satd` and `sad` ask for.  CG: planes written during the launch are read
// through L2.  two: a two-plane phase is possible.  idle: the group has no slots (its
// addresses are safe and its sums are not used).
template <int MODE, int REF, bool CG, bool INL>
__device__ __forceinline__ void price_pass(const MbLane& s, MbScratch& ws, const CandAddr<REF>& ta, const CandAddr<REF>& tb,
                                           int ax, int ay, int bx, int by, bool two, bool idle, bool satd, bool sad, int& a0,
                                           int& a1, int& b0, int& b1, int& sa, int& sb) {
    uint32_t p[16];
    pass_words<MODE, REF>(s, ws, ta.a, tb.a, p);
    if (two) {
        uint32_t r[16];
        pass_words<MODE, REF>(s, ws, ta.b, tb.b, r);
#pragma unroll
        for (int i = 0; i < 16; i++) p[i] = avg_up4(p[i], r[i]);
    }
    a0 = a1 = b0 = b1 = sa = sb = 0;
    if (satd) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            had_mma(s.had, p[i], s.src[i], a0, a1);
            had_mma(s.had, p[8 + i], s.src[MODE == 0 ? 8 + i : i], b0, b1);
        }
    }
    if (sad) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            sa += int(__vsadu4(p[i], s.src[i]));
            sb += int(__vsadu4(p[8 + i], s.src[MODE == 0 ? 8 + i : i]));
        }
    }
    const bool miss = !idle && !(ta.covered && (MODE == 0 || tb.covered));
    if (__any_sync(0xffffffffu, miss)) {
        int4 r = make_int4(a0 | (a1 << 16), b0 | (b1 << 16), sa, sb);
        if constexpr (INL)
            r = slow_columns<MODE, CG>(&ws, s.had, s.src, s.px, s.py, s.rw, ax, ay, bx, by, miss, r);
        else
            r = slow_pass<MODE, CG>(&ws, s.px, s.py, s.rw, ax, ay, bx, by, miss, r);
        a0 = r.x & 0xffff; a1 = int(uint32_t(r.x) >> 16);
        b0 = r.y & 0xffff; b1 = int(uint32_t(r.y) >> 16);
        sa = r.z; sb = r.w;
    }
    if (MODE == 0) { a0 += b0; a1 += b1; sa += sb; }
}

// The eight ring points (dx, dy) in the reference's order: (1,0) (-1,0) (0,1)
// (0,-1) (1,1) (-1,-1) (1,-1) (-1,1); the four-point diamond is the first four.
// Packed two bits per point as d+1, so a lane computes its point without a
// memory lookup.
constexpr uint32_t kRingXP = 0x2252u, kRingYP = 0x8225u;
__device__ __forceinline__ int ring_dx(int i) { return int((kRingXP >> (2 * i)) & 3u) - 1; }
__device__ __forceinline__ int ring_dy(int i) { return int((kRingYP >> (2 * i)) & 3u) - 1; }

// Proposals of the learned search's 16x16 search.
constexpr int N_PROP = 8;
constexpr int LOOP_GUARD = 1 << 20;  // iterations of one rung / sub-pel step

struct SearchOut {
    int x, y, cost, evals;
};

// ---------------------------------------------------------------------------
// The searches
// ---------------------------------------------------------------------------
// motion_search (mb16.rs:2433-3302) as a loop of rounds, each of a kind: the
// seeds (with the integer snaps of sub-pel predictors, mb16.rs:2597-2607), the
// learned search's proposals, a fixed-centre diamond of the full-pel ladder
// (all four points, first strict minimum, as the reference's argmin loops), a
// cascading ring (the centre moves mid-ring: the points left are priced
// around the current centre, the first improvement moves it, and the rest are
// priced again around the new one, the order in which the reference evaluates
// them), the B2 reprice, or a fixed-centre sub-pel ring (sp_fc).  The centre,
// `step` (quarter-pels; STEP_REPRICE between the ladder and the sub-pel steps)
// and the kind are the state; evals counts what the reference evaluates.
//
// Costs are dist + (λ·rate) as i64 held in 32 bits: distortions are below
// 2^21 and λ·rate below 2^28 for every λ the encoder forms, so the sum never
// saturates and comparisons match the reference's i64.
//
// BAL: the Balanced preset's knobs as constants, and the λ·rate products from
// a table per λ.  Host rule (balanced_preset): the preset's knobs and
// 0 <= λ < 2^23, so that every table entry and cost fits 31 bits.  Any other
// preset, or λ, runs the same rounds with its knobs read.  (One CIF frame,
// fast / walk to convergence / full ladder: 493, 1,607 and 1,641 us with four
// warps an MB and butterflies; 593, 2,004 and 2,852 with one warp and a search
// of their own for both modes, its state per lane and its sums by shuffles;
// 414, 1,472 and 1,615 this way, with the registers for it, see ME_ANY_BLOCKS.)
//
// Every decision of the 16x16 search, which every MB runs and the wavefront
// waits for, is warp-uniform: costs are compared through redux and ballots, a
// lane forms its column's candidate from the round's centre, step and ring
// index, the operand addresses come from a 16-entry table, and a pass's
// column sums cross the lanes through shared memory.
//
// LEARN with use_prop (the learned-proposal kernels' 16x16 search): after the
// seeds, the 8 proposals are priced, both with `cost` (SATD and λ also where
// the full-pel phase has a cost of its own, so that predictor and proposals
// compare); when the best proposal's distortion exceeds the predictor's by
// more than prop_t the plain search goes on from the seeds (fell = 1),
// otherwise it continues as motion_search with the cheapest of predictor and
// proposals as its start vector (mb16.rs:2445, 2579-2596: refine-only, no
// full-pel phase).  use_start: a refine-only search from `start`.

constexpr int LAM_TAB = 48;  // (λ·rate) as i64 for rates below LAM_TAB
constexpr double LAM_TAB_MAX = 8388608.0;  // of a λ whose products fit 31 bits (rates up to 126)
constexpr int STEP_REPRICE = 3;

// Per-warp tables and scratch of the searches.
struct SearchScratch {
    double lam;             // the λ the table holds (NaN: none)
    double lam_main, lam_dia;  // not BAL: the λ of `cost` and of the fixed diamond
    int lamtab[LAM_TAB];
    // a pass's shares, 64 words a tile: SATD [lane / 4][column], then SAD [column][lane % 4]
    alignas(16) int red[128];
};
static_assert(offsetof(SearchScratch, red) % 16 == 0 && sizeof(SearchScratch) % 16 == 0, "16-byte reads of the shares");
// Per-CTA operand table: byte offsets in the window of both operands of each
// quarter phase fx * 4 + fy (equal at one-plane phases).
struct PhaseTab {
    uint2 e[16];
};
__device__ __forceinline__ void phase_tab_init(PhaseTab& t, int i) {
    if (i >= 16) return;
    const uint32_t pb = phase_bits(i >> 2, i & 3);
    const uint32_t a = (pb & 3u) * WIN_PLANE + ((pb >> 5) & 1u) * WIN_STRIDE + ((pb >> 4) & 1u);
    const uint32_t b = ((pb >> 2) & 3u) * WIN_PLANE + ((pb >> 7) & 1u) * WIN_STRIDE + ((pb >> 6) & 1u);
    t.e[i] = make_uint2(a, ((pb >> 2) & 3u) ? b : a);
}
__device__ __forceinline__ void bal_lambda(SearchScratch& b, double lambda_me) {
    if (b.lam == lambda_me) return;  // warp-uniform
    __syncwarp();
    for (int r = int(threadIdx.x & 31); r < LAM_TAB; r += 32) b.lamtab[r] = int(lam_cost(lambda_me, uint32_t(r)));
    if ((threadIdx.x & 31) == 0) b.lam = lambda_me;
    __syncwarp();
}
// Exp-Golomb bits of an mvd component (mb16.rs:2454-2482, kind 0)
__device__ __forceinline__ uint32_t eg_bits(int d) {
    const uint32_t v = uint32_t(d > 0 ? 2 * d : 1 - 2 * d);
    return 63u - 2u * uint32_t(__clz(int(v)));
}
__device__ __forceinline__ int bal_rate_cost(const SearchScratch& b, double lam, int dx, int dy) {
    const uint32_t r = eg_bits(dx) + eg_bits(dy);
    return r < LAM_TAB ? b.lamtab[r] : int(lam_cost(lam, r));
}

// A preset's knobs as the searches read them: constants for BAL, else worked
// out once a search.  A round's cost is one of four: `cost`, the full-pel
// phase's cost_fp, the 16-wide fixed diamond's and the 16-wide sub-pel ring's.
constexpr int C_MAIN = 0, C_FP = 1, C_DIA = 2, C_SPFC = 3;
template <bool BAL>
struct Knobs {
    static constexpr bool kSnap = true, kFc = true, kSadfp = false, kSpFc = false;
    static constexpr int kFirst = 16, kSub = 2, kRing = 8, sads = 0, tabs = 15;
    __device__ __forceinline__ Knobs(const MeParamsDev&, double lambda_me, SearchScratch& b) { bal_lambda(b, lambda_me); }
    __device__ __forceinline__ int next_step(int step) const { return step >> 1; }
    __device__ __forceinline__ bool again(int) const { return false; }
    __device__ __forceinline__ bool sad(int) const { return false; }
};
template <>
struct Knobs<false> {
    bool kSnap, kFc, kSadfp, kSpFc, iterate;
    int kFirst, kSub, kRing;
    int ladder;  // the steps of the full-pel ladder, one bit each (64 .. 4 quarter-pels by dia_mask's bits 0..4)
    int maxit, sads, tabs;  // sads, tabs: a bit per cost
    __device__ __forceinline__ Knobs(const MeParamsDev& p, double lambda_me, SearchScratch& b) {
        const bool full = !p.fast;
        const int pat = p.subpel_pat >= 0 ? p.subpel_pat : (p.sp_single_pass ? 2 : 0);
        kSnap = p.me_snap;
        kFc = full && p.fc;
        kSadfp = full && p.sadfp;
        kSpFc = full && p.sp_fc && (pat & 1) == 0;
        iterate = p.me_subpel_iter && !(pat & 2);
        maxit = p.sp_maxit != 0 ? p.sp_maxit : INT_MAX;
        kRing = (pat & 1) ? 4 : 8;
        kSub = p.subpel ? 2 : 0;
        ladder = full ? int(__brev(p.dia_mask & 0x1fu) >> 25) : 16 + 4;
        kFirst = lower(128);
        const int m = p.use_sad ? 1 : 0, f = kSadfp ? 1 : 0;
        sads = m << C_MAIN | (f | m) << C_FP | f << C_DIA;
        // Exp-Golomb rates: the costs whose λ is λ itself read its table
        const bool tab = p.kind == 0 && lambda_me >= 0.0 && lambda_me < LAM_TAB_MAX;
        tabs = tab ? (kSadfp ? 1 << C_MAIN | 1 << C_SPFC : 15) : 0;
        if (b.lam != lambda_me) {  // warp-uniform
            __syncwarp();
            if ((threadIdx.x & 31) == 0) {
                b.lam_main = p.kind != 0 ? lambda_me * 0.25 : lambda_me;
                b.lam_dia = kSadfp ? lambda_me * p.sadfp_lambda : lambda_me;
            }
            if (!tab && (threadIdx.x & 31) == 0) b.lam = lambda_me;
            __syncwarp();
            if (tab) bal_lambda(b, lambda_me);
        }
    }
    __device__ __forceinline__ int lower(int step) const {
        const int r = ladder & (step - 1);
        return r ? 1 << (31 - __clz(r)) : (kSadfp ? STEP_REPRICE : kSub);
    }
    // the step after `step` (0: the search is done)
    __device__ __forceinline__ int next_step(int step) const {
        return step > STEP_REPRICE ? lower(step) : (step == STEP_REPRICE ? kSub : step >> 1);
    }
    // another sub-pel ring at the step after `iter` of them, the last of which improved
    __device__ __forceinline__ bool again(int iter) const { return iterate && iter < maxit; }
    __device__ __forceinline__ bool sad(int cost) const { return (sads >> cost) & 1; }
};
// (λ·rate) of an mvd, and a cost
template <bool BAL>
__device__ __forceinline__ long long rate_cost(const MeParamsDev& p, const SearchScratch& b, double lambda_me, int tabs, bool sadfp,
                                               int cost, int dx, int dy) {
    if (BAL || tabs == 15 || (tabs >> cost) & 1) return bal_rate_cost(b, lambda_me, dx, dy);
    const double l = cost == C_MAIN || (cost == C_FP && !sadfp) ? b.lam_main : (cost == C_SPFC ? lambda_me : b.lam_dia);
    return lam_cost(l, mvbits(p.kind, p.tab, dx) + mvbits(p.kind, p.tab, dy));
}
template <bool BAL>
__device__ __forceinline__ int cost_sum(int d, long long rc) {
    if constexpr (BAL) return d + int(rc);
    const long long c = (long long)d + rc;
    return c > INT_MAX - 1 ? INT_MAX - 1 : int(c);
}

// Every point of the w x h block's ring at full-pel distance st inside the picture.
__device__ __forceinline__ bool ring_inside(const MbLane& s, int cw, int ch, int x, int y, int st) {
    const int ox = s.px + (x >> 2), oy = s.py + (y >> 2);
    return ox - st >= 0 && oy - st >= 0 && ox + st + s.rw <= cw && oy + st + s.rh <= ch;
}
// hpel_qpel_refs / hpel_ref resolve the ring point (inter.rs:1015, 1060): inside
// the planes with a slack of 1, and at step 1 a quarter phase
__device__ __forceinline__ bool point_resolves(const MbLane& s, const MbScratch& ws, int x, int y, int step) {
    const int ox = s.px + (x >> 2) + ws.pad, oy = s.py + (y >> 2) + ws.pad;
    return ox >= 0 && oy >= 0 && ox + s.rw + 1 <= ws.pw && oy + s.rh + 1 <= ws.ph && (step == 2 || ((x | y) & 1));
}

// The 16x16 search (predictor p0 the mvd centre), warp-uniform.  propc / propg:
// proposals lane / 4 and lane % 8.
template <bool BAL, bool LEARN, int REF, bool CG>
__device__ __forceinline__ SearchOut search16(const MbLane& s, const MeParamsDev& prm, MbScratch& ws, SearchScratch& bs, uint32_t lut,
                                              int2 p0, double lambda_me, bool use_prop, int2 propc, int2 propg, int prop_t,
                                              int* fell) {
    constexpr int SEED = 0, DIA = 1, RING = 2, PROP = 3, SPFC = 4, REPRICE = 5;
    constexpr unsigned FULL = 0xffffffffu;
    const Knobs<BAL> kn(prm, lambda_me, bs);
    const int lane = s.lane, gl = s.gl, col = lane >> 2, cw = ws.cw, ch = ws.ch;
    const int2 q0 = make_int2(((p0.x + 2) >> 2) * 4, ((p0.y + 2) >> 2) * 4);  // its integer snap
    const bool sub = ((p0.x | p0.y) & 3) != 0;
    const int step0 = kn.kFirst;
    bool prop_next = LEARN && use_prop;  // the proposals are still to be priced
    // the first rung's ring around p0's (snapped) position in the seeds' round, where both have one cost
    const bool seed_ring = !prop_next && step0 >= 4 && kn.kFc && (kn.kSnap || !sub) && (BAL || kn.kSadfp || (!prm.use_sad && prm.kind == 0)) &&
                           ring_inside(s, cw, ch, q0.x, q0.y, step0 >> 2);
    int evals = 0, best = 0, seed_c = 0, seed_x = 0, seed_y = 0, cp = 0, dp = 0;
    int cx = q0.x, cy = q0.y, step = step0, kind = SEED, ri = 0, rn = 4;
    int iter = 0, loops = 0;  // rings at this step (not counted for BAL, whose steps end by themselves)
    int low = step0, cost = prop_next ? C_MAIN : C_FP;  // DIA: the next rung where it is >= 4; the round's cost
    bool improved = false;
    for (;;) {
        // the candidates of the lane's mma column and of its cost slot: SEED
        // 0 the zero MV, 1 p0, 2 its snap, 4..7 the first rung's ring around
        // the snap; DIA this rung's ring and the next's; RING and SPFC the
        // points from ri; REPRICE the centre and the seed
        int mx, my, rx, ry;
        {
            const int ic = kind == RING ? min(ri + col, 7) : (kind == SPFC ? col : col & 3),
                      ig = kind == RING ? min(ri + gl, 7) : (kind == SPFC ? gl : gl & 3);
            const int lw = BAL ? step >> 1 : low;
            const int sc = kind == DIA && col >= 4 ? lw : step, sg = kind == DIA && gl >= 4 ? lw : step;
            mx = cx + ring_dx(ic) * sc; my = cy + ring_dy(ic) * sc;
            rx = cx + ring_dx(ig) * sg; ry = cy + ring_dy(ig) * sg;
            if (kind == SEED) {
                if (col < 4 || !seed_ring) { mx = col == 0 ? 0 : (col == 1 ? p0.x : q0.x); my = col == 0 ? 0 : (col == 1 ? p0.y : q0.y); }
                if (gl < 4 || !seed_ring) { rx = gl == 0 ? 0 : (gl == 1 ? p0.x : q0.x); ry = gl == 0 ? 0 : (gl == 1 ? p0.y : q0.y); }
            }
            if (LEARN && kind == PROP) { mx = propc.x; my = propc.y; rx = propg.x; ry = propg.y; }
            if (!BAL && kind == REPRICE) {
                mx = col == 1 ? seed_x : cx; my = col == 1 ? seed_y : cy;
                rx = gl == 1 ? seed_x : cx; ry = gl == 1 ? seed_y : cy;
            }
        }
        const bool sad = kn.sad(cost);
        const CandAddr<REF> ta = cand_addr<REF>(s, ws, lut, mx, my);
        const long long rc = rate_cost<BAL>(prm, bs, lambda_me, kn.tabs, kn.kSadfp, cost, rx - p0.x, ry - p0.y);
        int a0, a1, b0, b1, sa, sb;
        // a two-plane phase is possible among the seeds, at quarter-pel steps
        // and, from a start vector, around a quarter-pel centre
        const bool two = BAL ? kind == SEED || step == 1 || (LEARN && (kind == PROP || ((cx | cy) & 1))) : __any_sync(FULL, (mx | my) & 1);
        price_pass<0, REF, CG, !BAL>(s, ws, ta, ta, mx, my, mx, my, two, false, !sad, sad, a0, a1, b0, b1, sa, sb);
        // column sums through shared memory: slot gl's eight shares, or four rows' SADs
        int d = 0;
        if (!sad) {
            *reinterpret_cast<int2*>(&bs.red[8 * col + 2 * (lane & 3)]) = make_int2(a0, a1);
            __syncwarp();
#pragma unroll
            for (int g = 0; g < 8; g++) d += bs.red[8 * g + gl];
        } else {
            bs.red[lane] = sa;
            __syncwarp();
            const int4 r = *reinterpret_cast<const int4*>(&bs.red[4 * gl]);
            d = r.x + r.y + r.z + r.w;
        }
        __syncwarp();  // read by every lane: the next round stores its own
        const int cc = cost_sum<BAL>(d, rc);
        bool stay = false;  // another ring at this step
        if (kind == RING) {
            const unsigned hit = __ballot_sync(FULL, gl < rn - ri && cc < best) & 0xffu;
            if (hit) {
                const int j = __ffs(hit) - 1;
                best = __reduce_min_sync(FULL, gl == j ? cc : INT_MAX);
                evals += j + 1;
                cx += ring_dx(ri + j) * step;
                cy += ring_dy(ri + j) * step;
                improved = true;
                ri += j + 1;
            } else {
                evals += rn - ri;
                ri = rn;
            }
            if (ri < rn) continue;  // the rest of the ring around the moved centre
            stay = improved && (step >= 4 || kn.again(iter));
        } else {
            // the minima of slots 0..3 and 4..7 and their first slots
            const int m0 = __reduce_min_sync(FULL, gl < 4 ? cc : INT_MAX), m1 = __reduce_min_sync(FULL, gl < 4 ? INT_MAX : cc);
            const unsigned at = __ballot_sync(FULL, cc == (gl < 4 ? m0 : m1)) & 0xffu;
            const int j0 = __ffs(at) - 1, j1 = __ffs(at >> 4) - 1;
            if (kind == DIA) {
                evals += 4;
                stay = true;
                if (m0 < best) {
                    best = m0;
                    cx += ring_dx(j0) * step;
                    cy += ring_dy(j0) * step;
                } else if ((BAL ? step >> 1 : low) >= 4) {  // the next rung's first ring, priced beside it
                    step = BAL ? step >> 1 : low;
                    loops = 0;
                    evals += 4;
                    if (m1 < best) {
                        best = m1;
                        cx += ring_dx(j1) * step;
                        cy += ring_dy(j1) * step;
                    } else {
                        stay = false;
                    }
                } else {
                    stay = false;
                }
            } else if (kind == SEED) {
                // sequential strict-< scan: (0,0), then the predictor; the
                // winner's integer snap is the centre
                const int c0 = __reduce_min_sync(FULL, gl == 0 ? cc : INT_MAX), c1 = __reduce_min_sync(FULL, gl == 1 ? cc : INT_MAX),
                          c2 = __reduce_min_sync(FULL, gl == 2 ? cc : INT_MAX);
                if (LEARN) {
                    cp = c1;
                    dp = __reduce_min_sync(FULL, gl == 1 ? d : INT_MAX);
                }
                evals += 2;
                if (c1 < c0) {
                    best = seed_c = c1;
                    seed_x = p0.x; seed_y = p0.y;
                    if (sub && kn.kSnap) {
                        best = c2;
                        evals += 1;
                    } else if (!BAL) {
                        cx = p0.x; cy = p0.y;
                    }
                } else {
                    best = seed_c = c0;
                    seed_x = seed_y = 0;
                    cx = cy = 0;
                }
                if (LEARN && (BAL ? use_prop : prop_next)) {  // (the seeds come once for BAL)
                    kind = PROP;
                    continue;
                }
                stay = true;
                if (seed_ring && cx == q0.x && cy == q0.y) {
                    evals += 4;
                    if (m1 < best) {
                        best = m1;
                        cx += ring_dx(j1) * step;
                        cy += ring_dy(j1) * step;
                    } else {
                        stay = false;
                    }
                }
            } else if (!BAL && kind == SPFC) {
                const int m = min(m0, m1), j = m0 == m ? j0 : 4 + j1;
                evals += 8;
                if (m < best) {
                    best = m;
                    cx += ring_dx(j) * step;
                    cy += ring_dy(j) * step;
                    stay = kn.again(iter);
                }
            } else if (!BAL && kind == REPRICE) {
                best = __reduce_min_sync(FULL, gl == 0 ? cc : INT_MAX);
                seed_c = __reduce_min_sync(FULL, gl == 1 ? cc : INT_MAX);
                evals += 2;
            } else {  // PROP: the cheapest proposal (first wins) against the predictor
                const int m = min(m0, m1), j = m0 == m ? j0 : 4 + j1;
                const int dprop = __reduce_min_sync(FULL, gl == j ? d : INT_MAX);
                const bool fb = dprop - dp > prop_t;
                *fell = fb ? 1 : 0;
                prop_next = false;
                stay = true;
                if (!fb) {
                    evals = N_PROP + 1;
                    best = cp;
                    cx = p0.x; cy = p0.y;
                    if (m < cp) {
                        best = m;
                        cx = __shfl_sync(FULL, propg.x, j);
                        cy = __shfl_sync(FULL, propg.y, j);
                    }
                    seed_c = best; seed_x = cx; seed_y = cy;
                    step = kn.kSub;  // a start vector: the sub-pel steps only
                } else if (kn.kSadfp) {
                    // the plain search's seeds, priced again with its full-pel cost
                    evals = N_PROP + 1;
                    cx = q0.x; cy = q0.y;
                    kind = SEED;
                    cost = C_FP;
                    continue;
                } else {
                    evals += N_PROP + 1;  // the plain search goes on from its seeds
                }
            }
        }
        if (BAL) {
            if (!stay) step >>= 1;
        } else if (!stay || ++loops >= LOOP_GUARD) {
            step = kn.next_step(step);
            iter = loops = 0;
        }
        if (step == 0) break;
        improved = false;
        ri = 0;
        rn = step >= 4 ? 4 : kn.kRing;
        kind = RING;
        if constexpr (BAL) {
            if (step >= 4 && ring_inside(s, cw, ch, cx, cy, step >> 2)) kind = DIA;
        } else {
            iter++;
            cost = C_MAIN;
            if (step >= 4) {
                cost = C_FP;
                if (kn.kFc && ((cx | cy) & 3) == 0 && ring_inside(s, cw, ch, cx, cy, step >> 2)) {
                    kind = DIA;
                    cost = C_DIA;
                    low = kn.lower(step);
                }
            } else if (step == STEP_REPRICE) {
                kind = REPRICE;
            } else if (kn.kSpFc && (step == 1 || ((cx | cy) & 3) == 0) &&
                       __all_sync(FULL, point_resolves(s, ws, cx + ring_dx(gl) * step, cy + ring_dy(gl) * step, step))) {
                kind = SPFC;
                cost = C_SPFC;
            }
        }
    }
    // ---- seed restore (mb16.rs:3297-3300) ----
    if (kn.kSnap && seed_c < best) {
        cx = seed_x; cy = seed_y; best = seed_c;
    }
    return SearchOut{cx, cy, best, evals};
}

// The four partitions, group g of eight lanes searching partition g (mode 1):
// seeds (0,0), p0 (the mvd centre), p1, then as search16, four slots a round
// (a fixed-centre ring of eight takes two).  use_start: refine-only from `start`.
template <bool BAL, bool LEARN, int REF, bool CG>
__device__ __forceinline__ SearchOut search_parts(const MbLane& s, const MeParamsDev& prm, MbScratch& ws, SearchScratch& bs, uint32_t lut,
                                                  int2 p0, int2 p1, double lambda_me, bool use_start, int2 start) {
    constexpr int SEED = 0, DIA = 1, RING = 2, SNAP = 3, START = 4, DONE = 5, SPFC = 6, REPRICE = 7;
    constexpr unsigned FULL = 0xffffffffu;
    const Knobs<BAL> kn(prm, lambda_me, bs);
    const int gl = s.gl, gb = s.gb, sl = gl & 3, grp = gb >> 3, half = (s.lane >> 2) & 1, cw = ws.cw, ch = ws.ch;
    auto snap = [](int v) { return ((v + 2) >> 2) * 4; };
    const bool two = p1.x != p0.x || p1.y != p0.y;  // equal predictors: p1 cannot win
    // seed slots: 0 the zero MV, 1 p0, 2 p1, 3 the snap of p1 (the likely winner)
    const int2 q0 = make_int2(snap(p0.x), snap(p0.y)), q1 = make_int2(snap(p1.x), snap(p1.y));
    const bool sub1 = ((p1.x | p1.y) & 3) != 0;
    int evals = 0, best = 0, seed_c = 0, seed_x = 0, seed_y = 0;
    int cx = 0, cy = 0, step = kn.kFirst, kind = SEED, ri = 0, rn = 4;
    int iter = 0, loops = 0, fm = 0, fj = 0;  // SPFC: the first four points' minimum and its point
    int cost = C_FP;
    bool improved = false;
    if (LEARN && use_start) {
        kind = START;
        cost = C_MAIN;
        cx = seed_x = start.x;
        cy = seed_y = start.y;
    }
    while (!__all_sync(FULL, kind == DONE)) {
        // the MV of slot i of this round
        auto slot_mv = [&](int i, int& x, int& y) {
            const int ir = kind == RING || (!BAL && kind == SPFC) ? min(ri + i, 7) : i;
            x = cx + ring_dx(ir) * step;
            y = cy + ring_dy(ir) * step;
            if (kind == SEED) {
                x = i == 0 ? 0 : (i == 1 ? p0.x : (i == 2 ? p1.x : q1.x));
                y = i == 0 ? 0 : (i == 1 ? p0.y : (i == 2 ? p1.y : q1.y));
            } else if (kind >= SNAP && (BAL || kind <= DONE)) {  // (DONE: a position the window covers)
                x = cx;
                y = cy;
            } else if (!BAL && kind == REPRICE) {
                x = i == 1 ? seed_x : cx;
                y = i == 1 ? seed_y : cy;
            }
        };
        int ax, ay, bx, by, rx, ry;
        slot_mv(half, ax, ay);
        slot_mv(half + 2, bx, by);
        slot_mv(sl, rx, ry);
        const bool sad = kn.sad(cost);
        bool any_satd = true, any_sad = false;
        if (!BAL && kn.sads != 0) {
            any_satd = __any_sync(FULL, kind != DONE && !sad);
            any_sad = __any_sync(FULL, kind != DONE && sad);
        }
        const CandAddr<REF> ta = cand_addr<REF>(s, ws, lut, ax, ay), tb = cand_addr<REF>(s, ws, lut, bx, by);
        const long long rc = rate_cost<BAL>(prm, bs, lambda_me, kn.tabs, kn.kSadfp, cost, rx - p0.x, ry - p0.y);
        const bool planes2 = __any_sync(FULL, ((ax | ay | bx | by) & 1) != 0 && kind != DONE);  // quarter phases
        int a0, a1, b0, b1, sa, sb;
        price_pass<1, REF, CG, !BAL>(s, ws, ta, tb, ax, ay, bx, by, planes2, kind == DONE, any_satd, any_sad, a0, a1, b0, b1, sa, sb);
        // column sums through shared memory: columns 2g, 2g+1 of tile A are
        // slots 0, 1 of group g, of tile B slots 2, 3
        int d = 0;
        if (any_satd) {
            int* const mine = &bs.red[8 * (s.lane >> 2) + 2 * (s.lane & 3)];
            *reinterpret_cast<int2*>(mine) = make_int2(a0, a1);
            *reinterpret_cast<int2*>(mine + 64) = make_int2(b0, b1);
            __syncwarp();
#pragma unroll
            for (int g = 0; g < 8; g++) d += bs.red[64 * (sl >> 1) + 8 * g + 2 * grp + (sl & 1)];
            __syncwarp();  // as in search16
        }
        if (any_sad) {
            bs.red[s.lane] = sa;
            bs.red[64 + s.lane] = sb;
            __syncwarp();
            const int4 r = *reinterpret_cast<const int4*>(&bs.red[64 * (sl >> 1) + 4 * (2 * grp + (sl & 1))]);
            if (sad) d = r.x + r.y + r.z + r.w;
            __syncwarp();
        }
        const int cc = cost_sum<BAL>(d, rc);
        // collectives of every group's fold
        const int n = rn - ri < 4 ? rn - ri : 4;
        const unsigned hit = (__ballot_sync(FULL, sl < n && cc < best) >> gb) & 0xfu;
        const int jh = hit ? __ffs(hit) - 1 : 0;
        int m = min(cc, __shfl_xor_sync(FULL, cc, 1));
        m = min(m, __shfl_xor_sync(FULL, m, 2));
        const int jm = __ffs((__ballot_sync(FULL, cc == m) >> gb) & 0xfu) - 1;
        const int cj = __shfl_sync(FULL, cc, gb + jh);
        const int c0 = __shfl_sync(FULL, cc, gb), c1 = __shfl_sync(FULL, cc, gb + 1), c2 = __shfl_sync(FULL, cc, gb + 2),
                  c3 = __shfl_sync(FULL, cc, gb + 3);
        bool next = false, stay = false;  // the round's ring or rung is done; another at its step
        if (kind == RING) {
            if (hit) {
                best = cj;
                evals += jh + 1;
                cx += ring_dx(ri + jh) * step;
                cy += ring_dy(ri + jh) * step;
                improved = true;
                ri += jh + 1;
            } else {
                evals += n;
                ri += n;
            }
            next = ri >= rn;
            stay = improved && (step >= 4 || kn.again(iter));
        } else if (kind == DIA) {
            evals += 4;
            if (m < best) {
                best = m;
                cx += ring_dx(jm) * step;
                cy += ring_dy(jm) * step;
                stay = true;
            }
            next = true;
        } else if (kind == SEED) {
            // sequential strict-< scan: (0,0), p0, p1; a sub-pel winner's
            // integer snap is the centre
            evals = 3;
            best = seed_c = c0;
            next = stay = true;
            if (c1 < best) { best = seed_c = c1; cx = seed_x = p0.x; cy = seed_y = p0.y; }
            if (two && c2 < best) { best = seed_c = c2; cx = seed_x = p1.x; cy = seed_y = p1.y; }
            if (kn.kSnap && best == c2 && two && cx == p1.x && cy == p1.y && sub1) {
                best = c3;
                cx = q1.x; cy = q1.y;
                evals = 4;
            } else if (kn.kSnap && ((cx | cy) & 3)) {  // p0 won
                evals = 4;
                cx = q0.x; cy = q0.y;
                if (cx == q1.x && cy == q1.y) {
                    best = c3;
                } else {
                    kind = SNAP;  // price its snap
                    next = false;
                }
            }
        } else if (kind == SNAP) {
            best = c0;
            next = stay = true;
        } else if (LEARN && kind == START) {
            best = seed_c = c0;
            evals = 1;
            step = kn.kSub;
            next = stay = true;
        } else if (!BAL && kind == SPFC) {
            if (ri == 0) {
                fm = m; fj = jm;
                ri = 4;
            } else {
                if (m < fm) { fm = m; fj = 4 + jm; }
                evals += 8;
                next = true;
                if (fm < best) {
                    best = fm;
                    cx += ring_dx(fj) * step;
                    cy += ring_dy(fj) * step;
                    stay = kn.again(iter);
                }
            }
        } else if (!BAL && kind == REPRICE) {
            best = c0;
            seed_c = c1;
            evals += 2;
            next = true;
        }
        if (next) {
            if (BAL) {
                if (!stay) step >>= 1;
            } else if (!stay || ++loops >= LOOP_GUARD) {
                step = kn.next_step(step);
                iter = loops = 0;
            }
            improved = false;
            ri = 0;
            rn = step >= 4 ? 4 : kn.kRing;
            if constexpr (BAL) {
                kind = step == 0 ? DONE : (step >= 4 && ring_inside(s, cw, ch, cx, cy, step >> 2) ? DIA : RING);
            } else {
                iter++;
                kind = step == 0 ? DONE : (step == STEP_REPRICE ? REPRICE : RING);
                cost = C_MAIN;
                if (step >= 4) {
                    cost = C_FP;
                    if (kn.kFc && ((cx | cy) & 3) == 0 && ring_inside(s, cw, ch, cx, cy, step >> 2)) {
                        kind = DIA;
                        if (s.rw == 16) cost = C_DIA;
                    }
                }
            }
        }
        if (!BAL && kn.kSpFc) {
            // a sub-pel ring about to start: all its points resolve
            const bool r = point_resolves(s, ws, cx + ring_dx(gl) * step, cy + ring_dy(gl) * step, step);
            const unsigned all = (__ballot_sync(FULL, r) >> gb) & 0xffu;
            if (next && kind == RING && step < STEP_REPRICE && (step == 1 || ((cx | cy) & 3) == 0) && all == 0xffu) {
                kind = SPFC;
                if (s.rw == 16) cost = C_SPFC;
            }
        }
    }
    if (kn.kSnap && seed_c < best) {
        cx = seed_x; cy = seed_y; best = seed_c;
    }
    return SearchOut{cx, cy, best, evals};
}

}  // namespace h264a

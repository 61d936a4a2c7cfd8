// deblock.cu -- §8f row 3: in-loop deblocking of the plain-ME P pictures
// (crates/rusty_h264-common/src/deblock.rs).
//
// The reference filters MBs in raster order, in place: per MB the luma
// vertical edges, the luma horizontal edges, then per chroma plane its
// vertical and horizontal edges.  An MB's filtering reads and writes three
// samples into its left and top neighbours, so MB (x, y)'s horizontal edges
// need MB (x + 1, y - 1)'s vertical ones: rows run as a wavefront, and a
// row's MBs one after another.
//
// deblock_bs_kernel first finds every MB's 32 edge strengths, in parallel, as
// two bit masks.  deblock_rows_kernel then gives each MB row to one warp,
// which keeps the running MB in shared-memory tiles, so the left neighbour's
// samples never leave the warp; a CTA holds several consecutive rows, which
// hand the three bottom sample rows of each finished MB to the row below
// through shared memory, and only a CTA's last row goes through global
// memory (bounded waits throughout).  One line per lane, luma rows / columns on
// lanes 0..15 and chroma on 16..31, filtered in registers through all edges of
// a direction by one code.  The chain is W MBs along a row and one more MB
// per row down, each a few hundred cycles; an MB per warp with its neighbours'
// samples and flags through L2 took 6.9 us per step of W + 2H - 3.
#include <algorithm>
#include <cstring>
#include <vector>

#include "deblock_device.cuh"

namespace h264a {

struct DbFrameDesc {
    uint8_t* y;
    uint8_t* uv[2];
    const int32_t* picks;
    const int16_t* coeffs;
    int cw, ch, mb_w, mb_h, flag_base, row_base;  // its first MB and MB row in the batch
    DbThresh th;
};
constexpr int DB_MAXF = 64;
struct DbBatch {
    DbFrameDesc f[DB_MAXF];  // most MB rows first
    int n;
};

// Edge strengths of an MB: bit 16 * horizontal + 4 * edge + segment of m1
// (bS 1) and m2 (bS 2).
struct DbStrength {
    uint32_t m1, m2;
};

constexpr int DB_BS_WARPS = 8;
__global__ void __launch_bounds__(32 * DB_BS_WARPS) deblock_bs_kernel(const __grid_constant__ DbBatch batch, long long total,
                                                                      DbStrength* __restrict__ out) {
    const long long g = (long long)blockIdx.x * DB_BS_WARPS + (threadIdx.x >> 5);
    if (g >= total) return;
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = batch.n - 1;  // the frame: last whose first MB is at or before g
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (batch.f[mid].flag_base <= g) lo = mid; else hi = mid - 1;
    }
    const DbFrameDesc& fd = batch.f[lo];
    const int m = int(g - fd.flag_base), mbx = m % fd.mb_w, mby = m / fd.mb_w;
    const bool left = mbx > 0, top = mby > 0;
    // coefficient flags: lanes 0..15 the MB's blocks in raster order, 16..19
    // the left MB's (3, 0..3), 20..23 the top MB's (0..3, 3)
    const int nb = lane < 16 ? m : (lane < 20 ? m - 1 : m - fd.mb_w);
    const int bx = lane < 16 ? lane & 3 : (lane < 20 ? 3 : lane & 3), by = lane < 16 ? lane >> 2 : (lane < 20 ? lane & 3 : 3);
    bool nz = false;
    if (lane < 16 || (lane < 20 && left) || (lane >= 20 && lane < 24 && top)) {
        const int qi = (by >= 2 ? 2 : 0) + (bx >= 2 ? 1 : 0), k = (by & 1) * 2 + (bx & 1);
        const uint4* c = reinterpret_cast<const uint4*>(fd.coeffs + (long long)nb * 256 + (qi * 4 + k) * 16);
        const uint4 u = __ldg(c), v = __ldg(c + 1);
        nz = (u.x | u.y | u.z | u.w | v.x | v.y | v.z | v.w) != 0u;
    }
    const unsigned nzm = __ballot_sync(0xffffffffu, nz);
    // the lane's segment: block (qbx, qby) against the block left of or above it
    const int hor = lane >> 4, e = (lane >> 2) & 3, sg = lane & 3;
    const bool edge = e > 0 || (hor ? top : left);
    int bs = 0;
    if (edge) {
        const int qbx = hor ? sg : e, qby = hor ? e : sg;
        const int pbx = e > 0 ? (hor ? sg : e - 1) : (hor ? sg : 3), pby = e > 0 ? (hor ? e - 1 : sg) : (hor ? 3 : sg);
        auto mv = [&](int mb, int x4, int y4) {
            const int32_t* p = fd.picks + 6LL * mb;
            const int shape = __ldg(p);
            const int part = shape == 1 ? (y4 >= 2) : (shape == 2 ? (x4 >= 2) : 0);
            return make_int2(__ldg(p + 1 + 2 * part), __ldg(p + 2 + 2 * part));
        };
        const int2 qm = mv(m, qbx, qby), pm = mv(e > 0 ? m : (hor ? m - fd.mb_w : m - 1), pbx, pby);
        const int pbit = e > 0 ? 4 * pby + pbx : (hor ? 20 + sg : 16 + sg);
        bs = bs_of((nzm >> pbit) & 1u, (nzm >> (4 * qby + qbx)) & 1u, pm.x, pm.y, qm.x, qm.y);
    }
    const unsigned m1 = __ballot_sync(0xffffffffu, bs == 1), m2 = __ballot_sync(0xffffffffu, bs == 2);
    if (lane == 0) out[g] = DbStrength{m1, m2};
}

// A line's filter parameters: luma and chroma lanes run the same code, chroma
// with tc = tc0 + 1 and p1, q1 untouched (filter_chroma_line).
struct DbLine {
    int alpha, beta, tc1, tc2;
    bool luma;
};
// filter_luma_line / filter_chroma_line (deblock.rs:67-137) at bS 1..2 across
// p2 p1 p0 | q0 q1 q2; bs 0 leaves them.
__device__ __forceinline__ void db_filter(const DbLine& d, int bs, int p2, int& p1, int& p0, int& q0, int& q1, int q2) {
    const bool on = bs != 0 && abs(p0 - q0) < d.alpha && abs(p1 - p0) < d.beta && abs(q1 - q0) < d.beta;
    const int tc0 = bs == 1 ? d.tc1 : d.tc2;
    const bool ap = d.luma && abs(p2 - p0) < d.beta, aq = d.luma && abs(q2 - q0) < d.beta;
    const int tc = tc0 + (d.luma ? int(ap) + int(aq) : 1);
    const int delta = clip3(-tc, tc, (((q0 - p0) << 2) + (p1 - q1) + 4) >> 3);
    const int avg = (p0 + q0 + 1) >> 1;
    const int np1 = p1 + clip3(-tc0, tc0, (p2 + avg - 2 * p1) >> 1), nq1 = q1 + clip3(-tc0, tc0, (q2 + avg - 2 * q1) >> 1);
    p0 = on ? clip1(p0 + delta) : p0;
    q0 = on ? clip1(q0 - delta) : q0;
    p1 = on && ap ? np1 : p1;  // between p1 and its neighbours: no clip needed
    q1 = on && aq ? nq1 : q1;
}
// The edges of one direction of the lane's line px[0..19] (luma edges at 4, 8,
// 12, 16; chroma at 4 and 8); bits: two per edge.
__device__ __forceinline__ void db_line(const DbLine& d, unsigned bits, int px[20]) {
    const unsigned any = __reduce_or_sync(0xffffffffu, bits);  // edges no line of the MB filters are skipped
#pragma unroll
    for (int e = 0; e < 4; e++)
        if ((any >> (2 * e)) & 3u)
            db_filter(d, int((bits >> (2 * e)) & 3u), px[4 * e + 1], px[4 * e + 2], px[4 * e + 3], px[4 * e + 4],
                      px[4 * e + 5], px[4 * e + 6]);
}

// (eight 1080p pictures with 4, 6, 8, 16 rows a CTA: 529, 520, 524, 565 us for
// luma and chroma T/Q and this; publishing every 1, 2, 4 MBs: 532, 524, 534)
constexpr int DB_ROWS = 8;              // MB rows (warps) per CTA
constexpr int DB_STRIP = 80;            // a finished MB's bottom rows: luma 3 x 16, chroma 2 x 2 x 8
constexpr int DB_PUBLISH = 2;           // MBs between releases of a CTA's last row
constexpr int DB_MAX_SMEM = 200 * 1024; // a CTA's strips; wider pictures take fewer rows per CTA
struct DbTiles {
    uint8_t lt[LT * LT];
    uint8_t ct[2][CR * CT];
};

// Tickets: row group g of frame f, the first groups of all frames first, so a
// group's predecessor was taken earlier.  rows: MB rows per CTA (its warps);
// strips: room for (rows - 1) * max mb_w strips; prog: one word per MB row of
// every frame (zeroed), the MBs of the row whose samples the row below may read.
__global__ void __launch_bounds__(32 * DB_ROWS) deblock_rows_kernel(const __grid_constant__ DbBatch batch, int rows, int max_w,
                                                                    int ntickets, const DbStrength* __restrict__ strength,
                                                                    int* __restrict__ counter, int* __restrict__ prog,
                                                                    int* __restrict__ status, int spin_limit) {
    extern __shared__ __align__(16) uint8_t db_strips[];
    __shared__ __align__(16) DbTiles tiles[DB_ROWS];
    __shared__ int done[DB_ROWS];
    __shared__ int ticket;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (;;) {
        if (threadIdx.x == 0) ticket = atomicAdd(counter, 1);
        if (lane == 0) *reinterpret_cast<volatile int*>(&done[w]) = 0;
        __syncthreads();
        const int t = ticket;
        if (t >= ntickets) return;
        // frames are sorted by rows, descending: group g exists for the first
        // seg frames with more than g * rows rows
        int g = 0, base = 0, f = 0;
        for (;; g++) {
            int nf = 0;
            while (nf < batch.n && batch.f[nf].mb_h > g * rows) nf++;
            if (t < base + nf) { f = t - base; break; }
            base += nf;
        }
        const DbFrameDesc& fd = batch.f[f];
        const int y = g * rows + w, W = fd.mb_w, H = fd.mb_h;
        if (w < rows && y < H) {
            const bool has_c = fd.uv[0] != nullptr, top = y > 0;
            const bool top_shared = top && w > 0;           // the row above is this CTA's previous warp
            const bool last = w == rows - 1 || y == H - 1;  // the row below (if any) is another CTA's
            const bool hand = !last;                        // bottom rows go to the next warp
            const int cw = fd.cw, ccw = cw >> 1;
            uint8_t* const Y = fd.y + (long long)y * 16 * cw;
            uint8_t* const C0 = has_c ? fd.uv[0] + (long long)y * 8 * ccw : nullptr;
            uint8_t* const C1 = has_c ? fd.uv[1] + (long long)y * 8 * ccw : nullptr;
            int* const gprog = prog + fd.row_base + y;
            const DbStrength* const st = strength + fd.flag_base + (long long)y * W;
            DbTiles& tl = tiles[w];
            uint32_t* const lt32 = reinterpret_cast<uint32_t*>(tl.lt);
            // the lane's line: luma row / column lane, or chroma line li of plane pl
            const bool luma = lane < 16;
            const int pl = (lane >> 3) & 1, li = lane & 7;
            uint8_t* const ct = tl.ct[pl];
            uint32_t* const ct32 = reinterpret_cast<uint32_t*>(ct);
            uint8_t* const cplane = pl ? C1 : C0;
            const DbLine dl{luma ? fd.th.alpha_y : fd.th.alpha_c, luma ? fd.th.beta_y : fd.th.beta_c, luma ? fd.th.tc_y[0] : fd.th.tc_c[0],
                            luma ? fd.th.tc_y[1] : fd.th.tc_c[1], luma};
            const int sg = luma ? lane >> 2 : li >> 1;
            auto edge_bits = [&](const DbStrength& s, int dir) {
                unsigned bits = 0;
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int ee = luma ? e : 2 * e;  // chroma: luma edges 0 and 2
                    const int i = 16 * dir + 4 * (ee & 3) + sg;
                    const unsigned b = ((s.m1 >> i) & 1u) | (((s.m2 >> i) & 1u) << 1);
                    if (luma || (e < 2 && has_c)) bits |= b << (2 * e);
                }
                return bits;
            };
            // own samples of MB x: luma words lane and lane + 32 (row i / 4,
            // word i % 4), chroma word (plane lane / 16, row (lane / 2) % 8)
            const int r0 = lane >> 2, r1 = 8 + (lane >> 2), wc = lane & 3;
            const int cpl = lane >> 4, cr = (lane >> 1) & 7, cwd = lane & 1;
            uint8_t* const cown = cpl ? C1 : C0;
            auto ldw32 = [](const uint8_t* p) { return __ldcg(reinterpret_cast<const unsigned int*>(p)); };
            auto stw32 = [](uint8_t* p, uint32_t v) { __stcg(reinterpret_cast<unsigned int*>(p), v); };
            uint32_t n0 = ldw32(Y + (long long)r0 * cw + 4 * wc), n1 = ldw32(Y + (long long)r1 * cw + 4 * wc), nc = 0;
            if (has_c) nc = ldw32(cown + (long long)cr * ccw + 4 * cwd);
            DbStrength ns = st[0];
            int avail = 0;  // MBs of the row above seen ready
            const unsigned poll_ns = top_shared ? 20 : 100;
            const int polls = poll_limit(spin_limit, poll_ns);
            // a row whose upper neighbour is another CTA's: the lane's word of
            // the next MB's top strip, fetched a step ahead when it is ready
            uint32_t tw = 0;
            bool tw_ok = false;
            auto top_word = [&](int mb) -> uint32_t {
                if (lane < 12) return ldw32(Y + (long long)((lane >> 2) - 3) * cw + 16 * mb + 4 * (lane & 3));
                if (lane < 20 && has_c) {
                    const int i = lane - 12;
                    return ldw32(((i >> 2) ? C1 : C0) + (long long)(((i >> 1) & 1) - 2) * ccw + 8 * mb + 4 * (i & 1));
                }
                return 0u;
            };
            for (int x = 0; x < W; x++) {
                const DbStrength s = ns;
                lt32[(4 + r0) * (LT / 4) + 1 + wc] = n0;
                lt32[(4 + r1) * (LT / 4) + 1 + wc] = n1;
                if (has_c) *reinterpret_cast<uint32_t*>(&tl.ct[cpl][(2 + cr) * CT + 4 + 4 * cwd]) = nc;
                if (x + 1 < W) {  // the next MB's, under this one's filtering
                    n0 = ldw32(Y + (long long)r0 * cw + 16 * (x + 1) + 4 * wc);
                    n1 = ldw32(Y + (long long)r1 * cw + 16 * (x + 1) + 4 * wc);
                    if (has_c) nc = ldw32(cown + (long long)cr * ccw + 8 * (x + 1) + 4 * cwd);
                    ns = st[x + 1];
                }
                __syncwarp();
                // ---- vertical edges ----
                int px[20];
                {
                    const uint32_t* const row = luma ? lt32 + (4 + lane) * (LT / 4) : ct32 + (2 + li) * (CT / 4);
#pragma unroll
                    for (int i = 0; i < 5; i++) {
                        const uint32_t v = i < 3 || luma ? row[i] : 0u;
#pragma unroll
                        for (int k = 0; k < 4; k++) px[4 * i + k] = byte_of(v, k);
                    }
                    db_line(dl, edge_bits(s, 0), px);
                    uint32_t* const rw = const_cast<uint32_t*>(row);
#pragma unroll
                    for (int i = 0; i < 5; i++) {
                        const uint32_t v = uint32_t(px[4 * i]) | uint32_t(px[4 * i + 1]) << 8 | uint32_t(px[4 * i + 2]) << 16 |
                                           uint32_t(px[4 * i + 3]) << 24;
                        if (i < 3 || luma) rw[i] = v;
                    }
                }
                __syncwarp();
                // the left MB is final: its last word column goes out (rows the
                // row below finishes are its), its bottom rows to the row below
                if (x > 0) {
                    if (luma) {
                        if (!hand || lane < 13) stw32(Y + (long long)lane * cw + 16 * x - 4, lt32[(4 + lane) * (LT / 4)]);
                    } else if (has_c) {
                        if (!hand || li < 6) stw32(cplane + (long long)li * ccw + 8 * x - 4, ct32[(2 + li) * (CT / 4)]);
                    }
                    if (hand) {
                        uint32_t* const sp = reinterpret_cast<uint32_t*>(db_strips + ((long long)w * max_w + x - 1) * DB_STRIP);
                        if (lane < 3) sp[4 * lane + 3] = lt32[(4 + 13 + lane) * (LT / 4)];
                        else if (lane >= 4 && lane < 8) sp[12 + 2 * (lane - 4) + 1] = *reinterpret_cast<uint32_t*>(&tl.ct[(lane - 4) >> 1][(2 + 6 + (lane & 1)) * CT]);
                        __syncwarp();
                        if (lane == 0) {
                            __threadfence_block();
                            *reinterpret_cast<volatile int*>(&done[w]) = x;
                        }
                    } else if (y < H - 1 && x % DB_PUBLISH == 0) {
                        __syncwarp();
                        if (lane == 0) st_release(gprog, x);
                    }
                }
                // ---- the row above's bottom rows of this MB ----
                if (top) {
                    if (avail < x + 1) {
                        if (lane == 0) {
                            int it = 0;
                            for (;; it++) {
                                avail = top_shared ? *reinterpret_cast<volatile int*>(&done[w - 1]) : ld_acquire(gprog - 1);
                                if (avail >= x + 1) break;
                                if (it >= polls || ((it & 255) == 255 && *reinterpret_cast<volatile int*>(status) != 0)) {
                                    atomicCAS(status, 0, 1);
                                    avail = W;
                                    break;
                                }
                                __nanosleep(poll_ns);
                            }
                            if (top_shared) __threadfence_block();
                        }
                        __syncwarp();  // what lane 0 has seen is every lane's to read
                        avail = __shfl_sync(0xffffffffu, avail, 0);
                    }
                    // luma rows -3..-1: lanes 0..11; chroma rows -2, -1: lanes 12..19
                    if (top_shared) {
                        if (lane < 20) tw = reinterpret_cast<const uint32_t*>(db_strips + ((long long)(w - 1) * max_w + x) * DB_STRIP)[lane];
                    } else if (!tw_ok) {
                        tw = top_word(x);
                    }
                    if (lane < 12) lt32[(1 + (lane >> 2)) * (LT / 4) + 1 + (lane & 3)] = tw;
                    else if (lane < 20 && has_c)
                        *reinterpret_cast<uint32_t*>(&tl.ct[(lane - 12) >> 2][(((lane - 12) >> 1) & 1) * CT + 4 + 4 * (lane & 1)]) = tw;
                    tw_ok = !top_shared && avail >= x + 2;
                    if (tw_ok) tw = top_word(x + 1);
                    __syncwarp();
                }
                // ---- horizontal edges ----
                {
                    const unsigned bits = edge_bits(s, 1);
                    uint8_t* const colp = luma ? tl.lt + 4 + lane : ct + 4 + li;
                    const int stride = luma ? LT : CT, skip = luma ? 0 : 2;  // chroma tiles start at row -2
                    const int lo = top ? (luma ? 1 : 2) : 4;
#pragma unroll
                    for (int i = 1; i < 20; i++) px[i] = i >= lo && (i < 12 || luma) ? colp[(i - skip) * stride] : 0;
                    db_line(dl, bits, px);
#pragma unroll
                    for (int i = 2; i < 18; i++)
                        if (i >= lo && (i < 12 || luma)) colp[(i - skip) * stride] = uint8_t(px[i]);
                }
                __syncwarp();
                // ---- out: the row above's bottom rows, this MB but for its last
                // word column (the next MB's left edge) and the rows that the row
                // below finishes ----
                if (top) {
                    if (lane < 12) {
                        const int r = lane >> 2;
                        stw32(Y + (long long)(r - 3) * cw + 16 * x + 4 * (lane & 3), lt32[(1 + r) * (LT / 4) + 1 + (lane & 3)]);
                    } else if (lane < 20 && has_c) {
                        const int i = lane - 12, p = i >> 2, r = (i >> 1) & 1, k = i & 1;
                        stw32((p ? C1 : C0) + (long long)(r - 2) * ccw + 8 * x + 4 * k, *reinterpret_cast<const uint32_t*>(&tl.ct[p][r * CT + 4 + 4 * k]));
                    }
                }
                const bool end = x == W - 1;
                const int lrows = hand ? 13 : 16, crows = hand ? 6 : 8;
                if (wc < 3 || end) {
                    stw32(Y + (long long)r0 * cw + 16 * x + 4 * wc, lt32[(4 + r0) * (LT / 4) + 1 + wc]);
                    if (r1 < lrows) stw32(Y + (long long)r1 * cw + 16 * x + 4 * wc, lt32[(4 + r1) * (LT / 4) + 1 + wc]);
                }
                if (has_c && (cwd == 0 || end) && cr < crows)
                    stw32(cown + (long long)cr * ccw + 8 * x + 4 * cwd, *reinterpret_cast<const uint32_t*>(&tl.ct[cpl][(2 + cr) * CT + 4 + 4 * cwd]));
                if (hand) {
                    uint32_t* const sp = reinterpret_cast<uint32_t*>(db_strips + ((long long)w * max_w + x) * DB_STRIP);
                    if (lane < 12 && ((lane & 3) < 3 || end)) sp[lane] = lt32[(4 + 13 + (lane >> 2)) * (LT / 4) + 1 + (lane & 3)];
                    else if (lane >= 12 && lane < 20 && ((lane & 1) == 0 || end)) {
                        const int i = lane - 12;
                        sp[12 + i] = *reinterpret_cast<const uint32_t*>(&tl.ct[i >> 2][(2 + 6 + ((i >> 1) & 1)) * CT + 4 + 4 * (i & 1)]);
                    }
                }
                if (end) {
                    __syncwarp();
                    if (lane == 0) {
                        if (hand) {
                            __threadfence_block();
                            *reinterpret_cast<volatile int*>(&done[w]) = W;
                        } else if (y < H - 1) {
                            st_release(gprog, W);
                        }
                    }
                } else {
                    // the last word column is the next MB's left strip
                    uint32_t v = 0;
                    if (luma) v = lt32[(4 + lane) * (LT / 4) + 4];
                    else v = ct32[(2 + li) * (CT / 4) + 2];
                    __syncwarp();
                    if (luma) lt32[(4 + lane) * (LT / 4)] = v;
                    else ct32[(2 + li) * (CT / 4)] = v;
                }
            }
        }
        __syncthreads();  // the strips and progress words are free for the next ticket
    }
}

}  // namespace h264a

using namespace h264a;

extern "C" int h264a_deblock_frames(h264a_ctx* ctx, const h264a_deblock_frame* h_frames, int nframes, void* stream) {
    if (!ctx || !h_frames || nframes < 1) return fail(H264A_E_ARG, "deblock_frames: bad arguments");
    for (int i = 0; i < nframes; i++) {
        const h264a_deblock_frame& f = h_frames[i];
        if (!f.d_y || !f.d_picks || !f.d_coeffs) return fail(H264A_E_ARG, "deblock_frames: null frame pointer");
        if ((f.d_u == nullptr) != (f.d_v == nullptr))
            return fail(H264A_E_ARG, "deblock_frames: give both chroma planes or neither");
        if (f.cw < 16 || f.ch < 16 || f.cw % 16 || f.ch % 16 || (long long)(f.cw / 16) * (f.ch / 16) > (1 << 24))
            return fail(H264A_E_ARG, "deblock_frames: frames must be MB-aligned");
        const uintptr_t a = reinterpret_cast<uintptr_t>(f.d_y) | reinterpret_cast<uintptr_t>(f.d_u) |
                            reinterpret_cast<uintptr_t>(f.d_v);
        if ((a & 3) != 0 || (reinterpret_cast<uintptr_t>(f.d_coeffs) & 15) != 0)
            return fail(H264A_E_ARG, "deblock_frames: planes must be 4-byte and coefficients 16-byte aligned");
        if (f.qp < 0 || f.qp > 51) return fail(H264A_E_ARG, "deblock_frames: qp out of 0..51");
    }
    cudaStream_t st = pick_stream(ctx, stream);
    std::vector<int> order(nframes);
    for (int i = 0; i < nframes; i++) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        return h_frames[a].ch > h_frames[b].ch;
    });
    for (int g0 = 0; g0 < nframes; g0 += DB_MAXF) {
        const int gn = nframes - g0 < DB_MAXF ? nframes - g0 : DB_MAXF;
        DbBatch b;
        memset(&b, 0, sizeof b);
        b.n = gn;
        long long total = 0;
        int nrows = 0, max_w = 0;
        for (int k = 0; k < gn; k++) {
            const h264a_deblock_frame& f = h_frames[order[g0 + k]];
            DbFrameDesc& d = b.f[k];
            d.y = f.d_y;
            d.uv[0] = f.d_u;
            d.uv[1] = f.d_v;
            d.picks = f.d_picks;
            d.coeffs = f.d_coeffs;
            d.cw = f.cw;
            d.ch = f.ch;
            d.mb_w = f.cw / 16;
            d.mb_h = f.ch / 16;
            d.flag_base = int(total);
            d.row_base = nrows;
            d.th = db_thresholds(f.qp, f.offset_a, f.offset_b, f.chroma_qp_offset);
            total += (long long)d.mb_w * d.mb_h;
            nrows += d.mb_h;
            max_w = std::max(max_w, d.mb_w);
        }
        if (total >= (1LL << 31)) return fail(H264A_E_ARG, "deblock_frames: too many macroblocks in one call");
        // the strengths, then the rows' progress words, in the queue's word space
        const size_t nwords = size_t(total) + size_t(nrows + 1) / 2;
        int rc = ensure_me_words(ctx, nwords, Q_MAIN);
        if (rc) return rc;
        WorkQueue& q = ctx->q[Q_MAIN];
        DbStrength* strength = reinterpret_cast<DbStrength*>(q.d_words);
        int* prog = reinterpret_cast<int*>(q.d_words + total);
        H264A_CUDA(cudaMemsetAsync(q.d_counter, 0, sizeof(int32_t), st));
        H264A_CUDA(cudaMemsetAsync(prog, 0, sizeof(int) * size_t(nrows), st));
        deblock_bs_kernel<<<unsigned((total + DB_BS_WARPS - 1) / DB_BS_WARPS), 32 * DB_BS_WARPS, 0, st>>>(b, total, strength);
        rc = check_launch("deblock_bs_kernel");
        if (rc) return rc;
        // rows per CTA: as many as the strips' shared memory allows, at most
        // DB_ROWS (1 for a picture too wide: every row through global memory)
        int rows = DB_ROWS;
        while (rows > 1 && (long long)(rows - 1) * max_w * DB_STRIP > DB_MAX_SMEM) rows--;
        const int smem = (rows - 1) * max_w * DB_STRIP;
        H264A_CUDA(cudaFuncSetAttribute(deblock_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DB_MAX_SMEM));
        int ntickets = 0;
        for (int k = 0; k < gn; k++) ntickets += (b.f[k].mb_h + rows - 1) / rows;
        int per_sm = 0;
        H264A_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, deblock_rows_kernel, 32 * DB_ROWS, smem));
        const int blocks = std::min(ntickets, ctx->num_sms * std::max(per_sm, 1));
        deblock_rows_kernel<<<unsigned(blocks), 32 * DB_ROWS, smem, st>>>(b, rows, max_w, ntickets, strength, q.d_counter, prog,
                                                                          ctx->d_status, SPIN_LIMIT);
        rc = check_launch("deblock_rows_kernel");
        if (rc) return rc;
    }
    return H264A_OK;
}

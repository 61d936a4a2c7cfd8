// me.cu -- a10/a11/a12: motion_search (crates/rusty_h264-encoder/src/mb16.rs:
// 2433-3302), best_part (:4921) and the plain-ME frame pass.
//
// One warp runs one search.  The frame kernels price an MB's 16x16 and its
// four partitions on the tensor cores (mb_search.cuh).  h264a_me_search's jobs
// (any shape and preset) run motion_search_warp below: each lane owns one 4x4
// sub-block of the partition, so a pass over 32 lanes prices 32/nb candidates
// at once (nb = sub-blocks per partition); a candidate's distortion is the sum
// of its lanes' blocks, added with shared-memory atomics.  Control flow
// replays the reference exactly:
//  * fixed-centre diamond passes and batched rings price their 4/8 candidates
//    together, then take the first strict-minimum like the reference's argmin;
//  * cascading rings (the centre moves mid-ring) are priced speculatively
//    against the current centre; the first improving point is taken and the
//    remaining points are re-priced around the new centre, which is exactly
//    the order in which the reference evaluates them.
// λ·rate is computed as an IEEE double product truncated toward zero, the
// same arithmetic as `(λ·rate as f64) as i64`.
#include <algorithm>
#include <climits>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "deblock_device.cuh"
#include "hpel_device.cuh"
#include "mb_search.cuh"
#include "tq_device.cuh"


namespace h264a {

// Warps per CTA of the frame kernels (one MB per warp).
constexpr int ME_WARPS = 4;

// Of h264a_me_search's jobs: metrics, search phases and what an evaluation
// round's results are for.
constexpr int MET_SATD = 0, MET_SAD = 1;
constexpr int PH_SEEDS = 0, PH_DIA = 1, PH_REPRICE = 2, PH_SUB = 3, PH_DONE = 4;
constexpr int EV_START = 0, EV_SEEDS = 1, EV_FIXED = 2, EV_RING = 3, EV_REPRICE = 4;

// Per-warp shared state of an h264a_me_search job: the round's candidates and
// distortions, and the search's cold parameters (read a few times per round,
// so they live here rather than in registers).
struct WarpScratch {
    int2 cand[32];
    int dist[32];
    const uint8_t* base;  // F|H|V|C planes
    int pw, ph, pad, cw, ch, rw, rh;
    int cx, cy;           // mvd centre, predictors[0]
    double lam_r;         // cost's λ (λ/4 for the table kinds)
    double lam_fp;        // cost_fp's λ (λ·RFF_ME_SADL under B2, else λ)
    double lam_me;        // λ itself (the batched sub-pel arms)
};

// Register-resident part of one search (every function below is inlined, so
// nothing of it is ever addressed in local memory); the rest is in the
// warp's WarpScratch.
struct SearchGeom {
    int lx, ly, lg_nb, lane, bxo, byo;
    uint32_t spa[4], spb[4];  // this lane's source 4x4 rows, split into column pairs
};

__device__ __forceinline__ void geom_init(SearchGeom& g, WarpScratch& ws, const h264a_picture& pc, int x, int y, int w,
                                          int h) {
    g.lx = x; g.ly = y;
    g.lane = threadIdx.x & 31;
    if (g.lane == 0) {
        ws.base = pc.d_planes;
        ws.pad = pc.pad;
        ws.pw = pc.cw + 2 * pc.pad;
        ws.ph = pc.ch + 2 * pc.pad;
        ws.cw = pc.cw;
        ws.ch = pc.ch;
        ws.rw = w;
        ws.rh = h;
    }
    g.lg_nb = (w == 16 ? 2 : (w == 8 ? 1 : 0)) + (h == 16 ? 2 : (h == 8 ? 1 : 0));
    const int nbx = w >> 2;
    const int blk = g.lane & ((1 << g.lg_nb) - 1);
    g.bxo = (blk % nbx) * 4;
    g.byo = (blk / nbx) * 4;
    uint32_t srow[4];
    // x + bxo is a multiple of 4 and the row lies inside the picture: aligned loads
#pragma unroll
    for (int r = 0; r < 4; r++)
        srow[r] = __ldg(reinterpret_cast<const uint32_t*>(pc.d_src + (long long)(y + g.byo + r) * pc.cw + x + g.bxo));
    split_pairs(srow, g.spa, g.spb);
    __syncwarp();
}

// Distortions of ws.cand[0..n) under `metric` added into ws.dist (zeroed by
// the caller) by shared-memory atomics of the lanes' 4x4 blocks.
__device__ __forceinline__ void eval_round(const SearchGeom& g, WarpScratch& ws, int n, int metric) {
    const int npass = ((n << g.lg_nb) + 31) >> 5;
    for (int k = 0; k < npass; k++) {
        const int c = (32 * k + g.lane) >> g.lg_nb;
        if (c >= n) continue;
        const int2 mv = ws.cand[c];
        Planes P;
        P.base = ws.base; P.pw = ws.pw; P.ph = ws.ph; P.pad = ws.pad; P.ps = (long long)ws.pw * ws.ph;
        uint32_t p4[4];
        pred_rows(P, g.lx + g.bxo + (mv.x >> 2), g.ly + g.byo + (mv.y >> 2), mv.x & 3, mv.y & 3, p4);
        int d;
        if (metric == MET_SAD) {
            uint32_t srow[4];
#pragma unroll
            for (int r = 0; r < 4; r++) srow[r] = g.spa[r] | (g.spb[r] << 8);
            d = sad4x4_rows(srow, p4);
        } else {
            d = satd4x4_packed(g.spa, g.spb, p4);
        }
        atomicAdd(&ws.dist[c], d);  // the candidate's blocks, summed in shared memory
    }
    __syncwarp();
}

// Rate of an MV against the search's mvd centre (mb16.rs:2454-2482).
__device__ __forceinline__ uint32_t rate_of(const MeParamsDev& pr, const WarpScratch& ws, int mvx, int mvy) {
    return mvbits(pr.kind, pr.tab, mvx - ws.cx) + mvbits(pr.kind, pr.tab, mvy - ws.cy);
}

// dist + (lam·rate) as i64 for candidate `lane` (< n), held in 32 bits: the
// distortions are below 2^21 and λ·rate below 2^28 for every λ the encoder
// forms (sqrt of 0.85·2^13 times a scale <= 4, rates < 2^17), so the sum
// never saturates and comparisons match the reference's i64.
__device__ __forceinline__ int lane_cost(const MeParamsDev& pr, const WarpScratch& ws, int lane, int n, double lam) {
    if (lane >= n) return INT_MAX;
    const int2 mv = ws.cand[lane];
    const long long c = (long long)ws.dist[lane] + lam_cost(lam, rate_of(pr, ws, mv.x, mv.y));
    return c > INT_MAX - 1 ? INT_MAX - 1 : int(c);
}

__device__ __forceinline__ bool in_plane_window(const SearchGeom& g, const WarpScratch& ws, int mvx, int mvy) {
    const int px = g.lx + (mvx >> 2) + ws.pad, py = g.ly + (mvy >> 2) + ws.pad;
    return px >= 0 && py >= 0 && px + ws.rw + 1 <= ws.pw && py + ws.rh + 1 <= ws.ph;
}

// dist + λ·rate of candidate i as the reference's i64 (every lane the same value).
__device__ __forceinline__ long long cand_cost64(const MeParamsDev& pr, const WarpScratch& ws, int i, double lam) {
    const int2 mv = ws.cand[i];
    return (long long)ws.dist[i] + lam_cost(lam, rate_of(pr, ws, mv.x, mv.y));
}

// Points of a cascading ring priced per round: the first round prices
// RING_FIRST of them, later rounds (after the centre moved, or none improved)
// up to RING_REST.  A ring of eight sub-pel points usually improves once or
// twice, mostly early, so pricing a few points at a time wastes fewer
// evaluations on points the walk reaches from a different centre; the order
// of the walk and its result do not depend on these sizes.
#ifndef RING_FIRST
#define RING_FIRST 2
#endif
#ifndef RING_REST
#define RING_REST 4
#endif

// motion_search (mb16.rs:2433-3302) of the partition in `g` (warp-cooperative,
// uniform control flow).  preds: npred (x,y) pairs, preds[0] the mvd centre;
// start: refine-only start MV or nullptr.  Returns the reference's evaluation
// count in `evals`.
//
// The search is written as one loop around a single evaluation round, so the
// round's code exists once per kernel: each iteration plans the next batch of
// candidates from the phase state (seeds together with the snaps of sub-pel
// predictors, diamond ladder, B2 reprice, sub-pel rings), prices it, and folds
// the result back into the state.
//  * fixed-centre batches (the FC diamond, sp_fc rings) price all points and
//    take the first strict minimum, like the reference's argmin loops;
//  * cascading rings (the centre moves mid-ring) price the remaining points
//    against the current centre; at the first improvement the centre moves and
//    the points after it are priced again around the new centre, which is the
//    order in which the reference evaluates them.
__device__ __forceinline__ void motion_search_warp(const SearchGeom& g, const MeParamsDev& pr, WarpScratch& ws,
                                                   const int* preds, int npred, const int* start, double lambda_me,
                                                   int& out_x, int& out_y, long long& out_c, int& evals) {
    const bool refine_only = start != nullptr;
    const bool sadfp = !pr.fast && !refine_only && pr.sadfp;
    const int m_main = pr.use_sad ? MET_SAD : MET_SATD;
    if (g.lane == 0) {
        ws.cx = preds[0];
        ws.cy = preds[1];
        ws.lam_me = lambda_me;
        ws.lam_r = pr.kind != 0 ? lambda_me * 0.25 : lambda_me;
        ws.lam_fp = lambda_me * (sadfp ? pr.sadfp_lambda : 1.0);
    }
    // Seeds in ws.cand[0..npred]; with the integer snap on, the snapped
    // position of every sub-pel predictor follows them, so the snap
    // (mb16.rs:2597-2607) is priced in the seed round: slot npred+1+k holds the
    // snap of the k-th sub-pel predictor (bit i of `snaps` set for predictor i).
    unsigned snaps = 0u;
    if (!refine_only) {
        int qx = 0, qy = 0;
        const bool mine = g.lane >= 1 && g.lane <= npred;
        if (mine) {
            qx = preds[2 * (g.lane - 1)];
            qy = preds[2 * (g.lane - 1) + 1];
            ws.cand[g.lane] = make_int2(qx, qy);
        }
        snaps = __ballot_sync(0xffffffffu, pr.me_snap && mine && ((qx & 3) != 0 || (qy & 3) != 0));
        if ((snaps >> g.lane) & 1u)
            ws.cand[npred + 1 + __popc(snaps & ((1u << g.lane) - 1u))] = make_int2(((qx + 2) >> 2) * 4, ((qy + 2) >> 2) * 4);
    }
    __syncwarp();
    const int m_fp = sadfp ? MET_SAD : m_main;
    const double l_fp = sadfp ? ws.lam_fp : ws.lam_r;  // cost_fp's λ (cost's λ when B2 is off)
    const int rw = ws.rw, rh = ws.rh;
    const bool x4shape = (rw == 16 || rw == 8) && (rh == 16 || rh == 8);
    const bool fc = !pr.fast && pr.fc && x4shape;
    const uint32_t dmask = pr.fast ? 0u : ((rw < 8 || rh < 8) ? pr.dia_sub_mask : pr.dia_mask);
    const int spat = pr.subpel_pat >= 0 ? pr.subpel_pat : ((rw < 8 || rh < 8) ? pr.sub_pat : (pr.sp_single_pass ? 2 : 0));
    const bool sp_fc = pr.sp_fc && !pr.fast && x4shape;
    const int sp_nring = (spat & 1) ? 4 : 8;

    evals = 0;
    int bx = 0, by = 0, seed_x = 0, seed_y = 0;
    long long best_c = 0, seed_c = 0;
    int phase = PH_SEEDS;
    int si = -1;        // diamond rung, -1 before the first
    int sk = -1;        // sub-pel step index (0: step 2, 1: step 1), -1 before the first
    int loops = 0;      // iterations of the current rung / sub-pel step
    int iter = 0;       // sub-pel iterations of the current step
    int step = 0;
    bool ring_open = false, ring_improved = false;  // a cascading ring in progress
    int ring_i = 0, ring_n = 0;
    for (;;) {
        // ---------- plan the next round ----------
        int kind = -1, n = 0, metric = m_main;
        double lam = ws.lam_r;
        while (kind < 0 && phase != PH_DONE) {
            if (phase == PH_SEEDS) {
                // seeds (mb16.rs:2580-2596): the start MV, or (0,0) then the predictors
                if (refine_only) {
                    bx = start[0]; by = start[1];
                    if (g.lane == 0) ws.cand[0] = make_int2(bx, by);
                    kind = EV_START; n = 1; metric = m_main; lam = ws.lam_r;
                } else {
                    if (g.lane == 0) ws.cand[0] = make_int2(0, 0);
                    kind = EV_SEEDS; n = npred + 1 + __popc(snaps); metric = m_fp; lam = l_fp;
                }
            } else if (phase == PH_DIA) {
                // diamond ladder (mb16.rs:2616-2727)
                if (ring_open) {
                    kind = EV_RING; n = min(ring_n - ring_i, RING_REST); metric = m_fp; lam = l_fp;
                    if (g.lane < n)
                        ws.cand[g.lane] = make_int2(bx + ring_dx(ring_i + g.lane) * step, by + ring_dy(ring_i + g.lane) * step);
                    break;
                }
                if (si < 0 || loops >= LOOP_GUARD) {
                    // next enabled rung
                    int nsi = si + 1;
                    if (pr.fast) nsi = nsi >= 2 ? 5 : nsi;
                    else
                        while (nsi < 5 && !(dmask & (1u << nsi))) nsi++;
                    if (nsi >= 5) {
                        phase = PH_REPRICE;
                        continue;
                    }
                    si = nsi;
                    step = pr.fast ? (si == 0 ? 16 : 4) : (64 >> si);  // rungs [64,32,16,8,4] quarter-pel
                    loops = 0;
                }
                loops++;
                bool fixed = false;
                if (fc && (bx & 3) == 0 && (by & 3) == 0) {
                    const int st = step >> 2;
                    const int px = g.lx + (bx >> 2), py = g.ly + (by >> 2);
                    fixed = px - st >= 0 && py - st >= 0 && px + st + rw <= ws.cw && py + st + rh <= ws.ch;
                }
                if (g.lane < 4) ws.cand[g.lane] = make_int2(bx + ring_dx(g.lane) * step, by + ring_dy(g.lane) * step);
                if (fixed) {
                    // 16-wide: sad_x4 / satd_x4 batch priced with lam_fp (mb16.rs:2676-2690);
                    // 8-wide shapes price each point with cost_fp (mb16.rs:2691)
                    kind = EV_FIXED; n = 4;
                    metric = rw == 16 ? (sadfp ? MET_SAD : MET_SATD) : m_fp;
                    lam = rw == 16 ? ws.lam_fp : l_fp;
                } else {
                    ring_open = true; ring_improved = false; ring_i = 0; ring_n = 4;
                    kind = EV_RING; n = 4; metric = m_fp; lam = l_fp;
                }
            } else if (phase == PH_REPRICE) {
                // B2 reprice into the SATD domain (mb16.rs:2744-2747)
                if (sadfp) {
                    if (g.lane == 0) {
                        ws.cand[0] = make_int2(bx, by);
                        ws.cand[1] = make_int2(seed_x, seed_y);
                    }
                    kind = EV_REPRICE; n = 2; metric = m_main; lam = ws.lam_r;
                } else {
                    phase = PH_SUB;
                }
            } else {  // PH_SUB: sub-pel rings (mb16.rs:2956-3283)
                if (ring_open) {
                    kind = EV_RING; n = min(ring_n - ring_i, RING_REST); metric = m_main; lam = ws.lam_r;
                    if (g.lane < n)
                        ws.cand[g.lane] = make_int2(bx + ring_dx(ring_i + g.lane) * step, by + ring_dy(ring_i + g.lane) * step);
                    break;
                }
                if (!pr.subpel) {
                    phase = PH_DONE;
                    continue;
                }
                if (sk < 0 || loops >= LOOP_GUARD) {
                    if (++sk >= 2) {
                        phase = PH_DONE;
                        continue;
                    }
                    step = sk == 0 ? 2 : 1;
                    loops = 0;
                    iter = 0;
                }
                loops++;
                if (sp_fc && (spat & 1) == 0 && (step == 1 || ((bx & 3) == 0 && (by & 3) == 0))) {
                    // hpel_qpel_refs / hpel_ref resolve every ring point (inter.rs:1015, 1060):
                    // inside the +1-slack window, and at step 1 a quarter phase
                    bool all = true;
                    for (int i = 0; i < 8; i++) {
                        const int qx = bx + ring_dx(i) * step, qy = by + ring_dy(i) * step;
                        all = all && in_plane_window(g, ws, qx, qy) && (step == 2 || ((qx | qy) & 1));
                    }
                    if (all) {
                        iter++;
                        if (g.lane < 8)
                            ws.cand[g.lane] = make_int2(bx + ring_dx(g.lane) * step, by + ring_dy(g.lane) * step);
                        // 16-wide: satd_avg_x4 / satd_x4p priced with lambda_me; 8-wide: cost()
                        kind = EV_FIXED; n = 8;
                        metric = rw == 16 ? MET_SATD : m_main;
                        lam = rw == 16 ? ws.lam_me : ws.lam_r;
                        break;
                    }
                }
                iter++;
                n = min(sp_nring, RING_FIRST);
                if (g.lane < n)
                    ws.cand[g.lane] = make_int2(bx + ring_dx(g.lane) * step, by + ring_dy(g.lane) * step);
                ring_open = true; ring_improved = false; ring_i = 0; ring_n = sp_nring;
                kind = EV_RING; metric = m_main; lam = ws.lam_r;
            }
        }
        if (kind < 0) break;
        if (g.lane < n) ws.dist[g.lane] = 0;  // eval_round adds each lane's block into its candidate's slot
        __syncwarp();

        // ---------- price the round ----------
        eval_round(g, ws, n, metric);
        const int cc = lane_cost(pr, ws, g.lane, n, lam);

        // ---------- fold the result into the state ----------
        if (kind == EV_START) {
            best_c = cand_cost64(pr, ws, 0, lam);
            evals += 1;
            seed_x = bx; seed_y = by; seed_c = best_c;
            phase = PH_REPRICE;  // refine-only: no snap, no ladder, no B2 reprice; on to the sub-pel rings
        } else if (kind == EV_SEEDS) {
            // sequential strict-< scan: (0,0) first, then the predictors in order
            best_c = __shfl_sync(0xffffffffu, cc, 0);
            bx = 0; by = 0;
            int wi = 0;
            for (int i = 1; i <= npred; i++) {
                const long long ci = __shfl_sync(0xffffffffu, cc, i);
                if (ci < best_c) {
                    best_c = ci;
                    bx = ws.cand[i].x;
                    by = ws.cand[i].y;
                    wi = i;
                }
            }
            evals += npred + 1;
            seed_x = bx; seed_y = by; seed_c = best_c;
            if ((snaps >> wi) & 1u) {
                // the winner is a sub-pel predictor: take its snap, priced in this round
                const int si_ = npred + 1 + __popc(snaps & ((1u << wi) - 1u));
                bx = ws.cand[si_].x; by = ws.cand[si_].y;
                best_c = cand_cost64(pr, ws, si_, lam);
                evals += 1;
            }
            phase = PH_DIA;
        } else if (kind == EV_REPRICE) {
            best_c = cand_cost64(pr, ws, 0, lam);
            seed_c = cand_cost64(pr, ws, 1, lam);
            evals += 2;
            phase = PH_SUB;
        } else if (kind == EV_FIXED) {
            const int m = __reduce_min_sync(0xffffffffu, cc);
            const unsigned at = __ballot_sync(0xffffffffu, cc == m);
            evals += n;
            const int bi = (long long)m < best_c ? __ffs(at) - 1 : -1;
            if (bi >= 0) {
                best_c = m;
                bx += ring_dx(bi) * step;
                by += ring_dy(bi) * step;
            }
            if (phase == PH_DIA) {
                if (bi < 0) loops = LOOP_GUARD;  // rung done
            } else {
                const bool stop = bi < 0 || !pr.me_subpel_iter || (spat & 2) || (pr.sp_maxit != 0 && iter >= pr.sp_maxit);
                if (stop) loops = LOOP_GUARD;  // step done
            }
        } else {  // EV_RING
            const unsigned hit = __ballot_sync(0xffffffffu, g.lane < n && (long long)cc < best_c);
            if (hit == 0) {
                evals += n;
                ring_i += n;
                ring_open = ring_i < ring_n;  // the rest of the ring, around the same centre
            } else {
                const int j = __ffs(hit) - 1;
                best_c = __shfl_sync(0xffffffffu, cc, j);
                const int2 mv = ws.cand[j];
                evals += j + 1;
                bx = mv.x;
                by = mv.y;
                ring_improved = true;
                ring_i += j + 1;
                ring_open = ring_i < ring_n;
            }
            if (!ring_open) {
                if (phase == PH_DIA) {
                    if (!ring_improved) loops = LOOP_GUARD;  // rung done
                } else if (!ring_improved || !pr.me_subpel_iter || (spat & 2) ||
                           (pr.sp_maxit != 0 && iter >= pr.sp_maxit)) {
                    loops = LOOP_GUARD;  // step done
                }
            }
        }
        __syncwarp();
    }
    // ---- seed restore (mb16.rs:3297-3300) ----
    if (pr.me_snap && seed_c < best_c) {
        bx = seed_x; by = seed_y; best_c = seed_c;
    }
    out_x = bx; out_y = by; out_c = best_c;
}
__device__ __forceinline__ bool job_shape_ok(int w, int h) {
    return (w == 16 && (h == 16 || h == 8)) || (w == 8 && (h == 16 || h == 8 || h == 4)) ||
           (w == 4 && (h == 8 || h == 4));
}

// CTAs per SM that the frame kernels' registers allow: three with Balanced,
// whose searches need some 140 registers a thread; at the 128 of four CTAs their
// reloads cost more than the further warps give (1080p closed loop 25.4 and 24.1
// ms, one 720p frame with its reconstruction 1.88 and 1.78, 75 mixed frames
// 4.52 and 4.12).  Two with other presets, whose searches hold more: reloads at
// 128 and 168 registers cost a round 20% and 5%, also in calls of many frames
// (fifteen 720p frames walked to convergence: 4.24, 3.72 and 3.65 ms).
constexpr int ME_MIN_BLOCKS = 3, ME_ANY_BLOCKS = 2;

__global__ void __launch_bounds__(32 * ME_WARPS) me_search_kernel(const h264a_picture* __restrict__ pics, int npics,
                                                                 const __grid_constant__ MeParamsDev prm,
                                                                 const h264a_me_job* __restrict__ jobs, int n,
                                                                 h264a_me_result* __restrict__ out) {
    __shared__ WarpScratch scratch[ME_WARPS];
    const int w = threadIdx.x >> 5;
    const long long j = (long long)blockIdx.x * ME_WARPS + w;
    if (j >= n) return;
    const h264a_me_job job = jobs[j];
    h264a_me_result res{};
    const bool ok = job.pic >= 0 && job.pic < npics && job_shape_ok(job.w, job.h) && job.npred >= 1 && job.npred <= 4;
    h264a_picture pc{};
    bool inside = false;
    if (ok) {
        pc = pics[job.pic];
        inside = job.x >= 0 && job.y >= 0 && job.x + job.w <= pc.cw && job.y + job.h <= pc.ch;
    }
    if (!ok || !inside) {
        res.status = -1;
        if ((threadIdx.x & 31) == 0) out[j] = res;
        return;
    }
    SearchGeom g;
    geom_init(g, scratch[w], pc, job.x, job.y, job.w, job.h);
    int mx, my, evals;
    long long c;
    motion_search_warp(g, prm, scratch[w], job.preds, job.npred, job.has_start ? job.start : nullptr, job.lambda_me, mx,
                       my, c, evals);
    if ((threadIdx.x & 31) == 0) {
        res.mvx = mx; res.mvy = my; res.cost = c; res.evals = evals; res.status = 0;
        out[j] = res;
    }
}

// ---------------------------------------------------------------------------
// Plain-ME frames: persistent work-queue kernel
// ---------------------------------------------------------------------------

struct FrameDesc {
    // the reference picture's F|H|V|C planes as a 3D tensor (x, y, plane)
    // with an 80 x 42 x 4 box, the shape of an MB's window; tmap_ok 0 means
    // the window is staged row by row instead
    CUtensorMap tmap;
    h264a_picture pic;
    double lambda_me;
    long long split_gate;
    int32_t* picks;
    int64_t* costs;
    int flag_base;
    int mb_w, mb_h;
    // the fused MC + luma T/Q (h264a_me_tq_frames): coefficients out, or
    // nullptr for none, and the frame QP's quant row
    int16_t* coeffs;
    int16_t qff[8], qmf[8];
    // optional row completion (h264a_pixel_path_host): one counter per MB row
    // (zeroed), and a host-visible word per row set to row_token once every
    // MB of the row has its pick and coefficients stored
    int32_t* row_count;
    int32_t* row_done;
    int32_t row_token;
    int32_t tmap_ok;
    // the learned-proposal kernels (h264a_me_frames_learned): 16 i32 per MB
    // of proposals, the fallback threshold, and an optional fallback flag per MB
    const int32_t* props;
    int32_t* fallback;
    int32_t prop_t;
};

// One launch's frames, passed by value.  Frames are sorted by MB count
// (descending) and the work queue deals the k-th MB of every frame that has
// one before the (k+1)-th of any frame: segment j covers positions
// [nmb[j+1], nmb[j]) of frames 0..j, so its tickets are (nmb[j]-nmb[j+1])*(j+1),
// and segments are dealt from j = n-1 (every frame) down to j = 0 (the
// largest frame's tail).  Only the non-empty segments are stored (one per
// distinct frame size): seg_start[s] is the first ticket of segment seg_j[s],
// seg_start[nseg] the ticket count.
// Within a frame the k-th MB is taken in wavefront order (anti-diagonals
// t = x + 2y, then y): every MB's neighbours (left, top, top-left, top-right)
// lie on earlier diagonals, so a window of resident warps always holds MBs
// that are ready, and no MB ever waits on a ticket dealt after its own.
constexpr int ME_MAXF = 96;
// Launches of at most this many frames use the work queue of the closed loop
// (Q_WIDE), larger ones Q_MAIN.
constexpr int ME_FEW_FRAMES = 2;
// The pipelined closed loop: the width of a band's column segments in MBs, the
// number of warp pools (frames dealt round-robin to them) and the CTAs per SM,
// by the picture's size.  A narrower segment is final sooner, so the next frame
// follows closer; it also means more tickets and plane strips with idle lanes.
// So a 24th of the width: what the wavefront of a small picture waits for is
// the frame before, a large one's segments are too many (30 frames, segments
// of 1, 2, 3, 4, 7 MBs: 640x360 7.9, 8.4, 8.9, 9.3, 10.4 ms; 960x540 9.7, 8.1,
// 8.4, 8.8, 10.1; 1920x1080, 60 frames, -, 29.4, 28.4, 27.5, 27.7; 3840x2160,
// 16 frames, 4 and 7: 20.0, 18.8).  Pools: about the frames whose wavefronts
// fit one after another; more pools only hold warps that wait (learned 720p at
// 6, 8, 10, 13: 7.5, 6.8, 7.0, 8.0 ms; 1080p at 8, 10, 13: 28.4, 26.5, 27.1).
// CTAs: about a warp per MB of the pools' longest anti-diagonals: more hold MBs
// that wait, and slow the warps that run (60 1080p frames at 1 and 2 an SM: 24.1
// and 26.1 ms; 30 of 2560x1440 at 2 and 3: 19.4 and 20.9; 16 of 3840x2160: 18.3
// and 19.6).  (The segment and pool sweeps, and fewer CTAs than that -- 2560x1440
// at 1 and 2: 18.9 and 17.0, 3840x2160 27.0 and 20.0 -- on an earlier build at
// 128 registers a thread.)
constexpr int PIPE_SEGW = 7, PIPE_POOLS = 10;
static inline int wave_mbs(int mb_w, int mb_h) { return std::min((mb_w + 1) / 2, mb_h); }  // of the longest anti-diagonal
static inline int pipe_segw(int mb_w) { return std::min(std::max(mb_w / 24, 1), PIPE_SEGW); }
static inline int pipe_pools(int mb_w, int mb_h) {
    return std::min(std::max((mb_w + 2 * mb_h) / 16, 6), PIPE_POOLS);
}
static inline int pipe_ctas_per_sm(int mb_w, int mb_h, int pools, int num_sms, int most) {
    const int warps = ME_WARPS * num_sms;
    const int n = (pools * wave_mbs(mb_w, mb_h) + warps * 3 / 4 - 1) / warps;  // a quarter short is near enough
    return std::min(std::max(n, 1), most);
}
// Dynamic shared memory of such a launch: its windows, or as much as keeps one
// CTA more than its share off an SM.  Beside another kernel (the lookahead of
// the next frames on its own stream) the CTAs would otherwise crowd onto the
// SMs that are free first (60 1080p frames with their lookahead: 64.8 ms, the
// loop alone 41.7).  The price: launches of one CTA an SM from two contexts do
// not share SMs, although one of them keeps 5% of an SM's warps active.
constexpr int SM_SHARED = 228 * 1024, FRAME_SMEM_MAX = SM_SHARED / 2;
static inline size_t frame_smem(long long blocks, int num_sms) {
    const long long share = (blocks + num_sms - 1) / num_sms;
    return std::max<size_t>(ME_WARPS * WIN_BYTES, size_t(SM_SHARED / (share + 1)));
}
struct FrameBatch {
    FrameDesc f[ME_MAXF];
    long long seg_start[ME_MAXF + 1];
    int seg_j[ME_MAXF];
    int n, nseg;
};
// The frame table as the kernel body reads it: the launch's parameters
// (FrameBatch, up to ME_MAXF frames) or arrays in device memory (any count).
struct ParamTable {
    static constexpr bool kGlobal = false;  // tensor maps in the kernel's parameters
    const FrameBatch& b;
    __device__ __forceinline__ int n() const { return b.n; }
    __device__ __forceinline__ int nseg() const { return b.nseg; }
    __device__ __forceinline__ long long seg(int s) const { return b.seg_start[s]; }
    __device__ __forceinline__ int segj(int s) const { return b.seg_j[s]; }
    __device__ __forceinline__ const FrameDesc& fr(int i) const { return b.f[i]; }
};
struct DeviceTable {
    static constexpr bool kGlobal = true;  // tensor maps in device memory
    const FrameDesc* f;
    const long long* seg_start;
    const int* seg_j;
    int nf, ns;
    __device__ __forceinline__ int n() const { return nf; }
    __device__ __forceinline__ int nseg() const { return ns; }
    __device__ __forceinline__ long long seg(int s) const { return __ldg(seg_start + s); }
    __device__ __forceinline__ int segj(int s) const { return __ldg(seg_j + s); }
    __device__ __forceinline__ const FrameDesc& fr(int i) const { return f[i]; }
};
static_assert(sizeof(FrameBatch) + 512 <= 32764, "me_frames_kernel's parameters must fit the 32 KB parameter space");

// The MV of neighbour MB `m`'s 4x4 block at (bx4, by4) under its pick.
__device__ __forceinline__ int2 pick_mv_at(const int32_t* picks, int m, int bx4, int by4) {
    const int32_t* p = picks + 6 * m;
    const int shape = __ldcg(p);
    const int part = shape == 1 ? (by4 >= 2) : (shape == 2 ? (bx4 >= 2) : 0);
    return make_int2(__ldcg(p + 1 + 2 * part), __ldcg(p + 2 + 2 * part));
}

// predict_mv (inter.rs:36-69) with every available neighbour inter, ref 0.
__device__ __forceinline__ int2 predict_mv_ref0(bool aa, int2 a, bool ba, int2 b, bool ca, int2 c) {
    int2 mva = aa ? a : make_int2(0, 0);
    int2 mvb = ba ? b : make_int2(0, 0);
    int2 mvc = ca ? c : make_int2(0, 0);
    int ra = aa ? 0 : -1, rb = ba ? 0 : -1, rc = ca ? 0 : -1;
    if (!ba && !ca && aa) { mvb = mva; rb = ra; mvc = mva; rc = ra; }
    const int matches = (ra == 0) + (rb == 0) + (rc == 0);
    if (matches == 1) return ra == 0 ? mva : (rb == 0 ? mvb : mvc);
    auto med = [](int x, int y, int z) { return x + y + z - min(min(x, y), z) - max(max(x, y), z); };
    return make_int2(med(mva.x, mvb.x, mvc.x), med(mva.y, mvb.y, mvc.y));
}

// ---------------------------------------------------------------------------
// One MB of the frame kernels
// ---------------------------------------------------------------------------

// The closed loop's reconstruction of a frame, fused into the frame kernels:
// after an MB's pick is published, the same warp runs its luma and chroma MC +
// T/Q + reconstruction and then the in-loop deblocking of the MB in shared
// tiles, once the deblocking of its left and top-right neighbours is done
// (bounded waits on a second run of flags, the same wavefront order as the
// search).
struct RecDesc {
    const uint8_t* src_c[2];  // the frame's chroma source (U, V)
    const uint8_t* ref_c[2];  // the chroma reconstruction of the previous frame
    uint8_t* rec_y;           // the frame's reconstruction
    uint8_t* rec_c[2];
    int16_t* ccoeffs;         // chroma levels, 128 per MB
    int qp, qpc;              // luma and chroma QP
    int16_t cff[8], cmf[8];   // the chroma QP's quant row (inter dead-zone)
    int dflag_base, nz_base;  // the deblocking flags' and coefficient masks' offsets in the flag array
    DbThresh th;
};

// Where pictures allow it an MB's pick is published to the wavefront as three
// 64-bit words, each the launch's epoch (high half) and one MV (x, y as i16,
// low half): the MVs of its blocks (3,0), (0,3) and (3,3), which are what its
// right, lower (and lower-left) and lower-right neighbours' median predictors
// read (mv_neighbors_block, mb16.rs:1871).  A waiting MB polls the words it
// needs until their epoch is the launch's, so the flag and the data arrive in
// one load and no release fence orders anything else.  An MV that does not fit
// (a caller's proposal may lie anywhere, and a search walks on from it) is the
// word MV_FAR: the pick is in memory before it, for the reader to take from
// there.  Pictures more than 8191 samples wide or high, whose MVs seldom fit,
// and launches whose scratch holds one flag per MB (h264a_me_frames_noalloc),
// publish a flag after the pick instead.
constexpr int EW_PER_MB = 3;
// Nanoseconds between polls of a warp diagonals ahead of the wavefront, and of
// one waiting for its left or top-right neighbour.
constexpr unsigned POLL_FAR_NS = 1000, POLL_NEAR_NS = 40;
constexpr int EW_MAX_SIDE = 8191;
constexpr int MV_FAR = -32768;  // both components of the word of an MV beyond +-32767
__device__ __forceinline__ bool mv_far(int v) { return v < -32767 || v > 32767; }
__device__ __forceinline__ unsigned long long mv_word(int epoch, int x, int y) {
    return ((unsigned long long)(unsigned)epoch << 32) | (uint32_t(uint16_t(x)) | (uint32_t(uint16_t(y)) << 16));
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// Waits (bounded; status 1 on timeout) for the word to carry `epoch`, polling
// every `ns` nanoseconds; returns its MV.
__device__ __forceinline__ int2 wait_mv_word(const unsigned long long* p, int epoch, int* status, int limit, unsigned ns) {
    unsigned long long v = 0;
    const int polls = poll_limit(limit, ns);
    for (int it = 0;; it++) {
        asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
        if (int(v >> 32) == epoch) break;
        if (it >= polls || ((it & 255) == 255 && *reinterpret_cast<volatile int*>(status) != 0)) {
            atomicCAS(status, 0, 1);
            break;
        }
        __nanosleep(ns);
    }
    return make_int2(int(int16_t(v & 0xffffu)), int(int16_t((v >> 16) & 0xffffu)));
}

// The launch's synchronisation as one MB sees it: the frame's MV words (or
// null: its flags), its deblocking flags and coefficient masks, the reference's segment readiness
// (pipelined closed loop, or null) and the bounded waits' parameters.
struct MbSync {
    unsigned long long* ew;
    int* flags;
    int* dfl;
    int* nz;  // REC: each MB's mask of luma blocks with coefficients (raster order), stored before its deblocking flag
    const BandWait* bw;
    int epoch;
    int* status;
    int limit;
};

// The reconstruction tiles of an MB (deblock_device.cuh's layout) and its
// edges' bS.  They live in the MB's window buffer once its motion compensation
// has read the window.
struct RecTiles {
    uint8_t lt[LT * LT];
    uint8_t ct[2][CR * CT];
    int bs[32];
};
static_assert(sizeof(RecTiles) <= WIN_BYTES && alignof(RecTiles) <= 16, "the tiles fit the window buffer");

// Stages the reference window around MV `mv` of the MB at (lx, ly): WIN_R rows
// and columns up-left of the position, the x origin on a 16-byte boundary
// (bulk-copy alignment); one TMA tensor copy, or a bulk copy per plane row
// when the planes have no tensor map.  Returns whether a window is on its way
// (wait_window on `bar`).  The warp is converged; its earlier accesses to the
// buffer are ordered before the copy.
__device__ __forceinline__ bool stage_window(MbScratch& ws, const CUtensorMap* tmap, bool tmap_ok, bool tmap_global,
                                             int lx, int ly, int2 mv, uint32_t win, uint32_t bar) {
    const int lane = threadIdx.x & 31;
    const bool ok = ((reinterpret_cast<uintptr_t>(ws.base) | uintptr_t(ws.pw)) & 15) == 0 && ws.pw >= WIN_W && ws.ph >= WIN_H;
    if (!ok) return false;
    const int wx0 = min(max((lx + ws.pad + (mv.x >> 2) - WIN_R) & ~15, 0), ws.pw - WIN_W);
    const int wy0 = min(max(ly + ws.pad + (mv.y >> 2) - WIN_R, 0), ws.ph - WIN_H);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) {
        ws.wx0 = wx0;
        ws.wy0 = wy0;
        // the window's reference rows are built (pipelined loop), and the
        // generic-proxy writes of them are visible to the copy
        band_wait_px(ws.bw, &ws.bready, wy0 - ws.pad + WIN_H - 1, wx0 - ws.pad + WIN_W - 1);
        if (ws.bw != nullptr) asm volatile("fence.proxy.async.global;" ::: "memory");
        if (tmap_ok) {
            mbar_expect_tx(bar, uint32_t(WIN_BYTES));
            // a tensor map written to device memory by the host since an
            // earlier launch read that address: acquire it for the copy
            if (tmap_global) asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(tmap) : "memory");
            tma_load_3d(win, tmap, wx0, wy0, 0, bar);
        } else {
            mbar_expect_tx(bar, uint32_t(4 * WIN_H * WIN_W));
        }
    }
    __syncwarp();
    if (!tmap_ok) {
        const long long ps = (long long)ws.pw * ws.ph;
        for (int i = lane; i < 4 * WIN_H; i += 32) {
            const int pl = i / WIN_H, r = i - pl * WIN_H;
            bulk_g2s(win + uint32_t(pl * WIN_PLANE + r * WIN_STRIDE),
                     ws.base + ps * pl + (long long)(wy0 + r) * ws.pw + wx0, WIN_W, bar);
        }
    }
    return true;
}

// A warp's window buffer (dynamic shared memory), its mbarrier and the CTA's
// operand table (shared address).
struct WarpWindow {
    uint8_t* p;
    uint32_t win, bar, lut;
};
__device__ __forceinline__ WarpWindow warp_window(uint8_t* dyn, unsigned long long* bars, PhaseTab& pt, SearchScratch* bs) {
    const int w = threadIdx.x >> 5;
    WarpWindow o;
    o.p = dyn + w * WIN_BYTES;
    o.win = uint32_t(__cvta_generic_to_shared(o.p));
    o.bar = uint32_t(__cvta_generic_to_shared(bars + w));
    o.lut = uint32_t(__cvta_generic_to_shared(&pt));
    phase_tab_init(pt, int(threadIdx.x));
    if ((threadIdx.x & 31) == 0) {
        bs[w].lam = __longlong_as_double(0x7ff8000000000000ll);  // NaN: no table yet
        mbar_init(o.bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    return o;
}

// One MB by one warp: the predictor from the neighbours' picks, the reference
// window, best_part for 16x16 and, when its J exceeds the gate, for the four
// partitions (mb16.rs:8869-8913), the pick published to the wavefront, then
// off its path the MB's MC + T/Q when the frame has coefficients, and with
// REC its reconstruction and deblocking.
//
// The neighbours above were published a row earlier; only the left one is on
// the wavefront's path.  So the window's origin comes from the top MB's MV
// and its copy overlaps the wait for the left MB; any origin gives the same
// picks, as candidates the window misses read the planes.
template <bool BAL, bool LEARN, bool REC, bool PIPE>
__device__ __forceinline__ void frame_mb(const FrameDesc& fd, const RecDesc* rdp, int mbx, int mby,
                                         const MeParamsDev& prm, const MbSync& sy, MbScratch& ws, SearchScratch& bs,
                                         const WarpWindow& ww, uint32_t& parity, bool tmap_global) {
    const uint32_t win = ww.win, bar = ww.bar;
    uint8_t* const winp = ww.p;
    const int lane = threadIdx.x & 31;
    const int mb_w = fd.mb_w, m = mby * mb_w + mbx;
    const int lx = mbx * 16, ly = mby * 16;
    const h264a_picture pc = fd.pic;
    const int pw = pc.cw + 2 * pc.pad, ph = pc.ch + 2 * pc.pad;
    MbLane s;
    mb_load_src(s, pc.d_src, pc.cw, lx, ly);  // inputs: before any wait
    int2 prop = make_int2(0, 0), propc = prop;  // proposals lane % 8 and lane / 4
    if (LEARN) {
        prop = make_int2(__ldg(fd.props + 16LL * m + 2 * (lane & 7)), __ldg(fd.props + 16LL * m + 2 * (lane & 7) + 1));
        propc = make_int2(__ldg(fd.props + 16LL * m + 2 * (lane >> 2)), __ldg(fd.props + 16LL * m + 2 * (lane >> 2) + 1));
    }
    if (lane == 0) {
        ws.base = pc.d_planes;
        ws.src = pc.d_src;
        ws.bw = sy.bw;
        ws.pw = pw; ws.ph = ph; ws.pad = pc.pad; ws.cw = pc.cw; ws.ch = pc.ch;
        ws.bready = -1;
    }
    // the neighbours' MVs: lane 0 the left MB's block (3,0), lane 1 the top
    // MB's (0,3), lane 2 the top-right MB's (0,3), lane 3 the top-left MB's
    // (3,3) when there is no top-right (mv_neighbors_block, mb16.rs:1871)
    const bool aa = mbx > 0, ba = mby > 0, ca = mby > 0 && mbx < mb_w - 1, da = mbx > 0 && mby > 0;
    const bool need = lane < 4 && (lane == 0 ? aa : (lane == 1 ? ba : (lane == 2 ? ca : (!ca && da))));
    const int nb = m + (lane == 0 ? -1 : (lane == 1 ? -mb_w : (lane == 2 ? 1 - mb_w : -1 - mb_w)));
    auto fetch = [&](unsigned ns) {
        if (sy.ew != nullptr) {
            const int2 v = wait_mv_word(sy.ew + EW_PER_MB * (long long)nb + (lane == 0 ? 0 : (lane == 3 ? 2 : 1)), sy.epoch,
                                        sy.status, sy.limit, ns);
            if (v.x != MV_FAR) return v;
            __threadfence();  // the word first, then the pick
        } else {
            wait_flag(sy.flags + nb, sy.epoch, sy.status, 1, sy.limit);
        }
        return pick_mv_at(fd.picks, nb, lane == 0 || lane == 3 ? 3 : 0, lane == 0 ? 0 : 3);
    };
    // most resident warps hold MBs some diagonals ahead of the wavefront: they
    // wait for the top MB (two diagonals back) with long sleeps, so that their
    // polling does not slow the warps on the path
    int2 nv = make_int2(0, 0);
    if (need && (lane == 1 || !ba)) nv = fetch(ba ? POLL_FAR_NS : POLL_NEAR_NS);
    __syncwarp();
    const int2 top = make_int2(__shfl_sync(0xffffffffu, nv.x, 1), __shfl_sync(0xffffffffu, nv.y, 1));
    const int2 first = make_int2(__shfl_sync(0xffffffffu, nv.x, 0), __shfl_sync(0xffffffffu, nv.y, 0));
    const int2 guess = ba ? top : first;  // (the first row predicts from the left MB alone)
    const bool win_ok = stage_window(ws, &fd.tmap, fd.tmap_ok != 0, tmap_global, lx, ly, guess, win, bar);
    if (need && lane != 1 && ba) nv = fetch(POLL_NEAR_NS);
    __syncwarp();
    const int2 left = make_int2(__shfl_sync(0xffffffffu, nv.x, 0), __shfl_sync(0xffffffffu, nv.y, 0));
    const int2 corner = make_int2(__shfl_sync(0xffffffffu, nv.x, ca ? 2 : 3), __shfl_sync(0xffffffffu, nv.y, ca ? 2 : 3));
    const int2 pmv = predict_mv_ref0(aa, left, ba, top, ca || da, corner);
    mb_lane_16x16(s, lx, ly, win);
    mb_lane_window(s, ws, win_ok);
    if (win_ok) {
        wait_window(bar, parity, sy.status, 3, sy.limit);
        parity ^= 1u;
    }
    // best_part for 16x16, then, J above the gate, the four partitions seeded
    // [pmv, mv16] side by side
    int shape = 0, fell = 0;
    const SearchOut r16 =
        search16<BAL, LEARN, REF_WINDOW, PIPE>(s, prm, ws, bs, ww.lut, pmv, fd.lambda_me, LEARN, propc, prop, fd.prop_t, &fell);
    int evals = r16.evals << 4;  // 4x4-block evaluations
    const int c16 = r16.cost;
    long long best = c16;
    int mv0x = r16.x, mv0y = r16.y, mv1x = r16.x, mv1y = r16.y;
    if (fd.split_gate >= 0 && c16 > fd.split_gate) {
        mb_lane_parts(s);
        // the learned search's partitions, when its 16x16 search took a
        // proposal: refine-only from the 16x16 MV
        const int2 mv16 = make_int2(mv0x, mv0y);
        const SearchOut r =
            search_parts<BAL, LEARN, REF_WINDOW, PIPE>(s, prm, ws, bs, ww.lut, pmv, mv16, fd.lambda_me, LEARN && !fell, mv16);
        int px[4], py[4];
        long long pcost[4];
#pragma unroll
        for (int gi = 0; gi < 4; gi++) {
            px[gi] = __shfl_sync(0xffffffffu, r.x, 8 * gi);
            py[gi] = __shfl_sync(0xffffffffu, r.y, 8 * gi);
            pcost[gi] = __shfl_sync(0xffffffffu, r.cost, 8 * gi);
            evals += __shfl_sync(0xffffffffu, r.evals, 8 * gi) << 3;
        }
        if (pcost[0] + pcost[1] < best) {  // 16x8 top + bottom
            best = pcost[0] + pcost[1]; shape = 1;
            mv0x = px[0]; mv0y = py[0]; mv1x = px[1]; mv1y = py[1];
        }
        if (pcost[2] + pcost[3] < best) {  // 8x16 left + right
            best = pcost[2] + pcost[3]; shape = 2;
            mv0x = px[2]; mv0y = py[2]; mv1x = px[3]; mv1y = py[3];
        }
    }
    int32_t* const p = fd.picks + 6LL * m;
    if (sy.ew != nullptr) {
        // the pick to the wavefront: blocks (3,0), (0,3), (3,3)
        const bool second = lane == 0 ? shape == 2 : (lane == 1 ? shape == 1 : shape != 0);
        int wx = second ? mv1x : mv0x, wy = second ? mv1y : mv0y;
        if (mv_far(mv0x) || mv_far(mv0y) || mv_far(mv1x) || mv_far(mv1y)) {  // warp-uniform
            if (lane == 0) { p[0] = shape; p[1] = mv0x; p[2] = mv0y; p[3] = mv1x; p[4] = mv1y; }
            __syncwarp();
            __threadfence();  // the pick before the words
            if (mv_far(wx) || mv_far(wy)) wx = wy = MV_FAR;
        }
        if (lane < EW_PER_MB) st_relaxed_u64(sy.ew + EW_PER_MB * (long long)m + lane, mv_word(sy.epoch, wx, wy));
    }
    if (lane == 0) {
        p[0] = shape; p[1] = mv0x; p[2] = mv0y; p[3] = mv1x; p[4] = mv1y; p[5] = evals;
        fd.costs[2LL * m] = best;
        fd.costs[2LL * m + 1] = c16;
        if (LEARN && fd.fallback) fd.fallback[m] = fell;
        if (sy.ew == nullptr) st_release(sy.flags + m, sy.epoch);  // orders the pick's stores before the flag
    }
    // MC + T/Q of the MB under its pick (mb16.rs:3436-3450): lanes 0..15 the
    // luma 4x4 blocks, the prediction from the staged window when it covers
    // the block's MV; with REC, lanes 16..23 the chroma blocks (plane, block k
    // in SUBBLOCKS order; lanes 24..31 shadow them) and the reconstruction of both
    if (!REC && fd.coeffs == nullptr) {
        __syncwarp();  // the warp's scratch is read: lane 0 writes the next MB's
        return;
    }
    const bool chroma = REC && lane >= 16;
    const int bx = (lane & 3) * 4, by = ((lane >> 2) & 3) * 4;             // luma block
    const int cpl = (lane >> 2) & 1, kb = lane & 3, cbx = (kb & 1) * 4, cby = (kb >> 1) * 4;  // chroma block
    const bool hi_y = chroma ? cby >= 4 : by >= 8, hi_x = chroma ? cbx >= 4 : bx >= 8;
    const bool part = shape == 1 ? hi_y : (shape == 2 ? hi_x : false);
    const int mvx = part ? mv1x : mv0x, mvy = part ? mv1y : mv0y;
    const int cx0 = mbx * 8, cy0 = mby * 8;
    uint32_t sr[4], prd[4];
    const int ccw = pc.cw / 2, cch = pc.ch / 2;
    const int wx = lx + bx + pc.pad - ws.wx0 + (mvx >> 2), wy = ly + by + pc.pad - ws.wy0 + (mvy >> 2);
    const bool in_win = win_ok && win_covers(wx, wy);
    if constexpr (REC) {
        if (sy.bw != nullptr) {
            // the rows of the previous reconstruction that the lane reads
            // outside the window are final, then the warp together: a lane may
            // have it from another that its segment was seen ready
            if (chroma)
                band_wait_px(sy.bw, &ws.bready, 2 * min(cy0 + cby + 4 + (mvy >> 3), cch - 1) + 1,
                             2 * min(cx0 + cbx + 4 + (mvx >> 3), ccw - 1) + 1);
            else if (!in_win)
                band_wait_px(sy.bw, &ws.bready, ly + by + (mvy >> 2) + 5, lx + bx + (mvx >> 2) + 5);
            __syncwarp();
        }
    }
    if (chroma) {
        const uint8_t* sp = rdp->src_c[cpl] + (long long)(cy0 + cby) * ccw + cx0 + cbx;
#pragma unroll
        for (int r = 0; r < 4; r++) sr[r] = __ldg(reinterpret_cast<const uint32_t*>(sp + (long long)r * ccw));
        chroma_rows(rdp->ref_c[cpl], ccw, cch, cx0 + cbx + (mvx >> 3), cy0 + cby + (mvy >> 3), mvx & 7, mvy & 7, prd);
    } else if (lane < 16) {
        const int x = lx + bx, y = ly + by;
#pragma unroll
        for (int r = 0; r < 4; r++) sr[r] = ld4u(pc.d_src + (long long)(y + r) * pc.cw + x);
        if (in_win) {
            win_rows(win, wx, wy, mvx & 3, mvy & 3, prd);
        } else {
            const uint4 r = plane_rows(&ws, x, y, mvx, mvy);
            prd[0] = r.x; prd[1] = r.y; prd[2] = r.z; prd[3] = r.w;
        }
    }
    __syncwarp();  // the window is read: REC's tiles take its place
    const int qi = (by >= 8 ? 2 : 0) + (bx >= 8 ? 1 : 0), kk = ((by & 4) ? 2 : 0) + ((bx & 4) ? 1 : 0);
    int16_t* const co = fd.coeffs + (long long)m * 256 + qi * 64 + kk * 16;
    if (!REC) {
        if (lane < 16) tq4x4_store(sr, prd, fd.qff, fd.qmf, co);
        if (fd.row_count != nullptr) {
            __syncwarp();  // the lanes' stores ordered before lane 0's count
            if (lane == 0 && atom_add_acq_rel(fd.row_count + mby, 1) == mb_w - 1)
                st_release_sys(fd.row_done + mby, fd.row_token);  // the row's last MB: tell the host
        }
    }
    if constexpr (REC) {
        const RecDesc& rd = *rdp;
        RecTiles& rt = *reinterpret_cast<RecTiles*>(winp);
        const BlockQuant bq = block_quant(chroma ? rd.cff : fd.qff, chroma ? rd.cmf : fd.qmf, chroma ? rd.qpc : rd.qp);
        uint32_t r4[4];
        const bool any = mb_code_block(sr, prd, bq, chroma, kb,
                                       chroma ? (lane < 24 ? rd.ccoeffs + (long long)m * 128 + cpl * 64 + kb * 16 : nullptr) : co, r4);
        const unsigned nz = __ballot_sync(0xffffffffu, any) & 0xffffu;
        if (lane < 24) {
            uint8_t* const t = chroma ? &rt.ct[cpl][(2 + cby) * CT + 4 + cbx] : rt.lt + (4 + by) * LT + 4 + bx;
#pragma unroll
            for (int r = 0; r < 4; r++) *reinterpret_cast<uint32_t*>(t + r * (chroma ? CT : LT)) = r4[r];
        }
        if (lane == 0) sy.nz[m] = int(nz);
        // the left and top-right neighbours' deblocking (so the top
        // neighbour's too), then the strips their edges reach, and on lanes
        // 0..3 and 16..19 the left and top MBs' blocks at this MB's edges:
        // their MVs from the published words, their coefficient masks
        const DbStrips strips(lane, rd.rec_y, pc.cw, lx, ly, rd.rec_c, cx0, cy0, rt.lt, rt.ct[0], rt.ct[1], aa, ba, true);
        if (lane == 0 && aa) wait_flag(sy.dfl + m - 1, sy.epoch, sy.status, 1, sy.limit);
        if (lane == 1 && ba) wait_flag(sy.dfl + m - mb_w + (mbx < mb_w - 1 ? 1 : 0), sy.epoch, sy.status, 1, sy.limit);
        __syncwarp();
        // bS: lanes 0..15 the vertical edges (edge e, block row sg),
        // lanes 16..31 the horizontal ones (edge e, block column sg)
        const int hor = lane >> 4, e = (lane >> 2) & 3, sg = lane & 3;
        const bool edge = e > 0 || (hor ? ba : aa);
        unsigned long long nw = 0;
        unsigned nnz = 0;
        if (e == 0 && edge) {
            const int n = hor ? m - mb_w : m - 1;
            nw = __ldcg(sy.ew + EW_PER_MB * (long long)n + (sg >= 2 ? 2 : hor));
            nnz = (unsigned(__ldcg(sy.nz + n)) >> (hor ? 12 + sg : 4 * sg + 3)) & 1u;
        }
        strips.load();
        auto own = [&](int bx4, int by4) {
            const bool second = shape == 1 ? by4 >= 2 : (shape == 2 ? bx4 >= 2 : false);
            return second ? make_int2(mv1x, mv1y) : make_int2(mv0x, mv0y);
        };
        int bs = 0;
        if (edge) {
            const int qbx = hor ? sg : e, qby = hor ? e : sg;
            int2 pm = make_int2(int(int16_t(nw & 0xffffu)), int(int16_t((nw >> 16) & 0xffffu)));
            if (e == 0 && pm.x == MV_FAR) pm = pick_mv_at(fd.picks, hor ? m - mb_w : m - 1, hor ? sg : 3, hor ? 3 : sg);
            if (e > 0) {
                const int pbx = hor ? sg : e - 1, pby = hor ? e - 1 : sg;
                pm = own(pbx, pby);
                nnz = (nz >> (4 * pby + pbx)) & 1u;
            }
            const int2 qm = own(qbx, qby);
            bs = bs_of(nnz != 0, ((nz >> (4 * qby + qbx)) & 1u) != 0, pm.x, pm.y, qm.x, qm.y);
        }
        rt.bs[lane] = bs;
        __syncwarp();
        deblock_mb_tiles(lane, rt.lt, rt.ct[0], rt.ct[1], rt.bs, aa, ba, true, rd.th);
        db_store_mb(lane, rt.lt, rt.ct[0], rt.ct[1], rd.rec_y, pc.cw, lx, ly, rd.rec_c, cx0, cy0, true);
        strips.store();
        __syncwarp();  // every lane's stores ordered before lane 0's release
        if (lane == 0) st_release(sy.dfl + m, sy.epoch);
    }
    __syncwarp();
}

// The persistent plain-ME kernel.  Each warp takes MB tickets dealt in
// wavefront order (frames interleaved) and runs frame_mb on them.  words: the
// launch's MV words (EW_PER_MB per MB), or null to use its flags.  Dynamic
// shared memory: ME_WARPS windows of WIN_BYTES.
template <bool BAL, bool LEARN, bool REC, class TAB>
__device__ __forceinline__ void me_frames_body(const TAB& tab, long long total, const MeParamsDev& prm,
                                               int* __restrict__ counter, int* __restrict__ flags,
                                               unsigned long long* __restrict__ words, int epoch,
                                               int* __restrict__ status, int spin_limit) {
    __shared__ MbScratch scratch[ME_WARPS];
    __shared__ __align__(16) SearchScratch scr[ME_WARPS];
    __shared__ PhaseTab ptab;
    __shared__ __align__(8) unsigned long long win_bar[ME_WARPS];
    extern __shared__ __align__(128) uint8_t me_win[];
    const WarpWindow ww = warp_window(me_win, win_bar, ptab, scr);
    MbScratch& ws = scratch[threadIdx.x >> 5];
    uint32_t parity = 0;
    for (;;) {
        int t = 0;
        if ((threadIdx.x & 31) == 0) t = atomicAdd(counter, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= total) return;
        // the ticket's segment (dealt in order), frame and wavefront position
        int sg = 0;
        while (sg + 1 < tab.nseg() && tab.seg(sg + 1) <= t) sg++;
        const int j = tab.segj(sg);
        const long long u = t - tab.seg(sg);
        const int nxt = j + 1 < tab.n() ? tab.fr(j + 1).mb_w * tab.fr(j + 1).mb_h : 0;
        const int fi = int(u % (j + 1));
        const FrameDesc& fd = tab.fr(fi);
        const int k = nxt + int(u / (j + 1));  // position in the frame's wavefront order
        int mbx, mby;
        wave_mb(fd.mb_w, fd.mb_h, k, mbx, mby);
        const RecDesc* rd = nullptr;
        if constexpr (REC) rd = tab.rec(fi);
        const MbSync sy{words ? words + EW_PER_MB * (long long)fd.flag_base : nullptr, flags + fd.flag_base,
                        REC ? flags + rd->dflag_base : nullptr, REC ? flags + rd->nz_base : nullptr, nullptr, epoch,
                        status, spin_limit};
        frame_mb<BAL, LEARN, REC, false>(fd, rd, mbx, mby, prm, sy, ws, scr[threadIdx.x >> 5], ww, parity, TAB::kGlobal);
    }
}

template <bool BAL, bool LEARN = false>
__global__ void __launch_bounds__(32 * ME_WARPS, BAL ? ME_MIN_BLOCKS : ME_ANY_BLOCKS)
    me_frames_kernel(const __grid_constant__ FrameBatch batch, long long total, const __grid_constant__ MeParamsDev prm,
                     int* __restrict__ counter, int* __restrict__ flags, unsigned long long* __restrict__ words,
                     int epoch, int* __restrict__ status, int spin_limit) {
    me_frames_body<BAL, LEARN, false>(ParamTable{batch}, total, prm, counter, flags, words, epoch, status, spin_limit);
}

// The same kernel over a frame table in device memory (more than ME_MAXF
// frames in one wavefront launch); the frames' tensor maps are read there.
template <bool BAL, bool LEARN = false>
__global__ void __launch_bounds__(32 * ME_WARPS, BAL ? ME_MIN_BLOCKS : ME_ANY_BLOCKS)
    me_frames_dkernel(const FrameDesc* __restrict__ frames, const long long* __restrict__ seg_start,
                      const int* __restrict__ seg_j, int nframes, int nseg, long long total,
                      const __grid_constant__ MeParamsDev prm, int* __restrict__ counter, int* __restrict__ flags,
                      unsigned long long* __restrict__ words, int epoch, int* __restrict__ status, int spin_limit) {
    me_frames_body<BAL, LEARN, false>(DeviceTable{frames, seg_start, seg_j, nframes, nseg}, total, prm, counter, flags,
                                      words, epoch, status, spin_limit);
}

// One or two P frames with the fused reconstruction (h264a_closed_step_frame):
// the frame table with its reconstruction descriptors, by value.
struct StepBatch {
    FrameDesc f[ME_FEW_FRAMES];
    RecDesc rec[ME_FEW_FRAMES];
    long long seg_start[ME_FEW_FRAMES + 1];
    int seg_j[ME_FEW_FRAMES];
    int n, nseg;
};
struct StepTable {
    static constexpr bool kGlobal = false;
    const StepBatch& b;
    __device__ __forceinline__ int n() const { return b.n; }
    __device__ __forceinline__ int nseg() const { return b.nseg; }
    __device__ __forceinline__ long long seg(int s) const { return b.seg_start[s]; }
    __device__ __forceinline__ int segj(int s) const { return b.seg_j[s]; }
    __device__ __forceinline__ const FrameDesc& fr(int i) const { return b.f[i]; }
    __device__ __forceinline__ const RecDesc* rec(int i) const { return &b.rec[i]; }
};
template <bool BAL, bool LEARN>
__global__ void __launch_bounds__(32 * ME_WARPS, BAL ? ME_MIN_BLOCKS : ME_ANY_BLOCKS)
    me_step_kernel(const __grid_constant__ StepBatch batch, long long total, const __grid_constant__ MeParamsDev prm,
                   int* __restrict__ counter, int* __restrict__ flags, unsigned long long* __restrict__ words, int epoch,
                   int* __restrict__ status, int spin_limit) {
    me_frames_body<BAL, LEARN, true>(StepTable{batch}, total, prm, counter, flags, words, epoch, status, spin_limit);
}

// ---------------------------------------------------------------------------
// The pipelined closed loop: every P frame of a clip in one launch
// ---------------------------------------------------------------------------
// Frame h searches the planes of the deblocked reconstruction of frame h-1,
// but an MB only reads the reference pixels its window (and any candidate
// off the window) reaches.  So the launch runs the frames' wavefronts
// overlapped: each frame's tickets are its MBs in wavefront order with
// segment tickets among them.  Segment (b, s) covers picture rows
// 16b .. 16b+15 (band b) and columns 16*segw*s .. (segment s, the first and
// last segments reaching into the padding); its ticket comes after the MB
// whose deblocking makes those reconstruction pixels final, MB
// (min(segw*(s+1), mb_w-1), min(b+1, mb_h-1)) (deblocking runs as a
// wavefront too, so that MB done means every MB up and left of it is), and
// builds the planes of the segment (hpel_strip_rows, its own columns only).
// An MB of frame h waits (bounded) for the segments of frame h-1 its reads
// need (band_wait_px); a segment's flag is published after the flags of the
// segments above and left of it, so one flag stands for all of those.  The
// next frame can therefore start a few MB columns and rows behind the
// previous one instead of a whole frame width behind.  The planes of nbuf
// consecutive frames live in nbuf buffers (frame h's in buffer h % nbuf),
// and a segment ticket of frame h first waits until frame h-nbuf+1, the last
// reader of the buffer's previous picture, has finished every MB.
//
// Deadlock freedom: the warps form `pools` pools, warp i taking frames
// 1 + i % pools, 1 + i % pools + pools, ..., each pool its frames in order, a
// warp moving to the pool's next frame only once the current frame's tickets
// are all dealt.  A ticket waits only on earlier tickets of its own frame, on
// frame h-1 and on frame h-nbuf+1's completion; the oldest unfinished frame
// therefore depends on nothing unfinished, its tickets are all dealt or held
// by warps of its own pool that are not blocked by a later frame, and it
// always progresses.  Every wait is still bounded, and after the first
// timeout the others give up (status 1).
struct PipeParams {
    const FrameDesc* fds;  // per frame 0..n-1 (entry 0 unused), in device memory
    const RecDesc* rds;
    const int* items;      // a frame's tickets: MB index, or -(1 + b * nseg + s)
    int nitems, n, mb_w, mb_h, nbands, nseg, segw, nbuf, pools;
    int* flags;            // per frame fstride ints: MV words, deblocking flags, segment flags
    long long fstride;
    int ew_off, dfl_off, nz_off, band_off;
    int* ctr;              // n ticket counters and n completed-MB counters, zeroed
    int* done;
    const uint8_t* rec_y;  // frame h's luma reconstruction at h * fs
    long long fs;
    uint8_t* planes;       // nbuf plane buffers, pbytes apart
    long long pbytes;
    int cw, ch, pad, word_in, word_out;
    int32_t* frame_words;  // mapped host words: frame h's set to ftoken when it is final (or null)
    int32_t ftoken;
    const int32_t* arrive;  // frame h's sources uploaded once arrive[h] == atoken (or null: all resident)
    int32_t atoken;
};

// Segment (b, s) of frame h: the planes of its reconstruction for padded rows
// [pad + 16b, pad + 16b + 16) (band 0 from row 0, the last band to the end)
// and padded columns [pad + 16*segw*s, pad + 16*segw*(s+1)) (segment 0 from
// column 0, the last segment to the end), into buffer h % nbuf.  One warp,
// in strips of HP_STRIP columns from the segment's first.
__device__ __forceinline__ void pipe_band(const PipeParams& pp, int h, int b, int sg, int epoch, int* status,
                                          int limit) {
    int* const ff = pp.flags + pp.fstride * h;
    const int lane = threadIdx.x & 31;
    if (lane == 0) {
        const int r = min(b + 1, pp.mb_h - 1), x = min(pp.segw * (sg + 1), pp.mb_w - 1);
        wait_flag(ff + pp.dfl_off + r * pp.mb_w + x, epoch, status, 1, limit, POLL_FAR_NS);
        if (h - pp.nbuf + 1 >= 1) {
            const int nmb = pp.mb_w * pp.mb_h;
            for (int it = 0; ld_acquire(pp.done + h - pp.nbuf + 1) < nmb; it++) {
                if (it >= limit || ((it & 255) == 255 && *reinterpret_cast<volatile int*>(status) != 0)) {
                    atomicCAS(status, 0, 1);
                    break;
                }
                __nanosleep(SPIN_NS);
            }
        }
    }
    __syncwarp();
    const int pw = pp.cw + 2 * pp.pad, ph = pp.ch + 2 * pp.pad;
    const int y0 = b == 0 ? 0 : pp.pad + 16 * b;
    const int y1 = b == pp.nbands - 1 ? ph : pp.pad + 16 * b + 16;
    const int x0 = sg == 0 ? 0 : pp.pad + 16 * pp.segw * sg;
    const int x1 = sg == pp.nseg - 1 ? pw : pp.pad + 16 * pp.segw * (sg + 1);
    for (int xs = x0; xs < x1; xs += HP_STRIP)
        hpel_strip_rows<true, true>(pp.rec_y + pp.fs * h, pp.cw, pp.ch, pp.pad, pp.planes + pp.pbytes * (h % pp.nbuf), pw,
                              ph, xs, y0, y1, pp.word_in, pp.word_out, x1);
    // the planes' generic-proxy writes, visible to the readers' bulk copies
    asm volatile("fence.proxy.async.global;" ::: "memory");
    __syncwarp();
    if (lane == 0) {
        int* const sf = ff + pp.band_off + b * pp.nseg + sg;
        if (b > 0) wait_flag(sf - pp.nseg, epoch, status, 1, limit);
        if (sg > 0) wait_flag(sf - 1, epoch, status, 1, limit);
        st_release(sf, epoch);
    }
    __syncwarp();
}

template <bool BAL, bool LEARN>
__global__ void __launch_bounds__(32 * ME_WARPS, BAL ? ME_MIN_BLOCKS : ME_ANY_BLOCKS)
    closed_pipe_kernel(const __grid_constant__ PipeParams pp, const __grid_constant__ MeParamsDev prm, int epoch,
                       int* __restrict__ status, int spin_limit) {
    __shared__ MbScratch scratch[ME_WARPS];
    __shared__ __align__(16) SearchScratch scr[ME_WARPS];
    __shared__ PhaseTab ptab;
    __shared__ __align__(8) unsigned long long win_bar[ME_WARPS];
    __shared__ BandWait bwait[ME_WARPS];
    extern __shared__ __align__(128) uint8_t me_win[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const WarpWindow ww = warp_window(me_win, win_bar, ptab, scr);
    uint32_t parity = 0;
    int fenced = -1;   // the frame whose tensor map this warp has acquired and whose sources it has seen
    int h = 1 + int((blockIdx.x * ME_WARPS + w) % unsigned(pp.pools));  // this warp's pool: frames h, h + pools, ...
    while (h < pp.n) {
        int t = 0;
        if (lane == 0) t = atomicAdd(pp.ctr + h, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= pp.nitems) {
            h += pp.pools;  // every ticket of frame h is dealt: the pool's next frame
            continue;
        }
        const int item = __ldg(pp.items + t);
        if (item < 0) {
            pipe_band(pp, h, (-item - 1) / pp.nseg, (-item - 1) % pp.nseg, epoch, status, spin_limit);
            continue;
        }
        int* const ff = pp.flags + pp.fstride * h;
        if (lane == 0) {
            if (pp.arrive != nullptr && fenced != h) {
                // the frame's sources are still being uploaded beside the launch
                for (int it = 0; ld_acquire(pp.arrive + h) != pp.atoken; it++) {
                    if (it >= spin_limit || ((it & 255) == 255 && *reinterpret_cast<volatile int*>(status) != 0)) {
                        atomicCAS(status, 0, 1);
                        break;
                    }
                    __nanosleep(SPIN_NS);
                }
            }
            if (fenced != h)
                bwait[w] = BandWait{pp.flags + pp.fstride * (h - 1) + pp.band_off, pp.nbands, pp.nseg, 16 * pp.segw, epoch,
                                    spin_limit, status};
        }
        __syncwarp();
        // frame 1's reference (frame 0) is built before the launch
        const MbSync sy{reinterpret_cast<unsigned long long*>(ff + pp.ew_off), nullptr, ff + pp.dfl_off, ff + pp.nz_off,
                        h > 1 ? &bwait[w] : nullptr, epoch, status, spin_limit};
        frame_mb<BAL, LEARN, true, true>(pp.fds[h], pp.rds + h, item % pp.mb_w, item / pp.mb_w, prm, sy, scratch[w], scr[w], ww,
                                   parity, fenced != h);
        fenced = h;
        if (lane == 0 && pp.frame_words == nullptr) {
            red_add_release(pp.done + h, 1);
        } else if (lane == 0) {
            const int c = atom_add_acq_rel(pp.done + h, 1);
            if (c == pp.mb_w * pp.mb_h - 1) {
                // the frame's last MB: its outputs are final, for the host
                __threadfence_system();
                st_release_sys(pp.frame_words + h, pp.ftoken);
            }
        }
        __syncwarp();
    }
}

// One warp waits on a flag that nothing sets; the bounded wait must give up
// after `limit` polls and record status code 2.
__global__ void bounded_wait_selftest_kernel(const int* flag, int* status, int limit) {
    if (threadIdx.x == 0) wait_flag(flag, 1, status, 2, limit);
}

}  // namespace h264a

using namespace h264a;

namespace h264a {
int encode_u8_map_3d(CUtensorMap* map, const uint8_t* base, int w, int h, int d, int bw, int bh, int bd) {
    static const PFN_cuTensorMapEncodeTiled_v12000 encode = [] {  // looked up once, thread-safely
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
        cudaGetLastError();
        return PFN_cuTensorMapEncodeTiled_v12000(nullptr);
    }();
    if (!encode || (reinterpret_cast<uintptr_t>(base) & 15) != 0 || w % 16 != 0 || bw % 16 != 0 || w < bw || h < bh ||
        d < bd || bw > 256 || bh > 256 || bd > 256 || bd < 1)
        return 0;
    const cuuint64_t dim[3] = {cuuint64_t(w), cuuint64_t(h), cuuint64_t(d)};
    const cuuint64_t stride[2] = {cuuint64_t(w), cuuint64_t(w) * cuuint64_t(h)};  // bytes, dims 1 and 2
    const cuuint32_t box[3] = {cuuint32_t(bw), cuuint32_t(bh), cuuint32_t(bd)};
    const cuuint32_t estride[3] = {1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<uint8_t*>(base), dim, stride, box, estride,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
               ? 1
               : 0;
}
}  // namespace h264a

// The F|H|V|C planes of a reference picture as a 3D u8 tensor (pw, ph, 4)
// whose 80 x 42 x 4 box is an MB's window in the WIN_STRIDE / WIN_PLANE
// layout.  Returns 0 when the planes cannot be described (alignment, or no
// driver entry point), and the kernel then stages the window row by row.
static int encode_window_map(CUtensorMap* map, const uint8_t* planes, int pw, int ph) {
    static_assert(WIN_STRIDE % 16 == 0 && WIN_PLANE == WIN_H * WIN_STRIDE && WIN_BYTES == 4 * WIN_PLANE,
                  "the window is one dense 3D box");
    return encode_u8_map_3d(map, planes, pw, ph, 4, WIN_STRIDE, WIN_H, 4);
}

// Dynamic shared memory of me_frames_kernel, its opt-in above 48 KB, and the
// CTAs per SM it reaches.
static int me_frames_setup_once(int& per_sm, bool bal, bool learn);
// Cached per device: the attributes and the occupancy of the frame kernels
// (queried once, not on every launch).
static int me_frames_setup(int& per_sm, bool bal, bool learn = false) {
    constexpr int kMaxDev = 64;
    static int cached[kMaxDev][4];  // CTAs per SM + 1, 0 while unknown
    static std::mutex mu;
    int dev = 0;
    H264A_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDev) return me_frames_setup_once(per_sm, bal, learn);
    std::lock_guard<std::mutex> lock(mu);
    int& c = cached[dev][(bal ? 2 : 0) + (learn ? 1 : 0)];
    if (!c) {
        const int rc = me_frames_setup_once(per_sm, bal, learn);
        if (rc) return rc;
        c = per_sm + 1;
    }
    per_sm = c - 1;
    return H264A_OK;
}

static int me_frames_setup_once(int& per_sm, bool bal, bool learn) {
    const int smem = ME_WARPS * WIN_BYTES;
    H264A_CUDA(cudaFuncSetAttribute(me_frames_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, FRAME_SMEM_MAX));
    H264A_CUDA(cudaFuncSetAttribute(me_frames_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, FRAME_SMEM_MAX));
    H264A_CUDA(cudaFuncSetAttribute(me_frames_dkernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, FRAME_SMEM_MAX));
    H264A_CUDA(cudaFuncSetAttribute(me_frames_dkernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, FRAME_SMEM_MAX));
    H264A_CUDA(cudaFuncSetAttribute(me_frames_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, FRAME_SMEM_MAX));
    H264A_CUDA(cudaFuncSetAttribute(me_frames_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, FRAME_SMEM_MAX));
    H264A_CUDA(cudaFuncSetAttribute(me_frames_dkernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, FRAME_SMEM_MAX));
    H264A_CUDA(cudaFuncSetAttribute(me_frames_dkernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, FRAME_SMEM_MAX));
    H264A_CUDA(cudaFuncSetAttribute(me_step_kernel<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, FRAME_SMEM_MAX));
    H264A_CUDA(cudaFuncSetAttribute(me_step_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, FRAME_SMEM_MAX));
    H264A_CUDA(cudaFuncSetAttribute(me_step_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, FRAME_SMEM_MAX));
    H264A_CUDA(cudaFuncSetAttribute(me_step_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, FRAME_SMEM_MAX));
    per_sm = 0;
    auto kern = bal ? (learn ? me_frames_kernel<true, true> : me_frames_kernel<true, false>)
                    : (learn ? me_frames_kernel<false, true> : me_frames_kernel<false, false>);
    H264A_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * ME_WARPS, smem));
    if (per_sm < 1) per_sm = 1;
    return H264A_OK;
}

// A λ that the Balanced searches' tables hold: every (λ·rate) as i64 (rates
// up to 126) and every cost (distortions below 2^21) fits 31 bits.  The
// encoder's are below 1,500; others run the general search.
static bool balanced_lambda(double lam) { return lam >= 0.0 && lam < LAM_TAB_MAX; }
// True when the parameters are the Balanced preset's (h264a_me_params_default)
// and the frames' λ allow it (lam_ok): the frame kernels then run the searches
// written for it.
static bool balanced_preset(const MeParamsDev& p, bool lam_ok) {
    return lam_ok && p.fast == 0 && p.use_sad == 0 && p.sadfp == 0 && p.kind == 0 && p.me_snap == 1 && p.fc == 1 &&
           p.dia_mask == 0x1cu && p.subpel == 1 && p.subpel_pat == -1 && p.sp_single_pass == 1 &&
           p.me_subpel_iter == 1 && p.sp_maxit == 0 && p.sp_fc == 0;
}

// The non-empty segments of the ticket order of nf frames sorted by MB count,
// descending: segment j (positions [nmb(j+1), nmb(j)) of frames 0..j) has
// (nmb(j) - nmb(j+1)) * (j+1) tickets, and segments are dealt from
// j = nf-1 down.  Writes their first tickets (start[nseg] = the ticket count,
// which equals the frames' MB count) and j values; returns nseg.
static int make_segments(const FrameDesc* f, int nf, long long* start, int* segj) {
    long long acc = 0;
    int ns = 0;
    for (int j = nf - 1; j >= 0; j--) {
        const long long nj = (long long)f[j].mb_w * f[j].mb_h;
        const long long nn = j + 1 < nf ? (long long)f[j + 1].mb_w * f[j + 1].mb_h : 0;
        if (nj == nn) continue;
        start[ns] = acc;
        segj[ns] = j;
        ns++;
        acc += (nj - nn) * (j + 1);
    }
    start[ns] = acc;
    return ns;
}

// CTAs of a frame launch: of those that fit (per_sm on each SM), as many as
// give a warp to every MB of the frames' longest anti-diagonals.  More hold MBs
// that wait: 1, 2, 4 CTAs an SM, one 720p frame with its reconstruction 1,806,
// 1,847, 1,858 us; five 1080p frames (300 MBs, 592 warps) 2,565, 2,579, 2,605;
// fifteen (900) 3,191, 3,177, 3,168; 75 of mixed sizes (2,430) 4,981, 4,494,
// 4,360.
static long long frame_ctas(const FrameDesc* f, int n, long long total, int num_sms, int per_sm) {
    long long wave = 0;
    for (int i = 0; i < n; i++) wave += wave_mbs(f[i].mb_w, f[i].mb_h);
    const long long warps = (long long)ME_WARPS * num_sms, want = std::max(1LL, (wave + warps - 1) / warps);
    return std::min(num_sms * std::min<long long>(per_sm, want), (total + ME_WARPS - 1) / ME_WARPS);
}

// fb.nseg and the segment arrays of a batch of fb.n sorted frames; returns the
// ticket count.
static long long fill_segments(FrameBatch& fb) {
    fb.nseg = make_segments(fb.f, fb.n, fb.seg_start, fb.seg_j);
    return fb.seg_start[fb.nseg];
}

static void launch_me_frames_dtab(const MeParamsDev& prm, unsigned blocks, size_t sm, cudaStream_t st, const FrameDesc* frames,
                                  const long long* seg_start, const int* seg_j, int nframes, int nseg, long long total,
                                  int* counter, int* flags, unsigned long long* words, int epoch, int* status,
                                  bool lam_ok, bool learn = false) {
    const bool bal = balanced_preset(prm, lam_ok);
    if (learn && bal)
        me_frames_dkernel<true, true><<<blocks, 32 * ME_WARPS, sm, st>>>(frames, seg_start, seg_j, nframes, nseg, total,
                                                                        prm, counter, flags, words, epoch, status, SPIN_LIMIT);
    else if (learn)
        me_frames_dkernel<false, true><<<blocks, 32 * ME_WARPS, sm, st>>>(frames, seg_start, seg_j, nframes, nseg, total,
                                                                         prm, counter, flags, words, epoch, status, SPIN_LIMIT);
    else if (bal)
        me_frames_dkernel<true><<<blocks, 32 * ME_WARPS, sm, st>>>(frames, seg_start, seg_j, nframes, nseg, total, prm,
                                                                  counter, flags, words, epoch, status, SPIN_LIMIT);
    else
        me_frames_dkernel<false><<<blocks, 32 * ME_WARPS, sm, st>>>(frames, seg_start, seg_j, nframes, nseg, total, prm,
                                                                   counter, flags, words, epoch, status, SPIN_LIMIT);
}

static void launch_me_step(const MeParamsDev& prm, unsigned blocks, size_t sm, cudaStream_t st, const StepBatch& sb, long long total,
                           int* counter, int* flags, unsigned long long* words, int epoch, int* status, bool lam_ok,
                           bool learn) {
    auto kern = balanced_preset(prm, lam_ok) ? (learn ? me_step_kernel<true, true> : me_step_kernel<true, false>)
                                     : (learn ? me_step_kernel<false, true> : me_step_kernel<false, false>);
    kern<<<blocks, 32 * ME_WARPS, sm, st>>>(sb, total, prm, counter, flags, words, epoch, status, SPIN_LIMIT);
}

static void launch_me_frames(const MeParamsDev& prm, unsigned blocks, size_t sm, cudaStream_t st, const FrameBatch& fb,
                             long long total, int* counter, int* flags, unsigned long long* words, int epoch,
                             int* status, bool lam_ok, bool learn = false) {
    const bool bal = balanced_preset(prm, lam_ok);
    if (learn && bal)
        me_frames_kernel<true, true><<<blocks, 32 * ME_WARPS, sm, st>>>(fb, total, prm, counter, flags, words, epoch, status,
                                                                       SPIN_LIMIT);
    else if (learn)
        me_frames_kernel<false, true><<<blocks, 32 * ME_WARPS, sm, st>>>(fb, total, prm, counter, flags, words, epoch, status,
                                                                        SPIN_LIMIT);
    else if (bal)
        me_frames_kernel<true><<<blocks, 32 * ME_WARPS, sm, st>>>(fb, total, prm, counter, flags, words, epoch, status,
                                                                 SPIN_LIMIT);
    else
        me_frames_kernel<false><<<blocks, 32 * ME_WARPS, sm, st>>>(fb, total, prm, counter, flags, words, epoch, status,
                                                                  SPIN_LIMIT);
}

extern "C" int h264a_selftest_bounded_wait(h264a_ctx* ctx, int spin_limit, void* stream) {
    if (!ctx || spin_limit < 0 || spin_limit > SPIN_LIMIT) return fail(H264A_E_ARG, "selftest_bounded_wait: bad limit");
    int rc = ensure_me_scratch(ctx, 1);
    if (rc) return rc;
    cudaStream_t st = pick_stream(ctx, stream);
    // the counter word is zero-initialised scratch that no kernel of this call writes
    H264A_CUDA(cudaMemsetAsync(ctx->q[Q_MAIN].d_counter, 0, sizeof(int32_t), st));
    bounded_wait_selftest_kernel<<<1, 32, 0, st>>>(ctx->q[Q_MAIN].d_counter, ctx->d_status, spin_limit);
    return check_launch("bounded_wait_selftest_kernel");
}

extern "C" int h264a_me_search(h264a_ctx* ctx, const h264a_picture* d_pics, int npics, const h264a_me_params* params,
                               const h264a_me_job* d_jobs, int n, h264a_me_result* d_out, void* stream) {
    if (!ctx || !d_pics || !params || !d_jobs || !d_out) return fail(H264A_E_ARG, "me_search: null pointer");
    if (n < 0 || npics < 1) return fail(H264A_E_ARG, "me_search: bad count");
    if ((params->mv_cost_kind == 1 || params->mv_cost_kind == 2) && !params->d_mv_cost_tab)
        return fail(H264A_E_ARG, "me_search: mv cost kinds 1 and 2 need d_mv_cost_tab");
    if (n == 0) return H264A_OK;
    const MeParamsDev prm = to_dev(*params);
    me_search_kernel<<<unsigned((n + ME_WARPS - 1) / ME_WARPS), 32 * ME_WARPS, 0, pick_stream(ctx, stream)>>>(
        d_pics, npics, prm, d_jobs, n, d_out);
    return check_launch("me_search_kernel");
}

// Plain-ME of a batch of frames (h264a_me_frames); with `tq`, each frame's
// MC + luma T/Q is fused in (h264a_me_tq_frames, h264a_pixel_path_host).
// A frame table's pinned staging buffer (at least `bytes`), then its upload
// into the device copy on `st`; table_done after the launch that reads it
// records the event both wait for before they are reused.
static int table_host(h264a_ctx* ctx, size_t bytes, char** host) {
    if (!ctx->me_tab_ev) H264A_CUDA(cudaEventCreateWithFlags(&ctx->me_tab_ev, cudaEventDisableTiming));
    H264A_CUDA(cudaEventSynchronize(ctx->me_tab_ev));
    if (bytes > ctx->me_tab_cap) {
        if (ctx->me_tab) cudaFree(ctx->me_tab);
        if (ctx->me_tab_host) cudaFreeHost(ctx->me_tab_host);
        ctx->me_tab = ctx->me_tab_host = nullptr;
        ctx->me_tab_cap = 0;
        if (cudaMalloc(&ctx->me_tab, bytes) != cudaSuccess || cudaMallocHost(&ctx->me_tab_host, bytes) != cudaSuccess) {
            cudaGetLastError();
            return fail(H264A_E_NOMEM, "frame table allocation failed");
        }
        ctx->me_tab_cap = bytes;
    }
    *host = static_cast<char*>(ctx->me_tab_host);
    return H264A_OK;
}
static int table_upload(h264a_ctx* ctx, size_t bytes, cudaStream_t st) {
    H264A_CUDA(cudaMemcpyAsync(ctx->me_tab, ctx->me_tab_host, bytes, cudaMemcpyHostToDevice, st));
    return H264A_OK;
}
static int table_done(h264a_ctx* ctx, cudaStream_t st) {
    H264A_CUDA(cudaEventRecord(ctx->me_tab_ev, st));
    return H264A_OK;
}

int h264a::me_frames_run(h264a_ctx* ctx, const h264a_me_frame* h_frames, int nframes,
                         const h264a_me_params* params, const MeTqOut* tq, void* stream, const MeLearnIn* learn,
                         const MeRecIn* rec) {
    if (!ctx || !h_frames || !params) return fail(H264A_E_ARG, "me_frames: null pointer");
    if (nframes < 1) return fail(H264A_E_ARG, "me_frames: need at least one frame");
    if (rec && (!tq || nframes > ME_FEW_FRAMES))
        return fail(H264A_E_ARG, "me_frames: the fused reconstruction needs T/Q outputs and at most two frames");
    if ((params->mv_cost_kind == 1 || params->mv_cost_kind == 2) && !params->d_mv_cost_tab)
        return fail(H264A_E_ARG, "me_frames: mv cost kinds 1 and 2 need d_mv_cost_tab");
    for (int i = 0; i < nframes; i++) {
        const h264a_me_frame& f = h_frames[i];
        if (!f.pic.d_src || !f.pic.d_planes || !f.d_picks || !f.d_costs)
            return fail(H264A_E_ARG, "me_frames: null frame pointer");
        if (f.pic.cw < 16 || f.pic.ch < 16 || f.pic.cw % 16 || f.pic.ch % 16 || f.pic.pad < 3 || f.pic.pad > 128)
            return fail(H264A_E_ARG, "me_frames: frames must be MB-aligned with 3 <= pad <= 128");
        if ((long long)(f.pic.cw / 16) * (f.pic.ch / 16) > (1 << 24))
            return fail(H264A_E_ARG, "me_frames: frame too large");
    }
    cudaStream_t st = pick_stream(ctx, stream);
    const MeParamsDev prm = to_dev(*params);
    // One wavefront launch over all frames, largest first: the frame table in
    // the kernel's parameters up to ME_MAXF frames, in device memory beyond.
    std::vector<int> order(nframes);
    for (int i = 0; i < nframes; i++) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        return (long long)h_frames[a].pic.cw * h_frames[a].pic.ch > (long long)h_frames[b].pic.cw * h_frames[b].pic.ch;
    });
    std::vector<FrameDesc> desc(nframes);
    memset(desc.data(), 0, sizeof(FrameDesc) * nframes);
    RecDesc rdesc[ME_FEW_FRAMES];
    memset(rdesc, 0, sizeof rdesc);
    long long total = 0;
    bool lam_ok = true;
    for (int k = 0; k < nframes; k++) {
        const h264a_me_frame& f = h_frames[order[k]];
        FrameDesc& d = desc[k];
        lam_ok = lam_ok && balanced_lambda(f.lambda_me);
        d.pic = f.pic;
        d.tmap_ok = encode_window_map(&d.tmap, f.pic.d_planes, f.pic.cw + 2 * f.pic.pad, f.pic.ch + 2 * f.pic.pad);
        d.lambda_me = f.lambda_me;
        d.split_gate = f.split_gate;
        d.picks = f.d_picks;
        d.costs = f.d_costs;
        d.mb_w = f.pic.cw / 16;
        d.mb_h = f.pic.ch / 16;
        d.flag_base = int(total);
        if (tq) {
            const MeTqOut& t = tq[order[k]];
            d.coeffs = t.coeffs;
            make_quant_row4(t.qp, t.dz_div, d.qff, d.qmf);
            d.row_count = t.row_count;
            d.row_done = t.row_done;
            d.row_token = t.row_token;
        }
        if (learn) {
            const MeLearnIn& l = learn[order[k]];
            d.props = l.props;
            d.fallback = l.fallback;
            d.prop_t = l.prop_t;
        }
        if (rec) {
            const MeRecIn& r = rec[order[k]];
            if (!r.src_u || !r.src_v || !r.ref_u || !r.ref_v || !r.rec_y || !r.rec_u || !r.rec_v || !r.ccoeffs)
                return fail(H264A_E_ARG, "me_frames: null reconstruction pointer");
            if (((reinterpret_cast<uintptr_t>(r.src_u) | reinterpret_cast<uintptr_t>(r.src_v) |
                  reinterpret_cast<uintptr_t>(r.ref_u) | reinterpret_cast<uintptr_t>(r.ref_v) |
                  reinterpret_cast<uintptr_t>(r.rec_y) | reinterpret_cast<uintptr_t>(r.rec_u) |
                  reinterpret_cast<uintptr_t>(r.rec_v)) & 3) ||
                ((reinterpret_cast<uintptr_t>(r.ccoeffs) | reinterpret_cast<uintptr_t>(tq[order[k]].coeffs)) & 15))
                return fail(H264A_E_ARG, "me_frames: planes must be 4-byte and levels 16-byte aligned");
            const int qp = tq[order[k]].qp;
            if (qp < 0 || qp > 51) return fail(H264A_E_ARG, "me_frames: qp out of 0..51");
            RecDesc& rd = rdesc[k];
            rd.src_c[0] = r.src_u; rd.src_c[1] = r.src_v;
            rd.ref_c[0] = r.ref_u; rd.ref_c[1] = r.ref_v;
            rd.rec_y = r.rec_y;
            rd.rec_c[0] = r.rec_u; rd.rec_c[1] = r.rec_v;
            rd.ccoeffs = r.ccoeffs;
            rd.qp = qp;
            rd.qpc = chroma_qp_of(qp);
            make_quant_row4(rd.qpc, 6, rd.cff, rd.cmf);  // chroma: the inter dead-zone
            rd.th = db_thresholds(qp, 0, 0, 0);
        }
        total += (long long)d.mb_w * d.mb_h;
        if (total >= (1LL << 31)) return fail(H264A_E_ARG, "me_frames: too many macroblocks in one call");
    }
    int per_sm = 0;
    int rc = me_frames_setup(per_sm, balanced_preset(prm, lam_ok), learn != nullptr);
    if (rc) return rc;
    std::vector<long long> seg(nframes + 1);
    std::vector<int> segj(nframes);
    const int nseg = make_segments(desc.data(), nframes, seg.data(), segj.data());
    if (seg[nseg] != total) return fail(H264A_E_ARG, "me_frames: internal queue layout error");
    // Launches of few frames run on the closed loop's queue, larger ones on the
    // main one.  Picks go to the wavefront as MV words where the pictures'
    // sides allow it and the words stay below 400 MB, else by flags.  The
    // words, and the few-frame queue's flags (which also hold other layouts),
    // are cleared ahead of the launch.
    const bool few = nframes <= ME_FEW_FRAMES;
    bool words_ok = total <= (1LL << 24);
    for (int k = 0; k < nframes; k++)
        if (desc[k].pic.cw + 2 * desc[k].pic.pad > EW_MAX_SIDE || desc[k].pic.ch + 2 * desc[k].pic.pad > EW_MAX_SIDE)
            words_ok = false;
    if (rec && !words_ok)
        return fail(H264A_E_ARG, "me_frames: the fused reconstruction needs pictures of at most 8191 - 2 pad samples");
    const int qi = few ? Q_WIDE : Q_MAIN;
    WorkQueue& qw = ctx->q[qi];
    const size_t nflags = size_t(rec ? 3 * total : total);  // with rec: then deblocking flags and coefficient masks
    rc = ensure_me_scratch(ctx, nflags, qi);
    if (!rc && words_ok) rc = ensure_me_words(ctx, size_t(EW_PER_MB) * size_t(total), qi);
    if (rc) return rc;
    H264A_CUDA(cudaMemsetAsync(qw.d_counter, 0, sizeof(int32_t), st));
    if (few) H264A_CUDA(cudaMemsetAsync(qw.d_flags, 0, sizeof(int32_t) * nflags, st));
    unsigned long long* words = words_ok ? qw.d_words : nullptr;
    if (words) H264A_CUDA(cudaMemsetAsync(words, 0, sizeof(unsigned long long) * EW_PER_MB * size_t(total), st));
    const int epoch = next_epoch(ctx, st, qi);
    if (epoch < 0) return H264A_E_CUDA;
    const long long blocks = frame_ctas(desc.data(), nframes, total, ctx->num_sms, per_sm);
    if (rec) {
        StepBatch sb;
        memset(&sb, 0, sizeof sb);
        sb.n = nframes;
        memcpy(sb.f, desc.data(), sizeof(FrameDesc) * nframes);
        for (int k = 0; k < nframes; k++) {
            sb.rec[k] = rdesc[k];
            sb.rec[k].dflag_base = int(total) + desc[k].flag_base;
            sb.rec[k].nz_base = int(2 * total) + desc[k].flag_base;
        }
        sb.nseg = make_segments(sb.f, sb.n, sb.seg_start, sb.seg_j);
        if (sb.seg_start[sb.nseg] != total) return fail(H264A_E_ARG, "me_frames: internal queue layout error");
        launch_me_step(prm, unsigned(blocks), frame_smem(blocks, ctx->num_sms), st, sb, total, qw.d_counter, qw.d_flags, words, epoch, ctx->d_status,
                       lam_ok, learn != nullptr);
        return check_launch("me_step_kernel");
    }
    if (nframes <= ME_MAXF) {
        FrameBatch fb;
        memset(&fb, 0, sizeof fb);
        fb.n = nframes;
        memcpy(fb.f, desc.data(), sizeof(FrameDesc) * nframes);
        if (fill_segments(fb) != total) return fail(H264A_E_ARG, "me_frames: internal queue layout error");
        launch_me_frames(prm, unsigned(blocks), frame_smem(blocks, ctx->num_sms), st, fb, total, qw.d_counter, qw.d_flags, words, epoch, ctx->d_status,
                         lam_ok, learn != nullptr);
        return check_launch("me_frames_kernel");
    }
    // the table, its segment starts and j values in one device buffer
    const size_t b_desc = sizeof(FrameDesc) * nframes, b_seg = sizeof(long long) * (nseg + 1),
                 b_j = sizeof(int) * nseg, bytes = b_desc + b_seg + b_j;
    char* hst = nullptr;
    rc = table_host(ctx, bytes, &hst);
    if (rc) return rc;
    memcpy(hst, desc.data(), b_desc);
    memcpy(hst + b_desc, seg.data(), b_seg);
    memcpy(hst + b_desc + b_seg, segj.data(), b_j);
    rc = table_upload(ctx, bytes, st);
    if (rc) return rc;
    char* dv = static_cast<char*>(ctx->me_tab);
    launch_me_frames_dtab(prm, unsigned(blocks), frame_smem(blocks, ctx->num_sms), st, reinterpret_cast<const FrameDesc*>(dv),
                          reinterpret_cast<const long long*>(dv + b_desc), reinterpret_cast<const int*>(dv + b_desc + b_seg),
                          nframes, nseg, total, qw.d_counter, qw.d_flags, words, epoch, ctx->d_status,
                          lam_ok, learn != nullptr);
    rc = check_launch("me_frames_dkernel");
    if (rc) return rc;
    return table_done(ctx, st);
}

extern "C" int h264a_me_frames(h264a_ctx* ctx, const h264a_me_frame* h_frames, int nframes,
                               const h264a_me_params* params, void* stream) {
    return me_frames_run(ctx, h_frames, nframes, params, nullptr, stream);
}

extern "C" int h264a_me_frames_learned(h264a_ctx* ctx, const h264a_me_learned_frame* h_frames, int nframes,
                                       const h264a_me_params* params, void* stream) {
    if (!ctx || !h_frames || !params) return fail(H264A_E_ARG, "me_frames_learned: null pointer");
    if (nframes < 1) return fail(H264A_E_ARG, "me_frames_learned: need at least one frame");
    std::vector<h264a_me_frame> me(nframes);
    std::vector<MeLearnIn> ln(nframes);
    for (int i = 0; i < nframes; i++) {
        const h264a_me_learned_frame& f = h_frames[i];
        if (!f.d_props) return fail(H264A_E_ARG, "me_frames_learned: null proposals");
        if (f.fallback_t < 0) return fail(H264A_E_ARG, "me_frames_learned: negative fallback threshold");
        me[i] = f.me;
        ln[i] = MeLearnIn{f.d_props, f.d_fallback, f.fallback_t};
    }
    return me_frames_run(ctx, me.data(), nframes, params, nullptr, stream, ln.data());
}

extern "C" int h264a_me_tq_frames(h264a_ctx* ctx, const h264a_me_tq_frame* h_frames, int nframes,
                                  const h264a_me_params* params, void* stream) {
    if (!ctx || !h_frames || !params) return fail(H264A_E_ARG, "me_tq_frames: null pointer");
    if (nframes < 1) return fail(H264A_E_ARG, "me_tq_frames: need at least one frame");
    std::vector<h264a_me_frame> me(nframes);
    std::vector<MeTqOut> tq(nframes);
    for (int i = 0; i < nframes; i++) {
        const h264a_me_tq_frame& f = h_frames[i];
        if (!f.d_coeffs || (reinterpret_cast<uintptr_t>(f.d_coeffs) & 15) != 0)
            return fail(H264A_E_ARG, "me_tq_frames: coefficients must be non-null and 16-byte aligned");
        if (f.qp < 0 || f.qp > 51 || f.dz_div < 1) return fail(H264A_E_ARG, "me_tq_frames: qp out of 0..51 or dz_div < 1");
        me[i] = f.me;
        tq[i] = MeTqOut{f.d_coeffs, f.qp, f.dz_div, nullptr, nullptr, 0};
    }
    return me_frames_run(ctx, me.data(), nframes, params, tq.data(), stream);
}

// ---------------------------------------------------------------------------
// Plain-ME frames without any allocation
// ---------------------------------------------------------------------------
//
// Some callers cannot allocate device memory at the moment they run motion
// estimation: a real-time encoder thread that must not block on the CUDA
// allocator (cudaMalloc can synchronise the device and take a global lock),
// or a host application that hands this library a fixed memory budget and
// owns every buffer itself.  h264a_me_frames needs a context, and the
// context allocates the persistent kernel's scratch (the work-queue counter
// and one done flag per macroblock).  The entry below runs the same kernel
// with that scratch taken from this fixed array instead: one counter word
// plus one flag word per macroblock, for at most H264A_NOALLOC_MAX_MBS
// macroblocks per call (256 KiB per device, held by every device that loads
// the library until the process exits).

namespace h264a {

// [0] work-queue counter, [1..] per-MB done flags.
static __device__ __align__(256) int g_noalloc_scratch[1 + H264A_NOALLOC_MAX_MBS];

// The device address of g_noalloc_scratch on each device (nullptr: not yet
// looked up).  It is looked up once per device and kept; a caller that resets
// a device's primary context (cudaDeviceReset) must not call this entry point
// on that device again in the same process.
struct NoallocDevice {
    int* scratch;
};
constexpr int kNoallocMaxDevices = 64;
constexpr int kNoallocFlag = 1;  // the value a published MB's flag takes
static NoallocDevice g_noalloc_dev[kNoallocMaxDevices];
static std::mutex g_noalloc_mu;

}  // namespace h264a

extern "C" int h264a_me_frames_noalloc(const h264a_me_frame* h_frames, int nframes, const h264a_me_params* params,
                                       int32_t* d_status, void* stream) {
    if (!h_frames || !params || !d_status) return fail(H264A_E_ARG, "me_frames_noalloc: null pointer");
    if (nframes < 1 || nframes > ME_MAXF)
        return fail(H264A_E_ARG, "me_frames_noalloc: 1 to " + std::to_string(ME_MAXF) + " frames per call");
    if ((params->mv_cost_kind == 1 || params->mv_cost_kind == 2) && !params->d_mv_cost_tab)
        return fail(H264A_E_ARG, "me_frames_noalloc: mv cost kinds 1 and 2 need d_mv_cost_tab");
    long long total = 0;
    for (int i = 0; i < nframes; i++) {
        const h264a_me_frame& f = h_frames[i];
        if (!f.pic.d_src || !f.pic.d_planes || !f.d_picks || !f.d_costs)
            return fail(H264A_E_ARG, "me_frames_noalloc: null frame pointer");
        if (f.pic.cw < 16 || f.pic.ch < 16 || f.pic.cw % 16 || f.pic.ch % 16 || f.pic.pad < 3 || f.pic.pad > 128)
            return fail(H264A_E_ARG, "me_frames_noalloc: frames must be MB-aligned with 3 <= pad <= 128");
        total += (long long)(f.pic.cw / 16) * (f.pic.ch / 16);
    }
    if (total > H264A_NOALLOC_MAX_MBS)
        return fail(H264A_E_ARG, "me_frames_noalloc: " + std::to_string(total) + " macroblocks exceed the " +
                                     std::to_string(H264A_NOALLOC_MAX_MBS) + "-macroblock scratch of this entry point");
    int dev = 0;
    H264A_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoallocMaxDevices) return fail(H264A_E_ARG, "me_frames_noalloc: device index too large");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    int* scratch;
    {
        std::lock_guard<std::mutex> lock(g_noalloc_mu);
        NoallocDevice& nd = g_noalloc_dev[dev];
        if (!nd.scratch) {
            // first call on this device: the array's device address (the
            // symbol itself is only a host-side stand-in)
            void* p = nullptr;
            H264A_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
            nd.scratch = static_cast<int*>(p);
        }
        scratch = nd.scratch;
    }
    // frames largest first, dealt round-robin in wavefront order (as h264a_me_frames)
    int order[ME_MAXF];
    for (int i = 0; i < nframes; i++) order[i] = i;
    for (int i = 1; i < nframes; i++) {  // stable insertion sort by size, descending
        const int v = order[i];
        const long long sv = (long long)h_frames[v].pic.cw * h_frames[v].pic.ch;
        int k = i;
        while (k > 0 && (long long)h_frames[order[k - 1]].pic.cw * h_frames[order[k - 1]].pic.ch < sv) {
            order[k] = order[k - 1];
            k--;
        }
        order[k] = v;
    }
    FrameBatch fb;
    memset(&fb, 0, sizeof fb);
    fb.n = nframes;
    total = 0;
    bool lam_ok = true;
    for (int k = 0; k < nframes; k++) {
        const h264a_me_frame& f = h_frames[order[k]];
        FrameDesc& d = fb.f[k];
        lam_ok = lam_ok && balanced_lambda(f.lambda_me);
        d.pic = f.pic;
        d.tmap_ok = encode_window_map(&d.tmap, f.pic.d_planes, f.pic.cw + 2 * f.pic.pad, f.pic.ch + 2 * f.pic.pad);
        d.lambda_me = f.lambda_me;
        d.split_gate = f.split_gate;
        d.picks = f.d_picks;
        d.costs = f.d_costs;
        d.mb_w = f.pic.cw / 16;
        d.mb_h = f.pic.ch / 16;
        d.flag_base = int(total);
        total += (long long)d.mb_w * d.mb_h;
    }
    fill_segments(fb);
    // The counter, this call's flags and the caller's status word start at
    // zero: they are cleared on the stream ahead of the launch (at most
    // 256 KiB), and each MB's flag is set to 1 when its pick is published.
    // Nothing of an earlier call's array contents is read.
    H264A_CUDA(cudaMemsetAsync(scratch, 0, sizeof(int) * size_t(1 + total), st));
    H264A_CUDA(cudaMemsetAsync(d_status, 0, sizeof(int32_t), st));
    int per_sm = 0, sms = 0;
    const MeParamsDev prm = to_dev(*params);
    const int rc0 = me_frames_setup(per_sm, balanced_preset(prm, lam_ok));
    if (rc0) return rc0;
    H264A_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const long long blocks = frame_ctas(fb.f, fb.n, total, sms, per_sm);
    launch_me_frames(prm, unsigned(blocks), frame_smem(blocks, sms), st, fb, total, scratch, scratch + 1, nullptr, kNoallocFlag, d_status, lam_ok);
    return check_launch("me_frames_kernel (no-alloc)");
}

// ---------------------------------------------------------------------------
// The pipelined closed loop's launch
// ---------------------------------------------------------------------------

static int closed_pipe_setup_once() {
    H264A_CUDA(cudaFuncSetAttribute(closed_pipe_kernel<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, FRAME_SMEM_MAX));
    H264A_CUDA(cudaFuncSetAttribute(closed_pipe_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, FRAME_SMEM_MAX));
    H264A_CUDA(cudaFuncSetAttribute(closed_pipe_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, FRAME_SMEM_MAX));
    H264A_CUDA(cudaFuncSetAttribute(closed_pipe_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, FRAME_SMEM_MAX));
    return H264A_OK;
}

// The per-device kernel attributes and the CTAs per SM of the pipelined loop.
static int closed_pipe_setup(int& per_sm, bool bal) {
    constexpr int kMaxDev = 64;
    static int cached[kMaxDev][2];
    static std::mutex mu;
    int dev = 0;
    H264A_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    const bool known = dev >= 0 && dev < kMaxDev;
    if (known && cached[dev][bal]) {
        per_sm = cached[dev][bal];
        return H264A_OK;
    }
    const int rc = closed_pipe_setup_once();
    if (rc) return rc;
    auto kern = bal ? closed_pipe_kernel<true, true> : closed_pipe_kernel<false, true>;
    H264A_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * ME_WARPS, ME_WARPS * WIN_BYTES));
    if (per_sm < 1) per_sm = 1;
    if (known) cached[dev][bal] = per_sm;
    return H264A_OK;
}

int h264a::closed_pipe_run(h264a_ctx* ctx, const ClosedPipeIn& in, const h264a_me_params* params, cudaStream_t st,
                           int32_t* frame_words, int32_t token) {
    const int n = in.n, cw = in.cw, ch = in.ch, pad = in.pad;
    const int pw = cw + 2 * pad, ph = ch + 2 * pad;
    if (n < 2) return H264A_OK;
    if (pw > 8191 || ph > 8191) return fail(H264A_E_ARG, "closed loop: pictures too large for the pipelined loop");
    const int mb_w = cw / 16, mb_h = ch / 16, nmb = mb_w * mb_h, nbands = mb_h;
    const long long fs = (long long)cw * ch, cs = fs / 4, pbytes = 4LL * pw * ph;
    const MeParamsDev prm = to_dev(*params);
    const bool bal = balanced_preset(prm, balanced_lambda(in.lambda_me)), learn = in.props != nullptr;
    int per_sm = 0;
    int rc = closed_pipe_setup(per_sm, bal);
    if (rc) return rc;
    // the frame and reconstruction descriptors (entry 0 unused)
    std::vector<FrameDesc> fds(n);
    std::vector<RecDesc> rds(n);
    memset(fds.data(), 0, sizeof(FrameDesc) * n);
    memset(rds.data(), 0, sizeof(RecDesc) * n);
    // the plane buffers (frame h's planes in buffer h % nbuf), the column
    // segments of the bands, the warp pools
    const int nbuf = std::min(n, H264A_CLOSED_PLANE_PICTURES);
    const int segw = pipe_segw(mb_w), nseg = (mb_w + segw - 1) / segw;
    const int pools = std::min(pipe_pools(mb_w, mb_h), n - 1);
    if (pad % 4) return fail(H264A_E_ARG, "closed loop: the plane padding must be a multiple of 4");
    std::vector<CUtensorMap> maps(nbuf);
    std::vector<int> maps_ok(nbuf);
    for (int k = 0; k < nbuf; k++) maps_ok[k] = encode_window_map(&maps[k], in.planes + pbytes * k, pw, ph);
    for (int h = 1; h < n; h++) {
        FrameDesc& d = fds[h];
        const int buf = (h - 1) % nbuf;
        d.tmap = maps[buf];
        d.tmap_ok = maps_ok[buf];
        d.pic = h264a_picture{in.y + fs * h, in.planes + pbytes * buf, cw, ch, pad};
        d.lambda_me = in.lambda_me;
        d.split_gate = in.split_gate;
        d.picks = in.picks + 6LL * nmb * h;
        d.costs = in.costs + 2LL * nmb * h;
        d.mb_w = mb_w;
        d.mb_h = mb_h;
        d.coeffs = in.coeffs + 256LL * nmb * h;
        make_quant_row4(in.qp, in.dz_div, d.qff, d.qmf);
        if (in.props) {
            d.props = in.props + 16LL * nmb * h;
            d.fallback = in.fallback ? in.fallback + (long long)nmb * h : nullptr;
            d.prop_t = in.prop_t;
        }
        RecDesc& r = rds[h];
        r.src_c[0] = in.u + cs * h;
        r.src_c[1] = in.v + cs * h;
        r.ref_c[0] = in.rec_u + cs * (h - 1);
        r.ref_c[1] = in.rec_v + cs * (h - 1);
        r.rec_y = in.rec_y + fs * h;
        r.rec_c[0] = in.rec_u + cs * h;
        r.rec_c[1] = in.rec_v + cs * h;
        r.ccoeffs = in.ccoeffs + 128LL * nmb * h;
        r.qp = in.qp;
        r.qpc = chroma_qp_of(in.qp);
        make_quant_row4(r.qpc, 6, r.cff, r.cmf);
        r.th = db_thresholds(in.qp, 0, 0, 0);
    }
    // a frame's tickets: its MBs in wavefront order (anti-diagonals t = x + 2y,
    // then y), and segment (b, s) right after MB (min(segw*(s+1), mb_w-1),
    // min(b+1, mb_h-1)), segments of one MB in (b, s) order
    std::vector<std::vector<int>> trig(nmb);
    for (int b = 0; b < nbands; b++)
        for (int sg = 0; sg < nseg; sg++)
            trig[std::min(b + 1, mb_h - 1) * mb_w + std::min(segw * (sg + 1), mb_w - 1)].push_back(-(1 + b * nseg + sg));
    std::vector<int> items;
    items.reserve(nmb + nbands * nseg);
    for (int t = 0; t <= (mb_w - 1) + 2 * (mb_h - 1); t++) {
        for (int y = 0; y < mb_h; y++) {
            const int x = t - 2 * y;
            if (x < 0 || x >= mb_w) continue;
            items.push_back(y * mb_w + x);
            for (int it : trig[y * mb_w + x]) items.push_back(it);
        }
    }
    if ((int)items.size() != nmb + nbands * nseg) return fail(H264A_E_ARG, "closed loop: internal ticket layout error");
    const size_t b_fd = sizeof(FrameDesc) * n, b_rd = (sizeof(RecDesc) * n + 63) & ~size_t(63),
                 b_it = sizeof(int) * items.size();
    char* hst = nullptr;
    rc = table_host(ctx, b_fd + b_rd + b_it, &hst);
    if (rc) return rc;
    memcpy(hst, fds.data(), b_fd);
    memcpy(hst + b_fd, rds.data(), sizeof(RecDesc) * n);
    memcpy(hst + b_fd + b_rd, items.data(), b_it);
    rc = table_upload(ctx, b_fd + b_rd + b_it, st);
    if (rc) return rc;
    char* dv = static_cast<char*>(ctx->me_tab);
    // flags: n ticket counters, n completed-MB counters, then per frame its
    // MV words, deblocking flags, coefficient masks and band flags (an even count per frame)
    PipeParams pp;
    memset(&pp, 0, sizeof pp);
    pp.fds = reinterpret_cast<const FrameDesc*>(dv);
    pp.rds = reinterpret_cast<const RecDesc*>(dv + b_fd);
    pp.items = reinterpret_cast<const int*>(dv + b_fd + b_rd);
    pp.nitems = int(items.size());
    pp.n = n;
    pp.mb_w = mb_w;
    pp.mb_h = mb_h;
    pp.nbands = nbands;
    pp.nseg = nseg;
    pp.segw = segw;
    pp.nbuf = nbuf;
    pp.pools = pools;
    pp.ew_off = 0;
    pp.dfl_off = 2 * EW_PER_MB * nmb;
    pp.nz_off = pp.dfl_off + nmb;
    pp.band_off = pp.nz_off + nmb;
    pp.fstride = (pp.band_off + (long long)nbands * nseg + 1) & ~1LL;
    const long long head = (2LL * n + 1) & ~1LL;
    const long long need = head + pp.fstride * n;
    if (need >= (1LL << 31)) return fail(H264A_E_ARG, "closed loop: too many macroblocks for one launch");
    rc = ensure_me_scratch(ctx, size_t(need), Q_WIDE);
    if (rc) return rc;
    int* fl = ctx->q[Q_WIDE].d_flags;
    pp.ctr = fl;
    pp.done = fl + n;
    pp.flags = fl + head;
    pp.rec_y = in.rec_y;
    pp.fs = fs;
    pp.planes = in.planes;
    pp.pbytes = pbytes;
    pp.cw = cw;
    pp.ch = ch;
    pp.pad = pad;
    pp.word_in = (cw % 4 == 0) && (pad % 4 == 0) && ((reinterpret_cast<uintptr_t>(in.rec_y) & 3) == 0);
    pp.word_out = (pw % 4 == 0) && ((reinterpret_cast<uintptr_t>(in.planes) & 3) == 0) && (pbytes % 4 == 0);
    pp.frame_words = frame_words;
    pp.ftoken = token;
    pp.arrive = in.arrive;
    pp.atoken = in.atoken;
    // counters zero, and no word of an earlier launch's layout left to be
    // mistaken for a flag of this one
    H264A_CUDA(cudaMemsetAsync(fl, 0, sizeof(int) * size_t(need), st));
    const int epoch = next_epoch(ctx, st, Q_WIDE);
    if (epoch < 0) return H264A_E_CUDA;
    const long long blocks = (long long)ctx->num_sms * pipe_ctas_per_sm(mb_w, mb_h, pools, ctx->num_sms, per_sm);
    auto kern = bal ? (learn ? closed_pipe_kernel<true, true> : closed_pipe_kernel<true, false>)
                    : (learn ? closed_pipe_kernel<false, true> : closed_pipe_kernel<false, false>);
    kern<<<unsigned(blocks), 32 * ME_WARPS, frame_smem(blocks, ctx->num_sms), st>>>(pp, prm, epoch, ctx->d_status, SPIN_LIMIT);
    rc = check_launch("closed_pipe_kernel");
    if (rc) return rc;
    return table_done(ctx, st);
}

// ---------------------------------------------------------------------------
// Plain-ME frames over several reference pictures
// ---------------------------------------------------------------------------
// best_part's loop over references (mb16.rs:4921-4960) in the frame model:
// every search (the 16x16, and the four partitions when its J exceeds the
// gate) runs on each reference r with seeds [predict_mv(a, b, c, r), extra],
// costs plus (lambda * ref_bits(r, nref)) truncated to i64, the strictly
// cheapest kept (references in order).  An MV predicts only from neighbours
// of the same reference (inter.rs:36-69), so a pick carries each half's
// reference index: 8 i32 per MB (shape, ref0, mv0x, mv0y, ref1, mv1x, mv1y,
// 4x4-block evaluations).  One warp per MB, tickets in the frame kernels'
// order, readiness by a flag per MB; the window is staged again for each reference.
constexpr int ME_MAXREF = 4;
struct FrameDescMR {
    CUtensorMap tmap[ME_MAXREF];  // each reference's planes as the window's 3D tensor
    const uint8_t* planes[ME_MAXREF];
    const uint8_t* src;
    double lambda_me;
    long long split_gate;
    int32_t* picks;
    int64_t* costs;
    int nref, cw, ch, pad, mb_w, mb_h, flag_base, tmap_ok;
};

// ref_bits (mb16.rs:5967-5981).
__device__ __forceinline__ uint32_t ref_bits_of(int r, int nref) {
    if (nref <= 1) return 0;
    if (nref == 2) return 1;
    return 1u + 2u * (31u - uint32_t(__clz(r + 1)));
}

// predict_mv (inter.rs:36-69) against reference cur: neighbours with their
// reference indices (available ones are inter, index >= 0).
__device__ __forceinline__ int2 predict_mv_ref(bool aa, int2 a, int ra, bool ba, int2 b, int rb, bool ca, int2 c, int rc,
                                               int cur) {
    int2 mva = aa ? a : make_int2(0, 0), mvb = ba ? b : make_int2(0, 0), mvc = ca ? c : make_int2(0, 0);
    int qa = aa ? ra : -1, qb = ba ? rb : -1, qc = ca ? rc : -1;
    if (!ba && !ca && aa) { mvb = mva; qb = qa; mvc = mva; qc = qa; }
    const int matches = (qa == cur) + (qb == cur) + (qc == cur);
    if (matches == 1) return qa == cur ? mva : (qb == cur ? mvb : mvc);
    auto med = [](int x, int y, int z) { return x + y + z - min(min(x, y), z) - max(max(x, y), z); };
    return make_int2(med(mva.x, mvb.x, mvc.x), med(mva.y, mvb.y, mvc.y));
}

// The MV and reference of neighbour MB `m`'s 4x4 block (bx4, by4).
__device__ __forceinline__ int2 pick_mr_at(const int32_t* picks, int m, int bx4, int by4, int& ref) {
    const int32_t* p = picks + 8 * m;
    const int shape = __ldcg(p);
    const int part = shape == 1 ? (by4 >= 2) : (shape == 2 ? (bx4 >= 2) : 0);
    ref = __ldcg(p + 1 + 3 * part);
    return make_int2(__ldcg(p + 2 + 3 * part), __ldcg(p + 3 + 3 * part));
}

// Launch shapes (the batch runtime's autotuner picks one): NW warps per CTA,
// one MB each (the MBs a CTA holds at once), and STAGE: each search's window
// staged in shared memory by TMA, or every candidate read from L2 through the
// search's global path (no window, no shared memory, the same results).
template <bool BAL, int NW, bool STAGE>
__global__ void __launch_bounds__(32 * NW, (BAL ? 16 : 4 * ME_ANY_BLOCKS) / NW)
    me_frames_mr_kernel(const FrameDescMR* __restrict__ fds, const long long* __restrict__ seg_start,
                        const int* __restrict__ seg_j, int nf, int ns, long long total,
                        const __grid_constant__ MeParamsDev prm, int* __restrict__ counter, int* __restrict__ flags,
                        int epoch, int* __restrict__ status, int spin_limit) {
    __shared__ MbScratch scratch[NW];
    __shared__ __align__(16) SearchScratch scr[NW];
    __shared__ PhaseTab ptab;
    __shared__ __align__(8) unsigned long long win_bar[NW];
    extern __shared__ __align__(128) uint8_t me_win[];
    const int lane = threadIdx.x & 31;
    const WarpWindow ww = warp_window(me_win, win_bar, ptab, scr);
    MbScratch& ws = scratch[threadIdx.x >> 5];
    uint32_t parity = 0;
    for (;;) {
        int t = 0;
        if (lane == 0) t = atomicAdd(counter, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= total) return;
        int sg = 0;
        while (sg + 1 < ns && __ldg(seg_start + sg + 1) <= t) sg++;
        const int j = __ldg(seg_j + sg);
        const long long u = t - __ldg(seg_start + sg);
        const int nxt = j + 1 < nf ? fds[j + 1].mb_w * fds[j + 1].mb_h : 0;
        const FrameDescMR& fd = fds[int(u % (j + 1))];
        const int k = nxt + int(u / (j + 1));
        int mbx, mby;
        wave_mb(fd.mb_w, fd.mb_h, k, mbx, mby);
        const int m = mby * fd.mb_w + mbx;
        int* fl = flags + fd.flag_base;
        const int lx = mbx * 16, ly = mby * 16;
        MbLane s;
        mb_load_src(s, fd.src, fd.cw, lx, ly);
        if (lane == 0) {
            ws.src = fd.src;
            ws.bw = nullptr;
            ws.pw = fd.cw + 2 * fd.pad; ws.ph = fd.ch + 2 * fd.pad;
            ws.pad = fd.pad; ws.cw = fd.cw; ws.ch = fd.ch;
        }
        if (lane == 0) {
            if (mbx > 0) wait_flag(fl + m - 1, epoch, status, 1, spin_limit);
            if (mby > 0) wait_flag(fl + m - fd.mb_w + (mbx < fd.mb_w - 1 ? 1 : 0), epoch, status, 1, spin_limit);
        }
        __syncwarp();
        const bool aa = mbx > 0, ba = mby > 0, ca = mby > 0 && mbx < fd.mb_w - 1, da = mbx > 0 && mby > 0;
        int ra = -1, rb = -1, rc = -1;
        const int2 a = aa ? pick_mr_at(fd.picks, m - 1, 3, 0, ra) : make_int2(0, 0);
        const int2 bb = ba ? pick_mr_at(fd.picks, m - fd.mb_w, 0, 3, rb) : make_int2(0, 0);
        int2 c = make_int2(0, 0);
        if (ca) c = pick_mr_at(fd.picks, m - fd.mb_w + 1, 0, 3, rc);
        else if (da) c = pick_mr_at(fd.picks, m - fd.mb_w - 1, 3, 3, rc);
        const bool cav = ca || da;
        // best_part of the 16x16 over the references, then, J above the gate,
        // of each partition (lane group g = partition g) over the references
        mb_lane_16x16(s, lx, ly, ww.win);
        int evals = 0, shape = 0;
        int ref16 = 0, mv16x = 0, mv16y = 0;
        long long c16 = LLONG_MAX;
        int pref = 0, pmx = 0, pmy = 0;  // the lane's partition's best (mode 1)
        long long pcost = LLONG_MAX;
#pragma unroll 1
        for (int mode = 0; mode < 2; mode++) {
            if (mode == 1) {
                if (!(fd.split_gate >= 0 && c16 > fd.split_gate)) break;
                mb_lane_parts(s);
            }
            for (int r = 0; r < fd.nref; r++) {
                const int2 pmv = predict_mv_ref(aa, a, ra, ba, bb, rb, cav, c, rc, r);
                if (lane == 0) ws.base = fd.planes[r];
                __syncwarp();
                const bool win_ok = STAGE && stage_window(ws, &fd.tmap[r], fd.tmap_ok != 0, true, lx, ly, pmv, ww.win, ww.bar);
                mb_lane_window(s, ws, win_ok);
                if (win_ok) {
                    wait_window(ww.bar, parity, status, 3, spin_limit);
                    parity ^= 1u;
                }
                constexpr int REF = STAGE ? REF_WINDOW : REF_PLANES;
                SearchScratch& bs = scr[threadIdx.x >> 5];
                const int2 mv16 = make_int2(mv16x, mv16y);
                const SearchOut o =
                    mode == 0 ? search16<BAL, false, REF, false>(s, prm, ws, bs, ww.lut, pmv, fd.lambda_me, false, pmv, pmv, 0, nullptr)
                              : search_parts<BAL, false, REF, false>(s, prm, ws, bs, ww.lut, pmv, mv16, fd.lambda_me, false, mv16);
                const long long cst = o.cost + __double2ll_rz(__dmul_rn(fd.lambda_me, double(ref_bits_of(r, fd.nref))));
                if (mode == 0) {
                    evals += o.evals << 4;
                    if (cst < c16) { c16 = cst; ref16 = r; mv16x = o.x; mv16y = o.y; }
                } else {
                    // every lane of group g holds partition g's result
                    evals += (__shfl_sync(0xffffffffu, o.evals, 0) + __shfl_sync(0xffffffffu, o.evals, 8) +
                              __shfl_sync(0xffffffffu, o.evals, 16) + __shfl_sync(0xffffffffu, o.evals, 24)) << 3;
                    if (cst < pcost) { pcost = cst; pref = r; pmx = o.x; pmy = o.y; }
                }
            }
        }
        // the shape decision (mb16.rs:8869-8913)
        int s0r = ref16, s0x = mv16x, s0y = mv16y, s1r = ref16, s1x = mv16x, s1y = mv16y;
        long long best = c16;
        if (fd.split_gate >= 0 && c16 > fd.split_gate) {
            long long pc4[4];
            int pr4[4], px4[4], py4[4];
#pragma unroll
            for (int gi = 0; gi < 4; gi++) {
                pc4[gi] = __shfl_sync(0xffffffffu, pcost, 8 * gi);
                pr4[gi] = __shfl_sync(0xffffffffu, pref, 8 * gi);
                px4[gi] = __shfl_sync(0xffffffffu, pmx, 8 * gi);
                py4[gi] = __shfl_sync(0xffffffffu, pmy, 8 * gi);
            }
            if (pc4[0] + pc4[1] < best) {
                best = pc4[0] + pc4[1]; shape = 1;
                s0r = pr4[0]; s0x = px4[0]; s0y = py4[0]; s1r = pr4[1]; s1x = px4[1]; s1y = py4[1];
            }
            if (pc4[2] + pc4[3] < best) {
                best = pc4[2] + pc4[3]; shape = 2;
                s0r = pr4[2]; s0x = px4[2]; s0y = py4[2]; s1r = pr4[3]; s1x = px4[3]; s1y = py4[3];
            }
        }
        if (lane == 0) {
            int32_t* p = fd.picks + 8 * m;
            p[0] = shape; p[1] = s0r; p[2] = s0x; p[3] = s0y; p[4] = s1r; p[5] = s1x; p[6] = s1y; p[7] = evals;
            fd.costs[2 * m] = best;
            fd.costs[2 * m + 1] = c16;
            st_release(fl + m, epoch);  // orders the pick's stores before the flag
        }
        __syncwarp();
    }
}

// The launch shapes, variant 0 the default of h264a_me_frames_multiref.
struct MrShape {
    int nw;
    bool stage;
};
constexpr MrShape kMrShapes[H264A_BATCH_VARIANTS] = {{4, true}, {2, true}, {8, true}, {4, false}, {2, false}, {8, false}};

template <bool BAL, int NW, bool STAGE>
static int mr_attr() {
    if (STAGE)
        H264A_CUDA(cudaFuncSetAttribute(me_frames_mr_kernel<BAL, NW, STAGE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        NW * WIN_BYTES));
    return H264A_OK;
}

static int me_mr_setup_once() {
    int rc = mr_attr<false, 4, true>();
    if (!rc) rc = mr_attr<true, 4, true>();
    if (!rc) rc = mr_attr<true, 2, true>();
    if (!rc) rc = mr_attr<true, 8, true>();
    return rc;
}
// Once per device, as me_frames_setup.
static int me_mr_setup() {
    constexpr int kMaxDev = 64;
    static bool done[kMaxDev];
    static std::mutex mu;
    int dev = 0;
    H264A_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDev) return me_mr_setup_once();
    std::lock_guard<std::mutex> lock(mu);
    if (!done[dev]) {
        const int rc = me_mr_setup_once();
        if (rc) return rc;
        done[dev] = true;
    }
    return H264A_OK;
}

template <bool BAL, int NW, bool STAGE>
static int mr_launch_t(h264a_ctx* ctx, const MeParamsDev& prm, const char* dv, const MrTable& t, int32_t* counter,
                       int32_t* flags, int epoch, cudaStream_t st) {
    const size_t sm = STAGE ? size_t(NW) * WIN_BYTES : 0;
    int per_sm = 0;
    H264A_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, me_frames_mr_kernel<BAL, NW, STAGE>, 32 * NW, sm));
    if (per_sm < 1) per_sm = 1;
    long long blocks = (long long)ctx->num_sms * per_sm;
    const long long need = (t.total + NW - 1) / NW;
    if (blocks > need) blocks = need;
    me_frames_mr_kernel<BAL, NW, STAGE><<<unsigned(blocks), 32 * NW, sm, st>>>(
        reinterpret_cast<const FrameDescMR*>(dv), reinterpret_cast<const long long*>(dv + t.b_desc),
        reinterpret_cast<const int*>(dv + t.b_desc + t.b_seg), t.nframes, t.nseg, t.total, prm, counter, flags, epoch,
        ctx->d_status, SPIN_LIMIT);
    return check_launch("me_frames_mr_kernel");
}

int h264a::mr_table_build(const h264a_me_mr_frame* h_frames, int nframes, MrTable& t) {
    if (!h_frames) return fail(H264A_E_ARG, "me_frames_multiref: null pointer");
    if (nframes < 1) return fail(H264A_E_ARG, "me_frames_multiref: need at least one frame");
    for (int i = 0; i < nframes; i++) {
        const h264a_me_mr_frame& f = h_frames[i];
        if (f.nref < 1 || f.nref > ME_MAXREF) return fail(H264A_E_ARG, "me_frames_multiref: 1 to 4 references per frame");
        if (!f.d_src || !f.d_picks || !f.d_costs) return fail(H264A_E_ARG, "me_frames_multiref: null frame pointer");
        if (reinterpret_cast<uintptr_t>(f.d_src) & 3) return fail(H264A_E_ARG, "me_frames_multiref: sources must be 4-byte aligned");
        for (int r = 0; r < f.nref; r++)
            if (!f.d_planes[r]) return fail(H264A_E_ARG, "me_frames_multiref: null reference planes");
        if (f.cw < 16 || f.ch < 16 || f.cw % 16 || f.ch % 16 || f.pad < 3 || f.pad > 128)
            return fail(H264A_E_ARG, "me_frames_multiref: frames must be MB-aligned with 3 <= pad <= 128");
        if ((long long)(f.cw / 16) * (f.ch / 16) > (1 << 24)) return fail(H264A_E_ARG, "me_frames_multiref: frame too large");
    }
    std::vector<int> order(nframes);
    for (int i = 0; i < nframes; i++) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        return (long long)h_frames[a].cw * h_frames[a].ch > (long long)h_frames[b].cw * h_frames[b].ch;
    });
    std::vector<FrameDescMR> desc(nframes);
    memset(desc.data(), 0, sizeof(FrameDescMR) * nframes);
    std::vector<FrameDesc> segd(nframes);  // the sizes, for the queue's segments
    memset(segd.data(), 0, sizeof(FrameDesc) * nframes);
    long long total = 0;
    for (int k = 0; k < nframes; k++) {
        const h264a_me_mr_frame& f = h_frames[order[k]];
        FrameDescMR& d = desc[k];
        const int pw = f.cw + 2 * f.pad, ph = f.ch + 2 * f.pad;
        d.tmap_ok = 1;
        for (int r = 0; r < f.nref; r++) {
            d.planes[r] = f.d_planes[r];
            d.tmap_ok &= encode_window_map(&d.tmap[r], f.d_planes[r], pw, ph);
        }
        d.src = f.d_src;
        d.lambda_me = f.lambda_me;
        d.split_gate = f.split_gate;
        d.picks = f.d_picks;
        d.costs = f.d_costs;
        d.nref = f.nref;
        d.cw = f.cw; d.ch = f.ch; d.pad = f.pad;
        d.mb_w = f.cw / 16;
        d.mb_h = f.ch / 16;
        d.flag_base = int(total);
        t.lam_ok = t.lam_ok && balanced_lambda(f.lambda_me);
        segd[k].mb_w = d.mb_w;
        segd[k].mb_h = d.mb_h;
        total += (long long)d.mb_w * d.mb_h;
        if (total >= (1LL << 31)) return fail(H264A_E_ARG, "me_frames_multiref: too many macroblocks in one call");
    }
    std::vector<long long> seg(nframes + 1);
    std::vector<int> segj(nframes);
    const int nseg = make_segments(segd.data(), nframes, seg.data(), segj.data());
    if (seg[nseg] != total) return fail(H264A_E_ARG, "me_frames_multiref: internal queue layout error");
    t.nframes = nframes;
    t.nseg = nseg;
    t.total = total;
    t.b_desc = sizeof(FrameDescMR) * nframes;
    t.b_seg = sizeof(long long) * (nseg + 1);
    const size_t b_j = sizeof(int) * nseg;
    t.bytes.assign(t.b_desc + t.b_seg + b_j, 0);
    memcpy(t.bytes.data(), desc.data(), t.b_desc);
    memcpy(t.bytes.data() + t.b_desc, seg.data(), t.b_seg);
    memcpy(t.bytes.data() + t.b_desc + t.b_seg, segj.data(), b_j);
    return H264A_OK;
}

int h264a::mr_launch(h264a_ctx* ctx, int variant, const MeParamsDev& prm, const void* d_table, const MrTable& t,
                     int32_t* counter, int32_t* flags, int epoch, cudaStream_t st) {
    if (variant < 0 || variant >= H264A_BATCH_VARIANTS) return fail(H264A_E_ARG, "me_frames_multiref: no such launch shape");
    const int rc = me_mr_setup();
    if (rc) return rc;
    const char* dv = static_cast<const char*>(d_table);
    if (!balanced_preset(prm, t.lam_ok)) return mr_launch_t<false, 4, true>(ctx, prm, dv, t, counter, flags, epoch, st);
    switch (variant) {
        case 1: return mr_launch_t<true, 2, true>(ctx, prm, dv, t, counter, flags, epoch, st);
        case 2: return mr_launch_t<true, 8, true>(ctx, prm, dv, t, counter, flags, epoch, st);
        case 3: return mr_launch_t<true, 4, false>(ctx, prm, dv, t, counter, flags, epoch, st);
        case 4: return mr_launch_t<true, 2, false>(ctx, prm, dv, t, counter, flags, epoch, st);
        case 5: return mr_launch_t<true, 8, false>(ctx, prm, dv, t, counter, flags, epoch, st);
        default: return mr_launch_t<true, 4, true>(ctx, prm, dv, t, counter, flags, epoch, st);
    }
}

extern "C" int h264a_batch_variant_shape(int variant, int* mbs_per_cta, int* staged) {
    if (variant < 0 || variant >= H264A_BATCH_VARIANTS) return fail(H264A_E_ARG, "batch_variant_shape: no such variant");
    if (mbs_per_cta) *mbs_per_cta = kMrShapes[variant].nw;
    if (staged) *staged = kMrShapes[variant].stage ? 1 : 0;
    return H264A_OK;
}

extern "C" int h264a_me_frames_multiref(h264a_ctx* ctx, const h264a_me_mr_frame* h_frames, int nframes,
                                        const h264a_me_params* params, void* stream) {
    if (!ctx || !h_frames || !params) return fail(H264A_E_ARG, "me_frames_multiref: null pointer");
    if ((params->mv_cost_kind == 1 || params->mv_cost_kind == 2) && !params->d_mv_cost_tab)
        return fail(H264A_E_ARG, "me_frames_multiref: mv cost kinds 1 and 2 need d_mv_cost_tab");
    MrTable t;
    int rc = mr_table_build(h_frames, nframes, t);
    if (rc) return rc;
    cudaStream_t st = pick_stream(ctx, stream);
    const MeParamsDev prm = to_dev(*params);
    char* hst = nullptr;
    rc = table_host(ctx, t.bytes.size(), &hst);
    if (rc) return rc;
    memcpy(hst, t.bytes.data(), t.bytes.size());
    rc = table_upload(ctx, t.bytes.size(), st);
    if (rc) return rc;
    rc = ensure_me_scratch(ctx, size_t(t.total));
    if (rc) return rc;
    H264A_CUDA(cudaMemsetAsync(ctx->q[Q_MAIN].d_counter, 0, sizeof(int32_t), st));
    const int epoch = next_epoch(ctx, st);
    if (epoch < 0) return H264A_E_CUDA;
    rc = mr_launch(ctx, 0, prm, ctx->me_tab, t, ctx->q[Q_MAIN].d_counter, ctx->q[Q_MAIN].d_flags, epoch, st);
    if (rc) return rc;
    return table_done(ctx, st);
}

// density_stream.cuh — the FP32C density of a particle system, over work items
// of up to 32 i-particles.
//
// One warp streams its item's whole list; entries inside the list radius go
// to per-lane neighbour lists that the later passes read.  Items with longer
// lists are set apart for the LONG form, in which a block streams one item: same
// ring order, same tiles, same folds, so the same results bit for bit, with
// the loads, support tests and tiles of a round spread over its warps.
//
// Bound: latency of the streaming and of the listed gathers, and the last
// items: at 200k the SMs were active for 41% of this kernel and 56% of the LONG
// one until the long items came from a queue, longest first, beside the
// others (1.6 -> 0.9 ms for both).
//
// The rows kernels (density_rows.cuh) serve the FP64 density, the functors and
// the re-walks of few particles.  They are not used here: the hydro sums
// amplify a change of rounding in h and rho by up to 10^3, and the h of a few
// surface particles by more from evaluation to evaluation, so that runs would
// leave the trajectories they had before.
#pragma once

#include "density_rows.cuh"

#ifndef SPH_DENSITY_MIN_BLOCKS
#define SPH_DENSITY_MIN_BLOCKS 4
#endif
#ifndef SPH_DENSITY_UNROLL
#define SPH_DENSITY_UNROLL 4
#endif

namespace sphk {

// f32x2 iterations (two entries each) of the packed loop per unrolled round
constexpr int DENSITY_UNROLL = SPH_DENSITY_UNROLL;
constexpr int STREAM_LONG_WARPS = 8;

struct StreamArgs {
    const dbl4 *i_pm;       // x, y, z, mass
    F32Part fi, fj;         // double-float records (phi.w = mass)
    const long long *i_id;
    const long long *j_id;
    const double *i_ksr;    // first guess of h (DensityEPI::ksr)
    const double *i_rs;     // search radius (DensityEPI::rs)
    // work
    const WorkItem *items;
    int n_items;
    const int *n_items_dev; // when set, the item count is read from device memory
    const int *j_off;       // per walk: [j_off[w], j_off[w+1]) in j index space
    const int *j_idx;       // null: entries are j indices themselves
    const int *i_list;      // null: item i-particles are contiguous
    int *queue;             // item counter, 0 at launch
    // outputs, indexed like the i arrays
    double *o_dens, *o_divv, *o_rotv, *o_grdh, *o_ksr;
    long long *o_np;
    unsigned char *o_itr;
    double eta_ksrh;        // eta * ksrh
    double ksr_max;         // clamp of h (+inf disables)
    const double *ksr_max_dev;  // when set, the clamp is read from device memory
    // particles whose final h lies within amb_tol of rs (where
    // the search-radius decision h > rs of hdr_density.hpp:299 could come out
    // differently in FP64) are queued here for an FP64 recomputation
    int *amb_count;         // null disables the queue
    int2 *amb;              // (particle, walk)
    int amb_cap;
    float amb_tol;
    // Per-warp neighbour lists; null: every pass sweeps the walk's j-list.
    // Warp w of the grid (blockIdx.x * WARPS + warp) owns the int array
    // nbr[w * nbr_cap * 32, (w + 1) * nbr_cap * 32), entry c of lane l at
    // [c * 32 + l]; warps w >= nbr_warps sweep.  nbr_slack (> 1) is the list
    // radius in units of each i-particle's first-pass h.
    int *nbr = nullptr;
    int nbr_cap = 0;
    int nbr_warps = 0;
    float nbr_slack = 1.0f;
    LongQueue longs;        // items of the LONG form
    // when set: pair evaluations performed, [0] the three density passes
    // ((j-entries kept by the support test x i-particles) of the swept passes
    // plus the list entries of the listed ones), [1] the gradient pass
    unsigned long long *n_eval = nullptr;
    // when set: [0] item passes (second, third, gradient) served from the
    // neighbour lists, [1] item passes that swept the walk's j-list
    unsigned long long *n_pass = nullptr;
};

// The particles without a row, walk by walk in items of 32 (one warp per
// walk): their indices to `list`, which holds every walk's at its own offset.
// Nothing while no more than `most` (*n_rowless) are without.
__global__ inline void __launch_bounds__(128)
rowless_items(int n_walk, const int *i_off, const int *j_off, const int2 *info, const int *n_rowless, int most,
              int *list, WorkItem *items, int *n_items) {
    if (*n_rowless <= most) return;
    const int lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5;
    for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < n_walk; w += nw) {
        const int b = i_off[w], e = i_off[w + 1];
        int n = 0;
        for (int k = b; k < e; k += 32) {
            const bool out = k + lane < e && info[k + lane].x > ROW_CAP;
            const unsigned m = __ballot_sync(FULL, out);
            if (out) list[b + n + __popc(m & lanemask_lt())] = k + lane;
            n += __popc(m);
        }
        const int c = (n + 31) / 32;
        int pos = 0;
        if (lane == 0 && c > 0) pos = atomicAdd(n_items, c);
        pos = __shfl_sync(FULL, pos, 0);
        for (int q = lane; q < c; q += 32)
            items[pos + q] = make_int4(w, b + 32 * q, min(32, n - 32 * q), 0);
    }
}

template <bool B>
struct BTag {
    static constexpr bool value = B;
};

// The density functor of hdr_density.hpp:252-350 for one work item per warp:
// three fixed-point passes rho(h) -> h = eta ksrh (m / rho)^(1/3) from the
// first guess, then the gradient pass (grdh, divv, rotv) with the final h.
//
// Every pass can stream the walk's j-list through a shared ring (kept entries
// of each 32-entry chunk compacted by the item-box support test), which
// evaluates every kept entry for every i-particle of the item: ~10x more
// pairs than the kernel support holds.  With neighbour lists the first pass
// streams the list once with the support widened by nbr_slack and also writes,
// per lane, the j indices within nbr_slack * (first-pass h) of its
// i-particle; the second and third passes and the gradient pass then loop over
// each lane's own list (gathering the j records) whenever every h of the item
// has stayed within that radius and no lane's list overflowed nbr_cap;
// otherwise the pass sweeps.  Entries beyond a particle's support add exactly
// zero in both forms, so the two differ only in the grouping of the FP32
// partial sums.
//
// LONG: a block takes an item of the long-item queue.  Its warps hold the same
// lanes; a round of 32 WARPS U list entries is loaded and tested by all of
// them, compacted in list order, cut into 32-entry tiles that the warps sum
// one each, and every warp folds the tiles' partial sums in order.
template <int WARPS, bool LONG = false>
__global__ void __launch_bounds__(WARPS * 32, LONG ? 2 : SPH_DENSITY_MIN_BLOCKS) density_stream(const StreamArgs a) {
    // LONG: the compacted entries (< 32 left over + a round) and the tiles'
    // partial sums (1 or 5 per lane; the list-building pass keeps its marks in
    // the second slot)
    constexpr int U = 4, ROUND = 32 * U * WARPS, LBUF = LONG ? ROUND + 32 : 1, LT = LONG ? LBUF / 32 : 1;
    __shared__ __align__(16) float l_x[LBUF], l_y[LBUF], l_z[LBUF], l_m[LBUF];
    __shared__ int l_j[LBUF];
    __shared__ float l_part[LT][5][32];
    __shared__ int l_cnt[LONG ? WARPS : 1];
    __shared__ unsigned l_any[LT];
    constexpr int RW = LONG ? 1 : WARPS, RN = LONG ? 1 : 64;   // the per-warp ring
    // per warp a 64-entry ring of compacted j records: entries accumulate
    // until 32 are ready, the pair loop consumes one 32-entry half at a time
    __shared__ float4 s_p[RW][RN];
    __shared__ float4 s_v[RW][RN];
    __shared__ float2 s_vl[RW][RN];
    __shared__ long long s_id[RW][RN];
    // density passes: the same ring as a structure of arrays, so that
    // two consecutive entries load as one f32x2 operand
    __shared__ __align__(16) float s_rx[RW][RN], s_ry[RW][RN], s_rz[RW][RN], s_rm[RW][RN];
    __shared__ int s_j[RW][RN];   // j index of each ring entry (list-building pass)
    const int lane = threadIdx.x & 31;
    const int wid = threadIdx.x >> 5;
    const unsigned lt = lanemask_lt();
    __shared__ int s_next;   // LONG
    const int n_items = LONG ? 0 : (a.n_items_dev ? *a.n_items_dev : a.n_items);
    const double ksr_max = a.ksr_max_dev ? *a.ksr_max_dev : a.ksr_max;
    // (LONG: the last gridDim.x slots, one per block)
    const int gw = LONG ? a.nbr_warps - gridDim.x + blockIdx.x : blockIdx.x * WARPS + wid;
    // the ring (LONG: the compacted entries)
    const float *bx = LONG ? l_x : s_rx[LONG ? 0 : wid], *by = LONG ? l_y : s_ry[LONG ? 0 : wid];
    const float *bz = LONG ? l_z : s_rz[LONG ? 0 : wid], *bm = LONG ? l_m : s_rm[LONG ? 0 : wid];
    const int *bj = LONG ? l_j : s_j[LONG ? 0 : wid];
    // this lane's neighbour list: entry c at a.nbr[nlb + c * 32]
    const bool has_nl = a.nbr != nullptr && gw < a.nbr_warps;
    const int nlb = has_nl ? gw * a.nbr_cap * 32 + lane : 0;
    // list radius^2 over (first-pass h)^2, and the largest h (over the
    // first-pass h) a listed pass accepts: every pair with q < 1 then has r^2
    // below the list radius with a margin of 2e-5 over the rounding of both
    // tests
    const float nl_lim = (float)a.nbr_slack * (float)a.nbr_slack;
    const double nl_hmax = (double)a.nbr_slack * 0.99998;

    for (;;) {
        WorkItem wi;
        if (LONG) {
            if (!a.longs.take(&s_next, wi)) return;
        } else {
            int item = 0;
            if (lane == 0) item = atomicAdd(a.queue, 1);
            item = __shfl_sync(FULL, item, 0);
            if (item >= n_items) return;
            wi = a.items[item];
        }
        const ItemRef r = decode(wi, a.j_off, a.i_list, lane);
        const int tpi = r.tpi, sub = r.sub, ii = r.ii, nj = r.nj, jb = r.jb;

        // i-particle relative to the centre particle c (velocity, id, mass
        // and search radius are read where they are used, keeping the
        // registers of the passes free)
        const float4 cph = a.fi.phi[r.ic], cpl = a.fi.plo[r.ic];
        float xi, yi, zi;
        {
            const float4 ph = a.fi.phi[ii], pl = a.fi.plo[ii];
            xi = df_diff(ph.x, pl.x, cph.x, cpl.x);
            yi = df_diff(ph.y, pl.y, cph.y, cpl.y);
            zi = df_diff(ph.z, pl.z, cph.z, cpl.z);
        }
        // The kernel is zero for r >= h, so a j-particle farther than the
        // largest h of the item from the item's box adds nothing to any sum
        // or count of this item: staging drops it before the pair loop.
        IBox<float> box;
        box.from_lanes(xi, yi, zi);
        double h = a.i_ksr[ii];
        // largest h a listed pass accepts for this lane
        const float nl_h = (float)(h * nl_hmax);
        float rho = 0;
        int np = 0;

        // One j record as loaded from memory.
        struct JRec {
            float4 ph, pl, vh, vl;
            long long id;
        };
        auto jlist = [&](int k) -> int { return a.j_idx ? a.j_idx[jb + k] : jb + k; };
        auto load = [&](int j, bool with_v, JRec &q) {
            q.ph = a.fj.phi[j];
            q.pl = a.fj.plo[j];
            if (with_v) {
                q.vh = a.fj.vhi[j];
                q.vl = a.fj.vlo[j];
                q.id = a.j_id[j];
            }
        };
        // position of particle j relative to the centre particle and its mass
        auto jpos = [&](int j) -> float4 {
            const float4 ph = __ldg(&a.fj.phi[j]), pl = __ldg(&a.fj.plo[j]);
            return make_float4(df_diff(ph.x, pl.x, cph.x, cpl.x), df_diff(ph.y, pl.y, cph.y, cpl.y),
                               df_diff(ph.z, pl.z, cph.z, cpl.z), ph.w);
        };
        // Streams the walk's list through the ring: lane k takes entry t+k,
        // entries that can lie within sqrt(rf2) of the item box are
        // compacted into the ring, and consume(base, n) runs whenever 32 are
        // ready (and once more for the rest).  Loads run one 32-entry chunk
        // ahead of their use (the list index two chunks ahead) so that their
        // latency overlaps the box test and the pair loops.  with_v also
        // stages velocities and ids (gradient pass), with_j the j indices.
        unsigned kept = 0;   // j-entries kept by the support test, all sweeps
        auto sweep = [&](const float rf2, const bool with_v, const bool with_j, auto &&consume) {
            int head = 0, fill = 0;
            JRec cur, nxt;
            int jn = 0, jnx = 0;
            if (lane < nj) {
                jnx = jlist(lane);
                load(jnx, with_v, nxt);
            }
            if (32 + lane < nj) jn = jlist(32 + lane);
            for (int t = 0; t < nj; t += 32) {
                cur = nxt;
                const int jc = jnx;
                const bool valid = t + lane < nj;
                if (t + 32 + lane < nj) {
                    jnx = jn;
                    load(jn, with_v, nxt);
                }
                if (t + 64 + lane < nj) jn = jlist(t + 64 + lane);
                bool keep = false;
                float4 p4;
                if (valid) {
                    p4 = make_float4(df_diff(cur.ph.x, cur.pl.x, cph.x, cpl.x),
                                     df_diff(cur.ph.y, cur.pl.y, cph.y, cpl.y),
                                     df_diff(cur.ph.z, cur.pl.z, cph.z, cpl.z), cur.ph.w);
                    keep = !(box.d2(p4.x, p4.y, p4.z) > rf2);
                }
                const unsigned m = __ballot_sync(FULL, keep);
                if (keep) {
                    const int slot = (head + fill + __popc(m & lt)) & 63;
                    if (!with_v) {
                        s_rx[LONG ? 0 : wid][slot] = p4.x;
                        s_ry[LONG ? 0 : wid][slot] = p4.y;
                        s_rz[LONG ? 0 : wid][slot] = p4.z;
                        s_rm[LONG ? 0 : wid][slot] = p4.w;
                    } else {
                        s_p[wid][slot] = p4;
                    }
                    if (with_v) {
                        s_v[wid][slot] = make_float4(cur.vh.x, cur.vh.y, cur.vh.z, cur.vl.x);
                        s_vl[wid][slot] = make_float2(cur.vl.y, cur.vl.z);
                        s_id[wid][slot] = cur.id;
                    }
                    if (with_j) s_j[wid][slot] = jc;
                }
                fill += __popc(m);
                kept += __popc(m);
                __syncwarp();
                if (fill >= 32) {
                    consume(head, 32);
                    head ^= 32;
                    fill -= 32;
                }
            }
            if (fill > 0) consume(head, fill);
        };

        // The LONG sweep: tile(head, n, out) sums the compacted entries
        // [head, head + n) for this lane into out[0..NV); fold(t, head) adds the
        // NV sums of tile t.  A run of tiles without any sum folds one zero
        // (further zeros leave a compensated sum as it is).
        auto sweep_long = [&](const float rf2, auto &&tile, auto &&fold) {
            int fill = 0;
            bool zero = false;
            int jn[U];   // the next round's list entries
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int k = 32 * (U * wid + u) + lane;
                jn[u] = (k < nj) ? jlist(k) : -1;
            }
            for (int t = 0; t < nj; t += ROUND) {
                float4 p4[U], lo[U];
                int jc[U];
                unsigned m[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    jc[u] = jn[u];
                    if (jc[u] >= 0) {
                        p4[u] = a.fj.phi[jc[u]];
                        lo[u] = a.fj.plo[jc[u]];
                    }
                    const int k = t + ROUND + 32 * (U * wid + u) + lane;
                    jn[u] = (k < nj) ? jlist(k) : -1;
                }
                int mine = 0;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    bool keep = false;
                    if (jc[u] >= 0) {
                        p4[u] = make_float4(df_diff(p4[u].x, lo[u].x, cph.x, cpl.x),
                                            df_diff(p4[u].y, lo[u].y, cph.y, cpl.y),
                                            df_diff(p4[u].z, lo[u].z, cph.z, cpl.z), p4[u].w);
                        keep = !(box.d2(p4[u].x, p4[u].y, p4[u].z) > rf2);
                    }
                    m[u] = __ballot_sync(FULL, keep);
                    mine += __popc(m[u]);
                }
                if (lane == 0) l_cnt[wid] = mine;
                __syncthreads();   // counts; the last round's tiles are folded
                int pos = fill, total = 0;
                for (int w = 0; w < WARPS; ++w) {
                    const int c = l_cnt[w];
                    if (w < wid) pos += c;
                    total += c;
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (m[u] >> lane & 1u) {
                        const int q = pos + __popc(m[u] & lt);
                        l_x[q] = p4[u].x;
                        l_y[q] = p4[u].y;
                        l_z[q] = p4[u].z;
                        l_m[q] = p4[u].w;
                        l_j[q] = jc[u];
                    }
                    pos += __popc(m[u]);
                }
                fill += total;
                kept += total;
                __syncthreads();   // entries
                const int nt = fill >> 5;
                for (int q = wid; q < nt; q += WARPS) {
                    const bool any = tile(32 * q, 32, q);
                    if (lane == 0) l_any[q] = any ? 1u : 0u;
                }
                __syncthreads();   // tiles
                for (int q = 0; q < nt; ++q) {
                    const bool any = l_any[q] != 0u;
                    if (any || !zero) fold(q, 32 * q);
                    zero = !any;
                }
                // the entries left over move to the front (one warp)
                if (wid == 0 && nt > 0) {
                    const int q = 32 * nt + lane;
                    const bool mv = q < fill;
                    const float x = mv ? l_x[q] : 0.0f, y = mv ? l_y[q] : 0.0f, z = mv ? l_z[q] : 0.0f;
                    const float w = mv ? l_m[q] : 0.0f;
                    const int j = mv ? l_j[q] : 0;
                    __syncwarp();
                    if (mv) {
                        l_x[lane] = x; l_y[lane] = y; l_z[lane] = z; l_m[lane] = w; l_j[lane] = j;
                    }
                }
                fill &= 31;
            }
            __syncthreads();   // the last round's folds and move
            if (fill > 0) {
                if (wid == 0) tile(0, fill, 0);
                __syncthreads();
                fold(0, 0);
                __syncthreads();
            }
        };

        // neighbour list of this lane: its length (above nbr_cap the list is
        // unusable), appended by the first pass from the ring
        int ncnt = 0;
        bool nl_ok = false;
        unsigned ev_list = 0, ev_list_g = 0;   // list entries evaluated (this lane)
        int n_listed = 0;                      // of the 3 item passes after the first
        auto nl_push = [&](int head, unsigned msk) {
            while (msk) {
                const int k = __ffs(msk) - 1;
                msk &= msk - 1;
                if (ncnt < a.nbr_cap && (!LONG || wid == 0)) a.nbr[nlb + ncnt * 32] = bj[head + k];
                ++ncnt;
            }
        };

        // three fixed-point passes, hdr_density.hpp:264-302
        for (int pass = 0; pass < 3; ++pass) {
            const float hinv = (float)1 / (float)h;
            const float hinv2 = hinv * hinv;
            const bool build = has_nl && pass == 0;
            const bool listed = pass > 0 && nl_ok && __all_sync(FULL, (float)h <= nl_h);
            Acc<false> acc;
            int cnt = 0;
            float part = 0;
            // rho pair term m_j W0(q)/c0; neighbour count only in the last
            // pass (the only np the reference stores, :297)
            auto term = [&](const float4 pj, bool count) -> float {
                const float dx = xi - pj.x, dy = yi - pj.y, dz = zi - pj.z;
                const float r2 = dx * dx + dy * dy + dz * dz;
                const float q = sqrt_q(r2, hinv2);
                const float u = max0((float)1 - q);
                const float u2 = u * u;
                if (count) cnt += (q < (float)1) ? 1 : 0;
                return pj.w * (u2 * u2 * ((float)1 + (float)4 * q));
            };
            // ring entry k; with mark set, bit k of *mark flags an entry
            // within the list radius
            auto pair = [&](int k, bool count, unsigned *mark) {
                const float4 pj = make_float4(bx[k], by[k], bz[k], bm[k]);
                part += term(pj, count);
                if (mark) {
                    const float dx = xi - pj.x, dy = yi - pj.y, dz = zi - pj.z;
                    if ((dx * dx + dy * dy + dz * dz) * hinv2 < nl_lim) *mark |= 1u << (k & 31);
                }
            };
            // full FP32C tile: two entries per instruction (f32x2); even and
            // odd entries summed apart and combined at the end of the tile;
            // the list-building form also flags the entries within the list
            // radius
            auto run_packed = [&](int head, bool count, auto build_tag) {
                constexpr bool B = decltype(build_tag)::value;
                const f2 XI = f2_make((float)xi, (float)xi), YI = f2_make((float)yi, (float)yi);
                const f2 ZI = f2_make((float)zi, (float)zi), H2 = f2_make((float)hinv2, (float)hinv2);
                const f2 NEG = f2_make(-1.0f, -1.0f), ONE = f2_make(1.0f, 1.0f), FOUR = f2_make(4.0f, 4.0f);
                const float lim = (float)nl_lim;
                f2 PART = f2_make(0.0f, 0.0f);
                int c2 = 0;
                unsigned msk = 0;
#pragma unroll DENSITY_UNROLL
                for (int k = 0; k < 32; k += 2) {
                    const f2 DX = f2_fma(f2_lds(&bx[head + k]), NEG, XI);
                    const f2 DY = f2_fma(f2_lds(&by[head + k]), NEG, YI);
                    const f2 DZ = f2_fma(f2_lds(&bz[head + k]), NEG, ZI);
                    const float2 x2 = f2_get(f2_mul(f2_fma(DZ, DZ, f2_fma(DY, DY, f2_mul(DX, DX))), H2));
                    if constexpr (B) msk |= (x2.x < lim ? 1u << k : 0u) | (x2.y < lim ? 2u << k : 0u);
                    float q0, q1;
                    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(q0) : "f"(x2.x));
                    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(q1) : "f"(x2.y));
                    const f2 Q = f2_make(q0, q1);
                    const float2 u = f2_get(f2_fma(Q, NEG, ONE));
                    const f2 U = f2_make(max0(u.x), max0(u.y));
                    const f2 U2 = f2_mul(U, U);
                    PART = f2_fma(f2_lds(&bm[head + k]), f2_mul(f2_mul(U2, U2), f2_fma(Q, FOUR, ONE)), PART);
                    if (count) c2 += (q0 < 1.0f ? 1 : 0) + (q1 < 1.0f ? 1 : 0);
                }
                const float2 ps = f2_get(PART);
                part = (float)(ps.x + ps.y);
                cnt += c2;
                return msk;
            };
            // sum of one tile in part, and its marks
            auto tile = [&](int head, int n) -> unsigned {
                part = 0;
                unsigned msk = 0;
                if (tpi == 1 && n == 32) {
                    if (build)
                        msk = run_packed(head, false, BTag<true>());
                    else
                        run_packed(head, pass == 2, BTag<false>());
                } else {
                    unsigned *mark = build ? &msk : nullptr;
                    for (int k = sub; k < n; k += tpi) pair(head + k, pass == 2, mark);
                }
                return msk;
            };
            auto run = [&](int head, int n) {
                const unsigned msk = tile(head, n);
                if (build) nl_push(head, msk);
                acc.add(part);
                __syncwarp();
            };
            if (listed) {
                // this lane's list, four entries per round (gathers first);
                // LONG: a round each for the warps, folded in order
                const int cmax = (int)__reduce_max_sync(FULL, (unsigned)ncnt);
                auto round4 = [&](int c0) {
                    int jj[4];
                    float4 pj[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) jj[u] = (c0 + u < ncnt) ? a.nbr[nlb + (c0 + u) * 32] : -1;
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (jj[u] >= 0) pj[u] = jpos(jj[u]);
                    part = 0;
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (jj[u] >= 0) part += term(pj[u], pass == 2);
                };
                if constexpr (LONG) {
                    for (int b0 = 0; b0 < cmax; b0 += 4 * LT) {
                        const int nq = min(LT, (cmax - b0 + 3) >> 2);
                        for (int q = wid; q < nq; q += WARPS) {
                            round4(b0 + 4 * q);
                            l_part[q][0][lane] = part;
                        }
                        __syncthreads();
                        for (int q = 0; q < nq; ++q) acc.add(l_part[q][0][lane]);
                        __syncthreads();
                    }
                } else {
                    for (int c0 = 0; c0 < cmax; c0 += 4) {
                        round4(c0);
                        acc.add(part);
                    }
                }
                if (r.act) ev_list += (unsigned)ncnt;
                ++n_listed;
            } else {
                const float rf2 = support2<float>(build ? h * (double)a.nbr_slack : h);
                if constexpr (LONG) {
                    sweep_long(rf2,
                               [&](int head, int n, int q) {
                                   const unsigned msk = tile(head, n);
                                   l_part[q][0][lane] = part;
                                   if (build) l_part[q][1][lane] = __uint_as_float(msk);
                                   return __any_sync(FULL, part != 0.0f || msk != 0u);
                               },
                               [&](int q, int head) {
                                   if (build) nl_push(head, __float_as_uint(l_part[q][1][lane]));
                                   acc.add(l_part[q][0][lane]);
                               });
                } else {
                    sweep(rf2, false, build, run);
                }
            }
            if (LONG && pass == 2) {
                // the warps' counts
                int *sum = reinterpret_cast<int *>(&l_part[0][0][0]);
                __syncthreads();
                if (wid == 0) sum[lane] = 0;
                __syncthreads();
                atomicAdd(&sum[lane], cnt);
                __syncthreads();
                cnt = sum[lane];
                __syncthreads();
            }
            if (LONG && build) __syncthreads();   // the lists
            if (build) nl_ok = __all_sync(FULL, ncnt <= a.nbr_cap);
            const double sum = seg_sum(acc.value(), tpi);
            const int c = (int)seg_sum((long long)cnt, tpi);
            const double mi = a.i_pm[ii].w;
            // FP32 per-particle update (relative error ~1e-7, far inside
            // the 1e-5 budget) keeps the FP64 pipe out of the loop
            const float hinv_f = (float)hinv;
            const float rho_f = (float)CEFF0 * hinv_f * hinv_f * hinv_f * (float)sum;
            rho = (float)rho_f;
            double hn = (double)((float)a.eta_ksrh * cbrtf((float)mi / rho_f));
            hn = (hn < ksr_max) ? hn : ksr_max;
            np = c;
            h = hn;
        }
        // the search-radius decision of the last pass (hdr_density.hpp:299)
        const double rs_i = a.i_rs[ii];
        const bool itr = h > rs_i;
        if (a.amb_count && (!LONG || wid == 0) && r.act && sub == 0 && fabs(h - rs_i) <= (double)a.amb_tol * rs_i) {
            const int k = atomicAdd(a.amb_count, 1);
            if (k < a.amb_cap) a.amb[k] = make_int2(ii, r.walk);
        }

        const unsigned kept_rho = kept;
        // gradient pass with the final h, hdr_density.hpp:304-349
        {
            const long long idi = a.i_id[ii];
            // velocities stay absolute hi/lo pairs and are differenced per
            // pair: an item may straddle two colliding streams
            const float4 ivh = a.fi.vhi[ii], ivl = a.fi.vlo[ii];
            const float vxi = ivh.x, vyi = ivh.y, vzi = ivh.z;
            const float lxi = ivl.x, lyi = ivl.y, lzi = ivl.z;
            const float hinv = (float)1 / (float)h;
            Acc<false> g_acc, d_acc, rx_acc, ry_acc, rz_acc;
            float pg = 0, pd = 0, prx = 0, pry = 0, prz = 0;
            // pair terms; (vx, vy, vz) the j velocity (FP32C: hi parts, with
            // the lo parts (lx, ly, lz) differenced apart)
            auto gpair = [&](const float4 pj, float vx, float vy, float vz, float lx, float ly, float lz, long long idj) {
                const float dx = xi - pj.x, dy = yi - pj.y, dz = zi - pj.z;
                float ux = vxi - vx, uy = vyi - vy, uz = vzi - vz;
                ux += lxi - lx;
                uy += lyi - ly;
                uz += lzi - lz;
                const float r2 = dx * dx + dy * dy + dz * dz;
                const float ri = (idi != idj) ? rsqrt_r(r2) : (float)0;
                const float q = r2 * ri * hinv;
                const float u = max0((float)1 - q);
                const float u2 = u * u;
                const float u3 = u2 * u;
                const float p14 = (float)1 + (float)4 * q;
                const float w0 = u2 * u2 * p14;            // W0 / c0
                const float w1 = w1_term(q, u, u2, u3, p14);   // W1 / c1
                pg += pj.w * ((float)(3.0 * CEFF0) * w0 + (float)CEFF1 * q * w1);
                const float dw = pj.w * w1 * ri;
                pd += (ux * dx + uy * dy + uz * dz) * dw;
                prx += (uy * dz - uz * dy) * dw;
                pry += (uz * dx - ux * dz) * dw;
                prz += (ux * dy - uy * dx) * dw;
            };
            auto pair = [&](int k) {
                if constexpr (LONG) {
                    const int j = bj[k];
                    const float4 vh = __ldg(&a.fj.vhi[j]), vl = __ldg(&a.fj.vlo[j]);
                    gpair(make_float4(bx[k], by[k], bz[k], bm[k]), vh.x, vh.y, vh.z, vl.x, vl.y, vl.z,
                          __ldg(&a.j_id[j]));
                } else {
                    const float4 vj = s_v[wid][k];
                    const float2 vl = s_vl[wid][k];
                    gpair(s_p[wid][k], vj.x, vj.y, vj.z, (float)vj.w, vl.x, vl.y, s_id[wid][k]);
                }
            };
            auto fold = [&]() {
                g_acc.add(pg);
                d_acc.add(pd);
                rx_acc.add(prx);
                ry_acc.add(pry);
                rz_acc.add(prz);
                pg = 0; pd = 0; prx = 0; pry = 0; prz = 0;
            };
            // Each lane first marks the tile entries inside its own support
            // (r^2/h^2 below 1 + 2e-5, so every pair with q < 1 is marked),
            // then evaluates the gradient terms of the marked entries only, in
            // tile order; the unmarked pairs contribute exactly zero.
            const float lim = hinv * hinv * (float)1.00002;
            auto mark = [&](int k, unsigned &msk) {
                const float4 pj = LONG ? make_float4(bx[k], by[k], bz[k], bm[k]) : s_p[LONG ? 0 : wid][LONG ? 0 : k];
                const float dx = xi - pj.x, dy = yi - pj.y, dz = zi - pj.z;
                const float r2 = dx * dx + dy * dy + dz * dz;
                if (!(r2 * lim >= (float)1)) msk |= 1u << (k & 31);
            };
            // sums of one tile in pg .. prz
            auto tile = [&](int head, int n) {
                unsigned msk = 0;
                if (tpi == 1 && n == 32) {
#pragma unroll 8
                    for (int k = 0; k < 32; ++k) mark(head + k, msk);
                } else {
                    for (int k = sub; k < n; k += tpi) mark(head + k, msk);
                }
                while (msk) {
                    const int k = __ffs(msk) - 1;
                    msk &= msk - 1;
                    pair(head + k);
                }
            };
            // LONG: this lane's sums to and from tile q
            auto put = [&](int q) {
                l_part[q][0][lane] = pg;
                l_part[q][1][lane] = pd;
                l_part[q][2][lane] = prx;
                l_part[q][3][lane] = pry;
                l_part[q][4][lane] = prz;
                pg = 0; pd = 0; prx = 0; pry = 0; prz = 0;
            };
            auto take = [&](int q) {
                pg = l_part[q][0][lane];
                pd = l_part[q][1][lane];
                prx = l_part[q][2][lane];
                pry = l_part[q][3][lane];
                prz = l_part[q][4][lane];
                fold();
            };
            auto run = [&](int head, int n) {
                tile(head, n);
                fold();
                __syncwarp();
            };
            if (nl_ok && __all_sync(FULL, (float)h <= nl_h)) {
                // this lane's list, two entries per round (gathers first),
                // folded after eight; LONG: eight entries each for the warps
                const int cmax = (int)__reduce_max_sync(FULL, (unsigned)ncnt);
                auto round2 = [&](int c0) {
                    int jj[2];
                    float4 pj[2];
                    float4 vh[2];
                    float4 vl[2];
                    long long idj[2];
#pragma unroll
                    for (int u = 0; u < 2; ++u) jj[u] = (c0 + u < ncnt) ? a.nbr[nlb + (c0 + u) * 32] : -1;
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        if (jj[u] >= 0) {
                            pj[u] = jpos(jj[u]);
                            vh[u] = __ldg(&a.fj.vhi[jj[u]]);
                            vl[u] = __ldg(&a.fj.vlo[jj[u]]);
                            idj[u] = __ldg(&a.j_id[jj[u]]);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 2; ++u)
                        if (jj[u] >= 0) gpair(pj[u], vh[u].x, vh[u].y, vh[u].z, vl[u].x, vl[u].y, vl[u].z, idj[u]);
                };
                if constexpr (LONG) {
                    const int n8 = (cmax + 1) / 8 + 1;   // folds (the last of what is left, or nothing)
                    for (int b0 = 0; b0 < n8; b0 += LT) {
                        const int nq = min(LT, n8 - b0);
                        for (int q = wid; q < nq; q += WARPS) {
                            for (int c0 = 8 * (b0 + q); c0 < min(cmax, 8 * (b0 + q) + 8); c0 += 2) round2(c0);
                            put(q);
                        }
                        __syncthreads();
                        for (int q = 0; q < nq; ++q) take(q);
                        __syncthreads();
                    }
                } else {
                    for (int c0 = 0; c0 < cmax; c0 += 2) {
                        round2(c0);
                        if ((c0 & 7) == 6) fold();
                    }
                    fold();
                }
                if (r.act) ev_list_g += (unsigned)ncnt;
                ++n_listed;
            } else {
                if constexpr (LONG) {
                    sweep_long(support2<float>(h),
                               [&](int head, int n, int q) {
                                   tile(head, n);
                                   const bool any = pg != 0.0f || pd != 0.0f || prx != 0.0f || pry != 0.0f || prz != 0.0f;
                                   put(q);
                                   return __any_sync(FULL, any);
                               },
                               [&](int q, int head) {
                                   (void)head;
                                   take(q);
                               });
                } else {
                    sweep(support2<float>(h), true, false, run);
                }
            }
            const double sg = seg_sum(g_acc.value(), tpi);
            const double sd = seg_sum(d_acc.value(), tpi);
            const double sx = seg_sum(rx_acc.value(), tpi);
            const double sy = seg_sum(ry_acc.value(), tpi);
            const double sz = seg_sum(rz_acc.value(), tpi);
            if (r.act && sub == 0 && (!LONG || wid == 0)) {
                const float hf = (float)h;
                const float hinv_f = 1.0f / hf;
                const float hinv4 = hinv_f * hinv_f * hinv_f * hinv_f;
                const float rinv = 1.0f / (float)rho;
                const float g = -hinv4 * (float)sg;
                const float xf = (float)CEFF1 * hinv4 * (float)sx, yf = (float)CEFF1 * hinv4 * (float)sy,
                            zf = (float)CEFF1 * hinv4 * (float)sz;
                const float om = 1.0f / (1.0f + hf * rinv * g / 3.0f);
                const float rot2 = xf * xf + yf * yf + zf * zf;
                const double omega = om;
                const double divv = -(float)CEFF1 * hinv4 * (float)sd * rinv * om;
                const double rotv = ((rot2 != 0.0f) ? sqrtf(rot2) : 0.0f) * rinv * om;
                a.o_dens[ii] = (double)rho;
                a.o_divv[ii] = divv;
                a.o_rotv[ii] = rotv;
                a.o_grdh[ii] = omega;
                a.o_ksr[ii] = h;
                a.o_np[ii] = (long long)np;
                a.o_itr[ii] = itr ? 1 : 0;
            }
        }
        if (a.n_eval) {
            const unsigned long long l0 = __reduce_add_sync(FULL, ev_list);
            const unsigned long long l1 = __reduce_add_sync(FULL, ev_list_g);
            if (lane == 0 && (!LONG || wid == 0)) {
                atomicAdd(a.n_eval, (unsigned long long)kept_rho * (unsigned long long)r.ni + l0);
                atomicAdd(a.n_eval + 1, (unsigned long long)(kept - kept_rho) * (unsigned long long)r.ni + l1);
            }
        }
        if (a.n_pass && lane == 0 && (!LONG || wid == 0)) {
            atomicAdd(a.n_pass, (unsigned long long)n_listed);
            atomicAdd(a.n_pass + 1, (unsigned long long)(3 - n_listed));
        }
    }
}

}  // namespace sphk

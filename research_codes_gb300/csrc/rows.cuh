// rows.cuh — per-particle neighbour rows: for every i-particle the j indices
// of its walk's list that can lie inside a given radius.
//
// The pair sums of the density (both precisions), of the FP64 hydro force and
// of the derivative run over these rows instead of the walk's whole list
// (~15x longer): a list entry is tested once, in FP32, and the pair arithmetic
// in either precision touches only ~60 entries per particle.
//
// mark_rows streams a walk's list through a shared ring (one warp per work
// item, as the pair kernels do), drops entries beyond the item's box, tests
// the rest against every i-particle with packed FP32 instructions and appends
// the hits to the particles' rows in list order.  The test is conservative:
// the radius is widened over every rounding of the FP32 frame, so a row is a
// superset of the pairs inside the radius and never depends on the precision
// of the sums that follow; entries beyond a support add exactly zero there.
// Bound: instruction issue and the latency of the list streaming.
#pragma once

#include "sph_device.cuh"

namespace sphk {

// Entries of a row; particles with more go to the sweep queue.
constexpr int ROW_CAP = 128;
static_assert(ROW_CAP % 32 == 0, "eight lanes read a row four entries at a time");
// Items with longer lists are marked by a whole block (LONG form of
// mark_rows): one warp would stream such a list for longer than the rest of
// the phase takes (a step of 64 entries costs ~0.3 us).
constexpr int LONG_LIST = 4096;
constexpr int MARK_LONG_WARPS = 16;
// Radii outside this range (or NaN) are left to the sweep: their squares
// leave the FP32 range.
constexpr float ROW_HMIN = 1.0e-15f, ROW_HMAX = 1.0e15f;

__device__ __forceinline__ float df_diff(float hi, float lo, float chi, float clo) {
    return (hi - chi) + (lo - clo);
}

// Double-float split of an FP64 value: hi = float(x), lo = float(x - hi).
__device__ __forceinline__ float2 df_split(double x) {
    const float h = (float)x;
    return make_float2(h, (float)(x - (double)h));
}

struct ItemRef {   // decoded work item
    int walk, jb, nj, ni, tpi, sub, li, ii, ic;
    bool act;
};

__device__ __forceinline__ ItemRef decode(const WorkItem &it, const int *j_off, const int *i_list, int lane) {
    ItemRef r;
    r.walk = it.x;
    r.jb = j_off[it.x];
    r.nj = j_off[it.x + 1] - r.jb;
    r.ni = it.z;
    r.tpi = lanes_per_i(it.z);
    const int sh = ilog2_pow2(r.tpi);
    r.li = lane >> sh;
    r.sub = lane & (r.tpi - 1);
    r.act = r.li < it.z;
    const int k = it.y + (r.act ? r.li : 0);
    r.ii = i_list ? i_list[k] : k;
    r.ic = i_list ? i_list[it.y] : it.y;   // the item's centre particle
    return r;
}

struct MarkArgs {
    // double-float positions; lo.w of the i (and, symmetric rows, the j)
    // records: h rounded up
    const float4 *i_hi, *i_lo, *j_hi, *j_lo;
    float slack;             // row radius over h_i
    const WorkItem *items;
    int n_items;
    const int *n_items_dev;  // when set, the item count is read from device memory
    const int *j_off;        // per walk: [j_off[w], j_off[w+1]) in j index space
    const int *j_idx;        // null: entries are j indices themselves
    const int *i_list;       // null: item i-particles are contiguous
    int *queue;              // item counter, 0 at launch
    int *rows;               // row of particle i: rows[i * ROW_CAP ...]
    int2 *info;              // per particle: entries (> ROW_CAP: none, see ovf), walk
    int2 *ovf;               // particles without a row: (particle, walk)
    int *n_ovf;
    WorkItem *long_items;    // items left to the LONG form, and their number
    int *n_long;
};

// Tests of 32 ring entries against this lane's particle, two per packed
// instruction: bit k of the result marks entry k.
template <bool SYM>
__device__ __forceinline__ unsigned mark_tile(const float *x, const float *y, const float *z, const float *h2, float xi,
                                              float yi, float zi, float lim) {
    const f2 XI = f2_make(xi, xi), YI = f2_make(yi, yi), ZI = f2_make(zi, zi), NEG = f2_make(-1.0f, -1.0f);
    unsigned msk = 0;
#pragma unroll
    for (int k = 0; k < 32; k += 2) {
        const f2 DX = f2_fma(f2_lds(x + k), NEG, XI);
        const f2 DY = f2_fma(f2_lds(y + k), NEG, YI);
        const f2 DZ = f2_fma(f2_lds(z + k), NEG, ZI);
        const float2 r2 = f2_get(f2_fma(DZ, DZ, f2_fma(DY, DY, f2_mul(DX, DX))));
        float l0 = lim, l1 = lim;
        if (SYM) {
            const float2 hj = f2_get(f2_lds(h2 + k));
            l0 = fmaxf(l0, hj.x);
            l1 = fmaxf(l1, hj.y);
        }
        if (!(r2.x > l0)) msk |= 1u << k;
        if (!(r2.y > l1)) msk |= 2u << k;
    }
    return msk;
}

// SYM: j inside max(h_i, h_j) (hydro); else inside slack * h_i (density).
// LONG: a block per item of the long-item queue, its warps streaming
// interleaved steps of the list; the hits of all warps meet in shared rows,
// which are put into list order at the end (the same rows as one warp writes).
template <bool SYM, int WARPS, bool LONG = false>
__global__ void __launch_bounds__(WARPS * 32) mark_rows(const MarkArgs a) {
    constexpr int RING = 128;   // < 32 left over + a step of 64
    __shared__ int s_row[LONG ? 32 : 1][ROW_CAP];   // list positions of the hits
    __shared__ int s_cnt[LONG ? 32 : 1];
    __shared__ __align__(16) float s_x[WARPS][RING], s_y[WARPS][RING], s_z[WARPS][RING];
    __shared__ __align__(16) float s_h[SYM ? WARPS : 1][RING];
    __shared__ int s_j[WARPS][RING];
    const int lane = threadIdx.x & 31;
    const int wid = threadIdx.x >> 5;
    const unsigned lt = lanemask_lt();
    const int n_items = LONG ? *a.n_long : (a.n_items_dev ? *a.n_items_dev : a.n_items);
    constexpr int STEP = 64, STRIDE = LONG ? WARPS * STEP : STEP;   // entries of a step, between a warp's steps
    int next = blockIdx.x;   // LONG
    for (;;) {
        int item = 0;
        if (LONG) {
            item = next;
            next += gridDim.x;
        } else {
            if (lane == 0) item = atomicAdd(a.queue, 1);
            item = __shfl_sync(FULL, item, 0);
        }
        if (item >= n_items) return;
        const WorkItem wi = LONG ? a.long_items[item] : a.items[item];
        ItemRef r = decode(wi, a.j_off, a.i_list, lane);
        if (LONG) {   // a lane per particle
            r.tpi = 1;
            r.sub = 0;
            r.li = lane;
            r.act = lane < r.ni;
            const int k = wi.y + (r.act ? lane : 0);
            r.ii = a.i_list ? a.i_list[k] : k;
            if (threadIdx.x < 32) s_cnt[threadIdx.x] = 0;
            __syncthreads();
        } else if (r.nj > LONG_LIST && a.long_items) {
            if (lane == 0) a.long_items[atomicAdd(a.n_long, 1)] = wi;
            continue;
        }
        const int tpi = r.tpi, sub = r.sub, ii = r.ii, nj = r.nj, jb = r.jb;
        const int t0 = LONG ? wid * STEP : 0;
        const float4 ch = a.i_hi[r.ic], cl = a.i_lo[r.ic], ph = a.i_hi[ii], pl = a.i_lo[ii];
        const bool use = r.act && a.slack > 0.0f && pl.w >= ROW_HMIN && pl.w <= ROW_HMAX;
        int lcount = use ? 0 : ROW_CAP + 1;
        if (__any_sync(FULL, use)) {
            const float xi = df_diff(ph.x, pl.x, ch.x, cl.x), yi = df_diff(ph.y, pl.y, ch.y, cl.y);
            const float zi = df_diff(ph.z, pl.z, ch.z, cl.z);
            IBox<float> box;
            box.from_lanes(xi, yi, zi);
            // widening over the rounding of the frame: 2^-24 per coordinate
            // of the item's extent, and 2^-47 of the global coordinates (lo
            // parts); the factor 1.0001 covers the same of the radius itself
            const float ext = fmaxf(fmaxf(fmaxf(-box.xl, box.xh), fmaxf(-box.yl, box.yh)), fmaxf(-box.zl, box.zh));
            const float pad = 5.0e-7f * ext + 3.0e-14f * (fabsf(ch.x) + fabsf(ch.y) + fabsf(ch.z) + 3.0f * ext);
            const float rad = pl.w * a.slack * 1.0001f + pad;
            const float lim = use ? rad * rad : -1.0f;
            const float rf2 = warp_max(use ? rad * rad : 0.0f);
            auto jlist = [&](int k) -> int { return a.j_idx ? a.j_idx[jb + k] : jb + k; };
            // two entries per lane and step, records one step ahead of their
            // use, list indices two
            float4 nh[2], nl[2];
            int jn[2], jx[2];
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const int k = t0 + 32 * s + lane;
                jx[s] = 0;
                jn[s] = 0;
                if (k < nj) {
                    jx[s] = jlist(k);
                    nh[s] = a.j_hi[jx[s]];
                    nl[s] = a.j_lo[jx[s]];
                }
                if (k + STRIDE < nj) jn[s] = jlist(k + STRIDE);
            }
            int head = 0, fill = 0;
            int *row = a.rows + (size_t)ii * ROW_CAP;
            auto consume = [&](int n) {
                unsigned m = 0;
                if (tpi == 1 && n == 32) {
                    m = mark_tile<SYM>(&s_x[wid][head], &s_y[wid][head], &s_z[wid][head], &s_h[SYM ? wid : 0][head],
                                       xi, yi, zi, lim);
                } else {
                    for (int k = sub; k < n; k += tpi) {
                        const float dx = xi - s_x[wid][head + k], dy = yi - s_y[wid][head + k];
                        const float dz = zi - s_z[wid][head + k];
                        float l = lim;
                        if (SYM) l = fmaxf(l, s_h[wid][head + k]);
                        if (!(dx * dx + dy * dy + dz * dz > l)) m |= 1u << k;
                    }
                }
                if (!use) m = 0;
                if (LONG) {
                    for (; m; m &= m - 1) {
                        const int pos = atomicAdd(&s_cnt[lane], 1);
                        if (pos < ROW_CAP) s_row[lane][pos] = s_j[wid][head + __ffs(m) - 1];
                    }
                    __syncwarp();
                    return;
                }
                // the tpi lanes of one particle write consecutive segments
                const int c = __popc(m);
                int pos = lcount;
                if (tpi == 1) {
                    lcount += c;
                } else {
                    int incl = c;
                    for (int o = 1; o < tpi; o <<= 1) {
                        const int v = __shfl_up_sync(FULL, incl, o, tpi);
                        if (sub >= o) incl += v;
                    }
                    pos += incl - c;
                    lcount += __shfl_sync(FULL, incl, tpi - 1, tpi);
                }
                for (; m; m &= m - 1) {
                    const int k = __ffs(m) - 1;
                    if (pos < ROW_CAP) row[pos] = s_j[wid][head + k];
                    ++pos;
                }
                __syncwarp();
            };
            for (int t = t0; t < nj; t += STRIDE) {
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    const int k = t + 32 * s + lane;
                    const float4 h = nh[s], l = nl[s];
                    const int jc = LONG ? k : jx[s];
                    if (k + STRIDE < nj) {
                        jx[s] = jn[s];
                        nh[s] = a.j_hi[jn[s]];
                        nl[s] = a.j_lo[jn[s]];
                    }
                    if (k + 2 * STRIDE < nj) jn[s] = jlist(k + 2 * STRIDE);
                    bool keep = false;
                    float px = 0, py = 0, pz = 0, hj2 = 0;
                    if (k < nj) {
                        px = df_diff(h.x, l.x, ch.x, cl.x);
                        py = df_diff(h.y, l.y, ch.y, cl.y);
                        pz = df_diff(h.z, l.z, ch.z, cl.z);
                        float lim_j = rf2;
                        if (SYM) {
                            const float rj = l.w * 1.0001f + pad;
                            hj2 = (l.w >= ROW_HMIN && l.w <= ROW_HMAX) ? rj * rj : INFINITY;
                            lim_j = fmaxf(rf2, hj2);
                        }
                        keep = !(box.d2(px, py, pz) > lim_j * 1.0002f);
                    }
                    const unsigned m = __ballot_sync(FULL, keep);
                    if (keep) {
                        const int slot = (head + fill + __popc(m & lt)) & (RING - 1);
                        s_x[wid][slot] = px;
                        s_y[wid][slot] = py;
                        s_z[wid][slot] = pz;
                        if (SYM) s_h[wid][slot] = hj2;
                        s_j[wid][slot] = jc;
                    }
                    fill += __popc(m);
                }
                __syncwarp();
                while (fill >= 32) {
                    consume(32);
                    head = (head + 32) & (RING - 1);
                    fill -= 32;
                }
            }
            if (fill > 0) consume(fill);
        }
        if (LONG) {
            // rows in list order: each hit's place is the number of hits at
            // earlier list positions
            __syncthreads();
            for (int i = wid; i < r.ni; i += WARPS) {
                const int c = s_cnt[i];
                int *row = a.rows + (size_t)__shfl_sync(FULL, ii, i) * ROW_CAP;
                if (c <= ROW_CAP)
                    for (int e = lane; e < c; e += 32) {
                        const int k = s_row[i][e];
                        int rank = 0;
                        for (int q = 0; q < c; ++q) rank += s_row[i][q] < k ? 1 : 0;
                        row[rank] = a.j_idx ? a.j_idx[jb + k] : jb + k;
                    }
            }
            if (use) lcount = s_cnt[lane];
            __syncthreads();   // s_cnt is cleared for the next item
            if (wid != 0) continue;
        }
        if (r.act && sub == 0) {
            a.info[ii] = make_int2(lcount, r.walk);
            if (lcount > ROW_CAP) a.ovf[atomicAdd(a.n_ovf, 1)] = make_int2(ii, r.walk);
        }
    }
}

// Positions as double-float records with h (rounded up) in lo.w, from FP64
// arrays; hinv: h holds 1/h.
__global__ inline void make_row_records(int n, const dbl4 *pm, const double *h, bool hinv, float4 *hi, float4 *lo) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const dbl4 p = pm[k];
        const float2 x = df_split(p.x), y = df_split(p.y), z = df_split(p.z);
        const double hk = h ? (hinv ? 1.0 / h[k] : h[k]) : 0.0;
        hi[k] = make_float4(x.x, y.x, z.x, (float)p.w);
        lo[k] = make_float4(x.y, y.y, z.y, __double2float_ru(hk));
    }
}

}  // namespace sphk

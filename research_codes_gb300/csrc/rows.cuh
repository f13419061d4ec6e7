// rows.cuh — per-particle neighbour rows: for every i-particle the j indices
// of its walk's list that can lie inside a given radius.
//
// The pair sums of the density and the hydro force run over these rows
// instead of the walk's whole list (~15x longer): a list entry is tested
// once, in FP32, and the pair arithmetic in either precision touches only ~60
// entries per particle.
//
// mark_rows streams a walk's list through a shared ring (one warp per work
// item, as the pair kernels do), drops entries beyond the item's box, tests
// the rest against every i-particle with packed FP32 instructions and appends
// the hits to the particles' rows in list order.  The test is conservative:
// the radius is widened over every rounding of the FP32 frame, so a row is a
// superset of the pairs inside the radius and never depends on the precision
// of the sums that follow; entries beyond a support add exactly zero there.
// Bound: instruction issue and the latency of the list streaming, so short
// launches live by how many warps they keep busy: long lists go to blocks
// (LONG), small systems get smaller items.  What rows replace: every pass over
// all listed pairs, in FP64 at 1/60 of the FP32 rate: FP64 density call of 64
// among 20k 2095 -> 105 us, FP64 run of 50k (density and hydro) 85 -> 40 ms.
#pragma once

#include "sph_device.cuh"

namespace sphk {

// Entries of a row; particles with more go to the sweep queue.  128 hold the 50
// to 64 neighbours of eta 1.18 to 1.28 within 3%; at eta 1.6 (125 neighbours) most
// particles have no row and are swept (FP32C density: rowless_items).  Times
// there, by the lists before rows and now: density batch of 20k in walks of 300
// 4.8 and 2.9 ms in FP32C, 21.4 and 3.7 in FP64; hydro batch 10.5 and 4.6, 37.9 and
// 5.7; evaluation of 200k 16.4 and 16.1 ms in FP32C, 86.2 and 60.3 in FP64.
constexpr int ROW_CAP = 128;
static_assert(ROW_CAP % 32 == 0, "eight lanes read a row four entries at a time");
// Items with longer lists than this are taken by a whole block (the LONG forms
// of mark_rows and density_stream).  On a full SM a warp streams ~1.6e7 entries
// per second, the chip ~5e11 listed pairs: beyond pairs / 131072 entries one
// warp's item lasts about a quarter of the whole walk's time (200k head-on run: 37.8 ms at
// 2^16, 37.1 at 2^17, 38.6 at 2^18, 45.9 at 2^19).
__device__ __forceinline__ int long_list(long long pairs, int least = 768) {
    return (int)min(max(pairs >> 17, (long long)least), 1LL << 30);
}
constexpr int MARK_LONG_WARPS = 16, HYDRO_LONG_WARPS = 8;
// FP32C hydro rows: longest list (in steps of 64 entries) whose LONG form
// keeps the row order of a warp's item.  Calls leave longer ones to a warp;
// in a system they go to blocks too, and their rows are in list order.
constexpr int LONG_STEPS = 2048;
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

// The same for records that FP64 sums follow: a value beyond the FP32 range
// keeps an infinite hi part (NaN with the lo part that goes with it), so that
// it lies outside every finite radius, as in FP64.
__device__ __forceinline__ float2 df_split_far(double x) {
    const float2 s = df_split(x);
    return make_float2(s.x, isinf(s.x) ? 0.0f : s.y);
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

// Which rows mark_rows writes: density rows (j inside slack * h_i), or hydro
// rows (j inside max(h_i, h_j), equal ids dropped), whose kernel also takes
// the signal-velocity maximum, accurate values in FP32 or FP64.
enum RowKind { ROWS_DENSITY = 0, ROWS_HYDRO32 = 1, ROWS_HYDRO64 = 2 };

// Double-float particle records of FP32C mode.
struct F32Part {
    const float4 *phi;   // x_hi, y_hi, z_hi, mass
    const float4 *plo;   // x_lo, y_lo, z_lo, aux
    const float4 *vhi;   // vx_hi, vy_hi, vz_hi, aux
    const float4 *vlo;   // vx_lo, vy_lo, vz_lo, aux
};

// Items of the LONG form: n[0] of them from the front of the array, the
// longest, n[1] from its end (cap entries); n[2] counts those taken.
struct LongQueue {
    WorkItem *items;
    int *n;
    int cap;
    __device__ __forceinline__ void push(const WorkItem &wi) const { items[atomicAdd(n, 1)] = wi; }
    // the block's next item; false when there is none (slot: shared)
    __device__ __forceinline__ bool take(int *slot, WorkItem &wi) const {
        __syncthreads();
        if (threadIdx.x == 0) *slot = atomicAdd(&n[2], 1);
        __syncthreads();
        const int k = *slot, front = n[0];
        if (k >= front + n[1]) return false;
        wi = items[k < front ? k : cap - 1 - (k - front)];
        return true;
    }
};

struct MarkArgs {
    // double-float positions; h (rounded up) in lo.w (density: i records) or
    // hi.w (hydro: i and j records)
    const float4 *i_hi, *i_lo, *j_hi, *j_lo;
    float slack;             // density: row radius over h_i
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
    LongQueue longs;         // items of the LONG form
    // push_long: the kernel itself moves items with lists beyond long_nj (with
    // pairs set: beyond long_list of the walks' listed pairs) to that queue
    bool push_long;
    const long long *pairs;
    int long_nj;
    // hydro: velocity and sound speed in FP32
    const float4 *i_v, *j_v;
    const long long *i_id, *j_id;
    // accurate signal-velocity terms: double-float records and (.y) sound
    // speeds (FP32C) or FP64 records
    F32Part fi, fj;
    const float4 *fi_g2, *fj_g2;
    const dbl4 *i_pm, *i_vel, *i_h2, *j_pm, *j_vel, *j_h2;
    double *o_vsmx;
    const float *csmax;      // per walk: largest sound speed of its list (null: unknown)
    int sv_skip;             // nonzero: entries whose bound cannot raise any maximum skip their terms
    // when set: list entries x i-particles [0] tested against the supports,
    // [1] beyond them; 32-entry tiles [0] skipped, [1] tested; [0] marked
    // pairs, [1] lane slots of the loops over them
    unsigned long long *n_near, *n_far, *n_skip, *n_mark;
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

// Signal velocity c_i + c_j - 3 min(w, 0) of one pair (hdr_hydro.hpp:368-372)
// in the precision of the hydro outputs.
template <int KIND>
struct Signal {
    typedef float R;
    float4 ph, pl, vh, vl;
    float cs;
    __device__ __forceinline__ void load_i(const MarkArgs &a, int ii) {
        ph = a.fi.phi[ii]; pl = a.fi.plo[ii]; vh = a.fi.vhi[ii]; vl = a.fi.vlo[ii];
        cs = a.fi_g2[ii].y;
    }
    __device__ __forceinline__ R pair(const MarkArgs &a, int j, bool self) const {
        const float4 qh = __ldg(&a.fj.phi[j]), ql = __ldg(&a.fj.plo[j]);
        const float4 uh = __ldg(&a.fj.vhi[j]), ul = __ldg(&a.fj.vlo[j]);
        const float dx = (ph.x - qh.x) + (pl.x - ql.x), dy = (ph.y - qh.y) + (pl.y - ql.y);
        const float dz = (ph.z - qh.z) + (pl.z - ql.z);
        const float ux = (vh.x - uh.x) + (vl.x - ul.x), uy = (vh.y - uh.y) + (vl.y - ul.y);
        const float uz = (vh.z - uh.z) + (vl.z - ul.z);
        const float r2 = dx * dx + dy * dy + dz * dz;
        const float w = (dx * ux + dy * uy + dz * uz) * (self ? 0.0f : rsqrt_r(r2));
        return cs + __ldg(&a.fj_g2[j]).y - 3.0f * (w < 0.0f ? w : 0.0f);
    }
};
template <>
struct Signal<ROWS_HYDRO64> {
    typedef double R;
    dbl4 p, v;
    double cs;
    __device__ __forceinline__ void load_i(const MarkArgs &a, int ii) {
        p = a.i_pm[ii]; v = a.i_vel[ii];
        cs = a.i_h2[ii].y;
    }
    __device__ __forceinline__ R pair(const MarkArgs &a, int j, bool self) const {
        const dbl4 q = a.j_pm[j], u = a.j_vel[j];
        const double dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
        const double r2 = dx * dx + dy * dy + dz * dz;
        const double w = (dx * (v.x - u.x) + dy * (v.y - u.y) + dz * (v.z - u.z)) * (self ? 0.0 : rsqrt_r(r2));
        return cs + a.j_h2[j].y - 3.0 * (w < 0.0 ? w : 0.0);
    }
};

// One warp per work item streams the walk's list in steps of 64 entries.
// LONG: a block per item of the long-item queue, its warps streaming
// interleaved steps; the hits of all warps meet in the rows by shared
// counters and are put into order at the end (the same rows as one warp
// writes; FP32C hydro: up to LONG_STEPS).
//
// Hydro: the signal-velocity maximum runs over every entry of the list.  A
// term is at most c_i + c_j + 3 (|v_i - v_c| + |v_j - v_c|) with v_c the
// centre particle's velocity, so 32 entries whose largest bound stays below
// every lane's lb, a lower bound of its maximum, skip their terms.  Otherwise
// each pair gets an FP32 upper bound of its term (item-frame positions and
// velocities, widened by their rounding, two pairs per packed instruction),
// and only pairs whose bound exceeds lb, a handful per particle, are evaluated
// accurately (Signal).  lb starts at c_i + the walk's largest sound speed,
// which no maximum undercuts, where that is known, and grows with the accurate
// terms.  The result is the maximum over the accurate terms of all pairs,
// whether or not entries skip.
template <int KIND, int WARPS, bool LONG = false>
__global__ void __launch_bounds__(WARPS * 32, (KIND == ROWS_DENSITY ? 24 : 16) / WARPS) mark_rows(const MarkArgs a) {
    constexpr bool HYDRO = KIND != ROWS_DENSITY;
    constexpr int RING = 128;   // < 32 left over + a step of 64
    constexpr int STEP = 64, STRIDE = LONG ? WARPS * STEP : STEP;   // entries of a step, between a warp's steps
    constexpr int HW = HYDRO ? WARPS : 1, HN = HYDRO ? 32 : 1;
    typedef typename Signal<KIND>::R R;
    __shared__ __align__(16) float s_x[WARPS][RING], s_y[WARPS][RING], s_z[WARPS][RING];
    __shared__ __align__(16) float s_h[HW][HYDRO ? RING : 1];
    __shared__ int s_j[WARPS][RING];   // LONG: list positions
    __shared__ long long s_id[HW][HYDRO ? RING : 1];
    __shared__ int s_cnt[LONG ? 32 : 1];
    constexpr bool KEYS = LONG && KIND == ROWS_HYDRO32;
    __shared__ int s_step[KEYS ? LONG_STEPS : 1];   // staged entries per step, then before it
    // hydro: 32 entries whose signal-velocity terms are due (item-frame
    // position and velocity, sound speed, |v - v_c|)
    __shared__ __align__(16) float s_sig[HW][8][HN];
    __shared__ int s_sj[HW][HN];
    const int lane = threadIdx.x & 31;
    const int wid = threadIdx.x >> 5;
    const int hw = HYDRO ? wid : 0;
    const unsigned lt = lanemask_lt();
    __shared__ int s_next;   // LONG
    const int n_items = LONG ? 0 : (a.n_items_dev ? *a.n_items_dev : a.n_items);
    const int long_nj = a.pairs ? long_list(*a.pairs) : a.long_nj;
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
        ItemRef r = decode(wi, a.j_off, a.i_list, lane);
        const int item_tpi = r.tpi;
        const bool keyed = KEYS && r.nj <= 64 * LONG_STEPS;
        if (LONG) {   // a lane per particle
            r.tpi = 1;
            r.sub = 0;
            r.li = lane;
            r.act = lane < r.ni;
            const int k = wi.y + (r.act ? lane : 0);
            r.ii = a.i_list ? a.i_list[k] : k;
            if (threadIdx.x < 32) s_cnt[threadIdx.x] = 0;
            __syncthreads();
        } else if (a.push_long && r.nj > long_nj && (KIND != ROWS_HYDRO32 || r.nj <= 64 * LONG_STEPS)) {
            if (lane == 0) a.longs.push(wi);
            continue;
        }
        const int tpi = r.tpi, sub = r.sub, ii = r.ii, nj = r.nj, jb = r.jb;
        const int t0 = LONG ? wid * STEP : 0;
        const float4 ch = a.i_hi[r.ic], cl = a.i_lo[r.ic], ph = a.i_hi[ii], pl = a.i_lo[ii];
        const float h_i = HYDRO ? ph.w : pl.w;
        const bool use = r.act && (HYDRO || a.slack > 0.0f) && h_i >= ROW_HMIN && h_i <= ROW_HMAX;
        int lcount = use ? 0 : ROW_CAP + 1;
        R vsmx = 0;
        unsigned n_near = 0, n_steps = 0, n_skipped = 0, n_marked = 0, n_slots = 0;
        if (HYDRO || __any_sync(FULL, use)) {
            const float xi = df_diff(ph.x, pl.x, ch.x, cl.x), yi = df_diff(ph.y, pl.y, ch.y, cl.y);
            const float zi = df_diff(ph.z, pl.z, ch.z, cl.z);
            IBox<float> box;
            box.from_lanes(xi, yi, zi);
            // widening over the rounding of the frame: 2^-24 per coordinate
            // of the item's extent, and 2^-47 of the global coordinates (lo
            // parts); the factor 1.0001 covers the same of the radius itself
            const float ext = fmaxf(fmaxf(fmaxf(-box.xl, box.xh), fmaxf(-box.yl, box.yh)), fmaxf(-box.zl, box.zh));
            // (a centre without a position has no frame: every entry is marked)
            float pad = 5.0e-7f * ext + 3.0e-14f * (fabsf(ch.x) + fabsf(ch.y) + fabsf(ch.z) + 3.0f * ext);
            if (!(pad < 1.0e30f)) pad = INFINITY;
            // (FP32C hydro rows widen h^2 by 2e-4 alone, what FP32 sums need)
            auto reach2 = [&](float h) -> float {
                if (KIND == ROWS_HYDRO32) return h * h * 1.0002f;
                const float rad = h * 1.0001f + pad;
                return rad * rad;
            };
            const float lim = use ? reach2(h_i * (HYDRO ? 1.0f : a.slack)) : -1.0f;
            const float rf2 = warp_max(use ? lim : 0.0f);
            const float boxf = KIND == ROWS_HYDRO32 ? 1.0f : 1.0002f;
            auto jlist = [&](int k) -> int { return a.j_idx ? a.j_idx[jb + k] : jb + k; };
            // hydro: velocity in the frame of the centre particle's, its
            // rounding included in |v - v_c|, and the bounds
            float4 vc, vi;
            float verr = 0, di = 0, ub_i = 0, lb = 0;
            bool exact_i = false;   // FP32 bounds do not hold for this particle's values
            long long idi = 0;
            auto speed = [&](float x, float y, float z) { return sqrt_bound(x * x + y * y + z * z) * 1.000002f + verr; };
            if (HYDRO) {
                vc = a.i_v[r.ic];
                vi = a.i_v[ii];
                verr = 4.0e-7f * (fabsf(vc.x) + fabsf(vc.y) + fabsf(vc.z));
                vi.x -= vc.x; vi.y -= vc.y; vi.z -= vc.z;
                di = speed(vi.x, vi.y, vi.z);
                ub_i = vi.w + 3.0f * di;
                exact_i = !(vi.w >= 1.0e-15f && di < 1.0e15f && ext < 1.0e15f && pad < 1.0e15f);
                if (a.csmax) lb = fmaxf((vi.w + a.csmax[r.walk]) * 0.999997f, 0.0f);
                idi = a.i_id[ii];
            }
            // two entries per lane and step, records one step ahead of their
            // use, list indices two
            float4 nh[2], nl[2], nv[2];
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
                    if (HYDRO) nv[s] = a.j_v[jx[s]];
                }
                if (k + STRIDE < nj) jn[s] = jlist(k + STRIDE);
            }
            int head = 0, fill = 0;
            int *row = a.rows + (size_t)ii * ROW_CAP;
            auto consume = [&](int n) {
                unsigned m = 0;
                if (tpi == 1 && n == 32) {
                    m = mark_tile<HYDRO>(&s_x[wid][head], &s_y[wid][head], &s_z[wid][head], &s_h[hw][HYDRO ? head : 0],
                                         xi, yi, zi, lim);
                } else {
                    for (int k = sub; k < n; k += tpi) {
                        const float dx = xi - s_x[wid][head + k], dy = yi - s_y[wid][head + k];
                        const float dz = zi - s_z[wid][head + k];
                        float l = lim;
                        if (HYDRO) l = fmaxf(l, s_h[hw][head + k]);
                        if (!(dx * dx + dy * dy + dz * dz > l)) m |= 1u << k;
                    }
                }
                if (!use) m = 0;
                if (HYDRO && a.n_mark) {
                    const unsigned c = __popc(m);
                    n_marked += c;
                    n_slots += 32u * __reduce_max_sync(FULL, c);
                }
                if (LONG) {
                    for (; m; m &= m - 1) {
                        const int k = __ffs(m) - 1;
                        if (HYDRO && s_id[hw][head + k] == idi) continue;
                        const int pos = atomicAdd(&s_cnt[lane], 1);
                        if (pos < ROW_CAP) row[pos] = s_j[wid][head + k];
                    }
                } else if (tpi == 1) {
                    for (; m; m &= m - 1) {
                        const int k = __ffs(m) - 1;
                        if (HYDRO && s_id[hw][head + k] == idi) continue;   // self pairs, hdr_hydro.hpp:356
                        if (lcount < ROW_CAP) row[lcount] = s_j[wid][head + k];
                        ++lcount;
                    }
                } else {
                    // the tpi lanes of one particle write consecutive segments
                    if (HYDRO)
                        for (unsigned t = m; t; t &= t - 1) {
                            const int k = __ffs(t) - 1;
                            if (s_id[hw][head + k] == idi) m &= ~(1u << k);
                        }
                    int incl = __popc(m);
                    int pos = lcount - incl;
                    for (int o = 1; o < tpi; o <<= 1) {
                        const int v = __shfl_up_sync(FULL, incl, o, tpi);
                        if (sub >= o) incl += v;
                    }
                    pos += incl;
                    lcount += __shfl_sync(FULL, incl, tpi - 1, tpi);
                    for (; m; m &= m - 1) {
                        if (pos < ROW_CAP) row[pos] = s_j[wid][head + __ffs(m) - 1];
                        ++pos;
                    }
                }
                __syncwarp();
            };
            // upper bound of the signal velocity with staged entry k and its
            // successor: base + 3 max(e - w, 0), e the rounding of w
            auto upper = [&](int k) -> float2 {
                const f2 NEG = f2_make(-1.0f, -1.0f);
                const auto at = [&](int q) { return f2_lds(&s_sig[hw][q][k]); };
                const f2 DX = f2_fma(at(0), NEG, f2_make(xi, xi)), DY = f2_fma(at(1), NEG, f2_make(yi, yi));
                const f2 DZ = f2_fma(at(2), NEG, f2_make(zi, zi));
                const f2 UX = f2_fma(at(3), NEG, f2_make(vi.x, vi.x)), UY = f2_fma(at(4), NEG, f2_make(vi.y, vi.y));
                const f2 UZ = f2_fma(at(5), NEG, f2_make(vi.z, vi.z));
                const float2 r2 = f2_get(f2_fma(DZ, DZ, f2_fma(DY, DY, f2_mul(DX, DX))));
                const f2 DOT = f2_fma(DZ, UZ, f2_fma(DY, UY, f2_mul(DX, UX)));
                const f2 RI = f2_make(rsqrt_r(r2.x), rsqrt_r(r2.y));
                const f2 E = f2_fma(f2_add(at(7), f2_make(di, di)),
                                    f2_fma(f2_make(4.0f * pad, 4.0f * pad), RI, f2_make(4.0e-6f, 4.0e-6f)),
                                    f2_make(2.0f * verr, 2.0f * verr));
                // NaN (r = 0 in the frame: nothing is known of w) stays NaN,
                // which no comparison with lb skips
                const float2 t = f2_get(f2_fma(f2_mul(DOT, NEG), RI, E));
                return f2_get(f2_fma(f2_make(max0_nan(t.x), max0_nan(t.y)), f2_make(3.0f, 3.0f),
                                     f2_add(at(6), f2_make(vi.w, vi.w))));
            };
            // signal-velocity terms of the nb <= 32 staged entries; lb is kept
            // a margin of 2e-6 below accurate terms
            auto signals = [&](int nb) {
                unsigned m = 0;
                if (tpi == 1) {
#pragma unroll 4
                    for (int k = 0; k < 32; k += 2) {
                        const float2 up = upper(k);
                        if (!(up.x <= lb)) m |= 1u << k;
                        if (!(up.y <= lb)) m |= 2u << k;
                    }
                } else {
                    // two consecutive entries, as a packed bound holds; one
                    // each for 32 lanes
                    for (int k = 2 * sub & 31; k < 32; k += 2 * tpi) {
                        const float2 up = upper(k);
                        if (!(up.x <= lb)) m |= 1u << k;
                        if (!(up.y <= lb)) m |= 2u << k;
                    }
                    if (tpi == 32) m &= sub < 16 ? 0x55555555u : 0xaaaaaaaau;
                }
                if (exact_i) {
                    m = 0;
                    for (int k = sub; k < nb; k += tpi) m |= 1u << k;
                }
                m &= nb >= 32 ? FULL : (1u << nb) - 1u;   // entries of the list
                Signal<KIND> sig;
                if (m) sig.load_i(a, ii);
                for (; m; m &= m - 1) {
                    const int k = __ffs(m) - 1;
                    const float2 up = upper(k & ~1);   // lb has grown since
                    if (!exact_i && ((k & 1) ? up.y : up.x) <= lb) continue;
                    const int j = s_sj[hw][k];
                    const R vs = sig.pair(a, j, a.j_id[j] == idi);
                    if (vs > vsmx) {   // (not for NaN, which raises neither)
                        vsmx = vs;
                        lb = fmaxf(lb, fminf((float)vs * 0.999997f, 3.0e38f));
                    }
                }
                for (int o = 1; o < tpi; o <<= 1) lb = fmaxf(lb, __shfl_xor_sync(FULL, lb, o));
                __syncwarp();
            };
            for (int t = t0; t < nj; t += STRIDE) {
                int staged = 0;   // of this step
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    const int k = t + 32 * s + lane;
                    const float4 h = nh[s], l = nl[s], v = nv[s];
                    const int j = jx[s], jc = LONG ? k : j;
                    if (k + STRIDE < nj) {
                        jx[s] = jn[s];
                        nh[s] = a.j_hi[jn[s]];
                        nl[s] = a.j_lo[jn[s]];
                        if (HYDRO) nv[s] = a.j_v[jn[s]];
                    }
                    if (k + 2 * STRIDE < nj) jn[s] = jlist(k + 2 * STRIDE);
                    bool keep = false;
                    float px = 0, py = 0, pz = 0, hj2 = 0;
                    float bmax = 0;
                    float4 sp = make_float4(0.0f, 0.0f, 0.0f, 0.0f), sv = sp;
                    if (k < nj) {
                        px = df_diff(h.x, l.x, ch.x, cl.x);
                        py = df_diff(h.y, l.y, ch.y, cl.y);
                        pz = df_diff(h.z, l.z, ch.z, cl.z);
                        float lim_j = rf2;
                        if (HYDRO) {
                            hj2 = (h.w >= 0.0f && h.w <= ROW_HMAX) ? reach2(fmaxf(h.w, ROW_HMIN)) : INFINITY;
                            lim_j = fmaxf(rf2, hj2);
                            const float ux = v.x - vc.x, uy = v.y - vc.y, uz = v.z - vc.z;
                            const float d = speed(ux, uy, uz);
                            const float bj = v.w + 3.0f * d;
                            // non-negative floats (or NaN) order like their bit patterns
                            bmax = (bj < 0.0f) ? 0.0f : bj;
                            // an entry outside the FP32 range gets an infinite bound
                            const bool in = fmaxf(fmaxf(fabsf(px), fabsf(py)), fabsf(pz)) < 1.0e15f && d < 1.0e15f;
                            sp = in ? make_float4(px, py, pz, v.w) : make_float4(0.0f, 0.0f, 0.0f, v.w);
                            sv = in ? make_float4(ux, uy, uz, d) : make_float4(0.0f, 0.0f, 0.0f, INFINITY);
                            if (!in) bmax = INFINITY;
                        }
                        keep = !(box.d2(px, py, pz) > lim_j * boxf);
                    }
                    const unsigned m = __ballot_sync(FULL, keep);
                    if (keep) {
                        const int slot = (head + fill + __popc(m & lt)) & (RING - 1);
                        s_x[wid][slot] = px;
                        s_y[wid][slot] = py;
                        s_z[wid][slot] = pz;
                        s_j[wid][slot] = keyed ? (jc << 6) | (staged + __popc(m & lt)) : jc;
                        if (HYDRO) {
                            s_h[hw][slot] = hj2;
                            s_id[hw][slot] = a.j_id[j];
                        }
                    }
                    fill += __popc(m);
                    staged += __popc(m);
                    if (HYDRO) {
                        n_near += __popc(m);
                        const int nb = nj - t - 32 * s;
                        if (nb > 0) {
                            const float b = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(bmax)));
                            ++n_steps;
                            if (a.sv_skip && __all_sync(FULL, !exact_i && (ub_i + b) * 1.00001f <= lb)) {
                                ++n_skipped;
                            } else {
                                s_sig[hw][0][lane] = sp.x;
                                s_sig[hw][1][lane] = sp.y;
                                s_sig[hw][2][lane] = sp.z;
                                s_sig[hw][3][lane] = sv.x;
                                s_sig[hw][4][lane] = sv.y;
                                s_sig[hw][5][lane] = sv.z;
                                s_sig[hw][6][lane] = sp.w;
                                s_sig[hw][7][lane] = sv.w;
                                s_sj[hw][lane] = j;
                                __syncwarp();
                                signals(min(32, nb));
                            }
                        }
                    }
                }
                if (KEYS && keyed && lane == 0) s_step[t >> 6] = staged;
                __syncwarp();
                while (fill >= 32) {
                    consume(32);
                    head = (head + 32) & (RING - 1);
                    fill -= 32;
                }
            }
            if (fill > 0) consume(fill);
            for (int o = 1; o < tpi; o <<= 1) {
                const R v = __shfl_xor_sync(FULL, vsmx, o);
                vsmx = v > vsmx ? v : vsmx;
            }
        }
        if (HYDRO && a.n_near && lane == 0) {
            const unsigned mine = (nj > t0) ? n_near : 0u;
            atomicAdd(a.n_near, (unsigned long long)mine * (unsigned long long)r.ni);
            if (wid == 0 || !LONG) atomicAdd(a.n_far, (unsigned long long)nj * (unsigned long long)r.ni);
            atomicAdd(a.n_far, 0ull - (unsigned long long)mine * (unsigned long long)r.ni);
            atomicAdd(a.n_skip, (unsigned long long)n_skipped);
            atomicAdd(a.n_skip + 1, (unsigned long long)n_steps);
        }
        if (HYDRO && a.n_mark) {
            const unsigned m = __reduce_add_sync(FULL, n_marked);
            if (lane == 0) {
                atomicAdd(a.n_mark, (unsigned long long)m);
                atomicAdd(a.n_mark + 1, (unsigned long long)n_slots);
            }
        }
        if (LONG) {
            __syncthreads();
            // rows in list order: each hit's place is the number of hits at
            // earlier list positions.  FP32C hydro: in the order of a warp's
            // item, whose tpi lanes take a tile of 32 staged entries each
            // their own residue
            if (KEYS && keyed) {
                if (wid == 0) {
                    int before = 0;
                    for (int k0 = 0; 64 * k0 < nj; k0 += 32) {
                        const int v = 64 * (k0 + lane) < nj ? s_step[k0 + lane] : 0;
                        int incl = v;
                        for (int o = 1; o < 32; o <<= 1) {
                            const int x = __shfl_up_sync(FULL, incl, o);
                            if (lane >= o) incl += x;
                        }
                        if (64 * (k0 + lane) < nj) s_step[k0 + lane] = before + incl - v;
                        before += __shfl_sync(FULL, incl, 31);
                    }
                }
                __syncthreads();
            }
            auto key = [&](int q) {
                if (!(KEYS && keyed)) return q;
                const int e = s_step[q >> 12] + (q & 63);   // staged entries before it
                return (e & ~31) << 5 | ((e & (item_tpi - 1)) << 5) | (e & 31);
            };
            for (int i = wid; i < r.ni; i += WARPS) {
                const int c = s_cnt[i];
                int *row = a.rows + (size_t)__shfl_sync(FULL, ii, i) * ROW_CAP;
                if (c > ROW_CAP) continue;
                int pos[ROW_CAP / 32], keys[ROW_CAP / 32], rank[ROW_CAP / 32];
#pragma unroll
                for (int u = 0; u < ROW_CAP / 32; ++u) {
                    const bool in = 32 * u + lane < c;
                    pos[u] = in ? row[32 * u + lane] : 0;
                    keys[u] = in ? key(pos[u]) : 0x7fffffff;
                    rank[u] = 0;
                }
#pragma unroll
                for (int v = 0; v < ROW_CAP / 32; ++v)
                    for (int q = 0; q < 32; ++q) {
                        const int other = __shfl_sync(FULL, keys[v], q);
#pragma unroll
                        for (int u = 0; u < ROW_CAP / 32; ++u) rank[u] += other < keys[u] ? 1 : 0;
                    }
                __syncwarp();
#pragma unroll
                for (int u = 0; u < ROW_CAP / 32; ++u)
                    if (32 * u + lane < c) {
                        const int k = KEYS && keyed ? pos[u] >> 6 : pos[u];
                        row[rank[u]] = a.j_idx ? a.j_idx[jb + k] : jb + k;
                    }
            }
            if (use) lcount = s_cnt[lane];
            if (HYDRO) {
                // the warps' maxima, in the staging buffer
                R *best = reinterpret_cast<R *>(&s_sig[0][0][0]);
                best[wid * 32 + lane] = vsmx;
                __syncthreads();
                for (int w = 0; w < WARPS; ++w) {
                    const R v = best[w * 32 + lane];
                    vsmx = v > vsmx ? v : vsmx;
                }
            }
            __syncthreads();   // the shared arrays are reused by the next item
            if (wid != 0) continue;
        }
        if (r.act && sub == 0) {
            if (HYDRO) a.o_vsmx[ii] = (double)vsmx;
            a.info[ii] = make_int2(lcount, r.walk);
            if (lcount > ROW_CAP) a.ovf[atomicAdd(a.n_ovf, 1)] = make_int2(ii, r.walk);
        }
    }
}

// Position and mass as a double-float record with h (rounded up) in lo.w.
// F64: of FP64 sums (df_split_far).
template <bool F64>
__device__ __forceinline__ void row_record(const dbl4 &p, double h, float4 &hi, float4 &lo) {
    const float2 x = F64 ? df_split_far(p.x) : df_split(p.x);
    const float2 y = F64 ? df_split_far(p.y) : df_split(p.y);
    const float2 z = F64 ? df_split_far(p.z) : df_split(p.z);
    hi = make_float4(x.x, y.x, z.x, (float)p.w);
    lo = make_float4(x.y, y.y, z.y, __double2float_ru(h));
}
__device__ __forceinline__ void velocity_record(const dbl4 &v, float4 &hi, float4 &lo) {
    const float2 x = df_split(v.x), y = df_split(v.y), z = df_split(v.z);
    hi = make_float4(x.x, y.x, z.x, 0.0f);
    lo = make_float4(x.y, y.y, z.y, 0.0f);
}

__global__ inline void make_row_records(int n, const dbl4 *pm, const double *h, float4 *hi, float4 *lo) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        float4 a, b;
        row_record<true>(pm[k], h[k], a, b);
        hi[k] = a;
        lo[k] = b;
    }
}

// The hydro mark records of one particle: position hi parts with h (rounded
// up) in w, velocity with the sound speed in w.
__device__ __forceinline__ void hydro_mark_records(const dbl4 &p, const dbl4 &v, double hinv, double cs, float4 &mp,
                                                   float4 &mv) {
    mp = make_float4((float)p.x, (float)p.y, (float)p.z, __frcp_ru(__double2float_rd(hinv)));
    mv = make_float4((float)v.x, (float)v.y, (float)v.z, (float)cs);
}

// The same for FP64 runs, with the position lo parts (h1: 1/h in x; h2: sound
// speed in y).
__global__ inline void make_hydro_row_records(int n, const dbl4 *pm, const dbl4 *vel, const dbl4 *h1, const dbl4 *h2,
                                              float4 *mp, float4 *lo, float4 *mv) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const dbl4 p = pm[k];
        const float2 x = df_split_far(p.x), y = df_split_far(p.y), z = df_split_far(p.z);
        float4 a, b;
        hydro_mark_records(p, vel[k], h1[k].x, h2[k].y, a, b);
        mp[k] = a;
        lo[k] = make_float4(x.y, y.y, z.y, 0.0f);
        mv[k] = b;
    }
}

}  // namespace sphk

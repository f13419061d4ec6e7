// pair_kernels.cuh — the three SPH pair-interaction kernels.
//
// Design (shared by density, hydro and gravity):
//  * Work is a list of WorkItems (<= 32 i-particles of one walk).  A
//    persistent grid of warps pulls items from a global queue counter
//    (atomicAdd), so walks with very different neighbour counts balance across
//    the SMs.  Items may address their i-particles through an index list
//    (search-radius re-walks recompute only the particles still iterating).
//  * A warp streams its walk's j-list through a private 32-entry shared-memory
//    tile: lane k loads entry t+k (gathered through j_idx), converts it and
//    stores it; every lane then reads the tile by broadcast.  With n_i < 32
//    several lanes share one i-particle (tpi lanes, strided over the tile) and
//    are combined with warp shuffles.
//  * FP32C mode (F64 == false): the engine keeps double-float copies of the
//    particle state (hi = float(x), lo = float(x - hi)).  Staging forms
//    (hi_j - hi_c) + (lo_j - lo_c) relative to the item's first i-particle c
//    in FP32, so pair differences keep FP32 relative accuracy far from the
//    origin and across colliding streams, and no FP64 instruction runs in the
//    pair loops (GB300's FP64 rate is ~1/60 of FP32).  Each lane's per-tile
//    FP32 partial sums are folded into Kahan accumulators.
//  * FP64 mode (F64 == true): the same kernels in plain FP64 on global
//    coordinates without compensation: the "plain FP64 GPU" comparator.
#pragma once

#include "density_rows.cuh"
#include "density_stream.cuh"
#include "hydro_df.cuh"
#include "rows.cuh"
#include "sph_device.cuh"

// Minimum resident blocks per SM requested from the compiler for the FP32C
// gravity and hydro kernels (register budget 65536 / (128 threads x blocks)).
#ifndef SPH_GRAVITY_MIN_BLOCKS
#define SPH_GRAVITY_MIN_BLOCKS 4
#endif
// Unroll factors of the full-tile FP32C loops: f32x2 iterations (two entries
// each) of the gravity loop.
#ifndef SPH_GRAVITY_UNROLL
#define SPH_GRAVITY_UNROLL 16
#endif
// The double-float hydro pass (128 threads): 3 blocks per SM, 168 registers.
#ifndef SPH_HYDRO_DF_MIN_BLOCKS
#define SPH_HYDRO_DF_MIN_BLOCKS 3
#endif

namespace sphk {

constexpr int GRAVITY_UNROLL = SPH_GRAVITY_UNROLL;

// ---------------------------------------------------------------- hydro
struct HydroArgs {
    // FP64 mode records
    const dbl4 *i_pm;    // x, y, z, (mass unused)
    const dbl4 *i_vel;
    const dbl4 *i_h1;    // hinv, pres, presc, bswt
    const dbl4 *i_h2;    // dens, vsnd, alph, alphu
    const double2 *i_h3; // thrm, eta
    const dbl4 *j_pm;    // x, y, z, mass
    const dbl4 *j_vel;
    const dbl4 *j_h1;
    const dbl4 *j_h2;
    const double2 *j_h3;
    // FP32C mode records: vhi.w = hinv, vlo.w = hinv^4,
    // g1 = (P_hi, P_lo, presc, bswt), g2 = (dens, vsnd, alph, alphu),
    // g3 = (thrm_hi, thrm_lo, eta, -)
    F32Part fi, fj;
    const float4 *fi_g1, *fi_g2, *fi_g3, *fj_g1, *fj_g2, *fj_g3;
    const long long *i_id;
    const long long *j_id;
    const int *j_off;
    const int *j_idx;
    // outputs (the signal velocity is mark_rows')
    double *o_acch;      // 3 per particle
    double *o_accg;      // 3 per particle
    double *o_udot, *o_diffu;
    // rows (mark_rows): the pairs inside either support, self pairs excluded;
    // particles without a row in the sweep queue.  g4 records: (1/h hi, 1/h lo,
    // h^-4 hi, h^-4 lo).
    const float4 *fi_g4 = nullptr, *fj_g4 = nullptr;
    const int *rows = nullptr;
    const int2 *info = nullptr;
    const int2 *ovf = nullptr;
    const int *n_ovf = nullptr;
    int n_i = 0;   // i-particles (the sums cover [0, n_i))
    // FP64: double-float positions with h in hi.w, for the sweep's distance test
    const float4 *mi_p = nullptr, *mi_l = nullptr, *mj_p = nullptr, *mj_l = nullptr;
};

// ---- FP64 hydro sums over the rows, hdr_hydro.hpp:349-398 ----
struct Hydro64P {   // one particle's fields
    dbl4 p, v, h1, h2;
    double2 h3;
    double hinv4;
};
__device__ __forceinline__ Hydro64P hydro64_load(const dbl4 *pm, const dbl4 *vel, const dbl4 *h1, const dbl4 *h2,
                                                 const double2 *h3, int k) {
    Hydro64P q;
    q.p = pm[k]; q.v = vel[k]; q.h1 = h1[k]; q.h2 = h2[k]; q.h3 = h3[k];
    q.hinv4 = q.h1.x * q.h1.x * q.h1.x * q.h1.x;
    return q;
}
struct Hydro64Acc {
    double ax = 0, ay = 0, az = 0, gx = 0, gy = 0, gz = 0, ud = 0, df = 0;
};
__device__ __forceinline__ void hydro64_pair(const Hydro64P &i, const Hydro64P &j, Hydro64Acc &s) {
    const double dx = i.p.x - j.p.x, dy = i.p.y - j.p.y, dz = i.p.z - j.p.z;
    const double ux = i.v.x - j.v.x, uy = i.v.y - j.v.y, uz = i.v.z - j.v.z;
    const double r2 = dx * dx + dy * dy + dz * dz;
    const double ri = rsqrt_r(r2);
    const double rr = infinite(r2) ? r2 : r2 * ri;   // (inf * 0 is NaN)
    // kernel gradients W1(q) for both smoothing lengths
    const double qi = rr * i.h1.x, qj = rr * j.h1.x;
    if (qi >= 1.0 && qj >= 1.0) return;   // beyond both supports: every term is zero
    const double ui = max0(1.0 - qi), uj = max0(1.0 - qj);
    const double ui2 = ui * ui, uj2 = uj * uj;
    const double w1i = w1_term(qi, ui, ui2, ui2 * ui, 1.0 + 4.0 * qi);
    const double w1j = w1_term(qj, uj, uj2, uj2 * uj, 1.0 + 4.0 * qj);
    const double dw_i = CEFF1 * i.hinv4 * w1i;
    const double dw_j = CEFF1 * j.hinv4 * w1j;
    const double mj = j.p.w;
    const double ka = (dw_i + dw_j) * mj;
    // viscosity, :368-376
    const double w = (dx * ux + dy * uy + dz * uz) * ri;
    const double wneg = w < 0.0 ? w : 0.0;
    const double vs = i.h2.y + j.h2.y - 3.0 * wneg;
    const double rhi = rcp_r(i.h2.x + j.h2.x);
    const double av = (i.h1.w + j.h1.w) * (i.h2.z + j.h2.z) * vs * wneg;
    // pressure gradient, :378-382
    const double ta = (i.h1.z + j.h1.z - 0.5 * av * rhi) * ka * ri;
    s.ax -= ta * dx;
    s.ay -= ta * dy;
    s.az -= ta * dz;
    // energy equation with conduction, :384-393
    const double du = i.h3.x - j.h3.x;
    const double alphu = i.h2.w + j.h2.w;
    double cond = 0.0;
    if (alphu != 0.0) {
        const double vsu2 = fabs(i.h1.y - j.h1.y) * rhi * 2.0;
        cond = alphu * (vsu2 > 0.0 ? vsu2 * rsqrt_r(vsu2) : 0.0) * du;
    }
    s.ud += ka * (i.h1.z * w - rhi * (0.25 * av * wneg - cond));
    s.df += rhi * du * ka * ri;
    // softening correction, :395-398
    const double dg = mj * ri * (i.h3.y * dw_i + j.h3.y * dw_j);
    s.gx += dg * dx;
    s.gy += dg * dy;
    s.gz += dg * dz;
}
__device__ __forceinline__ void hydro64_store(const HydroArgs &a, int p, const double (&v)[8]) {
    for (int c = 0; c < 3; ++c) {
        a.o_acch[3 * p + c] = 0.5 * v[c];
        a.o_accg[3 * p + c] = 0.5 * v[3 + c];
    }
    a.o_udot[p] = 0.5 * v[6];
    a.o_diffu[p] = 2.0 * v[7];
}

// Eight lanes per particle over its row; particles without one are left to
// the sweep.  FP64 pipe bound (~120 instructions per pair): rows hold ~57 pairs
// where the list holds ~900, and the old kernel tested each of those in FP64
// (call of 256 among 20k: 2690 -> 179 us).
// L = 32 in small calls (warp_per_row): the call of 256 162 -> 143 us.
constexpr int HROWS_LANES = 8, HROWS_THREADS = 128;
template <int L>
__global__ void __launch_bounds__(HROWS_THREADS) hydro64_rows(const HydroArgs a) {
    const int lane = threadIdx.x & 31, sub = lane & (L - 1);
    const int gw = (blockIdx.x * HROWS_THREADS + threadIdx.x) >> 5, nw = (gridDim.x * HROWS_THREADS) >> 5;
    for (int k0 = gw * (32 / L); k0 < a.n_i; k0 += nw * (32 / L)) {
        const int p = k0 + lane / L;
        const int cnt = p < a.n_i ? a.info[p].x : ROW_CAP + 1;
        const bool ok = cnt <= ROW_CAP;
        Hydro64Acc s;
        if (ok) {
            const Hydro64P I = hydro64_load(a.i_pm, a.i_vel, a.i_h1, a.i_h2, a.i_h3, p);
            const int *row = a.rows + (size_t)p * ROW_CAP;
            for (int e = sub; e < cnt; e += L)
                hydro64_pair(I, hydro64_load(a.j_pm, a.j_vel, a.j_h1, a.j_h2, a.j_h3, row[e]), s);
        }
        double v[8] = {s.ax, s.ay, s.az, s.gx, s.gy, s.gz, s.ud, s.df};
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = seg_sum(v[q], L);
        if (ok && sub == 0) hydro64_store(a, p, v);
    }
}

// One block per particle of the sweep queue over its walk's whole list.  A
// warp's entries within reach are summed 32 at a time: the FP64 pipe takes a
// warp's instruction whole, and a step of 32 entries holds two or three (sums of
// 200k particles at 125 neighbours 23.8 -> 20.0 ms, batch of 20k 8.9 -> 5.7).
__global__ inline void __launch_bounds__(DSWEEP_THREADS) hydro64_sweep(const HydroArgs a) {
    constexpr int T = DSWEEP_THREADS, U = 4, RING = 256;   // U entries per thread in flight
    static_assert(32 * (U + 1) <= RING, "hits of a round");
    __shared__ double red[8][T / 32];
    __shared__ int s_hit[T / 32][RING];
    const int n = *a.n_ovf;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned lt = lanemask_lt();
    for (int e = blockIdx.x; e < n; e += gridDim.x) {
        const int p = a.ovf[e].x, w = a.ovf[e].y;
        const Hydro64P I = hydro64_load(a.i_pm, a.i_vel, a.i_h1, a.i_h2, a.i_h3, p);
        const long long idi = a.i_id[p];
        const float4 ph = a.mi_p[p], pl = a.mi_l[p];
        const float pad = 3.0e-14f * (fabsf(ph.x) + fabsf(ph.y) + fabsf(ph.z));
        const int je = a.j_off[w + 1];
        int head = 0, fill = 0;
        Hydro64Acc s;
        auto pair = [&](int j) {
            if (a.j_id[j] != idi) hydro64_pair(I, hydro64_load(a.j_pm, a.j_vel, a.j_h1, a.j_h2, a.j_h3, j), s);
        };
        for (int b = a.j_off[w] + 32 * wid; b < je; b += T * U) {
            int j[U];
            float4 qh[U], ql[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int k = b + u * T + lane;
                j[u] = k < je ? (a.j_idx ? a.j_idx[k] : k) : -1;
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (j[u] >= 0) {
                    qh[u] = a.mj_p[j[u]];
                    ql[u] = a.mj_l[j[u]];
                }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                // pairs beyond both supports add zero: an FP32 distance test with
                // the margins of mark_rows (h outside its range: no test)
                bool hit = j[u] >= 0;
                if (hit) {
                    const float dx = df_diff(qh[u].x, ql[u].x, ph.x, pl.x), dy = df_diff(qh[u].y, ql[u].y, ph.y, pl.y);
                    const float dz = df_diff(qh[u].z, ql[u].z, ph.z, pl.z);
                    const float h = fmaxf(ph.w, qh[u].w) * 1.0001f + pad;
                    const bool test = ph.w >= ROW_HMIN && ph.w <= ROW_HMAX && qh[u].w >= ROW_HMIN && qh[u].w <= ROW_HMAX;
                    hit = !(test && square_sum(dx, dy, dz) > h * h);
                }
                const unsigned m = __ballot_sync(FULL, hit);
                if (hit) s_hit[wid][(head + fill + __popc(m & lt)) & (RING - 1)] = j[u];
                fill += __popc(m);
            }
            __syncwarp();
            for (; fill >= 32; fill -= 32, head += 32) pair(s_hit[wid][(head + lane) & (RING - 1)]);
            __syncwarp();
        }
        if (lane < fill) pair(s_hit[wid][(head + lane) & (RING - 1)]);
        double v[8] = {s.ax, s.ay, s.az, s.gx, s.gy, s.gz, s.ud, s.df};
        block_sum(v, red);
        if (threadIdx.x == 0) hydro64_store(a, p, v);
    }
}

// FP32C hydro, double-float pass over the marked-pair rows: one thread per
// i-particle (particles in index order, so a warp's particles share most of
// their neighbours in L1), two row entries at a time in the two halves of
// packed f32x2 instructions (even and odd entries summed apart and combined
// at the end), an odd last entry alone.  Rows that overflowed are left to
// hydro_df_sweep.
constexpr int HYDRO_DF_THREADS = 128;
__device__ __forceinline__ HydroDFP<float> hydro_df_load(const F32Part &f, const float4 *g1, const float4 *g2,
                                                         const float4 *g3, const float4 *g4, int j) {
    return hydro_df_rec(f.phi[j], f.plo[j], f.vhi[j], f.vlo[j], g1[j], g2[j], g3[j], g4[j]);
}
__device__ __forceinline__ void hydro_df_store(const HydroArgs &a, int p, const HydroDFAcc<float> &acc,
                                               dfk::df presc) {
    double h[3], g[3], ud, dif;
    hydro_df_finish(acc, presc, CEFF1, h, g, &ud, &dif);
    a.o_acch[3 * p + 0] = h[0];
    a.o_acch[3 * p + 1] = h[1];
    a.o_acch[3 * p + 2] = h[2];
    a.o_accg[3 * p + 0] = g[0];
    a.o_accg[3 * p + 1] = g[1];
    a.o_accg[3 * p + 2] = g[2];
    a.o_udot[p] = ud;
    a.o_diffu[p] = dif;
}
__global__ inline void __launch_bounds__(HYDRO_DF_THREADS, SPH_HYDRO_DF_MIN_BLOCKS) hydro_df_lists(const HydroArgs a) {
    using dfk::pk;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < a.n_i; p += gridDim.x * blockDim.x) {
        const int c = a.info[p].x;
        if (c > ROW_CAP) continue;
        const HydroDFP<float> I = hydro_df_load(a.fi, a.fi_g1, a.fi_g2, a.fi_g3, a.fi_g4, p);
        const HydroDFP<pk> I2 = hydro_df_pack(I, I);
        HydroDFAcc<pk> acc2 = hydro_df_zero<pk>();
        HydroDFAcc<float> acc = hydro_df_zero<float>();
        const int *row = a.rows + (size_t)p * ROW_CAP;
        int k = 0;
        for (; k + 1 < c; k += 2) {
            const HydroDFP<float> J0 = hydro_df_load(a.fj, a.fj_g1, a.fj_g2, a.fj_g3, a.fj_g4, row[k]);
            const HydroDFP<float> J1 = hydro_df_load(a.fj, a.fj_g1, a.fj_g2, a.fj_g3, a.fj_g4, row[k + 1]);
            hydro_df_pair(I2, hydro_df_pack(J0, J1), acc2);
        }
        if (k < c) hydro_df_pair(I, hydro_df_load(a.fj, a.fj_g1, a.fj_g2, a.fj_g3, a.fj_g4, row[k]), acc);
        // (even + odd) + last, each addition renormalised
        dfk::df *v[9] = {&acc.ax, &acc.ay, &acc.az, &acc.gx, &acc.gy, &acc.gz, &acc.ud, &acc.uv, &acc.dif};
        const dfk::dv<pk> *w[9] = {&acc2.ax, &acc2.ay, &acc2.az, &acc2.gx, &acc2.gy, &acc2.gz,
                                   &acc2.ud, &acc2.uv, &acc2.dif};
#pragma unroll
        for (int q = 0; q < 9; ++q) *v[q] = dfk::add(dfk::add(lane0(*w[q]), lane1(*w[q])), *v[q]);
        hydro_df_store(a, p, acc, I.presc);
    }
}

// The same for the particles whose row overflowed: one block per particle
// over its walk's whole j-list (such walks have long lists: a warp alone
// would wait on one load after another), pairs beyond both supports skipped
// (they add exactly zero), the threads' double-float sums combined by warp
// shuffles and then across the warps in a fixed order.
constexpr int HYDRO_SWEEP_THREADS = 512;
__device__ __forceinline__ dfk::df warp_sum_df(dfk::df x) {
    for (int o = 16; o > 0; o >>= 1) {
        const dfk::df y = dfk::make(__shfl_xor_sync(FULL, x.h, o), __shfl_xor_sync(FULL, x.l, o));
        x = dfk::add(x, y);
    }
    return x;
}
__global__ inline void __launch_bounds__(HYDRO_SWEEP_THREADS) hydro_df_sweep(const HydroArgs a) {
    constexpr int NW = HYDRO_SWEEP_THREADS / 32;
    __shared__ dfk::df part[9][NW];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int n_ovf = *a.n_ovf;
    for (int e = blockIdx.x; e < n_ovf; e += gridDim.x) {
        const int2 ent = a.ovf[e];
        const int p = ent.x, w = ent.y;
        const int jb = a.j_off[w], je = a.j_off[w + 1];
        const long long idi = a.i_id[p];
        const HydroDFP<float> I = hydro_df_load(a.fi, a.fi_g1, a.fi_g2, a.fi_g3, a.fi_g4, p);
        HydroDFAcc<float> acc = hydro_df_zero<float>();
        const float hi2 = 1.0f / (I.hinv.h * I.hinv.h);
        for (int k = jb + threadIdx.x; k < je; k += HYDRO_SWEEP_THREADS) {
            const int j = a.j_idx ? a.j_idx[k] : k;
            if (a.j_id[j] == idi) continue;
            // pairs beyond both supports add exactly zero: skip them on an
            // FP32 distance test with a margin far above its rounding
            const float4 ph = a.fj.phi[j], pl = a.fj.plo[j], vh = a.fj.vhi[j];
            const float dx = (I.xh - ph.x) + (I.xl - pl.x), dy = (I.yh - ph.y) + (I.yl - pl.y);
            const float dz = (I.zh - ph.z) + (I.zl - pl.z);
            const float hj2 = 1.0f / (vh.w * vh.w);
            if (dx * dx + dy * dy + dz * dz > fmaxf(hi2, hj2) * 1.001f) continue;
            hydro_df_pair(I, hydro_df_rec(ph, pl, vh, a.fj.vlo[j], a.fj_g1[j], a.fj_g2[j], a.fj_g3[j], a.fj_g4[j]),
                          acc);
        }
        dfk::df *v[9] = {&acc.ax, &acc.ay, &acc.az, &acc.gx, &acc.gy, &acc.gz, &acc.ud, &acc.uv, &acc.dif};
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            const dfk::df t = warp_sum_df(*v[q]);
            if (lane == 0) part[q][wid] = t;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
#pragma unroll
            for (int q = 0; q < 9; ++q) {
                dfk::df t = part[q][0];
                for (int u = 1; u < NW; ++u) t = dfk::add(t, part[q][u]);
                *v[q] = t;
            }
            hydro_df_store(a, p, acc, I.presc);
        }
        __syncthreads();   // part[] is rewritten by the next particle
    }
}

// ---------------------------------------------------------------- gravity
struct GravityArgs {
    // FP64 mode: i (x, y, z, eps2); j sources split at n_split: index
    // k < n_split reads (j_pm, j_eps2)[k], k >= n_split reads
    // (s_pm, s_eps2)[k - n_split] (superparticles / tree-node monopoles)
    const dbl4 *i_pe;
    const dbl4 *j_pm;       // x, y, z, mass
    const double *j_eps2;
    const dbl4 *s_pm;
    const double *s_eps2;
    // FP32C mode: hi = (x, y, z, mass), lo = (x, y, z, eps2); fi_* for the
    // i-particles, f_* for the j particles and f_s* for the monopoles
    const float4 *fi_phi, *fi_plo, *f_phi, *f_plo, *f_shi, *f_slo;
    int n_split;
    const WorkItem *items;
    int n_items;
    const int *n_items_dev;
    const int *j_off;
    const int *j_idx;
    const int *i_list;
    int *queue;
    double *o_acc;          // 3 per particle (assigned)
    double *o_pot, *o_eta;
    // work units: each item's list in `slices` parts (0: 1), the results of
    // part s at particle index + s * o_stride, to be added in the order of s
    int slices;
    size_t o_stride;
    // quadrupole of the sources k >= n_split (tree nodes), traceless, about
    // their centre of mass; null: monopoles only (the reference's SPJ).
    // FP64: 6 per node (xx, yy, zz, xy, xz, yz); FP32C: (xx, yy, zz, xy) and
    // (xz, yz, -, -)
    const double *s_quad;
    const float4 *f_sq0, *f_sq1;
};

// Parts of an item's list so that n_items items make `units` work units, of at
// least 128 entries each.  One unit is a warp's turn: a few more units than
// resident warps leave most of the last round empty, and a call of a few
// items leaves most of the chip idle.
inline int gravity_slices(long long n_items, long long nj, long long units, int most) {
    const long long want = n_items > 0 ? (units + n_items - 1) / n_items : 1;
    const long long fit = nj / 128 > 1 ? nj / 128 : 1;
    const long long s = want < fit ? want : fit;
    return (int)(s < 1 ? 1 : (s > most ? most : s));
}

// Adds the parts' results of particle p: g = (acc, pot, eta).
__device__ __forceinline__ void gravity_gather(const double *acc, const double *pot, const double *eta, int p,
                                               int slices, size_t stride, double (&g)[5]) {
    for (int q = 0; q < 5; ++q) g[q] = 0.0;
    for (int s = 0; s < slices; ++s) {
        const size_t o = p + s * stride;
        g[0] += acc[3 * o];
        g[1] += acc[3 * o + 1];
        g[2] += acc[3 * o + 2];
        g[3] += pot[o];
        g[4] += eta[o];
    }
}
// The same by the 32 lanes of a warp, parts l, l + 32, ... per lane.
__device__ __forceinline__ void gravity_gather_warp(const double *acc, const double *pot, const double *eta, int p,
                                                    int slices, size_t stride, int lane, double (&g)[5]) {
    for (int q = 0; q < 5; ++q) g[q] = 0.0;
    for (int s = lane; s < slices; s += 32) {
        const size_t o = p + s * stride;
        g[0] += acc[3 * o];
        g[1] += acc[3 * o + 1];
        g[2] += acc[3 * o + 2];
        g[3] += pot[o];
        g[4] += eta[o];
    }
    for (int q = 0; q < 5; ++q) g[q] = seg_sum(g[q], 32);
}

// Bound: FP32C by instruction issue (packed FMAs and rsqrt), FP64 by the FP64
// pipe (88% busy, 30 operations per pair).  Units of an item's list fill the
// chip where items are few: 500 targets x 20k 411 -> 40 us, gravity of a 50k
// FP64 evaluation 9.9 -> 6.3 ms.
// JT: the j-tile, list entries a warp stages in shared memory per pass (32
// or 64; each lane loads JT / 32 of them one tile ahead) and sums in FP32
// before folding into the compensated accumulators.
template <bool F64, int WARPS, int JT = 32>
__global__ void __launch_bounds__(WARPS * 32, F64 ? 1 : SPH_GRAVITY_MIN_BLOCKS)
gravity_kernel(const GravityArgs a) {
    typedef typename Real<F64>::T R;
    typedef typename Real<F64>::T4 R4;
    static_assert(JT == 32 || JT == 64, "j-tile of 32 or 64 entries");
    constexpr int S = JT / 32;        // entries per lane and tile
    constexpr int QR = 64 * S;        // quadrupole ring: < 32 left + a tile
    // FP64: one record per entry; FP32C: structure of arrays, so that two
    // consecutive entries load as one f32x2 operand
    __shared__ R4 s_p[F64 ? WARPS : 1][JT];   // dx, dy, dz, mass
    __shared__ R s_e[F64 ? WARPS : 1][JT];    // eps2
    __shared__ __align__(16) float s_x[F64 ? 1 : WARPS][JT], s_y[F64 ? 1 : WARPS][JT], s_z[F64 ? 1 : WARPS][JT],
        s_m[F64 ? 1 : WARPS][JT], s_q[F64 ? 1 : WARPS][JT];
    // tree-node entries of the list with their quadrupoles, compacted into a
    // ring (position in the item frame + eps^2; Q xx yy zz xy; Q xz yz)
    __shared__ R4 q_p[WARPS][QR];
    __shared__ R4 q_a[WARPS][QR];
    __shared__ typename Real<F64>::T2 q_b[WARPS][QR];
    const unsigned lt = lanemask_lt();
    const int slices = a.slices > 0 ? a.slices : 1;
    const bool quad = F64 ? (a.s_quad != nullptr) : (a.f_sq0 != nullptr);
    const int lane = threadIdx.x & 31;
    const int wid = threadIdx.x >> 5;
    const int n_items = a.n_items_dev ? *a.n_items_dev : a.n_items;

    for (;;) {
        int item = 0;
        if (lane == 0) item = atomicAdd(a.queue, 1);
        item = __shfl_sync(FULL, item, 0);
        if (item >= n_items * slices) return;
        const int slice = item % slices;
        const ItemRef r = decode(a.items[item / slices], a.j_off, a.i_list, lane);
        const int tpi = r.tpi, sub = r.sub, ii = r.ii;
        // whole tiles per part
        const int tiles = (r.nj + JT - 1) / JT;
        const int t_lo = (int)((long long)tiles * slice / slices), t_hi = (int)((long long)tiles * (slice + 1) / slices);
        const int jb = r.jb + t_lo * JT, nj = min(r.nj, t_hi * JT) - t_lo * JT;

        R xi, yi, zi, e2i;
        float4 ch = make_float4(0, 0, 0, 0), cl = ch;
        if (F64) {
            const dbl4 p = a.i_pe[ii];
            xi = p.x; yi = p.y; zi = p.z; e2i = p.w;
        } else {
            ch = a.fi_phi[r.ic]; cl = a.fi_plo[r.ic];
            const float4 h = a.fi_phi[ii], l = a.fi_plo[ii];
            xi = df_diff(h.x, l.x, ch.x, cl.x);
            yi = df_diff(h.y, l.y, ch.y, cl.y);
            zi = df_diff(h.z, l.z, ch.z, cl.z);
            e2i = l.w;
        }
        Acc<F64> ax, ay, az, pt, et;
        // j records are loaded one tile ahead of their use, list indices
        // two tiles ahead, so that their latency overlaps the pair loop
        auto jlist = [&](int k) -> int { return a.j_idx ? a.j_idx[jb + k] : jb + k; };
        float4 nh[S], nl[S];   // next tile (FP32C)
        dbl4 np64[S];          // next tile (FP64)
        double ne64[S];
        auto load = [&](int s, int j) {
            if constexpr (F64) {
                if (j < a.n_split) {
                    np64[s] = a.j_pm[j];
                    ne64[s] = a.j_eps2[j];
                } else {
                    np64[s] = a.s_pm[j - a.n_split];
                    ne64[s] = a.s_eps2[j - a.n_split];
                }
            } else {
                if (j < a.n_split) {
                    nh[s] = a.f_phi[j];
                    nl[s] = a.f_plo[j];
                } else {
                    nh[s] = a.f_shi[j - a.n_split];
                    nl[s] = a.f_slo[j - a.n_split];
                }
            }
        };
        int jn[S], jnx[S];   // list index two tiles ahead, of the next tile
#pragma unroll
        for (int s = 0; s < S; ++s) {
            nh[s] = make_float4(0, 0, 0, 0);
            nl[s] = nh[s];
            np64[s] = make_dbl4(0, 0, 0, 0);
            ne64[s] = 0.0;
            jn[s] = 0;
            jnx[s] = 0;
            if (32 * s + lane < nj) {
                jnx[s] = jlist(32 * s + lane);
                load(s, jnx[s]);
            }
            if (JT + 32 * s + lane < nj) jn[s] = jlist(JT + 32 * s + lane);
        }
        int qhead = 0, qfill = 0;
        // quadrupole terms of the node entries in the ring: the potential
        // -(1/2) r.Q.r R^5 and acceleration Q r R^5 - (5/2)(r.Q.r) r R^7 with
        // r = x_i - c and R = (r^2 + eps_node^2)^(-1/2), accumulated doubled
        // like the monopole sums (halved once at the end)
        auto run_quad = [&](int n_q) {
            R qax = 0, qay = 0, qaz = 0, qpt = 0;
            auto quad_term = [&](int k) {
                const R4 P = q_p[wid][qhead + k];
                const R4 A = q_a[wid][qhead + k];
                const typename Real<F64>::T2 B = q_b[wid][qhead + k];
                const R dx = xi - P.x, dy = yi - P.y, dz = zi - P.z;
                const R rr = rsqrt_r(dz * dz + (dy * dy + (dx * dx + P.w)));
                const R rr2 = rr * rr;
                const R rr5 = rr2 * rr2 * rr;
                const R rr7 = rr5 * rr2;
                const R qx = A.x * dx + A.w * dy + B.x * dz;
                const R qy = A.w * dx + A.y * dy + B.y * dz;
                const R qz = B.x * dx + B.y * dy + A.z * dz;
                const R rqr = dx * qx + dy * qy + dz * qz;
                const R f = (R)5 * rqr * rr7;
                const R g = (R)2 * rr5;
                // two fused multiply-adds per component
                qax += qx * g;
                qax -= f * dx;
                qay += qy * g;
                qay -= f * dy;
                qaz += qz * g;
                qaz -= f * dz;
                qpt -= rqr * rr5;
            };
            if (tpi == 1 && n_q == 32) {
#pragma unroll 8
                for (int k = 0; k < 32; ++k) quad_term(k);
            } else {
                for (int k = sub; k < n_q; k += tpi) quad_term(k);
            }
            ax.add(qax);
            ay.add(qay);
            az.add(qaz);
            pt.add(qpt);
            __syncwarp();
        };
        for (int t = 0; t < nj; t += JT) {
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const int jk = t + 32 * s + lane;
                const float4 h = nh[s], l = nl[s];
                const dbl4 p64 = np64[s];
                const double e64 = ne64[s];
                const int jcur = jnx[s];
                if (jk + JT < nj) {
                    jnx[s] = jn[s];
                    load(s, jn[s]);
                }
                if (jk + 2 * JT < nj) jn[s] = jlist(jk + 2 * JT);
                if (quad) {
                    const bool node = jk < nj && jcur >= a.n_split;
                    const unsigned mq = __ballot_sync(FULL, node);
                    if (node) {
                        const int slot = (qhead + qfill + __popc(mq & lt)) & (QR - 1);
                        const int nd = jcur - a.n_split;
                        if constexpr (F64) {
                            const double *q = a.s_quad + 6 * (size_t)nd;
                            q_p[wid][slot] = Real<F64>::make4(p64.x, p64.y, p64.z, e64);
                            q_a[wid][slot] = Real<F64>::make4(q[0], q[1], q[2], q[3]);
                            q_b[wid][slot] = Real<F64>::make2(q[4], q[5]);
                        } else {
                            const float4 q0 = a.f_sq0[nd], q1 = a.f_sq1[nd];
                            q_p[wid][slot] = Real<F64>::make4(df_diff(h.x, l.x, ch.x, cl.x),
                                                              df_diff(h.y, l.y, ch.y, cl.y),
                                                              df_diff(h.z, l.z, ch.z, cl.z), l.w);
                            q_a[wid][slot] = q0;
                            q_b[wid][slot] = make_float2(q1.x, q1.y);
                        }
                    }
                    qfill += __popc(mq);
                }
                if (jk < nj) {
                    const int e = 32 * s + lane;
                    if (F64) {
                        s_p[wid][e] = Real<F64>::make4(p64.x, p64.y, p64.z, p64.w);
                        s_e[wid][e] = e64;
                    } else {
                        s_x[wid][e] = df_diff(h.x, l.x, ch.x, cl.x);
                        s_y[wid][e] = df_diff(h.y, l.y, ch.y, cl.y);
                        s_z[wid][e] = df_diff(h.z, l.z, ch.z, cl.z);
                        s_m[wid][e] = h.w;
                        s_q[wid][e] = l.w;
                    }
                }
            }
            __syncwarp();
            const int n = min(JT, nj - t);
            R pax = 0, pay = 0, paz = 0, ppt = 0, pet = 0;
            auto pair = [&](int k) {
                R4 pj;
                R ej;
                if constexpr (F64) {
                    pj = s_p[wid][k];
                    ej = s_e[wid][k];
                } else {
                    pj = Real<F64>::make4(s_x[wid][k], s_y[wid][k], s_z[wid][k], s_m[wid][k]);
                    ej = s_q[wid][k];
                }
                const R dx = xi - pj.x, dy = yi - pj.y, dz = zi - pj.z;
                const R r2 = dx * dx + dy * dy + dz * dz;
                const R rei = rsqrt_r(r2 + e2i);
                const R rej = rsqrt_r(r2 + ej);
                const R rei3 = rei * rei * rei;
                const R rej3 = rej * rej * rej;
                const R g = pj.w * (rei3 + rej3);
                ppt -= pj.w * (rei + rej);
                pax -= dx * g;
                pay -= dy * g;
                paz -= dz * g;
                pet += pj.w * rei3;
            };
            if (!F64 && tpi == 1 && n == JT) {
                // full tile, FP32C: two entries per instruction (f32x2); the
                // even and odd entries are summed separately and combined
                // at the end of the tile.  Sums of -x are kept as sums of x
                // and negated once (exact).
                const f2 XI = f2_make((float)xi, (float)xi), YI = f2_make((float)yi, (float)yi);
                const f2 ZI = f2_make((float)zi, (float)zi), EI = f2_make((float)e2i, (float)e2i);
                const f2 NEG = f2_make(-1.0f, -1.0f);
                f2 AX = f2_make(0.0f, 0.0f), AY = AX, AZ = AX, PT = AX, ET = AX;
#pragma unroll GRAVITY_UNROLL
                for (int k = 0; k < JT; k += 2) {
                    const f2 DX = f2_fma(f2_lds(&s_x[wid][k]), NEG, XI);
                    const f2 DY = f2_fma(f2_lds(&s_y[wid][k]), NEG, YI);
                    const f2 DZ = f2_fma(f2_lds(&s_z[wid][k]), NEG, ZI);
                    const f2 M = f2_lds(&s_m[wid][k]);
                    const f2 R2 = f2_fma(DZ, DZ, f2_fma(DY, DY, f2_mul(DX, DX)));
                    const float2 ai = f2_get(f2_add(R2, EI));
                    const float2 aj = f2_get(f2_add(R2, f2_lds(&s_q[wid][k])));
                    const f2 REI = f2_make(rsqrt_r(ai.x), rsqrt_r(ai.y));
                    const f2 REJ = f2_make(rsqrt_r(aj.x), rsqrt_r(aj.y));
                    const f2 REI3 = f2_mul(f2_mul(REI, REI), REI);
                    const f2 REJ3 = f2_mul(f2_mul(REJ, REJ), REJ);
                    const f2 G = f2_mul(M, f2_add(REI3, REJ3));
                    PT = f2_fma(M, f2_add(REI, REJ), PT);
                    AX = f2_fma(DX, G, AX);
                    AY = f2_fma(DY, G, AY);
                    AZ = f2_fma(DZ, G, AZ);
                    ET = f2_fma(M, REI3, ET);
                }
                const float2 ax2 = f2_get(AX), ay2 = f2_get(AY), az2 = f2_get(AZ), pt2 = f2_get(PT), et2 = f2_get(ET);
                pax = -(R)(ax2.x + ax2.y);
                pay = -(R)(ay2.x + ay2.y);
                paz = -(R)(az2.x + az2.y);
                ppt = -(R)(pt2.x + pt2.y);
                pet = (R)(et2.x + et2.y);
            } else if (tpi == 1 && n == JT) {
#pragma unroll 8
                for (int k = 0; k < JT; ++k) pair(k);
            } else {
                for (int k = sub; k < n; k += tpi) pair(k);
            }
            ax.add(pax);
            ay.add(pay);
            az.add(paz);
            pt.add(ppt);
            et.add(pet);
            __syncwarp();
            while (qfill >= 32) {
                run_quad(32);
                qhead = (qhead + 32) & (QR - 1);
                qfill -= 32;
            }
        }
        if (qfill > 0) run_quad(qfill);
        const double sax = seg_sum(ax.value(), tpi), say = seg_sum(ay.value(), tpi);
        const double saz = seg_sum(az.value(), tpi), spt = seg_sum(pt.value(), tpi);
        const double set = seg_sum(et.value(), tpi);
        if (r.act && sub == 0) {
            const size_t o = ii + slice * a.o_stride;
            a.o_acc[3 * o + 0] = 0.5 * sax;
            a.o_acc[3 * o + 1] = 0.5 * say;
            a.o_acc[3 * o + 2] = 0.5 * saz;
            a.o_pot[o] = 0.5 * spt;
            a.o_eta[o] = set;
        }
    }
}

// ---------------------------------------------------------------- records
// Builders of the FP32C double-float records from FP64 arrays (one thread
// per particle).  Each fills hi/lo pairs; aux lanes as documented at the
// consumers above.
// Density records; lo.w: h rounded up.
__global__ inline void make_density_records(int n, const dbl4 *pm, const dbl4 *vel, const double *h, float4 *phi,
                                            float4 *plo, float4 *vhi, float4 *vlo) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        float4 a, b;
        row_record<false>(pm[k], h[k], a, b);
        phi[k] = a;
        plo[k] = b;
        velocity_record(vel[k], a, b);
        vhi[k] = a;
        vlo[k] = b;
    }
}

// Gravity records: hi = (x, y, z, mass), lo = (x, y, z, eps2).
__device__ __forceinline__ void gravity_record(const dbl4 &p, double mass, double eps2, float4 &hi, float4 &lo) {
    const float2 x = df_split(p.x), y = df_split(p.y), z = df_split(p.z);
    hi = make_float4(x.x, y.x, z.x, (float)mass);
    lo = make_float4(x.y, y.y, z.y, (float)eps2);
}
__global__ inline void make_gravity_records(int n, const dbl4 *pm, const double *eps2, float4 *phi, float4 *plo) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const dbl4 p = pm[k];
        float4 a, b;
        gravity_record(p, p.w, eps2[k], a, b);
        phi[k] = a;
        plo[k] = b;
    }
}

// Hydro records (layout in hydro_df.cuh): from h1 = (1/h, P, P Omega / rho^2,
// bswt / 2), h2 = (rho, c_s, alpha, alpha_u), h3 = (thrm, eta); 1/h, h^-4 and
// P Omega / rho^2 also as hi/lo splits of their FP64 values; and the mark
// records (hydro_mark_records).
struct HydroRecords {
    float4 phi, plo, vhi, vlo, g1, g2, g3, g4;
    __device__ __forceinline__ void fill(const dbl4 &p, const dbl4 &v, const dbl4 &a, const dbl4 &b, const double2 &c) {
        const float2 x = df_split(p.x), y = df_split(p.y), z = df_split(p.z);
        // (velocities beyond the FP32 range: infinite signal velocities, not NaN)
        const float2 u = df_split_far(v.x), w = df_split_far(v.y), s = df_split_far(v.z);
        const float2 P = df_split(a.y), T = df_split(c.x), Q = df_split(a.z);
        const double h4d = (a.x * a.x) * (a.x * a.x);
        const float2 H = df_split(a.x), H4 = df_split(h4d), M = df_split(p.w);
        phi = make_float4(x.x, y.x, z.x, M.x);
        plo = make_float4(x.y, y.y, z.y, M.y);
        vhi = make_float4(u.x, w.x, s.x, H.x);
        vlo = make_float4(u.y, w.y, s.y, H4.x);
        g1 = make_float4(P.x, P.y, Q.x, (float)a.w);
        g2 = make_float4((float)b.x, (float)b.y, (float)b.z, (float)b.w);
        g3 = make_float4(T.x, T.y, (float)c.y, Q.y);
        g4 = make_float4(H.x, H.y, H4.x, H4.y);
    }
};
__global__ inline void make_hydro_records(int n, const dbl4 *pm, const dbl4 *vel, const dbl4 *h1, const dbl4 *h2,
                                          const double2 *h3, float4 *phi, float4 *plo, float4 *vhi, float4 *vlo,
                                          float4 *g1, float4 *g2, float4 *g3, float4 *g4, float4 *mp, float4 *mv) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const dbl4 p = pm[k], v = vel[k], a = h1[k], b = h2[k];
        HydroRecords r;
        r.fill(p, v, a, b, h3[k]);
        phi[k] = r.phi; plo[k] = r.plo; vhi[k] = r.vhi; vlo[k] = r.vlo;
        g1[k] = r.g1; g2[k] = r.g2; g3[k] = r.g3; g4[k] = r.g4;
        float4 m0, m1;
        hydro_mark_records(p, v, a.x, b.y, m0, m1);
        mp[k] = m0;
        mv[k] = m1;
    }
}

}  // namespace sphk

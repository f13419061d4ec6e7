// density_rows.cuh — the density sums over per-particle neighbour rows.
//
// The functor of hdr_density.hpp:252-350: three fixed-point passes
// rho(h) -> h = eta ksrh (m / rho)^(1/3) from the first guess, then the
// gradient pass (grdh, divv, rotv) with the final h.
//
//   density_rows   eight lanes per particle over its row (mark_rows): the
//                  separations are formed once and kept in registers as
//                  (r, m), so the three passes read no memory; the gradient
//                  pass gathers the velocities.  A row holds every j within
//                  slack * (first guess of h): a particle whose h leaves that
//                  radius before the last pass is queued for the sweep.
//   density_sweep  one block per queued particle over its walk's whole list:
//                  particles without a row (overflow, very long lists, h
//                  outside the row range; many of them in an FP32C dispatch go
//                  to density_stream instead, in FP64 to density_sweep_warps),
//                  re-walks of few particles, and the FP64 recomputation of
//                  FP32C results whose search-radius decision is ambiguous.
//   density_sweep_warps  the same with a warp per particle (FP64).
//
// Bound: density_rows by the FP64 pipe (FP64) or by its launch and the latency of
// the rows (calls: 64 targets in 13 us where one warp per 32 targets took
// 100); eight lanes per particle keep a call of 64 on 16 warps and each pass at
// ~8 entries per lane (FP64 calls: a warp per particle).  density_sweep by the
// longest list of a batch (29k entries: 100 us, 150 without the distance test; a
// warp took 1.6 ms); indices a round ahead of the records, 8 entries in flight
// and no velocities beyond the support: 500k evaluation with five re-walks
// 10.29 -> 9.93 ms.  FP64: a step of 32 list entries holds two or three within
// reach, and the FP64 pipe takes a warp's instruction whole; collected and summed
// 32 at a time, a call of 64 without rows takes 135 us, 154 one by one.
//
// Both form the separations relative to the particle itself; FP32C sums a few
// terms in FP32, folds them into Kahan pairs per lane and adds the lanes with
// error-free transformations.
#pragma once

#include "rows.cuh"

namespace sphk {

struct DensityArgs {
    // FP64 records (i_pm is read in both modes for the i-particle's mass)
    const dbl4 *i_pm;       // x, y, z, mass
    const dbl4 *i_vel;      // vx, vy, vz, -
    const dbl4 *j_pm;
    const dbl4 *j_vel;
    // double-float positions (both modes: the sweep's distance test) and
    // velocities (FP32C)
    F32Part fi, fj;
    const long long *i_id;
    const long long *j_id;
    const double *i_ksr;    // first guess of h (DensityEPI::ksr)
    const double *i_rs;     // search radius (DensityEPI::rs)
    const int *i_list;      // null: particles [0, n_i)
    int n_i;
    const int *n_i_dev;     // when set, the particle count is read from device memory
    const int *j_off;       // per walk: [j_off[w], j_off[w+1]) in j index space
    const int *j_idx;       // null: entries are j indices themselves
    // rows (mark_rows)
    const int *rows;
    int2 *info;             // particles whose h leaves its row lose it
    int2 *ovf;              // sweep queue
    int *n_ovf;
    float slack;            // row radius over the first guess of h
    // when set: nothing runs while any of these error bits / this flag is set
    const int *err;
    int err_mask;
    const int *skip_rows;
    // bounds of the sweep's indices (n_j > 0: an index outside sets bounds_bit
    // in *err_out and that access is skipped)
    int n_j;
    long long list_cap;
    int *err_out;
    int bounds_bit;
    // outputs, indexed like the i arrays
    double *o_dens, *o_divv, *o_rotv, *o_grdh, *o_ksr;
    long long *o_np;
    unsigned char *o_itr;
    double eta_ksrh;        // eta * ksrh
    double ksr_max;         // clamp of h (+inf disables)
    const double *ksr_max_dev;  // when set, the clamp is read from device memory
    // FP32C only: particles whose final h lies within amb_tol of rs (where
    // the search-radius decision h > rs of hdr_density.hpp:299 could come out
    // differently in FP64) are queued here for an FP64 recomputation
    int *amb_count;         // null disables the queue
    int2 *amb;              // (particle, walk)
    int amb_cap;
    float amb_tol;
    // when set: pair evaluations performed, [0] the three density passes,
    // [1] the gradient pass
    unsigned long long *n_eval = nullptr;
    // when set: particle passes after the first (second, third, gradient)
    // [0] served from rows, [1] that swept the walk's j-list
    unsigned long long *n_pass = nullptr;
};

// Two-float sum of a value over the L lanes of a segment, every lane
// receiving the total (hi + lo); exact but for the rounding of lo.
struct sum2 {
    float h, l;
};
template <int L>
__device__ __forceinline__ sum2 lane_sum(sum2 v) {
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
        const float oh = __shfl_xor_sync(FULL, v.h, o), ol = __shfl_xor_sync(FULL, v.l, o);
        const float s = v.h + oh, b = s - v.h;
        const float e = (v.h - (s - b)) + (oh - b);
        v.l = (v.l + ol) + e;
        v.h = s;
    }
    return v;
}
template <int L>
__device__ __forceinline__ float lane_total(const Acc<false> &a) {
    const sum2 t = lane_sum<L>(sum2{a.s, -a.c});
    return t.h + t.l;
}
template <int L>
__device__ __forceinline__ double lane_total(const Acc<true> &a) {
    return seg_sum(a.s, L);
}

__device__ __forceinline__ float cbrt_r(float x) { return cbrtf(x); }
__device__ __forceinline__ double cbrt_r(double x) { return cbrt(x); }

// rho and the next h of one pass from its sum of m W0 / c0 (FP32C: FP32
// arithmetic, relative error ~1e-7)
template <typename R>
struct HState {
    R h, hinv, rho;
    bool clamped;
    __device__ __forceinline__ void start(double h0) {
        h = (R)h0;
        hinv = (R)1 / h;
        clamped = false;
    }
    __device__ __forceinline__ void update(R sum, R mass, R eta_ksrh, R ksr_max) {
        rho = (R)CEFF0 * hinv * hinv * hinv * sum;
        const R hn = eta_ksrh * cbrt_r(mass / rho);
        clamped = !(hn < ksr_max);   // also NaN, as the reference's comparison
        h = clamped ? ksr_max : hn;
        hinv = (R)1 / h;
    }
};

// Gradient-pass sums and one pair's terms (hdr_density.hpp:304-349).
template <bool F64>
struct GradSums {
    typedef typename Real<F64>::T R;
    Acc<F64> g, d, rx, ry, rz;
    R pg, pd, px, py, pz;
    __device__ __forceinline__ GradSums() : pg(0), pd(0), px(0), py(0), pz(0) {}
    // separation d, velocity difference u, mass m; self: equal ids
    __device__ __forceinline__ void add(R dx, R dy, R dz, R ux, R uy, R uz, R m, bool self, R hinv) {
        const R r2 = dx * dx + dy * dy + dz * dz;
        const R ri = self ? (R)0 : rsqrt_r(r2);
        const R q = r2 * ri * hinv;
        const R u = max0((R)1 - q);
        const R u2 = u * u;
        const R u3 = u2 * u;
        const R p14 = (R)1 + (R)4 * q;
        const R w0 = u2 * u2 * p14;               // W0 / c0
        const R w1 = w1_term(q, u, u2, u3, p14);  // W1 / c1
        pg += m * ((R)(3.0 * CEFF0) * w0 + (R)CEFF1 * q * w1);
        const R dw = m * w1 * ri;
        pd += (ux * dx + uy * dy + uz * dz) * dw;
        px += (uy * dz - uz * dy) * dw;
        py += (uz * dx - ux * dz) * dw;
        pz += (ux * dy - uy * dx) * dw;
    }
    __device__ __forceinline__ void fold() {
        g.add(pg);
        d.add(pd);
        rx.add(px);
        ry.add(py);
        rz.add(pz);
        pg = 0; pd = 0; px = 0; py = 0; pz = 0;
    }
};

// Omega, div v, |rot v| and the write-back of one particle.
template <typename R>
__device__ __forceinline__ void density_finish(const DensityArgs &a, int ii, int walk, const HState<R> &s, R sg, R sd,
                                               R sx, R sy, R sz, int np, double ksr_max) {
    const R hinv4 = s.hinv * s.hinv * s.hinv * s.hinv;
    const R rinv = (R)1 / s.rho;
    const R grdh = -hinv4 * sg;
    const R rx = (R)CEFF1 * hinv4 * sx, ry = (R)CEFF1 * hinv4 * sy, rz = (R)CEFF1 * hinv4 * sz;
    const R om = (R)1 / ((R)1 + s.h * rinv * grdh / (R)3);
    const R rot2 = rx * rx + ry * ry + rz * rz;
    const R rot = (rot2 != (R)0) ? sqrt(rot2) : (R)0;
    // the clamp itself is FP64
    const double h = s.clamped ? ksr_max : (double)s.h;
    const double rs_i = a.i_rs[ii];
    a.o_dens[ii] = (double)s.rho;
    a.o_divv[ii] = (double)(-(R)CEFF1 * hinv4 * sd * rinv * om);
    a.o_rotv[ii] = (double)(rot * rinv * om);
    a.o_grdh[ii] = (double)om;
    a.o_ksr[ii] = h;
    a.o_np[ii] = (long long)np;
    a.o_itr[ii] = h > rs_i ? 1 : 0;   // the search-radius decision, hdr_density.hpp:299
    if (a.amb_count && fabs(h - rs_i) <= (double)a.amb_tol * rs_i) {
        const int k = atomicAdd(a.amb_count, 1);
        if (k < a.amb_cap) a.amb[k] = make_int2(ii, walk);
    }
}

// j-particle q of particle i: separation (i - j), in the precision of the sums.
template <bool F64>
struct PairPos {
    typedef typename Real<F64>::T R;
    float4 hi, lo;   // FP32C
    dbl4 p;          // FP64
    __device__ __forceinline__ void load_i(const DensityArgs &a, int ii) {
        if constexpr (F64) {
            p = a.i_pm[ii];
        } else {
            hi = a.fi.phi[ii];
            lo = a.fi.plo[ii];
        }
    }
    __device__ __forceinline__ R rel(const DensityArgs &a, int j, R &dx, R &dy, R &dz) const {
        if constexpr (F64) return rel(a, j, hi, lo, dx, dy, dz);
        else return rel(a, j, __ldg(&a.fj.phi[j]), __ldg(&a.fj.plo[j]), dx, dy, dz);
    }
    // FP32C: (qh, ql) are j's records
    __device__ __forceinline__ R rel(const DensityArgs &a, int j, const float4 &qh, const float4 &ql, R &dx, R &dy,
                                     R &dz) const {
        if constexpr (F64) {
            const dbl4 q = a.j_pm[j];
            dx = p.x - q.x; dy = p.y - q.y; dz = p.z - q.z;
            return q.w;
        } else {
            dx = -df_diff(qh.x, ql.x, hi.x, lo.x);
            dy = -df_diff(qh.y, ql.y, hi.y, lo.y);
            dz = -df_diff(qh.z, ql.z, hi.z, lo.z);
            return qh.w;
        }
    }
};
template <bool F64>
struct PairVel {
    typedef typename Real<F64>::T R;
    float4 hi, lo;
    dbl4 v;
    __device__ __forceinline__ void load_i(const DensityArgs &a, int ii) {
        if constexpr (F64) {
            v = a.i_vel[ii];
        } else {
            hi = a.fi.vhi[ii];
            lo = a.fi.vlo[ii];
        }
    }
    // velocity difference; FP32C differences hi and lo parts apart, so that
    // it keeps FP32 relative accuracy across two colliding streams
    __device__ __forceinline__ void rel(const DensityArgs &a, int j, R &ux, R &uy, R &uz) const {
        if constexpr (F64) {
            const dbl4 w = a.j_vel[j];
            ux = v.x - w.x; uy = v.y - w.y; uz = v.z - w.z;
        } else {
            const float4 wh = __ldg(&a.fj.vhi[j]), wl = __ldg(&a.fj.vlo[j]);
            ux = (hi.x - wh.x) + (lo.x - wl.x);
            uy = (hi.y - wh.y) + (lo.y - wl.y);
            uz = (hi.z - wh.z) + (lo.z - wl.z);
        }
    }
};

template <typename R>
__device__ __forceinline__ R density_term(R q, R m) {   // m W0(q) / c0
    const R u = max0((R)1 - q);
    const R u2 = u * u;
    return m * (u2 * u2 * ((R)1 + (R)4 * q));
}

// q >= 1, not NaN; FP64 by the high word, off the FP64 pipe
__device__ __forceinline__ bool beyond(float q) { return q >= 1.0f; }
__device__ __forceinline__ bool beyond(double q) {
    return (unsigned)(__double2hiint(q) - 0x3ff00000) <= 0x7ff00000u - 0x3ff00000u;
}

constexpr int DROWS_LANES = 8;        // lanes per particle
constexpr int DROWS_THREADS = 128;
#ifndef SPH_DROWS_MIN_BLOCKS
#define SPH_DROWS_MIN_BLOCKS 4
#endif

// L lanes per particle: 8, or all 32 of the warp in small FP64 calls (warp_per_row).
template <bool F64, int L = DROWS_LANES>
__global__ void __launch_bounds__(DROWS_THREADS, F64 ? 2 : SPH_DROWS_MIN_BLOCKS) density_rows(const DensityArgs a) {
    typedef typename Real<F64>::T R;
    // a lane's entries, G groups of four: four consecutive ones of the row, or
    // (L = 32, one group) every 32nd, those beyond the row skipped
    constexpr int G = ROW_CAP / (4 * L);
    static_assert(L == 8 || (L == 32 && G == 1), "8 or 32 lanes");
    if (a.err && (*a.err & a.err_mask)) return;
    if (a.skip_rows && *a.skip_rows) return;
    const int n = a.n_i_dev ? *a.n_i_dev : a.n_i;
    const double ksr_max = a.ksr_max_dev ? *a.ksr_max_dev : a.ksr_max;
    const int lane = threadIdx.x & 31, sub = lane & (L - 1);
    const int per_warp = 32 / L;
    const int gw = (blockIdx.x * DROWS_THREADS + threadIdx.x) >> 5, nw = (gridDim.x * DROWS_THREADS) >> 5;
    unsigned ev_rows = 0, ev_swept = 0;   // of this lane's particles (sub 0): row entries; particles queued
    unsigned n_rows = 0;
    for (int k0 = gw * per_warp; k0 < n; k0 += nw * per_warp) {
        const int k = k0 + lane / L;
        const int ii = (k < n) ? (a.i_list ? a.i_list[k] : k) : -1;
        int2 inf = make_int2(ROW_CAP + 1, 0);
        if (ii >= 0) inf = a.info[ii];
        const bool row_ok = inf.x <= ROW_CAP;
        const int cnt = row_ok ? inf.x : 0;
        const int is = ii >= 0 ? ii : 0;
        const int cmax = (int)__reduce_max_sync(FULL, (unsigned)cnt);
        const double h0 = a.i_ksr[is];
        PairPos<F64> P;
        P.load_i(a, is);
        R mi;
        if constexpr (F64) mi = P.p.w;
        else mi = P.hi.w;
        const int *row = a.rows + (size_t)is * ROW_CAP;
        int4 jv[G];
        R r[4 * G], m[4 * G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            if (g * 4 * L < cmax) {
                const int e = g * 4 * L + 4 * sub;
                jv[g] = make_int4(-1, -1, -1, -1);
                if (L == 32) {
                    if (sub < cnt) jv[g].x = row[sub];
                    if (32 + sub < cnt) jv[g].y = row[32 + sub];
                    if (64 + sub < cnt) jv[g].z = row[64 + sub];
                    if (96 + sub < cnt) jv[g].w = row[96 + sub];
                } else if (e < cnt) {
                    jv[g] = *reinterpret_cast<const int4 *>(row + e);
                    if (e + 1 >= cnt) jv[g].y = -1;
                    if (e + 2 >= cnt) jv[g].z = -1;
                    if (e + 3 >= cnt) jv[g].w = -1;
                }
                int jj[4] = {jv[g].x, jv[g].y, jv[g].z, jv[g].w};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    R dx, dy, dz;
                    r[4 * g + u] = 0;
                    m[4 * g + u] = 0;   // a missing entry adds 0 * W0(0)
                    if (jj[u] >= 0) {
                        m[4 * g + u] = P.rel(a, jj[u], dx, dy, dz);
                        r[4 * g + u] = sqrt_r(dx * dx + dy * dy + dz * dz);
                        // at an infinite distance W0(q) would be 0 * inf
                        if (F64 && infinite(r[4 * g + u])) {
                            r[4 * g + u] = 0;
                            m[4 * g + u] = 0;
                            jj[u] = -1;
                        }
                    }
                }
                jv[g] = make_int4(jj[0], jj[1], jj[2], jj[3]);
            }
        }
        // three fixed-point passes, hdr_density.hpp:264-302
        HState<R> s;
        s.start(h0);
        // every pair with q < 1 is in the row while h stays below this
        const R h_row = (R)(h0 * (double)a.slack * 0.99998);
        bool valid = row_ok && s.h <= (R)(h0 * (double)a.slack);
        int np = 0;
#pragma unroll
        for (int pass = 0; pass < 3; ++pass) {
            Acc<F64> acc;
            int c = 0;
#pragma unroll
            for (int g = 0; g < G; ++g) {
                if (g * 4 * L < cmax) {
                    const int jj[4] = {jv[g].x, jv[g].y, jv[g].z, jv[g].w};
                    R part = 0;
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (L == 32 && 32 * u >= cmax) continue;
                        const R q = r[4 * g + u] * s.hinv;
                        const R sum = part + density_term(q, m[4 * g + u]);
                        part = beyond(q) ? part : sum;   // no term, whatever the mass
                        if (pass == 2) c += (jj[u] >= 0 && q < (R)1) ? 1 : 0;
                    }
                    acc.add(part);
                }
            }
            const R sum = (R)lane_total<L>(acc);
            if (pass == 2) {
                for (int o = L / 2; o > 0; o >>= 1) c += __shfl_xor_sync(FULL, c, o);
                np = c;
            }
            s.update(sum, mi, (R)a.eta_ksrh, (R)ksr_max);
            valid = valid && s.h >= (R)0 && s.h <= h_row;   // (h < 0, from a negative sum, has no radius)
        }
        // gradient pass with the final h, hdr_density.hpp:304-349
        GradSums<F64> gs;
        const long long idi = a.i_id[is];
        PairVel<F64> V;
        V.load_i(a, is);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            if (g * 4 * L < cmax) {
                const int jj[4] = {jv[g].x, jv[g].y, jv[g].z, jv[g].w};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (jj[u] >= 0 && r[4 * g + u] * s.hinv < (R)1.0001) {
                        R dx, dy, dz, ux, uy, uz;
                        const R mj = P.rel(a, jj[u], dx, dy, dz);
                        V.rel(a, jj[u], ux, uy, uz);
                        gs.add(dx, dy, dz, ux, uy, uz, mj, a.j_id[jj[u]] == idi, s.hinv);
                    }
                }
                gs.fold();
            }
        }
        const R sg = (R)lane_total<L>(gs.g), sd = (R)lane_total<L>(gs.d);
        const R sx = (R)lane_total<L>(gs.rx), sy = (R)lane_total<L>(gs.ry), sz = (R)lane_total<L>(gs.rz);
        if (sub == 0 && ii >= 0) {
            if (valid) {
                density_finish<R>(a, ii, inf.y, s, sg, sd, sx, sy, sz, np, ksr_max);
                ev_rows += (unsigned)cnt;
                ++n_rows;
            } else {
                ++ev_swept;
                if (row_ok) {
                    a.ovf[atomicAdd(a.n_ovf, 1)] = make_int2(ii, inf.y);
                    a.info[ii].x = ROW_CAP + 1;
                }
            }
        }
    }
    if (a.n_eval) {
        const unsigned e = __reduce_add_sync(FULL, ev_rows);
        const unsigned nr = __reduce_add_sync(FULL, n_rows), ns = __reduce_add_sync(FULL, ev_swept);
        if (lane == 0 && (nr | ns)) {
            atomicAdd(a.n_eval, 3ull * e);
            atomicAdd(a.n_eval + 1, (unsigned long long)e);
            atomicAdd(a.n_pass, 3ull * nr);
            atomicAdd(a.n_pass + 1, 3ull * ns);
        }
    }
}

constexpr int DSWEEP_THREADS = 256;
template <int N>
__device__ __forceinline__ void block_sum(double (&v)[N], double (*red)[DSWEEP_THREADS / 32]) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < N; ++q) {
        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(FULL, v[q], o);
        if (lane == 0) red[q][wid] = v[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < N; ++q) {
        double t = 0.0;
        for (int u = 0; u < DSWEEP_THREADS / 32; ++u) t += red[q][u];
        v[q] = t;
    }
    __syncthreads();
}

// queue / n_queue: (particle, walk) to sweep (n_queue capped at queue_cap;
// with more than `most` in FP32C nothing, in FP64 the lists that are left by
// density_sweep_warps); total (optional): the count is added to it.
#ifndef SPH_SWEEP_U
#define SPH_SWEEP_U 8
#endif
// FP64: longest list of a queue of n that a warp takes: up to 12 n entries, but
// not so many that a warp would need longer for it than the chip for the rest of
// the queue (n), or 0.2 ms (16384).  50k FP64 steps, whose few hundred particles
// without rows have lists of up to 50k: 27.7 ms; with 16384 for every queue 40.4.
__device__ __forceinline__ int sweep_long(int n) { return n < 1366 ? 12 * n : (n > 16384 ? n : 16384); }
template <bool F64>
__global__ void __launch_bounds__(DSWEEP_THREADS) density_sweep(const DensityArgs a, const int2 *queue,
                                                               const int *n_queue, int queue_cap, int *total,
                                                               int most = 0x7fffffff) {
    typedef typename Real<F64>::T R;
    constexpr int T = DSWEEP_THREADS, U = SPH_SWEEP_U;   // U list entries per thread in flight
    constexpr int RING = 512;                            // < 32 left over + a round of 32 U
    static_assert(32 * (U + 1) <= RING, "hits of a round");
    __shared__ double red[5][T / 32];
    __shared__ int s_hit[F64 ? T / 32 : 1][RING];        // a warp's entries within reach
    __shared__ int s_todo[F64 ? T : 1], s_n;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned lt = lanemask_lt();
    if (a.err && (*a.err & a.err_mask)) return;
    const int nq = min(*n_queue, queue_cap);
    const bool many = *n_queue > most;
    if (!F64 && many) return;
    if (total && blockIdx.x == 0 && threadIdx.x == 0) *total += *n_queue;
    const double ksr_max = a.ksr_max_dev ? *a.ksr_max_dev : a.ksr_max;
    // many: of T particles of the queue at a time those with the longest lists
    const int step = many ? T : 1, nj_warp = sweep_long(nq);
    for (int e0 = blockIdx.x; e0 < nq; e0 += gridDim.x * step)
    for (int td = 0;; ++td) {
        int e = e0;
        if (many) {
            if (td == 0) {
                __syncthreads();
                if (threadIdx.x == 0) s_n = 0;
                __syncthreads();
                const int k = e0 + threadIdx.x * gridDim.x;
                if (F64 && k < nq) {
                    const int w = queue[k].y;
                    if (a.j_off[w + 1] - a.j_off[w] > nj_warp) s_todo[atomicAdd(&s_n, 1)] = k;
                }
                __syncthreads();
            }
            if (td >= s_n) break;
            e = s_todo[F64 ? td : 0];
        } else if (td > 0) {
            break;
        }
        const int2 pw = queue[e];
        const int ii = pw.x;
        if (a.n_j > 0 && (ii < 0 || ii >= a.n_j)) {
            if (threadIdx.x == 0) atomicOr(a.err_out, a.bounds_bit);
            continue;   // block-uniform
        }
        const int jb = a.j_off[pw.y], je = a.j_off[pw.y + 1];
        if (a.n_j > 0 && (jb < 0 || je < jb || (long long)je > a.list_cap)) {
            if (threadIdx.x == 0) atomicOr(a.err_out, a.bounds_bit);
            continue;   // block-uniform
        }
        PairPos<F64> P;
        P.load_i(a, ii);
        const float4 ph = a.fi.phi[ii], pl = a.fi.plo[ii];
        const double mi = a.i_pm[ii].w;
        // visits the list entries; FP64: those that can lie within h of the
        // particle by an FP32 distance test on the double-float positions,
        // with the margins of mark_rows (h outside its range: every entry), 32
        // at a time; in FP32C f itself tests.  A coordinate that is NaN counts
        // as the particle's own, as in the box test of mark_rows.  Indices are
        // read a round ahead of the records.
        auto over_list = [&](R h, auto &&f) {
            const float hf = (float)h;
            const float pad = 3.0e-14f * (fabsf(ph.x) + fabsf(ph.y) + fabsf(ph.z));
            const float rad = hf * 1.0001f + pad;
            const bool test = F64 && hf >= ROW_HMIN && hf <= ROW_HMAX;
            const float lim = test ? rad * rad : INFINITY;
            int next[U];
            auto indices = [&](int k0) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int k = k0 + u * T;
                    next[u] = (k < je) ? (a.j_idx ? a.j_idx[k] : k) : -1;
                }
            };
            int head = 0, fill = 0;
            indices(jb + threadIdx.x);
            for (int b = jb + 32 * wid; b < je; b += T * U) {
                int j[U];
                float4 qh[U], ql[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    j[u] = next[u];
                    if (a.n_j > 0 && j[u] >= a.n_j) {
                        atomicOr(a.err_out, a.bounds_bit);
                        j[u] = -1;
                    }
                    if (j[u] >= 0) {
                        qh[u] = __ldg(&a.fj.phi[j[u]]);
                        ql[u] = __ldg(&a.fj.plo[j[u]]);
                    }
                }
                indices(b + lane + T * U);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if constexpr (F64) {
                        bool hit = j[u] >= 0;
                        if (hit) {
                            const float dx = df_diff(qh[u].x, ql[u].x, ph.x, pl.x);
                            const float dy = df_diff(qh[u].y, ql[u].y, ph.y, pl.y);
                            const float dz = df_diff(qh[u].z, ql[u].z, ph.z, pl.z);
                            hit = !(square_sum(dx, dy, dz) > lim);
                        }
                        const unsigned m = __ballot_sync(FULL, hit);
                        if (hit) s_hit[wid][(head + fill + __popc(m & lt)) & (RING - 1)] = j[u];
                        fill += __popc(m);
                    } else if (j[u] >= 0) {
                        f(j[u], qh[u], ql[u]);
                    }
                }
                if constexpr (F64) {
                    __syncwarp();
                    for (; fill >= 32; fill -= 32, head += 32) f(s_hit[wid][(head + lane) & (RING - 1)], ph, pl);
                    __syncwarp();
                }
            }
            if constexpr (F64) {
                if (lane < fill) f(s_hit[wid][(head + lane) & (RING - 1)], ph, pl);
                __syncwarp();
            }
        };
        // farther than r2_far; a coordinate that is NaN counts as zero
        auto far_off = [](R r2, R dx, R dy, R dz, R r2_far) {
            return r2 > r2_far || (r2 != r2 && square_sum(dx, dy, dz) > r2_far);
        };
        // Terms beyond the support are zero, whatever the mass, and need no
        // velocity; in FP32C a run of them folds one zero (further ones leave
        // the sums as they are).
        HState<R> s;
        s.start(a.i_ksr[ii]);
        int np = 0;
        for (int pass = 0; pass < 3; ++pass) {
            Acc<F64> acc;
            int cnt = 0;
            const R hinv2 = s.hinv * s.hinv, r2_far = (R)1.0002 * s.h * s.h;
            bool zero = false;
            over_list(s.h, [&](int j, const float4 &qh, const float4 &ql) {
                R dx, dy, dz;
                const R m = P.rel(a, j, qh, ql, dx, dy, dz), r2 = dx * dx + dy * dy + dz * dz;
                if (far_off(r2, dx, dy, dz, r2_far)) {
                    if (!F64 && !zero) acc.add((R)0);
                    zero = true;
                    return;
                }
                zero = false;
                const R q = sqrt_q(r2, hinv2);
                cnt += (q < (R)1) ? 1 : 0;
                acc.add(density_term(q, m));
            });
            double v[2] = {acc.value(), (double)cnt};
            block_sum(v, red);
            np = (int)v[1];
            s.update((R)v[0], (R)mi, (R)a.eta_ksrh, (R)ksr_max);
        }
        GradSums<F64> gs;
        const long long idi = a.i_id[ii];
        PairVel<F64> V;
        V.load_i(a, ii);
        const R r2_far = (R)1.0002 * s.h * s.h;
        bool zero = false;
        over_list(s.h, [&](int j, const float4 &qh, const float4 &ql) {
            R dx, dy, dz, ux, uy, uz;
            const R m = P.rel(a, j, qh, ql, dx, dy, dz), r2 = dx * dx + dy * dy + dz * dz;
            if (far_off(r2, dx, dy, dz, r2_far)) {
                if (!F64 && !zero) gs.fold();
                zero = true;
                return;
            }
            zero = false;
            V.rel(a, j, ux, uy, uz);
            gs.add(dx, dy, dz, ux, uy, uz, m, a.j_id[j] == idi, s.hinv);
            gs.fold();
        });
        double v[5] = {gs.g.value(), gs.d.value(), gs.rx.value(), gs.ry.value(), gs.rz.value()};
        block_sum(v, red);
        if (threadIdx.x == 0) {
            density_finish<R>(a, ii, pw.y, s, (R)v[0], (R)v[1], (R)v[2], (R)v[3], (R)v[4], np, ksr_max);
            if (a.n_eval) {
                atomicAdd(a.n_eval, 3ull * (unsigned long long)(je - jb));
                atomicAdd(a.n_eval + 1, (unsigned long long)(je - jb));
            }
        }
    }
}

// FP64: a warp per queued particle where there are many (more than `least`) and
// its list is not far longer than the others' (sweep_long).  Entries within
// 1.1 h are kept in shared memory for the passes whose h stays within that;
// SWEEP_CAP hold 125 neighbours four times.
// Bound by FP64 pairs and the latency of the list's records (a block of
// density_sweep fills an SM and waits for both and for its barriers).  Density of
// 200k particles at 125 neighbours 58.7 -> 12.6 ms (36.0 by the lists before rows;
// 17.7 at 12 warps per SM, 13.4 at 20), with a first guess of h 20% low at 55
// neighbours 134 -> 23 ms (42.7).
constexpr int SWEEP_CAP = 512, SWEEP_WARPS = 4;
__global__ inline void __launch_bounds__(SWEEP_WARPS * 32, 4)
density_sweep_warps(const DensityArgs a, const int2 *queue, const int *n_queue, int queue_cap, int least) {
    constexpr int U = 4;   // list entries per lane in flight
    static_assert(SWEEP_CAP >= 64 * U, "a round of hits and the room for another");
    __shared__ int s_hit[SWEEP_WARPS][SWEEP_CAP];
    if (a.err && (*a.err & a.err_mask)) return;
    if (*n_queue <= least) return;
    const int nq = min(*n_queue, queue_cap), nj_warp = sweep_long(nq);
    const double ksr_max = a.ksr_max_dev ? *a.ksr_max_dev : a.ksr_max;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned lt = lanemask_lt();
    int *hits = s_hit[wid];
    for (int e = blockIdx.x * SWEEP_WARPS + wid; e < nq; e += gridDim.x * SWEEP_WARPS) {
        const int2 pw = queue[e];
        const int ii = pw.x;
        if (a.n_j > 0 && (ii < 0 || ii >= a.n_j)) {
            if (lane == 0) atomicOr(a.err_out, a.bounds_bit);
            continue;   // warp-uniform
        }
        const int jb = a.j_off[pw.y], je = a.j_off[pw.y + 1];
        if (je - jb > nj_warp) continue;
        if (a.n_j > 0 && (jb < 0 || je < jb || (long long)je > a.list_cap)) {
            if (lane == 0) atomicOr(a.err_out, a.bounds_bit);
            continue;   // warp-uniform
        }
        PairPos<true> P;
        P.load_i(a, ii);
        const float4 ph = a.fi.phi[ii], pl = a.fi.plo[ii];
        const float pad = 3.0e-14f * (fabsf(ph.x) + fabsf(ph.y) + fabsf(ph.z));
        int n = 0;            // hits
        double h_hits = -1.0;   // all within this radius are there
        // f(j) for the entries that can lie within h, as in density_sweep
        auto over_list = [&](double h, auto &&f) {
            const bool scan = !(h >= 0.0 && h <= h_hits);
            bool all = true;
            float lim = INFINITY;
            int b = jb;
            if (scan) {
                const float hf = (float)(1.1 * h), rad = hf * 1.0001f + pad;
                if (hf >= ROW_HMIN && hf <= ROW_HMAX) lim = rad * rad;
                n = 0;
            }
            for (bool last = false; !last;) {
                if (scan && b < je) {
                    int j[U];
                    float4 qh[U], ql[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int k = b + 32 * u + lane;
                        j[u] = k < je ? (a.j_idx ? a.j_idx[k] : k) : -1;
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        if (a.n_j > 0 && j[u] >= a.n_j) {
                            atomicOr(a.err_out, a.bounds_bit);
                            j[u] = -1;
                        }
                        if (j[u] >= 0) {
                            qh[u] = __ldg(&a.fj.phi[j[u]]);
                            ql[u] = __ldg(&a.fj.plo[j[u]]);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        bool hit = j[u] >= 0;
                        if (hit) {
                            const float dx = df_diff(qh[u].x, ql[u].x, ph.x, pl.x);
                            const float dy = df_diff(qh[u].y, ql[u].y, ph.y, pl.y);
                            const float dz = df_diff(qh[u].z, ql[u].z, ph.z, pl.z);
                            hit = !(square_sum(dx, dy, dz) > lim);
                        }
                        const unsigned m = __ballot_sync(FULL, hit);
                        if (hit) hits[n + __popc(m & lt)] = j[u];
                        n += __popc(m);
                    }
                    b += 32 * U;
                    __syncwarp();
                }
                last = !scan || b >= je;
                if (last || n > SWEEP_CAP - 32 * U) {
                    for (int k = lane; k < n; k += 32) f(hits[k]);
                    if (!last) {
                        n = 0;
                        all = false;
                    }
                    __syncwarp();
                }
            }
            if (scan) h_hits = all && lim < INFINITY ? 1.1 * h : -1.0;
        };
        auto far_off = [](double r2, double dx, double dy, double dz, double r2_far) {
            return r2 > r2_far || (r2 != r2 && square_sum(dx, dy, dz) > r2_far);
        };
        HState<double> s;
        s.start(a.i_ksr[ii]);
        int np = 0;
        for (int pass = 0; pass < 3; ++pass) {
            double sum = 0.0;
            int cnt = 0;
            const double hinv2 = s.hinv * s.hinv, r2_far = 1.0002 * s.h * s.h;
            over_list(s.h, [&](int j) {
                double dx, dy, dz;
                const double m = P.rel(a, j, dx, dy, dz), r2 = dx * dx + dy * dy + dz * dz;
                if (far_off(r2, dx, dy, dz, r2_far)) return;
                const double q = sqrt_q(r2, hinv2);
                cnt += (q < 1.0) ? 1 : 0;
                sum += density_term(q, m);
            });
            np = __reduce_add_sync(FULL, cnt);
            s.update(seg_sum(sum, 32), P.p.w, a.eta_ksrh, ksr_max);
        }
        GradSums<true> gs;
        const long long idi = a.i_id[ii];
        PairVel<true> V;
        V.load_i(a, ii);
        const double r2_far = 1.0002 * s.h * s.h;
        over_list(s.h, [&](int j) {
            double dx, dy, dz, ux, uy, uz;
            const double m = P.rel(a, j, dx, dy, dz), r2 = dx * dx + dy * dy + dz * dz;
            if (far_off(r2, dx, dy, dz, r2_far)) return;
            V.rel(a, j, ux, uy, uz);
            gs.add(dx, dy, dz, ux, uy, uz, m, a.j_id[j] == idi, s.hinv);
        });
        gs.fold();
        const double sg = seg_sum(gs.g.value(), 32), sd = seg_sum(gs.d.value(), 32);
        const double sx = seg_sum(gs.rx.value(), 32), sy = seg_sum(gs.ry.value(), 32), sz = seg_sum(gs.rz.value(), 32);
        if (lane == 0) {
            density_finish<double>(a, ii, pw.y, s, sg, sd, sx, sy, sz, np, ksr_max);
            if (a.n_eval) {
                atomicAdd(a.n_eval, 3ull * (unsigned long long)(je - jb));
                atomicAdd(a.n_eval + 1, (unsigned long long)(je - jb));
            }
        }
    }
}

}  // namespace sphk

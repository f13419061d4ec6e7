// capi.cu — the C ABI of include/sph_gb300.h: contexts, the single-group
// functors and the batched Dispatch/Retrieve pairs.
//
// Data path of one dispatch (one CUDA stream per context):
//   host  : offsets, work items and the walk arrays into one pinned buffer
//           [offsets | items | EPI | EPJ], large ones by several threads
//   device: a kernel copies the buffer in, a segment at a time while the host
//           fills the next; one kernel turns the reference AoS structs into
//           records; the pair kernels; a pack kernel writes the reference Force
//           structs to pinned memory (finite check)
//   Retrieve waits on the stream and copies to the caller's per-walk arrays.
//
// One thread's memcpy into the buffer took 5 of a 7 ms dispatch of 64 MB.  The
// device can read pageable arrays where they are (0.33 ms), but its first
// access to a 4 MB region of memory that was freed and mapped again costs a
// fault of 0.6 ms: up to 18 ms for fresh arrays scattered over the heap.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstddef>
#include <cstdio>
#include <cstring>
#include <limits>
#include <new>
#include <vector>

#include "../../include/sph_gb300.h"
#include "capi_internal.h"
#include "host_copy.h"
#include "pair_kernels.cuh"

// ---- ABI layout checks: the reference classes' member order and padding ----
#define SPH_OFF(T, f, v) static_assert(offsetof(T, f) == (v), #T "::" #f " offset")
SPH_OFF(sph_DensityEPI, id, 0); SPH_OFF(sph_DensityEPI, mass, 8); SPH_OFF(sph_DensityEPI, pos, 16);
SPH_OFF(sph_DensityEPI, vel, 40); SPH_OFF(sph_DensityEPI, ksr, 64); SPH_OFF(sph_DensityEPI, rs, 72);
static_assert(sizeof(sph_DensityEPI) == 80, "DensityEPI size");
SPH_OFF(sph_DensityEPJ, mass, 8); SPH_OFF(sph_DensityEPJ, vel, 40);
static_assert(sizeof(sph_DensityEPJ) == 64, "DensityEPJ size");
SPH_OFF(sph_Density, ksr, 32); SPH_OFF(sph_Density, np, 40); SPH_OFF(sph_Density, itr, 48);
static_assert(sizeof(sph_Density) == 56, "Density size");
SPH_OFF(sph_HydroEPI, pos, 8); SPH_OFF(sph_HydroEPI, ksr, 56); SPH_OFF(sph_HydroEPI, eta, 136);
static_assert(sizeof(sph_HydroEPI) == 144, "HydroEPI size");
SPH_OFF(sph_HydroEPJ, mass, 8); SPH_OFF(sph_HydroEPJ, ksr, 64); SPH_OFF(sph_HydroEPJ, eta, 144);
static_assert(sizeof(sph_HydroEPJ) == 152, "HydroEPJ size");
SPH_OFF(sph_Hydro, accg, 24); SPH_OFF(sph_Hydro, diffu, 64);
static_assert(sizeof(sph_Hydro) == 72, "Hydro size");
static_assert(sizeof(sph_GravityEPI) == 32 && sizeof(sph_GravityEPJ) == 40 &&
              sizeof(sph_GravitySPJ) == 40 && sizeof(sph_Gravity) == 40, "gravity sizes");
SPH_OFF(sph_GravityEPJ, pos, 8); SPH_OFF(sph_GravityEPJ, eps2, 32); SPH_OFF(sph_Gravity, eta, 32);

using sphk::WorkItem;

namespace sphrt {

// Relative band |h - rs| <= AMB_TOL * rs in which an FP32C density result is
// recomputed in FP64 (FP32 h carries ~1e-7 relative error).
const float AMB_TOL = 4.0e-6f;

int set_error(sph_context *ctx, int status, const char *fmt, ...) {
    if (ctx) {
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(ctx->err, sizeof(ctx->err), fmt, ap);
        va_end(ap);
    }
    return status;
}

int cuda_error(sph_context *ctx, cudaError_t e, const char *what) {
    return set_error(ctx, SPH_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

template <class K>
static int occupancy_grid(K kernel, int threads, int sm_count, int *out) {
    int nb = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, threads, 0);
    if (e != cudaSuccess) return (int)e;
    *out = std::max(1, nb) * sm_count;
    return 0;
}

int init_grids(sph_context *ctx) {
    const int th = PAIR_WARPS * 32;
    int e = 0;
    e |= occupancy_grid(sphk::mark_rows<sphk::ROWS_DENSITY, PAIR_WARPS>, th, ctx->sm_count, &ctx->grid[0][0]);
    e |= occupancy_grid(sphk::density_stream<PAIR_WARPS>, th, ctx->sm_count, &ctx->grid_stream);
    ctx->grid[0][1] = ctx->grid[0][0];   // the rows are marked in FP32 in both precisions
    e |= occupancy_grid(sphk::mark_rows<sphk::ROWS_HYDRO32, PAIR_WARPS>, th, ctx->sm_count, &ctx->grid[1][0]);
    e |= occupancy_grid(sphk::mark_rows<sphk::ROWS_HYDRO64, PAIR_WARPS>, th, ctx->sm_count, &ctx->grid[1][1]);
    e |= occupancy_grid(sphk::gravity_kernel<false, PAIR_WARPS>, th, ctx->sm_count, &ctx->grid[2][0]);
    e |= occupancy_grid(sphk::gravity_kernel<true, PAIR_WARPS>, th, ctx->sm_count, &ctx->grid[2][1]);
    e |= occupancy_grid(sphk::hydro_df_lists, sphk::HYDRO_DF_THREADS, ctx->sm_count, &ctx->grid_df);
    e |= occupancy_grid(sphk::gravity_kernel<false, PAIR_WARPS, 64>, th, ctx->sm_count, &ctx->grid_g64);
    return e;
}

int pair_grid(const sph_context *ctx, int kind, int precision, int n_items) {
    const int full = ctx->grid[kind][precision == SPH_PREC_FP64 ? 1 : 0];
    const int need = (n_items + PAIR_WARPS - 1) / PAIR_WARPS;
    return std::max(1, std::min(full, need));
}

// Long items run beside the others: first(side stream), then rest(s), joined
// after both (in a capture the two become parallel branches).  One block per
// SM takes half of its registers; the items of the usual kind fill the rest.
template <class A, class B>
static void beside(const LongSide &side, cudaStream_t s, A first, B rest) {
    cudaEventRecord(side.fork, s);
    cudaStreamWaitEvent(side.stream, side.fork, 0);
    first(side.stream);
    cudaEventRecord(side.join, side.stream);
    rest(s);
    cudaStreamWaitEvent(s, side.join, 0);
}

// The queued long items: a block each.
template <int KIND>
static void mark_long(const sph_context *ctx, const sphk::MarkArgs &m, int n_max, cudaStream_t s) {
    constexpr int W = KIND == sphk::ROWS_DENSITY ? sphk::MARK_LONG_WARPS : sphk::HYDRO_LONG_WARPS;
    sphk::mark_rows<KIND, W, true><<<std::max(1, std::min(n_max, 2 * ctx->sm_count)), W * 32, 0, s>>>(m);
}

// Rows of the items of m and of its long items: beside them where the caller
// has queued them and gives a side stream, else after the kernel that queues
// them (push_long).  No long items without either.
template <int KIND>
static void mark_all(const sph_context *ctx, const sphk::MarkArgs &m, int grid, int n_max, cudaStream_t s,
                     const LongSide *side) {
    auto usual = [&](cudaStream_t t) {
        sphk::mark_rows<KIND, PAIR_WARPS><<<grid, PAIR_WARPS * 32, 0, t>>>(m);
    };
    auto lng = [&](cudaStream_t t) { mark_long<KIND>(ctx, m, n_max, t); };
    if (side) {
        beside(*side, s, lng, usual);
    } else {
        usual(s);
        if (m.push_long) lng(s);
    }
}

// FP64 recomputation of the FP32C results queued as ambiguous (their number
// is added to amb_total).
static void recheck_density(const sph_context *ctx, const sphk::DensityArgs &a, int n_max, cudaStream_t s,
                            int *amb_total) {
    sphk::DensityArgs f = a;
    f.amb_count = nullptr;
    f.n_eval = nullptr;
    sphk::density_sweep<true><<<std::max(1, std::min(n_max, ctx->sm_count)), sphk::DSWEEP_THREADS, 0, s>>>(
        f, a.amb, a.amb_count, a.amb_cap, amb_total);
}

// FP64 rows of up to 8 particles per SM are summed by a whole warp each: their
// chain of dependent FP64 operations is what such a call waits for.  A call of one
// target: density 93.9 us with eight lanes, 71.3 so (78.1 by the list, before
// rows); hydro 82.3 and 67.1 (66.3).  1000 targets: 197 and 189, hydro 391 and
// 381; at 2000 the FP64 pipe is busy with either (326 and 358, 819 and 820).
static bool warp_per_row(const sph_context *ctx, int n) { return n <= 8 * ctx->sm_count; }

// The density sums of the particles of a.i_list (at most n_max) over their
// rows, the sweep of the queued particles and, in FP32C, the FP64
// recomputation of the ambiguous ones.  *a.n_ovf and *a.amb_count hold the
// queues' counts.
static void launch_density_sums(const sph_context *ctx, const sphk::DensityArgs &a, int n_max, int precision,
                                cudaStream_t s, int *amb_total, const RowlessItems *rowless) {
    const bool whole_warp = precision == SPH_PREC_FP64 && warp_per_row(ctx, n_max);
    const int per_block = sphk::DROWS_THREADS / (whole_warp ? 32 : sphk::DROWS_LANES);
    const int rg = std::max(1, std::min((n_max + per_block - 1) / per_block, ctx->sm_count * 16));
    const int sg = std::max(1, std::min(n_max, ctx->sm_count * 6));
    if (precision == SPH_PREC_FP64) {
        if (whole_warp)
            sphk::density_rows<true, 32><<<rg, sphk::DROWS_THREADS, 0, s>>>(a);
        else
            sphk::density_rows<true><<<rg, sphk::DROWS_THREADS, 0, s>>>(a);
        // More particles without a row than SMs: a warp each.  Calls (list of
        // ~1100 to 4500) of 128: 146 us by warps and 135 by blocks; of 256: 166 and
        // 183, of 600: 217 and 300; of 4096 (~12500) 1.2 and 2.4 ms.
        const int most = ctx->sm_count;
        if (n_max > most)
            sphk::density_sweep_warps<<<std::min(n_max / sphk::SWEEP_WARPS + 1, 4 * ctx->sm_count),
                                        sphk::SWEEP_WARPS * 32, 0, s>>>(a, a.ovf, a.n_ovf, n_max, most);
        sphk::density_sweep<true><<<sg, sphk::DSWEEP_THREADS, 0, s>>>(a, a.ovf, a.n_ovf, n_max, nullptr, most);
        return;
    }
    sphk::density_rows<false><<<rg, sphk::DROWS_THREADS, 0, s>>>(a);
    const int most = rowless ? rowless->most : 0x7fffffff;
    sphk::density_sweep<false><<<sg, sphk::DSWEEP_THREADS, 0, s>>>(a, a.ovf, a.n_ovf, n_max, nullptr, most);
    if (rowless) {
        const RowlessItems &r = *rowless;
        sphk::rowless_items<<<std::max(1, std::min((r.n_walk + 3) / 4, 8 * ctx->sm_count)), 128, 0, s>>>(
            r.n_walk, r.i_off, a.j_off, a.info, a.n_ovf, most, r.list, r.items, r.n_items);
        sphk::StreamArgs w{};
        w.i_pm = a.i_pm; w.fi = a.fi; w.fj = a.fj; w.i_id = a.i_id; w.j_id = a.j_id;
        w.i_ksr = a.i_ksr; w.i_rs = a.i_rs;
        w.items = r.items; w.n_items_dev = r.n_items; w.j_off = a.j_off; w.j_idx = a.j_idx;
        w.i_list = r.list; w.queue = r.queue;
        w.o_dens = a.o_dens; w.o_divv = a.o_divv; w.o_rotv = a.o_rotv; w.o_grdh = a.o_grdh; w.o_ksr = a.o_ksr;
        w.o_np = a.o_np; w.o_itr = a.o_itr;
        w.eta_ksrh = a.eta_ksrh; w.ksr_max = a.ksr_max; w.ksr_max_dev = a.ksr_max_dev;
        w.amb_count = a.amb_count; w.amb = a.amb; w.amb_cap = a.amb_cap; w.amb_tol = a.amb_tol;
        sphk::density_stream<PAIR_WARPS><<<ctx->grid_stream, PAIR_WARPS * 32, 0, s>>>(w);
    }
    recheck_density(ctx, a, n_max, s, amb_total);
}

// Density rows of the items of m.
void launch_mark_density(const sph_context *ctx, const sphk::MarkArgs &m, int mark_grid, int n_max, cudaStream_t s,
                         const LongSide *side) {
    mark_all<sphk::ROWS_DENSITY>(ctx, m, mark_grid, n_max, s, side);
}

// Rows of the items of m, then the density sums over them.
void launch_density(const sph_context *ctx, const sphk::MarkArgs &m, int mark_grid, const sphk::DensityArgs &a,
                    int n_max, int precision, cudaStream_t s, int *amb_total, const LongSide *side,
                    const RowlessItems *rowless) {
    launch_mark_density(ctx, m, mark_grid, n_max, s, side);
    launch_density_sums(ctx, a, n_max, precision, s, amb_total, rowless);
}

// The FP32C density of a particle system (n_max particles): the streamed walk
// over the items of w (those with long lists a block each), the sweep of the queued particles (re-walks of few) and
// the FP64 recomputation of the ambiguous ones.
void launch_density_stream(const sph_context *ctx, const sphk::StreamArgs &w, bool sweep, const sphk::DensityArgs &a,
                           int n_max, cudaStream_t s, int *amb_total, const LongSide &side) {
    beside(
        side, s,
        [&](cudaStream_t t) {
            sphk::density_stream<sphk::STREAM_LONG_WARPS, true>
                <<<std::max(1, std::min(n_max, 2 * ctx->sm_count)), sphk::STREAM_LONG_WARPS * 32, 0, t>>>(w);
        },
        [&](cudaStream_t t) { sphk::density_stream<PAIR_WARPS><<<ctx->grid_stream, PAIR_WARPS * 32, 0, t>>>(w); });
    if (sweep)
        sphk::density_sweep<false><<<std::max(1, std::min(n_max, ctx->sm_count * 6)), sphk::DSWEEP_THREADS, 0, s>>>(
            a, a.ovf, a.n_ovf, n_max, nullptr);
    recheck_density(ctx, a, n_max, s, amb_total);
}

// Hydro: signal velocities and rows of the items of m, then the pair sums
// over them (FP32C: the double-float pass) and over the lists of the particles
// without a row.  *a.n_ovf and *m.longs.n must be zero at launch.
void launch_hydro_marks(const sph_context *ctx, const sphk::MarkArgs &m, int mark_grid, int n_i, int precision,
                        cudaStream_t s, const LongSide *side) {
    if (precision == SPH_PREC_FP64)
        mark_all<sphk::ROWS_HYDRO64>(ctx, m, mark_grid, n_i, s, side);
    else
        mark_all<sphk::ROWS_HYDRO32>(ctx, m, mark_grid, n_i, s, side);
}

void launch_hydro_sums(const sph_context *ctx, const sphk::HydroArgs &a, int precision, cudaStream_t s) {
    if (a.n_i <= 0) return;
    if (precision == SPH_PREC_FP64) {
        const bool whole_warp = warp_per_row(ctx, a.n_i);
        const int per_block = sphk::HROWS_THREADS / (whole_warp ? 32 : sphk::HROWS_LANES);
        const int grid = std::max(1, std::min((a.n_i + per_block - 1) / per_block, 16 * ctx->sm_count));
        if (whole_warp)
            sphk::hydro64_rows<32><<<grid, sphk::HROWS_THREADS, 0, s>>>(a);
        else
            sphk::hydro64_rows<sphk::HROWS_LANES><<<grid, sphk::HROWS_THREADS, 0, s>>>(a);
        sphk::hydro64_sweep<<<std::max(1, std::min(a.n_i, 2 * ctx->sm_count)), sphk::DSWEEP_THREADS, 0, s>>>(a);
        return;
    }
    const int need = (a.n_i + sphk::HYDRO_DF_THREADS - 1) / sphk::HYDRO_DF_THREADS;
    sphk::hydro_df_lists<<<std::max(1, std::min(need, ctx->grid_df)), sphk::HYDRO_DF_THREADS, 0, s>>>(a);
    // one block per particle without a row, up to one per SM and round
    sphk::hydro_df_sweep<<<std::max(1, std::min(a.n_i, 2 * ctx->grid_df / 5 + 1)), sphk::HYDRO_SWEEP_THREADS, 0, s>>>(
        a);
}

// jtile: entries a warp stages per pass in FP32C (32 or 64; FP64 uses 32).
void launch_gravity(const sphk::GravityArgs &a, int precision, int grid, cudaStream_t s, int jtile) {
    if (precision == SPH_PREC_FP64)
        sphk::gravity_kernel<true, PAIR_WARPS><<<grid, PAIR_WARPS * 32, 0, s>>>(a);
    else if (jtile == 64)
        sphk::gravity_kernel<false, PAIR_WARPS, 64><<<grid, PAIR_WARPS * 32, 0, s>>>(a);
    else
        sphk::gravity_kernel<false, PAIR_WARPS><<<grid, PAIR_WARPS * 32, 0, s>>>(a);
}

}  // namespace sphrt

using namespace sphrt;

// ---------------------------------------------------------------- kernels
namespace {

__device__ __forceinline__ bool finite3(double a, double b, double c) {
    return isfinite(a) && isfinite(b) && isfinite(c);
}

// Copies n 16-byte words from pinned memory; the first launch of a dispatch
// clears its counters.
__global__ void __launch_bounds__(256) copy_inputs(const uint4 *src, uint4 *dst, size_t n, int *queue) {
    if (queue && blockIdx.x == 0 && threadIdx.x < 12) queue[threadIdx.x] = 0;
    const size_t stride = (size_t)gridDim.x * 256;
    for (size_t k = (size_t)blockIdx.x * 256 + threadIdx.x; k < n; k += 4 * stride) {
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (k + u * stride < n) v[u] = src[k + u * stride];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (k + u * stride < n) dst[k + u * stride] = v[u];
    }
}

// Records of one side (i or j) of a dispatch.
struct DensitySide {
    dbl4 *pm, *vel;
    long long *id;
    double *ksr, *rs;                     // i side
    float4 *phi, *plo, *vhi, *vlo;
};
template <class E>
__device__ __forceinline__ void prepare_density_one(const E *in, int k, const DensitySide &s, bool f32) {
    const E e = in[k];
    const dbl4 p = make_dbl4(e.pos[0], e.pos[1], e.pos[2], e.mass), v = make_dbl4(e.vel[0], e.vel[1], e.vel[2], 0.0);
    double h = 0.0;
    if constexpr (sizeof(E) == sizeof(sph_DensityEPI)) {
        h = e.ksr;
        s.ksr[k] = e.ksr;
        s.rs[k] = e.rs;
    }
    s.pm[k] = p;
    s.vel[k] = v;
    s.id[k] = e.id;
    float4 a, b;
    if (f32)
        sphk::row_record<false>(p, h, a, b);
    else
        sphk::row_record<true>(p, h, a, b);
    s.phi[k] = a;
    s.plo[k] = b;
    if (f32) {
        sphk::velocity_record(v, a, b);
        s.vhi[k] = a;
        s.vlo[k] = b;
    }
}
__global__ void prepare_density(const sph_DensityEPI *epi, int ni, const sph_DensityEPJ *epj, int nj, DensitySide si,
                                DensitySide sj, bool f32) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < ni + nj; k += gridDim.x * blockDim.x) {
        if (k < ni)
            prepare_density_one(epi, k, si, f32);
        else
            prepare_density_one(epj, k - ni, sj, f32);
    }
}

struct HydroSide {
    dbl4 *pm, *vel, *h1, *h2;
    double2 *h3;
    long long *id;
    float4 *phi, *plo, *vhi, *vlo, *g1, *g2, *g3, *g4, *mp, *mv;
};
template <class E>
__device__ __forceinline__ void prepare_hydro_one(const E *in, int k, const HydroSide &s, bool f32) {
    const E &e = in[k];
    double m = 0.0;
    if constexpr (sizeof(E) == sizeof(sph_HydroEPJ)) m = e.mass;
    const dbl4 p = make_dbl4(e.pos[0], e.pos[1], e.pos[2], m), v = make_dbl4(e.vel[0], e.vel[1], e.vel[2], 0.0);
    const dbl4 h1 = make_dbl4(e.hinv, e.pres, e.presc, e.bswt), h2 = make_dbl4(e.dens, e.vsnd, e.alph, e.alphu);
    const double2 h3 = make_double2(e.thrm, e.eta);
    s.pm[k] = p;
    s.vel[k] = v;
    s.id[k] = e.id;
    s.h1[k] = h1;
    s.h2[k] = h2;
    s.h3[k] = h3;
    float4 a, b;
    if (f32) {
        sphk::HydroRecords r;
        r.fill(p, v, h1, h2, h3);
        s.phi[k] = r.phi; s.plo[k] = r.plo; s.vhi[k] = r.vhi; s.vlo[k] = r.vlo;
        s.g1[k] = r.g1; s.g2[k] = r.g2; s.g3[k] = r.g3; s.g4[k] = r.g4;
    } else {
        sphk::row_record<true>(p, 0.0, a, b);
        s.plo[k] = b;
    }
    sphk::hydro_mark_records(p, v, h1.x, h2.y, a, b);
    s.mp[k] = a;
    s.mv[k] = b;
}
__global__ void prepare_hydro(const sph_HydroEPI *epi, int ni, const sph_HydroEPJ *epj, int nj, HydroSide si,
                              HydroSide sj, bool f32) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < ni + nj; k += gridDim.x * blockDim.x) {
        if (k < ni)
            prepare_hydro_one(epi, k, si, f32);
        else
            prepare_hydro_one(epj, k - ni, sj, f32);
    }
}

// GravityEPJ and GravitySPJ share one layout (mass, pos[3], eps2).
__global__ void prepare_gravity(const sph_GravityEPI *epi, int ni, const sph_GravityEPJ *epj, int nj, dbl4 *i_pe,
                                float4 *i_hi, float4 *i_lo, dbl4 *j_pm, double *j_eps2, float4 *j_hi, float4 *j_lo,
                                bool f32) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < ni + nj; k += gridDim.x * blockDim.x) {
        float4 a, b;
        if (k < ni) {
            const sph_GravityEPI e = epi[k];
            const dbl4 p = make_dbl4(e.pos[0], e.pos[1], e.pos[2], e.eps2);
            if (f32) {
                sphk::gravity_record(p, 0.0, e.eps2, a, b);
                i_hi[k] = a;
                i_lo[k] = b;
            } else {
                i_pe[k] = p;
            }
        } else {
            const int j = k - ni;
            const sph_GravityEPJ e = epj[j];
            const dbl4 p = make_dbl4(e.pos[0], e.pos[1], e.pos[2], e.mass);
            if (f32) {
                sphk::gravity_record(p, e.mass, e.eps2, a, b);
                j_hi[j] = a;
                j_lo[j] = b;
            } else {
                j_pm[j] = p;
                j_eps2[j] = e.eps2;
            }
        }
    }
}

// Results go to pinned memory: a block's structs through shared memory, so that
// the link sees consecutive words (bound by it: 40k density structs took 89 us
// written struct by struct, 16 us so).
constexpr int PACK_THREADS = 256;
template <class T>
__device__ __forceinline__ void write_structs(T *s, const T &v, T *out, int k0, int n) {
    static_assert(sizeof(T) % 8 == 0, "structs of 8-byte words");
    s[threadIdx.x] = v;
    __syncthreads();
    const unsigned long long *w = reinterpret_cast<const unsigned long long *>(s);
    unsigned long long *o = reinterpret_cast<unsigned long long *>(out + k0);
    const int words = min(PACK_THREADS, n - k0) * (int)(sizeof(T) / 8);
    for (int k = threadIdx.x; k < words; k += PACK_THREADS) o[k] = w[k];
    __syncthreads();
}

__global__ void __launch_bounds__(PACK_THREADS)
pack_density(int n, const double *dens, const double *divv, const double *rotv, const double *grdh,
             const double *ksr, const long long *np, const unsigned char *itr, sph_Density *out, int *flag) {
    __shared__ sph_Density s[PACK_THREADS];
    for (int k0 = blockIdx.x * PACK_THREADS; k0 < n; k0 += gridDim.x * PACK_THREADS) {
        const int k = min(k0 + (int)threadIdx.x, n - 1);
        sph_Density d;
        d.dens = dens[k];
        d.divv = divv[k];
        d.rotv = rotv[k];
        d.grdh = grdh[k];
        d.ksr = ksr[k];
        d.np = np[k];
        d.itr = itr[k] != 0;
        write_structs(s, d, out, k0, n);
        if (!(finite3(d.dens, d.divv, d.rotv) && finite3(d.grdh, d.ksr, 0.0))) *flag = 1;
    }
}

__global__ void __launch_bounds__(PACK_THREADS)
pack_hydro(int n, const double *acch, const double *accg, const double *udot, const double *vsmx,
           const double *diffu, sph_Hydro *out, int *flag) {
    __shared__ sph_Hydro s[PACK_THREADS];
    for (int k0 = blockIdx.x * PACK_THREADS; k0 < n; k0 += gridDim.x * PACK_THREADS) {
        const int k = min(k0 + (int)threadIdx.x, n - 1);
        sph_Hydro h;
        for (int c = 0; c < 3; ++c) {
            h.acch[c] = acch[3 * k + c];
            h.accg[c] = accg[3 * k + c];
        }
        h.udot = udot[k];
        h.vsmx = vsmx[k];
        h.diffu = diffu[k];
        write_structs(s, h, out, k0, n);
        if (!(finite3(h.acch[0], h.acch[1], h.acch[2]) && finite3(h.accg[0], h.accg[1], h.accg[2]) &&
              finite3(h.udot, h.vsmx, h.diffu)))
            *flag = 1;
    }
}

// Few parts per list (many particles): a thread per particle.
constexpr int PACK_SLICES = 8;
__global__ void __launch_bounds__(PACK_THREADS)
pack_gravity_block(int n, const double *acc, const double *pot, const double *eta, int slices, sph_Gravity *out,
                   int *flag) {
    __shared__ sph_Gravity s[PACK_THREADS];
    for (int k0 = blockIdx.x * PACK_THREADS; k0 < n; k0 += gridDim.x * PACK_THREADS) {
        const int k = min(k0 + (int)threadIdx.x, n - 1);
        double v[5];
        sphk::gravity_gather(acc, pot, eta, k, slices, n, v);
        sph_Gravity g;
        for (int c = 0; c < 3; ++c) g.acc[c] = v[c];
        g.pot = v[3];
        g.eta = v[4];
        write_structs(s, g, out, k0, n);
        if (!(finite3(g.acc[0], g.acc[1], g.acc[2]) && finite3(g.pot, g.eta, 0.0))) *flag = 1;
    }
}

// One warp per particle, over the parts of its list.
__global__ void pack_gravity(int n, const double *acc, const double *pot, const double *eta, int slices,
                             sph_Gravity *out, int *flag) {
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < n; k += nw) {
        double v[5];
        sphk::gravity_gather_warp(acc, pot, eta, k, slices, n, lane, v);
        if (lane != 0) continue;
        sph_Gravity g;
        for (int c = 0; c < 3; ++c) g.acc[c] = v[c];
        g.pot = v[3];
        g.eta = v[4];
        out[k] = g;
        if (!(finite3(g.acc[0], g.acc[1], g.acc[2]) && finite3(g.pot, g.eta, 0.0))) *flag = 1;
    }
}

inline int eltwise_grid(long long n) {
    long long b = (n + 255) / 256;
    return (int)std::max(1LL, std::min(b, 4096LL));
}

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Warps that the pair kernels keep resident, about (4 blocks of 4 per SM).
int resident_warps(const sph_context *ctx) { return 16 * ctx->sm_count; }

// Splits every walk into work items of <= chunk i-particles; largest first.
// split_nj > 0: walks with longer lists are cut finer (down to 4), so that no
// item outlasts the rest.
void build_items(int n_walk, const int *i_off, const int *j_off, int chunk, int split_nj,
                 std::vector<WorkItem> &items) {
    items.clear();
    for (int w = 0; w < n_walk; ++w) {
        const int ni = i_off[w + 1] - i_off[w];
        const int nj = j_off[w + 1] - j_off[w];
        int ch = chunk;
        if (split_nj > 0)
            for (long long lim = split_nj; ch > 4 && nj > lim; lim <<= 1) ch >>= 1;
        for (int k = 0; k < ni; k += ch) {
            const int c = std::min(ch, ni - k);
            const long long cost = (long long)nj * c;
            items.push_back(make_int4(w, i_off[w] + k, c, (int)std::min<long long>(cost, 0x7fffffff)));
        }
    }
    std::stable_sort(items.begin(), items.end(),
                     [](const WorkItem &a, const WorkItem &b) { return a.w > b.w; });
}

// i-particles per work item: halved from 32 while that leaves resident warps
// without an item (a small call's time is the streaming of one item's list,
// whatever its number of i-particles).
int item_size(const sph_context *ctx, long long n_i) {
    int chunk = 32;
    while (chunk > 1 && n_i < (long long)chunk * resident_warps(ctx)) chunk >>= 1;
    return chunk;
}

}  // namespace

// ---------------------------------------------------------------- context
extern "C" void sph_params_default(sph_params *p) {
    if (!p) return;
    p->device = 0;
    p->precision = SPH_PREC_FP32C;
    p->eta = 1.6;
    p->ksr_max = 0.0;
    p->max_walks = 1000;
    p->max_i = 1000000;
    p->max_j = 10000000;
    p->check_finite = 1;
}

extern "C" const char *sph_status_string(int s) {
    switch (s) {
        case SPH_OK: return "ok";
        case SPH_ERR_INVALID_ARGUMENT: return "invalid argument";
        case SPH_ERR_CAPACITY: return "capacity exceeded";
        case SPH_ERR_CUDA: return "CUDA error";
        case SPH_ERR_NONFINITE: return "non-finite value in an output";
        case SPH_ERR_NOT_CONVERGED: return "search radius expansion did not converge";
        case SPH_ERR_STATE: return "call out of sequence";
        case SPH_ERR_NO_DEVICE: return "no usable CUDA device";
        default: return "unknown status";
    }
}

extern "C" const char *sph_version(void) { return "sph_gb300 0.1 (sm_103a)"; }

extern "C" int sph_context_create(const sph_params *p, sph_context **out) {
    if (!out) return SPH_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    sph_params prm;
    if (p) prm = *p; else sph_params_default(&prm);
    if (prm.precision != SPH_PREC_FP32C && prm.precision != SPH_PREC_FP64) return SPH_ERR_INVALID_ARGUMENT;
    if (!(prm.eta > 0.0) || prm.max_walks <= 0 || prm.max_i <= 0 || prm.max_j <= 0 ||
        prm.max_i > 0x7fffffffLL || prm.max_j > 0x7fffffffLL)
        return SPH_ERR_INVALID_ARGUMENT;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) {
        cudaGetLastError();
        return SPH_ERR_NO_DEVICE;
    }
    if (prm.device < 0 || prm.device >= ndev) return SPH_ERR_NO_DEVICE;
    sph_context *ctx = new (std::nothrow) sph_context();
    if (!ctx) return SPH_ERR_CAPACITY;
    ctx->prm = prm;
    cudaError_t e = cudaSetDevice(prm.device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&ctx->sm_count, cudaDevAttrMultiProcessorCount, prm.device);
    int cc_major = 0;
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&cc_major, cudaDevAttrComputeCapabilityMajor, prm.device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMalloc(&ctx->d_queue, 12 * sizeof(int));
    if (e == cudaSuccess) e = cudaMallocHost(&ctx->h_flags, 8 * sizeof(int));
    if (e == cudaSuccess && init_grids(ctx) != 0) e = cudaErrorInvalidDeviceFunction;
    if (e != cudaSuccess) {
        cudaGetLastError();
        int st = (e == cudaErrorNoKernelImageForDevice || e == cudaErrorInvalidDeviceFunction)
                     ? SPH_ERR_NO_DEVICE : SPH_ERR_CUDA;
        sph_context_destroy(ctx);
        return st;
    }
    *out = ctx;
    return SPH_OK;
}

extern "C" int sph_context_destroy(sph_context *ctx) {
    if (!ctx) return SPH_ERR_INVALID_ARGUMENT;
    // systems hold the context's stream: they must go first
    if (ctx->n_systems > 0)
        return set_error(ctx, SPH_ERR_STATE, "%d system(s) still use this context", ctx->n_systems);
    cudaSetDevice(ctx->prm.device);
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    for (int k = 0; k < 3; ++k) ctx->kind[k].release();
    if (ctx->d_queue) cudaFree(ctx->d_queue);
    if (ctx->h_flags) cudaFreeHost(ctx->h_flags);
    if (ctx->stream) cudaStreamDestroy(ctx->stream);
    delete ctx;
    return SPH_OK;
}

extern "C" int sph_context_set_eta(sph_context *ctx, double eta) {
    if (!ctx || !(eta > 0.0)) return SPH_ERR_INVALID_ARGUMENT;
    ctx->prm.eta = eta;
    return SPH_OK;
}

extern "C" int sph_context_set_ksr_max(sph_context *ctx, double v) {
    if (!ctx || std::isnan(v)) return SPH_ERR_INVALID_ARGUMENT;
    ctx->prm.ksr_max = v;
    return SPH_OK;
}

extern "C" int sph_context_set_precision(sph_context *ctx, int32_t precision) {
    if (!ctx || (precision != SPH_PREC_FP32C && precision != SPH_PREC_FP64)) return SPH_ERR_INVALID_ARGUMENT;
    ctx->prm.precision = precision;
    return SPH_OK;
}

extern "C" int sph_context_stream(const sph_context *ctx, void **stream) {
    if (!ctx || !stream) return SPH_ERR_INVALID_ARGUMENT;
    *stream = (void *)ctx->stream;
    return SPH_OK;
}

namespace {
// Eight independent FMA chains per thread keep the FP32 pipe full.
__global__ void fma_probe(float *out, int iters, float b, float c) {
    float a0 = threadIdx.x, a1 = a0 + 1, a2 = a0 + 2, a3 = a0 + 3, a4 = a0 + 4, a5 = a0 + 5, a6 = a0 + 6, a7 = a0 + 7;
    for (int k = 0; k < iters; ++k) {
        a0 = fmaf(a0, b, c); a1 = fmaf(a1, b, c); a2 = fmaf(a2, b, c); a3 = fmaf(a3, b, c);
        a4 = fmaf(a4, b, c); a5 = fmaf(a5, b, c); a6 = fmaf(a6, b, c); a7 = fmaf(a7, b, c);
    }
    const float s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
    if (s == 1234.5f) out[0] = s;   // keeps the chains live
}
}  // namespace

extern "C" int sph_probe_fp32_peak(sph_context *ctx, double *tflops) {
    if (!ctx || !tflops) return SPH_ERR_INVALID_ARGUMENT;
    cudaSetDevice(ctx->prm.device);
    float *d = nullptr;
    cudaEvent_t e0, e1;
    if (cudaMalloc(&d, sizeof(float)) != cudaSuccess) return sphrt::set_error(ctx, SPH_ERR_CUDA, "probe alloc");
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int threads = 256, blocks = ctx->sm_count * 8, iters = 1 << 16;
    fma_probe<<<blocks, threads, 0, ctx->stream>>>(d, 256, 0.999f, 1e-3f);   // warm-up
    cudaEventRecord(e0, ctx->stream);
    fma_probe<<<blocks, threads, 0, ctx->stream>>>(d, iters, 0.999f, 1e-3f);
    cudaEventRecord(e1, ctx->stream);
    cudaError_t e = cudaEventSynchronize(e1);
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(d);
    if (e != cudaSuccess) return sphrt::cuda_error(ctx, e, "probe");
    *tflops = 2.0 * 8.0 * (double)iters * threads * blocks / (ms * 1e-3) / 1e12;
    return SPH_OK;
}

extern "C" int sph_context_last_error(const sph_context *ctx, char *buf, size_t n) {
    if (!ctx || !buf || n == 0) return SPH_ERR_INVALID_ARGUMENT;
    std::snprintf(buf, n, "%s", ctx->err);
    return SPH_OK;
}

// ---------------------------------------------------------------- dispatch
namespace {

enum { K_DENS = 0, K_HYDRO = 1, K_GRAV = 2 };
constexpr float ROW_SLACK = 1.03f;   // row radius of the density over the first guess of h
// Lists beyond this are marked by a block per item (hydro 21k batch 2.86 ms with none,
// 2.23 at 4096, 1.93 at 1536, 1.98 at 1024; density 40k 2.13 / 2.04 / 2.07).
constexpr int LONG_NJ = 1536;
// FP32C hydro calls of few items (32 targets each, so that rows keep a warp's
// order): a warp per list leaves the chip idle.  Calls of 16, 32 and 64 targets 158,
// 172 and 199 us by warps at 125 neighbours, 123, 125 and 132 by blocks; at 55
// neighbours 145, 163 and 180, 139, 153 and 161; of 8 (list of 187) 124 and 127.
constexpr int LONG_NJ_FEW = 256;
constexpr int SPLIT_NJ = 1024;   // density and hydro: lists beyond this make smaller items

int longest(const int32_t *n, int n_walk) {
    int m = 0;
    for (int w = 0; w < n_walk; ++w) m = std::max(m, (int)n[w]);
    return m;
}

// FP32C density: with more rowless particles than this (a first guess of h far
// off, or more neighbours than a row holds) items of 32, which share every list
// entry, stream the lists instead of a block per particle.  A block takes ~0.1 us
// of the chip per particle and 1000 entries; an item's four passes take 0.24 us
// per entry, however many items there are.  Calls of 2000 targets (list of ~5500):
// 0.78 ms by blocks, 1.61 by items; of 5000 (~10000) 2.12 and 2.97; batches of 10000
// (~700) 2.2 and 1.7; of 40000 (1000 per walk) 10.5 and 3.9 (5.1 by the lists,
// before rows); at 125 neighbours 12.8 and 5.3 (8.3).
int rowless_most(const sph_context *ctx, int longest_list) { return ctx->sm_count * (8 + longest_list / 256); }

// Validates walk counts and fills the int32 offsets.  n_extra (gravity SPJ
// counts) may be null.
int walk_offsets(sph_context *ctx, int32_t n_walk, const int32_t *n_i, const int32_t *n_j,
                 const int32_t *n_extra, std::vector<int> &i_off, std::vector<int> &j_off) {
    if (n_walk < 0) return set_error(ctx, SPH_ERR_INVALID_ARGUMENT, "n_walk < 0");
    if (n_walk > ctx->prm.max_walks)
        return set_error(ctx, SPH_ERR_CAPACITY, "n_walk %d > max_walks %d", n_walk, ctx->prm.max_walks);
    if (n_walk > 0 && (!n_i || !n_j)) return set_error(ctx, SPH_ERR_INVALID_ARGUMENT, "null counts");
    i_off.assign(n_walk + 1, 0);
    j_off.assign(n_walk + 1, 0);
    long long ti = 0, tj = 0;
    for (int w = 0; w < n_walk; ++w) {
        const long long e = n_extra ? n_extra[w] : 0;
        if (n_i[w] < 0 || n_j[w] < 0 || e < 0)
            return set_error(ctx, SPH_ERR_INVALID_ARGUMENT, "negative count in walk %d", w);
        ti += n_i[w];
        tj += n_j[w] + e;
        if (ti > ctx->prm.max_i) return set_error(ctx, SPH_ERR_CAPACITY, "i total %lld > max_i", ti);
        if (tj > ctx->prm.max_j) return set_error(ctx, SPH_ERR_CAPACITY, "j total %lld > max_j", tj);
        i_off[w + 1] = (int)ti;
        j_off[w + 1] = (int)tj;
    }
    return SPH_OK;
}

// Device buffer [i_off | j_off | items | EPI | EPJ].
struct Layout {
    size_t off_ioff, off_joff, off_items, off_epi, off_epj, total;
};

Layout make_layout(int n_walk, size_t n_items, size_t bytes_epi, size_t bytes_epj) {
    Layout L;
    size_t o = 0;
    L.off_ioff = o; o = align_up(o + sizeof(int) * (n_walk + 1), 256);
    L.off_joff = o; o = align_up(o + sizeof(int) * (n_walk + 1), 256);
    L.off_items = o; o = align_up(o + sizeof(WorkItem) * n_items, 256);
    L.off_epi = o; o = align_up(o + bytes_epi, 256);
    L.off_epj = o; o = align_up(o + bytes_epj, 256);
    L.total = o;
    return L;
}

// One array of each walk: entries of `size` bytes, the walk's at index off of
// the region at `base` of the device buffer.
struct WalkArrays {
    const void *const *ptr;
    const int32_t *n;
    size_t size, base;
};

// Copies bytes [from, to) of the pinned buffer in; the first copy of a dispatch
// (from = 0) clears its counters.
void launch_copy(sph_context *ctx, KindState &ks, size_t from, size_t to) {
    const size_t n = (to - from + 15) / 16;
    const int grid = (int)std::max<size_t>(1, std::min<size_t>((n + 255) / 256, 8 * ctx->sm_count));
    copy_inputs<<<grid, 256, 0, ctx->stream>>>(reinterpret_cast<const uint4 *>(ks.h_in.p + from),
                                               reinterpret_cast<uint4 *>(ks.d_in.p + from), n,
                                               from == 0 ? ctx->d_queue : nullptr);
}

// Builds the items, fills the pinned buffer and copies it to the device.
// place: byte offset of array a of walk w in the buffer.
template <class P>
int stage(sph_context *ctx, KindState &ks, const std::vector<int> &i_off, const std::vector<int> &j_off,
          size_t epi_size, size_t epj_size, int chunk, int split_nj, const WalkArrays *arrays, int n_arrays,
          P place, Layout &L) {
    const int n_walk = (int)i_off.size() - 1;
    build_items(n_walk, i_off.data(), j_off.data(), chunk, split_nj, ks.items);
    L = make_layout(n_walk, ks.items.size(), epi_size * (size_t)i_off[n_walk],
                    epj_size * (size_t)j_off[n_walk]);
    if (ks.h_in.ensure(L.total) || ks.d_in.ensure(L.total, false))
        return set_error(ctx, SPH_ERR_CUDA, "staging allocation of %zu bytes failed", L.total);
    std::vector<CopyTask> tasks;
    tasks.reserve((size_t)n_arrays * n_walk + L.total / TASK_BYTES);
    auto add = [&](int a, int w) {
        const size_t bytes = arrays[a].n ? arrays[a].size * (size_t)arrays[a].n[w] : 0;
        if (!bytes) return true;
        const char *src = static_cast<const char *>(arrays[a].ptr[w]);
        if (!src) return false;
        const size_t dst = place(a, w);
        for (size_t o = 0; o < bytes; o += TASK_BYTES)
            tasks.push_back(CopyTask{src + o, dst + o, std::min(bytes - o, TASK_BYTES)});
        return true;
    };
    // in the order of the buffer: EPI of every walk, then each walk's lists
    for (int w = 0; w < n_walk; ++w)
        if (!add(0, w)) return set_error(ctx, SPH_ERR_INVALID_ARGUMENT, "null array in walk %d", w);
    for (int w = 0; w < n_walk; ++w)
        for (int a = 1; a < n_arrays; ++a)
            if (!add(a, w)) return set_error(ctx, SPH_ERR_INVALID_ARGUMENT, "null array in walk %d", w);
    char *h = ks.h_in.p;
    std::memcpy(h + L.off_ioff, i_off.data(), sizeof(int) * (n_walk + 1));
    std::memcpy(h + L.off_joff, j_off.data(), sizeof(int) * (n_walk + 1));
    if (!ks.items.empty()) std::memcpy(h + L.off_items, ks.items.data(), sizeof(WorkItem) * ks.items.size());
    ctx->h_flags[ks.flag_slot] = 0;
    const size_t bytes = tasks.empty() ? 0 : tasks.back().dst + tasks.back().bytes - tasks.front().dst;
    run_copies(h, tasks, L.total, extra_copy_threads(bytes),
               [&](size_t from, size_t to) { launch_copy(ctx, ks, from, to); });
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error(ctx, e, "input copy");
    return SPH_OK;
}

// After the launches of a dispatch.
int finish_dispatch(sph_context *ctx, KindState &ks, int n_walk, const std::vector<int> &i_off) {
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error(ctx, e, "kernel launch");
    ks.pending = true;
    ks.n_walk = n_walk;
    ks.i_off = i_off;
    return SPH_OK;
}

int begin_kind(sph_context *ctx, KindState &ks) {
    if (!ctx) return SPH_ERR_INVALID_ARGUMENT;
    if (ks.pending)
        return set_error(ctx, SPH_ERR_STATE, "a dispatch of this kind is outstanding; retrieve it first");
    cudaError_t e = cudaSetDevice(ctx->prm.device);
    if (e != cudaSuccess) return cuda_error(ctx, e, "cudaSetDevice");
    // The pinned staging buffer may still feed a copy of an earlier dispatch
    // that failed after its upload was queued; never overwrite it in flight.
    e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_error(ctx, e, "stream synchronize");
    return SPH_OK;
}

template <class F>
int retrieve_common(sph_context *ctx, KindState &ks, int32_t n_walk, const int32_t *n_i, F **force,
                    size_t out_size) {
    if (!ctx) return SPH_ERR_INVALID_ARGUMENT;
    if (!ks.pending) return set_error(ctx, SPH_ERR_STATE, "retrieve without a dispatch");
    cudaError_t e = cudaSetDevice(ctx->prm.device);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    ks.pending = false;
    if (e != cudaSuccess) return cuda_error(ctx, e, "stream synchronize");
    if (n_walk != ks.n_walk)
        return set_error(ctx, SPH_ERR_INVALID_ARGUMENT, "n_walk %d differs from dispatch %d", n_walk, ks.n_walk);
    if (n_walk > 0 && (!n_i || !force)) return set_error(ctx, SPH_ERR_INVALID_ARGUMENT, "null arrays");
    for (int w = 0; w < n_walk; ++w) {
        const int ni = ks.i_off[w + 1] - ks.i_off[w];
        if (n_i[w] != ni)
            return set_error(ctx, SPH_ERR_INVALID_ARGUMENT, "walk %d: n_i %d differs from dispatch %d", w, n_i[w], ni);
        if (ni > 0 && !force[w]) return set_error(ctx, SPH_ERR_INVALID_ARGUMENT, "null force[%d]", w);
        if (ni > 0) std::memcpy(force[w], ks.h_out.p + out_size * ks.i_off[w], out_size * ni);
    }
    if (ctx->prm.check_finite && ctx->h_flags[ks.flag_slot])
        return set_error(ctx, SPH_ERR_NONFINITE, "non-finite value in the outputs");
    return SPH_OK;
}

}  // namespace

extern "C" int sph_dispatch_density(sph_context *ctx, int32_t tag, int32_t n_walk,
                                    const sph_DensityEPI **epi, const int32_t *n_epi,
                                    const sph_DensityEPJ **epj, const int32_t *n_epj) {
    (void)tag;
    KindState *ksp = ctx ? &ctx->kind[K_DENS] : nullptr;
    int st = begin_kind(ctx, *ksp);
    if (st) return st;
    KindState &ks = *ksp;
    ks.flag_slot = K_DENS;
    std::vector<int> i_off, j_off;
    if ((st = walk_offsets(ctx, n_walk, n_epi, n_epj, nullptr, i_off, j_off))) return st;
    if (n_walk > 0 && (!epi || !epj)) return set_error(ctx, SPH_ERR_INVALID_ARGUMENT, "null walk arrays");
    const int ni = i_off[n_walk], nj = j_off[n_walk];
    const int cap = std::max(256, ni / 16);
    const WalkArrays arrays[2] = {{(const void *const *)epi, n_epi, sizeof(sph_DensityEPI), 0},
                                  {(const void *const *)epj, n_epj, sizeof(sph_DensityEPJ), 0}};
    Layout L;
    auto place = [&](int a, int w) {
        return a == 0 ? L.off_epi + sizeof(sph_DensityEPI) * i_off[w] : L.off_epj + sizeof(sph_DensityEPJ) * j_off[w];
    };
    if ((st = stage(ctx, ks, i_off, j_off, sizeof(sph_DensityEPI), sizeof(sph_DensityEPJ), item_size(ctx, ni),
                    SPLIT_NJ, arrays, 2, place, L)))
        return st;
    const bool f32 = ctx->prm.precision == SPH_PREC_FP32C;
    const int most = rowless_most(ctx, longest(n_epj, n_walk));
    const bool many = f32 && ni > most;
    if (ks.ensure_density(ni, nj, cap, ks.items.size(), many ? ni : 0, n_walk))
        return set_error(ctx, SPH_ERR_CUDA, "device allocation failed");
    if (ks.h_out.ensure(sizeof(sph_Density) * (size_t)std::max(ni, 1)))
        return set_error(ctx, SPH_ERR_CUDA, "output allocation failed");
    char *d = ks.d_in.p;
    const DensitySide si{ks.a4[0].p, ks.a4[1].p, ks.id[0].p, ks.d1[0].p, ks.d1[1].p,
                         ks.f4[0].p, ks.f4[1].p, ks.f4[2].p, ks.f4[3].p};
    const DensitySide sj{ks.a4[2].p, ks.a4[3].p, ks.id[1].p, nullptr, nullptr,
                         ks.f4[4].p, ks.f4[5].p, ks.f4[6].p, ks.f4[7].p};
    if (ni + nj > 0)
        prepare_density<<<eltwise_grid((long long)ni + nj), 256, 0, ctx->stream>>>(
            (const sph_DensityEPI *)(d + L.off_epi), ni, (const sph_DensityEPJ *)(d + L.off_epj), nj, si, sj, f32);
    if (!ks.items.empty()) {
        sphk::MarkArgs m{};
        m.i_hi = ks.f4[0].p; m.i_lo = ks.f4[1].p; m.j_hi = ks.f4[4].p; m.j_lo = ks.f4[5].p;
        m.slack = ROW_SLACK;
        m.items = (const WorkItem *)(d + L.off_items);
        m.n_items = (int)ks.items.size();
        m.j_off = (const int *)(d + L.off_joff);
        m.queue = ctx->d_queue + K_DENS;
        m.rows = ks.hl_list.p; m.info = ks.r_info.p; m.ovf = ks.hl_ovf.p; m.n_ovf = ctx->d_queue + 7;
        m.longs = sphk::LongQueue{ks.long_items.p, ctx->d_queue + 9, 0}; m.long_nj = LONG_NJ;
        m.push_long = longest(n_epj, n_walk) > LONG_NJ;
        sphk::DensityArgs a{};
        a.i_pm = ks.a4[0].p; a.i_vel = ks.a4[1].p; a.i_id = ks.id[0].p; a.i_ksr = ks.d1[0].p; a.i_rs = ks.d1[1].p;
        a.j_pm = ks.a4[2].p; a.j_vel = ks.a4[3].p; a.j_id = ks.id[1].p;
        a.fi = sphk::F32Part{ks.f4[0].p, ks.f4[1].p, ks.f4[2].p, ks.f4[3].p};
        a.fj = sphk::F32Part{ks.f4[4].p, ks.f4[5].p, ks.f4[6].p, ks.f4[7].p};
        a.n_i = ni;
        a.j_off = m.j_off;
        a.rows = m.rows; a.info = m.info; a.ovf = m.ovf; a.n_ovf = m.n_ovf;
        a.slack = m.slack;
        a.o_dens = ks.o[0].p; a.o_divv = ks.o[1].p; a.o_rotv = ks.o[2].p; a.o_grdh = ks.o[3].p;
        a.o_ksr = ks.o[4].p; a.o_np = ks.o_np.p; a.o_itr = ks.o_itr.p;
        a.eta_ksrh = ctx->prm.eta * sphk::KSRH;
        a.ksr_max = ctx->prm.ksr_max > 0.0 ? ctx->prm.ksr_max : std::numeric_limits<double>::infinity();
        a.amb_count = f32 ? ctx->d_queue + 3 : nullptr;
        a.amb = ks.amb.p;
        a.amb_cap = cap;
        a.amb_tol = AMB_TOL;
        const RowlessItems rowless{(const int *)(d + L.off_ioff), n_walk, most, ks.rowless.p, ks.rowless_items.p,
                                   ctx->d_queue + 4, ctx->d_queue + 5};
        launch_density(ctx, m, pair_grid(ctx, K_DENS, ctx->prm.precision, m.n_items), a, ni, ctx->prm.precision,
                       ctx->stream, nullptr, nullptr, many ? &rowless : nullptr);
    }
    if (ni > 0)
        pack_density<<<eltwise_grid(ni), 256, 0, ctx->stream>>>(
            ni, ks.o[0].p, ks.o[1].p, ks.o[2].p, ks.o[3].p, ks.o[4].p, ks.o_np.p, ks.o_itr.p,
            (sph_Density *)ks.h_out.p, ctx->h_flags + K_DENS);
    return finish_dispatch(ctx, ks, n_walk, i_off);
}

extern "C" int sph_retrieve_density(sph_context *ctx, int32_t tag, int32_t n_walk, const int32_t *n_i,
                                    sph_Density **force) {
    (void)tag;
    if (!ctx) return SPH_ERR_INVALID_ARGUMENT;
    return retrieve_common(ctx, ctx->kind[K_DENS], n_walk, n_i, force, sizeof(sph_Density));
}

extern "C" int sph_dispatch_hydro(sph_context *ctx, int32_t tag, int32_t n_walk,
                                  const sph_HydroEPI **epi, const int32_t *n_epi,
                                  const sph_HydroEPJ **epj, const int32_t *n_epj) {
    (void)tag;
    KindState *ksp = ctx ? &ctx->kind[K_HYDRO] : nullptr;
    int st = begin_kind(ctx, *ksp);
    if (st) return st;
    KindState &ks = *ksp;
    ks.flag_slot = K_HYDRO;
    std::vector<int> i_off, j_off;
    if ((st = walk_offsets(ctx, n_walk, n_epi, n_epj, nullptr, i_off, j_off))) return st;
    if (n_walk > 0 && (!epi || !epj)) return set_error(ctx, SPH_ERR_INVALID_ARGUMENT, "null walk arrays");
    const int ni = i_off[n_walk], nj = j_off[n_walk];
    const WalkArrays arrays[2] = {{(const void *const *)epi, n_epi, sizeof(sph_HydroEPI), 0},
                                  {(const void *const *)epj, n_epj, sizeof(sph_HydroEPJ), 0}};
    Layout L;
    auto place = [&](int a, int w) {
        return a == 0 ? L.off_epi + sizeof(sph_HydroEPI) * i_off[w] : L.off_epj + sizeof(sph_HydroEPJ) * j_off[w];
    };
    // FP32C: items of 32 i-particles, whose rows and so sums do not depend on
    // the size of the call
    const bool f32 = ctx->prm.precision == SPH_PREC_FP32C, f64 = !f32;
    if ((st = stage(ctx, ks, i_off, j_off, sizeof(sph_HydroEPI), sizeof(sph_HydroEPJ), f64 ? item_size(ctx, ni) : 32,
                    f64 ? SPLIT_NJ : 0, arrays, 2, place, L)))
        return st;
    if (ks.ensure_hydro(ni, nj, ks.items.size()))
        return set_error(ctx, SPH_ERR_CUDA, "device allocation failed");
    if (ks.h_out.ensure(sizeof(sph_Hydro) * (size_t)std::max(ni, 1)))
        return set_error(ctx, SPH_ERR_CUDA, "output allocation failed");
    char *d = ks.d_in.p;
    const HydroSide si{ks.a4[0].p, ks.a4[1].p, ks.a4[4].p, ks.a4[5].p, ks.a2[0].p, ks.id[0].p, ks.f4[0].p, ks.f4[1].p,
                       ks.f4[2].p, ks.f4[3].p, ks.f4[8].p, ks.f4[9].p, ks.f4[10].p, ks.f4[14].p, ks.f4[16].p,
                       ks.f4[17].p};
    const HydroSide sj{ks.a4[2].p, ks.a4[3].p, ks.a4[6].p, ks.a4[7].p, ks.a2[1].p, ks.id[1].p, ks.f4[4].p, ks.f4[5].p,
                       ks.f4[6].p, ks.f4[7].p, ks.f4[11].p, ks.f4[12].p, ks.f4[13].p, ks.f4[15].p, ks.f4[18].p,
                       ks.f4[19].p};
    if (ni + nj > 0)
        prepare_hydro<<<eltwise_grid((long long)ni + nj), 256, 0, ctx->stream>>>(
            (const sph_HydroEPI *)(d + L.off_epi), ni, (const sph_HydroEPJ *)(d + L.off_epj), nj, si, sj, f32);
    if (!ks.items.empty()) {
        sphk::MarkArgs m{};
        m.i_hi = ks.f4[16].p; m.i_lo = ks.f4[1].p; m.j_hi = ks.f4[18].p; m.j_lo = ks.f4[5].p;
        m.i_v = ks.f4[17].p; m.j_v = ks.f4[19].p;
        m.items = (const WorkItem *)(d + L.off_items);
        m.n_items = (int)ks.items.size();
        m.j_off = (const int *)(d + L.off_joff);
        m.queue = ctx->d_queue + K_HYDRO;
        m.rows = ks.hl_list.p; m.info = ks.r_info.p; m.ovf = ks.hl_ovf.p; m.n_ovf = ctx->d_queue + 8;
        m.longs = sphk::LongQueue{ks.long_items.p, ctx->d_queue + 9, 0};
        m.long_nj = f32 && m.n_items <= ctx->sm_count ? LONG_NJ_FEW : LONG_NJ;
        m.push_long = longest(n_epj, n_walk) > m.long_nj;
        m.o_vsmx = ks.o[3].p;
        m.sv_skip = 1;
        sphk::HydroArgs a{};
        a.i_pm = ks.a4[0].p; a.i_vel = ks.a4[1].p; a.i_id = ks.id[0].p;
        a.i_h1 = ks.a4[4].p; a.i_h2 = ks.a4[5].p; a.i_h3 = ks.a2[0].p;
        a.j_pm = ks.a4[2].p; a.j_vel = ks.a4[3].p; a.j_id = ks.id[1].p;
        a.j_h1 = ks.a4[6].p; a.j_h2 = ks.a4[7].p; a.j_h3 = ks.a2[1].p;
        a.fi = sphk::F32Part{ks.f4[0].p, ks.f4[1].p, ks.f4[2].p, ks.f4[3].p};
        a.fj = sphk::F32Part{ks.f4[4].p, ks.f4[5].p, ks.f4[6].p, ks.f4[7].p};
        a.fi_g1 = ks.f4[8].p; a.fi_g2 = ks.f4[9].p; a.fi_g3 = ks.f4[10].p;
        a.fj_g1 = ks.f4[11].p; a.fj_g2 = ks.f4[12].p; a.fj_g3 = ks.f4[13].p;
        a.fi_g4 = ks.f4[14].p; a.fj_g4 = ks.f4[15].p;
        a.j_off = m.j_off;
        a.o_acch = ks.o[0].p; a.o_accg = ks.o[1].p; a.o_udot = ks.o[2].p; a.o_diffu = ks.o[4].p;
        a.rows = m.rows; a.info = m.info; a.ovf = m.ovf; a.n_ovf = m.n_ovf; a.n_i = ni;
        a.mi_p = m.i_hi; a.mi_l = m.i_lo; a.mj_p = m.j_hi; a.mj_l = m.j_lo;
        m.i_id = a.i_id; m.j_id = a.j_id; m.fi = a.fi; m.fj = a.fj; m.fi_g2 = a.fi_g2; m.fj_g2 = a.fj_g2;
        m.i_pm = a.i_pm; m.i_vel = a.i_vel; m.i_h2 = a.i_h2; m.j_pm = a.j_pm; m.j_vel = a.j_vel; m.j_h2 = a.j_h2;
        launch_hydro_marks(ctx, m, pair_grid(ctx, K_HYDRO, ctx->prm.precision, m.n_items), ni, ctx->prm.precision,
                           ctx->stream);
        launch_hydro_sums(ctx, a, ctx->prm.precision, ctx->stream);
    }
    if (ni > 0)
        pack_hydro<<<eltwise_grid(ni), 256, 0, ctx->stream>>>(
            ni, ks.o[0].p, ks.o[1].p, ks.o[2].p, ks.o[3].p, ks.o[4].p, (sph_Hydro *)ks.h_out.p,
            ctx->h_flags + K_HYDRO);
    return finish_dispatch(ctx, ks, n_walk, i_off);
}

extern "C" int sph_retrieve_hydro(sph_context *ctx, int32_t tag, int32_t n_walk, const int32_t *n_i,
                                  sph_Hydro **force) {
    (void)tag;
    if (!ctx) return SPH_ERR_INVALID_ARGUMENT;
    return retrieve_common(ctx, ctx->kind[K_HYDRO], n_walk, n_i, force, sizeof(sph_Hydro));
}

extern "C" int sph_dispatch_gravity(sph_context *ctx, int32_t tag, int32_t n_walk,
                                    const sph_GravityEPI **epi, const int32_t *n_epi,
                                    const sph_GravityEPJ **epj, const int32_t *n_epj,
                                    const sph_GravitySPJ **spj, const int32_t *n_spj) {
    (void)tag;
    KindState *ksp = ctx ? &ctx->kind[K_GRAV] : nullptr;
    int st = begin_kind(ctx, *ksp);
    if (st) return st;
    KindState &ks = *ksp;
    ks.flag_slot = K_GRAV;
    std::vector<int> i_off, j_off;
    if ((st = walk_offsets(ctx, n_walk, n_epi, n_epj, n_spj, i_off, j_off))) return st;
    if (n_walk > 0 && (!epi || !epj)) return set_error(ctx, SPH_ERR_INVALID_ARGUMENT, "null walk arrays");
    if (n_spj && !spj) return set_error(ctx, SPH_ERR_INVALID_ARGUMENT, "null spj");
    const int ni = i_off[n_walk], nj = j_off[n_walk];
    static_assert(sizeof(sph_GravitySPJ) == sizeof(sph_GravityEPJ), "SPJ appended to EPJ");
    const WalkArrays arrays[3] = {{(const void *const *)epi, n_epi, sizeof(sph_GravityEPI), 0},
                                  {(const void *const *)epj, n_epj, sizeof(sph_GravityEPJ), 0},
                                  {(const void *const *)spj, n_spj, sizeof(sph_GravitySPJ), 0}};
    Layout L;
    auto place = [&](int a, int w) {
        if (a == 0) return L.off_epi + sizeof(sph_GravityEPI) * i_off[w];
        return L.off_epj + sizeof(sph_GravityEPJ) * ((size_t)j_off[w] + (a == 2 ? n_epj[w] : 0));
    };
    if ((st = stage(ctx, ks, i_off, j_off, sizeof(sph_GravityEPI), sizeof(sph_GravityEPJ), 32, 0, arrays, 3, place, L)))
        return st;
    const int slices = sphk::gravity_slices((long long)ks.items.size(), nj / std::max(n_walk, 1),
                                            2LL * resident_warps(ctx), 512);
    if (ks.ensure_gravity(ni, nj, slices)) return set_error(ctx, SPH_ERR_CUDA, "device allocation failed");
    if (ks.h_out.ensure(sizeof(sph_Gravity) * (size_t)std::max(ni, 1)))
        return set_error(ctx, SPH_ERR_CUDA, "output allocation failed");
    char *d = ks.d_in.p;
    const bool f32 = ctx->prm.precision == SPH_PREC_FP32C;
    if (ni + nj > 0)
        prepare_gravity<<<eltwise_grid((long long)ni + nj), 256, 0, ctx->stream>>>(
            (const sph_GravityEPI *)(d + L.off_epi), ni, (const sph_GravityEPJ *)(d + L.off_epj), nj, ks.a4[0].p,
            ks.f4[0].p, ks.f4[1].p, ks.a4[2].p, ks.d1[0].p, ks.f4[4].p, ks.f4[5].p, f32);
    if (!ks.items.empty()) {
        sphk::GravityArgs a{};
        a.i_pe = ks.a4[0].p;
        a.j_pm = ks.a4[2].p; a.j_eps2 = ks.d1[0].p;
        a.s_pm = ks.a4[2].p; a.s_eps2 = ks.d1[0].p;
        a.fi_phi = ks.f4[0].p; a.fi_plo = ks.f4[1].p;
        a.f_phi = ks.f4[4].p; a.f_plo = ks.f4[5].p; a.f_shi = ks.f4[4].p; a.f_slo = ks.f4[5].p;
        a.i_list = nullptr;
        a.n_split = 0x7fffffff;
        a.items = (const WorkItem *)(d + L.off_items);
        a.n_items = (int)ks.items.size();
        a.n_items_dev = nullptr;
        a.j_off = (const int *)(d + L.off_joff);
        a.j_idx = nullptr;
        a.queue = ctx->d_queue + K_GRAV;
        a.o_acc = ks.o[0].p; a.o_pot = ks.o[1].p; a.o_eta = ks.o[2].p;
        a.s_quad = nullptr; a.f_sq0 = nullptr; a.f_sq1 = nullptr;   // SPJ are monopoles
        a.slices = slices;
        a.o_stride = ni;
        launch_gravity(a, ctx->prm.precision, pair_grid(ctx, K_GRAV, ctx->prm.precision, a.n_items * slices),
                       ctx->stream, 32);
    }
    if (ni > 0) {
        sph_Gravity *out = (sph_Gravity *)ks.h_out.p;
        int *flag = ctx->h_flags + K_GRAV;
        if (slices <= PACK_SLICES)
            pack_gravity_block<<<eltwise_grid(ni), PACK_THREADS, 0, ctx->stream>>>(ni, ks.o[0].p, ks.o[1].p,
                                                                                  ks.o[2].p, slices, out, flag);
        else
            pack_gravity<<<eltwise_grid(32LL * ni), 256, 0, ctx->stream>>>(ni, ks.o[0].p, ks.o[1].p, ks.o[2].p,
                                                                          slices, out, flag);
    }
    return finish_dispatch(ctx, ks, n_walk, i_off);
}

extern "C" int sph_retrieve_gravity(sph_context *ctx, int32_t tag, int32_t n_walk, const int32_t *n_i,
                                    sph_Gravity **force) {
    (void)tag;
    if (!ctx) return SPH_ERR_INVALID_ARGUMENT;
    return retrieve_common(ctx, ctx->kind[K_GRAV], n_walk, n_i, force, sizeof(sph_Gravity));
}

// ---------------------------------------------------------------- functors
extern "C" int sph_calc_density(sph_context *ctx, const sph_DensityEPI *epi, int32_t n_i,
                                const sph_DensityEPJ *epj, int32_t n_j, sph_Density *force) {
    if (!ctx) return SPH_ERR_INVALID_ARGUMENT;
    if (n_i < 0 || n_j < 0 || (n_i && (!epi || !force)) || (n_j && !epj))
        return set_error(ctx, SPH_ERR_INVALID_ARGUMENT, "bad functor arguments");
    int st = sph_dispatch_density(ctx, 0, 1, &epi, &n_i, &epj, &n_j);
    if (st) return st;
    return sph_retrieve_density(ctx, 0, 1, &n_i, &force);
}

extern "C" int sph_calc_hydro(sph_context *ctx, const sph_HydroEPI *epi, int32_t n_i,
                              const sph_HydroEPJ *epj, int32_t n_j, sph_Hydro *force) {
    if (!ctx) return SPH_ERR_INVALID_ARGUMENT;
    if (n_i < 0 || n_j < 0 || (n_i && (!epi || !force)) || (n_j && !epj))
        return set_error(ctx, SPH_ERR_INVALID_ARGUMENT, "bad functor arguments");
    int st = sph_dispatch_hydro(ctx, 0, 1, &epi, &n_i, &epj, &n_j);
    if (st) return st;
    return sph_retrieve_hydro(ctx, 0, 1, &n_i, &force);
}

namespace {
int gravity_accumulate(sph_context *ctx, const sph_GravityEPI *epi, int32_t n_i,
                       const sph_GravityEPJ *epj, int32_t n_ep, const sph_GravitySPJ *spj,
                       int32_t n_sp, sph_Gravity *force) {
    if (!ctx) return SPH_ERR_INVALID_ARGUMENT;
    if (n_i < 0 || n_ep < 0 || n_sp < 0 || (n_i && (!epi || !force)) || (n_ep && !epj) || (n_sp && !spj))
        return set_error(ctx, SPH_ERR_INVALID_ARGUMENT, "bad functor arguments");
    int st = sph_dispatch_gravity(ctx, 0, 1, &epi, &n_i, &epj, &n_ep, &spj, &n_sp);
    if (st) return st;
    std::vector<sph_Gravity> tmp((size_t)std::max(n_i, 1));
    sph_Gravity *tp = tmp.data();
    st = sph_retrieve_gravity(ctx, 0, 1, &n_i, &tp);
    if (st && st != SPH_ERR_NONFINITE) return st;
    for (int k = 0; k < n_i; ++k) {
        for (int c = 0; c < 3; ++c) force[k].acc[c] += tmp[k].acc[c];
        force[k].pot += tmp[k].pot;
        force[k].eta += tmp[k].eta;
    }
    return st;
}
}  // namespace

extern "C" int sph_calc_gravity_ep(sph_context *ctx, const sph_GravityEPI *epi, int32_t n_i,
                                   const sph_GravityEPJ *epj, int32_t n_j, sph_Gravity *force) {
    return gravity_accumulate(ctx, epi, n_i, epj, n_j, nullptr, 0, force);
}

extern "C" int sph_calc_gravity_sp(sph_context *ctx, const sph_GravityEPI *epi, int32_t n_i,
                                   const sph_GravitySPJ *spj, int32_t n_j, sph_Gravity *force) {
    return gravity_accumulate(ctx, epi, n_i, nullptr, 0, spj, n_j, force);
}

// ---------------------------------------------------------------- bindings
// For the Python binding alone (functors.py), not in the ABI header: the
// pointers `offset` bytes into n objects.
extern "C" void sph_member_pointers(const void *const *obj, int64_t n, int64_t offset, void **out) {
    for (int64_t k = 0; k < n; ++k)
        std::memcpy(&out[k], static_cast<const char *>(obj[k]) + offset, sizeof(void *));
}

// ---------------------------------------------------------------- layout
extern "C" int64_t sph_abi_layout(int64_t *out, int64_t n) {
    std::vector<int64_t> v;
#define S(T) v.push_back(sizeof(T))
#define F(T, f) v.push_back(offsetof(T, f))
    S(sph_DensityEPI); F(sph_DensityEPI, id); F(sph_DensityEPI, mass); F(sph_DensityEPI, pos);
    F(sph_DensityEPI, vel); F(sph_DensityEPI, ksr); F(sph_DensityEPI, rs);
    S(sph_DensityEPJ); F(sph_DensityEPJ, id); F(sph_DensityEPJ, mass); F(sph_DensityEPJ, pos);
    F(sph_DensityEPJ, vel);
    S(sph_Density); F(sph_Density, dens); F(sph_Density, divv); F(sph_Density, rotv);
    F(sph_Density, grdh); F(sph_Density, ksr); F(sph_Density, np); F(sph_Density, itr);
#define HYDRO_TAIL(T) F(T, ksr); F(T, hinv); F(T, pres); F(T, presc); F(T, bswt); F(T, dens); \
    F(T, vsnd); F(T, alph); F(T, alphu); F(T, thrm); F(T, eta)
    S(sph_HydroEPI); F(sph_HydroEPI, id); F(sph_HydroEPI, pos); F(sph_HydroEPI, vel);
    HYDRO_TAIL(sph_HydroEPI);
    S(sph_HydroEPJ); F(sph_HydroEPJ, id); F(sph_HydroEPJ, mass); F(sph_HydroEPJ, pos);
    F(sph_HydroEPJ, vel); HYDRO_TAIL(sph_HydroEPJ);
    S(sph_Hydro); F(sph_Hydro, acch); F(sph_Hydro, accg); F(sph_Hydro, udot); F(sph_Hydro, vsmx);
    F(sph_Hydro, diffu);
    S(sph_GravityEPI); F(sph_GravityEPI, pos); F(sph_GravityEPI, eps2);
    S(sph_GravityEPJ); F(sph_GravityEPJ, mass); F(sph_GravityEPJ, pos); F(sph_GravityEPJ, eps2);
    S(sph_GravitySPJ); F(sph_GravitySPJ, mass); F(sph_GravitySPJ, pos); F(sph_GravitySPJ, eps2);
    S(sph_Gravity); F(sph_Gravity, acc); F(sph_Gravity, pot); F(sph_Gravity, eta);
#undef S
#undef F
#undef HYDRO_TAIL
    const int64_t m = (int64_t)v.size();
    if (out)
        for (int64_t k = 0; k < std::min(m, n); ++k) out[k] = v[k];
    return m;
}

// capi_internal.h — context state behind the C ABI (not installed).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <vector>

#include "../../include/sph_gb300.h"
#include "pair_kernels.cuh"

#define PAIR_WARPS 4

namespace sphrt {

// Device buffer that grows on demand (never inside stream capture).
template <class T>
struct DevBuf {
    T *p = nullptr;
    size_t cap = 0;
    int ensure(size_t n, bool zero = true) {
        if (n <= cap && p) return 0;
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
        size_t want = n + n / 4 + 64;
        if (cudaMalloc(&p, want * sizeof(T)) != cudaSuccess) {
            cudaGetLastError();
            p = nullptr;
            return 1;
        }
        // no buffer is ever read before it is written, but a field that a
        // caller leaves unset (e.g. the signal velocity before the first
        // force evaluation) then holds zeros, not stale memory; the memset is
        // waited for, as no other stream is ordered after it
        if (zero && (cudaMemset(p, 0, want * sizeof(T)) != cudaSuccess ||
                     cudaStreamSynchronize(cudaStreamLegacy) != cudaSuccess)) {
            cudaGetLastError();
            cudaFree(p);
            p = nullptr;
            return 1;
        }
        cap = want;
        return 0;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
    }
};

// Pinned host buffer that grows on demand.
template <class T>
struct HostBuf {
    T *p = nullptr;
    size_t cap = 0;
    int ensure(size_t n) {
        if (n <= cap && p) return 0;
        if (p) cudaFreeHost(p);
        p = nullptr;
        cap = 0;
        size_t want = n + n / 4 + 64;
        if (cudaMallocHost(&p, want * sizeof(T)) != cudaSuccess) {
            cudaGetLastError();
            p = nullptr;
            return 1;
        }
        cap = want;
        return 0;
    }
    void release() {
        if (p) cudaFreeHost(p);
        p = nullptr;
        cap = 0;
    }
};

// Buffers and dispatch state of one interaction kind (density/hydro/gravity).
struct KindState {
    HostBuf<char> h_in, h_out;
    DevBuf<char> d_in;
    // Device buffers of a dispatch, slices of one allocation: a new context's
    // first call makes one cudaMalloc instead of ~30 (density call of 64: 254 -> 163 us).
    DevBuf<char> arena;
    template <class T>
    struct Slice {
        T *p = nullptr;
    };
    Slice<dbl4> a4[8];
    Slice<float4> f4[20];   // FP32C double-float records; 16..19 hydro mark records
    Slice<int> hl_list;               // rows of the density and hydro sums
    Slice<int2> hl_ovf;               // particles without a row (particle, walk)
    Slice<double2> a2[2];
    Slice<long long> id[2];
    Slice<double> d1[2];
    Slice<double> o[5];
    Slice<long long> o_np;
    Slice<unsigned char> o_itr;
    Slice<int2> r_info;               // rows: entries and walk per particle
    Slice<int2> amb;                  // FP64 re-check queue of the density
    Slice<int4> long_items;           // items with lists left to a block each
    Slice<int> rowless;               // FP32C density: particles without a row, and items of them
    Slice<int4> rowless_items;
    std::vector<int4> items;
    std::vector<int> i_off;
    bool pending = false;
    int n_walk = 0;
    int flag_slot = 0;

    // places the slices: with a base, else only adds up their bytes
    struct Placer {
        char *base;
        size_t bytes = 0;
        template <class T>
        void operator()(Slice<T> &b, size_t n) {
            if (base) b.p = reinterpret_cast<T *>(base + bytes);
            bytes += (n * sizeof(T) + 256) / 256 * 256;
        }
    };
    template <class F>
    int ensure(F layout) {
        Placer size{nullptr};
        layout(size);
        if (arena.ensure(size.bytes, false)) return 1;
        Placer place{arena.p};
        layout(place);
        return 0;
    }
    int ensure_density(size_t ni, size_t nj, size_t n_amb, size_t n_items, size_t n_rowless, size_t n_walk) {
        return ensure([&](Placer &put) {
            put(a4[0], ni), put(a4[1], ni), put(id[0], ni), put(d1[0], ni), put(d1[1], ni);
            put(a4[2], nj), put(a4[3], nj), put(id[1], nj);
            for (int k = 0; k < 5; ++k) put(o[k], ni);
            put(o_np, ni), put(o_itr, ni);
            for (int k = 0; k < 4; ++k) put(f4[k], ni), put(f4[4 + k], nj);
            put(hl_list, ni * sphk::ROW_CAP), put(r_info, ni), put(hl_ovf, ni);
            put(amb, n_amb), put(long_items, n_items);
            if (n_rowless) put(rowless, n_rowless), put(rowless_items, n_rowless / 32 + n_walk);
        });
    }
    int ensure_hydro(size_t ni, size_t nj, size_t n_items) {
        return ensure([&](Placer &put) {
            put(a4[0], ni), put(a4[1], ni), put(a4[4], ni), put(a4[5], ni);
            put(a2[0], ni), put(id[0], ni);
            put(a4[2], nj), put(a4[3], nj), put(a4[6], nj), put(a4[7], nj);
            put(a2[1], nj), put(id[1], nj);
            put(o[0], 3 * ni), put(o[1], 3 * ni);
            for (int k = 2; k < 5; ++k) put(o[k], ni);
            for (int k = 0; k < 4; ++k) put(f4[k], ni), put(f4[4 + k], nj);
            for (int k = 8; k < 11; ++k) put(f4[k], ni), put(f4[k + 3], nj);
            put(f4[14], ni), put(f4[15], nj);
            put(f4[16], ni), put(f4[17], ni), put(f4[18], nj), put(f4[19], nj);
            put(hl_list, ni * sphk::ROW_CAP), put(r_info, ni), put(hl_ovf, ni);
            put(long_items, n_items);
        });
    }
    int ensure_gravity(size_t ni, size_t nj, size_t slices) {
        return ensure([&](Placer &put) {
            put(a4[0], ni), put(a4[2], nj), put(d1[0], nj);
            put(o[0], 3 * ni * slices), put(o[1], ni * slices), put(o[2], ni * slices);
            put(f4[0], ni), put(f4[1], ni), put(f4[4], nj), put(f4[5], nj);
        });
    }
    void release() {
        h_in.release();
        h_out.release();
        d_in.release();
        arena.release();
    }
};

}  // namespace sphrt

struct sph_context {
    sph_params prm;
    int sm_count = 0;
    cudaStream_t stream = nullptr;
    int *d_queue = nullptr;   // [0..2] work-queue counters, [3] density re-check count,
                              // [4] items of rowless particles, [5] their counter, [7] density
                              // sweep queue, [8] hydro rows that overflowed, [9..11] long items
    int *h_flags = nullptr;   // pinned: per kind, non-finite values in the outputs
    int grid[3][2] = {{0}};   // persistent grid per kind and precision
    int grid_stream = 0;      // persistent grid of the FP32C streamed density walk
    int grid_df = 0;          // resident blocks of the double-float hydro pass
    int grid_g64 = 0;         // persistent grid of the FP32C gravity kernel with a 64-entry j-tile
    sphrt::KindState kind[3];
    int n_systems = 0;        // live sph_system objects using this context
    char err[512] = {0};
};

namespace sphrt {
extern const float AMB_TOL;
int set_error(sph_context *ctx, int status, const char *fmt, ...);
int cuda_error(sph_context *ctx, cudaError_t e, const char *what);
// A stream for long items, with the events that fork it from the caller's
// stream and join it again.
struct LongSide {
    cudaStream_t stream = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
};
// FP32C density of a dispatch: what the items of its rowless particles need
// (density_stream over them where they are many).
struct RowlessItems {
    const int *i_off;
    int n_walk;
    int most;   // up to this many are swept by a block each
    int *list;
    int4 *items;
    int *n_items, *queue;
};
int pair_grid(const sph_context *ctx, int kind, int precision, int n_items);
void launch_mark_density(const sph_context *ctx, const sphk::MarkArgs &m, int mark_grid, int n_max, cudaStream_t s,
                         const LongSide *side = nullptr);
void launch_density(const sph_context *ctx, const sphk::MarkArgs &m, int mark_grid, const sphk::DensityArgs &a,
                    int n_max, int precision, cudaStream_t s, int *amb_total = nullptr, const LongSide *side = nullptr,
                    const RowlessItems *rowless = nullptr);
void launch_density_stream(const sph_context *ctx, const sphk::StreamArgs &w, bool sweep, const sphk::DensityArgs &a,
                           int n_max, cudaStream_t s, int *amb_total, const LongSide &side);
void launch_hydro_marks(const sph_context *ctx, const sphk::MarkArgs &m, int mark_grid, int n_i, int precision,
                        cudaStream_t s, const LongSide *side = nullptr);
void launch_hydro_sums(const sph_context *ctx, const sphk::HydroArgs &a, int precision, cudaStream_t s);
void launch_gravity(const sphk::GravityArgs &a, int precision, int grid, cudaStream_t s, int jtile);
}  // namespace sphrt

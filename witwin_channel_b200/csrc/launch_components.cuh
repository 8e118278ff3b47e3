// Definition of launch_components (launch.h); included by solve_f32.cu and
// solve_f64.cu.
#pragma once

#include "internal.h"
#include "kernels.cuh"
#include "launch.h"

namespace wcb {

// Warps per 32-cell tile of the reflection and diffraction kernels.  Few warps
// per tile keep their batches full and wait for nobody, but tiles take unequal
// times, so they need many waves to even out; eight warps share a tile when
// tiles are few.  Measured on one B200, ms of the kernels: reflection and
// visibility of the 1024^2 large city (32,768 tiles) 23.5 + 55.1 at 1, 22.7 + 53.2
// at 2; reflection of four transmitters on 128^2 and 320^2 (2,048 and 12,800
// tiles) 5.89 at 4, 5.71 at 2 for the larger; a 90 x 70 town (216 tiles) 4.5 at 8,
// 7.3 at 1 (whole call).  The UTD kernel, whose batches are dealt out evenly,
// wants more: 0.34 at 4 and 0.25 at 8 on the canyon (2,048 tiles), the same at 1
// and 2 on the city.  FP64 keeps eight: its warps' sums are rounded to FP32 before
// they are added, so another grouping would be another result.  In mixed precision
// the grouping, and with it the rounding of a cell's sum, follows the tile count of
// the whole call: a shard or a single transmitter of a larger map agrees with that
// map to FP32 rounding, not bit for bit.
template <typename T>
static int trace_tile_warps(long long tiles) {
    if (sizeof(T) == 8) return 8;
    return tiles >= 4096 ? 2 : tiles >= 1024 ? 4 : 8;
}
template <typename T>
static int utd_tile_warps(long long tiles) {
    if (sizeof(T) == 8) return 8;
    return tiles >= 16384 ? 2 : tiles >= 4096 ? 4 : 8;
}

// LoS+transmission and diffraction go on `stream`, reflection on `side` (its
// candidate tables were built there); the caller joins the streams before
// the finalize kernel.
template <typename T, int NF>
static void launch_nf(const MainParams& q0, unsigned blocks, int sdepth, size_t stack_bytes, cudaStream_t stream,
               cudaStream_t side, ComponentEvents* evs, const DiffractionPlan& dp) {
    const long long tiles = tiles_per_tx(q0) * q0.num_tx;
    const int tw = trace_tile_warps<T>(tiles), uw = utd_tile_warps<T>(tiles);
    const unsigned grid = unsigned((tiles * tw + kSplitWarps - 1) / kSplitWarps);
    const unsigned utd_grid = unsigned((tiles * uw + kSplitWarps - 1) / kSplitWarps);
    const size_t split_stack = size_t(sdepth) * kSplitBlock * 4;
    const int c = q0.components;
    MainParams q = q0;
    unsigned long long* rc = q0.ray_counter;
    if (c & 2) {
        if (evs) cudaEventRecord(evs->start[1], side);
        q.ray_counter = rc ? rc + 1 : nullptr;
        const size_t bytes = split_stack + kSplitWarps * sizeof(ReflShared<NF>) + size_t(kSplitWarps) * 32 * NF * 3 * 4;
        static std::atomic<unsigned long long> raised{0};
        raise_shared_limit((const void*)k_reflect<T, NF>, 200 * 1024, raised);
        k_reflect<T, NF><<<grid, kSplitBlock, bytes, side>>>(q, sdepth, tw);
        note_launch();
        if (evs) cudaEventRecord(evs->end[1], side);
    }
    if (evs) cudaEventRecord(evs->start[0], stream);
    if (c & (1 | 8)) {
        q.ray_counter = rc ? rc + 0 : nullptr;
        k_los_trans<T, NF><<<blocks, kCompBlock, stack_bytes, stream>>>(q);
        note_launch();
    }
    if (evs) cudaEventRecord(evs->end[0], stream);
    if (evs) cudaEventRecord(evs->start[2], stream);
    if ((c & 4) && dp.chunks > 0) {
        q.ray_counter = rc ? rc + 2 : nullptr;
        const size_t bytes = kSplitWarps * sizeof(DiffShared<NF>) + size_t(kSplitWarps) * 32 * NF * 9 * 4;
        static std::atomic<unsigned long long> raised_vis{0}, raised_utd{0};
        raise_shared_limit((const void*)k_diffract_vis<T>, 200 * 1024, raised_vis);
        raise_shared_limit((const void*)k_diffract_utd<T, NF>, 200 * 1024, raised_utd);
        for (int k = 0; k < dp.chunks; ++k) {
            const int j0 = k * dp.chunk;
            if (dp.run_vis) {
                std::pair<cudaEvent_t, cudaEvent_t> ev{nullptr, nullptr};
                if (evs) {
                    cudaEventCreate(&ev.first);
                    cudaEventCreate(&ev.second);
                    cudaEventRecord(ev.first, stream);
                }
                k_diffract_vis<T><<<grid, kSplitBlock, split_stack, stream>>>(q, tw, j0, dp.chunk, dp.words);
                note_launch();
                if (evs) {
                    cudaEventRecord(ev.second, stream);
                    evs->vis.push_back(ev);
                }
            }
            k_diffract_utd<T, NF><<<utd_grid, kSplitBlock, bytes, stream>>>(q, uw, j0, dp.chunk, dp.words,
                                                                           static_cast<T*>(dp.carry));
            note_launch();
        }
    }
    if (evs) cudaEventRecord(evs->end[2], stream);
}

template <typename T>
void launch_components(const MainParams& q, int nf, unsigned blocks, int sdepth, size_t stack_bytes, cudaStream_t stream,
                       cudaStream_t side, ComponentEvents* evs, const DiffractionPlan& dp) {
    switch (nf) {
        case 1: launch_nf<T, 1>(q, blocks, sdepth, stack_bytes, stream, side, evs, dp); break;
        case 2: launch_nf<T, 2>(q, blocks, sdepth, stack_bytes, stream, side, evs, dp); break;
        case 3: launch_nf<T, 3>(q, blocks, sdepth, stack_bytes, stream, side, evs, dp); break;
        default: launch_nf<T, 4>(q, blocks, sdepth, stack_bytes, stream, side, evs, dp); break;
    }
}

}  // namespace wcb

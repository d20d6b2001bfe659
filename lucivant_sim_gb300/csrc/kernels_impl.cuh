// Definitions behind kernels.cuh, included by the per-type translation units only.
#pragma once

#include "kernels.cuh"

namespace lsg {

static_assert(offsetof(BlockDesc, gb) == kDescGb && offsetof(BlockDesc, lob) == kDescOb && offsetof(BlockDesc, sob) == kDescOb + 8 &&
                  offsetof(BlockDesc, lconst) == kDescConst && offsetof(BlockDesc, lead) == kDescConst + 4 &&
                  offsetof(BlockDesc, lvec) == kDescConst + 8 && sizeof(OpRec) == 16,
              "the staged descriptors' layout");

template <typename T>
const void* PassKernels<T>::pipe() {
    return reinterpret_cast<const void*>(k_tile_pipe<T>);
}
template <typename T>
const void* PassKernels<T>::swz(int mode) {
    if constexpr (Elem<T>::complex) {
        if constexpr (sizeof(T) == 8)
            if (mode == kDrawn) return reinterpret_cast<const void*>(k_tile_pipe_swz<T, kDrawn>);
        if (mode == kRounds) return reinterpret_cast<const void*>(k_tile_pipe_swz<T, kRounds>);
        if (mode == kMixed) return reinterpret_cast<const void*>(k_tile_pipe_swz<T, kMixed>);
    }
    return reinterpret_cast<const void*>(k_tile_pipe_swz<T, kSwz>);
}
template <typename T>
const void* PassKernels<T>::pass() {
    return reinterpret_cast<const void*>(k_tile_pass<T>);
}
template <typename T>
const void* PassKernels<T>::ragged() {
    return reinterpret_cast<const void*>(k_tile_pipe_ragged<T>);
}
template <typename T>
void PassKernels<T>::launch_pipe(unsigned grid, size_t smem, cudaStream_t st, T* state, int64_t member_elems,
                                 const PassDesc* pass, const TileOp* ops, const BlockDesc* blocks, const T* data,
                                 int64_t tiles_per_member, int64_t total_tiles, int* status, const TrajCtx& ctx) {
    launch_chained(total_tiles <= 16 * (int64_t)grid, k_tile_pipe<T>, grid, kPipeThreads, smem, st, state, member_elems, pass, ops, blocks, data,
                   tiles_per_member, total_tiles, status, ctx);
}
template <typename T>
void PassKernels<T>::launch_swz(int mode, unsigned grid, size_t smem, cudaStream_t st, T* state, int64_t member_elems,
                                const PassDesc* pass, const TileOp* ops, const BlockDesc* blocks, const T* data,
                                int64_t tiles_per_member, int64_t total_tiles, int* status, const TrajCtx& ctx,
                                const Tmap& tmap) {
    auto launch = [&](auto kern, int threads) {
        launch_chained(total_tiles <= 16 * (int64_t)grid, kern, grid, threads, smem, st, state, member_elems, pass, ops, blocks, data, tiles_per_member,
                       total_tiles, status, ctx, tmap);
    };
    if constexpr (Elem<T>::complex) {
        if constexpr (sizeof(T) == 8)
            if (mode == kDrawn) return launch(k_tile_pipe_swz<T, kDrawn>, compute_threads<kDrawn>() + 32);
        if (mode == kRounds) return launch(k_tile_pipe_swz<T, kRounds>, compute_threads<kRounds>() + 32);
        if (mode == kMixed) return launch(k_tile_pipe_swz<T, kMixed>, kPipeThreads);
    }
    launch(k_tile_pipe_swz<T, kSwz>, kPipeThreads);
}
template <typename T>
void PassKernels<T>::launch_pass(unsigned grid, size_t smem, cudaStream_t st, T* state, int64_t member_elems,
                                 const PassDesc* pass, const TileOp* ops, const BlockDesc* blocks, const T* data,
                                 int64_t tiles_per_member, int64_t total_tiles, int* status, const TrajCtx& ctx) {
    k_tile_pass<T><<<grid, 256, smem, st>>>(state, member_elems, pass, ops, blocks, data, tiles_per_member, total_tiles,
                                            status, ctx);
}
template <typename T>
void PassKernels<T>::launch_ragged(unsigned grid, size_t smem, cudaStream_t st, const RaggedJob* jobs, int njobs,
                                   int* status) {
    k_tile_pipe_ragged<T><<<grid, kPipeThreads, smem, st>>>(jobs, njobs, status);
}

}  // namespace lsg

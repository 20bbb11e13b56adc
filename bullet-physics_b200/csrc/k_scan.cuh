// Ordered one-pass scans and compactions over tiles of items: each tile publishes its total, looks
// back over the tiles before it (decoupled look-back, Merrill and Garland 2016) and so learns
// where its output starts. One launch where a flag pass, a selection of two launches and a copy took
// four; on the small worlds that bound it is the launches that count.
#pragma once
#include "bgpu_kernels.cuh"

namespace bgpu {

constexpr uint32_t TILE_TB = 256;                  // threads of a tile's block
// ROUNDS: items a thread; round r holds items r * 256 + thread of the tile.
template <uint32_t ROUNDS>
__host__ __device__ __forceinline__ uint32_t tile_count(uint32_t n) {
    return (n + TILE_TB * ROUNDS - 1) / (TILE_TB * ROUNDS);
}

// The block's tile: tiles are dealt in order, so every tile before it has a running block. Every block of
// the launch takes one; the last to do so puts the ticket back.
__device__ __forceinline__ uint32_t tile_take(const TileScan& t) {
    __shared__ uint32_t s_tile;
    if (threadIdx.x == 0) {
        s_tile = atomicAdd(t.ticket, 1u);
        if (s_tile + 1u == gridDim.x) *t.ticket = 0u;
    }
    __syncthreads();
    return s_tile;
}

// A tile's word: epoch of the launch << 34 | state << 32 | value; state 1: the tile's total, 2: the
// total of all tiles up to it. The value travels in the word that says it is there.
__device__ __forceinline__ void tile_publish(const TileScan& t, uint32_t tile, uint32_t state, uint32_t value) {
    const unsigned long long w = (uint64_t(t.epoch) << 34) | (uint64_t(state) << 32) | value;
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(t.words + tile), "l"(w) : "memory");
}

// The sum of the totals of tiles [first, tile), for the whole block (all its threads call it; its
// last step is a block barrier). Each warp looks at 32 tiles, the block at 256 a round: a round
// costs a trip through L2, and with one warp's 32 the 900 tiles of a large pile's pairs took 28 of them
// (18 us). Bounded like every wait on the device: a tile that never publishes sets the status word.
__device__ __forceinline__ uint32_t tile_prefix(const TileScan& t, uint32_t tile, uint32_t first, uint32_t total) {
    constexpr uint32_t WARPS = TILE_TB / 32;
    __shared__ uint32_t s_sum[WARPS], s_full[WARPS];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (tile > first && threadIdx.x == 0) tile_publish(t, tile, 1u, total);
    uint32_t sum = 0;
    for (uint32_t back = 0, found = tile == first; !found; back += TILE_TB) {  // uniform across the block
        const uint32_t d = back + threadIdx.x + 1u;  // this thread looks d tiles back
        uint32_t state = 2u, value = 0u;             // before the first tile the sum is known to be 0
        if (tile - first >= d) {
            for (uint32_t spins = 0;;) {
                unsigned long long w;
                asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(t.words + (tile - d)));
                value = uint32_t(w);
                state = uint32_t(w >> 32) & 3u;
                if (uint32_t(w >> 34) == t.epoch && state != 0u) break;
                if (++spins > BARRIER_SPIN_LIMIT / 64u) {
                    atomicOr(t.status, ST_BARRIER_TIMEOUT);
                    state = 2u;
                    value = 0u;
                    break;
                }
            }
        }
        __syncwarp();
        const uint32_t full = __ballot_sync(0xffffffffu, state == 2u);
        const uint32_t last = full ? uint32_t(__ffs(int(full)) - 1) : 31u;
        const uint32_t part = __reduce_add_sync(0xffffffffu, lane <= last ? value : 0u);
        if (lane == 0) {
            s_sum[warp] = part;
            s_full[warp] = full;
        }
        __syncthreads();
        for (uint32_t k = 0; k < WARPS && !found; ++k) {
            sum += s_sum[k];
            found = s_full[k] != 0u;
        }
        __syncthreads();  // the sums are rewritten in the next round
    }
    if (threadIdx.x == 0) tile_publish(t, tile, 2u, sum + total);
    __syncthreads();
    return sum;
}

// Ranks of the flagged items of a block's tile in item order; returns their number.
template <uint32_t ROUNDS>
__device__ __forceinline__ uint32_t tile_ranks(const bool (&flag)[ROUNDS], uint32_t (&rank)[ROUNDS]) {
    constexpr uint32_t WARPS = TILE_TB / 32, N = WARPS * ROUNDS, PER = (N + 31) / 32;
    __shared__ uint32_t s_cnt[N], s_total;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (uint32_t r = 0; r < ROUNDS; ++r) {
        const uint32_t b = __ballot_sync(0xffffffffu, flag[r]);
        rank[r] = __popc(b & ((1u << lane) - 1u));
        if (lane == 0) s_cnt[r * WARPS + warp] = __popc(b);
    }
    __syncthreads();
    if (warp == 0) {
        uint32_t c[PER], own = 0;
#pragma unroll
        for (uint32_t k = 0; k < PER; ++k) {
            c[k] = lane * PER + k < N ? s_cnt[lane * PER + k] : 0u;
            own += c[k];
        }
        uint32_t x = own;
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31u) s_total = x;
        x -= own;
#pragma unroll
        for (uint32_t k = 0; k < PER; ++k) {
            if (lane * PER + k < N) s_cnt[lane * PER + k] = x;
            x += c[k];
        }
    }
    __syncthreads();
#pragma unroll
    for (uint32_t r = 0; r < ROUNDS; ++r) rank[r] += s_cnt[r * WARPS + warp];
    return s_total;
}

// Exclusive sums of the items' values over the tile in item order; returns the tile's total.
template <uint32_t ROUNDS>
__device__ __forceinline__ uint32_t tile_sums(const uint32_t (&value)[ROUNDS], uint32_t (&before)[ROUNDS]) {
    constexpr uint32_t WARPS = TILE_TB / 32, N = WARPS * ROUNDS;
    static_assert(N <= 32, "one warp scans the sums");
    __shared__ uint32_t s_sum[32], s_total;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (uint32_t r = 0; r < ROUNDS; ++r) {
        uint32_t x = value[r];
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        before[r] = x - value[r];
        if (lane == 31u) s_sum[r * WARPS + warp] = x;
    }
    __syncthreads();
    if (warp == 0) {
        const uint32_t c = lane < N ? s_sum[lane] : 0u;
        uint32_t x = c;
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        s_sum[lane] = x - c;
        if (lane == 31u) s_total = x;
    }
    __syncthreads();
#pragma unroll
    for (uint32_t r = 0; r < ROUNDS; ++r) before[r] += s_sum[r * WARPS + warp];
    return s_total;
}

}  // namespace bgpu

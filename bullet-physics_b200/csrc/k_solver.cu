// Sequential-impulse (PGS) solve over graph-coloured row groups, and the
// post-solve manifold writeback / lifecycle prune.
//
// The reference solves rows one by one in pair order (solver/
// sequential_impulse.rs:692-735, 743-802). Here the row group of each pair
// (its <= 4 contacts, solved in order by one thread) is a graph vertex; two
// groups conflict when they share a body with nonzero inverse mass. A
// Jones-Plassmann colouring with first-fit colour choice splits the groups
// into batches of pairwise-independent groups. Within a batch no dynamic body
// is touched twice, so the result is bit-identical to the reference's
// sequential solve over the same rows taken in (colour, pair) order.
//
// Worlds without joints use the chunked PGS (k_solve_flow): the bodies are cut into chunks (in Morton
// order where the broad phase has a tree, in index order where it has none), one per block of a
// cooperative launch, and each warp solves its share of the chunk's groups colour by colour,
// waiting only for the versions of its groups' own velocities (a version rides in the fourth word
// of a velocity). A group's contacts are spread over lanes (one
// contact per lane, the velocities handed from lane to lane in contact order), and the split
// sweep s rides in the phases of velocity sweep s + 1. Worlds with joints use the team kernel
// (k_solve): a persistent cooperative launch split into two teams of blocks with their own
// grid barriers, the velocity team running the warm start, the velocity sweeps and the joint
// rows, the split team the split-impulse sweeps, which touch only the push velocities and so
// run at the same time. The warm start computes the per-contact terms that stay fixed during
// the solve (tangent basis, Iw^-1 (r x d)) once and stores them in a contact table in
// batch-slot order, so the later sweeps run only the impulse update, reading the table with
// coalesced loads.
//
// Rows store only the contact frame (normal, lever arms), the bias terms, the
// effective masses and the accumulated impulses; the tangent basis, the
// angular components Iw^-1 (r x d) and the velocity couplings are recomputed
// from the per-body world inverse inertia with the reference's arithmetic, so
// they equal the values the reference precomputes in prepare().
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <cooperative_groups.h>
#include <cub/cub.cuh>
#include "k_scan.cuh"

namespace bgpu {

namespace {

constexpr uint32_t NO_COLOUR = 0xffffffffu;
constexpr int MAX_ROUNDS = 1024;

__device__ __forceinline__ uint32_t mix32(uint64_t k) {
    uint32_t h = uint32_t(k) ^ uint32_t(k >> 32) * 0x9E3779B1u;
    h ^= h >> 16;
    h *= 0x85EBCA6Bu;
    h ^= h >> 13;
    h *= 0xC2B2AE35u;
    h ^= h >> 16;
    return h;
}

__device__ __forceinline__ float inv_mass_of(const float4* __restrict__ iw, uint32_t i) { return iw[3 * i + 2].y; }

__device__ __forceinline__ M3 load_iw(const float4* __restrict__ iw, uint32_t i, float& inv_mass) {
    float4 a = __ldg(&iw[3 * i]), b = __ldg(&iw[3 * i + 1]), c = __ldg(&iw[3 * i + 2]);
    inv_mass = c.y;
    return M3{V3{a.x, a.y, a.z}, V3{a.w, b.x, b.y}, V3{b.z, b.w, c.x}};
}

// The pairs with rows, ascending, and their number; scalars[12]: every world prunes (step.rs:1006-1010).
template <uint32_t ROUNDS>
__global__ void __launch_bounds__(TILE_TB) k_contact_list(uint32_t npairs, const uint32_t* __restrict__ row_count,
                                                          uint32_t* contact_pairs, uint32_t* scalars,
                                                          const uint32_t* __restrict__ simulate,
                                                          const uint32_t* __restrict__ prev_simulate, uint32_t worlds,
                                                          TileScan ts) {
    const uint32_t tile = tile_take(ts), base = tile * (TILE_TB * ROUNDS);
    bool flag[ROUNDS];
    uint32_t rank[ROUNDS];
#pragma unroll
    for (uint32_t r = 0; r < ROUNDS; ++r) {
        const uint32_t p = base + r * TILE_TB + threadIdx.x;
        flag[r] = p < npairs && row_count[p] > 0;
    }
    const uint32_t total = tile_ranks(flag, rank);
    const uint32_t at = tile_prefix(ts, tile, 0u, total);
#pragma unroll
    for (uint32_t r = 0; r < ROUNDS; ++r)
        if (flag[r]) contact_pairs[at + rank[r]] = base + r * TILE_TB + threadIdx.x;
    if (base + TILE_TB * ROUNDS >= npairs && threadIdx.x == 0) scalars[2] = at + total;
    if (tile == 0u && worlds) {
        bool all = true;
#pragma unroll 4
        for (uint32_t w = threadIdx.x; w < worlds; w += TILE_TB)
            all &= (simulate[w] != 0u) & (prev_simulate[w] != 0u);  // (no short cut: the loads overlap)
        if (__syncthreads_and(all ? 1 : 0) && threadIdx.x == 0) scalars[12] = 1u;
    }
}

// Tiles of 4,096 pairs from 256k pairs on: the look-back's rounds count there (918k pairs: 13.7 us
// with tiles of 1,024), with fewer pairs the blocks.
void launch_contact_list(uint32_t npairs, PairData& pd, const StepParams& sp, uint32_t* status, cudaStream_t s) {
    auto go = [&](auto kernel, uint32_t tiles) {
        kernel<<<tiles, TILE_TB, 0, s>>>(npairs, pd.row_count.p, pd.contact_pairs.p, pd.scalars.p, sp.simulate,
                                         sp.prev_simulate, sp.worlds, pd.list_scan.begin(tiles, status, s));
    };
    if (npairs > (1u << 18)) go(k_contact_list<16>, tile_count<16>(npairs));
    else go(k_contact_list<4>, tile_count<4>(npairs));
}

struct ColourArgs {
    const uint32_t* count;  // number of contact pairs
    const uint32_t* contact_pairs;
    const uint64_t* pairs;
    const float4* iw;
    uint32_t* colour;
    unsigned long long* prio;
    unsigned long long* mask;
    unsigned long long* dup;      // 2 words per body: colours seeded twice at the body
    unsigned long long* used;     // 4 words per body, zeroed here for the histogram pass (null: not wanted)
    const float4* entries;        // this step's manifold entries (their meta carries last step's colour)
    uint32_t seed;                // 1: start from last step's colours
    unsigned int* bar;  // [0] barrier counter, [5] colour max, [6] [7] uncoloured-list lengths
    uint32_t* status;
    uint32_t* zero;     // nzero words to clear for the kernels after this one
    uint32_t nzero;
};

__device__ __forceinline__ unsigned long long* colour_word(unsigned long long* m, uint32_t x, uint32_t c) {
    return &m[2 * x + (c >> 6)];
}

// Seeding, then Jones-Plassmann rounds. Seeding: a group whose pair kept its
// manifold starts from the colour it had last step (kept in the entry's meta
// bits); a seed is dropped, for every group that claims it, when two groups
// claim the same colour at one dynamic body - so the result does not depend on
// the order of the atomics. The bits of dropped seeds stay in the masks and
// only make those colours unavailable there. Jones-Plassmann: an uncoloured
// group wins when its priority is the maximum over the uncoloured groups at
// both of its dynamic bodies; winners take the lowest colour free at both.
//
// The rounds walk a list of the still-uncoloured groups (rebuilt by each round
// from its losers), so a round costs what is left to colour, not the whole
// set; once the list fits one block, that block finishes the rounds alone with
// block-local syncs and the rest of the grid exits. Which groups win in a
// round depends only on the priorities, so the colours do not depend on the
// list order or on which threads run the rounds.
struct JpList {
    uint32_t* items[2];
    unsigned int* len[2];
};

// Appends k to a list: one atomicAdd per group of lanes that append together.
__device__ __forceinline__ void list_append(uint32_t* items, unsigned int* len, uint32_t k) {
    cooperative_groups::coalesced_group g = cooperative_groups::coalesced_threads();
    unsigned int base = 0;
    if (g.thread_rank() == 0) base = atomicAdd(len, g.size());
    base = g.shfl(base, 0);
    items[base + g.thread_rank()] = k;
}

// One Jones-Plassmann round over list r & 1; losers go to list (r + 1) & 1.
// [lo, n) with step `step` is this thread's share of the list.
__device__ __forceinline__ void jp_clear(const ColourArgs& a, const uint32_t* list, uint32_t n, uint32_t lo, uint32_t step) {
    for (uint32_t i = lo; i < n; i += step) {
        const uint64_t key = a.pairs[a.contact_pairs[list[i]]];
        a.prio[key_lo(key)] = 0ull;
        a.prio[key_hi(key)] = 0ull;
    }
}

__device__ __forceinline__ void jp_bid(const ColourArgs& a, const uint32_t* list, uint32_t n, uint32_t lo, uint32_t step) {
    for (uint32_t i = lo; i < n; i += step) {
        const uint32_t k = list[i];
        const uint64_t key = a.pairs[a.contact_pairs[k]];
        const uint32_t u = key_lo(key), v = key_hi(key);
        const unsigned long long pr = (uint64_t(mix32(key)) << 32) | k;
        if (inv_mass_of(a.iw, u) > 0.0f) atomicMax(&a.prio[u], pr);
        if (inv_mass_of(a.iw, v) > 0.0f) atomicMax(&a.prio[v], pr);
    }
}

// The colour count (bar[5]) is raised once per block: each warp folds its lanes'
// colours into the block's shared maximum, which colour_max_flush publishes.
__device__ __forceinline__ void warp_colour_max(unsigned int* s_cmax, uint32_t top) {
    top = __reduce_max_sync(0xffffffffu, top);
    if ((threadIdx.x & 31u) == 0 && top) atomicMax(s_cmax, top);
}

__device__ __forceinline__ void colour_max_flush(const unsigned int* s_cmax, unsigned int* bar5) {
    __syncthreads();
    if (threadIdx.x == 0 && *s_cmax) atomicMax(bar5, *s_cmax);
}

__device__ __forceinline__ void jp_pick(const ColourArgs& a, const uint32_t* list, uint32_t n, uint32_t lo, uint32_t step,
                                        uint32_t* losers, unsigned int* nlosers, unsigned int* s_cmax) {
    uint32_t top = 0;
    for (uint32_t i = lo; i < n; i += step) {
        const uint32_t k = list[i];
        const uint64_t key = a.pairs[a.contact_pairs[k]];
        const uint32_t u = key_lo(key), v = key_hi(key);
        const unsigned long long pr = (uint64_t(mix32(key)) << 32) | k;
        const bool du = inv_mass_of(a.iw, u) > 0.0f, dv = inv_mass_of(a.iw, v) > 0.0f;
        const bool win = (!du || __ldcg(&a.prio[u]) == pr) && (!dv || __ldcg(&a.prio[v]) == pr);
        if (!win) {
            list_append(losers, nlosers, k);
            continue;
        }
        unsigned long long m0 = 0, m1 = 0;
        if (du) { m0 |= __ldcg(&a.mask[2 * u]); m1 |= __ldcg(&a.mask[2 * u + 1]); }
        if (dv) { m0 |= __ldcg(&a.mask[2 * v]); m1 |= __ldcg(&a.mask[2 * v + 1]); }
        uint32_t c;
        if (~m0) c = uint32_t(__ffsll((long long)~m0) - 1);
        else if (~m1) c = 64u + uint32_t(__ffsll((long long)~m1) - 1);
        else { c = MAX_COLOURS - 1; atomicOr(a.status, ST_COLOUR_OVERFLOW); }
        a.colour[k] = c;
        const unsigned long long b0 = c < 64 ? (1ull << c) : 0ull, b1 = c >= 64 ? (1ull << (c - 64)) : 0ull;
        if (du) { a.mask[2 * u] |= b0; a.mask[2 * u + 1] |= b1; }
        if (dv) { a.mask[2 * v] |= b0; a.mask[2 * v + 1] |= b1; }
        top = max(top, c + 1u);
    }
    warp_colour_max(s_cmax, top);
}

__global__ void k_colour(ColourArgs a, JpList wl) {
    const uint32_t K = *a.count;
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t stride = gridDim.x * blockDim.x;
    const unsigned int nblocks = gridDim.x;
    unsigned int nbar = 0;
    __shared__ unsigned int s_cmax;
    if (threadIdx.x == 0) s_cmax = 0u;
    for (uint32_t k = tid; k < a.nzero; k += stride) a.zero[k] = 0u;
    for (uint32_t k = tid; k < K; k += stride) {
        a.colour[k] = NO_COLOUR;
        uint64_t key = a.pairs[a.contact_pairs[k]];
        uint32_t u = key_lo(key), v = key_hi(key);
        a.mask[2 * u] = 0ull; a.mask[2 * u + 1] = 0ull;
        a.mask[2 * v] = 0ull; a.mask[2 * v + 1] = 0ull;
        if (a.seed) {
            a.dup[2 * u] = 0ull; a.dup[2 * u + 1] = 0ull;
            a.dup[2 * v] = 0ull; a.dup[2 * v + 1] = 0ull;
        } else {
            wl.items[0][k] = k;  // every group starts uncoloured
        }
        if (a.used) {
            for (uint32_t x = 0; x < 4; ++x) a.used[4 * u + x] = a.used[4 * v + x] = 0ull;
        }
    }
    if (tid == 0) {
        a.bar[5] = 0;
        *wl.len[0] = a.seed ? 0u : K;
        *wl.len[1] = 0u;
    }
    team_barrier(a.bar, ++nbar * nblocks, a.status);
    if (a.seed) {
        for (uint32_t k = tid; k < K; k += stride) {  // claim last step's colour at both bodies
            const uint32_t p = a.contact_pairs[k];
            const uint32_t cs = (__float_as_uint(a.entries[size_t(p) * ENTRY_F4 + 2].w) >> META_COLOUR_SHIFT) & 0xffu;
            if (cs == 0u || cs > MAX_COLOURS) continue;
            const uint32_t c = cs - 1u;
            const unsigned long long bit = 1ull << (c & 63u);
            const uint64_t key = a.pairs[p];
            const uint32_t u = key_lo(key), v = key_hi(key);
            if (inv_mass_of(a.iw, u) > 0.0f && (atomicOr(colour_word(a.mask, u, c), bit) & bit))
                atomicOr(colour_word(a.dup, u, c), bit);
            if (inv_mass_of(a.iw, v) > 0.0f && (atomicOr(colour_word(a.mask, v, c), bit) & bit))
                atomicOr(colour_word(a.dup, v, c), bit);
        }
        team_barrier(a.bar, ++nbar * nblocks, a.status);
        uint32_t top = 0;
        for (uint32_t k = tid; k < K; k += stride) {  // keep the seeds claimed once at each body
            const uint32_t p = a.contact_pairs[k];
            const uint32_t cs = (__float_as_uint(a.entries[size_t(p) * ENTRY_F4 + 2].w) >> META_COLOUR_SHIFT) & 0xffu;
            bool keep = false;
            uint32_t c = 0;
            if (cs != 0u && cs <= MAX_COLOURS) {
                c = cs - 1u;
                const unsigned long long bit = 1ull << (c & 63u);
                const uint64_t key = a.pairs[p];
                const uint32_t u = key_lo(key), v = key_hi(key);
                const bool du = inv_mass_of(a.iw, u) > 0.0f && (__ldcg(colour_word(a.dup, u, c)) & bit);
                const bool dv = inv_mass_of(a.iw, v) > 0.0f && (__ldcg(colour_word(a.dup, v, c)) & bit);
                keep = !du && !dv;
            }
            if (keep) {
                a.colour[k] = c;
                top = max(top, c + 1u);
            } else {
                list_append(wl.items[0], wl.len[0], k);
            }
        }
        warp_colour_max(&s_cmax, top);
        colour_max_flush(&s_cmax, &a.bar[5]);
        team_barrier(a.bar, ++nbar * nblocks, a.status);
    }
    // Rounds on the whole grid while the list is longer than one block. The list
    // length is read once per block, so every thread of a block takes the same path
    // (even after a barrier timeout, when lengths may still be changing).
    __shared__ unsigned int s_len;
    auto list_len = [&](uint32_t which) -> uint32_t {
        if (threadIdx.x == 0) s_len = *(volatile unsigned int*)wl.len[which];
        __syncthreads();
        const uint32_t v = s_len;
        __syncthreads();
        return v;
    };
    int round = 0;
    for (; round < MAX_ROUNDS; ++round) {
        const uint32_t cur = uint32_t(round) & 1u, nxt = cur ^ 1u;
        const uint32_t n = list_len(cur);
        if (n <= blockDim.x) break;
        jp_clear(a, wl.items[cur], n, tid, stride);
        if (tid == 0) *wl.len[nxt] = 0u;  // last read (as this list's length) before the previous barrier
        team_barrier(a.bar, ++nbar * nblocks, a.status);
        jp_bid(a, wl.items[cur], n, tid, stride);
        team_barrier(a.bar, ++nbar * nblocks, a.status);
        jp_pick(a, wl.items[cur], n, tid, stride, wl.items[nxt], wl.len[nxt], &s_cmax);
        colour_max_flush(&s_cmax, &a.bar[5]);
        team_barrier(a.bar, ++nbar * nblocks, a.status);
        if (__syncthreads_or((*(volatile uint32_t*)a.status & ST_BARRIER_TIMEOUT) != 0u)) return;
    }
    // The short tail: block 0 alone, one group per thread.
    if (blockIdx.x != 0) return;
    for (; round < MAX_ROUNDS; ++round) {
        const uint32_t cur = uint32_t(round) & 1u, nxt = cur ^ 1u;
        const uint32_t n = list_len(cur);
        if (n == 0) break;
        jp_clear(a, wl.items[cur], n, threadIdx.x, blockDim.x);
        if (threadIdx.x == 0) *wl.len[nxt] = 0u;
        __syncthreads();
        jp_bid(a, wl.items[cur], n, threadIdx.x, blockDim.x);
        __syncthreads();
        jp_pick(a, wl.items[cur], n, threadIdx.x, blockDim.x, wl.items[nxt], wl.len[nxt], &s_cmax);
        __syncthreads();
    }
    colour_max_flush(&s_cmax, &a.bar[5]);
    if (round >= MAX_ROUNDS && threadIdx.x == 0) atomicOr(a.status, ST_COLOUR_ROUNDS);
}

// Colour histograms of all groups and of the groups with split-active rows,
// plus the row and split-row totals.
// With chunk histograms (vhist non-null) the pass also counts each group into its (colour,
// chunk) bins and marks its colour at its dynamic bodies (chunk_count, with the chunked PGS's
// code below).
__device__ __forceinline__ void chunk_count(const uint64_t* __restrict__ pairs, uint32_t p, uint32_t c, uint32_t rows,
                                            bool split, const float4* __restrict__ iw,
                                            const uint32_t* __restrict__ chunk_of, uint32_t P, uint32_t* vhist,
                                            uint32_t* shist, unsigned long long* used);

__global__ void k_colour_hist(const uint32_t* __restrict__ count, const uint32_t* __restrict__ contact_pairs,
                              const uint32_t* __restrict__ colour, const uint32_t* __restrict__ row_count,
                              const float4* __restrict__ rows, uint32_t* hist, uint32_t* split_hist, uint32_t* split_flag,
                              uint32_t* sub_hist, const uint64_t* __restrict__ pairs, const float4* __restrict__ iw,
                              const uint32_t* __restrict__ chunk_of, uint32_t P, uint32_t* vhist, uint32_t* shist,
                              unsigned long long* used) {
    // Block-local histograms; [MAX_COLOURS] rows, [MAX_COLOURS + 1] split-active rows;
    // shc: groups per (colour, row count - 1).
    __shared__ uint32_t sh[MAX_COLOURS + 2], ssh[MAX_COLOURS], shc[MAX_COLOURS * 4];
    for (uint32_t i = threadIdx.x; i < MAX_COLOURS + 2; i += blockDim.x) sh[i] = 0;
    for (uint32_t i = threadIdx.x; i < MAX_COLOURS; i += blockDim.x) ssh[i] = 0;
    for (uint32_t i = threadIdx.x; i < MAX_COLOURS * 4; i += blockDim.x) shc[i] = 0;
    __syncthreads();
    uint32_t K = *count;
    uint32_t nrows = 0, nsplit_rows = 0;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < K; k += gridDim.x * blockDim.x) {
        uint32_t c = colour[k];
        if (c >= MAX_COLOURS) {  // colouring gave up (its status bit is set): the group is not solved
            split_flag[k] = 0u;
            continue;
        }
        atomicAdd(&sh[c], 1u);
        uint32_t p = contact_pairs[k];
        uint32_t n = row_count[p];
        atomicAdd(&shc[c * 4 + (n - 1)], 1u);
        nrows += n;
        uint32_t nsr = 0;  // split-active rows
        for (uint32_t r = 0; r < n; ++r) nsr += rows[(size_t(p) * 4 + r) * ROW_F4 + 5].z != 0.0f ? 1u : 0u;
        split_flag[k] = nsr ? 1u : 0u;
        if (nsr) {
            nsplit_rows += nsr;
            atomicAdd(&ssh[c], 1u);
        }
        if (vhist) chunk_count(pairs, p, c, n, nsr != 0u, iw, chunk_of, P, vhist, shist, used);
    }
    nrows = __reduce_add_sync(0xffffffffu, nrows);
    nsplit_rows = __reduce_add_sync(0xffffffffu, nsplit_rows);
    if ((threadIdx.x & 31u) == 0u) {
        if (nrows) atomicAdd(&sh[MAX_COLOURS], nrows);
        if (nsplit_rows) atomicAdd(&sh[MAX_COLOURS + 1], nsplit_rows);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < MAX_COLOURS; i += blockDim.x) {
        if (sh[i]) atomicAdd(&hist[i], sh[i]);
        if (ssh[i]) atomicAdd(&split_hist[i], ssh[i]);
    }
    for (uint32_t i = threadIdx.x; i < MAX_COLOURS * 4; i += blockDim.x)
        if (shc[i]) atomicAdd(&sub_hist[i], shc[i]);
    if (threadIdx.x == 0) {
        if (sh[MAX_COLOURS]) atomicAdd(&hist[MAX_COLOURS + 1], sh[MAX_COLOURS]);
        if (sh[MAX_COLOURS + 1]) atomicAdd(&hist[MAX_COLOURS + 2], sh[MAX_COLOURS + 1]);
    }
}

// Offsets of the colour batches; scalars [3] rows [4] colours [5] split groups
// [10] split rows [11] largest split batch. One warp, four raw colours a lane.
// Colours without groups are dropped (remap: colour -> dense colour), batches start on
// multiples of 32 (one warp's slots never straddle two batches), so a batch's start is the sum
// of the earlier batches' sizes rounded up to 32. Inside a batch the groups with 4 rows come
// first, then 3, 2, 1 (sub_cursor: the scatter's cursor of each part), so most warps hold
// groups of one size: their lanes run the same number of contacts and read the table's contact
// planes without gaps. The split batches keep their cursors; after the scatter they hold the
// split batch ends. (chunked: the scatter takes per-(colour, chunk) cursors, so the batch ends
// are written here.)
__global__ void k_colour_scan(uint32_t* hist, uint32_t* offset, uint32_t* cursor, uint32_t* split_hist,
                              uint32_t* split_offset, uint32_t* split_cursor, const unsigned int* bar, uint32_t* scalars,
                              uint32_t* remap, const uint32_t* sub_hist, uint32_t* sub_cursor, uint32_t chunked) {
    static_assert(MAX_COLOURS == 128, "four raw colours a lane");
    if (blockIdx.x != 0 || threadIdx.x >= 32u) return;
    const uint32_t lane = threadIdx.x;
    const uint32_t nraw = bar[5];
    uint32_t h[4], sh[4], cnt = 0, pad = 0, spad = 0, smax = 0, sg = 0;
    for (uint32_t k = 0; k < 4; ++k) {
        const uint32_t c = 4u * lane + k;
        h[k] = c < nraw ? hist[c] : 0u;
        sh[k] = h[k] ? split_hist[c] : 0u;
        if (h[k]) {
            ++cnt;
            pad += (h[k] + 31u) & ~31u;
            spad += (sh[k] + 31u) & ~31u;
            smax = max(smax, sh[k]);
            sg += sh[k];
        }
    }
    uint32_t d = cnt, acc = pad, sacc = spad;  // inclusive scans, then exclusive
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, d, o), y = __shfl_up_sync(0xffffffffu, acc, o),
                       z = __shfl_up_sync(0xffffffffu, sacc, o);
        if (lane >= o) { d += x; acc += y; sacc += z; }
    }
    const uint32_t ncol = __shfl_sync(0xffffffffu, d, 31);
    d -= cnt;
    acc -= pad;
    sacc -= spad;
    for (uint32_t k = 0; k < 4; ++k) {
        if (!h[k]) continue;
        const uint32_t c = 4u * lane + k;
        remap[c] = d;
        offset[d] = acc;
        uint32_t part = acc;
        for (uint32_t n = 4; n >= 1; --n) {
            sub_cursor[d * 4 + (n - 1)] = part;
            part += sub_hist[c * 4 + (n - 1)];
        }
        cursor[d] = acc + h[k];  // the batch end
        split_offset[d] = sacc;
        split_cursor[d] = chunked ? sacc + sh[k] : sacc;
        if (d + 1u == ncol) {  // the last batch: the ends, unpadded
            offset[ncol] = acc + h[k];
            split_offset[ncol] = sacc + sh[k];
        }
        acc += (h[k] + 31u) & ~31u;
        sacc += (sh[k] + 31u) & ~31u;
        ++d;
    }
    for (uint32_t o = 16; o > 0; o >>= 1) {
        smax = max(smax, __shfl_xor_sync(0xffffffffu, smax, o));
        sg += __shfl_xor_sync(0xffffffffu, sg, o);
    }
    if (lane == 0) {
        if (ncol == 0) {
            offset[0] = 0u;
            split_offset[0] = 0u;
        }
        scalars[3] = hist[MAX_COLOURS + 1];
        scalars[4] = ncol;
        scalars[5] = sg;
        scalars[10] = hist[MAX_COLOURS + 2];
        scalars[11] = smax;
    }
}

// One atomicAdd per distinct colour among the calling lanes of a warp.
__device__ __forceinline__ uint32_t claim_slot(uint32_t* cursor, uint32_t c) {
    uint32_t active = __activemask();
    uint32_t peers = __match_any_sync(active, c);
    uint32_t lane = threadIdx.x & 31u;
    uint32_t leader = uint32_t(__ffs(int(peers)) - 1);
    uint32_t rank = uint32_t(__popc(peers & ((1u << lane) - 1u)));
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(&cursor[c], uint32_t(__popc(int(peers))));
    base = __shfl_sync(peers, base, int(leader));
    return base + rank;
}

// ---------------------------------------------------------------- chunks (chunked PGS)
// The chunked PGS deals each colour batch to the blocks of the launch by chunk: a chunk is a
// run of bodies in Morton order (the broad phase's tree leaves; without a tree in index order), and a
// group belongs to the chunk of its first dynamic body. Block b solves chunk b's groups of every colour.
//
// Ordering: within a sweep a dynamic body is updated by its groups in colour order, so its
// velocity goes through a chain of versions known before the solve starts: the group with rank r
// among the body's d groups finds version s d + r in sweep s and leaves version s d + r + 1.
// The colours of a body's groups are a bit mask (two 64-bit words), so d is its population count
// and r the count of the bits below the group's colour; both ride in the group's slot record.
constexpr uint32_t CHUNK_MAX = 1024;         // blocks of a chunked launch
constexpr uint32_t CHUNK_TB = 384;           // threads of a chunk block (one block per SM)
constexpr uint32_t SMALL_TB = 128;           // threads of a block when one chunk has many (a warp a scheduler)

__device__ __forceinline__ uint32_t group_owner(uint32_t ia, uint32_t ib, const float4* __restrict__ iw,
                                                const uint32_t* __restrict__ chunk_of, uint32_t P) {
    return min(chunk_of[inv_mass_of(iw, ia) > 0.0f ? ia : ib], P - 1u);
}

// Bodies in Morton order cut into P equal runs; with no tree, runs of body indices. (Dynamic
// bodies are all in the tree when there is one; other bodies own no group.) Also clears the version
// tags of the bodies' velocity words (vel, 2 float4 a body, velocities then push velocities).
__global__ void k_chunk_of(uint32_t n, uint32_t P, const uint32_t* __restrict__ leaf, uint32_t m, uint32_t* chunk_of,
                           float4* vel) {
    const uint32_t lim = leaf ? m : n;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 4u * n; i += gridDim.x * blockDim.x) {
        vel[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (i < lim) chunk_of[leaf ? leaf[i] : i] = uint32_t(uint64_t(i) * P / lim);
    }
}

// Groups per (colour, chunk, row count) and split groups per (colour, chunk), and the colours of
// the groups (words 0, 1) and split groups (words 2, 3) at their dynamic bodies (k_colour_hist's
// pass, for each group).
__device__ __forceinline__ void chunk_count(const uint64_t* __restrict__ pairs, uint32_t p, uint32_t c, uint32_t rows,
                                            bool split, const float4* __restrict__ iw,
                                            const uint32_t* __restrict__ chunk_of, uint32_t P, uint32_t* vhist,
                                            uint32_t* shist, unsigned long long* used) {
    const uint64_t key = pairs[p];
    const uint32_t ia = key_lo(key), ib = key_hi(key);
    const uint32_t B = group_owner(ia, ib, iw, chunk_of, P);
    atomicAdd(&vhist[(size_t(c) * P + B) * 4 + (rows - 1)], 1u);
    if (split) atomicAdd(&shist[size_t(c) * P + B], 1u);
    const unsigned long long bit = 1ull << (c & 63u);
    for (uint32_t side = 0; side < 2; ++side) {
        const uint32_t x = side ? ib : ia;
        if (!(inv_mass_of(iw, x) > 0.0f)) continue;
        atomicOr(&used[4 * size_t(x) + (c >> 6)], bit);
        if (split) atomicOr(&used[4 * size_t(x) + 2 + (c >> 6)], bit);
    }
}

// A group's rank among its body's groups | the number of them << 8 (0: the body is not dynamic);
// m: the two mask words.
__device__ __forceinline__ uint32_t colour_rank(const unsigned long long* __restrict__ m, uint32_t c) {
    const unsigned long long lo = m[0], hi = m[1];
    const unsigned long long below = (1ull << (c & 63u)) - 1ull;
    const uint32_t r = c < 64u ? __popcll(lo & below) : __popcll(lo) + __popcll(hi & below);
    return r | ((__popcll(lo) + __popcll(hi)) << 8);
}

// One block per raw colour: the colour's batch is laid out chunk by chunk (inside a chunk the
// groups with 4 rows first, then 3, 2, 1), so the counts become the scatter's cursors and the
// chunk bins [voff[d (P + 1) + b], voff[d (P + 1) + b + 1]) of dense colour d with the bin's
// groups of 4, 3, 2 and 1 rows in vsec[(d P + b) 4 + 0..3]; the same for the split batch (one
// part per chunk).
template <int TB>
__global__ void __launch_bounds__(TB) k_chunk_scan(uint32_t P, const uint32_t* __restrict__ hist,
                                                   const uint32_t* __restrict__ remap,
                                                   const uint32_t* __restrict__ offset,
                                                   const uint32_t* __restrict__ split_offset,
                                                   const unsigned int* __restrict__ bar, uint32_t* vhist,
                                                   uint32_t* shist, uint32_t* voff, uint32_t* soff, uint32_t* vsec) {
    using Scan = cub::BlockScan<uint32_t, TB>;
    __shared__ typename Scan::TempStorage tmp;
    const uint32_t c = blockIdx.x;
    if (c >= bar[5] || hist[c] == 0) return;
    const uint32_t d = remap[c];
    const uint32_t per = (P + TB - 1) / TB;  // chunks per thread
    const uint32_t b0 = min(P, threadIdx.x * per), b1 = min(P, b0 + per);
    uint32_t* vh = vhist + size_t(c) * P * 4;
    uint32_t* sh = shist + size_t(c) * P;
    uint32_t vsum = 0, ssum = 0;
    for (uint32_t b = b0; b < b1; ++b) {
        for (uint32_t n = 0; n < 4; ++n) vsum += vh[b * 4 + n];
        ssum += sh[b];
    }
    uint32_t vx, sx;
    Scan(tmp).ExclusiveSum(vsum, vx);
    __syncthreads();  // the scan's temporary storage is reused
    Scan(tmp).ExclusiveSum(ssum, sx);
    uint32_t vpos = offset[d] + vx, spos = split_offset[d] + sx;
    for (uint32_t b = b0; b < b1; ++b) {
        voff[size_t(d) * (P + 1) + b] = vpos;
        for (int n = 3; n >= 0; --n) {  // 4 rows first
            const uint32_t cnt = vh[b * 4 + n];
            vsec[(size_t(d) * P + b) * 4 + (3 - n)] = cnt;
            vh[b * 4 + n] = vpos;
            vpos += cnt;
        }
        soff[size_t(d) * (P + 1) + b] = spos;
        const uint32_t cnt = sh[b];
        sh[b] = spos;
        spos += cnt;
    }
    if (threadIdx.x == TB - 1) {
        voff[size_t(d) * (P + 1) + P] = vpos;
        soff[size_t(d) * (P + 1) + P] = spos;
    }
}

// Slot record of a group: its two bodies and its pair index with the row count
// in the top three bits. With chunk cursors (vcur / scur, by raw colour) the slot is taken
// in the group's (colour, chunk, row count) part, and the record's last word holds the
// group's rank and the group count of each body (colour_rank, body b's in the upper half).
__global__ void k_colour_scatter(const uint32_t* __restrict__ count, const uint32_t* __restrict__ contact_pairs,
                                 const uint64_t* __restrict__ pairs, const uint32_t* __restrict__ row_count,
                                 const uint32_t* __restrict__ colour, const uint32_t* __restrict__ split_flag,
                                 uint32_t* sub_cursor, uint32_t* split_cursor, uint4* batch_rec, uint4* split_rec,
                                 float4* entries, const uint32_t* __restrict__ remap,
                                 const uint32_t* __restrict__ chunk_of, const float4* __restrict__ iw, uint32_t P,
                                 uint32_t* vcur, uint32_t* scur, const unsigned long long* __restrict__ used) {
    uint32_t K = *count;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < K; k += gridDim.x * blockDim.x) {
        if (colour[k] >= MAX_COLOURS) continue;  // colouring gave up (its status bit is set)
        const uint32_t raw = colour[k];
        uint32_t c = remap[raw];
        uint32_t p = contact_pairs[k];
        uint64_t key = pairs[p];
        uint4 rec = make_uint4(key_lo(key), key_hi(key), p | (row_count[p] << 29), 0u);
        // The colour rides in the manifold's meta bits to seed next step's colouring.
        float* mw = &entries[size_t(p) * ENTRY_F4 + 2].w;
        *mw = __uint_as_float((__float_as_uint(*mw) & ~(0xffu << META_COLOUR_SHIFT)) | ((c + 1u) << META_COLOUR_SHIFT));
        if (vcur) {
            const uint32_t B = group_owner(rec.x, rec.y, iw, chunk_of, P);
            const unsigned long long *ua = used + 4 * size_t(rec.x), *ub = used + 4 * size_t(rec.y);
            const bool da = inv_mass_of(iw, rec.x) > 0.0f, db = inv_mass_of(iw, rec.y) > 0.0f;
            rec.w = (da ? colour_rank(ua, raw) : 0u) | ((db ? colour_rank(ub, raw) : 0u) << 16);
            batch_rec[claim_slot(vcur, (raw * P + B) * 4 + (row_count[p] - 1))] = rec;
            if (split_flag[k]) {
                rec.w = (da ? colour_rank(ua + 2, raw) : 0u) | ((db ? colour_rank(ub + 2, raw) : 0u) << 16);
                split_rec[claim_slot(scur, raw * P + B)] = rec;
            }
        } else {
            batch_rec[claim_slot(sub_cursor, c * 4 + (row_count[p] - 1))] = rec;
            if (split_flag[k]) split_rec[claim_slot(split_cursor, c)] = rec;
        }
    }
}

struct SolveArgs {
    float4* rows;
    const uint4* batch_rec;
    const uint32_t* offset;   // colour batch starts (multiples of 32)
    const uint32_t* end;      // colour batch ends
    const uint4* split_rec;
    const uint32_t* split_offset;
    const uint32_t* split_end;
    const uint32_t* scalars;  // [4] colours [5] split groups [11] largest split batch
    float4* linvel;
    float4* angvel;
    float4* push_lin;
    float4* push_ang;
    const float4* iw;
    float4* vtab;             // velocity contact table (VT_PLANES planes)
    float4* stab;             // split contact table (ST_PLANES planes)
    float4* srec;             // adjoint recording (else null): per (sweep, slot, contact) vn, impulse, clamp bits
    unsigned int* bar;        // [0] velocity-team barrier counter, [1] split-team counter, [8] flow_by_barriers
    uint32_t* status;
    float inv_dt;
    float restitution_threshold;
    uint32_t iterations;
    JointsDev j;              // joint rows, solved after the contacts of each sweep (j.ncol == 0: none)
    float damping;            // joint rows (info.rs damping)
};

// Only dynamic bodies move. Selects, not branches: a branch inside the contact's dependent chain
// costs more than the arithmetic it skips.
__device__ __forceinline__ V3 pick(bool c, V3 x, V3 y) { return V3{c ? x.x : y.x, c ? x.y : y.y, c ? x.z : y.z}; }

__device__ __forceinline__ void apply(V3& la, V3& wa, V3& lb, V3& wb, bool appa, bool appb, float ima, float imb, V3 d,
                                      V3 ca, V3 cb, float j) {
    la = pick(appa, la - d * (j * ima), la);
    wa = pick(appa, wa - ca * j, wa);
    lb = pick(appb, lb + d * (j * imb), lb);
    wb = pick(appb, wb + cb * j, wb);
}

enum Kind { WARM = 0, ITER = 1, SPLIT = 2 };

__device__ __forceinline__ float4 f4(V3 v, float w) { return make_float4(v.x, v.y, v.z, w); }

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// The per-contact terms of warm_start (sequential_impulse.rs:710-717) for contact k of pair p,
// written to the contact's velocity-table entries e (the terms sequential_impulse.rs:352-520
// computes in prepare()); the warm-start impulses are applied by warm_apply.
struct WarmTerms {
    V3 n, t1, t2, ana, anb, a1a, a1b, a2a, a2b;
    float4 r3;
};

__device__ __forceinline__ WarmTerms warm_terms(const SolveArgs& a, uint32_t p, uint32_t k, const M3& iwa,
                                                const M3& iwb, float ima, float imb, float4* e) {
    const float4* r = a.rows + (size_t(p) * 4 + k) * ROW_F4;
    const float4 r0 = r[0], r1 = r[1], r2 = r[2], r3 = r[3], r4 = r[4];
    WarmTerms w;
    w.n = from4(r0);
    const V3 ra = from4(r1), rb = from4(r2);
    tangent_basis_dev(w.n, w.t1, w.t2);
    w.ana = mul(iwa, cross(ra, w.n));
    w.anb = mul(iwb, cross(rb, w.n));
    w.a1a = mul(iwa, cross(ra, w.t1));
    w.a1b = mul(iwb, cross(rb, w.t1));
    w.a2a = mul(iwa, cross(ra, w.t2));
    w.a2b = mul(iwb, cross(rb, w.t2));
    w.r3 = r3;
    e[VT_N * PLANE_STRIDE] = r0;
    e[VT_RA * PLANE_STRIDE] = r1;
    e[VT_RB * PLANE_STRIDE] = r2;
    e[VT_T1 * PLANE_STRIDE] = f4(w.t1, ima);
    e[VT_ANA * PLANE_STRIDE] = f4(w.ana, r4.x);
    e[VT_ANB * PLANE_STRIDE] = f4(w.anb, r4.y);
    e[VT_A1A * PLANE_STRIDE] = f4(w.a1a, r4.z);
    e[VT_A1B * PLANE_STRIDE] = f4(w.a1b, r4.w);
    e[VT_A2A * PLANE_STRIDE] = f4(w.a2a, r3.w);
    e[VT_A2B * PLANE_STRIDE] = f4(w.a2b, imb);
    e[VT_IMP * PLANE_STRIDE] = r3;
    return w;
}

__device__ __forceinline__ void warm_apply(const WarmTerms& w, V3& la, V3& wa, V3& lb, V3& wb, bool appa, bool appb,
                                           float ima, float imb) {
    apply(la, wa, lb, wb, appa, appb, ima, imb, w.n, w.ana, w.anb, w.r3.x);
    apply(la, wa, lb, wb, appa, appb, ima, imb, w.t1, w.a1a, w.a1b, w.r3.y);
    apply(la, wa, lb, wb, appa, appb, ima, imb, w.t2, w.a2a, w.a2b, w.r3.z);
}

// warm_start for group slot t: every contact's terms into the slot's velocity table, its
// warm-start impulses onto the velocities in contact order.
__device__ __forceinline__ void warm_group(const SolveArgs& a, uint32_t t, uint32_t p, uint32_t cnt, uint32_t ia,
                                           uint32_t ib, V3& la, V3& wa, V3& lb, V3& wb, bool& appa, bool& appb) {
    float ima, imb;
    const M3 iwa = load_iw(a.iw, ia, ima);
    const M3 iwb = load_iw(a.iw, ib, imb);
    appa = ima > 0.0f;
    appb = imb > 0.0f;
    for (uint32_t k = 0; k < cnt; ++k) {
        const WarmTerms w = warm_terms(a, p, k, iwa, iwb, ima, imb, a.vtab + tix<VT_PLANES>(0, k, t));
        warm_apply(w, la, wa, lb, wb, appa, appb, ima, imb);
    }
}

// A contact's table entries and the terms of solve_contact that depend on nothing else: the second
// tangent and the velocity couplings (sequential_impulse.rs:352-520).
struct ContactTerms {
    V3 n, ra, rb, t1, t2, ana, anb, a1a, a1b, a2a, a2b, kn, kt1, kt2;
    float friction, bias_a, bias_b, mn, m1, m2, cfm, restitution;

    // Keeps the terms' computation where it stands (the compiler would sink it to their use).
    __device__ __forceinline__ void pin() {
        auto v = [](V3& x) { asm volatile("" : "+f"(x.x), "+f"(x.y), "+f"(x.z)); };
        v(n); v(ra); v(rb); v(t1); v(t2); v(ana); v(anb); v(a1a); v(a1b); v(a2a); v(a2b); v(kn); v(kt1); v(kt2);
        asm volatile("" : "+f"(friction), "+f"(bias_a), "+f"(bias_b), "+f"(mn), "+f"(m1), "+f"(m2), "+f"(cfm),
                     "+f"(restitution));
    }
};

__device__ __forceinline__ ContactTerms contact_terms(const float4* src, uint32_t st, float ima, float imb) {
    const float ims = ima + imb;
    const float4 r0 = src[VT_N * st], r1 = src[VT_RA * st], r2 = src[VT_RB * st], q3 = src[VT_T1 * st],
                 q5 = src[VT_ANA * st], q6 = src[VT_ANB * st], q7 = src[VT_A1A * st], q8 = src[VT_A1B * st],
                 q9 = src[VT_A2A * st], q10 = src[VT_A2B * st];
    ContactTerms c;
    c.n = from4(r0); c.ra = from4(r1); c.rb = from4(r2); c.t1 = from4(q3);
    c.t2 = cross(c.n, c.t1);  // tangent_basis (sequential_impulse.rs:620-629), as warm_terms made it
    c.ana = from4(q5); c.anb = from4(q6); c.a1a = from4(q7); c.a1b = from4(q8); c.a2a = from4(q9); c.a2b = from4(q10);
    // The velocity couplings of sequential_impulse.rs:352-520, in warm_terms's operand order.
    c.kn = c.n * ims + cross(c.anb, c.rb) + cross(c.ana, c.ra);
    c.kt1 = c.t1 * ims + cross(c.a1b, c.rb) + cross(c.a1a, c.ra);
    c.kt2 = c.t2 * ims + cross(c.a2b, c.rb) + cross(c.a2a, c.ra);
    c.friction = r0.w; c.bias_a = r1.w; c.bias_b = r2.w;
    c.mn = q5.w; c.m1 = q6.w; c.m2 = q7.w; c.cfm = q8.w; c.restitution = q9.w;
    return c;
}

// One solve_contact (sequential_impulse.rs:804-930): r3 holds the contact's accumulated impulses,
// and the new ones come back with the values the adjoint's records need.
struct ContactResult {
    float4 r3;
    float vn, u1, u2, maxf;
};

__device__ __forceinline__ ContactResult solve_contact(const SolveArgs& a, const ContactTerms& c, float4 r3, float ima,
                                                       float imb, bool appa, bool appb, V3& la, V3& wa, V3& lb, V3& wb) {
    V3 va = la + cross(wa, c.ra);
    V3 vb = lb + cross(wb, c.rb);
    V3 rel = vb - va;
    const float vn = dot(rel, c.n);
    float bias = vn < -a.restitution_threshold ? -c.restitution * vn : 0.0f;
    bias = c.bias_a != 0.0f ? bias + c.bias_a : bias;
    bias = c.bias_b != 0.0f ? bias + c.bias_b : bias;
    const float lam0 = c.mn * (bias - vn);
    const float lambda = c.cfm != 0.0f ? lam0 - c.cfm * r3.x : lam0;
    float old = r3.x;
    float nimp = fmaxf(old + lambda, 0.0f);
    float jn = nimp - old;
    apply(la, wa, lb, wb, appa, appb, ima, imb, c.n, c.ana, c.anb, jn);
    rel += c.kn * jn;
    float maxf = c.friction * nimp;
    float vt = dot(rel, c.t1);
    float lam = -c.m1 * (vt - 0.0f * a.inv_dt);
    float o1 = r3.y;
    const float u1 = o1 + lam;
    float n1 = fminf(fmaxf(u1, -maxf), maxf);
    float j1 = n1 - o1;
    apply(la, wa, lb, wb, appa, appb, ima, imb, c.t1, c.a1a, c.a1b, j1);
    rel += c.kt1 * j1;
    vt = dot(rel, c.t2);
    lam = -c.m2 * (vt - 0.0f * a.inv_dt);
    float o2 = r3.z;
    const float u2 = o2 + lam;
    float n2 = fminf(fmaxf(u2, -maxf), maxf);
    float j2 = n2 - o2;
    apply(la, wa, lb, wb, appa, appb, ima, imb, c.t2, c.a2a, c.a2b, j2);
    return ContactResult{make_float4(nimp, n1, n2, r3.w), vn, u1, u2, maxf};
}

// Contact k of slot t (pair p): its new impulses go back to the table entry e and, on the last sweep,
// to the pair's row.
__device__ __forceinline__ void store_contact(const SolveArgs& a, const ContactResult& x, float4* e, uint32_t sweep,
                                              uint32_t k, uint32_t t, bool last, uint32_t p) {
    if (a.srec) {  // the forward values the adjoint's frozen linearisation needs
        const uint32_t s1 = x.u1 > x.maxf ? 1u : (x.u1 < -x.maxf ? 2u : 0u);
        const uint32_t s2 = x.u2 > x.maxf ? 1u : (x.u2 < -x.maxf ? 2u : 0u);
        a.srec[sweep_index(sweep, k, t, a.iterations)] =
            make_float4(x.vn, x.r3.x, __uint_as_float(s1 | (s2 << 2)), 0.0f);
    }
    e[VT_IMP * PLANE_STRIDE] = x.r3;
    if (last) a.rows[(size_t(p) * 4 + k) * ROW_F4 + 3] = x.r3;
}

// One solve_contact sweep (sequential_impulse.rs:804-930) over group slot t;
// on the last sweep the impulses also go back to the pair's rows.
__device__ __forceinline__ void iter_group(const SolveArgs& a, uint32_t t, uint32_t p, uint32_t cnt, uint32_t sweep,
                                           bool last, V3& la, V3& wa, V3& lb, V3& wb, bool& appa, bool& appb) {
    const float4* e0 = a.vtab + tix<VT_PLANES>(0, 0, t);
    const float ima = e0[VT_T1 * PLANE_STRIDE].w, imb = e0[VT_A2B * PLANE_STRIDE].w;
    appa = ima > 0.0f;
    appb = imb > 0.0f;
    for (uint32_t k = 0; k < cnt; ++k) {
        float4* e = a.vtab + tix<VT_PLANES>(0, k, t);
        const float4 r3 = e[VT_IMP * PLANE_STRIDE];
        const ContactTerms c = contact_terms(e, PLANE_STRIDE, ima, imb);
        store_contact(a, solve_contact(a, c, r3, ima, imb, appa, appb, la, wa, lb, wb), e, sweep, k, t, last, p);
    }
}

// split_impulse_pass body (sequential_impulse.rs:759-786) for split slot t; the
// first sweep fills the slot's split table, the last writes row 5 back.
__device__ __forceinline__ void split_group(const SolveArgs& a, uint32_t t, uint32_t p, uint32_t cnt, uint32_t ia,
                                            uint32_t ib, bool first, bool last, V3& pla, V3& pwa, V3& plb, V3& pwb,
                                            bool& appa, bool& appb) {
    const float4* e0 = a.stab + tix<ST_PLANES>(0, 0, t);
    float ima, imb;
    M3 iwa, iwb;
    if (first) {
        iwa = load_iw(a.iw, ia, ima);
        iwb = load_iw(a.iw, ib, imb);
    } else {
        ima = e0[3 * PLANE_STRIDE].w;
        imb = e0[4 * PLANE_STRIDE].w;
    }
    appa = ima > 0.0f;
    appb = imb > 0.0f;
    for (uint32_t k = 0; k < cnt; ++k) {
        float4* e = a.stab + tix<ST_PLANES>(0, k, t);
        float4 q0, q1, q2, q3, q4, r5;
        if (first) {
            const float4* r = a.rows + (size_t(p) * 4 + k) * ROW_F4;
            const float4 r0 = r[0], r1 = r[1], r2 = r[2], r4 = r[4];
            r5 = r[5];
            const V3 n = from4(r0), ra = from4(r1), rb = from4(r2);
            const V3 ana = mul(iwa, cross(ra, n)), anb = mul(iwb, cross(rb, n));
            q0 = f4(n, r4.x);
            q1 = f4(ra, r4.w);
            q2 = f4(rb, 0.0f);
            q3 = f4(ana, ima);
            q4 = f4(anb, imb);
            e[0 * PLANE_STRIDE] = q0;
            e[1 * PLANE_STRIDE] = q1;
            e[2 * PLANE_STRIDE] = q2;
            e[3 * PLANE_STRIDE] = q3;
            e[4 * PLANE_STRIDE] = q4;
        } else {
            r5 = e[5 * PLANE_STRIDE];
        }
        if (r5.z == 0.0f) {
            if (first) e[5 * PLANE_STRIDE] = r5;
            continue;
        }
        if (!first) {
            q0 = e[0 * PLANE_STRIDE];
            q1 = e[1 * PLANE_STRIDE];
            q2 = e[2 * PLANE_STRIDE];
            q3 = e[3 * PLANE_STRIDE];
            q4 = e[4 * PLANE_STRIDE];
        }
        const V3 n = from4(q0), ra = from4(q1), rb = from4(q2), ana = from4(q3), anb = from4(q4);
        const float nmass = q0.w, cfm = q1.w;
        V3 pva = pla + cross(pwa, ra);
        V3 pvb = plb + cross(pwb, rb);
        float pvn = dot(pvb - pva, n);
        float delta = cfm != 0.0f ? r5.x - pvn * nmass - cfm * r5.y : r5.x - pvn * nmass;
        float old = r5.y;
        float np = fmaxf(old + delta, 0.0f);
        float j = np - old;
        if (j != 0.0f) {
            if (appa) { pla -= n * (j * ima); pwa -= ana * j; }
            if (appb) { plb += n * (j * imb); pwb += anb * j; }
        }
        const float4 nr5 = make_float4(r5.x, np, r5.z, r5.w);
        e[5 * PLANE_STRIDE] = nr5;
        if (last) a.rows[(size_t(p) * 4 + k) * ROW_F4 + 5] = nr5;
    }
}

// One group: velocities (or push velocities) from L2, the group's solve, the
// dynamic bodies' new velocities back to L2.
template <int KIND>
__device__ __forceinline__ void run_group(const SolveArgs& a, uint32_t t, uint4 rec, uint32_t sweep, uint32_t last) {
    const uint32_t ia = rec.x, ib = rec.y, p = rec.z & 0x1fffffffu, cnt = rec.z >> 29;
    float4* plin = KIND == SPLIT ? a.push_lin : a.linvel;
    float4* pang = KIND == SPLIT ? a.push_ang : a.angvel;
    V3 la = from4(__ldcg(&plin[ia])), wa = from4(__ldcg(&pang[ia]));
    V3 lb = from4(__ldcg(&plin[ib])), wb = from4(__ldcg(&pang[ib]));
    bool appa, appb;  // only dynamic bodies move
    if (KIND == WARM) warm_group(a, t, p, cnt, ia, ib, la, wa, lb, wb, appa, appb);
    else if (KIND == ITER) iter_group(a, t, p, cnt, sweep, sweep == last, la, wa, lb, wb, appa, appb);
    else split_group(a, t, p, cnt, ia, ib, sweep == 0, sweep == last, la, wa, lb, wb, appa, appb);
    if (appa) { __stcg(&plin[ia], to4(la, 0.0f)); __stcg(&pang[ia], to4(wa, 0.0f)); }
    if (appb) { __stcg(&plin[ib], to4(lb, 0.0f)); __stcg(&pang[ib], to4(wb, 0.0f)); }
}

// Bring all of a slot's table entries into L2 (the next phase's group, while the
// team waits at the barrier): the tables of a large pile outgrow L2, so without
// this the first loads after the barrier would wait for DRAM. (Into L1 instead
// measured the same: the barrier's acquire drops L1. Asking for a group's later
// contacts into L1 at the start of its solve measured slower.)
template <bool VELOCITY>
__device__ __forceinline__ void prefetch_slot_l2(const SolveArgs& a, uint32_t t, uint32_t cnt) {
    for (uint32_t k = 0; k < cnt; ++k) {
        if (VELOCITY) {
            const float4* e = a.vtab + tix<VT_PLANES>(0, k, t);
            for (uint32_t pl = 0; pl < VT_PLANES; ++pl) prefetch_l2(e + pl * PLANE_STRIDE);
        } else {
            const float4* e = a.stab + tix<ST_PLANES>(0, k, t);
            for (uint32_t pl = 0; pl < ST_PLANES; ++pl) prefetch_l2(e + pl * PLANE_STRIDE);
        }
    }
}

template <bool VELOCITY>
__device__ __forceinline__ void run_item(const SolveArgs& a, uint32_t sweep, uint32_t last, uint32_t t, uint4 rec) {
    if (!VELOCITY) run_group<SPLIT>(a, t, rec, sweep, last);
    else if (sweep == 0) run_group<WARM>(a, t, rec, sweep, last);
    else run_group<ITER>(a, t, rec, sweep, last);
}

__device__ __forceinline__ void shfl_v3(V3& v, int src) {
    v.x = __shfl_sync(0xffffffffu, v.x, src);
    v.y = __shfl_sync(0xffffffffu, v.y, src);
    v.z = __shfl_sync(0xffffffffu, v.z, src);
}

// Phases 0 .. nphases-1 of a team: phase q is colour q % ncol of sweep q / ncol.
// The team's threads deal the batch slots of each phase among themselves and
// meet at the team barrier between phases; each thread reads its next slot
// record while it solves the current one.
//
// A colour with at most one block's worth of groups (the tail colours of a
// pile, or every colour of a small scene) is solved by the team's first block
// alone, one group per thread. Between two such colours the block syncs
// locally instead of the team meeting at a barrier: the other blocks go on to
// the next barrier and wait there.
template <bool VELOCITY>
__device__ __forceinline__ void run_phases(const SolveArgs& a, const uint4* __restrict__ recs, const uint32_t* soff,
                                           const uint32_t* send, uint32_t ncol, uint32_t nphases, uint32_t last, uint32_t tid,
                                           uint32_t stride, unsigned int* ctr, uint32_t team_blocks, uint32_t team_block,
                                           uint32_t& nbar, uint32_t sweep0 = 0) {
    if (ncol == 0 || nphases == 0) return;
    auto small = [&](uint32_t c) { return send[c] - soff[c] <= blockDim.x; };
    auto first_slot = [&](uint32_t c) -> uint32_t {
        if (!small(c)) return soff[c] + tid;
        return team_block == 0 ? soff[c] + threadIdx.x : send[c];
    };
    auto first_rec = [&](uint32_t c) -> uint4 {
        const uint32_t t = first_slot(c);
        return t < send[c] ? __ldg(&recs[t]) : make_uint4(0u, 0u, 0u, 0u);
    };
    uint4 rec = first_rec(0);  // rec.z == 0 (no rows): no slot for this thread
    for (uint32_t q = 0; q < nphases; ++q) {
        const uint32_t c = q % ncol, sweep = sweep0 + q / ncol;
        const uint4 next = q + 1 < nphases ? first_rec((q + 1) % ncol) : make_uint4(0u, 0u, 0u, 0u);
        if (rec.z) {
            const uint32_t t0 = first_slot(c);
            run_item<VELOCITY>(a, sweep, last, t0, rec);
            if (!small(c))
                for (uint32_t t = t0 + stride; t < send[c]; t += stride) run_item<VELOCITY>(a, sweep, last, t, __ldg(&recs[t]));
        }
        rec = next;
        if (q + 1 < nphases) {
            const uint32_t cn = (q + 1) % ncol;
            if (small(c) && small(cn)) {
                __syncthreads();  // global writes of the block are visible to the block after it
                continue;
            }
            // The next phase's table entries (written in sweep 0) head for L2 while the team waits.
            if (rec.z && (q + 1) >= ncol) prefetch_slot_l2<VELOCITY>(a, first_slot(cn), rec.z >> 29);
            team_barrier(ctr, ++nbar * team_blocks, a.status);
        }
    }
}

// One joint colour: slots [first, end) with the given stride.
__device__ __forceinline__ void joint_phase(JointsDev j, float4* linvel, float4* angvel, const float4* iw, float damping,
                                         uint32_t first, uint32_t end, uint32_t stride) {
    for (uint32_t t = first; t < end; t += stride) solve_joint_slot(j, t, linvel, angvel, iw, damping);
}

// The velocity team's sweeps in a world with joints: sweep by sweep, the contact phases,
// then (velocity sweeps only) one phase per joint colour (sequential_impulse.rs:720-735).
// Between two phases that block 0 runs alone (at most one block's worth of slots) the
// block syncs locally; otherwise the team meets at its barrier. Only the k_solve built
// for worlds with joints contains it.
__device__ __forceinline__ void velocity_sweeps_with_joints(const SolveArgs& a, const uint32_t* s_off, const uint32_t* s_end,
                                                         const uint32_t* s_joff, uint32_t ncol, uint32_t njcol,
                                                         uint32_t iters, uint32_t tid, uint32_t stride,
                                                         uint32_t team_blocks, uint32_t team_block, uint32_t& nbar) {
    auto csmall = [&](uint32_t c) { return s_end[c] - s_off[c] <= blockDim.x; };
    auto jsmall = [&](uint32_t c) { return s_joff[c + 1] - s_joff[c] <= blockDim.x; };
    auto sync = [&](bool local) {
        if (local) __syncthreads();
        else team_barrier(a.bar, ++nbar * team_blocks, a.status);
    };
    for (uint32_t sw = 0; sw <= iters; ++sw) {
        run_phases<true>(a, a.batch_rec, s_off, s_end, ncol, ncol, iters, tid, stride, a.bar, team_blocks, team_block,
                         nbar, sw);
        bool prev_small = ncol ? csmall(ncol - 1) : true;
        if (sw >= 1) {
            for (uint32_t jc = 0; jc < njcol; ++jc) {
                const bool small = jsmall(jc);
                sync(prev_small && small);
                const uint32_t lo = s_joff[jc], hi = s_joff[jc + 1];
                if (small) {
                    if (team_block == 0 && lo + threadIdx.x < hi)
                        joint_phase(a.j, a.linvel, a.angvel, a.iw, a.damping, lo + threadIdx.x, hi, blockDim.x);
                } else {
                    joint_phase(a.j, a.linvel, a.angvel, a.iw, a.damping, lo + tid, hi, stride);
                }
                prev_small = small;
            }
        }
        if (sw < iters) sync(prev_small && (ncol ? csmall(0) : true));
    }
}

// solve() (sequential_impulse.rs:692-705): warm start and velocity sweeps on
// the velocity team; the split sweeps on the split team, which has enough
// blocks for the largest split batch and at most a quarter of the grid (none
// on a grid too small to split, where the velocity team runs them last).
// JOINTS: the build for worlds with joints (the contact-only build carries none of their code).
template <bool JOINTS>
__global__ void __launch_bounds__(256, 2) k_solve(SolveArgs a) {
    const uint32_t ncol = a.scalars[4];
    const uint32_t nsplit = a.scalars[5];
    const uint32_t iters = a.iterations;
    const uint32_t G = gridDim.x;
    uint32_t split_blocks = 0;
    if (nsplit && iters && G >= 4) {
        uint32_t need = (a.scalars[11] + blockDim.x - 1) / blockDim.x;
        split_blocks = min(max(need, 1u), G / 4);
    }
    const bool split_team = blockIdx.x >= G - split_blocks;
    const uint32_t team_blocks = split_team ? split_blocks : G - split_blocks;
    const uint32_t team_block = split_team ? blockIdx.x - (G - split_blocks) : blockIdx.x;
    const uint32_t tid = team_block * blockDim.x + threadIdx.x;
    const uint32_t stride = team_blocks * blockDim.x;
    __shared__ uint32_t s_off[MAX_COLOURS], s_end[MAX_COLOURS], s_split_off[MAX_COLOURS], s_split_end[MAX_COLOURS];
    for (uint32_t c = threadIdx.x; c < ncol; c += blockDim.x) {
        s_off[c] = a.offset[c];
        s_end[c] = a.end[c];
        s_split_off[c] = a.split_offset[c];
        s_split_end[c] = a.split_end[c];
    }
    const uint32_t njcol = JOINTS ? a.j.ncol : 0u;
    __shared__ uint32_t s_joff[JOINTS ? MAX_COLOURS + 1 : 1];
    if (JOINTS)
        for (uint32_t c = threadIdx.x; c <= njcol && njcol; c += blockDim.x) s_joff[c] = a.j.coff[c];
    __syncthreads();  // the batch ranges above are read by every thread of the block
    uint32_t nbar = 0;
    if (split_team) {
        run_phases<false>(a, a.split_rec, s_split_off, s_split_end, ncol, iters * ncol, iters - 1u, tid, stride, a.bar + 1,
                          team_blocks, team_block, nbar);
        return;
    }
    if (!JOINTS || njcol == 0) {
        run_phases<true>(a, a.batch_rec, s_off, s_end, ncol, (iters + 1) * ncol, iters, tid, stride, a.bar, team_blocks,
                         team_block, nbar);
    } else {
        velocity_sweeps_with_joints(a, s_off, s_end, s_joff, ncol, njcol, iters, tid, stride, team_blocks, team_block, nbar);
    }
    if (nsplit && iters && split_blocks == 0) {
        team_barrier(a.bar, ++nbar * team_blocks, a.status);
        run_phases<false>(a, a.split_rec, s_split_off, s_split_end, ncol, iters * ncol, iters - 1u, tid, stride, a.bar, team_blocks,
                          team_block, nbar);
    }
}

// ---------------------------------------------------------------- chunked PGS
// k_flow_table writes every contact's velocity table entries; k_solve_flow then runs the warm
// start, the velocity sweeps and the split sweeps in one cooperative launch without any barrier
// between warps.
struct FlowArgs {
    uint32_t P;             // chunks
    uint32_t bpc;           // blocks a chunk: the launch has P bpc blocks
    const uint32_t* voff;   // [d (P + 1) + b]: chunk b's part of colour batch d
    const uint32_t* soff;   // the same for the split batches
    const uint32_t* vsec;   // [(d P + b) 4 + i]: groups of 4 - i rows in chunk b's part of batch d
    float4* vel;            // 2 per body: linear velocity | version, angular velocity | version
    float4* push;           // 2 per body: the push velocities
};

constexpr uint32_t FLOW_PLANES = VT_PLANES - 1;  // every plane but the impulses is staged in shared memory
constexpr size_t flow_smem(uint32_t tb) { return size_t(2) * FLOW_PLANES * tb * sizeof(float4); }

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned int d = static_cast<unsigned int>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem) : "memory");
}

// A versioned velocity word: one 128-bit access carries the vector and its version, so a reader
// that finds the version it waits for has the vector that goes with it (no fence, no second
// round trip).
__device__ __forceinline__ float4 flow_load(const float4* p) {
    unsigned long long lo, hi;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(lo), "=l"(hi)
                 : "l"(p));
    return make_float4(__uint_as_float(uint32_t(lo)), __uint_as_float(uint32_t(lo >> 32)), __uint_as_float(uint32_t(hi)),
                       __uint_as_float(uint32_t(hi >> 32)));
}

__device__ __forceinline__ void flow_store(float4* p, V3 v, uint32_t version) {
    const unsigned long long lo = (uint64_t(__float_as_uint(v.y)) << 32) | __float_as_uint(v.x);
    const unsigned long long hi = (uint64_t(version) << 32) | __float_as_uint(v.z);
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p), "l"(lo),
                 "l"(hi)
                 : "memory");
}

// The two velocity vectors of one body of a group and their versions. deg: the body's groups a
// sweep (0: not dynamic; its velocities are constant), total: its versions over the whole
// solve. Version 0 is the body's own array (lin, ang), and the last version goes back there.
struct FlowBody {
    uint32_t i, want, total;

    __device__ __forceinline__ void init(uint32_t body, uint32_t rank_deg, uint32_t sweep, uint32_t sweeps) {
        const uint32_t deg = (rank_deg >> 8) & 0xffu;
        i = body;
        want = sweep * deg + (rank_deg & 0xffu);
        total = deg * sweeps;
    }
    // Reads the vectors; false: not yet at the version wanted.
    __device__ __forceinline__ bool read(const float4* lin, const float4* ang, const float4* ver, V3& l, V3& w) const {
        const bool own = want == 0u;
        const float4* v = ver + 2 * size_t(i);
        const float4 x = flow_load(own ? lin + i : v), y = flow_load(own ? ang + i : v + 1);
        l = from4(x);
        w = from4(y);
        return own || (__float_as_uint(x.w) == want && __float_as_uint(y.w) == want);
    }
    __device__ __forceinline__ void write(float4* lin, float4* ang, float4* ver, V3 l, V3 w) const {
        if (total == 0u) return;
        const bool end = want + 1u == total;
        float4* v = ver + 2 * size_t(i);
        flow_store(end ? lin + i : v, l, end ? 0u : want + 1u);
        flow_store(end ? ang + i : v + 1, w, end ? 0u : want + 1u);
    }
};

// Waits until every lane of the warp that takes part has both its bodies' versions. The wait is
// bounded like team_barrier's; false: it gave up (the status word says so).
__device__ __forceinline__ bool flow_wait(bool take, const FlowBody& A, const FlowBody& B, const float4* lin,
                                          const float4* ang, const float4* ver, V3& la, V3& wa, V3& lb, V3& wb,
                                          uint32_t* status) {
    bool ra = !take, rb = !take;
    uint32_t spins = 0;
    unsigned long long t0 = 0;
    for (;;) {
        if (!ra) ra = A.read(lin, ang, ver, la, wa);
        if (!rb) rb = B.read(lin, ang, ver, lb, wb);
        if (__all_sync(0xffffffffu, ra && rb)) return true;
        if ((++spins & 63u) == 0u) {
            const unsigned long long now = globaltimer_ns();
            if (t0 == 0) t0 = now;
            const bool stop = (*(volatile uint32_t*)status & ST_BARRIER_TIMEOUT) || now - t0 > BARRIER_TIMEOUT_NS ||
                              spins > BARRIER_SPIN_LIMIT;
            if (__any_sync(0xffffffffu, stop)) {
                if ((threadIdx.x & 31u) == 0u) atomicOr(status, ST_BARRIER_TIMEOUT);
                return false;
            }
        }
    }
}

// Every contact's table entries from its row and its bodies' inverse inertia: one warp per 32 slots
// and contact index, so the table's planes are written in whole lines.
__global__ void __launch_bounds__(256) k_flow_table(SolveArgs a) {
    __shared__ uint32_t s_off[MAX_COLOURS], s_end[MAX_COLOURS];
    const uint32_t ncol = a.scalars[4];
    for (uint32_t c = threadIdx.x; c < ncol; c += blockDim.x) {
        s_off[c] = a.offset[c];
        s_end[c] = a.end[c];
    }
    __syncthreads();
    if (ncol == 0) return;
    const uint32_t lane = threadIdx.x & 31u, nblk = (s_end[ncol - 1] + 31u) / 32u * 4u;
    for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nblk; w += (gridDim.x * blockDim.x) >> 5) {
        const uint32_t t = (w >> 2) * 32u + lane, k = w & 3u;
        uint32_t lo = 0, hi = ncol - 1;  // the batch this block of 32 slots belongs to
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1) >> 1;
            if (s_off[mid] <= t) lo = mid;
            else hi = mid - 1;
        }
        if (t >= s_end[lo]) continue;  // padding at the batch's end
        const uint4 rec = __ldg(&a.batch_rec[t]);
        if (k >= rec.z >> 29) continue;
        float ima, imb;
        const M3 iwa = load_iw(a.iw, rec.x, ima);
        const M3 iwb = load_iw(a.iw, rec.y, imb);
        warm_terms(a, rec.z & 0x1fffffffu, k, iwa, iwb, ima, imb, a.vtab + tix<VT_PLANES>(0, k, t));
    }
}

// The same solve with a grid barrier after every phase, for a colouring that overflowed: its surplus groups
// share the last colour with others at one body, so a colour is no longer one version of a body and a wait
// for one may never end. Every group is solved; only the order (and, as they run side by side, the velocity
// updates) of those at that one body is left open. A slot's table entries stay with one thread (the deal
// depends on the colour alone). Some 3 us a phase: 128 colours and 20 sweeps take 8 ms, under an error status.
// (The caller's parameters are __grid_constant__: a copy of them to pass on here cost every solve 1 to 2 %.)
template <uint32_t TB>
__device__ __noinline__ void flow_by_barriers(const SolveArgs& a, const FlowArgs& f) {
    const uint32_t ncol = a.scalars[4], iters = a.iterations;
    const uint32_t first = blockIdx.x * TB + threadIdx.x, stride = gridDim.x * TB;
    uint32_t nbar = 0;
    for (uint32_t sw = 0; sw <= iters; ++sw)
        for (uint32_t c = 0; c < ncol; ++c) {
            for (uint32_t t = a.offset[c] + first; t < a.end[c]; t += stride)
                run_item<true>(a, sw, iters, t, __ldg(&a.batch_rec[t]));
            const uint32_t* soff = f.soff + size_t(c) * (f.P + 1);
            if (sw)
                for (uint32_t t = soff[0] + first; t < soff[f.P]; t += stride)
                    run_item<false>(a, sw - 1u, iters - 1u, t, __ldg(&a.split_rec[t]));
            team_barrier(a.bar + 8, ++nbar * gridDim.x, a.status);
        }
}

// The items of a warp: 32 lanes of a phase (sweep, colour) of its chunk. A phase's lanes are its
// velocity lanes (a group of 4 or 3 rows takes 4 lanes, of 2 rows 2, of 1 row one), padded to a
// whole warp, then one lane per split group; split sweep s runs in the phases of velocity sweep
// s + 1 (it touches only the push velocities). Each colour starts its deal at another warp, so that
// the small colours do not all fall to the first.
struct FlowItem {
    uint32_t sweep, c, base;
};

// solve() (sequential_impulse.rs:692-705) for worlds without joints, one chunk per block. A warp
// walks its items in (sweep, colour) order and waits, item by item, only for the velocities the
// item's own bodies have in that order; nothing else holds it up. What a body's update waits
// for always lies in an earlier phase, every block is resident (cooperative launch) and each warp
// takes its items in phase order, so the wait always ends. Each body sees its groups in (sweep,
// colour) order, as under a barrier after every phase: the result is the sequential solve in
// (colour, pair) order.
//
// Lane k of a group's segment holds contact k: the table entries come by cp.async one item ahead
// (two stages of shared memory, private to the thread), the terms that need no velocity are computed
// before the wait, and the contacts are solved in order k = 0, 1, ..., the velocities handed from lane
// to lane by shuffles; the last contact's lane stores the new versions.
//
// What bounds it: the chain of dependent contacts. A phase costs a version's way through L2 (about
// 1,200 cycles from the store to the reader's poll) plus the item itself (about 390 cycles a contact
// for a lone warp, 700 when three warps share a scheduler); a warp that holds several items of a
// large colour does them one after the other. Measured against the block-level neighbour waits it
// replaces (release store, counter poll, then the velocity loads), warm start included, one step's
// launches: 131,072-body pile with 15 colours and 20 iterations 2,489 -> 1,575 us, 5,681-body pile 934
// -> 380 us, 16,384 mixed bodies with 15 colours and 10 iterations 604 -> 245 us. 384 threads: at 512 the
// 128 registers spill (1,628 us on the pile, 528 on the small one), at 320 too few groups are in
// flight (1,785 us). One group a lane instead of one contact a lane halves the instructions but holds
// a warp up for the slowest of 32 groups (1,887 us at 160 threads, the most its staging allows).
template <uint32_t TB>
__global__ void __launch_bounds__(TB, 1) k_solve_flow(const __grid_constant__ SolveArgs a,
                                                      const __grid_constant__ FlowArgs f) {
    extern __shared__ float4 s_pl[];  // [stage][plane][thread]
    // Per colour: the chunk's part of the batches, and the ends of its velocity lanes on 4 and on 2
    // lanes a group, of all of them, and the phase's lanes with the split groups.
    __shared__ uint32_t s_v0[MAX_COLOURS], s_s0[MAX_COLOURS];
    __shared__ uint4 s_end[MAX_COLOURS];
    const uint32_t ncol = a.scalars[4];
    const uint32_t iters = a.iterations;
    if (*a.status & ST_COLOUR_OVERFLOW) {  // set by the colouring, before this launch: the same for all blocks
        flow_by_barriers<TB>(a, f);
        return;
    }
    const uint32_t b = blockIdx.x / f.bpc, lane = threadIdx.x & 31u;  // the chunk
    const uint32_t nwarps = f.bpc * (TB / 32u), warp = (blockIdx.x % f.bpc) * (TB / 32u) + (threadIdx.x >> 5);
    for (uint32_t c = threadIdx.x; c < ncol; c += TB) {
        const uint32_t v0 = f.voff[size_t(c) * (f.P + 1) + b], nv = f.voff[size_t(c) * (f.P + 1) + b + 1] - v0;
        const uint32_t s0 = f.soff[size_t(c) * (f.P + 1) + b], ns = f.soff[size_t(c) * (f.P + 1) + b + 1] - s0;
        const uint32_t* sec = f.vsec + (size_t(c) * f.P + b) * 4;
        const uint32_t n4 = sec[0] + sec[1], n2 = sec[2];
        const uint32_t L4 = 4u * n4, L2 = L4 + 2u * n2, L1 = L2 + (nv - n4 - n2);
        s_v0[c] = v0;
        s_s0[c] = s0;
        s_end[c] = make_uint4(L4, L2, L1, ((L1 + 31u) & ~31u) + ns);
    }
    __syncthreads();
    auto start = [&](uint32_t c) { return ((warp + 5u * c) % nwarps) * 32u; };
    // The colours with an item for this warp, a bit each (from sweep 1 on; in sweep 0 some may
    // hold split groups only).
    unsigned long long mine0 = 0, mine1 = 0;
    for (uint32_t c0 = 0; c0 < ncol; c0 += 32u) {
        const uint32_t c = c0 + lane;
        const unsigned long long w = __ballot_sync(0xffffffffu, c < ncol && start(c) < s_end[c].w);
        if (c0 < 64u) mine0 |= w << c0;
        else mine1 |= w << (c0 - 64u);
    }
    if ((mine0 | mine1) == 0ull) return;
    // The next item at or after `it`; false: none.
    auto settle = [&](FlowItem& it) {
        while (it.base >= (it.sweep ? s_end[it.c].w : (s_end[it.c].z + 31u) & ~31u)) {
            const uint32_t c = it.c + 1u;
            unsigned long long lo = c < 64u ? mine0 & (~0ull << c) : 0ull;
            unsigned long long hi = c < 64u ? mine1 : (c < 128u ? mine1 & (~0ull << (c - 64u)) : 0ull);
            if ((lo | hi) == 0ull) {
                if (++it.sweep > iters) return false;
                lo = mine0;
                hi = mine1;
            }
            it.c = lo ? uint32_t(__ffsll((long long)lo) - 1) : 63u + uint32_t(__ffsll((long long)hi));
            it.base = start(it.c);
        }
        return true;
    };
    // What an item's lane needs: its slot, contact, record and the contact's impulses (which this
    // lane wrote a sweep before); its other table entries head for a stage.
    struct Lane {
        uint4 rec;
        uint32_t t, k;
        float4 r3;
    };
    auto fetch = [&](const FlowItem& it, uint32_t stage) {
        Lane L;
        L.rec = make_uint4(0u, 0u, 0u, 0u);
        L.t = 0;
        L.k = 0;
        L.r3 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const uint4 end = s_end[it.c];
        const uint32_t LV = (end.z + 31u) & ~31u, i = it.base + lane;
        if (it.base < LV) {
            if (i < end.z) {
                uint32_t g = end.x / 4u + (end.y - end.x) / 2u + (i - end.y);
                if (i < end.x) { g = i >> 2; L.k = i & 3u; }
                else if (i < end.y) { g = (end.x / 4u) + ((i - end.x) >> 1); L.k = i & 1u; }
                L.t = s_v0[it.c] + g;
                L.rec = __ldg(&a.batch_rec[L.t]);
                // (The fourth lane of a 3-row group copies entries nothing reads: no wait for the record.)
                const float4* e = a.vtab + tix<VT_PLANES>(0, L.k, L.t);
                L.r3 = e[VT_IMP * PLANE_STRIDE];
#pragma unroll
                for (uint32_t pl = 0; pl < FLOW_PLANES; ++pl)
                    cp_async16(&s_pl[(stage * FLOW_PLANES + pl) * TB + threadIdx.x], e + pl * PLANE_STRIDE);
            }
        } else if (i < end.w) {
            L.t = s_s0[it.c] + (i - LV);
            L.rec = __ldg(&a.split_rec[L.t]);
            if (it.sweep >= 2) prefetch_slot_l2<false>(a, L.t, L.rec.z >> 29);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        return L;
    };
    FlowItem cur{0u, 0u, start(0)};
    if (!settle(cur)) return;
    Lane L = fetch(cur, 0);
    uint32_t stage = 0;
    for (;;) {
        FlowItem nxt = cur;
        nxt.base += nwarps * 32u;
        const bool more = settle(nxt);
        const bool same = nxt.c == cur.c && nxt.base == cur.base;  // the warp's only item of a sweep
        Lane N = L;
        if (more && !same) {
            N = fetch(nxt, stage ^ 1u);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        const uint32_t cnt = L.rec.z >> 29, p = L.rec.z & 0x1fffffffu, ia = L.rec.x, ib = L.rec.y;
        V3 la{0.0f, 0.0f, 0.0f}, wa = la, lb = la, wb = la;
        FlowBody A, B;
        if (cur.base < ((s_end[cur.c].z + 31u) & ~31u)) {
            const uint32_t k = L.k, t = L.t;
            const bool mine = k < cnt;
            const uint32_t jmax = __reduce_max_sync(0xffffffffu, cnt);
            const uint32_t seg0 = lane - k;
            A.init(ia, L.rec.w & 0xffffu, cur.sweep, iters + 1u);
            B.init(ib, L.rec.w >> 16, cur.sweep, iters + 1u);
            const float4* sp = s_pl + stage * (FLOW_PLANES * TB) + threadIdx.x;
            ContactTerms C{};
            float ima = 0.0f, imb = 0.0f;
            if (mine) {
                ima = sp[VT_T1 * TB].w;
                imb = sp[VT_A2B * TB].w;
                C = contact_terms(sp, TB, ima, imb);
            }
            C.pin();  // before the wait, not after it
            const bool appa = ima > 0.0f, appb = imb > 0.0f;
            ContactResult X{};
            if (!flow_wait(mine && k == 0u, A, B, a.linvel, a.angvel, f.vel, la, wa, lb, wb, a.status)) break;
            for (uint32_t j = 0; j < jmax; ++j) {
                if (mine && k == j) {
                    if (cur.sweep == 0u) {
                        apply(la, wa, lb, wb, appa, appb, ima, imb, C.n, C.ana, C.anb, L.r3.x);
                        apply(la, wa, lb, wb, appa, appb, ima, imb, C.t1, C.a1a, C.a1b, L.r3.y);
                        apply(la, wa, lb, wb, appa, appb, ima, imb, C.t2, C.a2a, C.a2b, L.r3.z);
                    } else {
                        X = solve_contact(a, C, L.r3, ima, imb, appa, appb, la, wa, lb, wb);
                    }
                    if (k + 1u == cnt) {
                        A.write(a.linvel, a.angvel, f.vel, la, wa);
                        B.write(a.linvel, a.angvel, f.vel, lb, wb);
                    }
                }
                if (j + 1u < jmax) {
                    const int src = int(j < cnt ? seg0 + j : lane);
                    shfl_v3(la, src);
                    shfl_v3(wa, src);
                    shfl_v3(lb, src);
                    shfl_v3(wb, src);
                }
            }
            if (mine && cur.sweep) {
                store_contact(a, X, a.vtab + tix<VT_PLANES>(0, k, t), cur.sweep, k, t, cur.sweep == iters, p);
                if (same) N.r3 = X.r3;
            }
        } else {
            const uint32_t sw = cur.sweep - 1u;
            A.init(ia, L.rec.w & 0xffffu, sw, iters);
            B.init(ib, L.rec.w >> 16, sw, iters);
            if (!flow_wait(cnt != 0u, A, B, a.push_lin, a.push_ang, f.push, la, wa, lb, wb, a.status)) break;
            if (cnt) {
                bool appa, appb;
                split_group(a, L.t, p, cnt, ia, ib, sw == 0u, sw + 1u == iters, la, wa, lb, wb, appa, appb);
                A.write(a.push_lin, a.push_ang, f.push, la, wa);
                B.write(a.push_lin, a.push_ang, f.push, lb, wb);
            }
        }
        if (!more) break;
        cur = nxt;
        L = N;
        if (!same) stage ^= 1u;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// ---------------------------------------------------------------- per-world PGS (batched worlds)
// Every world of a batch is solved on its own by one CTA or one warp: its row groups are
// coloured in shared memory (Jones-Plassmann with the world's own priorities, colours from
// one 64-bit mask per body), sorted into colour batches, and solved phase by phase with only
// a block (or warp) sync between phases; its bodies' velocities and push velocities stay in
// shared memory for the whole solve. No barrier spans worlds. Within a world the order is the
// same (colour, pair) Gauss-Seidel order the global solver uses, so each world equals the
// reference's sequential solve over its rows in that order. The split sweeps touch only push
// velocities, so split sweep s runs in the phases of velocity sweep s + 1.
struct WorldSolveArgs {
    SolveArgs a;                       // rows, tables, adjoint sweep records, iw, constants
    const uint32_t* contact_pairs;     // pair ids with rows, ascending (so grouped by world)
    const uint32_t* ngroups;           // device count of contact_pairs
    const uint64_t* pairs;
    const uint32_t* row_count;
    const uint32_t* world_off;
    uint32_t* colour;                  // out: world-local colour per contact pair
    uint4* recs;                       // out: slot records, world by world, colour by colour
    uint32_t* wcol;                    // out: per world g0, ncol, offsets[ncol + 1]
    uint32_t* colour_count;            // out: groups per colour summed over worlds (stats)
    uint32_t* split_count;
    uint32_t* scalars;                 // out: [3] rows [4] colours (max) [5] split groups [10] split rows
    float4* linvel;
    float4* angvel;
    float4* push_lin;
    float4* push_ang;
    uint32_t* status;
    WorldPlanDev plan;
    float4* entries;                   // the pairs' new manifolds: their meta bits carry the colour
    uint32_t seed;                     // nonzero: start from the colours the manifolds carry
};

struct WorldCtx {  // per world being solved by a CTA or a warp
    uint32_t g0, g1, ncol, left, rows, split_groups, split_rows;
    uint32_t hist[WS_MAX_COLOURS], off[WS_MAX_COLOURS + 1], cur[WS_MAX_COLOURS], split_hist[WS_MAX_COLOURS];
};

template <bool WARP>
__device__ __forceinline__ void ws_sync() {
    if (WARP) __syncwarp();
    else __syncthreads();
}

__device__ __forceinline__ uint32_t lower_bound_lo(const uint64_t* __restrict__ pairs, const uint32_t* __restrict__ cp,
                                                   uint32_t n, uint32_t body) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (key_lo(pairs[cp[mid]]) < body) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// One group of a world: velocities from the world's shared-memory arrays (body i at i - b0).
template <int KIND>
__device__ __forceinline__ void run_group_shared(const SolveArgs& a, uint32_t t, uint4 rec, uint32_t sweep,
                                                 uint32_t last, float4* lin, float4* ang, uint32_t b0) {
    const uint32_t ia = rec.x, ib = rec.y, p = rec.z & 0x1fffffffu, cnt = rec.z >> 29;
    const uint32_t la_i = ia - b0, lb_i = ib - b0;
    V3 la = from4(lin[la_i]), wa = from4(ang[la_i]);
    V3 lb = from4(lin[lb_i]), wb = from4(ang[lb_i]);
    bool appa, appb;
    if (KIND == WARM) warm_group(a, t, p, cnt, ia, ib, la, wa, lb, wb, appa, appb);
    else if (KIND == ITER) iter_group(a, t, p, cnt, sweep, sweep == last, la, wa, lb, wb, appa, appb);
    else split_group(a, t, p, cnt, ia, ib, sweep == 0, sweep == last, la, wa, lb, wb, appa, appb);
    if (appa) { lin[la_i] = to4(la, 0.0f); ang[la_i] = to4(wa, 0.0f); }
    if (appb) { lin[lb_i] = to4(lb, 0.0f); ang[lb_i] = to4(wb, 0.0f); }
}

// The range of world w's groups and their colours (A.colour), by `nt` threads (lane = 0 .. nt - 1):
// `mask` its 4 * nb words of shared memory, `C` its context. Every thread of the CTA (block mode) or
// of the warp (warp mode) calls it, and every sync is reached by all of them.
template <bool WARP>
__device__ __forceinline__ void colour_world(const WorldSolveArgs& A, uint32_t b0, uint32_t nb, uint32_t lane, uint32_t nt,
                                             unsigned long long* mask, WorldCtx& C) {
    const SolveArgs& a = A.a;
    unsigned long long* best0 = mask + nb;
    unsigned long long* best1 = best0 + nb;
    unsigned long long* dup = best1 + nb;  // seeded colours claimed twice at a body
    for (uint32_t i = lane; i < nb; i += nt) {
        mask[i] = 0ull;
        best0[i] = 0ull;
        best1[i] = 0ull;
        dup[i] = 0ull;
    }
    if (lane == 0) {
        const uint32_t K = *A.ngroups;
        C.g0 = lower_bound_lo(A.pairs, A.contact_pairs, K, b0);
        C.g1 = lower_bound_lo(A.pairs, A.contact_pairs, K, b0 + nb);
        C.left = C.g1 - C.g0;
        C.ncol = 0;
        C.rows = C.split_groups = C.split_rows = 0;
    }
    for (uint32_t c = lane; c < WS_MAX_COLOURS; c += nt) {
        C.hist[c] = 0;
        C.split_hist[c] = 0;
    }
    ws_sync<WARP>();
    const uint32_t g0 = C.g0, g1 = C.g1;
    auto dyn = [&](uint32_t i) { return inv_mass_of(a.iw, i) > 0.0f; };
    // Jones-Plassmann rounds: an uncoloured group wins when its priority is the largest
    //    among the uncoloured groups at each of its dynamic bodies; a winner takes the lowest
    //    colour free at both bodies (winners of one round share no dynamic body).
    auto seed_of = [&](uint32_t g) -> uint32_t {  // last step's colour + 1 (0: none)
        const uint32_t cs =
            (__float_as_uint(A.entries[size_t(A.contact_pairs[g]) * ENTRY_F4 + 2].w) >> META_COLOUR_SHIFT) & 0xffu;
        return cs <= WS_MAX_COLOURS ? cs : 0u;
    };
    if (A.seed) {
        //    Seeds: each group claims last step's colour at its dynamic bodies; a group keeps it
        //    when no other group claimed the same colour at either body. The others are coloured
        //    by the rounds below, first fit around every claimed colour.
        for (uint32_t g = g0 + lane; g < g1; g += nt) {
            const uint32_t cs = seed_of(g);
            if (cs == 0u) continue;
            const unsigned long long bit = 1ull << (cs - 1u);
            const uint64_t key = A.pairs[A.contact_pairs[g]];
            const uint32_t ia = key_lo(key), ib = key_hi(key);
            if (dyn(ia) && (atomicOr(&mask[ia - b0], bit) & bit)) atomicOr(&dup[ia - b0], bit);
            if (dyn(ib) && (atomicOr(&mask[ib - b0], bit) & bit)) atomicOr(&dup[ib - b0], bit);
        }
        ws_sync<WARP>();
        uint32_t kept = 0;
        for (uint32_t g = g0 + lane; g < g1; g += nt) {
            const uint32_t cs = seed_of(g);
            bool keep = false;
            if (cs != 0u) {
                const unsigned long long bit = 1ull << (cs - 1u);
                const uint64_t key = A.pairs[A.contact_pairs[g]];
                const uint32_t ia = key_lo(key), ib = key_hi(key);
                keep = !(dyn(ia) && (dup[ia - b0] & bit)) && !(dyn(ib) && (dup[ib - b0] & bit));
            }
            A.colour[g] = keep ? cs - 1u : NO_COLOUR;
            kept += keep ? 1u : 0u;
        }
        if (kept) atomicSub(&C.left, kept);
    } else {
        for (uint32_t g = g0 + lane; g < g1; g += nt) A.colour[g] = NO_COLOUR;
    }
    ws_sync<WARP>();
    for (uint32_t r = 0; C.left != 0; ++r) {
        if (r >= MAX_ROUNDS) {
            if (lane == 0) atomicOr(A.status, ST_COLOUR_ROUNDS);
            break;
        }
        unsigned long long* best = (r & 1) ? best1 : best0;
        unsigned long long* other = (r & 1) ? best0 : best1;
        for (uint32_t g = g0 + lane; g < g1; g += nt) {
            if (A.colour[g] != NO_COLOUR) continue;
            const uint64_t key = A.pairs[A.contact_pairs[g]];
            const unsigned long long v = (static_cast<unsigned long long>(mix32(key)) << 32) | (g - g0 + 1u);
            const uint32_t ia = key_lo(key), ib = key_hi(key);
            if (dyn(ia)) atomicMax(&best[ia - b0], v);
            if (dyn(ib)) atomicMax(&best[ib - b0], v);
        }
        ws_sync<WARP>();
        uint32_t won = 0;
        for (uint32_t g = g0 + lane; g < g1; g += nt) {
            if (A.colour[g] != NO_COLOUR) continue;
            const uint64_t key = A.pairs[A.contact_pairs[g]];
            const unsigned long long v = (static_cast<unsigned long long>(mix32(key)) << 32) | (g - g0 + 1u);
            const uint32_t ia = key_lo(key), ib = key_hi(key);
            const bool da = dyn(ia), db = dyn(ib);
            if ((da && best[ia - b0] != v) || (db && best[ib - b0] != v)) continue;
            const unsigned long long m = (da ? mask[ia - b0] : 0ull) | (db ? mask[ib - b0] : 0ull);
            int c = __ffsll(static_cast<long long>(~m)) - 1;
            if (c < 0) {  // 64 colours taken at one body
                atomicOr(A.status, ST_COLOUR_OVERFLOW);
                c = int(WS_MAX_COLOURS) - 1;
            }
            A.colour[g] = uint32_t(c);
            if (da) mask[ia - b0] |= 1ull << c;
            if (db) mask[ib - b0] |= 1ull << c;
            ++won;
        }
        for (uint32_t i = lane; i < nb; i += nt) other[i] = 0ull;
        if (won) atomicSub(&C.left, won);
        ws_sync<WARP>();
    }
}

// The whole PGS of world w by `nt` threads (lane = 0 .. nt - 1), `sm` its 4 * nb float4 of
// shared memory, `C` its context. Every thread of the CTA (block mode) or of the warp (warp
// mode) calls it; every early return is taken by all of them together, so every sync is
// reached by all of them.
template <bool WARP>
__device__ void solve_world(const WorldSolveArgs& A, uint32_t w, uint32_t lane, uint32_t nt, float4* sm, WorldCtx& C) {
    const SolveArgs& a = A.a;
    const uint32_t b0 = A.world_off[w], nb = A.world_off[w + 1] - b0;
    float4* lin = sm;
    float4* ang = sm + nb;
    float4* plin = sm + 2 * nb;
    float4* pang = sm + 3 * nb;
    for (uint32_t i = lane; i < nb; i += nt) {
        lin[i] = __ldcg(&A.linvel[b0 + i]);
        ang[i] = __ldcg(&A.angvel[b0 + i]);
    }
    // 1. Colours, with the push-velocity region as scratch.
    colour_world<WARP>(A, b0, nb, lane, nt, reinterpret_cast<unsigned long long*>(plin), C);
    const uint32_t g0 = C.g0, g1 = C.g1;
    if (g0 == g1 && !a.j.ncol) {  // no rows in this world: its velocities stay as they are
        if (lane == 0) {  // an empty record (the adjoint's reverse pass reads every world's)
            A.wcol[size_t(w) * WS_STRIDE] = g0;
            A.wcol[size_t(w) * WS_STRIDE + 1] = 0;
        }
        return;
    }
    // 2. Colour batches: histogram, offsets, scatter of the slot records.
    for (uint32_t g = g0 + lane; g < g1; g += nt) {
        const uint32_t c = A.colour[g];
        if (c >= WS_MAX_COLOURS) continue;  // left uncoloured (round limit; the status word says so)
        atomicAdd(&C.hist[c], 1u);
        atomicMax(&C.ncol, c + 1u);
    }
    ws_sync<WARP>();
    const uint32_t ncol = C.ncol;
    if (lane == 0) {
        uint32_t acc = 0;
        uint32_t* rec = A.wcol + size_t(w) * WS_STRIDE;
        rec[0] = g0;
        rec[1] = ncol;
        for (uint32_t c = 0; c < ncol; ++c) {
            C.off[c] = acc;
            C.cur[c] = acc;
            rec[2 + c] = acc;
            acc += C.hist[c];
        }
        C.off[ncol] = acc;
        rec[2 + ncol] = acc;
        if (ncol) atomicMax(&A.scalars[4], ncol);
    }
    ws_sync<WARP>();
    uint32_t my_rows = 0, my_split_groups = 0, my_split_rows = 0;
    for (uint32_t g = g0 + lane; g < g1; g += nt) {
        const uint32_t c = A.colour[g];
        if (c >= WS_MAX_COLOURS) continue;
        const uint32_t slot = g0 + atomicAdd(&C.cur[c], 1u);
        const uint32_t p = A.contact_pairs[g];
        const uint64_t key = A.pairs[p];
        const uint32_t cnt = A.row_count[p];
        uint32_t nsplit = 0;
        for (uint32_t k = 0; k < cnt; ++k) nsplit += a.rows[(size_t(p) * 4 + k) * ROW_F4 + 5].z != 0.0f ? 1u : 0u;
        A.recs[slot] = make_uint4(key_lo(key), key_hi(key), p | (cnt << 29), nsplit ? 1u : 0u);
        // The colour rides in the manifold's meta bits to seed next step's colouring.
        float* mw = &A.entries[size_t(p) * ENTRY_F4 + 2].w;
        *mw = __uint_as_float((__float_as_uint(*mw) & ~(0xffu << META_COLOUR_SHIFT)) | ((c + 1u) << META_COLOUR_SHIFT));
        my_rows += cnt;
        if (nsplit) {
            ++my_split_groups;
            my_split_rows += nsplit;
            atomicAdd(&C.split_hist[c], 1u);
        }
    }
    if (my_rows) atomicAdd(&C.rows, my_rows);
    if (my_split_groups) {
        atomicAdd(&C.split_groups, my_split_groups);
        atomicAdd(&C.split_rows, my_split_rows);
    }
    ws_sync<WARP>();  // the colouring scratch is free from here on
    for (uint32_t i = lane; i < nb; i += nt) {
        plin[i] = __ldcg(&A.push_lin[b0 + i]);
        pang[i] = __ldcg(&A.push_ang[b0 + i]);
    }
    if (lane == 0) {
        atomicAdd(&A.scalars[3], C.rows);
        if (C.split_groups) {
            atomicAdd(&A.scalars[5], C.split_groups);
            atomicAdd(&A.scalars[10], C.split_rows);
        }
    }
    for (uint32_t c = lane; c < ncol; c += nt) {
        atomicAdd(&A.colour_count[c], C.hist[c]);
        if (C.split_hist[c]) atomicAdd(&A.split_count[c], C.split_hist[c]);
    }
    ws_sync<WARP>();
    // 3. Warm start and velocity sweeps; split sweep s rides along velocity sweep s + 1.
    const uint32_t iters = a.iterations;
    for (uint32_t sweep = 0; sweep <= iters; ++sweep) {
        for (uint32_t c = 0; c < ncol; ++c) {
            const uint32_t hi = g0 + C.off[c + 1];
            for (uint32_t t = g0 + C.off[c] + lane; t < hi; t += nt) {
                const uint4 rec = A.recs[t];
                if (sweep == 0) run_group_shared<WARM>(a, t, rec, 0, iters, lin, ang, b0);
                else run_group_shared<ITER>(a, t, rec, sweep, iters, lin, ang, b0);
                if (sweep >= 1 && rec.w) run_group_shared<SPLIT>(a, t, rec, sweep - 1, iters - 1, plin, pang, b0);
            }
            ws_sync<WARP>();
        }
        // sequential_impulse.rs:720-735: a velocity sweep's joint rows follow its contacts (the
        // host allows joints here only for a plain world, whose bodies start at 0).
        if (sweep >= 1 && a.j.ncol) {
            for (uint32_t jc = 0; jc < a.j.ncol; ++jc) {
                const uint32_t hi = a.j.coff[jc + 1];
                for (uint32_t t = a.j.coff[jc] + lane; t < hi; t += nt)
                    solve_joint_slot<true>(a.j, t, lin, ang, a.iw, a.damping);
                ws_sync<WARP>();
            }
        }
    }
    // 4. The world's velocities and push velocities back to global memory.
    for (uint32_t i = lane; i < nb; i += nt) {
        __stcg(&A.linvel[b0 + i], lin[i]);
        __stcg(&A.angvel[b0 + i], ang[i]);
        __stcg(&A.push_lin[b0 + i], plin[i]);
        __stcg(&A.push_ang[b0 + i], pang[i]);
    }
}

// What k_world_prep leaves for k_solve_flow: the batches of one chunk.
struct WorldPrepOut {
    uint32_t *offset, *end;       // colour batch starts and ends (slots)
    uint4* split_rec;
    uint32_t *voff, *soff, *vsec; // FlowArgs
    uint32_t* split_flag;         // scratch, one a group
    float4* vel;                  // FlowArgs::vel and, 2 nb further on, push
};

// A plain world's colours and batches by one block, for k_solve_flow to solve with many: one launch
// instead of the global colouring's eleven, which for a world this small cost more than the solve.
// The colours are solve_world's; a batch holds its groups of 4 rows first, then 3, 2, 1.
__global__ void __launch_bounds__(512) k_world_prep(WorldSolveArgs A, WorldPrepOut O) {
    extern __shared__ float4 ws_dyn[];
    __shared__ WorldCtx C;
    __shared__ uint32_t hist[WS_MAX_COLOURS * 4], scur[WS_MAX_COLOURS];
    const SolveArgs& a = A.a;
    const uint32_t lane = threadIdx.x, nt = blockDim.x, nb = A.world_off[1];
    unsigned long long* mask = reinterpret_cast<unsigned long long*>(ws_dyn);
    for (uint32_t i = lane; i < 4 * nb; i += nt) O.vel[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (uint32_t i = lane; i < WS_MAX_COLOURS * 4; i += nt) hist[i] = 0;
    colour_world<false>(A, 0u, nb, lane, nt, mask, C);
    const uint32_t K = C.g1;
    // The colours of a body's groups and split groups (the masks above may hold dropped seeds too).
    unsigned long long *used = mask + nb, *split_used = used + nb;
    for (uint32_t i = lane; i < 2 * nb; i += nt) used[i] = 0ull;
    __syncthreads();
    auto dyn = [&](uint32_t i) { return inv_mass_of(a.iw, i) > 0.0f; };
    uint32_t rows = 0, split_groups = 0, split_rows = 0;
    for (uint32_t g = lane; g < K; g += nt) {
        const uint32_t c = A.colour[g];
        if (c >= WS_MAX_COLOURS) continue;  // left uncoloured (round limit; the status word says so)
        const uint32_t p = A.contact_pairs[g], cnt = A.row_count[p];
        const uint64_t key = A.pairs[p];
        uint32_t nsplit = 0;
        for (uint32_t k = 0; k < cnt; ++k) nsplit += a.rows[(size_t(p) * 4 + k) * ROW_F4 + 5].z != 0.0f ? 1u : 0u;
        O.split_flag[g] = nsplit;
        atomicAdd(&hist[c * 4 + (4u - cnt)], 1u);
        atomicMax(&C.ncol, c + 1u);
        rows += cnt;
        if (nsplit) {
            ++split_groups;
            split_rows += nsplit;
            atomicAdd(&C.split_hist[c], 1u);
        }
        const unsigned long long bit = 1ull << c;
        for (uint32_t side = 0; side < 2; ++side) {
            const uint32_t x = side ? key_hi(key) : key_lo(key);
            if (!dyn(x)) continue;
            atomicOr(&used[x], bit);
            if (nsplit) atomicOr(&split_used[x], bit);
        }
    }
    if (rows) atomicAdd(&C.rows, rows);
    if (split_groups) {
        atomicAdd(&C.split_groups, split_groups);
        atomicAdd(&C.split_rows, split_rows);
    }
    __syncthreads();
    const uint32_t ncol = C.ncol;
    if (lane < 32u) {  // batch offsets: two colours a lane
        uint32_t n[2], s[2], nsum = 0, ssum = 0;
        for (uint32_t k = 0; k < 2; ++k) {
            const uint32_t c = 2u * lane + k;
            n[k] = hist[4 * c] + hist[4 * c + 1] + hist[4 * c + 2] + hist[4 * c + 3];
            s[k] = C.split_hist[c];
            nsum += n[k];
            ssum += s[k];
        }
        uint32_t v = nsum, w = ssum;
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, v, o), y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) { v += x; w += y; }
        }
        v -= nsum;
        w -= ssum;
        for (uint32_t k = 0; k < 2; ++k) {
            const uint32_t c = 2u * lane + k;
            if (c < ncol) {
                O.offset[c] = O.voff[2 * c] = A.wcol[2 + c] = v;
                O.end[c] = O.voff[2 * c + 1] = v + n[k];
                O.soff[2 * c] = w;
                O.soff[2 * c + 1] = w + s[k];
                A.colour_count[c] = n[k];
                A.split_count[c] = s[k];
            }
            for (uint32_t r = 0; r < 4; ++r) {
                const uint32_t cnt = hist[4 * c + r];
                if (c < ncol) O.vsec[4 * c + r] = cnt;
                hist[4 * c + r] = v;  // the scatter's cursor
                v += cnt;
            }
            scur[c] = w;
            w += s[k];
            if (c + 1u == ncol) {
                O.offset[ncol] = A.wcol[2 + ncol] = v;
                A.scalars[3] = C.rows;
                A.scalars[4] = ncol;
                A.scalars[5] = C.split_groups;
                A.scalars[10] = C.split_rows;
            }
        }
        if (lane == 0) {
            A.wcol[0] = 0u;
            A.wcol[1] = ncol;
        }
    }
    __syncthreads();
    for (uint32_t g = lane; g < K; g += nt) {
        const uint32_t c = A.colour[g];
        if (c >= WS_MAX_COLOURS) continue;
        const uint32_t p = A.contact_pairs[g], cnt = A.row_count[p];
        const uint64_t key = A.pairs[p];
        const uint32_t ia = key_lo(key), ib = key_hi(key);
        const unsigned long long below = (1ull << c) - 1ull;
        auto rank = [&](const unsigned long long* m, uint32_t i) {
            return dyn(i) ? uint32_t(__popcll(m[i] & below)) | (uint32_t(__popcll(m[i])) << 8) : 0u;
        };
        uint4 rec = make_uint4(ia, ib, p | (cnt << 29), rank(used, ia) | (rank(used, ib) << 16));
        A.recs[atomicAdd(&hist[c * 4 + (4u - cnt)], 1u)] = rec;
        if (O.split_flag[g]) {
            rec.w = rank(split_used, ia) | (rank(split_used, ib) << 16);
            O.split_rec[atomicAdd(&scur[c], 1u)] = rec;
        }
        // The colour rides in the manifold's meta bits to seed next step's colouring.
        float* mw = &A.entries[size_t(p) * ENTRY_F4 + 2].w;
        *mw = __uint_as_float((__float_as_uint(*mw) & ~(0xffu << META_COLOUR_SHIFT)) | ((c + 1u) << META_COLOUR_SHIFT));
    }
}

// MAXT: the launch's largest block. Plans of up to 256 threads a CTA mix block and warp modes;
// the 512-thread build runs only plans whose worlds are all in block mode (one large world).
template <int MAXT>
__global__ void __launch_bounds__(MAXT) k_world_solve(WorldSolveArgs A) {
    extern __shared__ float4 ws_dyn[];
    __shared__ WorldCtx ctx[MAXT > 256 ? 1 : WS_MAX_WARPS];
    const uint2 c = A.plan.cta[blockIdx.x];
    const bool block_mode = (c.y >> 31) != 0u;
    const uint32_t count = c.y & 0x7fffffffu;
    if (block_mode) {
        solve_world<false>(A, A.plan.list[c.x], threadIdx.x, blockDim.x, ws_dyn, ctx[0]);
        return;
    }
    if (MAXT > 256) return;  // the plan builder gives this build block-mode plans only
    const uint32_t wi = threadIdx.x >> 5;
    if (wi >= count) return;  // warp mode: warps never sync with each other
    uint32_t off = 0;
    for (uint32_t j = 0; j < wi; ++j) {
        const uint32_t wj = A.plan.list[c.x + j];
        off += A.world_off[wj + 1] - A.world_off[wj];
    }
    solve_world<true>(A, A.plan.list[c.x + wi], threadIdx.x & 31u, 32u, ws_dyn + 4 * size_t(off), ctx[wi]);
}

// ---------------------------------------------------------------- cache update
// step.rs:982-1010. Tiles [0, ta): the solved normal impulse goes back to its manifold point, and the
// surviving manifolds of the current pairs go, in pair order, to the new cache. Tiles [ta, ..): the
// old manifolds that no pair took over and whose world does not prune (prune = simulate &&
// prev_simulate). When every world prunes there are none of these, the new cache's positions are
// the current manifolds' ranks, and their entries are copied here and now; otherwise the two lists go to
// k_merge.
// What bounds it: the 256-byte manifolds' traffic and, on small worlds, its own latency. One launch
// for what took nine (write-back, two flag passes and two selections): 1,000-box stack 8.5 us for 20,
// 131,072-body pile 100 us for 123 (write-back 43, merge 50, the rest the selections).
struct CacheArgs {
    uint32_t npairs, nold, ta;
    const uint32_t* row_count;
    const float4* rows;
    float4* entries;
    const uint64_t* pairs;
    const uint32_t* owned;
    const uint64_t* old_keys;
    const uint32_t *world_of, *simulate, *prev_simulate;
    uint32_t *sel_a, *sel_b, *scalars;  // scalars[8], [9]: the lists' lengths; [12]: every world prunes
    uint64_t* out_keys;
    float4* out_entries;
    uint32_t* out_count;
    uint32_t* rec_merge_pos;
};

template <uint32_t ROUNDS>
__global__ void __launch_bounds__(TILE_TB) k_cache_lists(CacheArgs a, TileScan ts) {
    constexpr uint32_t ITEMS = TILE_TB * ROUNDS;
    __shared__ uint32_t s_pair[ITEMS];  // the tile's surviving pairs | rows << 29
    const uint32_t tile = tile_take(ts);
    const bool prune_all = a.scalars[12] != 0u;
    bool flag[ROUNDS];
    uint32_t rank[ROUNDS];
    if (tile >= a.ta) {
        if (prune_all) return;
        const uint32_t base = (tile - a.ta) * ITEMS;
#pragma unroll
        for (uint32_t r = 0; r < ROUNDS; ++r) {
            const uint32_t o = base + r * TILE_TB + threadIdx.x;
            flag[r] = false;
            if (o < a.nold) {
                const uint32_t w = a.world_of ? a.world_of[key_lo(a.old_keys[o])] : 0u;
                flag[r] = !(a.simulate[w] != 0u && a.prev_simulate[w] != 0u) && !a.owned[o];
            }
        }
        const uint32_t total = tile_ranks(flag, rank);
        const uint32_t at = tile_prefix(ts, tile, a.ta, total);
#pragma unroll
        for (uint32_t r = 0; r < ROUNDS; ++r)
            if (flag[r]) a.sel_b[at + rank[r]] = base + r * TILE_TB + threadIdx.x;
        if (base + ITEMS >= a.nold && threadIdx.x == 0) a.scalars[9] = at + total;
        return;
    }
    const uint32_t base = tile * ITEMS;
    uint32_t rows[ROUNDS];
#pragma unroll
    for (uint32_t r = 0; r < ROUNDS; ++r) {
        const uint32_t p = base + r * TILE_TB + threadIdx.x;
        flag[r] = p < a.npairs && (__float_as_uint(a.entries[size_t(p) * ENTRY_F4 + 2].w) & META_VALID) != 0u;
        rows[r] = p < a.npairs ? a.row_count[p] : 0u;
    }
    const uint32_t total = tile_ranks(flag, rank);
#pragma unroll
    for (uint32_t r = 0; r < ROUNDS; ++r)
        if (flag[r]) s_pair[rank[r]] = (base + r * TILE_TB + threadIdx.x) | (rows[r] << 29);
    const uint32_t at = tile_prefix(ts, tile, 0u, total);  // (its last step is a block barrier: s_pair is ready)
    if (base + ITEMS >= a.npairs && threadIdx.x == 0) {
        a.scalars[8] = at + total;
        if (prune_all) *a.out_count = at + total;
    }
    // 16 threads a manifold, one float4 each: point k's impulse is word w of entry 5 + 3 k.
    const uint32_t q = threadIdx.x & 15u, k = (q - 5u) / 3u;
    const bool holds = q >= 5u && (q - 5u) % 3u == 0u;
    if (prune_all) {
        constexpr uint32_t BATCH = 4;  // manifolds in flight a thread
        for (uint32_t t0 = threadIdx.x >> 4; t0 < total; t0 += BATCH * (TILE_TB / 16u)) {
            float4 e[BATCH];
            float imp[BATCH];
#pragma unroll
            for (uint32_t u = 0; u < BATCH; ++u) {
                const uint32_t t = t0 + u * (TILE_TB / 16u);
                if (t >= total) continue;
                const uint32_t x = s_pair[t], p = x & 0x1fffffffu;
                e[u] = __ldcs(&a.entries[size_t(p) * ENTRY_F4 + q]);
                imp[u] = e[u].w;
                if (holds && k < x >> 29) imp[u] = a.rows[(size_t(p) * 4 + k) * ROW_F4 + 3].x;
            }
#pragma unroll
            for (uint32_t u = 0; u < BATCH; ++u) {
                const uint32_t t = t0 + u * (TILE_TB / 16u);
                if (t >= total) continue;
                e[u].w = imp[u];
                a.out_entries[size_t(at + t) * ENTRY_F4 + q] = e[u];
                if (q == 0u) {
                    const uint32_t p = s_pair[t] & 0x1fffffffu;
                    a.out_keys[at + t] = a.pairs[p];
                    if (a.rec_merge_pos) a.rec_merge_pos[p] = at + t;
                }
            }
        }
        return;
    }
    for (uint32_t t = threadIdx.x >> 4; t < total; t += TILE_TB / 16u) {
        const uint32_t p = s_pair[t] & 0x1fffffffu;
        if (holds && k < s_pair[t] >> 29)
            a.entries[size_t(p) * ENTRY_F4 + q].w = a.rows[(size_t(p) * 4 + k) * ROW_F4 + 3].x;
        if (q == 0u) a.sel_a[at + t] = p;
    }
}

__device__ __forceinline__ uint32_t lower_bound_pairs(const uint64_t* __restrict__ pairs, const uint32_t* __restrict__ sel,
                                                      uint32_t n, uint64_t key) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        uint32_t mid = (lo + hi) >> 1;
        if (pairs[sel[mid]] < key) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ uint32_t lower_bound_keys(const uint64_t* __restrict__ keys, const uint32_t* __restrict__ sel,
                                                     uint32_t n, uint64_t key) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        uint32_t mid = (lo + hi) >> 1;
        if (keys[sel[mid]] < key) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Merge the surviving current manifolds (A, pair order) with the surviving old ones (B, key order).
__global__ void k_merge(const uint64_t* __restrict__ pairs, const float4* __restrict__ cur_entries,
                        const uint32_t* __restrict__ sel_a, const uint32_t* __restrict__ na_ptr,
                        const uint64_t* __restrict__ old_keys, const float4* __restrict__ old_entries,
                        const uint32_t* __restrict__ sel_b, const uint32_t* __restrict__ nb_ptr, uint64_t* out_keys,
                        float4* out_entries, uint32_t* out_count, uint32_t* rec_merge_pos,
                        const uint32_t* __restrict__ done) {
    if (*done) return;  // every world pruned: k_cache_lists has filled the cache
    uint32_t na = *na_ptr, nb = *nb_ptr;
    uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0) *out_count = na + nb;
    if (t < na) {
        uint32_t p = sel_a[t];
        uint64_t key = pairs[p];
        uint32_t pos = t + (nb ? lower_bound_keys(old_keys, sel_b, nb, key) : 0u);
        out_keys[pos] = key;
        if (rec_merge_pos) rec_merge_pos[p] = pos;
        const float4* src = cur_entries + size_t(p) * ENTRY_F4;
        float4* dst = out_entries + size_t(pos) * ENTRY_F4;
        for (int q = 0; q < ENTRY_F4; ++q) dst[q] = src[q];
    } else if (t < na + nb) {
        uint32_t b = t - na;
        uint32_t o = sel_b[b];
        uint64_t key = old_keys[o];
        uint32_t pos = b + lower_bound_pairs(pairs, sel_a, na, key);
        out_keys[pos] = key;
        const float4* src = old_entries + size_t(o) * ENTRY_F4;
        float4* dst = out_entries + size_t(pos) * ENTRY_F4;
        for (int q = 0; q < ENTRY_F4; ++q) dst[q] = src[q];
    }
}

// A barrier whose target counts one block more than the grid has: nothing completes it.
__global__ void k_wait_selftest(unsigned int* ctr, uint32_t* status, unsigned long long limit_ns) {
    team_barrier(ctr, gridDim.x + 1u, status, limit_ns);
}

int device_sms() {
    static int sms = -1;
    if (sms < 0) {
        int dev = 0;
        check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
        check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "sm count");
    }
    return sms;
}

int coop_grid(const void* fn, int block, size_t smem) {
    static int sms = -1;
    if (sms < 0) {
        int dev = 0;
        check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
        check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "sm count");
    }
    int per_sm = 0;
    check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, block, smem), "occupancy");
    if (per_sm < 1) per_sm = 1;
    return sms * per_sm;
}

}  // namespace

// PGS (cooperative launch: the teams' barriers need every block resident).
static void launch_solve(const WorldView& w, PairData& pd, const StepParams& sp, uint32_t* status_dev, cudaStream_t s,
                         const JointsDev* joints) {
    const int TB = 256;
    check_cuda(cudaMemsetAsync(pd.barrier.p, 0, 2 * sizeof(unsigned int), s), "memset barrier");
    SolveArgs sa{pd.rows.p, pd.batch_rec.p, pd.colour_offset.p, pd.colour_cursor.p, pd.split_rec.p,
                 pd.split_offset.p, pd.split_cursor.p, pd.scalars.p, w.b.linvel, w.b.angvel, w.b.push_lin,
                 w.b.push_ang, w.b.iw, pd.vtab.p, pd.stab.p, pd.rec.sweeps,
                 pd.barrier.p, status_dev, sp.inv_dt, sp.info.restitution_velocity_threshold,
                 sp.info.num_iterations, joints ? *joints : JointsDev{}, sp.info.damping};
    const void* fn = joints ? (const void*)k_solve<true> : (const void*)k_solve<false>;
    static int solve_grid[2] = {0, 0};
    int& grid = solve_grid[joints ? 1 : 0];
    if (!grid) grid = coop_grid(fn, TB, 0);
    void* sargs[] = {&sa};
    check_cuda(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(TB), sargs, 0, s), "solve launch");
}

// The PGS kernel for worlds without joints is the chunked one; BGPU_PGS=team in the
// environment keeps the team-barrier kernel (which worlds with joints always use), for
// comparison.
static int pgs_mode() {
    static int mode = -1;
    if (mode < 0) {
        const char* e = std::getenv("BGPU_PGS");
        mode = (e && std::strcmp(e, "team") == 0) ? 1 : 2;
    }
    return mode;
}

// Plain worlds of up to 1,024 bodies: one block colours and batches, many solve, four warps each.
// A phase then costs a trip through L2 (1.8 us) but a warp holds only a few groups, where one block's
// threads solve theirs in turn, each contact after a table load. Measured on box stacks, colouring
// and solve: 1,000 bodies 504 us by one block, 209 / 200 / 196 us with 64 / 32 / 16 bodies a block;
// 512 bodies 262 and 137, 216 bodies 111 and 109, 125 bodies 88 and 105, 8 bodies 48 and 58. Hence
// the line at 256 bodies, below which one block solves the world alone.
constexpr uint32_t SMALL_BODIES_PER_BLOCK = 16;
constexpr uint32_t SMALL_FLOW_MIN_BODIES = 256;

static int g_last_solver_kind = 0;
int last_solver_kind() { return g_last_solver_kind; }

static int chunk_grid() {
    static int grid = 0;
    if (!grid) {
        check_cuda(cudaFuncSetAttribute((const void*)k_solve_flow<CHUNK_TB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        int(flow_smem(CHUNK_TB))), "smem attribute");
        grid = coop_grid((const void*)k_solve_flow<CHUNK_TB>, CHUNK_TB, flow_smem(CHUNK_TB));
    }
    if (grid > int(CHUNK_MAX)) throw CudaError{cudaErrorInvalidValue, "chunked PGS: more blocks than chunk slots"};
    return grid;
}

void run_wait_selftest(unsigned long long limit_ns, unsigned int* ctr, uint32_t* status, cudaStream_t s) {
    k_wait_selftest<<<2, 32, 0, s>>>(ctr, status, limit_ns);
}

void run_solver(const WorldView& w, const uint64_t* pairs, uint32_t npairs, PairData& pd, const StepParams& sp,
                uint32_t* status_dev, cudaStream_t s, const std::function<void(int)>& mark, bool seed_colours,
                const JointsDev* joints, const uint32_t* morton_leaf, uint32_t tree_m) {
    const bool with_joints = joints && joints->n && joints->ncol;
    g_last_solver_kind = 0;
    if (npairs == 0) {
        mark(5);
        if (with_joints) {
            launch_solve(w, pd, sp, status_dev, s, joints);
            g_last_solver_kind = 1;
        }
        mark(6);
        return;
    }
    const int mode = with_joints ? 1 : pgs_mode();
    const bool chunked = mode == 2;
    const int TB = 256;
    if (npairs >= (1u << 29)) throw CudaError{cudaErrorInvalidValue, "more than 2^29 pairs for the solver's slot records"};
    // Contact pairs (ascending pair order).
    launch_contact_list(npairs, pd, sp, status_dev, s);
    // Chunks: each body's chunk; the (colour, chunk) counts and the bodies' colour masks come with
    // the colour histograms.
    uint32_t P = 0;
    uint32_t *vhist = nullptr, *shist = nullptr;
    if (chunked) {
        P = uint32_t(chunk_grid());
        const uint32_t n = w.nbodies;
        pd.chunk_of.reserve(std::max<uint32_t>(n, 1));
        pd.chunk_hist.reserve(size_t(MAX_COLOURS) * P * 5);
        pd.chunk_off.reserve(2 * size_t(MAX_COLOURS) * (P + 1) + size_t(MAX_COLOURS) * P * 4);
        pd.flow_vel.reserve(4 * size_t(std::max<uint32_t>(n, 1)));
        vhist = pd.chunk_hist.p;
        shist = pd.chunk_hist.p + size_t(MAX_COLOURS) * P * 4;
    }
    // Colouring (cooperative launch).
    ColourArgs ca{pd.scalars.p + 2, pd.contact_pairs.p, pairs, w.b.iw, pd.colour.p, pd.body_prio.p, pd.body_mask.p,
                  pd.body_dup.p, chunked ? pd.body_used.p : nullptr, pd.entries.p, seed_colours ? 1u : 0u, pd.barrier.p,
                  status_dev, vhist, P * MAX_COLOURS * 5u};
    // Two blocks per SM: enough threads for a pile's groups, and the rounds' grid barriers
    // are cheaper than with every block the SM could hold.
    static int colour_grid = 0;
    if (!colour_grid) colour_grid = std::min(coop_grid((const void*)k_colour, TB, 0), 2 * device_sms());
    pd.colour_work.reserve(2 * size_t(npairs) + 2);
    JpList wl{{pd.colour_work.p, pd.colour_work.p + npairs}, {pd.barrier.p + 6, pd.barrier.p + 7}};
    void* cargs[] = {&ca, &wl};
    check_cuda(cudaLaunchCooperativeKernel((const void*)k_colour, dim3(colour_grid), dim3(TB), cargs, 0, s),
               "colour launch");
    // Batches.
    uint32_t* sub_hist = pd.colour_sub.p;
    uint32_t* sub_cursor = pd.colour_sub.p + 4 * MAX_COLOURS;
    uint32_t g = std::min<uint32_t>((npairs + TB - 1) / TB, 148u * 8u);
    if (chunked) {
        const uint32_t n = w.nbodies;
        const bool tree = morton_leaf && tree_m;
        k_chunk_of<<<std::min<uint32_t>((4 * n + TB - 1) / TB, 148u * 8u), TB, 0, s>>>(
            n, P, tree ? morton_leaf : nullptr, tree_m, pd.chunk_of.p, pd.flow_vel.p);
    }
    k_colour_hist<<<g, TB, 0, s>>>(pd.scalars.p + 2, pd.contact_pairs.p, pd.colour.p, pd.row_count.p, pd.rows.p,
                                   pd.colour_count.p, pd.split_count.p, pd.flags.p, sub_hist, pairs, w.b.iw,
                                   pd.chunk_of.p, P, vhist, shist, pd.body_used.p);
    k_colour_scan<<<1, 32, 0, s>>>(pd.colour_count.p, pd.colour_offset.p, pd.colour_cursor.p, pd.split_count.p,
                                   pd.split_offset.p, pd.split_cursor.p, pd.barrier.p, pd.scalars.p, pd.colour_remap.p,
                                   sub_hist, sub_cursor, chunked ? 1u : 0u);
    uint32_t *voff = nullptr, *soff = nullptr, *vsec = nullptr;
    if (chunked) {
        voff = pd.chunk_off.p;
        soff = pd.chunk_off.p + size_t(MAX_COLOURS) * (P + 1);
        vsec = pd.chunk_off.p + 2 * size_t(MAX_COLOURS) * (P + 1);
        k_chunk_scan<256><<<MAX_COLOURS, 256, 0, s>>>(P, pd.colour_count.p, pd.colour_remap.p, pd.colour_offset.p,
                                                      pd.split_offset.p, pd.barrier.p, vhist, shist, voff, soff, vsec);
    }
    k_colour_scatter<<<g, TB, 0, s>>>(pd.scalars.p + 2, pd.contact_pairs.p, pairs, pd.row_count.p, pd.colour.p,
                                      pd.flags.p, sub_cursor, pd.split_cursor.p, pd.batch_rec.p,
                                      pd.split_rec.p, pd.entries.p, pd.colour_remap.p, pd.chunk_of.p, w.b.iw, P,
                                      vhist, shist, pd.body_used.p);
    mark(5);
    // Slot capacity: every group plus the 32-alignment padding of each batch.
    const size_t slots = (size_t(npairs) + 32u * (MAX_COLOURS + 1) + 31u) & ~size_t(31);
    pd.vtab.reserve(size_t(VT_PLANES) * 4 * slots);
    pd.stab.reserve(size_t(ST_PLANES) * 4 * slots);
    if (chunked) {
        SolveArgs sa{pd.rows.p, pd.batch_rec.p, pd.colour_offset.p, pd.colour_cursor.p, pd.split_rec.p,
                     pd.split_offset.p, pd.split_cursor.p, pd.scalars.p, w.b.linvel, w.b.angvel, w.b.push_lin,
                     w.b.push_ang, w.b.iw, pd.vtab.p, pd.stab.p, pd.rec.sweeps,
                     pd.barrier.p, status_dev, sp.inv_dt, sp.info.restitution_velocity_threshold,
                     sp.info.num_iterations, JointsDev{}, sp.info.damping};
        FlowArgs fa{P, 1u, voff, soff, vsec, pd.flow_vel.p, pd.flow_vel.p + 2 * size_t(w.nbodies)};
        k_flow_table<<<std::min<uint32_t>((npairs + TB / 4 - 1) / (TB / 4), 148u * 8u), TB, 0, s>>>(sa);
        void* args[] = {&sa, &fa};
        check_cuda(cudaLaunchCooperativeKernel((const void*)k_solve_flow<CHUNK_TB>, dim3(P), dim3(CHUNK_TB), args,
                                               flow_smem(CHUNK_TB), s), "chunked solve launch");
        g_last_solver_kind = 2;
    } else {
        launch_solve(w, pd, sp, status_dev, s, with_joints ? joints : nullptr);
        g_last_solver_kind = 1;
    }
    mark(6);
}

bool build_world_plan(const std::vector<uint32_t>& world_off, uint32_t block, uint32_t tau, WorldPlan& plan,
                      cudaStream_t s) {
    plan.valid = false;
    // Up to 256 threads a CTA; 512 when every world runs in block mode (tau 0).
    if (block < 32 || block > (tau == 0 ? 512u : 32u * WS_MAX_WARPS) || block % 32) return false;
    const uint32_t nw = world_off.empty() ? 0u : uint32_t(world_off.size() - 1);
    std::vector<uint32_t> order(nw);
    for (uint32_t k = 0; k < nw; ++k) order[k] = k;
    auto size = [&](uint32_t k) { return world_off[k + 1] - world_off[k]; };
    std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return size(x) > size(y); });
    const size_t smem_cap = 200u * 1024u;  // leaves room for the static contexts and L1
    std::vector<uint2> cta;
    size_t smem = 0;
    const uint32_t per_cta = block / 32;
    uint32_t k = 0;
    while (k < nw) {
        const uint32_t nb = size(order[k]);
        if (nb > tau) {  // block mode: one world per CTA
            if (size_t(nb) * WS_SMEM_PER_BODY > smem_cap) return false;
            cta.push_back(make_uint2(k, 1u | (1u << 31)));
            smem = std::max(smem, size_t(nb) * WS_SMEM_PER_BODY);
            ++k;
            continue;
        }
        uint32_t cnt = 0;
        size_t bodies = 0;
        while (k + cnt < nw && cnt < per_cta && (bodies + size(order[k + cnt])) * WS_SMEM_PER_BODY <= smem_cap) {
            bodies += size(order[k + cnt]);
            ++cnt;
        }
        if (cnt == 0) return false;
        cta.push_back(make_uint2(k, cnt));
        smem = std::max(smem, bodies * WS_SMEM_PER_BODY);
        k += cnt;
    }
    plan.cta.reserve(std::max<size_t>(cta.size(), 1));
    plan.list.reserve(std::max<uint32_t>(nw, 1));
    if (!cta.empty())
        check_cuda(cudaMemcpyAsync(plan.cta.p, cta.data(), cta.size() * sizeof(uint2), cudaMemcpyHostToDevice, s), "h2d");
    if (nw) check_cuda(cudaMemcpyAsync(plan.list.p, order.data(), nw * sizeof(uint32_t), cudaMemcpyHostToDevice, s), "h2d");
    check_cuda(cudaStreamSynchronize(s), "sync");  // the host vectors go out of scope
    // Without this opt-in, dynamic shared memory is limited to 48 KB minus the kernel's static part.
    // The limit is the function's, for every world of the process: always the largest plan's.
    check_cuda(cudaFuncSetAttribute(block > 256 ? (const void*)k_world_solve<512> : (const void*)k_world_solve<256>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem_cap)), "smem attribute");
    plan.ncta = uint32_t(cta.size());
    plan.block = block;
    plan.tau = tau;
    plan.smem = smem;
    plan.valid = true;
    return true;
}

void run_world_solver(const WorldView& w, const uint64_t* pairs, uint32_t npairs, PairData& pd, const StepParams& sp,
                      uint32_t* status_dev, cudaStream_t s, const std::function<void(int)>& mark,
                      const uint32_t* world_off, uint32_t nworlds, const WorldPlan& plan, uint32_t* wcol,
                      const JointsDev* joints, bool seed_colours) {
    const bool with_joints = joints && joints->n && joints->ncol;
    if (nworlds == 0 || (npairs == 0 && !with_joints)) {
        mark(5);
        mark(6);
        return;
    }
    const int TB = 256;
    if (npairs >= (1u << 29)) throw CudaError{cudaErrorInvalidValue, "more than 2^29 pairs for the solver's slot records"};
    if (npairs) launch_contact_list(npairs, pd, sp, status_dev, s);
    mark(5);
    // A plain world's contacts go to many blocks; with joints, and a world of a few bodies, to one
    // block with its velocities in shared memory.
    const bool prep = !with_joints && nworlds == 1 && plan.block > 256 && w.nbodies >= SMALL_FLOW_MIN_BODIES;
    const size_t slots = (size_t(npairs) + 32u * (MAX_COLOURS + 1) + 31u) & ~size_t(31);
    pd.vtab.reserve(size_t(VT_PLANES) * 4 * slots);
    pd.stab.reserve(size_t(ST_PLANES) * 4 * slots);
    WorldSolveArgs A;
    A.a = SolveArgs{pd.rows.p, pd.batch_rec.p, pd.colour_offset.p, pd.colour_cursor.p, pd.split_rec.p,
                    pd.split_offset.p, pd.split_cursor.p, pd.scalars.p, w.b.linvel, w.b.angvel, w.b.push_lin,
                    w.b.push_ang, w.b.iw, pd.vtab.p, pd.stab.p, pd.rec.sweeps,
                    pd.barrier.p, status_dev, sp.inv_dt, sp.info.restitution_velocity_threshold,
                    sp.info.num_iterations, with_joints ? *joints : JointsDev{}, sp.info.damping};
    A.contact_pairs = pd.contact_pairs.p;
    A.ngroups = pd.scalars.p + 2;
    A.pairs = pairs;
    A.row_count = pd.row_count.p;
    A.world_off = world_off;
    A.colour = pd.colour.p;
    A.recs = pd.batch_rec.p;
    A.wcol = wcol;
    A.colour_count = pd.colour_count.p;
    A.split_count = pd.split_count.p;
    A.scalars = pd.scalars.p;
    A.linvel = w.b.linvel;
    A.angvel = w.b.angvel;
    A.push_lin = w.b.push_lin;
    A.push_ang = w.b.push_ang;
    A.status = status_dev;
    A.plan = plan.dev();
    A.entries = pd.entries.p;
    A.seed = seed_colours ? 1u : 0u;
    if (prep) {
        const uint32_t n = w.nbodies;
        pd.chunk_off.reserve(size_t(WS_MAX_COLOURS) * 8);
        pd.flow_vel.reserve(4 * size_t(n));
        uint32_t *voff = pd.chunk_off.p, *soff = voff + 2 * WS_MAX_COLOURS, *vsec = soff + 2 * WS_MAX_COLOURS;
        const WorldPrepOut O{pd.colour_offset.p, pd.colour_cursor.p, pd.split_rec.p, voff, soff, vsec, pd.flags.p,
                             pd.flow_vel.p};
        k_world_prep<<<1, 512, size_t(n) * 32, s>>>(A, O);
        const uint32_t blocks = std::min<uint32_t>((n + SMALL_BODIES_PER_BLOCK - 1) / SMALL_BODIES_PER_BLOCK,
                                                   uint32_t(device_sms()));
        k_flow_table<<<std::min<uint32_t>((npairs + TB / 4 - 1) / (TB / 4), 148u * 8u), TB, 0, s>>>(A.a);
        FlowArgs fa{1u, blocks, voff, soff, vsec, pd.flow_vel.p, pd.flow_vel.p + 2 * size_t(n)};
        void* args[] = {&A.a, &fa};
        check_cuda(cudaLaunchCooperativeKernel((const void*)k_solve_flow<SMALL_TB>, dim3(blocks), dim3(SMALL_TB), args,
                                               flow_smem(SMALL_TB), s), "solve launch");
    } else if (plan.block > 256) k_world_solve<512><<<plan.ncta, plan.block, plan.smem, s>>>(A);
    else k_world_solve<256><<<plan.ncta, plan.block, plan.smem, s>>>(A);
    check_cuda(cudaGetLastError(), "world solve launch");
    mark(6);
}

void run_cache_update(const uint64_t* pairs, uint32_t npairs, const Manifolds& old_cache, PairData& pd,
                      Manifolds& next, const uint32_t* world_of, const uint32_t* simulate_flag,
                      const uint32_t* prev_simulate, uint32_t* status_dev, cudaStream_t s) {
    // The exact old count: the world syncs on it before the step.
    const uint32_t nold = old_cache.count_host;
    const size_t cap = size_t(npairs) + nold + 1;
    next.keys.reserve(cap);
    next.entries.reserve(cap * ENTRY_F4);
    const uint32_t total = npairs + nold;
    if (!total) {
        check_cuda(cudaMemsetAsync(next.count_dev, 0, sizeof(uint32_t), s), "memset");
        return;
    }
    // Small tiles where blocks are few, so that many copy; large ones where the look-back counts.
    const bool large = npairs > (1u << 17);
    const uint32_t ta = std::max(large ? tile_count<4>(npairs) : tile_count<1>(npairs), 1u);
    const uint32_t tiles = ta + (large ? tile_count<4>(nold) : tile_count<1>(nold));
    const CacheArgs a{npairs, nold, ta, pd.row_count.p, pd.rows.p, pd.entries.p, pairs, pd.old_owned.p, old_cache.keys.p,
                      world_of, simulate_flag, prev_simulate, pd.sel_a.p, pd.sel_b.p, pd.scalars.p,
                      next.keys.p, next.entries.p, next.count_dev, pd.rec.merge_pos};
    if (large) k_cache_lists<4><<<tiles, TILE_TB, 0, s>>>(a, pd.cache_scan.begin(tiles, status_dev, s));
    else k_cache_lists<1><<<tiles, TILE_TB, 0, s>>>(a, pd.cache_scan.begin(tiles, status_dev, s));
    k_merge<<<(total + TILE_TB - 1) / TILE_TB, TILE_TB, 0, s>>>(
        pairs, pd.entries.p, pd.sel_a.p, pd.scalars.p + 8, old_cache.keys.p, old_cache.entries.p, pd.sel_b.p,
        pd.scalars.p + 9, next.keys.p, next.entries.p, next.count_dev, pd.rec.merge_pos, pd.scalars.p + 12);
    pd.old_owned.reserve(cap);  // the next step clears and fills a mark for each of its old manifolds
}

}  // namespace bgpu

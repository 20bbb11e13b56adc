// Broad phase: Morton-ordered linear BVH (Karras 2012 radix-tree build,
// bottom-up refit) over the bounded proxies, queried once per proxy.
//
// Output contract (crates/bullet-collision/src/broadphase/mod.rs:94-130,
// brute_force.rs:54-68): every pair (i < j) whose closed AABBs overlap on all
// three axes (util.rs:28-38), sorted lexicographically. Each proxy i owns the
// segment of partners j > i. One tree walk per proxy counts its partners and
// keeps them, sorted, in a fixed number of stash slots; an exclusive scan of
// the counts places the segments and a copy pass moves the stashed ones into
// place, so no global pair sort is needed. The few proxies with more partners
// than slots walk the tree a second time and write their segment directly.
// Unbounded proxies (planes) are kept out of the tree and joined by an ordered
// flag/scan compaction.
#include <cub/cub.cuh>
#include "k_scan.cuh"

namespace bgpu {

namespace {

constexpr int STACK_DEPTH = 64;
constexpr int LOCAL_SORT = 48;

__device__ __forceinline__ bool overlaps(float4 amin, float4 amax, float4 bmin, float4 bmax) {
    return amin.x <= bmax.x && amin.y <= bmax.y && amin.z <= bmax.z && bmin.x <= amax.x && bmin.y <= amax.y &&
           bmin.z <= amax.z;
}

// The same without branches, for the loops in which every lane tests.
__device__ __forceinline__ bool overlaps_all(float4 amin, float4 amax, float4 bmin, float4 bmax) {
    return (amin.x <= bmax.x) & (amin.y <= bmax.y) & (amin.z <= bmax.z) & (bmin.x <= amax.x) & (bmin.y <= amax.y) &
           (bmin.z <= amax.z);
}

__global__ void k_reset_bounds(int* bounds) {
    if (threadIdx.x < 3) bounds[threadIdx.x] = 0x7fffffff;
    else if (threadIdx.x < 6) bounds[threadIdx.x] = int(0x80000000);
}

__global__ void k_bounds(const float4* __restrict__ mn, const float4* __restrict__ mx, const uint32_t* __restrict__ is_unb,
                         uint32_t n, int* bounds) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    float cx = INFINITY, cy = INFINITY, cz = INFINITY, dx = -INFINITY, dy = -INFINITY, dz = -INFINITY;
    if (i < n && !is_unb[i]) {
        float4 a = mn[i], b = mx[i];
        cx = dx = 0.5f * (a.x + b.x);
        cy = dy = 0.5f * (a.y + b.y);
        cz = dz = 0.5f * (a.z + b.z);
    }
    typedef cub::BlockReduce<float, 256> BR;
    __shared__ typename BR::TempStorage t;
    float r;
    r = BR(t).Reduce(cx, cub::Min()); __syncthreads(); if (threadIdx.x == 0 && r < INFINITY) atomicMin(&bounds[0], float_to_ordered(r));
    r = BR(t).Reduce(cy, cub::Min()); __syncthreads(); if (threadIdx.x == 0 && r < INFINITY) atomicMin(&bounds[1], float_to_ordered(r));
    r = BR(t).Reduce(cz, cub::Min()); __syncthreads(); if (threadIdx.x == 0 && r < INFINITY) atomicMin(&bounds[2], float_to_ordered(r));
    r = BR(t).Reduce(dx, cub::Max()); __syncthreads(); if (threadIdx.x == 0 && r > -INFINITY) atomicMax(&bounds[3], float_to_ordered(r));
    r = BR(t).Reduce(dy, cub::Max()); __syncthreads(); if (threadIdx.x == 0 && r > -INFINITY) atomicMax(&bounds[4], float_to_ordered(r));
    r = BR(t).Reduce(dz, cub::Max()); __syncthreads(); if (threadIdx.x == 0 && r > -INFINITY) atomicMax(&bounds[5], float_to_ordered(r));
}

__device__ __forceinline__ uint32_t expand_bits(uint32_t v) {
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

__device__ __forceinline__ uint32_t quantize(float c, float lo, float hi) {
    float ext = hi - lo;
    float t = ext > 0.0f ? (c - lo) / ext : 0.0f;
    t = fminf(fmaxf(t, 0.0f), 1.0f);
    return uint32_t(t * 1023.0f);
}

// Morton code of each proxy's AABB centre (unbounded proxies: all ones, so they sort last),
// and the proxy index as the sort's value. A stable radix sort of the 32-bit codes with the
// indices as values orders the proxies exactly as sorting (code << 32 | index) would, in
// four 8-bit passes instead of eight.
__global__ void k_keys(const float4* __restrict__ mn, const float4* __restrict__ mx, const uint32_t* __restrict__ is_unb,
                       uint32_t n, const int* __restrict__ bounds, uint32_t* codes, uint32_t* index, uint32_t* zero) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0 && zero) *zero = 0u;  // the query's overflow count
    if (i >= n) return;
    index[i] = i;
    if (is_unb[i]) { codes[i] = 0xffffffffu; return; }
    float4 a = mn[i], b = mx[i];
    float lo0 = ordered_to_float(bounds[0]), lo1 = ordered_to_float(bounds[1]), lo2 = ordered_to_float(bounds[2]);
    float hi0 = ordered_to_float(bounds[3]), hi1 = ordered_to_float(bounds[4]), hi2 = ordered_to_float(bounds[5]);
    uint32_t x = quantize(0.5f * (a.x + b.x), lo0, hi0);
    uint32_t y = quantize(0.5f * (a.y + b.y), lo1, hi1);
    uint32_t z = quantize(0.5f * (a.z + b.z), lo2, hi2);
    codes[i] = (expand_bits(x) << 2) | (expand_bits(y) << 1) | expand_bits(z);
}

// Sorted leaves as unique 64-bit keys: code << 32 | proxy index.
struct LeafKeys {
    const uint32_t* __restrict__ code;
    const uint32_t* __restrict__ index;
    __device__ __forceinline__ uint64_t operator[](int i) const { return (uint64_t(code[i]) << 32) | index[i]; }
};

__device__ __forceinline__ int delta(const LeafKeys& k, int m, int i, int j) {
    if (j < 0 || j >= m) return -1;
    return __clzll(k[i] ^ k[j]);
}

// Karras 2012: internal node i spans a key range split at its highest differing bit.
__global__ void k_build(LeafKeys k, int m, uint32_t* left, uint32_t* right, uint32_t* parent,
                        uint32_t* leaf_body, uint32_t* refit_flag) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < m) leaf_body[i] = k.index[i];
    if (i >= m - 1) return;
    int d = (delta(k, m, i, i + 1) - delta(k, m, i, i - 1)) >= 0 ? 1 : -1;
    int dmin = delta(k, m, i, i - d);
    int lmax = 2;
    while (delta(k, m, i, i + lmax * d) > dmin) lmax *= 2;
    int l = 0;
    for (int t = lmax / 2; t >= 1; t /= 2)
        if (delta(k, m, i, i + (l + t) * d) > dmin) l += t;
    int j = i + l * d;
    int dnode = delta(k, m, i, j);
    int s = 0;
    int t = l;
    do {
        t = (t + 1) / 2;
        if (delta(k, m, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    int gamma = i + s * d + min(d, 0);
    int lo = min(i, j), hi = max(i, j);
    uint32_t lc = (lo == gamma) ? uint32_t(m - 1 + gamma) : uint32_t(gamma);
    uint32_t rc = (hi == gamma + 1) ? uint32_t(m - 1 + gamma + 1) : uint32_t(gamma + 1);
    left[i] = lc;
    right[i] = rc;
    refit_flag[i] = uint32_t(j) << 2;  // the other end of the node's leaves; low bits: children that arrived
    parent[lc] = uint32_t(i);
    parent[rc] = uint32_t(i);
}

// Leaf children are referenced as LEAF_REF | body index in the node records.
constexpr uint32_t LEAF_REF = 0x80000000u;

// Bottom-up refit: node boxes and the largest body index below each node; each internal
// node's record (4 float4: left child min | ref, left max | ref of right, right min | largest
// body index under left, right max | largest under right) is written by the thread that
// completes it, so a query reads one 64-byte record per node it visits.
// What bounds it: the climb, a fence, an atomic and two dependent loads a level. A node's number is one end of
// its leaves, so a node whose other end is in the same block of leaves has its whole subtree there: such
// nodes meet in shared memory, and only the climb from the blocks to the root goes through L2.
// There the records are written after the atomic, which has only the boxes to wait for, and the children's
// numbers are loaded with it. 16,384 / 60,000 / 131,072 leaves: 47 / 44 / 54 us with every node in L2,
// 37 / 38 / 47 us with blocks of 512 (256: 37 / 40 / 48, 128: 38 / 41 / 48), 30 / 31 / 38 us so.
constexpr int REFIT_TB = 512;

__global__ void __launch_bounds__(REFIT_TB) k_refit(int m, const uint32_t* __restrict__ leaf_body,
                                                    const uint32_t* __restrict__ parent, const uint32_t* __restrict__ left,
                                                    const uint32_t* __restrict__ right, uint32_t* refit_flag,
                                                    const float4* __restrict__ bmin, const float4* __restrict__ bmax,
                                                    float4* nmin, float4* nmax, float4* rec) {
    // The block's leaves, then its nodes; w of a minimum: the largest body index.
    __shared__ float4 s_min[2 * REFIT_TB], s_max[2 * REFIT_TB];
    __shared__ uint32_t s_left[REFIT_TB], s_right[REFIT_TB], s_parent[REFIT_TB], s_count[REFIT_TB];
    constexpr uint32_t ELSEWHERE = 1u << 31;  // in s_count: a node that other blocks' leaves belong to
    const uint32_t base = blockIdx.x * REFIT_TB, x = threadIdx.x, t = base + x, leaf0 = uint32_t(m - 1);
    uint32_t cur = 0, me = leaf0 + t;
    float4 lo{}, hi{};
    if (t < leaf0) {
        s_left[x] = left[t];
        s_right[x] = right[t];
        s_parent[x] = t ? parent[t] : 0u;
        s_count[x] = (refit_flag[t] >> 2) / REFIT_TB == blockIdx.x ? 0u : ELSEWHERE;
    }
    if (t < uint32_t(m)) {
        const uint32_t body = leaf_body[t];
        lo = bmin[body];
        hi = bmax[body];
        lo.w = __uint_as_float(body);
        s_min[x] = lo;
        s_max[x] = hi;
        if (m > 1) cur = parent[me];
    }
    __syncthreads();
    if (t >= uint32_t(m) || m == 1) return;
    constexpr uint32_t NONE = 0xffffffffu;
    uint32_t rec_of = NONE;  // a node whose record (q0 .. q3) is not written yet
    float4 q0{}, q1{}, q2{}, q3{};
    auto slot = [&](uint32_t node) { return node >= leaf0 ? node - leaf0 - base : REFIT_TB + node - base; };
    for (int guard = 0; guard < 128; ++guard) {
        const bool here = cur - base < uint32_t(REFIT_TB) && !(s_count[cur - base] & ELSEWHERE);
        uint32_t l, r, up;
        float4 a0, a1, b0, b1;
        if (here) {
            __threadfence_block();
            if (atomicAdd(&s_count[cur - base], 1u) == 0u) return;  // first child to arrive stops
            __threadfence_block();
            l = s_left[cur - base];
            r = s_right[cur - base];
            up = s_parent[cur - base];
            a0 = s_min[slot(l)]; a1 = s_max[slot(l)]; b0 = s_min[slot(r)]; b1 = s_max[slot(r)];
        } else {
            nmin[me] = lo;
            nmax[me] = hi;
            l = left[cur];  // on their way with the atomic
            r = right[cur];
            up = parent[cur];
            uint32_t arrived;
            asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(arrived) : "l"(refit_flag + cur) : "memory");
            if (rec_of != NONE) {  // the last node's record: nobody waits for it
                float4* rc = rec + size_t(rec_of) * 4;
                rc[0] = q0; rc[1] = q1; rc[2] = q2; rc[3] = q3;
                rec_of = NONE;
            }
            if ((arrived & 3u) == 0u) return;
            a0 = __ldcg(&nmin[l]); a1 = __ldcg(&nmax[l]); b0 = __ldcg(&nmin[r]); b1 = __ldcg(&nmax[r]);
        }
        const uint32_t il = __float_as_uint(a0.w), ir = __float_as_uint(b0.w);
        lo = make_float4(fminf(a0.x, b0.x), fminf(a0.y, b0.y), fminf(a0.z, b0.z), __uint_as_float(il > ir ? il : ir));
        hi = make_float4(fmaxf(a1.x, b1.x), fmaxf(a1.y, b1.y), fmaxf(a1.z, b1.z), 0.f);
        const uint32_t lref = l >= leaf0 ? (LEAF_REF | il) : l;
        const uint32_t rref = r >= leaf0 ? (LEAF_REF | ir) : r;
        q0 = make_float4(a0.x, a0.y, a0.z, __uint_as_float(lref));
        q1 = make_float4(a1.x, a1.y, a1.z, __uint_as_float(rref));
        q2 = make_float4(b0.x, b0.y, b0.z, __uint_as_float(il));
        q3 = make_float4(b1.x, b1.y, b1.z, __uint_as_float(ir));
        rec_of = cur;
        if (here || cur == 0) {
            float4* rc = rec + size_t(cur) * 4;
            rc[0] = q0; rc[1] = q1; rc[2] = q2; rc[3] = q3;
            rec_of = NONE;
        }
        if (cur == 0) return;
        me = cur;
        if (here) {
            s_min[REFIT_TB + cur - base] = lo;
            s_max[REFIT_TB + cur - base] = hi;
        }
        cur = up;
    }
}

// Partners j > i of bounded proxy i, in one of three modes:
//   Q_COUNT  counts[i] only;
//   Q_WRITE  the segment at offsets[i] (counts[i] from an earlier pass), sorted;
//   Q_STASH  counts[i], and when it is at most STASH_SLOTS the sorted partners in
//            stash slot a of Morton position t (stash[a * m + t], so a warp's
//            writes of one slot are contiguous); a proxy with more partners is
//            appended to `list` (its length in list_len) for a Q_WRITE pass.
// Q_COUNT and Q_WRITE take the proxies from `list` when it is given (t < list_len).
constexpr int Q_COUNT = 0, Q_WRITE = 1, Q_STASH = 2;
constexpr uint32_t STASH_SLOTS = 32;

template <int MODE>
__global__ void k_query(int m, uint32_t n, const uint32_t* __restrict__ is_unb, const float4* __restrict__ bmin,
                        const float4* __restrict__ bmax, const float4* __restrict__ rec,
                        const uint32_t* __restrict__ leaf_body, const uint32_t* __restrict__ unb, uint32_t nunb,
                        uint32_t* counts, const uint32_t* __restrict__ offsets, uint64_t* out, uint32_t* status,
                        uint32_t* list, uint32_t* list_len, uint32_t* stash) {
    constexpr bool WRITE = MODE == Q_WRITE;
    constexpr bool KEEP = MODE != Q_COUNT;
    // Threads take the bounded proxies in Morton (leaf) order, so a warp's
    // queries are neighbours in space and walk much the same part of the tree.
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t i;
    if (MODE != Q_STASH && list) {
        if (t >= *list_len) return;
        i = list[t];
    } else {
        if (t >= uint32_t(m)) return;
        i = leaf_body[t];
    }
    float4 qmin = bmin[i], qmax = bmax[i];
    uint32_t cnt = 0;
    uint32_t local[LOCAL_SORT];
    uint64_t base = 0;
    uint32_t expected = 0;
    if (WRITE) {
        base = offsets[i];
        expected = counts[i];
    }
    auto emit = [&](uint32_t j) {
        if (MODE == Q_STASH) {
            if (cnt < STASH_SLOTS) local[cnt] = j;
        } else if (WRITE) {
            if (expected <= LOCAL_SORT) {
                if (cnt < LOCAL_SORT) local[cnt] = j;
            } else if (cnt < expected) {
                out[base + cnt] = (uint64_t(i) << 32) | j;
            }
        }
        ++cnt;
    };
    if (m == 1) {  // the root is the single leaf
        const uint32_t j = leaf_body[0];
        if (j > i && overlaps(qmin, qmax, bmin[j], bmax[j])) emit(j);
    } else if (m > 1) {
        // Subtrees whose largest body index is at most i hold no partner j > i and are skipped.
        uint32_t stack[STACK_DEPTH];
        int sp = 0;
        stack[sp++] = 0u;
        while (sp > 0) {
            const float4* r = rec + size_t(stack[--sp]) * 4;
            const float4 a = r[0], b = r[1], c = r[2], d = r[3];
            const uint32_t ref[2] = {__float_as_uint(a.w), __float_as_uint(b.w)};
            const bool hit[2] = {__float_as_uint(c.w) > i && overlaps(qmin, qmax, a, b),
                                 __float_as_uint(d.w) > i && overlaps(qmin, qmax, c, d)};
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                if (!hit[k]) continue;
                if (ref[k] & LEAF_REF) {
                    emit(ref[k] & ~LEAF_REF);
                } else if (sp < STACK_DEPTH) {
                    stack[sp++] = ref[k];
                } else {
                    atomicOr(status, ST_TRAVERSAL_STACK);
                }
            }
        }
    }
    for (uint32_t u = 0; u < nunb; ++u) {
        uint32_t h = unb[u];
        if (h > i && overlaps(qmin, qmax, bmin[h], bmax[h])) emit(h);
    }
    if (!KEEP) {
        counts[i] = cnt;
        return;
    }
    if (MODE == Q_STASH) {
        counts[i] = cnt;
        if (cnt > STASH_SLOTS) {
            list[atomicAdd(list_len, 1u)] = i;
            return;
        }
    }
    if (MODE == Q_STASH || expected <= LOCAL_SORT) {
        uint32_t c = cnt < LOCAL_SORT ? cnt : LOCAL_SORT;
        for (uint32_t a = 1; a < c; ++a) {
            uint32_t v = local[a];
            uint32_t b = a;
            while (b > 0 && local[b - 1] > v) { local[b] = local[b - 1]; --b; }
            local[b] = v;
        }
        if (MODE == Q_STASH)
            for (uint32_t a = 0; a < c; ++a) stash[size_t(a) * uint32_t(m) + t] = local[a];
        else
            for (uint32_t a = 0; a < c; ++a) out[base + a] = (uint64_t(i) << 32) | local[a];
    } else {
        uint32_t c = cnt < expected ? cnt : expected;
        for (uint32_t a = 1; a < c; ++a) {
            uint64_t v = out[base + a];
            uint32_t b = a;
            while (b > 0 && out[base + b - 1] > v) { out[base + b] = out[base + b - 1]; --b; }
            out[base + b] = v;
        }
    }
}

// The partners j > h of each unbounded proxy h, tile by tile of proxies: their number (counts[h])
// and, for the pass that writes them, how many lie before each tile (before[u tiles + tile]).
constexpr uint32_t UNB_ROUNDS = 4;
constexpr uint32_t UNB_TILES_MAX = 65536;  // tiles a launch: many unbounded proxies take several launches

__device__ __forceinline__ uint32_t unb_ranks(uint32_t h, uint32_t base, uint32_t n, const float4* __restrict__ bmin,
                                              const float4* __restrict__ bmax, bool (&flag)[UNB_ROUNDS],
                                              uint32_t (&rank)[UNB_ROUNDS]) {
    const float4 hmin = bmin[h], hmax = bmax[h];
#pragma unroll
    for (uint32_t r = 0; r < UNB_ROUNDS; ++r) {
        const uint32_t j = base + r * TILE_TB + threadIdx.x;
        flag[r] = j > h && j < n && overlaps(hmin, hmax, bmin[j], bmax[j]);
    }
    return tile_ranks(flag, rank);
}

__global__ void __launch_bounds__(TILE_TB) k_unb_tiles(uint32_t n, uint32_t tiles, const uint32_t* __restrict__ unb,
                                                       const float4* __restrict__ bmin, const float4* __restrict__ bmax,
                                                       uint32_t* before, uint32_t* counts, TileScan ts) {
    const uint32_t tile = tile_take(ts), u = tile / tiles, t = tile % tiles;
    bool flag[UNB_ROUNDS];
    uint32_t rank[UNB_ROUNDS];
    const uint32_t total = unb_ranks(unb[u], t * (TILE_TB * UNB_ROUNDS), n, bmin, bmax, flag, rank);
    const uint32_t at = tile_prefix(ts, tile, u * tiles, total);
    if (threadIdx.x == 0) {
        before[tile] = at;
        if (t + 1u == tiles) counts[unb[u]] = at + total;
    }
}

// Where each proxy's segment starts, the number of pairs and of overflowing proxies (to the host).
__global__ void __launch_bounds__(TILE_TB) k_segments(uint32_t n, const uint32_t* __restrict__ counts, uint32_t* offsets,
                                                      const uint32_t* __restrict__ scalars, uint32_t* host, TileScan ts) {
    const uint32_t tile = tile_take(ts), base = tile * (TILE_TB * 4u);
    uint32_t v[4], before[4];
#pragma unroll
    for (uint32_t r = 0; r < 4; ++r) {
        const uint32_t i = base + r * TILE_TB + threadIdx.x;
        v[r] = i < n ? counts[i] : 0u;
    }
    const uint32_t total = tile_sums(v, before);
    const uint32_t at = tile_prefix(ts, tile, 0u, total);
#pragma unroll
    for (uint32_t r = 0; r < 4; ++r) {
        const uint32_t i = base + r * TILE_TB + threadIdx.x;
        if (i < n) offsets[i] = at + before[r];
    }
    if (base + TILE_TB * 4u >= n && threadIdx.x == 0) {
        host[0] = at + total;
        host[1] = scalars[1];
    }
}

// The segments at their place: the first stash_blocks blocks the stashed ones (slot t belongs to proxy
// leaf_body[t]), the others a tile of an unbounded proxy's partners.
__global__ void __launch_bounds__(TILE_TB) k_write_pairs(int m, const uint32_t* __restrict__ leaf_body,
                                                         const uint32_t* __restrict__ counts,
                                                         const uint32_t* __restrict__ offsets,
                                                         const uint32_t* __restrict__ stash, uint64_t* out,
                                                         uint32_t stash_blocks, uint32_t n, uint32_t tiles,
                                                         const uint32_t* __restrict__ unb, const float4* __restrict__ bmin,
                                                         const float4* __restrict__ bmax,
                                                         const uint32_t* __restrict__ before) {
    if (blockIdx.x < stash_blocks) {
        const uint32_t t = blockIdx.x * TILE_TB + threadIdx.x;
        if (t >= uint32_t(m)) return;
        const uint32_t i = leaf_body[t];
        const uint32_t c = counts[i];
        if (c > STASH_SLOTS) return;
        const uint64_t base = offsets[i];
        for (uint32_t a = 0; a < c; ++a) out[base + a] = (uint64_t(i) << 32) | stash[size_t(a) * uint32_t(m) + t];
        return;
    }
    const uint32_t tile = blockIdx.x - stash_blocks, h = unb[tile / tiles], base = tile % tiles * (TILE_TB * UNB_ROUNDS);
    bool flag[UNB_ROUNDS];
    uint32_t rank[UNB_ROUNDS];
    unb_ranks(h, base, n, bmin, bmax, flag, rank);
    const uint64_t at = uint64_t(offsets[h]) + before[tile];
#pragma unroll
    for (uint32_t r = 0; r < UNB_ROUNDS; ++r)
        if (flag[r]) out[at + rank[r]] = (uint64_t(h) << 32) | (base + r * TILE_TB + threadIdx.x);
}

// ---------------------------------------------------------------- all pairs (few proxies)
// Bit j of row i: i < j and their boxes overlap. A lane holds proxy j and a warp tests 32 of them against
// each row with one vote, so the partners come out in order and unbounded proxies are like any other. A
// block tests 256 proxies against 128 rows staged in shared memory.
constexpr uint32_t AP_ROWS = 128;

__global__ void __launch_bounds__(256) k_all_pairs(uint32_t n, uint32_t words, const float4* __restrict__ bmin,
                                                   const float4* __restrict__ bmax, uint32_t* masks) {
    __shared__ float4 s_min[AP_ROWS], s_max[AP_ROWS];
    const uint32_t i0 = blockIdx.y * AP_ROWS, j = blockIdx.x * 256u + threadIdx.x, lane = threadIdx.x & 31u;
    if (i0 >= (blockIdx.x + 1u) * 256u) return;  // no j of the block lies above a row
    if (threadIdx.x < AP_ROWS && i0 + threadIdx.x < n) {
        s_min[threadIdx.x] = bmin[i0 + threadIdx.x];
        s_max[threadIdx.x] = bmax[i0 + threadIdx.x];
    }
    float4 jmin = make_float4(0.f, 0.f, 0.f, 0.f), jmax = jmin;
    if (j < n) { jmin = bmin[j]; jmax = bmax[j]; }
    __syncthreads();
    const uint32_t word = j >> 5;
    if (word >= words) return;
    for (uint32_t r0 = 0; r0 < AP_ROWS; r0 += 32u) {
        uint32_t row = 0;
#pragma unroll 8
        for (uint32_t r = 0; r < 32u; ++r) {
            const uint32_t i = i0 + r0 + r;
            const uint32_t b = __ballot_sync(0xffffffffu, (j > i) & (j < n) &
                                                              overlaps_all(s_min[r0 + r], s_max[r0 + r], jmin, jmax));
            if (lane == r) row = b;
        }
        const uint32_t i = i0 + r0 + lane;
        if (i < n && word >= i >> 5) masks[size_t(i) * words + word] = row;
    }
}

// The rows' pairs, one warp a row and 16 rows a tile (many blocks: 1,000 proxies took 12 us with 64), as
// far as `out` holds them; the total to the host.
constexpr uint32_t AP_TILE = 16;

__global__ void __launch_bounds__(TILE_TB) k_all_pairs_rows(uint32_t n, uint32_t words, const uint32_t* __restrict__ masks,
                                                            uint64_t* out, uint64_t cap, uint32_t* host, TileScan ts) {
    __shared__ uint32_t s_cnt[AP_TILE], s_total;
    const uint32_t tile = tile_take(ts), lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    constexpr uint32_t PER = AP_TILE / (TILE_TB / 32);
#pragma unroll
    for (uint32_t r = 0; r < PER; ++r) {
        const uint32_t k = warp * PER + r, i = tile * AP_TILE + k;
        uint32_t c = 0;
        if (i < n)
            for (uint32_t w = (i >> 5) + lane; w < words; w += 32u) c += __popc(masks[size_t(i) * words + w]);
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0) s_cnt[k] = c;
    }
    __syncthreads();
    if (warp == 0) {
        const uint32_t a = lane < AP_TILE ? s_cnt[lane] : 0u;
        uint32_t x = a;
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31u) s_total = x;
        if (lane < AP_TILE) s_cnt[lane] = x - a;
    }
    __syncthreads();
    const uint32_t total = s_total, at = tile_prefix(ts, tile, 0u, total);
    if ((tile + 1u) * AP_TILE >= n && threadIdx.x == 0) {
        host[0] = at + total;
        host[1] = 0u;
    }
    if (uint64_t(at) + total > cap) return;  // the host makes room and comes again
#pragma unroll
    for (uint32_t r = 0; r < PER; ++r) {
        const uint32_t k = warp * PER + r, i = tile * AP_TILE + k;
        if (i >= n) break;
        uint64_t pos = uint64_t(at) + s_cnt[k];
        for (uint32_t w0 = i >> 5; w0 < words; w0 += 32u) {  // uniform across the warp
            const uint32_t w = w0 + lane;
            uint32_t m = w < words ? masks[size_t(i) * words + w] : 0u;
            const uint32_t c = __popc(m);
            uint32_t x = c;
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            uint64_t q = pos + x - c;
            for (; m; m &= m - 1u) out[q++] = (uint64_t(i) << 32) | (w * 32u + uint32_t(__ffs(int(m)) - 1));
            pos += __shfl_sync(0xffffffffu, x, 31);
        }
    }
}

// Unbounded proxy h: flags[j] = (j > h && overlap(h, j)) over all proxies.
__global__ void k_unb_flags(uint32_t h, uint32_t n, const float4* __restrict__ bmin, const float4* __restrict__ bmax,
                            uint32_t* flags) {
    uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    flags[j] = (j > h && overlaps(bmin[h], bmax[h], bmin[j], bmax[j])) ? 1u : 0u;
}

__global__ void k_unb_count(uint32_t h, uint32_t n, const uint32_t* __restrict__ flags, const uint32_t* __restrict__ scan,
                            uint32_t* counts) {
    if (blockIdx.x == 0 && threadIdx.x == 0) counts[h] = n ? scan[n - 1] + flags[n - 1] : 0u;
}

__global__ void k_unb_write(uint32_t h, uint32_t n, const uint32_t* __restrict__ flags, const uint32_t* __restrict__ scan,
                            const uint32_t* __restrict__ offsets, uint64_t* out) {
    uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n || !flags[j]) return;
    out[uint64_t(offsets[h]) + scan[j]] = (uint64_t(h) << 32) | j;
}

__global__ void k_total(uint32_t n, const uint32_t* __restrict__ counts, const uint32_t* __restrict__ offsets,
                        uint32_t* scalars) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        uint64_t t = n ? uint64_t(offsets[n - 1]) + counts[n - 1] : 0;
        scalars[0] = uint32_t(t > 0xffffffffull ? 0xffffffffull : t);
    }
}

__global__ void k_clear_u32(uint32_t n, uint32_t* a) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = 0;
}

__global__ void k_set_unbounded(const uint32_t* __restrict__ unb, uint32_t nunb, uint32_t* is_unb) {
    uint32_t u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u < nunb) is_unb[unb[u]] = 1;
}

// Batched worlds: world k owns proxies [off[k], off[k + 1]) and pairs only form inside a world.
//
// Bit j of row i of each world's masks (i < j, in the world's own numbers): their boxes overlap; counts[i]
// the row's bits. One CTA a world, a lane a proxy j, a vote per 32 tests (k_all_pairs, world by world). Rows
// [r0, r1) of the batch, which lie in worlds [w0, w1) and start at a multiple of 128 in theirs; without masks
// they are only counted.
// A thread per proxy that walked the others one by one and kept what it found took 91 us for 4,096
// worlds of 8 to 256 bodies and 79 us for 96 of them (a ground plane's 255 partners, one store after the
// other); this takes 41 and 12.
constexpr uint32_t WM_TILE = 128;

__global__ void __launch_bounds__(WM_TILE) k_world_masks(const float4* __restrict__ bmin, const float4* __restrict__ bmax,
                                                         const uint32_t* __restrict__ off, uint32_t w0, uint32_t w1,
                                                         uint32_t r0, uint32_t r1, const uint64_t* __restrict__ mask_off,
                                                         uint64_t mask_base, uint32_t* masks, uint32_t* counts) {
    __shared__ float4 s_min[WM_TILE], s_max[WM_TILE];
    __shared__ uint32_t s_cnt[WM_TILE];
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t w = w0 + blockIdx.x; w < w1; w += gridDim.x) {
        const uint32_t lo = off[w], nb = off[w + 1] - lo, words = (nb + 31u) / 32u;
        const uint32_t to = min(r1 - lo, nb);
        const uint64_t m = mask_off[w] - mask_base;  // (may be below 0 for rows that are not asked for)
        for (uint32_t i0 = r0 > lo ? r0 - lo : 0u; i0 < to; i0 += WM_TILE) {
            __syncthreads();  // the tile before is done with
            if (i0 + threadIdx.x < nb) {
                s_min[threadIdx.x] = bmin[lo + i0 + threadIdx.x];
                s_max[threadIdx.x] = bmax[lo + i0 + threadIdx.x];
            }
            s_cnt[threadIdx.x] = 0u;
            __syncthreads();
            const uint32_t rows = min(WM_TILE, to - i0);
            for (uint32_t j0 = i0; j0 < nb; j0 += WM_TILE) {
                const uint32_t j = j0 + threadIdx.x, word = j >> 5;
                if (word >= words) continue;  // uniform across the warp
                float4 jmin = make_float4(0.f, 0.f, 0.f, 0.f), jmax = jmin;
                if (j < nb) { jmin = bmin[lo + j]; jmax = bmax[lo + j]; }
                for (uint32_t q0 = 0; q0 < rows; q0 += 32u) {
                    if (word < (i0 + q0) >> 5) continue;  // no j of the word lies above these rows
                    uint32_t row = 0;
#pragma unroll 8
                    for (uint32_t q = 0; q < 32u; ++q) {
                        const uint32_t b = __ballot_sync(0xffffffffu, (j > i0 + q0 + q) & (j < nb) &
                                                                          overlaps_all(s_min[q0 + q], s_max[q0 + q], jmin, jmax));
                        if (lane == q) row = b;
                    }
                    if (q0 + lane < rows) {
                        if (masks) masks[m + uint64_t(i0 + q0 + lane) * words + word] = row;
                        if (row) atomicAdd(&s_cnt[q0 + lane], __popc(row));
                    }
                }
            }
            __syncthreads();
            if (threadIdx.x < rows) counts[lo + i0 + threadIdx.x] = s_cnt[threadIdx.x];
        }
    }
}

// The rows' pairs: a thread a row, but rows of many partners (a ground plane's) by the whole warp.
__global__ void __launch_bounds__(256) k_world_rows(uint32_t r0, uint32_t r1, const uint32_t* __restrict__ off,
                                                    const uint32_t* __restrict__ world_of,
                                                    const uint64_t* __restrict__ mask_off, uint64_t mask_base,
                                                    const uint32_t* __restrict__ masks, const uint32_t* __restrict__ counts,
                                                    const uint32_t* __restrict__ offsets, uint64_t* out) {
    const uint32_t i = r0 + blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u;
    uint32_t cnt = 0, lo = 0, words = 0;
    uint64_t pos = 0, first = 0;
    if (i < r1) {
        cnt = counts[i];
        if (cnt) {
            const uint32_t w = world_of[i];
            lo = off[w];
            words = (off[w + 1] - lo + 31u) / 32u;
            first = mask_off[w] - mask_base + uint64_t(i - lo) * words;
            pos = offsets[i];
        }
    }
    const bool wide = cnt > 48u;
    if (cnt && !wide) {
        for (uint32_t w = (i - lo) >> 5; w < words && cnt; ++w)
            for (uint32_t m = masks[first + w]; m; m &= m - 1u, --cnt)
                out[pos++] = (uint64_t(i) << 32) | (lo + w * 32u + uint32_t(__ffs(int(m)) - 1));
    }
    for (uint32_t todo = __ballot_sync(0xffffffffu, wide); todo; todo &= todo - 1u) {
        const int src = __ffs(int(todo)) - 1;
        const uint32_t ri = __shfl_sync(0xffffffffu, i, src), rlo = __shfl_sync(0xffffffffu, lo, src);
        const uint32_t rwords = __shfl_sync(0xffffffffu, words, src);
        const uint64_t rfirst = __shfl_sync(0xffffffffu, static_cast<unsigned long long>(first), src);
        uint64_t rpos = __shfl_sync(0xffffffffu, static_cast<unsigned long long>(pos), src);
        for (uint32_t w = (ri - rlo) >> 5; w < rwords; ++w) {
            const uint32_t m = masks[rfirst + w];
            if ((m >> lane) & 1u)
                out[rpos + __popc(m & ((1u << lane) - 1u))] = (uint64_t(ri) << 32) | (rlo + w * 32u + lane);
            rpos += __popc(m);
        }
    }
}

}  // namespace

uint64_t Broadphase::run_worlds(const float4* aabb_min, const float4* aabb_max, uint32_t n,
                                const std::vector<uint32_t>& world_off_host, const uint32_t* world_off,
                                const uint32_t* world_of, DevBuf<uint64_t>& out, uint32_t* status_dev, cudaStream_t s) {
    const uint32_t n_worlds = uint32_t(world_off_host.size() - 1);
    if (n == 0 || n_worlds == 0) return 0;
    counts.reserve(n);
    offsets.reserve(n);
    if (mask_worlds != n_worlds || mask_n != n) {  // worlds were added
        std::vector<uint64_t> first(n_worlds);
        mask_words = 0;
        for (uint32_t k = 0; k < n_worlds; ++k) {
            const uint64_t nb = world_off_host[k + 1] - world_off_host[k];
            first[k] = mask_words;
            mask_words += nb * ((nb + 31u) / 32u);
        }
        mask_off.reserve(n_worlds);
        check_cuda(cudaMemcpyAsync(mask_off.p, first.data(), n_worlds * sizeof(uint64_t), cudaMemcpyHostToDevice, s), "h2d");
        check_cuda(cudaStreamSynchronize(s), "sync");
        mask_worlds = n_worlds;
        mask_n = n;
    }
    auto make = [&](uint32_t w0, uint32_t w1, uint32_t r0, uint32_t r1, uint64_t base, uint32_t* to) {
        k_world_masks<<<std::min<uint32_t>(w1 - w0, 148u * 32u), WM_TILE, 0, s>>>(aabb_min, aabb_max, world_off, w0, w1, r0, r1,
                                                                               mask_off.p, base, to, counts.p);
    };
    auto write = [&](uint32_t r0, uint32_t r1, uint64_t base) {
        k_world_rows<<<(r1 - r0 + 255) / 256, 256, 0, s>>>(r0, r1, world_off, world_of, mask_off.p, base, masks.p, counts.p,
                                                           offsets.p, out.p);
    };
    const bool whole = mask_words <= WORLD_MASK_WORDS_MAX;
    if (whole) masks.reserve(mask_words);
    make(0, n_worlds, 0, n, 0, whole ? masks.p : nullptr);
    const uint32_t tiles = tile_count<4>(n);
    k_segments<<<tiles, TILE_TB, 0, s>>>(n, counts.p, offsets.p, scalars.p, host_scalars, scan.begin(tiles, status_dev, s));
    check_cuda(cudaStreamSynchronize(s), "broadphase sync");
    const uint64_t total = host_scalars[0];
    out.reserve(total + 1);
    if (!total) return 0;
    if (whole) {
        write(0, n, 0);
        return total;
    }
    // Too many masks: counted above, the tests are made again for as many rows at a time as the masks hold
    // (whole worlds, or a multiple of 128 rows of one; 128 rows at least).
    uint32_t k = 0, row = 0;  // the first world and its row still to do
    uint64_t base = 0;        // their mask word
    while (k < n_worlds) {
        const uint32_t w0 = k, r0 = world_off_host[k] + row;
        uint64_t words = 0;
        for (; k < n_worlds; ++k, row = 0) {
            const uint32_t nb = world_off_host[k + 1] - world_off_host[k], per = (nb + 31u) / 32u;
            const uint64_t fit = per ? (WORLD_MASK_WORDS_MAX - std::min(words, WORLD_MASK_WORDS_MAX)) / per : nb;
            uint32_t take = nb - row;
            if (take > fit) take = std::max(uint32_t(fit) / WM_TILE * WM_TILE, words ? 0u : std::min(take, WM_TILE));
            words += uint64_t(take) * per;
            row += take;
            if (row < nb) break;
        }
        const uint32_t r1 = k < n_worlds ? world_off_host[k] + row : n;
        masks.reserve(words);
        make(w0, std::min(k + 1u, n_worlds), r0, r1, base, masks.p);
        write(r0, r1, base);
        base += words;
    }
    return total;
}

Broadphase::Broadphase() {
    scalars.reserve(2);
    bounds.reserve(12);
    check_cuda(cudaMallocHost(&host_scalars, 4 * sizeof(uint32_t)), "cudaMallocHost");
}

Broadphase::~Broadphase() {
    if (host_scalars) cudaFreeHost(host_scalars);
}

uint64_t Broadphase::run(const float4* aabb_min, const float4* aabb_max, uint32_t n,
                         const std::vector<uint32_t>& unbounded_host, DevBuf<uint64_t>& out, bool all_pairs,
                         const int* centres, uint32_t* status_dev, cudaStream_t s) {
    if (n == 0) return 0;
    if (all_pairs) {
        tree_m = 0;
        nunb = 0;
        const uint32_t words = (n + 31u) / 32u, tiles = (n + AP_TILE - 1) / AP_TILE;
        masks.reserve(size_t(n) * words);
        k_all_pairs<<<dim3((n + 255u) / 256u, (n + AP_ROWS - 1) / AP_ROWS), 256, 0, s>>>(n, words, aabb_min, aabb_max,
                                                                                        masks.p);
        // Written at once when the last step's array has room, as it does but for growth.
        for (;;) {
            const uint64_t cap = out.cap;
            k_all_pairs_rows<<<tiles, TILE_TB, 0, s>>>(n, words, masks.p, out.p, cap, host_scalars,
                                                       scan.begin(tiles, status_dev, s));
            check_cuda(cudaStreamSynchronize(s), "broadphase sync");
            const uint64_t total = host_scalars[0];
            if (total <= cap) return total;
            out.reserve(total + 1);
        }
    }
    const uint32_t nunb = uint32_t(unbounded_host.size());
    const int m = int(n - nunb);
    tree_m = m;
    this->nunb = nunb;
    const int TB = 256;
    const uint32_t grid = (n + TB - 1) / TB;
    keys.reserve(n);
    keys_alt.reserve(n);
    leaf_body.reserve(n);
    parent.reserve(2 * size_t(n));
    left.reserve(n);
    right.reserve(n);
    refit_flag.reserve(n);
    node_min.reserve(2 * size_t(n));
    node_max.reserve(2 * size_t(n));
    node_rec.reserve(4 * size_t(n));
    counts.reserve(n);
    offsets.reserve(n);
    is_unb.reserve(n);
    unbounded.reserve(nunb + 1);
    if (unb_n != n || unb_listed != unbounded_host) {  // the list changes only when bodies are added
        unb_n = 0;
        if (nunb) check_cuda(cudaMemcpyAsync(unbounded.p, unbounded_host.data(), nunb * sizeof(uint32_t),
                                             cudaMemcpyHostToDevice, s), "upload unbounded");
        k_clear_u32<<<grid, TB, 0, s>>>(n, is_unb.p);
        if (nunb) k_set_unbounded<<<(nunb + TB - 1) / TB, TB, 0, s>>>(unbounded.p, nunb, is_unb.p);
        unb_listed = unbounded_host;
        unb_n = n;
    }
    if (!centres) {
        k_reset_bounds<<<1, 32, 0, s>>>(bounds.p);
        k_bounds<<<grid, TB, 0, s>>>(aabb_min, aabb_max, is_unb.p, n, bounds.p);
        centres = bounds.p;
    }
    // keys / keys_alt (n x 8 bytes each) hold the codes and indices and their sort buffers.
    uint32_t* codes = reinterpret_cast<uint32_t*>(keys.p);
    uint32_t* codes_alt = reinterpret_cast<uint32_t*>(keys_alt.p);
    k_keys<<<grid, TB, 0, s>>>(aabb_min, aabb_max, is_unb.p, n, centres, codes, codes + n, scalars.p + 1);

    size_t tmp_bytes = 0;
    cub::DoubleBuffer<uint32_t> dk(codes, codes_alt), dv(codes + n, codes_alt + n);
    check_cuda(cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, dk, dv, int(n), 0, 32, s), "sort size");
    cub_tmp.reserve(tmp_bytes);
    check_cuda(cub::DeviceRadixSort::SortPairs(cub_tmp.p, tmp_bytes, dk, dv, int(n), 0, 32, s), "sort");
    const LeafKeys sorted{dk.Current(), dv.Current()};

    if (m > 0) {
        k_build<<<(m + TB - 1) / TB, TB, 0, s>>>(sorted, m, left.p, right.p, parent.p, leaf_body.p, refit_flag.p);
        k_refit<<<(m + REFIT_TB - 1) / REFIT_TB, REFIT_TB, 0, s>>>(m, leaf_body.p, parent.p, left.p, right.p, refit_flag.p, aabb_min,
                                                 aabb_max, node_min.p, node_max.p, node_rec.p);
    }
    const uint32_t qgrid = m > 0 ? (uint32_t(m) + TB - 1) / TB : 1u;
    // One traversal per proxy: counts, plus the sorted partners of every proxy with at
    // most STASH_SLOTS of them; the rest are listed and walk the tree again below.
    stash.reserve(size_t(STASH_SLOTS) * uint32_t(m > 0 ? m : 1));
    overflow.reserve(uint32_t(m > 0 ? m : 1));
    k_query<Q_STASH><<<qgrid, TB, 0, s>>>(m, n, is_unb.p, aabb_min, aabb_max, node_rec.p, leaf_body.p, unbounded.p,
                                          nunb, counts.p, nullptr, nullptr, status_dev, overflow.p, scalars.p + 1,
                                          stash.p);
    const uint32_t utiles = tile_count<UNB_ROUNDS>(n), tiles = tile_count<4>(n);
    const uint32_t upart = std::max(UNB_TILES_MAX / utiles, 1u);  // unbounded proxies a launch
    unb_tiles.reserve(size_t(nunb) * utiles);
    for (uint32_t u = 0; u < nunb; u += upart) {
        const uint32_t blocks = std::min(upart, nunb - u) * utiles;
        k_unb_tiles<<<blocks, TILE_TB, 0, s>>>(n, utiles, unbounded.p + u, aabb_min, aabb_max,
                                               unb_tiles.p + size_t(u) * utiles, counts.p,
                                               scan.begin(blocks, status_dev, s));
    }
    k_segments<<<tiles, TILE_TB, 0, s>>>(n, counts.p, offsets.p, scalars.p, host_scalars, scan.begin(tiles, status_dev, s));
    check_cuda(cudaStreamSynchronize(s), "broadphase sync");
    uint64_t total = host_scalars[0];
    const uint32_t n_overflow = host_scalars[1];
    out.reserve(total + 1);
    if (total) {
        uint32_t sblocks = m > 0 ? (uint32_t(m) + TILE_TB - 1) / TILE_TB : 0u, u = 0;
        do {
            const uint32_t ublocks = std::min(upart, nunb - u) * utiles;
            if (sblocks + ublocks)
                k_write_pairs<<<sblocks + ublocks, TILE_TB, 0, s>>>(m, leaf_body.p, counts.p, offsets.p, stash.p, out.p,
                                                                    sblocks, n, utiles, unbounded.p + u, aabb_min, aabb_max,
                                                                    unb_tiles.p + size_t(u) * utiles);
            sblocks = 0;
            u += upart;
        } while (u < nunb);
        if (n_overflow)
            k_query<Q_WRITE><<<(n_overflow + TB - 1) / TB, TB, 0, s>>>(
                m, n, is_unb.p, aabb_min, aabb_max, node_rec.p, leaf_body.p, unbounded.p, nunb, counts.p, offsets.p,
                out.p, status_dev, overflow.p, scalars.p + 1, nullptr);
    }
    return total;
}

}  // namespace bgpu

// ---------------------------------------------------------------- allocation-free entry point
//
// For callers that cannot allocate device memory while they run: game and robotics
// loops with a fixed device-memory budget, code running inside another runtime
// that owns the allocator, or callers on a hard deadline that cannot afford a
// cudaMalloc / cudaFree round trip (both may synchronise the device). They pass
// device buffers for the input AABBs and the output pairs; every scratch array
// of the broad phase lives in one fixed file-scope device array instead.
//
// Limits: at most BGPU_NOALLOC_MAX_PROXIES proxies and BGPU_NOALLOC_MAX_UNBOUNDED
// unbounded proxies (extent >= 1e15, e.g. planes); larger inputs are rejected.
// The array is shared by every call in the process and keeps the last call's
// contents, so two calls that overlap on the GPU (different streams, or
// different host threads) race on it and must be serialised by the caller.
// Each GPU that loads the library holds the array until the process exits.
#include <mutex>
#include "../../include/bgpu.h"

namespace bgpu {
namespace {

constexpr size_t NOALLOC_SCRATCH_BYTES = size_t(24) << 20;
// Bytes per proxy of the arrays taken below (AABBs 32, sort keys 16, flags / scans / counts /
// offsets / tree links 36, parents 8, node boxes 64, node records 64),
// plus 256 B of alignment per array and room for CUB's sort / scan scratch (a few hundred KB
// at 65,536 keys; 4 MiB allowed). Each take() is also checked when the call runs.
constexpr size_t NOALLOC_PER_PROXY_BYTES = 220;
static_assert(NOALLOC_PER_PROXY_BYTES * BGPU_NOALLOC_MAX_PROXIES + 32 * 256 + (size_t(4) << 20) <= NOALLOC_SCRATCH_BYTES,
              "the allocation-free broad phase's scratch array is too small for its proxy limit");
static __device__ __align__(256) unsigned char g_bp_scratch[NOALLOC_SCRATCH_BYTES];

std::mutex g_bp_scratch_mutex;
constexpr int NOALLOC_MAX_DEVICES = 64;
unsigned char* g_bp_scratch_addr[NOALLOC_MAX_DEVICES] = {};

// Device address of the scratch array for the current device. In host code the
// array's name is only a stand-in, so the address comes from the runtime, once
// per device (the first call on a device does this lookup).
unsigned char* noalloc_scratch_address(int dev) {
    std::lock_guard<std::mutex> lock(g_bp_scratch_mutex);
    if (!g_bp_scratch_addr[dev]) {
        void* ptr = nullptr;
        check_cuda(cudaGetSymbolAddress(&ptr, g_bp_scratch), "cudaGetSymbolAddress(g_bp_scratch)");
        g_bp_scratch_addr[dev] = static_cast<unsigned char*>(ptr);
    }
    return g_bp_scratch_addr[dev];
}

struct Bump {
    unsigned char* base;
    size_t used, cap;
    template <class T>
    T* take(size_t n) {
        size_t off = (used + 255) & ~size_t(255);
        size_t bytes = n * sizeof(T);
        if (off + bytes > cap) return nullptr;
        used = off + bytes;
        return reinterpret_cast<T*>(base + off);
    }
};

__global__ void k_noalloc_unpack(const float* __restrict__ aabbs, uint32_t n, float4* mn, float4* mx,
                                 uint32_t* is_unb) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* a = aabbs + 6 * size_t(i);
    mn[i] = make_float4(a[0], a[1], a[2], 0.0f);
    mx[i] = make_float4(a[3], a[4], a[5], 0.0f);
    bool huge = !(a[3] - a[0] < 1e15f) || !(a[4] - a[1] < 1e15f) || !(a[5] - a[2] < 1e15f);
    is_unb[i] = huge ? 1u : 0u;
}

__global__ void k_unb_write_list(uint32_t n, const uint32_t* __restrict__ is_unb, const uint32_t* __restrict__ scan,
                                 uint32_t* list) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && is_unb[i]) list[scan[i]] = i;
}

// Keys (lo << 32 | hi) become (lo, hi) uint32 pairs in place.
__global__ void k_noalloc_keys_to_pairs(uint64_t* buf, uint64_t n) {
    uint64_t k = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k >= n) return;
    uint64_t key = buf[k];
    uint32_t* p = reinterpret_cast<uint32_t*>(buf + k);
    p[0] = uint32_t(key >> 32);
    p[1] = uint32_t(key & 0xffffffffu);
}

}  // namespace
}  // namespace bgpu

extern "C" bgpu_status bgpu_broadphase_pairs_noalloc(const float* aabbs_dev, uint32_t n, uint32_t* pairs_dev,
                                                     uint64_t cap, uint64_t* out_n, void* stream) {
    using namespace bgpu;
    if (out_n) *out_n = 0;
    if ((n && !aabbs_dev) || (cap && !pairs_dev) || (reinterpret_cast<uintptr_t>(pairs_dev) & 7u)) {
        set_last_error("allocation-free broad phase: NULL buffer or pairs buffer not 8-byte aligned");
        return BGPU_ERR_INVALID_ARGUMENT;
    }
    if (n > BGPU_NOALLOC_MAX_PROXIES) {
        set_last_error("allocation-free broad phase: more than BGPU_NOALLOC_MAX_PROXIES (65536) proxies");
        return BGPU_ERR_CAPACITY;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    try {
        int dev = 0;
        check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
        if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) {
            set_last_error("allocation-free broad phase: device ordinal out of range");
            return BGPU_ERR_CAPACITY;
        }
        if (n == 0) return BGPU_OK;
        Bump sb{noalloc_scratch_address(dev), 0, NOALLOC_SCRATCH_BYTES};
        float4* mn = sb.take<float4>(n);
        float4* mx = sb.take<float4>(n);
        uint64_t* keys = sb.take<uint64_t>(n);
        uint64_t* keys_alt = sb.take<uint64_t>(n);
        uint32_t* is_unb = sb.take<uint32_t>(n);
        uint32_t* leaf_body = sb.take<uint32_t>(n);
        uint32_t* parent = sb.take<uint32_t>(2 * size_t(n));
        uint32_t* left = sb.take<uint32_t>(n);
        uint32_t* right = sb.take<uint32_t>(n);
        uint32_t* refit_flag = sb.take<uint32_t>(n);
        uint32_t* counts = sb.take<uint32_t>(n);
        uint32_t* offsets = sb.take<uint32_t>(n);
        uint32_t* flags = sb.take<uint32_t>(n);
        uint32_t* scan = sb.take<uint32_t>(n);
        uint32_t* unb_list = sb.take<uint32_t>(BGPU_NOALLOC_MAX_UNBOUNDED + 1);
        float4* node_min = sb.take<float4>(2 * size_t(n));
        float4* node_max = sb.take<float4>(2 * size_t(n));
        float4* node_rec = sb.take<float4>(4 * size_t(n));
        int* bounds = sb.take<int>(8);
        uint32_t* scalars = sb.take<uint32_t>(8);
        const void* taken[] = {mn, mx, keys, keys_alt, is_unb, leaf_body, parent, left, right, refit_flag, counts,
                               offsets, flags, scan, unb_list, node_min, node_max, node_rec, bounds, scalars};
        for (const void* t : taken)
            if (!t) {
                set_last_error("allocation-free broad phase: scratch array too small");
                return BGPU_ERR_CAPACITY;
            }
        size_t sort_bytes = 0, scan_bytes = 0;
        uint32_t* codes = reinterpret_cast<uint32_t*>(keys);
        uint32_t* codes_alt = reinterpret_cast<uint32_t*>(keys_alt);
        cub::DoubleBuffer<uint32_t> dk(codes, codes_alt), dv(codes + n, codes_alt + n);
        check_cuda(cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, dk, dv, int(n), 0, 32, s), "sort size");
        check_cuda(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, counts, offsets, int(n), s), "scan size");
        size_t tmp_bytes = std::max(sort_bytes, scan_bytes);
        unsigned char* tmp = sb.take<unsigned char>(tmp_bytes);
        if (!tmp) {
            set_last_error("allocation-free broad phase: scratch array too small");
            return BGPU_ERR_CAPACITY;
        }
        const int TB = 256;
        const uint32_t grid = (n + TB - 1) / TB;
        // Nothing below relies on the previous call's contents; the status word and the
        // counters are cleared here, every other array is fully rewritten before it is read.
        check_cuda(cudaMemsetAsync(scalars, 0, 8 * sizeof(uint32_t), s), "memset");
        k_noalloc_unpack<<<grid, TB, 0, s>>>(aabbs_dev, n, mn, mx, is_unb);
        // Unbounded proxies, listed in index order (few by contract).
        check_cuda(cub::DeviceScan::ExclusiveSum(tmp, scan_bytes, is_unb, scan, int(n), s), "scan");
        uint32_t host_scan_last[2] = {0, 0};
        check_cuda(cudaMemcpyAsync(&host_scan_last[0], scan + (n - 1), 4, cudaMemcpyDeviceToHost, s), "d2h");
        check_cuda(cudaMemcpyAsync(&host_scan_last[1], is_unb + (n - 1), 4, cudaMemcpyDeviceToHost, s), "d2h");
        check_cuda(cudaStreamSynchronize(s), "sync");
        uint32_t nunb = host_scan_last[0] + host_scan_last[1];
        if (nunb > BGPU_NOALLOC_MAX_UNBOUNDED) {
            set_last_error("allocation-free broad phase: more than BGPU_NOALLOC_MAX_UNBOUNDED (16) unbounded proxies");
            return BGPU_ERR_CAPACITY;
        }
        uint32_t unb_host[BGPU_NOALLOC_MAX_UNBOUNDED + 1];
        if (nunb) {
            k_unb_write_list<<<grid, TB, 0, s>>>(n, is_unb, scan, unb_list);
            check_cuda(cudaMemcpyAsync(unb_host, unb_list, nunb * 4, cudaMemcpyDeviceToHost, s), "d2h");
        }
        const int m = int(n - nunb);
        k_reset_bounds<<<1, 32, 0, s>>>(bounds);
        k_bounds<<<grid, TB, 0, s>>>(mn, mx, is_unb, n, bounds);
        k_keys<<<grid, TB, 0, s>>>(mn, mx, is_unb, n, bounds, codes, codes + n, nullptr);
        check_cuda(cub::DeviceRadixSort::SortPairs(tmp, sort_bytes, dk, dv, int(n), 0, 32, s), "sort");
        const LeafKeys sorted{dk.Current(), dv.Current()};
        if (m > 0) {
            k_build<<<(m + TB - 1) / TB, TB, 0, s>>>(sorted, m, left, right, parent, leaf_body, refit_flag);
            k_refit<<<(m + REFIT_TB - 1) / REFIT_TB, REFIT_TB, 0, s>>>(m, leaf_body, parent, left, right, refit_flag, mn, mx, node_min,
                                                     node_max, node_rec);
        }
        uint32_t* status = scalars + 1;
        const uint32_t qgrid = m > 0 ? (uint32_t(m) + TB - 1) / TB : 1u;
        k_query<Q_COUNT><<<qgrid, TB, 0, s>>>(m, n, is_unb, mn, mx, node_rec, leaf_body, unb_list, nunb, counts,
                                              nullptr, nullptr, status, nullptr, nullptr, nullptr);
        uint32_t* unb_scan = dk.Alternate();  // free after the build
        check_cuda(cudaStreamSynchronize(s), "sync");
        for (uint32_t u = 0; u < nunb; ++u) {
            uint32_t h = unb_host[u];
            k_unb_flags<<<grid, TB, 0, s>>>(h, n, mn, mx, flags);
            check_cuda(cub::DeviceScan::ExclusiveSum(tmp, scan_bytes, flags, unb_scan, int(n), s), "scan");
            k_unb_count<<<1, 1, 0, s>>>(h, n, flags, unb_scan, counts);
        }
        check_cuda(cub::DeviceScan::ExclusiveSum(tmp, scan_bytes, counts, offsets, int(n), s), "scan");
        k_total<<<1, 1, 0, s>>>(n, counts, offsets, scalars);
        uint32_t host_scalars[2] = {0, 0};
        check_cuda(cudaMemcpyAsync(host_scalars, scalars, 2 * sizeof(uint32_t), cudaMemcpyDeviceToHost, s), "d2h");
        check_cuda(cudaStreamSynchronize(s), "sync");
        if (host_scalars[1]) {  // the count walk overflowed its stack: the total is not a pair count
            set_last_error("allocation-free broad phase: traversal stack overflow");
            return BGPU_ERR_DEVICE_STATUS;
        }
        uint64_t total = host_scalars[0];
        if (out_n) *out_n = total;
        if (total > cap) {
            set_last_error("allocation-free broad phase: output capacity too small (out_n holds the pair count)");
            return BGPU_ERR_CAPACITY;
        }
        uint64_t* out = reinterpret_cast<uint64_t*>(pairs_dev);
        if (total) {
            k_query<Q_WRITE><<<qgrid, TB, 0, s>>>(m, n, is_unb, mn, mx, node_rec, leaf_body, unb_list, nunb, counts,
                                                  offsets, out, status, nullptr, nullptr, nullptr);
            for (uint32_t u = 0; u < nunb; ++u) {
                uint32_t h = unb_host[u];
                k_unb_flags<<<grid, TB, 0, s>>>(h, n, mn, mx, flags);
                check_cuda(cub::DeviceScan::ExclusiveSum(tmp, scan_bytes, flags, unb_scan, int(n), s), "scan");
                k_unb_write<<<grid, TB, 0, s>>>(h, n, flags, unb_scan, offsets, out);
            }
            k_noalloc_keys_to_pairs<<<uint32_t((total + TB - 1) / TB), TB, 0, s>>>(out, total);
        }
        uint32_t st = 0;
        check_cuda(cudaMemcpyAsync(&st, status, 4, cudaMemcpyDeviceToHost, s), "d2h");
        check_cuda(cudaStreamSynchronize(s), "sync");
        check_cuda(cudaGetLastError(), "launch");
        if (st) {
            set_last_error("allocation-free broad phase: traversal stack overflow");
            return BGPU_ERR_DEVICE_STATUS;
        }
        return BGPU_OK;
    } catch (const CudaError& e) {
        set_last_error(e.where);
        return BGPU_ERR_CUDA;
    }
}

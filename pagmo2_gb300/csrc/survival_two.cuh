// Non-dominated sorting of 2-objective populations of up to kTwoPoints points
// (beyond the single block's limit). Included by survival.cu.
//
// Two objectives need no dominance matrix. In the order by (f0, f1, index) a
// point's dominators all come before it, and a front is the staircase of the
// points left: those whose f1 is below every earlier one's. The pass:
//  1. positions in each objective (sort_pos.cuh), two_scatter_kernel,
//     two_place_kernel: the lexicographic order, f0 and f1 as ranks (equal
//     values, equal ranks), 15 bits each.
//  2. two_peel_kernel, a cluster of blocks: the fronts, each the running minimum
//     of f1 over the positions left, passed from warp to warp;
//     two_lists_kernel: their sizes and unordered lists.
//  3. two_stairs_kernel: each front's distinct points by f0 (f1 falls along
//     them) and its points by index; two_ranges_kernel: for every point the run
//     of the front before that dominates it (f0 bounds it above, f1 below).
//  4. two_order_kernel, one block, front after front: a member's key is the
//     highest position in its run, the front's order is by (key, index), as the
//     reference appends them.
//  5. two_count_kernel, where the counts are asked for: earlier points with no
//     larger f1.
// Both sequences (2 and 4) are bound by the latency of their steps, some 1400
// and 2000 cycles a front. ZDT1, 20000 points in 153 fronts: peel 112 us and
// order 166 us (82 us for the fronts of the best 10000), where a grid barrier
// and row scans per front took 1542 us and the matrix 119 us. A population
// sampling it and the selection of its half: 1723 -> 284 us. Nested layers with
// crowding distances, n = 20000: 475 -> 316 us (1 layer), 1004 -> 342 us (30);
// n = 1100, 3 layers: 134 -> 98 us, 2000, 60: 408 -> 137 us. So the line lies at
// the single block's limit, below which that is faster, and at the 15 bits of
// a rank, above which the matrix pass remains.
#pragma once

#include "sort_pos.cuh"

namespace pgx
{
namespace
{

constexpr uint32_t kTwoPoints = 32768;
constexpr int kTwoThreads = 1024;
constexpr uint32_t kTwoInf = 0xffffu;
constexpr uint32_t kTwoRun = 64; // a run's elements (a level's, in a longer run) read one by one at most

// Scratch of the pass (in the room of the dominance matrix). A "position" is a
// place in the lexicographic order; equal points stand together, and the first
// of them stands for all until the members' lists.
struct two_scratch {
    void *runs;         // sort_pos.cuh
    uint2 *ent;         // n, by order: two_entry
    int32_t *pos;       // 2 n positions by objective
    int32_t *ord;       // 2 n: the points by position in an objective
    uint32_t *rr;       // n, by position: f0's rank << 16 | f1's rank
    uint32_t *ub;       // n, by position: points of no larger f1
    int32_t *id;        // n: the point of a position
    int32_t *uq;        // n: the first of its equals
    int32_t *rank_u;    // n: fronts of those
    int32_t *steps;     // n: the stairs' lengths
    int32_t *stair;     // n: the stairs' positions by f0, each stair where its front begins
    uint32_t *stair_v;  // n: their f1 ranks
    int32_t *at_u;      // n: index in its stair of a position
    int32_t *mem;       // n: positions by front, unordered
    int32_t *order;     // n: the same by front and point
    int32_t *deep;      // n: a run in the front's stair is longer than kTwoRun
};

constexpr uint32_t kTwoWords = 12; // the arrays of n + 1 words

constexpr size_t two_scratch_bytes(uint64_t n)
{
    return kTwoWords * align256((n + 1u) * 4u) + 2u * align256(2u * n * 4u) + align256(n * sizeof(uint2))
           + align256(pos_scratch_bytes(n, 2u));
}

two_scratch carve_two_scratch(void *base, uint64_t n)
{
    char *p = static_cast<char *>(base);
    const auto take = [&](size_t b) {
        void *q = p;
        p += align256(b);
        return q;
    };
    two_scratch s{};
    s.runs = take(pos_scratch_bytes(n, 2u));
    s.ent = static_cast<uint2 *>(take(n * sizeof(uint2)));
    s.pos = static_cast<int32_t *>(take(2u * n * 4u));
    s.ord = static_cast<int32_t *>(take(2u * n * 4u));
    int32_t **words[] = {&s.id, &s.uq, &s.rank_u, &s.steps, &s.stair, &s.at_u, &s.mem, &s.order, &s.deep};
    uint32_t **unsigned_words[] = {&s.rr, &s.ub, &s.stair_v};
    static_assert(sizeof(words) / sizeof(words[0]) + sizeof(unsigned_words) / sizeof(unsigned_words[0]) == kTwoWords,
                  "two_scratch_bytes counts the arrays");
    for (int32_t **a : words) *a = static_cast<int32_t *>(take((n + 1u) * 4u));
    for (uint32_t **a : unsigned_words) *a = static_cast<uint32_t *>(take((n + 1u) * 4u));
    return s;
}

__global__ void two_scatter_kernel(const double *__restrict__ pts, uint32_t n, const int32_t *__restrict__ pos,
                                   long long *__restrict__ keys, int32_t *__restrict__ ord,
                                   int32_t *__restrict__ deep, int32_t *__restrict__ front_offsets, peel_state *st)
{
    chain_wait();
    const uint32_t gt = blockIdx.x * blockDim.x + threadIdx.x, gn = gridDim.x * blockDim.x;
    for (uint32_t i = gt; i < n; i += gn) {
        keys[i] = order_key(pts[2u * i]);
        keys[n + i] = order_key(pts[2u * i + 1u]);
        ord[pos[i]] = static_cast<int32_t>(i);
        ord[n + pos[n + i]] = static_cast<int32_t>(i);
        front_offsets[i + 1u] = 0;
        deep[i] = 0;
    }
    if (gt == 0) front_offsets[0] = 0;
    for (uint32_t t = gt; t < sizeof(peel_state) / sizeof(int); t += gn) reinterpret_cast<int *>(st)[t] = 0;
}

// The end (dir = 1) or the beginning (dir = -1) of the run of keys equal to
// that at position p of an objective's order: steps of 1, 2, 4 .. beyond it,
// then halving (runs are mostly short).
__device__ __forceinline__ uint32_t two_tie_bound(const long long *keys, const int32_t *ord, uint32_t n, uint32_t p,
                                                  long long k, int dir)
{
    const auto equal = [&](uint32_t d) { // of the element d away
        if (dir > 0 ? p + d >= n : d > p) return false;
        return keys[ord[dir > 0 ? p + d : p - d]] == k;
    };
    uint32_t in = 0, out = 1;
    while (equal(out)) {
        in = out;
        out *= 2u;
    }
    while (out - in > 1u) {
        const uint32_t mid = (in + out) / 2u;
        if (equal(mid))
            in = mid;
        else
            out = mid;
    }
    return dir > 0 ? p + out : p - in;
}

__global__ void two_place_kernel(const long long *__restrict__ keys, uint32_t n, two_scratch s)
{
    chain_wait();
    const int32_t *o0 = s.ord, *o1 = s.ord + n, *pos1 = s.pos + n;
    const long long *keys1 = keys + n;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const long long k0 = keys[i], k1 = keys1[i];
        const uint32_t p0 = static_cast<uint32_t>(s.pos[i]), p1 = static_cast<uint32_t>(pos1[i]);
        const uint32_t r1 = two_tie_bound(keys1, o1, n, p1, k1, -1), e1 = two_tie_bound(keys1, o1, n, p1, k1, 1);
        const uint32_t lo = two_tie_bound(keys, o0, n, p0, k0, -1), hi = two_tie_bound(keys, o0, n, p0, k0, 1);
        uint32_t p = lo, first = lo; // among equal f0: by (f1, index), which f1's positions follow
        if (hi - lo > 1u)
            for (uint32_t x = lo; x < hi; ++x) {
                const uint32_t q = static_cast<uint32_t>(pos1[o0[x]]);
                p += q < p1 ? 1u : 0u;
                first += q < r1 ? 1u : 0u;
            }
        s.rr[p] = lo << 16 | r1;
        s.ub[p] = e1;
        s.id[p] = static_cast<int32_t>(i);
        s.uq[p] = static_cast<int32_t>(first);
    }
}

// Exclusive prefix sum of one value per thread over the block; *total gets the sum.
__device__ __forceinline__ uint32_t two_block_scan(uint32_t v, uint32_t *part, uint32_t *total)
{
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, o);
        if (static_cast<int>(lane) >= o) incl += t;
    }
    if (lane == 31u) part[warp] = incl;
    __syncthreads();
    const uint32_t t = lane < nw ? part[lane] : 0u;
    const uint32_t before = __reduce_add_sync(kFull, lane < warp ? t : 0u);
    *total = __reduce_add_sync(kFull, t);
    __syncthreads(); // part is free again
    return before + incl - v;
}

// ---- the fronts. Warp w of the cluster holds 2 Q rows of 32 consecutive
// positions, a value (f1's rank; kTwoInf once taken) per lane and row. A front
// k passes through the warps in order: warp w gets the minimum of the front so
// far from warp w - 1, sends its own minimum with it on to warp w + 1 at once,
// and only then takes its members out, the values below the front's minimum and
// below all before them in the warp, which a scan over the rows finds for the
// next front meanwhile. So the warps work on different fronts at a time. A
// minimum of kTwoInf says that no earlier warp has points left, now or later.
// Messages go through a ring of kTwoRing words per warp in its block's shared
// memory, (k + 1) << 16 | minimum, so that a word tells whose it is; the
// receiver acknowledges every half ring. Waits are bounded by spin_limit polls;
// when one runs out, those behind it do too, st->err is set and the number of
// fronts is -1, for which the kernels after this one do nothing.
// n = 20000, 153 fronts: 112 us, some 1400 cycles a front for the slowest warp
// (one block with barriers, 20 positions per thread: 220 us; rows behind
// branches on their number, not interleaved: 168 us).
constexpr uint32_t kTwoBlocks = 8; // of the cluster
constexpr uint32_t kTwoWarps = 16; // per block
constexpr uint32_t kTwoRows = kTwoPoints / (32u * kTwoBlocks * kTwoWarps);
constexpr uint32_t kTwoRing = 128;
constexpr uint32_t kTwoSpins = 1u << 22;

// p's address in another block of the cluster.
__device__ __forceinline__ uint32_t two_remote(const void *p, uint32_t block)
{
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;"
        : "=r"(a)
        : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))), "r"(block));
    return a;
}

__device__ __forceinline__ void two_send(uint32_t addr, uint32_t v)
{
    asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

__device__ __forceinline__ uint32_t two_peek(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.relaxed.cluster.shared::cta.u32 %0, [%1];"
                 : "=r"(v)
                 : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p)))
                 : "memory");
    return v;
}

__device__ __forceinline__ void two_cluster_sync()
{
    asm volatile("barrier.cluster.arrive;\nbarrier.cluster.wait;" ::: "memory");
}

// Q: registers of two rows each.
template <uint32_t Q>
__global__ void __cluster_dims__(kTwoBlocks, 1, 1) __launch_bounds__(kTwoWarps * 32, 1)
    two_peel_kernel(two_scratch s, uint32_t n, uint32_t spin_limit, int32_t *__restrict__ n_fronts, peel_state *st)
{
    chain_wait();
    __shared__ uint32_t ring[kTwoWarps][kTwoRing], acked[kTwoWarps];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, w = blockIdx.x * kTwoWarps + warp;
    const uint32_t rows = (n + 31u) / 32u, E = 2u * Q;
    const uint32_t warps = (rows + E - 1u) / E;
    for (uint32_t t = lane; t < kTwoRing; t += 32u) ring[warp][t] = 0u;
    if (lane == 0u) acked[warp] = 0u;
    two_cluster_sync();
    if (w < warps) {
        const uint32_t base = w * E * 32u + lane;
        // rows 2 q, 2 q + 1 in the halves of v[q]; bound: the least value before each (in the warp)
        uint32_t v[Q], bound[Q], least = kTwoInf;
        const auto value = [&](uint32_t r) {
            const uint32_t p = base + 32u * r;
            if (p >= n) return kTwoInf;
            return s.uq[p] == static_cast<int32_t>(p) ? s.rr[p] & 0xffffu : kTwoInf;
        };
        const auto scan = [&] {
            uint32_t incl[Q];
#pragma unroll
            for (uint32_t q = 0; q < Q; ++q) incl[q] = v[q];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
                for (uint32_t q = 0; q < Q; ++q) // (the lowest lanes get their own)
                    incl[q] = __vminu2(incl[q], __shfl_up_sync(kFull, incl[q], o));
            }
            least = kTwoInf;
#pragma unroll
            for (uint32_t q = 0; q < Q; ++q) {
                const uint32_t before = __shfl_up_sync(kFull, incl[q], 1);
                const uint32_t total = __shfl_sync(kFull, incl[q], 31);
                const uint32_t mid = min(least, total & 0xffffu);
                bound[q] = __vminu2(lane ? before : 0xffffffffu, mid << 16 | least);
                least = min(mid, total >> 16);
            }
        };
#pragma unroll
        for (uint32_t q = 0; q < Q; ++q) v[q] = value(2u * q + 1u) << 16 | value(2u * q);
        scan();
        // the next warp's ring and the word that the warp before reads our progress from
        const bool last = w + 1u == warps;
        const uint32_t to = two_remote(ring[(warp + 1u) % kTwoWarps], last ? blockIdx.x : (w + 1u) / kTwoWarps);
        const uint32_t back =
            two_remote(acked + (warp + kTwoWarps - 1u) % kTwoWarps, w == 0u ? 0u : (w - 1u) / kTwoWarps);
        bool waiting = w != 0u, failed = false; // waiting: earlier warps have points left
        uint32_t k = 0, room = kTwoRing;        // fronts below room fit in the next warp's ring
        for (;; ++k) {
            uint32_t T = kTwoInf;
            if (waiting) {
                const uint32_t *slot = ring[warp] + k % kTwoRing;
                uint32_t m = two_peek(slot), spins = 0;
                while (m >> 16 != k + 1u && ++spins < spin_limit) m = two_peek(slot);
                m = __shfl_sync(kFull, m, 0); // (lanes may have read it at different times)
                if (m >> 16 != k + 1u) {
                    failed = true;
                    break;
                }
                T = m & 0xffffu;
                waiting = T != kTwoInf;
                if ((k + 1u) % (kTwoRing / 2u) == 0u && lane == 0u) two_send(back, k + 1u);
            }
            const uint32_t out = min(T, least);
            if (!last) {
                if (k >= room) {
                    uint32_t a = two_peek(acked + warp), spins = 0;
                    while (k >= a + kTwoRing && ++spins < spin_limit) a = two_peek(acked + warp);
                    a = __shfl_sync(kFull, a, 0);
                    if (k >= a + kTwoRing) {
                        failed = true;
                        break;
                    }
                    room = a + kTwoRing;
                }
                if (lane == 0u) two_send(to + 4u * (k % kTwoRing), (k + 1u) << 16 | out);
            }
            if (out == kTwoInf) break; // no point is left up to here
            if (least < T) {
#pragma unroll
                for (uint32_t q = 0; q < Q; ++q) {
                    const uint32_t m = __vminu2(bound[q], T << 16 | T);
                    if ((v[q] & 0xffffu) < (m & 0xffffu)) {
                        v[q] |= kTwoInf;
                        s.rank_u[base + 64u * q] = static_cast<int32_t>(k);
                    }
                    if (v[q] >> 16 < m >> 16) {
                        v[q] |= kTwoInf << 16;
                        s.rank_u[base + 64u * q + 32u] = static_cast<int32_t>(k);
                    }
                }
                scan();
            }
        }
        if (failed && lane == 0u) st->err = 1;
        if (last && lane == 0u) {
            *n_fronts = failed ? -1 : static_cast<int32_t>(k);
            st->n_fronts = failed ? -1 : static_cast<int32_t>(k);
        }
    }
    two_cluster_sync(); // no block leaves while its shared memory may be written
}

// The number of fronts; 0, and nothing to do, where the waits ran out.
__device__ __forceinline__ uint32_t two_fronts(const int32_t *n_fronts)
{
    return static_cast<uint32_t>(max(*n_fronts, 0));
}

// The fronts' offsets and unordered lists of positions, written out in order
// (scattered to global memory from one SM: 36 us at n = 20000, 11 us now).
constexpr size_t two_lists_smem(uint32_t n)
{
    return align256(n * sizeof(uint32_t)) + align256(n * sizeof(uint16_t));
}

__global__ void __launch_bounds__(kTwoThreads, 1)
    two_lists_kernel(two_scratch s, uint32_t n, int32_t *__restrict__ front_offsets,
                     const int32_t *__restrict__ n_fronts)
{
    chain_wait();
    extern __shared__ __align__(256) unsigned char two_mem[];
    __shared__ uint32_t part[32];
    uint32_t *cnt = reinterpret_cast<uint32_t *>(two_mem);
    uint16_t *mem = reinterpret_cast<uint16_t *>(two_mem + align256(n * sizeof(uint32_t)));
    const uint32_t tid = threadIdx.x, F = two_fronts(n_fronts);
    if (F == 0u) return;
    for (uint32_t f = tid; f < F; f += kTwoThreads) cnt[f] = 0u;
    constexpr uint32_t kPer = kTwoPoints / kTwoThreads;
    uint32_t of[kPer];
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j) of[j] = static_cast<uint32_t>(s.uq[min(tid + j * kTwoThreads, n - 1u)]);
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j) of[j] = static_cast<uint32_t>(s.rank_u[of[j]]);
    __syncthreads();
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j)
        if (tid + j * kTwoThreads < n) atomicAdd(cnt + of[j], 1u);
    __syncthreads();
    const uint32_t fp = (F + kTwoThreads - 1u) / kTwoThreads, f0 = min(F, tid * fp), f1 = min(F, f0 + fp);
    uint32_t sum = 0, total = 0;
    for (uint32_t f = f0; f < f1; ++f) sum += cnt[f];
    uint32_t at = two_block_scan(sum, part, &total);
    for (uint32_t f = f0; f < f1; ++f) {
        const uint32_t c = cnt[f];
        cnt[f] = at;
        front_offsets[f] = static_cast<int32_t>(at);
        at += c;
    }
    if (tid == 0) front_offsets[F] = static_cast<int32_t>(total);
    __syncthreads();
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j) {
        const uint32_t p = tid + j * kTwoThreads;
        if (p < n) mem[atomicAdd(cnt + of[j], 1u)] = static_cast<uint16_t>(p);
    }
    __syncthreads();
    for (uint32_t p = tid; p < n; p += kTwoThreads) s.mem[p] = mem[p];
}

// A front's list in ascending order of its values (distinct, below n; kTwoNone
// is left out): place(t, value, rank) for each. A short list ranks by counting,
// a long one by a bit set of its values with the counts before each word.
// Returns how many there are.
constexpr int kStairThreads = 256;
constexpr uint32_t kStairShort = 256;
constexpr uint32_t kStairWords = kTwoPoints / 32u;
constexpr uint32_t kTwoNone = 0xffffffffu;

template <typename Value, typename Place>
__device__ __forceinline__ uint32_t two_rank_list(uint32_t L, uint32_t n, uint32_t *list, uint32_t *before,
                                                  uint32_t *part, Value value, Place place)
{
    const uint32_t tid = threadIdx.x;
    if (L <= kStairShort) {
        const uint32_t q = tid < L ? value(tid) : kTwoNone;
        const uint32_t some = static_cast<uint32_t>(__syncthreads_count(q != kTwoNone)); // (list is free, too)
        list[tid] = q;
        __syncthreads();
        if (q != kTwoNone) {
            uint32_t p = 0;
#pragma unroll 8
            for (uint32_t o = 0; o < L; ++o) p += list[o] < q ? 1u : 0u;
            place(tid, q, p);
        }
        return some;
    }
    const uint32_t W = (n + 31u) / 32u;
    __syncthreads(); // list is free
    for (uint32_t w = tid; w < kStairWords; w += kStairThreads) list[w] = 0u;
    __syncthreads();
    for (uint32_t t = tid; t < L; t += kStairThreads) {
        const uint32_t q = value(t);
        if (q != kTwoNone) atomicOr(list + q / 32u, 1u << (q & 31u));
    }
    __syncthreads();
    constexpr uint32_t kPer = kStairWords / kStairThreads;
    uint32_t c[kPer], sum = 0, total = 0;
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j) {
        const uint32_t w = tid * kPer + j;
        c[j] = w < W ? static_cast<uint32_t>(__popc(list[w])) : 0u;
        sum += c[j];
    }
    uint32_t at = two_block_scan(sum, part, &total);
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j) {
        before[tid * kPer + j] = at;
        at += c[j];
    }
    __syncthreads();
    for (uint32_t t = tid; t < L; t += kStairThreads) {
        const uint32_t q = value(t), w = q / 32u;
        if (q != kTwoNone) place(t, q, before[w] + static_cast<uint32_t>(__popc(list[w] & ((1u << (q & 31u)) - 1u))));
    }
    return total;
}

// Per front: its stair, by f0, and its positions by point.
__global__ void __launch_bounds__(kStairThreads)
    two_stairs_kernel(two_scratch s, uint32_t n, const int32_t *__restrict__ front_offsets,
                      const int32_t *__restrict__ n_fronts, int32_t *__restrict__ rank)
{
    chain_wait();
    __shared__ uint32_t list[kStairWords], before[kStairWords], part[32];
    const uint32_t F = two_fronts(n_fronts);
    for (uint32_t x = blockIdx.x; x < 2u * F; x += gridDim.x) {
        const uint32_t f = x >> 1, off = static_cast<uint32_t>(front_offsets[f]);
        const uint32_t L = static_cast<uint32_t>(front_offsets[f + 1u]) - off;
        if (x & 1u) {
            two_rank_list(
                L, n, list, before, part, [&](uint32_t t) { return static_cast<uint32_t>(s.id[s.mem[off + t]]); },
                [&](uint32_t t, uint32_t i, uint32_t p) {
                    s.order[off + p] = s.mem[off + t];
                    rank[i] = static_cast<int32_t>(f);
                });
        } else {
            const uint32_t S = two_rank_list(
                L, n, list, before, part,
                [&](uint32_t t) {
                    const int32_t q = s.mem[off + t];
                    return s.uq[q] == q ? static_cast<uint32_t>(q) : kTwoNone;
                },
                [&](uint32_t, uint32_t q, uint32_t p) {
                    s.stair[off + p] = static_cast<int32_t>(q);
                    s.stair_v[off + p] = s.rr[q] & 0xffffu;
                    s.at_u[q] = static_cast<int32_t>(p);
                });
            if (threadIdx.x == 0) s.steps[f] = static_cast<int32_t>(S);
        }
    }
}

// What the order of a front needs of a point: the point, its index in the
// front's stair (kTwoNoStep but for the last of equal points), its run in the
// stair of the front before, 15 + 16 + 15 + 16 bits.
constexpr uint32_t kTwoNoStep = 0xffffu;

__device__ __forceinline__ uint2 two_entry(uint32_t point, uint32_t step, uint32_t begin, uint32_t end)
{
    return make_uint2(point << 16 | step, begin << 16 | end);
}

__global__ void two_ranges_kernel(two_scratch s, uint32_t n, const int32_t *__restrict__ front_offsets,
                                  const int32_t *__restrict__ n_fronts)
{
    chain_wait();
    if (two_fronts(n_fronts) == 0u) return;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const uint32_t p = static_cast<uint32_t>(s.order[t]), u = static_cast<uint32_t>(s.uq[p]);
        const int32_t f = s.rank_u[u];
        const bool last = p + 1u == n || s.rr[p + 1u] != s.rr[p]; // of equal points: the highest index
        uint32_t begin = 0, end = 0;
        if (f > 0) {
            const uint32_t b = static_cast<uint32_t>(front_offsets[f - 1]), L = static_cast<uint32_t>(s.steps[f - 1]);
            const uint32_t v = s.rr[p] & 0xffffu;
            // the run: from the first step of no larger f1 to the last before u
            uint32_t lo0 = 0, hi0 = L, lo1 = 0, hi1 = L;
            while (lo0 < hi0 || lo1 < hi1) {
                const uint32_t m0 = (lo0 + hi0) / 2u, m1 = (lo1 + hi1) / 2u;
                const uint32_t x0 = lo0 < hi0 ? s.stair_v[b + m0] : 0u;
                const uint32_t x1 = lo1 < hi1 ? static_cast<uint32_t>(s.stair[b + m1]) : 0u;
                if (lo0 < hi0) {
                    if (x0 > v)
                        lo0 = m0 + 1u;
                    else
                        hi0 = m0;
                }
                if (lo1 < hi1) {
                    if (x1 < u)
                        lo1 = m1 + 1u;
                    else
                        hi1 = m1;
                }
            }
            begin = lo0;
            end = lo1; // one past the run
            if (end - begin > kTwoRun) s.deep[f - 1] = 1;
        }
        const uint32_t step = last ? static_cast<uint32_t>(s.at_u[u]) : kTwoNoStep;
        s.ent[t] = two_entry(static_cast<uint32_t>(s.id[p]), step, begin, end);
    }
}

// Room for the words of a front of L points: the block sorts 2, 4, 8 or 32 words
// per thread, at indexes skewed by a word in 32 (its threads' consecutive words
// would share banks).
constexpr uint32_t two_order_room(uint32_t L)
{
    return L <= 2048u ? 2048u : (L <= 4096u ? 4096u : (L <= 8192u ? 8192u : kTwoPoints));
}

__host__ __device__ constexpr uint32_t two_skew(uint32_t i)
{
    return i + (i >> 5);
}

constexpr size_t two_order_smem(uint32_t n) // a front's words, then positions of the stair before
{
    return align256(two_skew(two_order_room(n)) * sizeof(uint32_t)) + align256((n + 64u) * sizeof(uint16_t));
}

// The words at s ascending, by the block: E consecutive ones per thread
// ordered in registers, then merge levels as in sort_runs_kernel.
template <uint32_t E>
__device__ __noinline__ void two_block_sort(uint32_t *s)
{
    const uint32_t e0 = threadIdx.x * E;
    uint32_t r[E];
#pragma unroll
    for (uint32_t q = 0; q < E; ++q) r[q] = s[two_skew(e0 + q)];
    for (uint32_t round = 0; round < E; round += 2u) {
#pragma unroll
        for (uint32_t h = 0; h < 2u; ++h) {
#pragma unroll
            for (uint32_t q = h; q + 1u < E; q += 2u) {
                const uint32_t a = min(r[q], r[q + 1u]), b = max(r[q], r[q + 1u]);
                r[q] = a;
                r[q + 1u] = b;
            }
        }
    }
    for (uint32_t w = E; w < kTwoThreads * E; w <<= 1) {
        __syncthreads();
#pragma unroll
        for (uint32_t q = 0; q < E; ++q) s[two_skew(e0 + q)] = r[q];
        __syncthreads();
        const uint32_t d = e0 & (2u * w - 1u), A = e0 - d, B = A + w;
        uint32_t lo = d > w ? d - w : 0u, hi = d < w ? d : w;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (s[two_skew(A + mid)] <= s[two_skew(B + d - 1u - mid)])
                lo = mid + 1u;
            else
                hi = mid;
        }
        uint32_t ia = lo, ib = d - lo;
        uint32_t ka = ia < w ? s[two_skew(A + ia)] : 0xffffffffu, kb = ib < w ? s[two_skew(B + ib)] : 0xffffffffu;
#pragma unroll
        for (uint32_t q = 0; q < E; ++q) {
            // (words are distinct but for the highest, the padding: either side's will do)
            const bool from_a = ka <= kb;
            r[q] = from_a ? ka : kb;
            const uint32_t next = from_a ? ++ia : ++ib;
            const uint32_t k = next < w ? s[two_skew((from_a ? A : B) + next)] : 0xffffffffu;
            ka = from_a ? k : ka;
            kb = from_a ? kb : k;
        }
    }
    __syncthreads();
#pragma unroll
    for (uint32_t q = 0; q < E; ++q) s[two_skew(e0 + q)] = r[q];
    __syncthreads();
}

// c of the threads below room (a power of two, 64 .. 1024; the other threads
// pass too) ascending by thread: by shuffles within the warps, then levels in
// which a word's place is its own in its half plus a binary search in the
// other half. s: two buffers of 1024 words.
__device__ __forceinline__ uint32_t two_thread_sort(uint32_t c, uint32_t room, uint32_t *s)
{
    const uint32_t tid = threadIdx.x, lane = tid & 31u;
    const bool act = tid < room; // whole warps
    if (act) {
#pragma unroll
        for (uint32_t k = 2; k <= 32u; k <<= 1) {
#pragma unroll
            for (uint32_t j = k >> 1; j > 0u; j >>= 1) {
                const uint32_t o = __shfl_xor_sync(kFull, c, static_cast<int>(j));
                c = ((lane & j) == 0u) == ((lane & k) == 0u) ? min(c, o) : max(c, o);
            }
        }
        s[tid] = c;
    }
    uint32_t *from = s, *to = s + kTwoThreads;
    for (uint32_t w = 32u; w < room; w <<= 1) {
        __syncthreads();
        if (act) {
            c = from[tid];
            const uint32_t base = tid & ~(2u * w - 1u);
            const bool upper = (tid & w) != 0u;
            const uint32_t *o = from + base + (upper ? 0u : w);
            uint32_t at = 0;
            for (uint32_t step = w >> 1; step > 0u; step >>= 1) {
                const uint32_t y = o[at + step - 1u];
                if (upper ? y <= c : y < c) at += step;
            }
            const uint32_t y = o[at];
            at += (upper ? y <= c : y < c) ? 1u : 0u;
            to[base + (tid & (w - 1u)) + at] = c;
        }
        uint32_t *t = from;
        from = to;
        to = t;
    }
    __syncthreads();
    return act ? from[tid] : 0xffffffffu;
}

// Maxima of a stair's positions by blocks of 8, 64 and 512: a run of any length
// costs few reads (two long fronts: 10^8 otherwise).
struct two_high {
    uint16_t *pos, *by8, *by64, *by512;
};

// Maximum over [a, b).
__device__ __forceinline__ uint32_t two_run_max(const two_high &h, uint32_t a, uint32_t b)
{
    uint32_t key = 0;
    const auto over = [&](const uint16_t *p, uint32_t x, uint32_t y) {
        for (uint32_t q = x; q < y; q += 4u) {
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j) key = max(key, static_cast<uint32_t>(p[min(q + j, y - 1u)]));
        }
    };
    const uint16_t *p = h.pos;
    for (uint32_t level = 0; level < 3u && b > a + kTwoRun; ++level) {
        const uint32_t x = (a + 7u) / 8u, y = b / 8u;
        over(p, a, 8u * x);
        over(p, 8u * y, b);
        a = x;
        b = y;
        p = level == 0u ? h.by8 : (level == 1u ? h.by64 : h.by512);
    }
    over(p, a, b);
    return key;
}

__device__ __forceinline__ uint32_t two_max8(const uint16_t *p)
{
    const uint4 q = *reinterpret_cast<const uint4 *>(p);
    const uint32_t m = __vmaxu2(__vmaxu2(q.x, q.y), __vmaxu2(q.z, q.w));
    return max(m & 0xffffu, m >> 16);
}

// The fronts' orders, one front after the other. Its sequential steps bound it:
// a front of some 100 points takes about 2000 cycles. What a front needs is
// brought to shared memory two fronts ahead.
//  - Small fronts (up to 256 points and as many positions in the front before)
//    are the work of 8 warps, with barriers among these alone, while the others
//    wait for the next larger one: 1024 threads' common instructions alone took
//    more issue slots than the front's own work.
//    Up to kTwoPairs points: each word's place by counting the lower ones, two
//    threads per point; more: points per key counted, a scan of the counts, then
//    the few of equal keys among themselves.
//  - Up to 1024 points and positions: the same by all warps; many of a key, or
//    more positions: two_thread_sort; longer: two_block_sort.
constexpr uint32_t kTwoTeam = 256;  // threads (points, positions) of small fronts
constexpr uint32_t kTwoPairs = 128;
constexpr uint32_t kTwoAhead = 512; // fronts up to this size are brought in ahead
constexpr uint32_t kTwoSame = 32;   // points of one key compared among themselves at most
constexpr uint32_t kTwoOffs = 256;  // fronts per load of offsets

// Entries [b, e) of a front to shared memory, by `threads` threads.
__device__ __forceinline__ void two_bring(const uint2 *ent, uint32_t b, uint32_t e, uint2 *to, uint32_t threads)
{
    if (e - b <= kTwoAhead)
        for (uint32_t t = threadIdx.x; t < e - b; t += threads)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                             static_cast<uint32_t>(__cvta_generic_to_shared(to + t))),
                         "l"(ent + b + t)
                         : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// The small fronts fc + g .. fc + h - 1, by the threads below kTwoTeam.
__device__ __noinline__ void two_small_fronts(const uint2 *ent, const uint32_t *offs, uint32_t g, uint32_t h,
                                              uint32_t fc, uint2 (*ahead)[kTwoAhead], uint16_t *high, uint32_t *comp,
                                              uint32_t *cnt, uint16_t *list, uint32_t *part, int32_t *front_indices)
{
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const auto sync = [] { asm volatile("barrier.sync 1, %0;" ::"n"(kTwoTeam) : "memory"); };
    uint32_t slot = (fc + g) % 3u, off = offs[g], next = offs[g + 1u], after = offs[g + 2u];
    for (; g < h; ++g) {
        const uint32_t L = next - off, beyond = offs[g + 3u];
        const uint32_t to = slot == 0u ? 2u : slot - 1u; // (slot + 2) % 3
        two_bring(ent, after, beyond, ahead[to], kTwoTeam);
        asm volatile("cp.async.wait_group 1;" ::: "memory"); // the next front's have come
        const uint2 *ents = ahead[slot];
        const bool pairs = L <= kTwoPairs;
        const uint32_t t = pairs ? tid >> 1 : tid;
        const bool act = t < L;
        uint2 e = make_uint2(kTwoNoStep, 0u);
        if (act) e = ents[t];
        const uint32_t begin = e.y >> 16, end = e.y & 0xffffu;
        uint32_t key = 0;
        for (uint32_t q = begin; q < end; q += 4u) {
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j) key = max(key, static_cast<uint32_t>(high[min(q + j, end - 1u)]));
        }
        uint32_t p = 0;
        if (pairs) {
            const uint32_t mine = act ? key << 15 | t : 0xffffffffu;
            if (tid < 8u) comp[L + tid] = 0xffffffffu; // the last eight's rest: below no word
            if (act) comp[t] = mine;
            sync();
            const uint4 *words = reinterpret_cast<const uint4 *>(comp);
#pragma unroll 4
            for (uint32_t c = tid & 1u; 4u * c < L; c += 2u) {
                const uint4 q = words[c];
                p += (q.x < mine) + (q.y < mine) + (q.z < mine) + (q.w < mine);
            }
            p += __shfl_xor_sync(kFull, p, 1);
        } else {
            // (cnt is all 0)
            const uint32_t mine = act ? atomicAdd(cnt + key, 1u) : 0u;
            sync();
            const uint32_t c = cnt[tid];
            uint32_t incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t x = __shfl_up_sync(kFull, incl, o);
                if (static_cast<int>(lane) >= o) incl += x;
            }
            if (lane == 31u) part[warp] = incl;
            sync();
            const uint32_t before = __reduce_add_sync(kFull, lane < warp ? part[lane] : 0u);
            cnt[tid] = c << 16 | (before + incl - c);
            sync();
            uint32_t same = 0;
            if (act) {
                const uint32_t x = cnt[key];
                p = x & 0xffffu;
                same = x >> 16;
                list[p + mine] = static_cast<uint16_t>(t);
            }
            sync();
            cnt[tid] = 0u;
            if (same > 1u)
                for (uint32_t q = p, last = p + same; q < last; ++q) p += list[q] < t ? 1u : 0u;
        }
        if (act && (!pairs || (tid & 1u) == 0u)) {
            front_indices[off + p] = static_cast<int32_t>(e.x >> 16);
            if ((e.x & 0xffffu) != kTwoNoStep) high[e.x & 0xffffu] = static_cast<uint16_t>(p);
        }
        sync();
        off = next;
        next = after;
        after = beyond;
        slot = slot == 2u ? 0u : slot + 1u;
    }
}

__global__ void __launch_bounds__(kTwoThreads, 1)
    two_order_kernel(two_scratch s, uint32_t n, uint32_t need, const int32_t *__restrict__ front_offsets,
                     const int32_t *__restrict__ n_fronts, int32_t *__restrict__ front_indices)
{
    chain_wait();
    extern __shared__ __align__(256) unsigned char two_mem[];
    __shared__ __align__(16) uint16_t by8[kTwoPoints / 8u], by64[kTwoPoints / 64u], by512[kTwoPoints / 512u];
    __shared__ __align__(16) uint2 ahead[3][kTwoAhead];
    __shared__ uint32_t offs[kTwoOffs + 4u], part[32];
    __shared__ uint32_t cnt[kTwoThreads]; // points per key, then where the key's begin
    __shared__ uint16_t list[kTwoThreads];
    __shared__ int32_t deep[kTwoOffs], many;
    uint32_t *comp = reinterpret_cast<uint32_t *>(two_mem);
    uint16_t *high = reinterpret_cast<uint16_t *>(two_mem + align256(two_skew(two_order_room(n)) * sizeof(uint32_t)));
    const two_high run{high, by8, by64, by512};
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, F = two_fronts(n_fronts);
    uint32_t K = 1u; // positions of the front before
    cnt[tid] = 0u;
    if (tid == 0u) many = 0;
    for (uint32_t fc = 0; fc < F; fc += kTwoOffs) {
        __syncthreads();
        if (tid < kTwoOffs + 4u) offs[tid] = static_cast<uint32_t>(front_offsets[min(fc + tid, F)]);
        if (tid < kTwoOffs) deep[tid] = s.deep[min(fc + tid, F - 1u)];
        __syncthreads();
        // the fronts that hold the first `need` points
        const uint32_t g1 = static_cast<uint32_t>(__syncthreads_count(tid < min(kTwoOffs, F - fc) && offs[tid] < need));
        if (g1 == 0u) break;
        const auto bring = [&](uint32_t g) {
            two_bring(s.ent, offs[g], offs[g + 1u], ahead[(fc + g) % 3u], kTwoThreads);
        };
        if (fc == 0u) {
            bring(0u);
            bring(1u);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();
        }
        for (uint32_t g = 0; g < g1; ++g) {
            {
                const auto small = [&](uint32_t h) {
                    return offs[h + 1u] - offs[h] <= kTwoTeam && (h ? offs[h] - offs[h - 1u] : K) <= kTwoTeam
                           && !deep[h] && (h ? deep[h - 1u] == 0 : fc == 0u);
                };
                uint32_t h = g;
                while (h < g1 && small(h)) ++h;
                if (h > g) {
                    if (tid < kTwoTeam)
                        two_small_fronts(s.ent, offs, g, h, fc, ahead, high, comp, cnt, list, part, front_indices);
                    K = offs[h] - offs[h - 1u];
                    g = h;
                    __syncthreads();
                    if (g == g1) break;
                }
            }
            const uint32_t off = offs[g], L = offs[g + 1u] - off;
            bring(g + 2u);
            asm volatile("cp.async.wait_group 1;" ::: "memory"); // the next front's have come
            const uint2 *ents = L <= kTwoAhead ? ahead[(fc + g) % 3u] : s.ent + off;
            const auto key_of = [&](uint2 e) { return two_run_max(run, e.y >> 16, e.y & 0xffffu); };
            const auto put = [&](uint2 e, uint32_t p) {
                front_indices[off + p] = static_cast<int32_t>(e.x >> 16);
                if ((e.x & 0xffffu) != kTwoNoStep) high[e.x & 0xffffu] = static_cast<uint16_t>(p);
            };
            if (L <= kTwoThreads) {
                const bool act = tid < L;
                uint2 e = make_uint2(kTwoNoStep, 0u);
                uint32_t key = 0;
                if (act) {
                    e = ents[tid];
                    key = key_of(e);
                }
                bool sort = K > kTwoThreads;
                if (fc + g == 0u) { // (the first front's keys are all 0: it is in order)
                    if (act) put(e, tid);
                    __syncthreads();
                } else if (!sort) {
                    const uint32_t team = (max(L, K) + 31u) & ~31u; // threads; cnt is all 0
                    const auto sync = [&] { asm volatile("barrier.sync 1, %0;" ::"r"(team) : "memory"); };
                    if (tid < team) {
                        const uint32_t slot = act ? atomicAdd(cnt + key, 1u) : 0u;
                        sync();
                        const uint32_t c = cnt[tid];
                        uint32_t incl = c;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const uint32_t x = __shfl_up_sync(kFull, incl, o);
                            if (static_cast<int>(lane) >= o) incl += x;
                        }
                        if (lane == 31u) part[warp] = incl;
                        if (c > kTwoSame) many = 1;
                        sync();
                        const uint32_t before = __reduce_add_sync(kFull, lane < warp ? part[lane] : 0u);
                        cnt[tid] = c << 16 | (before + incl - c);
                        sync();
                        uint32_t from = 0, same = 0;
                        if (act) {
                            const uint32_t x = cnt[key];
                            from = x & 0xffffu;
                            same = x >> 16;
                            list[from + slot] = static_cast<uint16_t>(tid);
                        }
                        sync();
                        cnt[tid] = 0u;
                        if (act && !many) {
                            uint32_t p = from;
                            if (same > 1u)
                                for (uint32_t q = from; q < from + same; ++q) p += list[q] < tid ? 1u : 0u;
                            put(e, p);
                        }
                    }
                    __syncthreads();
                    sort = many != 0;
                }
                if (sort) {
                    uint32_t room = 64u;
                    while (room < L) room *= 2u;
                    const uint32_t c = two_thread_sort(act ? key << 15 | tid : 0xffffffffu, room, comp);
                    if (act) put(ents[c & 0x7fffu], tid);
                    if (tid == 0u) many = 0;
                    __syncthreads();
                }
            } else {
                const uint32_t room = two_order_room(L);
                for (uint32_t b = tid; b < room; b += 2u * kTwoThreads) {
                    uint2 e[2];
#pragma unroll
                    for (uint32_t j = 0; j < 2u; ++j) e[j] = s.ent[min(off + b + j * kTwoThreads, n - 1u)];
#pragma unroll
                    for (uint32_t j = 0; j < 2u; ++j) {
                        const uint32_t t = b + j * kTwoThreads;
                        comp[two_skew(t)] = t < L ? key_of(e[j]) << 15 | t : 0xffffffffu;
                    }
                }
                __syncthreads();
                if (fc + g > 0u) {
                    if (room == 2048u)
                        two_block_sort<2>(comp);
                    else if (room == 4096u)
                        two_block_sort<4>(comp);
                    else if (room == 8192u)
                        two_block_sort<8>(comp);
                    else
                        two_block_sort<32>(comp);
                }
                for (uint32_t b = tid; b < L; b += 4u * kTwoThreads) {
                    uint2 e[4];
#pragma unroll
                    for (uint32_t j = 0; j < 4u; ++j) {
                        const uint32_t t = b + j * kTwoThreads;
                        e[j] = s.ent[off + (t < L ? comp[two_skew(t)] & 0x7fffu : 0u)];
                    }
#pragma unroll
                    for (uint32_t j = 0; j < 4u; ++j)
                        if (b + j * kTwoThreads < L) put(e[j], b + j * kTwoThreads);
                }
                __syncthreads();
            }
            if (deep[g]) { // (what lies beyond the stair in its last blocks is in no run)
                for (uint32_t b = tid; 8u * (b - lane) < L; b += kTwoThreads) {
                    uint32_t v = 8u * b < n ? two_max8(high + 8u * b) : 0u;
                    by8[b] = static_cast<uint16_t>(v);
#pragma unroll
                    for (int o = 1; o < 8; o <<= 1) v = max(v, __shfl_xor_sync(kFull, v, o));
                    if ((lane & 7u) == 0u) by64[b / 8u] = static_cast<uint16_t>(v);
                }
                __syncthreads();
                if (L > 64u * kTwoRun) {
                    if (512u * tid < L) by512[tid] = static_cast<uint16_t>(two_max8(by64 + 8u * tid));
                    __syncthreads();
                }
            }
            K = L;
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// dom_count by lexicographic position: earlier points of no larger f1, less the
// equal points before. Block (c, part): chunk c's points as a bit set over f1's
// positions with the counts before each word, asked by part's share of the
// later points; the chunk's own points count their earlier ones one by one.
// (All earlier points one by one: 39 us at n = 20000, 16 us now.)
constexpr uint32_t kCountChunk = 512;
constexpr int kCountThreads = 256;
constexpr uint32_t kCountParts = 16;

__global__ void __launch_bounds__(kCountThreads)
    two_count_kernel(const uint32_t *__restrict__ rr, const uint32_t *__restrict__ ub, const int32_t *__restrict__ id,
                     const int32_t *__restrict__ pos1, uint32_t n, int32_t *__restrict__ dom_count)
{
    chain_wait();
    __shared__ uint32_t bits[kStairWords], before[kStairWords], part[32];
    __shared__ __align__(16) uint32_t v[kCountChunk];
    const uint32_t tid = threadIdx.x, b = blockIdx.x * kCountChunk, end = min(n, b + kCountChunk);
    for (uint32_t w = tid; w < kStairWords; w += kCountThreads) bits[w] = 0u;
    __syncthreads();
    for (uint32_t t = tid; t < kCountChunk; t += kCountThreads) {
        v[t] = b + t < end ? rr[b + t] & 0xffffu : 0xffffffffu;
        if (b + t < end) {
            const uint32_t q = static_cast<uint32_t>(pos1[id[b + t]]);
            atomicOr(bits + q / 32u, 1u << (q & 31u));
        }
    }
    __syncthreads();
    constexpr uint32_t kPer = kStairWords / kCountThreads;
    uint32_t c[kPer], sum = 0, total = 0;
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j) {
        c[j] = static_cast<uint32_t>(__popc(bits[tid * kPer + j]));
        sum += c[j];
    }
    uint32_t at = two_block_scan(sum, part, &total);
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j) {
        before[tid * kPer + j] = at;
        at += c[j];
    }
    __syncthreads();
    for (uint32_t p = end + blockIdx.y * kCountThreads + tid; p < n; p += kCountParts * kCountThreads) {
        const uint32_t own = rr[p], u = ub[p]; // u in 1 .. n: positions below u
        const uint32_t w = (u - 1u) / 32u, top = (u - 1u) & 31u;
        uint32_t k = before[w] + static_cast<uint32_t>(__popc(bits[w] & (0xffffffffu >> (31u - top))));
        for (uint32_t q = end; q > b && rr[q - 1u] == own; --q) k -= 1u; // equal points are no dominators
        if (k) atomicAdd(dom_count + id[p], static_cast<int32_t>(k));
    }
    if (blockIdx.y != kCountParts - 1u) return;
    for (uint32_t p = b + tid; p < end; p += kCountThreads) {
        const uint32_t own = rr[p], mine = own & 0xffffu, m = p - b;
        uint32_t k = 0, t = 0;
        for (; t + 4u <= m; t += 4u) {
            const uint4 q = *reinterpret_cast<const uint4 *>(v + t);
            k += (q.x <= mine) + (q.y <= mine) + (q.z <= mine) + (q.w <= mine);
        }
        for (; t < m; ++t) k += v[t] <= mine;
        for (uint32_t q = p; q > b && rr[q - 1u] == own; --q) k -= 1u;
        if (k) atomicAdd(dom_count + id[p], static_cast<int32_t>(k));
    }
}

bool two_fits(uint32_t n, uint32_t m)
{
    return m == 2u && n > kSmallPoints && n <= kTwoPoints;
}

// The fronts (and out.dom_count, with counts) of n points of 2 objectives; keys
// as order_keys_kernel writes them. need: fronts that begin at or after it keep
// their places in front_offsets and rank, and are not listed in front_indices.
// base: two_scratch_bytes(n).
int launch_two_survival(void *base, long long *keys, peel_state *st, const double *pts, uint32_t n,
                        const survival_out &out, bool counts, uint32_t need, int num_sms, cudaStream_t s,
                        uint64_t *launches, uint32_t spin_limit = kTwoSpins)
{
    const two_scratch sc = carve_two_scratch(base, n);
    const int pl = launch_positions(pts, n, 2u, 0u, 2u, sc.runs, sc.pos, num_sms, s);
    PGX_CUDA(cudaGetLastError());
    const unsigned g = static_cast<unsigned>(blocks_for(n, 128, num_sms));
    PGX_CUDA(launch_chained(two_scatter_kernel, g, 128, 0, s, pts, n, sc.pos, keys, sc.ord, sc.deep, out.front_offsets,
                            st));
    PGX_CUDA(launch_chained(two_place_kernel, g, 128, 0, s, keys, n, sc));
    if (counts) {
        PGX_CUDA(cudaMemsetAsync(out.dom_count, 0, static_cast<size_t>(n) * sizeof(int32_t), s));
        const dim3 grid((n + kCountChunk - 1u) / kCountChunk, kCountParts);
        PGX_CUDA(launch_chained(two_count_kernel, grid, kCountThreads, 0, s, sc.rr, sc.ub, sc.id, sc.pos + n, n,
                                out.dom_count));
        ++*launches;
    }
    const uint32_t rows = (n + 31u) / 32u, per = 2u * kTwoBlocks * kTwoWarps, q = (rows + per - 1u) / per;
    const auto peel = q <= 1u   ? two_peel_kernel<1>
                      : q == 2u ? two_peel_kernel<2>
                      : q == 3u ? two_peel_kernel<3>
                                : two_peel_kernel<4>;
    static_assert(kTwoRows == 8u, "four registers hold a warp's rows");
    PGX_CUDA(launch_chained(peel, kTwoBlocks, kTwoWarps * 32, 0, s, sc, n, spin_limit, out.n_fronts, st));
    PGX_CUDA(cudaFuncSetAttribute(two_lists_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(two_lists_smem(kTwoPoints))));
    PGX_CUDA(launch_chained(two_lists_kernel, 1, kTwoThreads, two_lists_smem(n), s, sc, n, out.front_offsets,
                            out.n_fronts));
    PGX_CUDA(launch_chained(two_stairs_kernel, static_cast<unsigned>(num_sms * 2), kStairThreads, 0, s, sc, n,
                            out.front_offsets, out.n_fronts, out.rank));
    PGX_CUDA(launch_chained(two_ranges_kernel, g, 128, 0, s, sc, n, out.front_offsets, out.n_fronts));
    PGX_CUDA(cudaFuncSetAttribute(two_order_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(two_order_smem(kTwoPoints))));
    PGX_CUDA(launch_chained(two_order_kernel, 1, kTwoThreads, two_order_smem(n), s, sc, n, need, out.front_offsets,
                            out.n_fronts, out.front_indices));
    *launches += static_cast<uint64_t>(pl) + 7u;
    return PGX_OK;
}

} // namespace
} // namespace pgx

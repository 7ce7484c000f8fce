// Non-dominated sorting and crowding of a small population (n <= kSmallPoints,
// m <= kSmallObjectives) by one thread block in one launch: every step of the
// general pass -- order keys, dominance bit matrix, counts, front peeling in
// the reference's order, crowding distances -- with block barriers between
// them instead of launches and grid barriers. Included by survival.cu.
//
// Thread j owns point j, so that warp w's ballots are word w of every bit set.
// The matrix and the keys are in shared memory (n = 1024, m = 8: 196 KB); the
// sort areas of the crowding step reuse the matrix's room. Beyond
// kSmallOwnMatrix points the pair tests, n^2 / 2 on one SM otherwise (1000 x 3:
// 100 us), come from a kernel on all of them before. Up to kSmallCrowd points the
// block sorts the fronts too: short ones by one warp each, all at the same time,
// the one that may be longer by the whole block; beyond, front_crowding_kernel
// gives each front a block.
//
// What bounds it: dependent instructions of few warps, in the exact sorts of
// the crowding (700 cycles per partition of 17 to 33 members) and in the peel
// (2700 cycles per front). By the general pass and now, us: 200 x 2 points in 12
// layers 135, 30, in one 84, 31; 512 x 3 in 10 114, 68; 1000 x 3 in 10 134, 94;
// 1024 x 2 in 40 278, 114. Beyond kSmallPoints a block has no thread per point.
#pragma once

namespace pgx
{
namespace
{

constexpr uint32_t kSmallPoints = 1024;
constexpr uint32_t kSmallObjectives = 8;
constexpr int kSmallThreads = 1024;
// Longest front one warp sorts: the block is quicker on one of more than
// kOneWarpFront members (one of 200: 31 against 40 us in all), and no two of
// these fit into the kSmallCrowd points that the block sorts at all.
constexpr int kOneWarpFront = 128;

// The sort arrays of all fronts, by position in front order: a front works in
// its own slice, whichever warp takes it.
struct warp_sort_area {
    long long *k;      // n
    int32_t *v;        // n
    int *pos_l, *pos_r; // n each
    int *stack;        // 3 (n / 16 + 1): ranges to come (first, last, depth budget); L / 16 for a front of L suffice,
                       // as ranges of at most 16 never wait
};

// std::sort's permutation (introsort.cuh) of x[0 .. n), n <= kOneWarpFront, by one
// warp: the ranges longer than 16 one after the other from a stack (they are
// disjoint, so at most kOneWarpFront / 17 wait), the shorter ones as they appear.
static_assert(kOneWarpFront <= dev::kShortRange, "the warp's partitions are short ones");
__device__ void warp_std_sort(const dev::sort_view<long long> &x, int n, const dev::sort_work &w, int *stack, int *err)
{
    const unsigned lane = threadIdx.x & 31u;
    if (n <= 16) {
        dev::halfwarp_leaf_sort(x, 0, lane < 16u ? n : 0);
        return;
    }
    int top = 0, first = 0, last = n, depth = 2 * dev::floor_log2_int(n);
    for (;;) {
        if (depth == 0) {
            if (lane == 0) dev::heap_sort(x, first, last);
            __syncwarp();
        } else {
            const int cut = dev::warp_partition_short(x, first, last, w, err);
            const int la = lane < 16u ? first : cut, len = lane < 16u ? cut - first : last - cut;
            dev::halfwarp_leaf_sort(x, la, len <= 16 ? len : 0);
            --depth;
            const bool lower = cut - first > 16, upper = last - cut > 16;
            if (lower && upper) {
                if (lane == 0) {
                    stack[3 * top] = cut;
                    stack[3 * top + 1] = last;
                    stack[3 * top + 2] = depth;
                }
                ++top;
                __syncwarp();
                last = cut;
                continue;
            }
            if (lower) {
                last = cut;
                continue;
            }
            if (upper) {
                first = cut;
                continue;
            }
        }
        if (top == 0) return;
        --top;
        first = stack[3 * top];
        last = stack[3 * top + 1];
        depth = stack[3 * top + 2];
        __syncwarp();
    }
}

// front_crowding for a front of 2 <= L <= kOneWarpFront members by one warp, the
// distances into s_cd (by point).
__device__ void warp_front_crowding(uint32_t n, uint32_t m, const long long *keys, const uint16_t *members, int L,
                                    const warp_sort_area &a, int *err, double *s_cd)
{
    const int lane = static_cast<int>(threadIdx.x & 31u);
    dev::sort_work w{};
    w.pos_l = a.pos_l;
    w.pos_r = a.pos_r;
    for (int p = lane; p < L; p += 32) {
        a.v[p] = members[p];
        s_cd[members[p]] = 0.0;
    }
    __syncwarp();
    for (uint32_t k = 0; k < m; ++k) {
        for (int p = lane; p < L; p += 32) a.k[p] = keys[k * n + static_cast<uint32_t>(a.v[p])];
        __syncwarp();
        warp_std_sort(dev::sort_view<long long>{a.k, a.v}, L, w, a.stack, err);
        __syncwarp();
        const double df = key_value(a.k[L - 1]) - key_value(a.k[0]);
        for (int p = 1 + lane; p < L - 1; p += 32) s_cd[a.v[p]] += (key_value(a.k[p + 1]) - key_value(a.k[p - 1])) / df;
        __syncwarp();
        if (lane == 0) {
            s_cd[a.v[0]] = HUGE_VAL;
            s_cd[a.v[L - 1]] = HUGE_VAL;
        }
        __syncwarp();
    }
}

struct small_args {
    const double *pts;
    uint32_t n, m;
    long long *keys; // n x m order keys, objective-major, for the kernels that follow (nullable)
    int32_t *rank, *dom_count, *front_offsets, *front_indices, *n_fronts;
    double *cd; // crowding distances, nullable
    int crowd_mode;
    peel_state *st;     // cleared here
    const uint32_t *Dt; // rows of small_row_words(n) words by small_dominance_kernel; null: built here
};

__host__ __device__ constexpr uint32_t small_row_words(uint32_t n) // words per row of the matrix, odd: a column of rows meets every bank
{
    return ((n + 31u) / 32u) | 1u;
}

// Threads of the block: one per point, at least 512 (a warp per member of a front, per front of the crowding).
constexpr int small_threads(uint32_t n)
{
    return n <= 512u ? 512 : kSmallThreads;
}

constexpr size_t small_smem(uint32_t n, uint32_t m, bool crowd) // grows with n
{
    const size_t keys = align256(static_cast<size_t>(n) * m * sizeof(long long));
    const size_t matrix = align256(static_cast<size_t>(n) * small_row_words(n) * sizeof(uint32_t));
    size_t sorts = 0;
    if (crowd) {
        sorts = align256(n * (sizeof(long long) + 3u * sizeof(int)) + 3u * (n / 16u + 1u) * sizeof(int));
        if (n > static_cast<uint32_t>(kOneWarpFront) && sorts < align256(kSortSmemBytes)) sorts = align256(kSortSmemBytes);
    }
    return keys + (matrix > sorts ? matrix : sorts);
}

// One warp: the pair tests of points 32 bi + lane against points 32 bj .. 32
// bj + 31, both directions at once (dominance_sym_kernel), into the rows of
// both sides. key(k, i): the order key of point i in objective k.
template <int MM, typename F>
__device__ __forceinline__ void small_tile(uint32_t bi, uint32_t bj, uint32_t n, uint32_t m, uint32_t *Dt, uint32_t R,
                                           const F &key)
{
    constexpr int KM = MM > 0 ? MM : static_cast<int>(kSmallObjectives);
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t i = bi * 32u + lane, J0 = bj * 32u;
    const bool iv = i < n;
    long long ik[KM], jk[KM]; // this lane's point of either side; the other's go round by shuffles
#pragma unroll
    for (int k = 0; k < KM; ++k) {
        const bool kv = MM > 0 || static_cast<uint32_t>(k) < m;
        ik[k] = iv && kv ? key(static_cast<uint32_t>(k), i) : 0;
        jk[k] = kv && J0 + lane < n ? key(static_cast<uint32_t>(k), J0 + lane) : 0;
    }
    const uint32_t jn = min(32u, n - J0);
    uint32_t row_i = 0u, word = 0u; // word: lane jj keeps row J0 + jj's
    for (uint32_t jj = 0; jj < jn; ++jj) {
        bool any_lt = false, any_gt = false;
#pragma unroll
        for (int k = 0; k < KM; ++k) {
            if (MM > 0 || static_cast<uint32_t>(k) < m) {
                const long long b = __shfl_sync(kFull, jk[k], static_cast<int>(jj));
                any_lt |= ik[k] < b;
                any_gt |= ik[k] > b;
            }
        }
        const uint32_t bal = __ballot_sync(kFull, iv && any_lt && !any_gt);
        if (lane == jj) word = bal;
        row_i |= static_cast<uint32_t>(iv && any_gt && !any_lt) << jj;
    }
    if (lane < jn) Dt[static_cast<size_t>(J0 + lane) * R + bi] = word;
    if (bi != bj && iv) Dt[static_cast<size_t>(i) * R + bj] = row_i;
}

// Tile t of the lower triangle, row by row: bi <= bj
__device__ __forceinline__ void small_tile_of(uint32_t t, uint32_t &bi, uint32_t &bj)
{
    bj = static_cast<uint32_t>((sqrtf(8.0f * static_cast<float>(t) + 1.0f) - 1.0f) * 0.5f);
    while (bj * (bj + 1u) / 2u > t) --bj;
    while ((bj + 1u) * (bj + 2u) / 2u <= t) ++bj;
    bi = t - bj * (bj + 1u) / 2u;
}

// The matrix on every SM, a warp per tile, for populations whose n^2 / 2 pair
// tests would take one block longer than a launch (1000 x 3: 100 us there).
constexpr uint32_t kSmallOwnMatrix = 160;
constexpr int kSmallTileThreads = 128;

template <int MM>
__global__ void __launch_bounds__(kSmallTileThreads)
    small_dominance_kernel(const double *__restrict__ pts, uint32_t n, uint32_t m, uint32_t *__restrict__ Dt)
{
    chain_wait();
    const uint32_t W = (n + 31u) / 32u;
    const uint32_t t = blockIdx.x * (kSmallTileThreads / 32) + (threadIdx.x >> 5);
    if (t >= W * (W + 1u) / 2u) return;
    uint32_t bi, bj;
    small_tile_of(t, bi, bj);
    small_tile<MM>(bi, bj, n, m, Dt, small_row_words(n),
                   [&](uint32_t k, uint32_t i) { return order_key(pts[static_cast<size_t>(i) * m + k]); });
}

// MM: the number of objectives, or 0 for any m up to kSmallObjectives.
template <int MM>
__global__ void __launch_bounds__(kSmallThreads, 1) small_survival_kernel(small_args a)
{
    chain_wait();
    extern __shared__ __align__(256) unsigned char small_mem[];
    __shared__ uint32_t s_rem[32], s_prev[32];
    __shared__ uint16_t s_pos[kSmallPoints];               // positions in the previous front
    __shared__ __align__(16) uint32_t s_new[kSmallPoints]; // the new front's members: key << 16 | index
    __shared__ uint16_t s_front[kSmallPoints];             // front_indices
    __shared__ uint16_t s_off[kSmallPoints + 1];           // front_offsets
    __shared__ double s_cd[kSmallPoints];
    __shared__ int s_cnt[2];
    __shared__ dev::sort_ctl ctl;
    __shared__ int slots[kSortWarps * 64];
    const uint32_t n = a.n, m = MM > 0 ? static_cast<uint32_t>(MM) : a.m;
    const uint32_t W = (n + 31u) / 32u, R = small_row_words(n);
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const uint32_t j = threadIdx.x;
    long long *keys = reinterpret_cast<long long *>(small_mem);
    unsigned char *area = small_mem + align256(static_cast<size_t>(n) * m * sizeof(long long));
    uint32_t *Dt = reinterpret_cast<uint32_t *>(area); // row j, word w: the points of word w that dominate j
    for (uint32_t t = threadIdx.x; t < n * m; t += blockDim.x) {
        const uint32_t i = t / m, k = t - i * m;
        const long long key = order_key(a.pts[t]);
        keys[k * n + i] = key;
        if (a.keys) a.keys[k * n + i] = key;
    }
    if (a.Dt)
        for (uint32_t t = threadIdx.x; t < n * R; t += blockDim.x) Dt[t] = __ldg(a.Dt + t);
    for (uint32_t t = threadIdx.x; t <= n; t += blockDim.x) a.front_offsets[t] = 0;
    for (uint32_t t = threadIdx.x; t < sizeof(peel_state) / sizeof(int); t += blockDim.x)
        reinterpret_cast<int *>(a.st)[t] = 0;
    if (threadIdx.x < 32u) {
        const uint32_t lo = 32u * threadIdx.x;
        s_rem[threadIdx.x] = lo + 32u <= n ? kFull : (lo < n ? (1u << (n - lo)) - 1u : 0u);
    }
    if (threadIdx.x < 2u) s_cnt[threadIdx.x] = 0;
    __syncthreads();
    if (!a.Dt) {
        for (uint32_t t = warp; t < W * (W + 1u) / 2u; t += nwarps) {
            uint32_t bi, bj;
            small_tile_of(t, bi, bj);
            small_tile<MM>(bi, bj, n, m, Dt, R, [&](uint32_t k, uint32_t i) { return keys[k * n + i]; });
        }
        __syncthreads();
    }
    const uint32_t *row = Dt + static_cast<size_t>(j < n ? j : 0u) * R;
    if (j < n) {
        int c = 0;
        for (uint32_t w = 0; w < W; ++w) c += __popc(row[w]);
        a.dom_count[j] = c;
    }
    // ---- peel: a thread keeps an unassigned dominator of its point and looks
    // for the next one, from the word of the last, when that one has gone
    bool open = j < n;
    uint32_t wit_w = 0, wit_b = 0, off = 0;
    int k = 0;
    for (;; ++k) {
        bool member = false;
        if (open && (k == 0 || !(s_rem[wit_w] >> wit_b & 1u))) {
            member = true;
            for (uint32_t w = wit_w; w < W; ++w) {
                const uint32_t x = row[w] & s_rem[w];
                if (x) {
                    wit_w = w;
                    wit_b = static_cast<uint32_t>(31 - __clz(x));
                    member = false;
                    break;
                }
            }
        }
        const uint32_t bal = __ballot_sync(kFull, member);
        uint32_t base = 0;
        if (lane == 0 && bal) base = static_cast<uint32_t>(atomicAdd(&s_cnt[k & 1], __popc(bal)));
        base = __shfl_sync(kFull, base, 0);
        if (member) s_new[base + __popc(bal & ((1u << lane) - 1u))] = j;
        __syncthreads(); // the members are listed
        const uint32_t L = static_cast<uint32_t>(s_cnt[k & 1]);
        if (L == 0u) break; // every point is assigned
        if (threadIdx.x == 0) {
            s_cnt[(k + 1) & 1] = 0;
            s_off[k] = static_cast<uint16_t>(off);
            a.front_offsets[k + 1] = static_cast<int32_t>(off + L);
        }
        if (k > 0) {
            // a member's key: the highest position, in the previous front, of one of its dominators; a warp per
            // member, a lane per word
            for (uint32_t t = warp; t < L; t += nwarps) {
                const uint32_t q = s_new[t];
                uint32_t x = lane < W ? Dt[static_cast<size_t>(q) * R + lane] & s_prev[lane] : 0u, key = 0;
                while (x) {
                    key = max(key, static_cast<uint32_t>(s_pos[lane * 32u + static_cast<uint32_t>(__ffs(x) - 1)]));
                    x &= x - 1u;
                }
                key = __reduce_max_sync(kFull, key);
                if (lane == 0) s_new[t] = key << 16 | q;
            }
            __syncthreads(); // every read of the previous front is done
        }
        if (lane == 0) {
            s_prev[warp] = bal;
            s_rem[warp] &= ~bal;
        }
        // positions: the members with a smaller (key, index); the packed words are distinct
        if (k > 0 && L <= 256u) {
            for (uint32_t t = warp; t < L; t += nwarps) {
                const uint32_t mine = s_new[t];
                uint32_t p = 0;
                for (uint32_t u = lane; u < L; u += 32u) p += s_new[u] < mine;
                p = __reduce_add_sync(kFull, p);
                if (lane == 0) {
                    const uint32_t q = mine & 0xffffu;
                    a.rank[q] = k;
                    a.front_indices[off + p] = static_cast<int32_t>(q);
                    s_front[off + p] = static_cast<uint16_t>(q);
                    s_pos[q] = static_cast<uint16_t>(p);
                }
            }
        } else if (k > 0) {
            if (j < L) {
                const uint32_t mine = s_new[j];
                uint32_t p = 0, t = 0;
                for (; t + 4u <= L; t += 4u) {
                    const uint4 q = *reinterpret_cast<const uint4 *>(s_new + t);
                    p += (q.x < mine) + (q.y < mine) + (q.z < mine) + (q.w < mine);
                }
                for (; t < L; ++t) p += s_new[t] < mine;
                const uint32_t q = mine & 0xffffu;
                a.rank[q] = k;
                a.front_indices[off + p] = static_cast<int32_t>(q);
                s_front[off + p] = static_cast<uint16_t>(q);
                s_pos[q] = static_cast<uint16_t>(p);
            }
        } else {
            // the first front is in index order: from the bit sets
            __syncthreads();
            if (member) {
                uint32_t p = static_cast<uint32_t>(__popc(bal & ((1u << lane) - 1u)));
                for (uint32_t w = 0; w < warp; ++w) p += static_cast<uint32_t>(__popc(s_prev[w]));
                a.rank[j] = 0;
                a.front_indices[p] = static_cast<int32_t>(j);
                s_front[p] = static_cast<uint16_t>(j);
                s_pos[j] = static_cast<uint16_t>(p);
            }
        }
        if (member) open = false;
        off += L;
        __syncthreads(); // positions and bit sets for the next front
    }
    if (threadIdx.x == 0) {
        s_off[k] = static_cast<uint16_t>(off);
        *a.n_fronts = k;
        a.st->n_fronts = k;
    }
    if (a.cd == nullptr) return;
    __syncthreads();
    // ---- crowding (the matrix's room is free)
    long long *ak = reinterpret_cast<long long *>(area);
    int *ai = reinterpret_cast<int *>(ak + n);
    for (int f = static_cast<int>(warp); f < k; f += static_cast<int>(nwarps)) {
        const int L = s_off[f + 1] - s_off[f];
        const uint16_t *mem = s_front + s_off[f];
        if (L == 1 || (L == 2 && a.crowd_mode == kCrowdNsga2)) {
            if (static_cast<int>(lane) < L) s_cd[mem[lane]] = a.crowd_mode == kCrowdNsga2 ? HUGE_VAL : 0.0;
        } else if (L <= kOneWarpFront) {
            const int at = s_off[f];
            const warp_sort_area mine{ak + at, ai + at, ai + n + at, ai + 2u * n + at, ai + 3u * n + 3 * (at / 16)};
            warp_front_crowding(n, m, keys, mem, L, mine, &a.st->sort_err, s_cd);
        }
    }
    __syncthreads();
    for (int f = 0; f < k; ++f) {
        const int L = s_off[f + 1] - s_off[f];
        if (L <= kOneWarpFront) continue; // uniform: the same front for every thread
        const sort_area<long long> sa = pick_area<long long>(area, L, nullptr, nullptr, nullptr, nullptr);
        front_crowding(n, m, keys, a.front_indices + s_off[f], L, sa, &ctl, slots, &a.st->sort_err, s_cd);
    }
    __syncthreads();
    if (j < n) a.cd[j] = s_cd[j];
}

bool small_fits(uint32_t n, uint32_t m, bool crowd)
{
    return n <= kSmallPoints && m >= 1u && m <= kSmallObjectives && (!crowd || m >= 2u);
}

// Whether the block computes the crowding distances too: it sorts its larger
// fronts one after the other, where front_crowding_kernel gives each a block
// (200 x 3 in 1 / 4 / 12 layers: 43 / 43 / 34 us by the block, 50 / 43 / 39 apart;
// 300 x 4: 71 / 92 / 101 and 81 / 75 / 72; 743 x 4: 123 / 203 / 149 and 122 / 115
// / 102; by the general pass 146 / 133 / 115).
constexpr uint32_t kSmallCrowd = 256;

bool small_crowd_inside(uint32_t n)
{
    return n <= kSmallCrowd;
}

// Dt: room for n rows of small_row_words(n) words. Returns the kernels launched through *launches.
template <int MM>
int launch_small_survival_mm(small_args a, uint32_t *Dt, cudaStream_t s, uint64_t *launches)
{
    const size_t smem = small_smem(a.n, a.m, a.cd != nullptr);
    a.Dt = nullptr;
    if (a.n > kSmallOwnMatrix) {
        const uint32_t W = (a.n + 31u) / 32u, tiles = W * (W + 1u) / 2u, per = kSmallTileThreads / 32;
        PGX_CUDA(launch_chained(small_dominance_kernel<MM>, (tiles + per - 1u) / per, kSmallTileThreads, 0, s, a.pts,
                                a.n, a.m, Dt));
        a.Dt = Dt;
        ++*launches;
    }
    // one limit for all calls: other contexts' threads launch the kernel at the same time
    constexpr uint32_t most_m = MM > 0 ? static_cast<uint32_t>(MM) : kSmallObjectives;
    constexpr size_t all = small_smem(kSmallPoints, most_m, false), inside = small_smem(kSmallCrowd, most_m, true);
    PGX_CUDA(cudaFuncSetAttribute(small_survival_kernel<MM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(all > inside ? all : inside)));
    PGX_CUDA(launch_chained(small_survival_kernel<MM>, 1, small_threads(a.n), smem, s, a));
    ++*launches;
    return PGX_OK;
}

int launch_small_survival(const small_args &a, uint32_t *Dt, cudaStream_t s, uint64_t *launches)
{
    switch (a.m) {
        case 2u: return launch_small_survival_mm<2>(a, Dt, s, launches);
        case 3u: return launch_small_survival_mm<3>(a, Dt, s, launches);
        default: return launch_small_survival_mm<0>(a, Dt, s, launches);
    }
}

} // namespace
} // namespace pgx

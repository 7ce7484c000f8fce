// Hypervolume of 2 or 3 objectives on the GPU (pagmo's hypervolume::compute,
// src/utils/hypervolume.cpp:203-228, which picks hv2d for two objectives and
// hv3d for three: src/utils/hv_algos/hv_hv2d.cpp:48-68, hv_hv3d.cpp:75-116),
// and the C ABI of the hypervolume queries: compute (4 or more objectives by
// hvwfg in hv_wfg.cu), exclusive, contributions and the least and greatest
// contributors (hypervolume.cpp:249-401).
//
// The dominated region is summed as non-negative slabs (no cancellation):
//  - 2D: with the points sorted by y, the staircase width W(t) = max over the
//    first t+1 points of (r_x - x), and HV = sum_t (y_{t+1} - y_t) W(t) with
//    y_n = r_y (hv2d's own sweep, summed as a tree).
//  - 3D: with the points taken in z order, point i adds to the 2D region
//    dominated so far the area G_i of its rectangle that no earlier point
//    covers, and that area counts from z_i up: HV = sum_i G_i (r_z - z_i).
//    G_i is a walk along the staircase of the earlier points from point i to
//    the first of them at least as wide. All points at once: a block of
//    consecutive points (in z order) first filters all points down to those
//    that one of its walks can meet.
// Order: positions in each coordinate's order (sort_pos.cuh, ties by index);
// a tie does not change any slab (its step is zero). The widths r_x - x are
// non-negative on valid input, so their running maximum is taken on integers:
// the IEEE bit patterns (2D) or the reversed x positions (3D).
#include "fitness_dev.cuh"
#include "sort_pos.cuh"
#include "pgx_internal.cuh"

#include <algorithm>
#include <climits>
#include <cmath>
#include <sstream>
#include <string>
#include <vector>

namespace pgx
{
namespace
{

constexpr unsigned kFull = 0xffffffffu;

// points into y order: ys and, for 2D, the widths r_x - x as bits; for 3D
// the 32-bit width keys (n - 1 - the x rank: a larger key never has a smaller
// width) beside the z ranks, the x values, and the z values in z order
__global__ void hv_scatter_kernel(const double *__restrict__ pts, uint32_t n, uint32_t m, double rx,
                                  const int32_t *__restrict__ rank, double *__restrict__ ys,
                                  long long *__restrict__ wbits, int2 *__restrict__ wk, double *__restrict__ xs,
                                  double *__restrict__ zs)
{
    chain_wait();
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const double *p = pts + static_cast<uint64_t>(t) * m;
        const int32_t ry = rank[t];
        ys[ry] = p[1];
        if (m == 3u) {
            const int32_t rz = rank[static_cast<uint64_t>(n) + t], rxk = rank[2ull * n + t];
            wk[ry] = make_int2(static_cast<int>(n) - 1 - rxk, rz);
            xs[ry] = p[0];
            zs[rz] = p[2];
        } else {
            wbits[ry] = __double_as_longlong(rx == p[0] ? 0.0 : rx - p[0]); // (also where both are infinite)
        }
    }
}

__device__ __forceinline__ long long warp_incl_max(long long v)
{
    const unsigned lane = threadIdx.x & 31u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long u = __shfl_up_sync(kFull, v, o);
        if (static_cast<int>(lane) >= o && u > v) v = u;
    }
    return v;
}

// 2D: A = sum_t (y_{t+1} - y_t) * max_{t' <= t} w[t'] over the points in y
// order (y_n = r_y). The running maximum W changes only at "records" (a point
// widening the staircase), so A is summed run by run, W_run * (y at the next
// record - y at this one), the last run ending at r_y: two FP64 operations per
// record instead of two per point. The points are cut into chunks of
// kAreaChunk, one block each; a run that crosses into a chunk is cut at the
// chunk's first point (a sum of two non-negative parts). hv_chunk_max_kernel
// gives each chunk's maximum width, of which a chunk takes the earlier ones'
// maximum; the partial sums are added by hv_sum_kernel. 60000 points: 3.3 us
// and 6.6 us (2226 us by one warp walking all points).
constexpr int kAreaThreads = 256;
constexpr uint32_t kAreaChunk = 2048;

__device__ __forceinline__ long long block_max(long long v, long long *part)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(kFull, v, o));
    if ((threadIdx.x & 31u) == 0u) part[threadIdx.x >> 5] = v;
    __syncthreads();
    v = part[threadIdx.x & (kAreaThreads / 32 - 1)];
#pragma unroll
    for (int o = kAreaThreads / 64; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(kFull, v, o));
    __syncthreads(); // part is free again
    return v;
}

__global__ void __launch_bounds__(kAreaThreads)
    hv_chunk_max_kernel(const long long *__restrict__ wbits, uint32_t n, long long *__restrict__ chunk_max)
{
    chain_wait();
    __shared__ long long part[kAreaThreads / 32];
    const uint32_t t0 = blockIdx.x * kAreaChunk, t1 = min(n, t0 + kAreaChunk);
    long long v = 0;
    for (uint32_t t = t0 + threadIdx.x; t < t1; t += kAreaThreads) v = max(v, wbits[t]);
    v = block_max(v, part);
    if (threadIdx.x == 0) chunk_max[blockIdx.x] = v;
}

__global__ void __launch_bounds__(kAreaThreads)
    hv_area2_kernel(const double *__restrict__ ys, const long long *__restrict__ wbits,
                    const long long *__restrict__ chunk_max, uint32_t n, double ry, double *__restrict__ term)
{
    chain_wait();
    constexpr uint32_t kPer = kAreaChunk / kAreaThreads;
    constexpr uint32_t kWarps = kAreaThreads / 32;
    __shared__ long long part[kWarps];
    __shared__ double head_y[kWarps]; // the first record's y of each warp's points (r_y's stand-in: no record)
    __shared__ uint32_t head_has[kWarps];
    __shared__ double sums[kWarps];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t t0 = blockIdx.x * kAreaChunk, t1 = min(n, t0 + kAreaChunk);
    // the widest point before the chunk
    long long before = 0;
    for (uint32_t b = threadIdx.x; b < blockIdx.x; b += kAreaThreads) before = max(before, chunk_max[b]);
    before = block_max(before, part);
    // each thread kPer consecutive points
    const uint32_t p0 = t0 + threadIdx.x * kPer;
    long long w[kPer];
    long long mine = 0;
#pragma unroll
    for (uint32_t u = 0; u < kPer; ++u) {
        w[u] = p0 + u < t1 ? wbits[p0 + u] : 0;
        mine = max(mine, w[u]);
    }
    long long incl = warp_incl_max(mine);
    if (lane == 31u) part[warp] = incl;
    __syncthreads();
    long long carry = before;
    for (uint32_t q = 0; q < warp; ++q) carry = max(carry, part[q]);
    long long run = __shfl_up_sync(kFull, incl, 1);
    if (lane == 0) run = 0;
    run = max(run, carry); // the maximum before this thread's points
    // the chunk starts a run of its own with the width found before it
    double a = 0.0, pend_w = __longlong_as_double(run), pend_y = 0.0, first_y = 0.0;
    const double run_w = pend_w;
    bool has = false;
#pragma unroll
    for (uint32_t u = 0; u < kPer; ++u) {
        if (w[u] > run) {
            const double y = ys[p0 + u];
            if (has && y != pend_y) a = fma(pend_w, y - pend_y, a); // (either side of a product may be infinite)
            if (!has) first_y = y;
            has = true;
            run = w[u];
            pend_w = __longlong_as_double(run);
            pend_y = y;
        }
    }
    // the y where the run open at a thread's end closes: the next record of
    // this warp, of a later warp, or the chunk's end
    const double end_y = t1 < n ? ys[t1] : ry;
    const uint32_t b = __ballot_sync(kFull, has);
    const double next_in_warp = __shfl_sync(kFull, first_y, b & ~((2u << lane) - 1u) ? __ffs(b & ~((2u << lane) - 1u)) - 1 : 0);
    const double warp_first = __shfl_sync(kFull, first_y, b ? __ffs(b) - 1 : 0);
    if (lane == 0) {
        head_y[warp] = warp_first;
        head_has[warp] = b ? 1u : 0u;
    }
    __syncthreads();
    double close = end_y;
    for (uint32_t q = kWarps; q-- > warp + 1u;)
        if (head_has[q]) close = head_y[q];
    if (b & ~((2u << lane) - 1u)) close = next_in_warp;
    // (an empty run is skipped: its width may be infinite)
    if (has && pend_w > 0.0 && close != pend_y) a = fma(pend_w, close - pend_y, a);
    // the run that reaches into the chunk: from the chunk's first point to its first record
    if (threadIdx.x == 0 && run_w > 0.0) {
        double stop = end_y;
        for (uint32_t q = kWarps; q-- > 0u;)
            if (head_has[q]) stop = head_y[q];
        if (stop != ys[t0]) a = fma(run_w, stop - ys[t0], a);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(kFull, a, o);
    if (lane == 0) sums[warp] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (uint32_t q = 0; q < kWarps; ++q) s += sums[q];
        term[blockIdx.x] = s;
    }
}

// 3D: one block per `levels` consecutive points in z order [i0, i0 + levels),
// one thread per point for its area, all threads for the filter. In y order,
// the staircase of the points before point i in z order is the running maximum
// of their widths; point i's area starts at its y with the staircase's x there
// (nothing when it is at least as wide) and ends at the first point at least
// as wide as itself, with one non-negative product per step of the staircase
// between. A point of z position below i0 is a step for no point of this block
// unless it is one of the staircase of the points below i0 alone (an earlier y
// at least as wide belongs to every walk here). So the filter, which reads
// every point once per block, kLvTile at a time and eight consecutive points
// per thread, keeps two lists in y order: that staircase (widths ascending
// too) and the block's own points. A thread looks up the staircase at its own
// point directly, takes the maximum with the own points before it, and walks
// on through both lists: integer compares, FP64 only for the steps of its own
// area (each point of a front is such a step about once in all). The staircase
// list is walked in pieces when it outgrows its room. A front of 20000 points
// on a sphere: 34 us (919 us when each of n levels summed its whole area
// over all points); the filter's barriers and loads are what is left.
// levels: the power of two that gives every SM two blocks, 8 to kLvLevels
// (fewer per block: more filtering).
constexpr int kLvThreads = 256;
constexpr uint32_t kLvPer = 8;
constexpr uint32_t kLvTile = kLvThreads * kLvPer;
constexpr uint32_t kLvLevels = 128; // most points per block
constexpr uint32_t kLvCap = 3072;   // staircase points: walked once fewer than a tile's room is left
constexpr size_t kLvSmem = kLvCap * (2u * sizeof(double) + sizeof(int) + sizeof(uint32_t));

__global__ void __launch_bounds__(kLvThreads)
    hv_levels3_kernel(const double *__restrict__ ys, const int2 *__restrict__ wk, const double *__restrict__ xs,
                      const double *__restrict__ zs, uint32_t n, uint32_t levels, double rx, double ry, double rz,
                      double *__restrict__ term)
{
    chain_wait();
    // the staircase: width keys, positions in y order, coordinates
    extern __shared__ __align__(16) double s_y[];
    double *s_x = s_y + kLvCap;
    int *s_key = reinterpret_cast<int *>(s_x + kLvCap);
    uint32_t *s_at = reinterpret_cast<uint32_t *>(s_key + kLvCap);
    // the block's own points in y order: width key, z position, staircase
    // points before it (in this piece), position in y order
    __shared__ int4 o_e[kLvLevels];
    __shared__ double o_y[kLvLevels], o_x[kLvLevels];
    __shared__ int own_at[kLvLevels]; // by z position: where the point is in o_e
    __shared__ int s_max[kLvThreads / 32];
    __shared__ uint32_t s_cnt[kLvThreads / 32];
    __shared__ double s_sum[kLvThreads / 32];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const int i0 = static_cast<int>(blockIdx.x * levels), i1 = static_cast<int>(min(n, (blockIdx.x + 1u) * levels));
    const int own = i0 + static_cast<int>(threadIdx.x); // this thread's point, by z position
    const bool level = own < i1;
    bool walking = false, done = !level;
    int v = -1, own_k = 0; // the staircase's width key so far, the own point's
    double step_x = rx, step_y = 0.0, own_x = 0.0, a = 0.0;
    // the step up to y; one of no width or no height adds nothing, even where
    // the other side, or both ends of this one, are infinite
    const auto add = [&](double y) {
        if (step_x != own_x && y != step_y) a = fma(step_x - own_x, y - step_y, a);
    };
    int carry = -1;                  // the widest earlier point of z position below i0
    uint32_t ns = 0, q0 = 0, q1 = 0; // staircase points, own points [q0, q1) of the piece
    if (level) own_at[threadIdx.x] = INT_MAX;
    const auto load = [&](uint32_t p, int2(&e)[kLvPer]) {
        if (p + kLvPer <= n) {
            const int4 *src = reinterpret_cast<const int4 *>(wk + p);
#pragma unroll
            for (uint32_t u = 0; u < kLvPer; u += 2u) {
                const int4 q = __ldg(src + u / 2u);
                e[u] = make_int2(q.x, q.y);
                e[u + 1u] = make_int2(q.z, q.w);
            }
        } else {
#pragma unroll
            for (uint32_t u = 0; u < kLvPer; ++u) e[u] = p + u < n ? __ldg(wk + p + u) : make_int2(-1, INT_MAX);
        }
    };
    int2 e[kLvPer], e_next[kLvPer]; // this tile's points and, in flight, the next one's
    load(threadIdx.x * kLvPer, e_next);
    for (uint32_t t0 = 0; t0 < n; t0 += kLvTile) {
        const uint32_t p0 = t0 + threadIdx.x * kLvPer;
#pragma unroll
        for (uint32_t u = 0; u < kLvPer; ++u) e[u] = e_next[u];
        load(p0 + kLvTile, e_next);
        int mine = -1;
        uint32_t keep_o = 0;
#pragma unroll
        for (uint32_t u = 0; u < kLvPer; ++u) {
            if (e[u].y < i0)
                mine = max(mine, e[u].x);
            else if (e[u].y < i1)
                keep_o |= 1u << u;
        }
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int q = __shfl_up_sync(kFull, incl, o);
            if (static_cast<int>(lane) >= o) incl = max(incl, q);
        }
        if (lane == 31u) s_max[warp] = incl;
        __syncthreads();
        int run = __shfl_up_sync(kFull, incl, 1);
        if (lane == 0) run = -1;
        run = max(run, carry);
#pragma unroll
        for (unsigned q = 0; q < kLvThreads / 32; ++q) {
            const int sm = s_max[q];
            if (q < warp) run = max(run, sm);
            carry = max(carry, sm);
        }
        uint32_t keep_s = 0;
#pragma unroll
        for (uint32_t u = 0; u < kLvPer; ++u) {
            if (e[u].y < i0 && e[u].x > run) {
                run = e[u].x;
                keep_s |= 1u << u;
            }
        }
        // kept points (staircase in the low half, own in the high half) of the
        // threads up to this one; at most kLvTile each: no carry between halves
        const uint32_t both = static_cast<uint32_t>(__popc(keep_s)) | static_cast<uint32_t>(__popc(keep_o)) << 16;
        uint32_t upto = both;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t q = __shfl_up_sync(kFull, upto, o);
            if (static_cast<int>(lane) >= o) upto += q;
        }
        if (lane == 31u) s_cnt[warp] = upto;
        __syncthreads();
        uint32_t at = ns + (q1 << 16) + upto - both;
#pragma unroll
        for (unsigned q = 0; q < kLvThreads / 32; ++q) {
            const uint32_t sc = s_cnt[q];
            if (q < warp) at += sc;
            ns += sc & 0xffffu;
            q1 += sc >> 16;
        }
        if (keep_s | keep_o) {
            uint32_t at_s = at & 0xffffu, at_o = at >> 16;
#pragma unroll
            for (uint32_t u = 0; u < kLvPer; ++u) {
                if (keep_s >> u & 1u) {
                    s_key[at_s] = e[u].x;
                    s_at[at_s] = p0 + u;
                    ++at_s;
                } else if (keep_o >> u & 1u) {
                    o_e[at_o] = make_int4(e[u].x, e[u].y, static_cast<int>(at_s), static_cast<int>(p0 + u));
                    own_at[e[u].y - i0] = static_cast<int>(at_o);
                    ++at_o;
                }
            }
        }
        // (the next tile's first barrier comes before its list writes)
        if (ns + kLvTile <= kLvCap && t0 + kLvTile < n) continue;
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < ns; j += kLvThreads) {
            s_y[j] = __ldg(ys + s_at[j]);
            s_x[j] = __ldg(xs + s_at[j]);
        }
        for (uint32_t j = q0 + threadIdx.x; j < q1; j += kLvThreads) {
            o_y[j] = __ldg(ys + o_e[j].w);
            o_x[j] = __ldg(xs + o_e[j].w);
        }
        __syncthreads();
        if (!done) {
            uint32_t sj = 0, oj = q0; // where the walk goes on
            if (!walking) {
                // the staircase up to the own point, or past this piece
                const int at_own = own_at[threadIdx.x];
                const bool here = at_own < static_cast<int>(q1);
                const uint32_t o_end = here ? static_cast<uint32_t>(at_own) : q1;
                const uint32_t s_end = here ? static_cast<uint32_t>(o_e[at_own].z) : ns;
                int from = -1; // an own point's index, or the staircase's last
                if (s_end > 0u && s_key[s_end - 1u] > v) {
                    v = s_key[s_end - 1u];
                    from = static_cast<int>(s_end - 1u);
                }
                int from_o = -1;
                for (uint32_t j = q0; j < o_end; ++j) {
                    const int4 k = o_e[j];
                    if (k.y < own && k.x > v) {
                        v = k.x;
                        from_o = static_cast<int>(j);
                    }
                }
                if (from_o >= 0)
                    step_x = o_x[from_o];
                else if (from >= 0)
                    step_x = s_x[from];
                if (here) {
                    own_k = o_e[at_own].x;
                    own_x = o_x[at_own];
                    step_y = o_y[at_own];
                    walking = true;
                    done = v > own_k; // an earlier point covers it
                    sj = s_end;
                    oj = o_end + 1u;
                }
            }
            while (walking && !done) {
                // the next wider point of either list, in y order (own points only as far as the staircase's)
                while (sj < ns && s_key[sj] <= v) ++sj;
                const bool has_s = sj < ns;
                const int s_pos = has_s ? static_cast<int>(s_at[sj]) : INT_MAX;
                int4 k = make_int4(0, 0, 0, 0);
                bool has_o = false;
                for (; oj < q1; ++oj) {
                    k = o_e[oj];
                    if (k.w > s_pos) break;
                    if (k.y < own && k.x > v) {
                        has_o = true;
                        break;
                    }
                }
                if (!has_s && !has_o) break; // goes on in the next piece, or to r_y
                double x, y;
                if (!has_o) {
                    v = s_key[sj];
                    x = s_x[sj];
                    y = s_y[sj];
                } else {
                    v = k.x;
                    x = o_x[oj];
                    y = o_y[oj];
                }
                add(y);
                step_x = x;
                step_y = y;
                done = v > own_k;
            }
        }
        ns = 0;
        q0 = q1;
    }
    double t = 0.0;
    if (level) {
        if (!done) add(ry);
        const double z = zs[own];
        t = a != 0.0 && rz != z ? (rz - z) * a : 0.0;
    }
    // the block's sum: 128 additions on this SM's FP64 pipe instead of n on hv_sum_kernel's
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(kFull, t, o);
    if (lane == 0) s_sum[warp] = t;
    __syncthreads();
    static_assert(kLvLevels <= 4u * 32u, "the block's points are the first four warps'");
    if (threadIdx.x == 0) term[blockIdx.x] = (s_sum[0] + s_sum[1]) + (s_sum[2] + s_sum[3]);
}

// out = sum of term[0 .. L), none negative, by one block: an integer sum
// (isum.h: within 2^-60 per addition, rounded once), as the last additions of a
// tree of doubles, each rounded at the volume's own size, were most of its error.
constexpr int kHvSumThreads = 256;

__global__ void __launch_bounds__(kHvSumThreads) hv_sum_kernel(const double *__restrict__ term, uint32_t L,
                                                               double *__restrict__ out)
{
    chain_wait();
    __shared__ unsigned long long part_m[kHvSumThreads / 32];
    __shared__ int part_e[kHvSumThreads / 32];
    __shared__ uint32_t part_flags[kHvSumThreads / 32];
    isum::sq_acc s = isum::make();
    for (uint32_t i = threadIdx.x; i < L; i += kHvSumThreads) isum::add(s, isum::magnitude(term[i], s.flags));
    s = dev::group_isum<32>(s, kFull);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (lane == 0u) {
        part_m[warp] = s.m;
        part_e[warp] = s.e;
        part_flags[warp] = s.flags;
    }
    __syncthreads();
    if (warp != 0u) return;
    const bool has = lane < kHvSumThreads / 32;
    s = has ? isum::sq_acc{part_m[lane], part_e[lane], part_flags[lane]} : isum::make();
    s = dev::group_isum<32>(s, kFull);
    if (lane == 0u) *out = isum::value(s);
}

// hypervolume::verify_after_construct and verify_before_compute with
// hv_algorithm::assert_minimisation (src/utils/hypervolume.cpp:406-449,
// src/utils/hv_algos/hv_algorithm.cpp:226-258), on host data.
int hv_check(const double *pts, uint64_t n, uint64_t m, const double *r)
{
    PGX_CHECK(n > 0u, PGX_ERR_INVALID, "Point set cannot be empty.");
    PGX_CHECK(m > 1u, PGX_ERR_INVALID, "Points of dimension > 1 required.");
    for (uint64_t i = 0; i < n * m; ++i)
        PGX_CHECK(!std::isnan(pts[i]), PGX_ERR_INVALID,
                  "A nan value has been encountered in the hypervolume points. Cannot construct the hypervolume object");
    PGX_CHECK(m <= kWfgMaxObjectives, PGX_ERR_NOTIMPL,
              "hypervolume on the GPU: at most " + std::to_string(kWfgMaxObjectives) + " objectives; " +
                  std::to_string(m) + " given");
    for (uint64_t i = 0; i < n; ++i) {
        bool outside = false, all_equal = true;
        for (uint64_t k = 0; k < m; ++k) {
            outside |= r[k] < pts[i * m + k];
            all_equal &= r[k] == pts[i * m + k];
        }
        if (outside || all_equal) {
            std::string sp("("), sr("(");
            for (uint64_t k = 0; k < m; ++k) {
                sp += std::to_string(pts[i * m + k]);
                sr += std::to_string(r[k]);
                sp += k + 1 < m ? ", " : ")";
                sr += k + 1 < m ? ", " : ")";
            }
            std::ostringstream ss;
            ss << "Reference point is invalid: another point seems to be outside the reference point boundary, or "
                  "be equal to it:"
               << std::endl
               << " P[" << i << "]\t= " << sp << std::endl
               << " R\t= " << sr << std::endl;
            set_error(ss.str());
            return PGX_ERR_INVALID;
        }
    }
    return PGX_OK;
}

size_t align256(size_t b)
{
    return (b + 255u) & ~size_t(255);
}

// All kernels on stream s over device points; *d_out receives the volume
// (4 or more objectives: hvwfg, hv_wfg.cu).
int launch_hypervolume(pgx_context *ctx, const double *d_pts, uint32_t n, uint32_t m, const double *r,
                       double *d_out, cudaStream_t s)
{
    if (m >= 4u) return launch_wfg_compute(ctx, d_pts, n, m, r, d_out, s);
    const uint32_t nc = m == 3u ? 3u : 1u; // coordinates ranked: y (and z, x for 3D)
    const int sms = ctx->num_sms;
    const int g1 = static_cast<int>(std::min<uint64_t>((n + 255u) / 256u, static_cast<uint64_t>(sms) * 8u));
    const size_t b_rank = align256(static_cast<size_t>(n) * nc * 4u);
    const size_t b_runs = align256(pos_scratch_bytes(n, nc));
    const size_t b_d = align256(static_cast<size_t>(n) * 8u);
    PGX_TRY(ctx->s_crowd.ensure(b_rank + b_runs + 6u * b_d + 256u));
    char *base = ctx->s_crowd.as<char>();
    void *runs = base;
    int32_t *rank = reinterpret_cast<int32_t *>(base + b_runs);
    char *arr = base + b_rank + b_runs; // six arrays of n doubles
    double *ys = reinterpret_cast<double *>(arr);
    long long *wbits = reinterpret_cast<long long *>(arr + b_d);
    double *zs = reinterpret_cast<double *>(arr + 2u * b_d);
    double *term = reinterpret_cast<double *>(arr + 3u * b_d);
    int2 *wk = reinterpret_cast<int2 *>(arr + 4u * b_d);
    double *xs = reinterpret_cast<double *>(arr + 5u * b_d);
    const int pl = launch_positions(d_pts, n, m, 1u, nc, runs, rank, sms, s);
    PGX_CUDA(cudaGetLastError());
    PGX_CUDA(launch_chained(hv_scatter_kernel, g1, 256, 0, s, d_pts, n, m, r[0], rank, ys, wbits, m == 3u ? wk : nullptr,
                                         m == 3u ? xs : nullptr, m == 3u ? zs : nullptr));
    uint32_t terms = 0; // partial sums, one per block
    if (m == 3u) {
        uint32_t levels = 8u;
        while (levels < kLvLevels && static_cast<uint64_t>(levels) * 2u * sms < n) levels *= 2u;
        terms = (n + levels - 1u) / levels;
        PGX_CUDA(cudaFuncSetAttribute(hv_levels3_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(kLvSmem)));
        PGX_CUDA(launch_chained(hv_levels3_kernel, terms, kLvThreads, kLvSmem, s, ys, wk, xs, zs, n, levels, r[0], r[1], r[2], term));
    } else {
        terms = (n + kAreaChunk - 1u) / kAreaChunk;
        long long *chunk_max = reinterpret_cast<long long *>(wk); // 3D's width keys: unused here
        PGX_CUDA(launch_chained(hv_chunk_max_kernel, terms, kAreaThreads, 0, s, wbits, n, chunk_max));
        PGX_CUDA(launch_chained(hv_area2_kernel, terms, kAreaThreads, 0, s, ys, wbits, chunk_max, n, r[1], term));
    }
    PGX_CUDA(launch_chained(hv_sum_kernel, 1, kHvSumThreads, 0, s, term, terms, d_out));
    ctx->launches += static_cast<uint64_t>(pl) + (m == 3u ? 3u : 4u);
    return PGX_OK;
}

// *out = a - b
__global__ void hv_sub_kernel(const double *__restrict__ a, const double *__restrict__ b, double *__restrict__ out)
{
    chain_wait();
    if (threadIdx.x == 0) *out = __dsub_rn(*a, *b);
}

// *idx = the first index of the smallest (greatest = 0) or largest
// (greatest = 1) of c[0 .. n): hv_algorithm::extreme_contributor's strict
// scan from index 0 (hv_algorithm.cpp:329-349), as a reduction that prefers
// the lower index on ties.
__global__ void __launch_bounds__(1024) hv_extreme_kernel(const double *__restrict__ c, uint32_t n, int greatest,
                                                          unsigned long long *__restrict__ idx)
{
    chain_wait();
    __shared__ double sv[1024];
    __shared__ uint32_t si[1024];
    double best = 0.0;
    uint32_t bi = UINT32_MAX;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const double v = c[i];
        if (bi == UINT32_MAX || (greatest ? v > best : v < best)) {
            best = v;
            bi = i;
        }
    }
    sv[threadIdx.x] = best;
    si[threadIdx.x] = bi;
    __syncthreads();
    for (unsigned h = blockDim.x / 2u; h > 0; h >>= 1) {
        if (threadIdx.x < h) {
            const double v = sv[threadIdx.x + h];
            const uint32_t j = si[threadIdx.x + h];
            const uint32_t i = si[threadIdx.x];
            const bool take = j != UINT32_MAX &&
                              (i == UINT32_MAX || (greatest ? v > sv[threadIdx.x] : v < sv[threadIdx.x]) ||
                               (v == sv[threadIdx.x] && j < i));
            if (take) {
                sv[threadIdx.x] = v;
                si[threadIdx.x] = j;
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) *idx = si[0];
}

// The checks of hypervolume's construction and compute on host data, the
// point count and the device, then the points on the device (s_points):
// returns their address; tail_bytes more are reserved after them.
int upload_points(pgx_context *ctx, const double *points, uint64_t n, uint64_t m, const double *ref,
                  size_t tail_bytes, double **dp, char **tail)
{
    PGX_CHECK(ctx != nullptr, PGX_ERR_INVALID, "null context");
    PGX_CHECK((points != nullptr || n == 0) && ref != nullptr, PGX_ERR_INVALID, "null buffer");
    PGX_TRY(hv_check(points, n, m, ref));
    PGX_CHECK(n < (1u << 24), PGX_ERR_CAPACITY, "hypervolume: more than 2^24 points");
    PGX_TRY(use_device(ctx));
    const size_t bp = align256(static_cast<size_t>(n) * m * 8u);
    PGX_TRY(ctx->s_points.ensure(bp + tail_bytes));
    *dp = ctx->s_points.as<double>();
    *tail = ctx->s_points.as<char>() + bp;
    PGX_CUDA(cudaMemcpyAsync(*dp, points, static_cast<size_t>(n) * m * 8u, cudaMemcpyHostToDevice, ctx->stream));
    return PGX_OK;
}

int wfg_ok(pgx_context *ctx)
{
    unsigned st = 0;
    PGX_TRY(wfg_status(ctx, &st));
    PGX_CHECK(st == 0u, PGX_ERR_CAPACITY, "hypervolume (WFG): a warp ran out of frame buffers");
    return PGX_OK;
}

} // namespace
} // namespace pgx

using namespace pgx;

extern "C" {

int pgx_hypervolume(pgx_context *ctx, const double *points, uint64_t n, uint64_t m, const double *ref, double *out)
{
    PGX_CHECK(ctx != nullptr, PGX_ERR_INVALID, "null context");
    PGX_CHECK(out != nullptr && (points != nullptr || n == 0) && ref != nullptr, PGX_ERR_INVALID, "null buffer");
    PGX_TRY(hv_check(points, n, m, ref));
    PGX_CHECK(n < (1u << 24), PGX_ERR_CAPACITY, "hypervolume: more than 2^24 points");
    std::lock_guard<std::mutex> g(ctx->lock);
    PGX_TRY(use_device(ctx));
    const size_t bp = align256(static_cast<size_t>(n) * m * 8u);
    PGX_TRY(ctx->s_points.ensure(bp + 256u));
    double *dp = ctx->s_points.as<double>();
    double *dout = reinterpret_cast<double *>(ctx->s_points.as<char>() + bp);
    cudaStream_t s = ctx->stream;
    PGX_CUDA(cudaMemcpyAsync(dp, points, static_cast<size_t>(n) * m * 8u, cudaMemcpyHostToDevice, s));
    PGX_TRY(launch_hypervolume(ctx, dp, static_cast<uint32_t>(n), static_cast<uint32_t>(m), ref, dout, s));
    PGX_CUDA(cudaMemcpyAsync(out, dout, sizeof(double), cudaMemcpyDeviceToHost, s));
    PGX_CUDA(cudaStreamSynchronize(s));
    return PGX_OK;
}

int pgx_hypervolume_device(pgx_context *ctx, const double *d_points, uint64_t n, uint64_t m, const double *ref,
                           double *d_out, void *stream)
{
    PGX_CHECK(ctx != nullptr, PGX_ERR_INVALID, "null context");
    PGX_CHECK(d_points != nullptr && d_out != nullptr && ref != nullptr, PGX_ERR_INVALID, "null buffer");
    PGX_CHECK(n > 0u, PGX_ERR_INVALID, "Point set cannot be empty.");
    PGX_CHECK(m > 1u, PGX_ERR_INVALID, "Points of dimension > 1 required.");
    PGX_CHECK(m <= kWfgMaxObjectives, PGX_ERR_NOTIMPL,
              "hypervolume on the GPU: at most " + std::to_string(kWfgMaxObjectives) + " objectives; " +
                  std::to_string(m) + " given");
    PGX_CHECK(n < (1u << 24), PGX_ERR_CAPACITY, "hypervolume: more than 2^24 points");
    std::lock_guard<std::mutex> g(ctx->lock);
    PGX_TRY(use_device(ctx));
    return launch_hypervolume(ctx, d_points, static_cast<uint32_t>(n), static_cast<uint32_t>(m), ref, d_out,
                              static_cast<cudaStream_t>(stream));
}

int pgx_hypervolume_exclusive(pgx_context *ctx, const double *points, uint64_t n, uint64_t m, const double *ref,
                              uint64_t p_idx, double *out)
{
    PGX_CHECK(ctx != nullptr, PGX_ERR_INVALID, "null context");
    PGX_CHECK(out != nullptr && (points != nullptr || n == 0) && ref != nullptr, PGX_ERR_INVALID, "null buffer");
    PGX_TRY(hv_check(points, n, m, ref)); // before the index, as hypervolume::exclusive (hypervolume.cpp:251-256)
    PGX_CHECK(p_idx < n, PGX_ERR_INVALID, "Index of the individual is out of bounds.");
    std::lock_guard<std::mutex> g(ctx->lock);
    const size_t bl = align256(static_cast<size_t>(n) * m * 8u);
    double *dp = nullptr;
    char *tail = nullptr;
    PGX_TRY(upload_points(ctx, points, n, m, ref, bl + 256u, &dp, &tail));
    double *less = reinterpret_cast<double *>(tail);
    double *d3 = reinterpret_cast<double *>(tail + bl); // volume of all, of all but p_idx, their difference
    cudaStream_t s = ctx->stream;
    const auto nn = static_cast<uint32_t>(n), mm = static_cast<uint32_t>(m);
    if (n == 1u) {
        // hv_algorithm::exclusive of a lone point: the volume (hv_algorithm.cpp:96-98)
        PGX_TRY(launch_hypervolume(ctx, dp, nn, mm, ref, d3 + 2, s));
    } else {
        const size_t row = static_cast<size_t>(m) * 8u;
        if (p_idx > 0u) PGX_CUDA(cudaMemcpyAsync(less, dp, p_idx * row, cudaMemcpyDeviceToDevice, s));
        if (p_idx + 1u < n)
            PGX_CUDA(cudaMemcpyAsync(less + p_idx * m, dp + (p_idx + 1u) * m, (n - p_idx - 1u) * row,
                                     cudaMemcpyDeviceToDevice, s));
        PGX_TRY(launch_hypervolume(ctx, dp, nn, mm, ref, d3, s));
        PGX_TRY(launch_hypervolume(ctx, less, nn - 1u, mm, ref, d3 + 1, s));
        PGX_CUDA(launch_chained(hv_sub_kernel, 1, 32, 0, s, d3, d3 + 1, d3 + 2));
        ++ctx->launches;
    }
    PGX_CUDA(cudaMemcpyAsync(out, d3 + 2, sizeof(double), cudaMemcpyDeviceToHost, s));
    PGX_CUDA(cudaStreamSynchronize(s));
    if (m >= 4u) PGX_TRY(wfg_ok(ctx));
    return PGX_OK;
}

int pgx_hypervolume_contributions(pgx_context *ctx, const double *points, uint64_t n, uint64_t m, const double *ref,
                                  double *out)
{
    PGX_CHECK(out != nullptr, PGX_ERR_INVALID, "null buffer");
    PGX_CHECK(ctx != nullptr, PGX_ERR_INVALID, "null context");
    std::lock_guard<std::mutex> g(ctx->lock);
    const size_t bo = align256(static_cast<size_t>(n) * 8u);
    double *dp = nullptr;
    char *tail = nullptr;
    PGX_TRY(upload_points(ctx, points, n, m, ref, bo, &dp, &tail));
    double *dc = reinterpret_cast<double *>(tail);
    PGX_TRY(launch_wfg_contributions(ctx, dp, static_cast<uint32_t>(n), static_cast<uint32_t>(m), ref, dc,
                                     ctx->stream));
    PGX_CUDA(cudaMemcpyAsync(out, dc, static_cast<size_t>(n) * 8u, cudaMemcpyDeviceToHost, ctx->stream));
    return wfg_ok(ctx);
}

int pgx_hypervolume_contributions_device(pgx_context *ctx, const double *d_points, uint64_t n, uint64_t m,
                                         const double *ref, double *d_out, void *stream)
{
    PGX_CHECK(ctx != nullptr, PGX_ERR_INVALID, "null context");
    PGX_CHECK(d_points != nullptr && d_out != nullptr && ref != nullptr, PGX_ERR_INVALID, "null buffer");
    PGX_CHECK(n > 0u, PGX_ERR_INVALID, "Point set cannot be empty.");
    PGX_CHECK(m > 1u, PGX_ERR_INVALID, "Points of dimension > 1 required.");
    PGX_CHECK(m <= kWfgMaxObjectives, PGX_ERR_NOTIMPL,
              "hypervolume on the GPU: at most " + std::to_string(kWfgMaxObjectives) + " objectives; " +
                  std::to_string(m) + " given");
    PGX_CHECK(n < (1u << 24), PGX_ERR_CAPACITY, "hypervolume: more than 2^24 points");
    std::lock_guard<std::mutex> g(ctx->lock);
    PGX_TRY(use_device(ctx));
    return launch_wfg_contributions(ctx, d_points, static_cast<uint32_t>(n), static_cast<uint32_t>(m), ref, d_out,
                                    static_cast<cudaStream_t>(stream));
}

int pgx_hypervolume_extreme_contributor(pgx_context *ctx, const double *points, uint64_t n, uint64_t m,
                                        const double *ref, int greatest, uint64_t *idx)
{
    PGX_CHECK(idx != nullptr, PGX_ERR_INVALID, "null buffer");
    PGX_CHECK(ctx != nullptr, PGX_ERR_INVALID, "null context");
    std::lock_guard<std::mutex> g(ctx->lock);
    const size_t bo = align256(static_cast<size_t>(n) * 8u);
    double *dp = nullptr;
    char *tail = nullptr;
    PGX_TRY(upload_points(ctx, points, n, m, ref, bo + 256u, &dp, &tail));
    if (n == 1u) { // hypervolume.cpp:339-342, hv_algorithm.cpp:332-335
        *idx = 0;
        return PGX_OK;
    }
    double *dc = reinterpret_cast<double *>(tail);
    auto *di = reinterpret_cast<unsigned long long *>(tail + bo);
    cudaStream_t s = ctx->stream;
    PGX_TRY(launch_wfg_contributions(ctx, dp, static_cast<uint32_t>(n), static_cast<uint32_t>(m), ref, dc, s));
    PGX_CUDA(launch_chained(hv_extreme_kernel, 1, 1024, 0, s, dc, static_cast<uint32_t>(n), greatest ? 1 : 0, di));
    ++ctx->launches;
    unsigned long long h = 0;
    PGX_CUDA(cudaMemcpyAsync(&h, di, sizeof(h), cudaMemcpyDeviceToHost, s));
    PGX_TRY(wfg_ok(ctx));
    *idx = h;
    return PGX_OK;
}

} // extern "C"

// WFG hypervolume on the GPU: pagmo's hvwfg with stop dimension 2
// (src/utils/hv_algos/hv_hvwfg.cpp), the algorithm hypervolume::compute picks
// for 4 or more objectives and hypervolume::contributions for 4 or more
// (src/utils/hypervolume.cpp:488-537); hv3d's contributions fall back to it
// (hv_hv3d.cpp:229-231), hv2d's run hv3d on the points with a third
// coordinate 0 and a reference 1 (hv_hv2d.cpp:133-146).
//
// The recursion, per frame of k points in d coordinates (hv_hvwfg.cpp:196-272):
//   k = 1: vol(p) = |prod over c = d-1 .. 0 of (r_c - p_c)|;
//   k = 2: vol(p0) + vol(p1) - prod over c = 0 .. d-1 of (r_c - max(p0_c, p1_c));
//   d = 2: hv2d's sweep over the points sorted by the second coordinate;
//   else: the frame sorted by hvwfg::cmp_points (descending, last coordinate
//   first) and H += |(p_j[d-1] - r_{d-1}) * (vol_{d-1}(p_j) - hv(L_j))| in
//   that order, L_j the limit set of p_j over the points after it: max(q, p_j)
//   over the first d-1 coordinates, non-dominated, one copy of equal points
//   (hvwfg::limitset, hv_hvwfg.cpp:134-193).
// A point's contribution is vol_m(p) - hv(limit set of p over every other
// point, m coordinates) (hvwfg::contributions, hv_hvwfg.cpp:79-105); the
// volume is the sum, in sorted order, of the top level's terms.
//
// GPU layout: one block per top-level term (compute) or per point
// (contributions), taken from a work counter in index order (the early terms
// of the sorted set have the most candidates); the frames of the first levels
// are split into one work item per sub-term, level by level (see wfg_level),
// a warp each, and the deepest level recurses on an explicit stack, its frames
// in the warp's slice of a scratch pool (m buffers of n rows). A warp's lanes
// share the limit-set filter (32 candidates at a time against the kept set,
// then against each other, then the kept points the survivors cover are
// removed) and the counting-rank sorts of a frame. Every coordinate of every
// frame is one of the points' (a limit set takes maxima), so the frames hold
// ranks, the number of points with a smaller value in that coordinate, two of
// 15 bits to a word: a maximum is one instruction for two coordinates, "no
// coordinate larger" a subtraction and a mask, and a word's order is that of
// its higher coordinate, then of its lower one. Only the volumes and terms look
// the values up in a table (rank_rows; n = 2000, m = 5: limit sets of the items
// 534 us on keys, 160 on ranks; of the rows 466, 254; the whole volume, with
// what is below, 1260 -> 349 us; n = 100, m = 5: 114 -> 69 us, n = 4000, m = 4:
// 554 -> 322 us). More than kRankLimit points hold 64-bit order keys instead
// (key_rows: the IEEE bit pattern with negatives mirrored, -0.0 read as +0.0,
// which the reference compares equal;
// the ranks are those of the keys). A frame's kept set is the unique
// non-dominated subset of its candidates whatever order they are filtered in,
// every frame of more than two points is sorted by a strict order before it is
// used, and the two-point form is symmetric, so the arithmetic is the
// reference's: every operation is the reference's IEEE double operation in the
// reference's order (explicit round-to-nearest intrinsics: no contraction into
// FMA), and the volumes and contributions equal the reference's bit for bit.
#include "pgx_internal.cuh"

#include <algorithm>

namespace pgx
{
namespace
{

constexpr unsigned kMask = 0xffffffffu;
constexpr int kWarpsPerBlock = 4;

struct wfg_ref {
    double r[kWfgMaxObjectives];
};

using okey = long long; // order key of a coordinate

__device__ __forceinline__ okey to_key(double v)
{
    const long long b = __double_as_longlong(v == 0.0 ? 0.0 : v);
    return b >= 0 ? b : (b ^ 0x7fffffffffffffffLL);
}

__device__ __forceinline__ double from_key(okey k)
{
    return __longlong_as_double(k >= 0 ? k : (k ^ 0x7fffffffffffffffLL));
}

__device__ __forceinline__ double std_max(double a, double b)
{
    return a < b ? b : a; // std::max(a, b)
}

// The values of ranks: tab[c n + rank].
struct wfg_values {
    const double *tab;
    uint32_t n;
};

constexpr uint32_t kRankLimit = 32768;
constexpr uint32_t kRankGuard = 0x80008000u;

// Rows of order keys, a word per coordinate (at most N).
template <int N_>
struct key_rows {
    using word = okey;
    static constexpr int N = N_;
    __device__ static uint32_t words(uint32_t d)
    {
        return d;
    }
    __device__ static word none(uint32_t, uint32_t) // (every bit of a word is in use)
    {
        return -1;
    }
    __device__ static word larger(word a, word b)
    {
        return max(a, b);
    }
    __device__ static bool le(word a, word b) // every coordinate of a <= b's
    {
        return a <= b;
    }
    __device__ static okey coord(const word *p, uint32_t c)
    {
        return p[c];
    }
    __device__ static double value(const wfg_values &, uint32_t, okey k)
    {
        return from_key(k);
    }
};

// Rows of ranks, two to a word (at most N words).
template <int N_>
struct rank_rows {
    using word = uint32_t;
    static constexpr int N = N_;
    __device__ static uint32_t words(uint32_t d)
    {
        return (d + 1u) / 2u;
    }
    __device__ static word none(uint32_t w, uint32_t d) // the bits of word w that d coordinates use
    {
        return 2u * w + 1u < d ? 0xffffffffu : 0xffffu;
    }
    __device__ static word larger(word a, word b)
    {
        return __vmaxu2(a, b);
    }
    __device__ static bool le(word a, word b)
    {
        return (((b | kRankGuard) - a) & kRankGuard) == kRankGuard;
    }
    __device__ static okey coord(const word *p, uint32_t c)
    {
        return (p[c >> 1] >> (16u * (c & 1u))) & 0xffffu;
    }
    __device__ static double value(const wfg_values &v, uint32_t c, okey k)
    {
        return __ldg(v.tab + c * v.n + static_cast<uint32_t>(k));
    }
};

// |prod over c = d-1 .. 0 of (r_c - p_c)| (hv_algorithm::volume_between on
// pointers, hv_algorithm.cpp:73-82)
template <class P>
__device__ __forceinline__ double vol(const wfg_values &vals, const double *r, const typename P::word *p, uint32_t d)
{
    double v = 1.0;
    for (int c = static_cast<int>(d) - 1; c >= 0; --c)
        v = __dmul_rn(v, __dsub_rn(r[c], P::value(vals, static_cast<uint32_t>(c), P::coord(p, static_cast<uint32_t>(c)))));
    return v < 0.0 ? -v : v;
}

// the same on plain doubles
__device__ __forceinline__ double vol_d(const double *r, const double *p, uint32_t d)
{
    double v = 1.0;
    for (int c = static_cast<int>(d) - 1; c >= 0; --c) v = __dmul_rn(v, __dsub_rn(r[c], p[c]));
    return v < 0.0 ? -v : v;
}

__device__ __forceinline__ unsigned lanes_below(unsigned lane)
{
    return (1u << lane) - 1u;
}

// The limit set of p over the rows t of src in [begin, end), t != skip
// (stride src_stride): max(row, p) over the first dc coordinates, filtered to
// the non-dominated ones with one copy of equal points, written to dst
// (rows of words(dc)). Returns the number kept. Warp-uniform arguments.
template <class P>
__device__ uint32_t limit_set(const typename P::word *src, uint32_t src_stride, uint32_t begin, uint32_t end,
                              uint32_t skip, const typename P::word *p, uint32_t dc, typename P::word *dst, unsigned lane)
{
    using word = typename P::word;
    const uint32_t nw = P::words(dc);
    word own[P::N];
#pragma unroll
    for (uint32_t w = 0; w < P::N; ++w) own[w] = w < nw ? p[w] : 0;
    uint32_t K = 0;
    for (uint32_t base = begin; base < end; base += 32u) {
        const uint32_t t = base + lane;
        const bool valid = t < end && t != skip;
        word s[P::N];
#pragma unroll
        for (uint32_t w = 0; w < P::N; ++w)
            s[w] = (valid && w < nw) ? P::larger(src[static_cast<uint64_t>(t) * src_stride + w], own[w]) & P::none(w, dc)
                                     : 0;
        bool alive = valid;
        // a kept point <= s in every coordinate (dominating or equal): s goes
        for (uint32_t q = 0; q < K; q += 4u) {
            if (!__any_sync(kMask, alive)) break;
            bool covered = false;
#pragma unroll
            for (uint32_t u = 0; u < 4u; ++u) {
                const word *kq = dst + static_cast<uint64_t>(min(q + u, K - 1u)) * nw;
                bool le = true;
#pragma unroll
                for (uint32_t w = 0; w < P::N; ++w)
                    if (w < nw) le &= P::le(kq[w], s[w]);
                covered |= le;
            }
            alive &= !covered;
        }
        // within the batch: a live candidate that dominates s, or equals it
        // from a higher lane (a candidate a kept point removed is no witness
        // needed: that kept point also covers whatever it dominates)
        const unsigned live = __ballot_sync(kMask, alive);
        if (__popc(live) > 1) {
            for (unsigned rest = live; rest; rest &= rest - 1u) {
                const int u = __ffs(rest) - 1;
                bool le = true, differs = false;
#pragma unroll
                for (uint32_t w = 0; w < P::N; ++w) {
                    if (w < nw) {
                        const word su = __shfl_sync(kMask, s[w], u);
                        le &= P::le(su, s[w]);
                        differs |= su != s[w];
                    }
                }
                if (u != static_cast<int>(lane) && le && (differs || u > static_cast<int>(lane))) alive = false;
            }
        }
        const unsigned surv = __ballot_sync(kMask, alive);
        if (surv == 0u) continue;
        // the kept points a survivor covers go (in place, order kept), the
        // survivors are appended
        uint32_t nk = 0;
        for (uint32_t c0 = 0; c0 < K; c0 += 32u) {
            const uint32_t q = c0 + lane;
            const bool has = q < K;
            word qr[P::N];
#pragma unroll
            for (uint32_t w = 0; w < P::N; ++w) qr[w] = (has && w < nw) ? dst[static_cast<uint64_t>(q) * nw + w] : 0;
            bool keep = has;
            for (unsigned rs = surv; rs; rs &= rs - 1u) {
                const int u = __ffs(rs) - 1;
                bool cov = true;
#pragma unroll
                for (uint32_t w = 0; w < P::N; ++w)
                    if (w < nw) cov &= P::le(__shfl_sync(kMask, s[w], u), qr[w]);
                keep &= !cov;
            }
            const unsigned km = __ballot_sync(kMask, keep);
            __syncwarp();
            if (keep && (nk != c0 || km != kMask)) {
                word *o = dst + static_cast<uint64_t>(nk + __popc(km & lanes_below(lane))) * nw;
#pragma unroll
                for (uint32_t w = 0; w < P::N; ++w)
                    if (w < nw) o[w] = qr[w];
            }
            nk += __popc(km);
            __syncwarp();
        }
        if (alive) {
            word *o = dst + static_cast<uint64_t>(nk + __popc(surv & lanes_below(lane))) * nw;
#pragma unroll
            for (uint32_t w = 0; w < P::N; ++w)
                if (w < nw) o[w] = s[w];
        }
        K = nk + __popc(surv);
        __syncwarp();
    }
    return K;
}

// Rows of src (K rows of d coordinates) into dst in order: by_y = false,
// hvwfg::cmp_points (descending, last coordinate first: hv_hvwfg.cpp:276-286);
// by_y = true (d = 2), ascending second coordinate (hv2d, hv_hv2d.cpp:79-81).
// Ties by row index (a frame's rows are distinct, so they never decide an
// order there).
// (Warp `part` of `parts` places its share of the rows.)
template <class P>
__device__ void sort_rows(const typename P::word *src, uint32_t K, uint32_t d, bool by_y, typename P::word *dst,
                          unsigned lane, uint32_t part = 0u, uint32_t parts = 1u)
{
    using word = typename P::word;
    const uint32_t nw = P::words(d);
    for (uint32_t i0 = 32u * part; i0 < K; i0 += 32u * parts) {
        const uint32_t i = i0 + lane;
        const bool has = i < K;
        word mine[P::N];
#pragma unroll
        for (uint32_t w = 0; w < P::N; ++w) mine[w] = (has && w < nw) ? src[static_cast<uint64_t>(i) * nw + w] : 0;
        uint32_t rank = 0;
        if (by_y) {
            const okey y = has ? P::coord(src + static_cast<uint64_t>(i) * nw, 1u) : 0;
            for (uint32_t j = 0; j < K; ++j) {
                const okey a = P::coord(src + static_cast<uint64_t>(j) * nw, 1u);
                rank += (a < y || (a == y && j < i)) ? 1u : 0u;
            }
        } else {
            for (uint32_t j = 0; j < K; ++j) {
                const word *rj = src + static_cast<uint64_t>(j) * nw;
                int dec = 0; // +1: row j first, -1: this row first
#pragma unroll
                for (int w = P::N - 1; w >= 0; --w) {
                    if (w < static_cast<int>(nw) && dec == 0) {
                        const word a = rj[w];
                        dec = a > mine[w] ? 1 : (a < mine[w] ? -1 : 0);
                    }
                }
                rank += (dec > 0 || (dec == 0 && j < i)) ? 1u : 0u;
            }
        }
        if (has) {
            word *o = dst + static_cast<uint64_t>(rank) * nw;
#pragma unroll
            for (uint32_t w = 0; w < P::N; ++w)
                if (w < nw) o[w] = mine[w];
        }
    }
    __syncwarp();
}

// The frames of a warp: m buffers of bd words, taken and given back by bit.
template <class P>
struct frame_pool {
    typename P::word *base;
    uint64_t bd;
    unsigned free;

    __device__ int take()
    {
        if (free == 0u) return -1;
        const int b = __ffs(free) - 1;
        free &= ~(1u << b);
        return b;
    }
    __device__ void give(int b)
    {
        free |= 1u << b;
    }
    __device__ typename P::word *at(int b) const
    {
        return base + static_cast<uint64_t>(b) * bd;
    }
};

// hv of a frame of 1 or 2 points, or of 2 coordinates with its rows by y
template <class P>
__device__ double closed_form(const wfg_values &vals, const double *r, const typename P::word *f, uint32_t K, uint32_t d)
{
    const uint32_t nw = P::words(d);
    if (K == 1u) return vol<P>(vals, r, f, d);
    if (K == 2u) {
        const double h = __dadd_rn(vol<P>(vals, r, f, d), vol<P>(vals, r, f + nw, d));
        double isect = 1.0;
        for (uint32_t c = 0; c < d; ++c)
            isect = __dmul_rn(isect, __dsub_rn(r[c], P::value(vals, c, max(P::coord(f, c), P::coord(f + nw, c)))));
        return __dsub_rn(h, isect);
    }
    double area = 0.0, w = __dsub_rn(r[0], P::value(vals, 0u, P::coord(f, 0u))), y = P::value(vals, 1u, P::coord(f, 1u));
    for (uint32_t t = 1; t < K; ++t) {
        const double x1 = P::value(vals, 0u, P::coord(f + t * nw, 0u)), y1 = P::value(vals, 1u, P::coord(f + t * nw, 1u));
        area = __dadd_rn(area, __dmul_rn(__dsub_rn(y1, y), w));
        w = std_max(w, __dsub_rn(r[0], x1));
        y = y1;
    }
    return __dadd_rn(area, __dmul_rn(__dsub_rn(r[1], y), w));
}

// |(p[d-1] - r[d-1]) * ex|, the term a point of a frame of d coordinates adds
template <class P>
__device__ __forceinline__ double slice_term(const wfg_values &vals, const double *r, const typename P::word *p, uint32_t d,
                                             double ex)
{
    return fabs(__dmul_rn(__dsub_rn(P::value(vals, d - 1u, P::coord(p, d - 1u)), r[d - 1u]), ex));
}

// hv of the frame in buffer `buf` (K points of d coordinates, K >= 1); the
// frame's buffer and every buffer taken below are given back. *fail is set
// when the pool runs dry (it cannot: a level holds one buffer, a sort or the
// sweep one more, and there are at most m - 1 levels).
template <class P>
__device__ double frame_hv(const wfg_values &vals, const double *r, frame_pool<P> &pool, int buf, uint32_t K, uint32_t d,
                           unsigned lane, bool *fail)
{
    using word = typename P::word;
    constexpr int kDepth = sizeof(word) == sizeof(okey) ? P::N : 2 * P::N + 1;
    int st_buf[kDepth];
    uint32_t st_k[kDepth], st_d[kDepth];
    int st_j[kDepth];
    double st_h[kDepth];
    int sp = 0;
    st_buf[0] = buf;
    st_k[0] = K;
    st_d[0] = d;
    st_j[0] = -1;
    st_h[0] = 0.0;
    for (;;) {
        const int j = st_j[sp];
        const uint32_t kk = st_k[sp], dd = st_d[sp];
        const word *f = pool.at(st_buf[sp]);
        double val;
        if (j < 0) {
            if (kk <= 2u || dd == 2u) {
                int tb = -1;
                if (kk > 2u) {
                    if ((tb = pool.take()) < 0) {
                        *fail = true;
                        return 0.0;
                    }
                    sort_rows<P>(f, kk, 2u, true, pool.at(tb), lane);
                }
                val = closed_form<P>(vals, r, tb >= 0 ? pool.at(tb) : f, kk, dd);
                if (tb >= 0) pool.give(tb);
            } else {
                const int sb = pool.take();
                if (sb < 0) {
                    *fail = true;
                    return 0.0;
                }
                sort_rows<P>(f, kk, dd, false, pool.at(sb), lane);
                pool.give(st_buf[sp]);
                st_buf[sp] = sb;
                st_j[sp] = 0;
                st_h[sp] = 0.0;
                continue;
            }
        } else if (static_cast<uint32_t>(j) < kk) {
            const uint32_t nw = P::words(dd);
            const word *p = f + static_cast<uint64_t>(j) * nw;
            const int cb = pool.take();
            if (cb < 0) {
                *fail = true;
                return 0.0;
            }
            word *child = pool.at(cb);
            const uint32_t ck = limit_set<P>(f, nw, static_cast<uint32_t>(j) + 1u, kk, kk, p, dd - 1u, child, lane);
            if (ck <= 1u) {
                double ex = vol<P>(vals, r, p, dd - 1u);
                if (ck == 1u) ex = __dsub_rn(ex, vol<P>(vals, r, child, dd - 1u));
                pool.give(cb);
                st_h[sp] = __dadd_rn(st_h[sp], slice_term<P>(vals, r, p, dd, ex));
                st_j[sp] = j + 1;
                continue;
            }
            ++sp;
            st_buf[sp] = cb;
            st_k[sp] = ck;
            st_d[sp] = dd - 1u;
            st_j[sp] = -1;
            st_h[sp] = 0.0;
            continue;
        } else {
            val = st_h[sp];
        }
        // level sp is done with value val: its parent's term j completes
        pool.give(st_buf[sp]);
        if (sp == 0) return val;
        --sp;
        const uint32_t pd = st_d[sp];
        const int pj = st_j[sp];
        const word *p = pool.at(st_buf[sp]) + static_cast<uint64_t>(pj) * P::words(pd);
        st_h[sp] = __dadd_rn(st_h[sp], slice_term<P>(vals, r, p, pd, __dsub_rn(vol<P>(vals, r, p, pd - 1u), val)));
        st_j[sp] = pj + 1;
    }
}

// The work of one volume or one set of contributions is split into levels of
// rows: wfg_top_kernel takes the items (the top-level terms of a volume, or
// the points of the contributions), builds each item's limit set (its
// "frame") and finishes the items whose frame has at most two points or two
// coordinates; every other frame is sorted into the level-1 row list, one row
// per sub-term. wfg_rows_kernel(l) takes the rows of level l: row j of a frame
// gives the sub-term |(f_j[d-1] - r_{d-1}) * (vol_{d-1}(f_j) - hv(limit set
// of f_j over the rows after it))|; the row's own frame (that limit set) goes
// to level l + 1 the same way while levels remain, else the recursion below it
// runs on the warp's own stack. wfg_join_kernel(l) adds each row's sub-terms
// of level l + 1 in order (compute_hv's H += ..., hv_hvwfg.cpp:262-266) and
// finishes the row, and wfg_items_kernel finishes the items from level 1. The
// operations and their order are those of one recursion, split between warps.
constexpr int kMaxLevels = 4;

template <class P>
struct wfg_level {
    typename P::word *frames;      // the frames of this level's rows, rows of words(d)
    uint32_t *row_parent;          // per row: its item (level 1) or its row of the level above
    double *row_term;              // per row: its sub-term
    uint32_t *frame_k;             // per parent: rows of its frame here (0: none)
    unsigned long long *frame_off; // per parent: its first row here
    unsigned long long *rows_used; // rows handed out (zero at launch)
    uint64_t row_cap;
    uint64_t parents;              // entries of frame_k / frame_off
};

template <class P>
struct wfg_args {
    const typename P::word *pts; // n rows of words(m); sorted by cmp_points for the terms of a volume
    wfg_values vals;
    uint32_t n, m;
    int contributions;  // 0: out[i] = the top-level term of sorted point i; 1: the contribution of point i
    double *out;        // n
    typename P::word *pool; // per warp: m buffers of bd words
    uint64_t bd;
    unsigned *next;     // work counters (zero at launch): [0] items, [2 + l] rows of level l
    unsigned *status;   // set when a warp's pool ran dry
    int levels;         // row levels in use, 1 .. kMaxLevels
    wfg_level<P> lv[kMaxLevels + 2]; // lv[1 .. levels]; lv[levels + 1] unused
};

template <class P>
__device__ __forceinline__ uint32_t first_dims(const wfg_args<P> &a)
{
    return a.contributions ? a.m : a.m - 1u; // coordinates of the items' frames
}

// The rows of level l from row0 to the list's end belong to no frame: the one
// that would have begun there does not fit (and none after it does). Unmarked
// they would hold what an earlier call left, whose ranks are no indexes into
// this call's table.
constexpr uint32_t kNoParent = 0xffffffffu;

template <class P>
__device__ __forceinline__ void mark_gap(const wfg_level<P> &L, unsigned long long row0, uint32_t t, uint32_t threads)
{
    for (unsigned long long g = row0 + t; g < L.row_cap; g += threads) L.row_parent[g] = kNoParent;
}

// Row g of level l when it belongs to a frame stored at that level: its frame's
// rows k, first row off and index j; false for marked rows.
template <class P>
__device__ __forceinline__ bool row_of(const wfg_args<P> &a, int l, unsigned long long g, uint32_t *k,
                                       unsigned long long *off)
{
    const wfg_level<P> &L = a.lv[l];
    const uint32_t parent = L.row_parent[g];
    if (parent >= L.parents) return false;
    *k = L.frame_k[parent];
    *off = L.frame_off[parent];
    return *k != 0u && g >= *off && g < *off + *k && *off + *k <= L.row_cap;
}

// The frame `buf` (k points of d coordinates, k > 2, d > 2) into level l's
// list, one row per point, sorted; the parent's entries set. Returns false
// when the list is full (the caller recurses instead).
template <class P>
__device__ bool store_frame(const wfg_args<P> &a, int l, uint64_t parent, const typename P::word *buf, uint32_t k,
                            uint32_t d, unsigned lane)
{
    const wfg_level<P> &L = a.lv[l];
    unsigned long long row0 = 0;
    if (lane == 0) row0 = atomicAdd(L.rows_used, static_cast<unsigned long long>(k));
    row0 = __shfl_sync(kMask, row0, 0);
    if (row0 + k > L.row_cap) {
        mark_gap<P>(L, row0, lane, 32u);
        return false;
    }
    sort_rows<P>(buf, k, d, false, L.frames + row0 * P::words(d), lane);
    for (uint32_t t = lane; t < k; t += 32u) L.row_parent[row0 + t] = static_cast<uint32_t>(parent);
    if (lane == 0) {
        L.frame_k[parent] = k;
        L.frame_off[parent] = row0;
    }
    return true;
}

template <class P>
__device__ __forceinline__ void mark_failed(const wfg_args<P> &a, uint32_t item, unsigned lane)
{
    if (lane == 0) {
        atomicOr(a.status, 1u);
        a.out[item] = __longlong_as_double(0x7ff8000000000000LL);
    }
}

// limit_set by a block, a batch of 32 candidates per warp at a time; the kept
// set starts in *kept and may end in *other (they are exchanged), in any order.
template <class P>
struct block_batch {
    typename P::word row[kWarpsPerBlock * 32][P::N];
    uint32_t live[kWarpsPerBlock], kept;
};

template <class P>
__device__ uint32_t block_limit_set(const typename P::word *src, uint32_t src_stride, uint32_t begin, uint32_t end,
                                    uint32_t skip, const typename P::word *p, uint32_t dc, typename P::word **kept,
                                    typename P::word **other, block_batch<P> &b)
{
    using word = typename P::word;
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t warp = threadIdx.x >> 5, nw = P::words(dc);
    word own[P::N];
#pragma unroll
    for (uint32_t w = 0; w < P::N; ++w) own[w] = w < nw ? p[w] : 0;
    uint32_t K = 0;
    for (uint32_t base = begin; base < end; base += kWarpsPerBlock * 32u) {
        const uint32_t t = base + threadIdx.x;
        const bool valid = t < end && t != skip;
        word s[P::N];
#pragma unroll
        for (uint32_t w = 0; w < P::N; ++w)
            s[w] = (valid && w < nw) ? P::larger(src[static_cast<uint64_t>(t) * src_stride + w], own[w]) & P::none(w, dc)
                                     : 0;
        bool alive = valid;
        const word *set = *kept;
        for (uint32_t q = 0; q < K; q += 4u) {
            if (!__any_sync(kMask, alive)) break;
            bool covered = false;
#pragma unroll
            for (uint32_t u = 0; u < 4u; ++u) {
                const word *kq = set + static_cast<uint64_t>(min(q + u, K - 1u)) * nw;
                bool le = true;
#pragma unroll
                for (uint32_t w = 0; w < P::N; ++w)
                    if (w < nw) le &= P::le(kq[w], s[w]);
                covered |= le;
            }
            alive &= !covered;
        }
        if (!__syncthreads_or(alive)) continue; // (nearly always, after the first batches)
        // the live candidates of all warps, against each other
        const unsigned live = __ballot_sync(kMask, alive);
        const uint32_t place = 32u * warp + __popc(live & lanes_below(lane));
        if (alive) {
#pragma unroll
            for (uint32_t w = 0; w < P::N; ++w) b.row[place][w] = s[w];
        }
        if (lane == 0) b.live[warp] = __popc(live);
        if (threadIdx.x == 0) b.kept = 0u;
        __syncthreads();
        if (live) {
            for (uint32_t v = 0; v < kWarpsPerBlock; ++v) {
                for (uint32_t q = 32u * v; q < 32u * v + b.live[v]; ++q) {
                    bool le = true, differs = q < place;
#pragma unroll
                    for (uint32_t w = 0; w < P::N; ++w) {
                        if (w < nw) {
                            const word x = b.row[q][w];
                            le &= P::le(x, s[w]);
                            differs |= x != s[w];
                        }
                    }
                    alive &= !(le && differs);
                }
            }
        }
        const unsigned surv = __ballot_sync(kMask, alive);
        __syncthreads(); // the rows are read no more
        if (lane == 0) b.live[warp] = __popc(surv);
        __syncthreads();
        uint32_t at = 0, S = 0;
#pragma unroll
        for (uint32_t v = 0; v < kWarpsPerBlock; ++v) {
            at += v < warp ? b.live[v] : 0u;
            S += b.live[v];
        }
        if (S == 0u) continue;
        at += __popc(surv & lanes_below(lane));
        if (alive) {
#pragma unroll
            for (uint32_t w = 0; w < P::N; ++w) b.row[at][w] = s[w];
        }
        __syncthreads();
        // the kept points that no survivor covers
        word *to = *other;
        for (uint32_t c0 = 32u * warp; c0 < K; c0 += kWarpsPerBlock * 32u) {
            const bool has = c0 + lane < K;
            word qr[P::N];
#pragma unroll
            for (uint32_t w = 0; w < P::N; ++w) qr[w] = (has && w < nw) ? set[static_cast<uint64_t>(c0 + lane) * nw + w] : 0;
            bool keep = has;
            for (uint32_t q = 0; q < S; ++q) {
                bool cov = true;
#pragma unroll
                for (uint32_t w = 0; w < P::N; ++w)
                    if (w < nw) cov &= P::le(b.row[q][w], qr[w]);
                keep &= !cov;
            }
            const unsigned km = __ballot_sync(kMask, keep);
            uint32_t from = 0;
            if (lane == 0) from = atomicAdd(&b.kept, static_cast<uint32_t>(__popc(km)));
            from = __shfl_sync(kMask, from, 0);
            if (keep) {
                word *o = to + static_cast<uint64_t>(from + __popc(km & lanes_below(lane))) * nw;
#pragma unroll
                for (uint32_t w = 0; w < P::N; ++w)
                    if (w < nw) o[w] = qr[w];
            }
        }
        __syncthreads();
        const uint32_t stay = b.kept;
        if (stay == K) { // all: the set stays where it is
            to = *kept;
        } else {
            *other = *kept;
            *kept = to;
        }
        if (alive) {
#pragma unroll
            for (uint32_t w = 0; w < P::N; ++w)
                if (w < nw) to[static_cast<uint64_t>(stay + at) * nw + w] = s[w];
        }
        K = stay + S;
        __syncthreads();
    }
    return K;
}

// A block takes an item. (A warp per item: the first items' sets, with the most
// candidates, took twice the average time of an SM: 362000 against 178000
// cycles at n = 2000, m = 5, 178 us; 122 now. A share of the candidates per
// warp, then the sets against each other: 864 us, the shares' own sets are far
// larger than what is kept of them.)
template <class P>
__global__ void __launch_bounds__(kWarpsPerBlock * 32) wfg_top_kernel(wfg_args<P> a, wfg_ref ref)
{
    chain_wait();
    using word = typename P::word;
    __shared__ double s_r[kWfgMaxObjectives];
    __shared__ block_batch<P> s_batch;
    __shared__ uint32_t s_item;
    __shared__ unsigned long long s_row0;
    if (threadIdx.x < kWfgMaxObjectives) s_r[threadIdx.x] = threadIdx.x < a.m ? ref.r[threadIdx.x] : 0.0;
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t m = a.m, mw = P::words(m);
    const uint32_t dc = first_dims(a), nw = P::words(dc);
    // buffers of the block's first warp (m, at least 3): 0 and 1 the frame, 2 a sort
    const uint64_t gw = static_cast<uint64_t>(blockIdx.x) * kWarpsPerBlock;
    word *const base = a.pool + gw * m * a.bd;
    const wfg_level<P> &L = a.lv[1];
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_item = atomicAdd(a.next, 1u);
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= a.n) break;
        const word *p = a.pts + static_cast<uint64_t>(item) * mw;
        word *frame = base, *other = base + a.bd;
        const uint32_t k0 = block_limit_set<P>(a.pts, mw, a.contributions ? 0u : item + 1u, a.n,
                                               a.contributions ? item : a.n, p, dc, &frame, &other, s_batch);
        if (k0 > 2u && dc > 2u) { // to the level-1 list, by all warps
            if (threadIdx.x == 0) s_row0 = atomicAdd(L.rows_used, static_cast<unsigned long long>(k0));
            __syncthreads();
            const unsigned long long row0 = s_row0;
            if (row0 + k0 <= L.row_cap) {
                sort_rows<P>(frame, k0, dc, false, L.frames + row0 * nw, lane, warp, kWarpsPerBlock);
                for (uint32_t t = threadIdx.x; t < k0; t += blockDim.x) L.row_parent[row0 + t] = item;
                if (threadIdx.x == 0) {
                    L.frame_k[item] = k0;
                    L.frame_off[item] = row0;
                }
                continue;
            }
            mark_gap<P>(L, row0, threadIdx.x, blockDim.x);
        }
        if (warp != 0u) continue;
        const int in = frame == base ? 0 : 1;
        frame_pool<P> pool{base, a.bd, ((1u << m) - 1u) & ~(1u << in)};
        double ex = vol<P>(a.vals, s_r, p, dc);
        bool fail = false;
        if (k0 == 0u) {
        } else if (k0 <= 2u || dc == 2u) {
            if (k0 > 2u) sort_rows<P>(frame, k0, 2u, true, other, lane);
            ex = __dsub_rn(ex, closed_form<P>(a.vals, s_r, k0 > 2u ? other : frame, k0, dc));
        } else {
            // the level-1 list is full: this warp finishes the item alone
            ex = __dsub_rn(ex, frame_hv<P>(a.vals, s_r, pool, in, k0, dc, lane, &fail));
        }
        if (fail) {
            mark_failed(a, item, lane);
            if (lane == 0) L.frame_k[item] = 0;
            continue;
        }
        if (lane == 0) {
            L.frame_k[item] = 0;
            a.out[item] = a.contributions ? ex : slice_term<P>(a.vals, s_r, p, m, ex);
        }
    }
}

// A warp takes up to 32 rows, builds their frames one after the other, and
// keeps those that a closed form finishes in shared memory; then each lane
// finishes a row, its FP64 operations beside the other lanes' (by the whole
// warp, row after row, the FP64 pipe took 314000 of 542000 cycles of the last
// level at n = 2000, m = 5).
constexpr uint32_t kStashBytes = 4096; // per warp

template <class P>
__global__ void __launch_bounds__(kWarpsPerBlock * 32) wfg_rows_kernel(wfg_args<P> a, wfg_ref ref, int l)
{
    chain_wait();
    using word = typename P::word;
    constexpr uint32_t kStash = kStashBytes / sizeof(word);
    __shared__ double s_r[kWfgMaxObjectives];
    __shared__ word s_stash[kWarpsPerBlock][kStash];
    if (threadIdx.x < kWfgMaxObjectives) s_r[threadIdx.x] = threadIdx.x < a.m ? ref.r[threadIdx.x] : 0.0;
    __syncthreads();
    const unsigned lane = threadIdx.x & 31u;
    const uint64_t gw = static_cast<uint64_t>(blockIdx.x) * kWarpsPerBlock + (threadIdx.x >> 5);
    word *stash = s_stash[threadIdx.x >> 5];
    const uint32_t m = a.m;
    const uint32_t d = first_dims(a) - static_cast<uint32_t>(l - 1); // coordinates of this level's rows
    const uint32_t nw = P::words(d), nc = P::words(d - 1u);
    const wfg_level<P> &L = a.lv[l];
    const unsigned long long used = *L.rows_used;
    const unsigned long long rows = used < L.row_cap ? used : L.row_cap;
    const bool deeper = l < a.levels; // a level below for the rows' own frames
    // rows per turn: all warps have work while there are few
    const unsigned long long share = rows / (static_cast<uint64_t>(gridDim.x) * kWarpsPerBlock * 4u);
    const unsigned turn = static_cast<unsigned>(share < 1u ? 1u : (share < 32u ? share : 32u));
    frame_pool<P> pool{a.pool + gw * m * a.bd, a.bd, (1u << m) - 1u};
    // the row that this lane finishes: its frame's rows in the stash
    const word *mine = nullptr;
    uint32_t mine_k = 0, mine_at = 0;
    unsigned mine_g = 0;
    uint32_t kept = 0, filled = 0; // rows and words waiting
    const auto finish = [&] {
        __syncwarp();
        if (lane < kept) {
            double ex = vol<P>(a.vals, s_r, mine, d - 1u);
            if (mine_k) ex = __dsub_rn(ex, closed_form<P>(a.vals, s_r, stash + mine_at, mine_k, d - 1u));
            L.row_term[mine_g] = slice_term<P>(a.vals, s_r, mine, d, ex);
        }
        kept = filled = 0;
        __syncwarp();
    };
    for (;;) {
        unsigned g0 = 0;
        if (lane == 0) g0 = atomicAdd(a.next + 2 + l, turn);
        g0 = __shfl_sync(kMask, g0, 0);
        if (g0 >= rows) break;
        const unsigned g1 = static_cast<unsigned>(rows - g0 < turn ? rows : static_cast<unsigned long long>(g0) + turn);
        for (unsigned g = g0; g < g1; ++g) {
            uint32_t k = 0;
            unsigned long long off = 0;
            if (!row_of(a, l, g, &k, &off)) continue;
            const uint32_t j = static_cast<uint32_t>(g - off);
            const word *f = L.frames + off * nw;
            const word *p = f + static_cast<uint64_t>(j) * nw;
            const int cb = pool.take();
            const uint32_t ck = limit_set<P>(f, nw, j + 1u, k, k, p, d - 1u, pool.at(cb), lane);
            if (lane == 0 && deeper) a.lv[l + 1].frame_k[g] = 0;
            if ((ck <= 2u || d - 1u == 2u) && ck * nc <= kStash) {
                if (kept == 32u || filled + ck * nc > kStash) finish();
                word *to = stash + filled;
                if (ck > 2u) {
                    sort_rows<P>(pool.at(cb), ck, 2u, true, to, lane);
                } else if (lane < ck * nc) {
                    to[lane] = pool.at(cb)[lane];
                }
                if (lane == kept) {
                    mine = p;
                    mine_k = ck;
                    mine_at = filled;
                    mine_g = g;
                }
                ++kept;
                filled += ck * nc;
                pool.give(cb);
                continue;
            }
            double ex = vol<P>(a.vals, s_r, p, d - 1u);
            bool fail = false;
            if (d - 1u == 2u) {
                const int tb = pool.take();
                sort_rows<P>(pool.at(cb), ck, 2u, true, pool.at(tb), lane);
                ex = __dsub_rn(ex, closed_form<P>(a.vals, s_r, pool.at(tb), ck, 2u));
                pool.give(tb);
                pool.give(cb);
            } else if (deeper && store_frame<P>(a, l + 1, g, pool.at(cb), ck, d - 1u, lane)) {
                pool.give(cb);
                continue; // wfg_join_kernel(l) finishes the row
            } else {
                ex = __dsub_rn(ex, frame_hv<P>(a.vals, s_r, pool, cb, ck, d - 1u, lane, &fail));
            }
            if (fail) {
                if (lane == 0) {
                    atomicOr(a.status, 1u);
                    L.row_term[g] = __longlong_as_double(0x7ff8000000000000LL);
                }
                pool.free = (1u << m) - 1u;
            } else if (lane == 0) {
                L.row_term[g] = slice_term<P>(a.vals, s_r, p, d, ex);
            }
        }
        finish();
    }
}

// The rows of level l whose frame went to level l + 1: H = the sum of that
// frame's sub-terms in order from 0.0, then the row's sub-term.
template <class P>
__global__ void wfg_join_kernel(wfg_args<P> a, wfg_ref ref, int l)
{
    chain_wait();
    const uint32_t d = first_dims(a) - static_cast<uint32_t>(l - 1), nw = P::words(d);
    const wfg_level<P> &L = a.lv[l], &C = a.lv[l + 1];
    const unsigned long long used = *L.rows_used;
    const unsigned long long rows = used < L.row_cap ? used : L.row_cap;
    for (unsigned long long g = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; g < rows;
         g += static_cast<unsigned long long>(gridDim.x) * blockDim.x) {
        uint32_t k = 0;
        unsigned long long off = 0;
        if (!row_of(a, l, g, &k, &off)) continue;
        const uint32_t ck = C.frame_k[g];
        const unsigned long long coff = C.frame_off[g];
        if (ck == 0u || coff + ck > C.row_cap) continue;
        double h = 0.0;
        for (uint32_t t = 0; t < ck; ++t) h = __dadd_rn(h, C.row_term[coff + t]);
        const typename P::word *p = L.frames + g * nw;
        L.row_term[g] = slice_term<P>(a.vals, ref.r, p, d, __dsub_rn(vol<P>(a.vals, ref.r, p, d - 1u), h));
    }
}

// The items with a frame at level 1: H = the sum of their rows' sub-terms in
// order from 0.0, then the item's value as wfg_top_kernel would give it.
template <class P>
__global__ void wfg_items_kernel(wfg_args<P> a, wfg_ref ref)
{
    chain_wait();
    const uint32_t m = a.m;
    const uint32_t dc = first_dims(a);
    const wfg_level<P> &L = a.lv[1];
    for (uint32_t item = blockIdx.x * blockDim.x + threadIdx.x; item < a.n; item += gridDim.x * blockDim.x) {
        const uint32_t k0 = L.frame_k[item];
        if (k0 == 0u) continue;
        const unsigned long long off = L.frame_off[item];
        double h = 0.0;
        for (uint32_t j = 0; j < k0; ++j) h = __dadd_rn(h, L.row_term[off + j]);
        const typename P::word *p = a.pts + static_cast<uint64_t>(item) * P::words(m);
        const double ex = __dsub_rn(vol<P>(a.vals, ref.r, p, dc), h);
        a.out[item] = a.contributions ? ex : slice_term<P>(a.vals, ref.r, p, m, ex);
    }
}

// The points as order keys (keys[i * m + c]).
__global__ void wfg_keys_kernel(const double *__restrict__ pts, uint64_t total, okey *__restrict__ keys)
{
    chain_wait();
    for (uint64_t e = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; e < total;
         e += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        keys[e] = to_key(pts[e]);
}

// Ranks of the points by hvwfg::cmp_points over m coordinates (ties by index),
// when order is set, and the number of smaller keys in each coordinate
// (coords[c n + i], when set): block (x, y) counts, for its 64 points, the
// points of slice y of the others (staged in shared memory); both arrays zero
// at launch. M: m itself up to 8, else at least m.
constexpr int kRankThreads = 64;
constexpr uint32_t kRankSlices = 32;

template <int M>
__global__ void __launch_bounds__(kRankThreads)
    wfg_rank_kernel(const okey *__restrict__ keys, uint32_t n, uint32_t m, unsigned *__restrict__ order,
                    unsigned *__restrict__ coords)
{
    chain_wait();
    __shared__ okey tile[kRankThreads * M];
    const uint32_t i = blockIdx.x * kRankThreads + threadIdx.x;
    okey mine[M];
    uint32_t below[M], cnt = 0;
#pragma unroll
    for (uint32_t c = 0; c < M; ++c) {
        mine[c] = i < n && c < m ? keys[static_cast<uint64_t>(i) * m + c] : 0;
        below[c] = 0u;
    }
    const uint32_t per = (n + kRankSlices - 1u) / kRankSlices;
    const uint32_t j_begin = blockIdx.y * per, j_end = min(n, j_begin + per);
    for (uint32_t j0 = j_begin; j0 < j_end; j0 += kRankThreads) {
        const uint32_t len = min(static_cast<uint32_t>(kRankThreads), j_end - j0);
        __syncthreads();
        for (uint32_t e = threadIdx.x; e < len * m; e += kRankThreads) tile[e] = keys[static_cast<uint64_t>(j0) * m + e];
        __syncthreads();
        if (i < n) {
            for (uint32_t jj = 0; jj < len; ++jj) {
                const okey *rj = tile + jj * m;
                bool first = j0 + jj < i; // of the coordinates so far: row jj before this one
#pragma unroll
                for (uint32_t c = 0; c < M; ++c) {
                    if (M <= 8 || c < m) {
                        const okey a = rj[c];
                        first = a > mine[c] || (a == mine[c] && first);
                        below[c] += a < mine[c] ? 1u : 0u;
                    }
                }
                cnt += first ? 1u : 0u;
            }
        }
    }
    if (i >= n) return;
    if (order != nullptr && cnt) atomicAdd(order + i, cnt);
    if (coords != nullptr) {
#pragma unroll
        for (uint32_t c = 0; c < M; ++c)
            if (c < m && below[c]) atomicAdd(coords + static_cast<uint64_t>(c) * n + i, below[c]);
    }
}

// sorted[rank[i]] = keys[i] (rows of m)
__global__ void wfg_scatter_kernel(const okey *__restrict__ keys, uint32_t n, uint32_t m,
                                   const unsigned *__restrict__ rank, okey *__restrict__ sorted)
{
    chain_wait();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        for (uint32_t c = 0; c < m; ++c) sorted[static_cast<uint64_t>(rank[i]) * m + c] = keys[static_cast<uint64_t>(i) * m + c];
}

// The points' rank rows (row order[i], or i), and the values of the ranks.
__global__ void wfg_pack_kernel(const okey *__restrict__ keys, uint32_t n, uint32_t m,
                                const unsigned *__restrict__ order, const unsigned *__restrict__ coords,
                                uint32_t *__restrict__ rows, double *__restrict__ tab)
{
    chain_wait();
    const uint32_t nw = (m + 1u) / 2u;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n * nw; t += gridDim.x * blockDim.x) {
        const uint32_t i = t / nw, w = t - i * nw;
        uint32_t word = 0;
        for (uint32_t c = 2u * w; c < min(m, 2u * w + 2u); ++c) {
            const uint32_t r = coords[static_cast<uint64_t>(c) * n + i];
            word |= r << (16u * (c & 1u));
            tab[static_cast<uint64_t>(c) * n + r] = from_key(keys[static_cast<uint64_t>(i) * m + c]);
        }
        rows[static_cast<uint64_t>(order != nullptr ? order[i] : i) * nw + w] = word;
    }
}

// out = the sum of term[0 .. n) in index order from 0.0 (compute_hv's
// H += ..., hv_hvwfg.cpp:262-266), each addition rounded as the reference's.
//
// One addition after the other is a chain of FP64 latencies (37 ns each: 74 us
// for 2000 terms). But while the sum h stays in one binade, with unit u, h is a
// multiple of u and h + t (t >= 0) rounds to h + u round(t / u), whatever h is,
// unless t / u lies halfway (then h's last bit decides): so such a run of
// additions is a sum of integers. The block scans the rounded terms of the
// next kSumThreads, takes all before the first that reaches the next binade,
// lies halfway or is no finite number in range, adds that one in FP64 (and some
// more after a short run, so that unlucky terms cost little beyond the chain),
// and goes on from the new h (n = 2000: 22 us).
constexpr int kSumThreads = 1024;
constexpr uint32_t kSumFew = 32; // terms added one by one at the start and after a shorter run

__global__ void __launch_bounds__(kSumThreads) wfg_sum_kernel(const double *__restrict__ term, uint32_t n,
                                                              double *__restrict__ out)
{
    chain_wait();
    __shared__ unsigned long long s_part[32], s_upto;
    __shared__ double s_h;
    __shared__ uint32_t s_stop;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    if (tid == 0) {
        double h = 0.0;
        for (uint32_t t = 0; t < min(n, kSumFew); ++t) h = __dadd_rn(h, term[t]);
        s_h = h;
    }
    __syncthreads();
    double h = s_h;
    for (uint32_t at = kSumFew; at < n;) {
        const uint32_t t = at + tid;
        const double a = t < n ? term[t] : 0.0;
        const unsigned long long hb = static_cast<unsigned long long>(__double_as_longlong(h));
        const int eh = static_cast<int>(hb >> 52);                    // (0 for a negative or subnormal h: below)
        const unsigned long long base = (hb & 0xfffffffffffffull) | (1ull << 52); // h = base 2^(eh - 1075)
        const bool usable = eh >= 1 && eh <= 2046;
        // a / u rounded to an integer, u = 2^(eh - 1075)
        const unsigned long long ab = static_cast<unsigned long long>(__double_as_longlong(a));
        const int ea = static_cast<int>((ab >> 52) & 0x7ffu);
        const unsigned long long ma = (ab & 0xfffffffffffffull) | (ea ? 1ull << 52 : 0ull);
        const int shift = eh - (ea ? ea : 1); // a / u = ma 2^-shift
        bool stop = !usable || (ab >> 63) != 0ull || shift < 0;
        unsigned long long q = 0;
        if (!stop) {
            if (shift == 0) {
                q = ma;
            } else if (shift <= 53) {
                const unsigned long long half = 1ull << (shift - 1), low = ma & ((1ull << shift) - 1ull);
                q = (ma >> shift) + (low > half ? 1ull : 0ull);
                stop = low == half;
            } // (else below half a unit)
        }
        if (t >= n) {
            stop = false;
            q = 0;
        }
        // inclusive sums, and the first term that cannot be taken this way
        unsigned long long incl = stop ? 0ull : q;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long x = __shfl_up_sync(kMask, incl, o);
            if (static_cast<int>(lane) >= o) incl += x;
        }
        if (tid == 0) s_stop = kSumThreads;
        if (lane == 31u) s_part[warp] = incl;
        __syncthreads();
        unsigned long long before = lane < warp ? s_part[lane] : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(kMask, before, o);
        incl += before;
        if (stop || base + incl >= (1ull << 53)) atomicMin(&s_stop, tid);
        __syncthreads();
        const uint32_t first = s_stop; // terms at .. at + first - 1 are taken, `more` are added one by one
        const uint32_t more = !usable ? kSumThreads : (first < kSumFew ? kSumFew : (first < kSumThreads ? 1u : 0u));
        if (tid + 1u == first || (first == 0u && tid == 0u)) s_upto = first ? base + incl : base;
        __syncthreads();
        if (tid == 0) {
            double v = h;
            if (first) // (below 2^53 units: exact)
                v = __longlong_as_double(static_cast<long long>((static_cast<unsigned long long>(eh) << 52)
                                                                | (s_upto & 0xfffffffffffffull)));
            for (uint32_t x = at + first; x < min(n, at + first + more); ++x) v = __dadd_rn(v, term[x]);
            s_h = v;
        }
        __syncthreads();
        h = s_h;
        at += first + more;
    }
    if (tid == 0) *out = h;
}

// The volume of one or two points (compute_hv's inclusion-exclusion,
// hv_hvwfg.cpp:201-211) and, with contribution_of_one, hypervolume's
// contribution of a lone point: |prod over c = 0 .. m-1 of (p_c - r_c)|
// (hypervolume.cpp:303-307 with volume_between on vectors,
// hv_algorithm.cpp:61-71).
__global__ void wfg_small_kernel(const double *__restrict__ pts, uint32_t n, uint32_t m, wfg_ref ref,
                                 int contribution_of_one, double *__restrict__ out)
{
    chain_wait();
    if (threadIdx.x != 0) return;
    const double *r = ref.r;
    if (contribution_of_one) {
        double v = 1.0;
        for (uint32_t c = 0; c < m; ++c) v = __dmul_rn(v, __dsub_rn(pts[c], r[c]));
        *out = v < 0.0 ? -v : v;
        return;
    }
    if (n == 1u) {
        *out = vol_d(r, pts, m);
        return;
    }
    const double h = __dadd_rn(vol_d(r, pts, m), vol_d(r, pts + m, m));
    double isect = 1.0;
    for (uint32_t c = 0; c < m; ++c) isect = __dmul_rn(isect, __dsub_rn(r[c], std_max(pts[c], pts[m + c])));
    *out = __dsub_rn(h, isect);
}

// 2-objective points as hv2d::contributions hands them to hv3d, as keys: a
// third coordinate 0 (hv_hv2d.cpp:135-143)
__global__ void wfg_lift2_kernel(const double *__restrict__ pts, uint32_t n, okey *__restrict__ out)
{
    chain_wait();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        out[3ull * i] = to_key(pts[2ull * i]);
        out[3ull * i + 1u] = to_key(pts[2ull * i + 1u]);
        out[3ull * i + 2u] = to_key(0.0);
    }
}

size_t round256(size_t b)
{
    return (b + 255u) & ~size_t(255);
}

// Scratch of the split kernels over n points of m coordinates: [counters,
// status, rows handed out | per level: per parent frame rows and first row,
// per row parent, sub-term and d keys | pool]; each level's list holds up to
// row_cap rows (past it a frame is finished by the warp that built it), the
// number of warps fits the pool in kPoolBytes (at least one warp).
constexpr size_t kPoolBytes = size_t(1) << 30;
constexpr uint64_t kRowCap = uint64_t(1) << 20;

template <class P>
int run_warps(pgx_context *ctx, const typename P::word *d_rows, const double *d_tab, uint32_t n, uint32_t m,
              const wfg_ref &ref, int contributions, double *d_out, cudaStream_t s)
{
    using word = typename P::word;
    const auto words = [](uint32_t d) { return sizeof(word) == sizeof(okey) ? d : (d + 1u) / 2u; };
    const uint64_t bd = static_cast<uint64_t>(n) * words(m); // a frame: at most n rows of at most m coordinates
    const size_t per_warp = static_cast<size_t>(m) * bd * sizeof(word);
    PGX_CHECK(per_warp <= (size_t(4) << 30), PGX_ERR_CAPACITY,
              "hypervolume (WFG): " + std::to_string(n) + " points of " + std::to_string(m) +
                  " objectives need more than 4 GiB of frames per warp");
    const uint32_t dc = contributions ? m : m - 1u;
    // levels 1 .. dc - 2 hold rows of dc .. 3 coordinates (a row of 3 has a frame of 2: closed form)
    const int levels = static_cast<int>(std::min<uint32_t>(kMaxLevels, dc > 3u ? dc - 2u : 1u));
    const uint64_t row_cap = std::max<uint64_t>(64u, std::min<uint64_t>(static_cast<uint64_t>(n) * n, kRowCap));
    // 32 warps per SM where the pool allows (the rows' kernels at n = 2000, m = 5: 165 us; 16: 255)
    const uint64_t want = static_cast<uint64_t>(ctx->num_sms) * 32u;
    const uint64_t fit = std::max<uint64_t>(1u, kPoolBytes / per_warp);
    uint64_t warps = std::min(want, fit);
    const unsigned blocks = static_cast<unsigned>((warps + kWarpsPerBlock - 1u) / kWarpsPerBlock);
    warps = static_cast<uint64_t>(blocks) * kWarpsPerBlock; // every warp of the grid has its slice
    const size_t b_ctl = 256u;
    size_t head = b_ctl;
    size_t lv_off[kMaxLevels + 2][5] = {};
    for (int l = 1; l <= levels; ++l) {
        const uint64_t parents = l == 1 ? n : row_cap;
        const uint32_t d = dc - static_cast<uint32_t>(l - 1);
        lv_off[l][0] = head; // frame_k
        head += round256(parents * sizeof(uint32_t));
        lv_off[l][1] = head; // frame_off
        head += round256(parents * sizeof(unsigned long long));
        lv_off[l][2] = head; // row_parent
        head += round256(row_cap * sizeof(uint32_t));
        lv_off[l][3] = head; // row_term
        head += round256(row_cap * sizeof(double));
        lv_off[l][4] = head; // frames
        head += round256(row_cap * words(d) * sizeof(word));
    }
    PGX_TRY(ctx->h_wfg.ensure(head + warps * per_warp));
    char *base = ctx->h_wfg.as<char>();
    unsigned *ctl = reinterpret_cast<unsigned *>(base);
    PGX_CUDA(cudaMemsetAsync(ctl, 0, b_ctl, s));
    wfg_args<P> a{};
    a.pts = d_rows;
    a.vals = wfg_values{d_tab, n};
    a.n = n;
    a.m = m;
    a.contributions = contributions;
    a.out = d_out;
    a.pool = reinterpret_cast<word *>(base + head);
    a.bd = bd;
    a.next = ctl;
    a.status = ctl + 1;
    a.levels = levels;
    for (int l = 1; l <= levels; ++l) {
        wfg_level<P> &L = a.lv[l];
        L.frame_k = reinterpret_cast<uint32_t *>(base + lv_off[l][0]);
        L.frame_off = reinterpret_cast<unsigned long long *>(base + lv_off[l][1]);
        L.row_parent = reinterpret_cast<uint32_t *>(base + lv_off[l][2]);
        L.row_term = reinterpret_cast<double *>(base + lv_off[l][3]);
        L.frames = reinterpret_cast<word *>(base + lv_off[l][4]);
        L.rows_used = reinterpret_cast<unsigned long long *>(base + 64u + 8u * static_cast<size_t>(l));
        L.row_cap = row_cap;
        L.parents = l == 1 ? n : row_cap;
    }
    const int threads = kWarpsPerBlock * 32;
    PGX_CUDA(launch_chained(wfg_top_kernel<P>, std::min<unsigned>(blocks, n), threads, 0, s, a, ref));
    for (int l = 1; l <= levels; ++l) PGX_CUDA(launch_chained(wfg_rows_kernel<P>, blocks, threads, 0, s, a, ref, l));
    const unsigned jb = static_cast<unsigned>(std::min<uint64_t>((row_cap + 127u) / 128u, 4096u));
    for (int l = levels - 1; l >= 1; --l) {
        PGX_CUDA(launch_chained(wfg_join_kernel<P>, jb, 128, 0, s, a, ref, l));
    }
    PGX_CUDA(launch_chained(wfg_items_kernel<P>, (n + 127u) / 128u, 128, 0, s, a, ref));
    ctx->launches += 2u + 2u * static_cast<uint64_t>(levels);
    return PGX_OK;
}

// Scratch of ranked_keys beyond the keys: rows | order | coords | table.
size_t ranked_bytes(uint32_t n, uint32_t m)
{
    const size_t nm = static_cast<size_t>(n) * m;
    return round256(nm * sizeof(uint32_t)) + round256((n + nm) * sizeof(unsigned)) + round256(nm * sizeof(double));
}

// The points' keys sorted (with sort) and ranked, then the kernels above.
// base: ranked_bytes(n, m) for up to kRankLimit points, else a second n m keys
// and n ranks.
int run_keys(pgx_context *ctx, const okey *d_keys, char *base, uint32_t n, uint32_t m, const wfg_ref &ref, bool sort,
             double *d_out, cudaStream_t s)
{
    const int contributions = sort ? 0 : 1;
    const bool ranked = n <= kRankLimit;
    const size_t nm = static_cast<size_t>(n) * m;
    const size_t b_rows = round256(nm * (ranked ? sizeof(uint32_t) : sizeof(okey)));
    unsigned *order = reinterpret_cast<unsigned *>(base + b_rows), *coords = order + n;
    double *tab = reinterpret_cast<double *>(base + b_rows + round256((n + nm) * sizeof(unsigned)));
    if (sort || ranked) {
        PGX_CUDA(cudaMemsetAsync(order, 0, (n + (ranked ? nm : 0u)) * sizeof(unsigned), s));
        const auto kernel = m == 2u   ? wfg_rank_kernel<2>
                            : m == 3u ? wfg_rank_kernel<3>
                            : m == 4u ? wfg_rank_kernel<4>
                            : m == 5u ? wfg_rank_kernel<5>
                            : m == 6u ? wfg_rank_kernel<6>
                            : m == 7u ? wfg_rank_kernel<7>
                            : m == 8u ? wfg_rank_kernel<8>
                                      : wfg_rank_kernel<16>;
        PGX_CUDA(launch_chained(kernel, dim3((n + kRankThreads - 1u) / kRankThreads, kRankSlices), kRankThreads, 0, s, d_keys,
                                n, m, sort ? order : nullptr, ranked ? coords : nullptr));
        ++ctx->launches;
    }
    if (ranked) {
        uint32_t *rows = reinterpret_cast<uint32_t *>(base);
        PGX_CUDA(launch_chained(wfg_pack_kernel, (n + 127u) / 128u, 128, 0, s, d_keys, n, m, sort ? order : nullptr, coords,
                                rows, tab));
        ++ctx->launches;
        const uint32_t dc = contributions ? m : m - 1u;
        if (dc <= 4u) return run_warps<rank_rows<2>>(ctx, rows, tab, n, m, ref, contributions, d_out, s);
        if (dc <= 6u) return run_warps<rank_rows<3>>(ctx, rows, tab, n, m, ref, contributions, d_out, s);
        if (dc <= 8u) return run_warps<rank_rows<4>>(ctx, rows, tab, n, m, ref, contributions, d_out, s);
        return run_warps<rank_rows<8>>(ctx, rows, tab, n, m, ref, contributions, d_out, s);
    }
    const okey *rows = d_keys;
    if (sort) {
        okey *sorted = reinterpret_cast<okey *>(base);
        PGX_CUDA(launch_chained(wfg_scatter_kernel, (n + 255u) / 256u, 256, 0, s, d_keys, n, m, order, sorted));
        ++ctx->launches;
        rows = sorted;
    }
    if (m <= 4u) return run_warps<key_rows<4>>(ctx, rows, nullptr, n, m, ref, contributions, d_out, s);
    if (m <= 8u) return run_warps<key_rows<8>>(ctx, rows, nullptr, n, m, ref, contributions, d_out, s);
    return run_warps<key_rows<16>>(ctx, rows, nullptr, n, m, ref, contributions, d_out, s);
}

size_t run_keys_bytes(uint32_t n, uint32_t m)
{
    return n <= kRankLimit ? ranked_bytes(n, m)
                           : round256(static_cast<size_t>(n) * m * sizeof(okey)) + round256(n * sizeof(unsigned));
}

// A call that runs no warp kernel leaves a zero status behind.
int clear_status(pgx_context *ctx, cudaStream_t s)
{
    if (ctx->h_wfg.ptr != nullptr) PGX_CUDA(cudaMemsetAsync(ctx->h_wfg.ptr, 0, 256u, s));
    return PGX_OK;
}

wfg_ref make_ref(const double *r, uint32_t m)
{
    wfg_ref w{};
    for (uint32_t c = 0; c < m; ++c) w.r[c] = r[c];
    return w;
}

} // namespace

int launch_wfg_compute(pgx_context *ctx, const double *d_pts, uint32_t n, uint32_t m, const double *r,
                       double *d_out, cudaStream_t s)
{
    PGX_CHECK(m >= 2u && m <= kWfgMaxObjectives, PGX_ERR_NOTIMPL,
              "hypervolume on the GPU: at most " + std::to_string(kWfgMaxObjectives) + " objectives; " +
                  std::to_string(m) + " given");
    const wfg_ref ref = make_ref(r, m);
    if (n <= 2u) {
        PGX_TRY(clear_status(ctx, s));
        PGX_CUDA(launch_chained(wfg_small_kernel, 1, 32, 0, s, d_pts, n, m, ref, 0, d_out));
        ++ctx->launches;
        return PGX_OK;
    }
    // keys | terms | run_keys' scratch
    const size_t b_keys = round256(static_cast<size_t>(n) * m * sizeof(okey));
    const size_t b_terms = round256(static_cast<size_t>(n) * sizeof(double));
    PGX_TRY(ctx->s_crowd.ensure(b_keys + b_terms + run_keys_bytes(n, m)));
    char *base = ctx->s_crowd.as<char>();
    okey *keys = reinterpret_cast<okey *>(base);
    double *terms = reinterpret_cast<double *>(base + b_keys);
    const uint64_t total = static_cast<uint64_t>(n) * m;
    const unsigned g = static_cast<unsigned>(std::min<uint64_t>((total + 255u) / 256u, 8192u));
    PGX_CUDA(launch_chained(wfg_keys_kernel, g, 256, 0, s, d_pts, total, keys));
    PGX_TRY(run_keys(ctx, keys, base + b_keys + b_terms, n, m, ref, true, terms, s));
    PGX_CUDA(launch_chained(wfg_sum_kernel, 1, kSumThreads, 0, s, terms, n, d_out));
    ctx->launches += 2;
    return PGX_OK;
}

int launch_wfg_contributions(pgx_context *ctx, const double *d_pts, uint32_t n, uint32_t m, const double *r,
                             double *d_out, cudaStream_t s)
{
    PGX_CHECK(m >= 2u && m <= kWfgMaxObjectives, PGX_ERR_NOTIMPL,
              "hypervolume on the GPU: at most " + std::to_string(kWfgMaxObjectives) + " objectives; " +
                  std::to_string(m) + " given");
    if (n == 1u) {
        PGX_TRY(clear_status(ctx, s));
        PGX_CUDA(launch_chained(wfg_small_kernel, 1, 32, 0, s, d_pts, n, m, make_ref(r, m), 1, d_out));
        ++ctx->launches;
        return PGX_OK;
    }
    const uint32_t mk = m == 2u ? 3u : m; // 2 objectives: hv3d's points with a third coordinate 0
    const size_t b_keys = round256(static_cast<size_t>(n) * mk * sizeof(okey));
    PGX_TRY(ctx->s_crowd.ensure(b_keys + run_keys_bytes(n, mk)));
    okey *keys = ctx->s_crowd.as<okey>();
    char *scratch = ctx->s_crowd.as<char>() + b_keys;
    if (m == 2u) {
        const unsigned g = static_cast<unsigned>(std::min<uint64_t>((n + 255u) / 256u, 4096u));
        PGX_CUDA(launch_chained(wfg_lift2_kernel, g, 256, 0, s, d_pts, n, keys));
        ++ctx->launches;
        const double r3[3] = {r[0], r[1], 1.0};
        return run_keys(ctx, keys, scratch, n, 3u, make_ref(r3, 3u), false, d_out, s);
    }
    const uint64_t total = static_cast<uint64_t>(n) * m;
    const unsigned g = static_cast<unsigned>(std::min<uint64_t>((total + 255u) / 256u, 8192u));
    PGX_CUDA(launch_chained(wfg_keys_kernel, g, 256, 0, s, d_pts, total, keys));
    ++ctx->launches;
    return run_keys(ctx, keys, scratch, n, m, make_ref(r, m), false, d_out, s);
}

int wfg_status(pgx_context *ctx, unsigned *status)
{
    *status = 0;
    if (ctx->h_wfg.ptr == nullptr) return PGX_OK;
    PGX_CUDA(cudaMemcpyAsync(status, ctx->h_wfg.as<unsigned>() + 1, sizeof(unsigned), cudaMemcpyDeviceToHost,
                             ctx->stream));
    PGX_CUDA(cudaStreamSynchronize(ctx->stream));
    return PGX_OK;
}

} // namespace pgx

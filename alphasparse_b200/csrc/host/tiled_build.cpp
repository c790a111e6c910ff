// Builds the column-tiled layout of a plan group (kernels_tiled.cu) from its template arrays, and decides whether the
// group is better off with it. One pass over the stored elements counts them per tile of x, one scatters them to
// their tiles (order of the rows kept). Then every tile is cut into blocks of whole rows that are turned into slices independently
// of one another, or, where rows have few elements in a tile, its elements stay in order and are units of a warp each.
#include <string.h>

#include <algorithm>
#include <cmath>

#include "../tiled.h"
#include "crew.hpp"

namespace asp
{
namespace
{
typedef uint64_t u64;
typedef uint32_t u32;

using host::for_each;
using host::share_pieces;
using host::share_ranges;
using host::share_steps;

// (What the threads of a shared loop work in is allocated before it: an exception that leaves a piece ends the process.)
// counters of every thread, on cache lines of their own
struct ThreadCounters
{
    const u64 stride;
    std::vector<u64> all;
    ThreadCounters(u64 count, unsigned threads) : stride((count + 15) / 8 * 8), all(stride * threads, 0) {}
    u64 *of(unsigned who) { return all.data() + stride * who; }
};

u64 row_in_y(const TiledSource &s, u64 r)
{
    if (s.a->sort_kind == ASP_SORT_GLOBAL) return s.perm->get(r + s.a->first_row);
    if (s.a->sort_kind == ASP_SORT_LOCAL) return s.perm->get(r) + s.a->first_row;
    return r + s.a->first_row;
}

// units (what a walk can start at) of a sub-matrix, 0: the template is not walked here
u64 unit_count(const TiledSource &s)
{
    switch (s.templ)
    {
    case ASP_DIRECT_ATOM_TEMPLATE_WARP_BLOCK_COMPRESS:
    case ASP_DIRECT_ATOM_TOTAL_WARP_REDUCE_TEMPLATE: return s.a->effective;
    case ASP_DIRECT_ATOM_TEMPLATE_WARP_COMPRESS:
    case ASP_SHARED_MEMORY_TEMPLATE_WARP_COMPRESS:
    case ASP_SHARED_MEMORY_TOTAL_WARP_REDUCE_TEMPLATE:
    case ASP_SHARED_MEMORY_LONG_ROW_TEMPLATE:
    case ASP_UNALIGNED_WARP_REDUCE_SAME_TLB_SIZE_TEMPLATE:
    case ASP_UNALIGNED_WARP_REDUCE_SAME_TLB_SIZE_TEMPLATE_WITH_WARP_REDUCE: return s.a->n_units;
    default: return 0;
    }
}

// (ASP_INLINE per element, in every template's loop: as calls, which the compiler makes of the seventh use, a third slower.)
// f(row of y, column of x, value) for every element that units [u0, u1) store. What a format adds to fill a TLB (a zero
// that repeats the column before it in the same row) is left out.
template <class VT, class CT, class F>
void walk(const TiledSource &s, u64 u0, u64 u1, F &&f)
{
    const VT *val = (const VT *)s.val;
    const CT *col = (const CT *)s.col;
    const KArgs &a = *s.a;
    const u64 c0 = a.first_col, radd = a.row_add ? a.first_row : 0;
    const HostMeta *m = s.m;
    u64 last_row = ~0ull, last_col = ~0ull;
    auto put = [&](u64 row, u64 at) ASP_INLINE {
        const u64 c = (u64)col[at] + c0;
        const VT v = val[at];
        if (v == VT(0) && row == last_row && c == last_col) return;
        last_row = row;
        last_col = c;
        f(row, c, v);
    };
    switch (s.templ)
    {
    case ASP_DIRECT_ATOM_TEMPLATE_WARP_BLOCK_COMPRESS:
        for (u64 t = u0; t < u1; t++)
        {
            const u64 row = m[MS_ROW_OF_TLB].get(t) + radd;
            for (u64 k = 0; k < a.tlb_size; k++) put(row, t + k * a.n_tlb);
        }
        return;
    case ASP_DIRECT_ATOM_TEMPLATE_WARP_COMPRESS:
        for (u64 b = u0; b < u1; b++)
        {
            const u64 nz = m[MS_BLK_NZ].get(b), t0 = m[MS_BLK_THR].get(b), n = m[MS_BLK_THR].get(b + 1) - t0, S = m[MS_TLB_SIZE].get(b);
            for (u64 i = 0; i < n && t0 + i < a.effective; i++)
            {
                const u64 row = m[MS_ROW_OF_TLB].get(t0 + i) + radd;
                for (u64 k = 0; k < S; k++) put(row, nz + i + k * n);
            }
        }
        return;
    case ASP_SHARED_MEMORY_TEMPLATE_WARP_COMPRESS:
        for (u64 b = u0; b < u1; b++)
        {
            const u64 nz = m[MS_BLK_NZ].get(b), n = m[MS_BLK_THR].get(b + 1) - m[MS_BLK_THR].get(b), S = m[MS_TLB_SIZE].get(b);
            const u64 r0 = m[MS_BLK_ROW].get(b), r1 = std::min<u64>(m[MS_BLK_ROW].get(b + 1), a.effective), g0 = m[MS_ROW_OFF].get(r0);
            for (u64 r = r0; r < r1; r++)
            {
                const u64 row = row_in_y(s, r), e = m[MS_ROW_OFF].get(r + 1) - g0;
                for (u64 i = m[MS_ROW_OFF].get(r) - g0; i < e; i++)
                    for (u64 k = 0; k < S; k++) put(row, nz + i + k * n);
            }
        }
        return;
    case ASP_SHARED_MEMORY_TOTAL_WARP_REDUCE_TEMPLATE:
        for (u64 b = u0; b < u1; b++)
        {
            const u64 w0 = m[MS_BLK_WARP].get(b), r0 = m[MS_BLK_ROW].get(b), r1 = std::min<u64>(m[MS_BLK_ROW].get(b + 1), a.effective), g0 = m[MS_ROW_OFF].get(r0);
            for (u64 r = r0; r < r1; r++)
            {
                const u64 row = row_in_y(s, r), e = w0 + m[MS_ROW_OFF].get(r + 1) - g0;
                for (u64 w = w0 + m[MS_ROW_OFF].get(r) - g0; w < e; w++)
                    for (u64 k = m[MS_WARP_NZ].get(w); k < m[MS_WARP_NZ].get(w + 1); k++) put(row, k);
            }
        }
        return;
    case ASP_DIRECT_ATOM_TOTAL_WARP_REDUCE_TEMPLATE:
    case ASP_SHARED_MEMORY_LONG_ROW_TEMPLATE:
    {
        const HostMeta &nz = m[s.templ == ASP_SHARED_MEMORY_LONG_ROW_TEMPLATE ? MS_BLK_NZ : MS_WARP_NZ];
        for (u64 u = u0; u < u1; u++)
        {
            const u64 row = m[MS_ROW_OF_UNIT].get(u) + radd, e = nz.get(u + 1);
            for (u64 k = nz.get(u); k < e; k++) put(row, k);
        }
        return;
    }
    default: // CSR5-like: the flags of a thread's word say which of its elements start a row; a warp's first element always does
        for (u64 w = u0; w < u1; w++)
        {
            const u64 R0 = m[MS_ROW_OF_UNIT].get(w), S = a.tlb_size;
            u64 row = ~0ull;
            for (u64 l = 0; l < 32; l++)
            {
                const u64 word = m[MS_COMBINE].get(w * 32 + l);
                u64 r = R0 + (word & ((1ull << a.bits_row) - 1));
                for (u64 k = 0; k < S; k++)
                {
                    if ((word >> (a.bits_word - 1 - (int)k)) & 1ull) row = row_in_y(s, r++);
                    if (row != ~0ull) put(row, w * 32 * S + k * 32 + l);
                }
            }
        }
    }
}

template <class VT, class F>
void walk_any(const TiledSource &s, u64 u0, u64 u1, F &&f)
{
    if (s.col_bytes == 1) walk<VT, uint8_t>(s, u0, u1, f);
    else if (s.col_bytes == 2) walk<VT, uint16_t>(s, u0, u1, f);
    else walk<VT, uint32_t>(s, u0, u1, f);
}

// Cache lines of x that one warp-wide gather of the group's own kernels touches, per lane (1: every lane another line).
// Sampled; the kernels with 16-byte lanes gather elements 4 l + j of 128 adjacent ones at a time, the others 32 adjacent ones.
double lines_per_gather(const TiledSource &s, bool f64)
{
    // (and so do those for whole rows)
    const bool by4 = !s.whole_rows && (s.templ == ASP_DIRECT_ATOM_TEMPLATE_WARP_BLOCK_COMPRESS || s.templ == ASP_DIRECT_ATOM_TEMPLATE_WARP_COMPRESS ||
                     s.templ == ASP_SHARED_MEMORY_TEMPLATE_WARP_COMPRESS || s.templ == ASP_SHARED_MEMORY_LONG_ROW_TEMPLATE);
    const u64 groups = s.stored / 128, samples = std::min<u64>(groups, 64), per_line = f64 ? 16 : 32;
    if (samples == 0) return 0.0;
    u64 lines = 0;
    for (u64 q = 0; q < samples; q++)
    {
        const u64 base = groups * q / samples * 128;
        for (int j = 0; j < 4; j++)
        {
            u64 ln[32];
            for (int l = 0; l < 32; l++)
            {
                const u64 at = base + (by4 ? 4 * l + j : 32 * j + l);
                const u64 c = s.col_bytes == 1 ? ((const uint8_t *)s.col)[at] : s.col_bytes == 2 ? ((const uint16_t *)s.col)[at] : ((const u32 *)s.col)[at];
                ln[l] = c / per_line;
            }
            std::sort(ln, ln + 32);
            lines += (u64)(std::unique(ln, ln + 32) - ln);
        }
    }
    return (double)lines / (double)(samples * 128);
}

// How close the elements of a row lie, 1: in adjacent columns. Sampled over some 4,000 of them (20,000 took 0.1 ms).
template <class VT>
double closeness(const TiledSource &s)
{
    const u64 units = unit_count(s), samples = std::min<u64>({units, 64, std::max<u64>(2, 4000 * units / std::max<u64>(1, s.stored))});
    u64 pairs = 0, columns = 0, last_row = ~0ull, last = 0;
    for (u64 q = 0; q < samples; q++)
    {
        const u64 u = units * q / samples;
        walk_any<VT>(s, u, u + 1, [&](u64 row, u64 c, VT) ASP_INLINE {
            if (row == last_row) pairs++, columns += c > last ? c - last : last - c;
            last_row = row;
            last = c;
        });
        last_row = ~0ull;
    }
    return pairs == 0 ? 0.0 : std::min(1.0, (double)pairs / (double)std::max<u64>(1, columns));
}

bool is_csr5(const TiledSource &s)
{
    return s.templ == ASP_UNALIGNED_WARP_REDUCE_SAME_TLB_SIZE_TEMPLATE || s.templ == ASP_UNALIGNED_WARP_REDUCE_SAME_TLB_SIZE_TEMPLATE_WITH_WARP_REDUCE;
}

// Microseconds of the longest serial chain of the template's own kernel: a thread of the SELL- and ELL-like kernels walks its
// TLB four elements a trip (index, then x: 1.4 us where few warps run), a CTA of the row-grouped kernel its strip's TLBs, a
// thread of the CSR5-like ones its TLB eight elements a trip and then the tails of its warp.
double chain_us(const TiledSource &s)
{
    u64 trips = 0;
    if (s.templ == ASP_DIRECT_ATOM_TEMPLATE_WARP_BLOCK_COMPRESS) trips = (s.a->tlb_size + 3) / 4;
    else if (s.templ == ASP_DIRECT_ATOM_TEMPLATE_WARP_COMPRESS)
        for (u64 b = 0; b < s.a->n_units; b++) trips = std::max<u64>(trips, (s.m[MS_TLB_SIZE].get(b) + 3) / 4);
    else if (s.templ == ASP_SHARED_MEMORY_TEMPLATE_WARP_COMPRESS)
        for (u64 b = 0; b < s.a->n_units; b++)
        {
            const u64 per_trip = 4 * std::max(32u, s.threads), n = s.m[MS_BLK_THR].get(b + 1) - s.m[MS_BLK_THR].get(b);
            trips = std::max<u64>(trips, (n + per_trip - 1) / per_trip * ((s.m[MS_TLB_SIZE].get(b) + 3) / 4));
        }
    else if (is_csr5(s)) return 3.5 + 1.4 * (double)((s.a->tlb_size + 7) / 8);
    return 1.4 * (double)trips;
}
// how far the template's own kernel stays below the rate of its gathers or bytes (measured, 80 non-zeros a row, random columns)
double slowness(const TiledSource &s)
{
    return s.templ == ASP_DIRECT_ATOM_TOTAL_WARP_REDUCE_TEMPLATE ? 1.45 : s.templ == ASP_SHARED_MEMORY_TOTAL_WARP_REDUCE_TEMPLATE ? 2.35 : 1.1;
}

// How many parts of a row may be added up in y itself: as many as its template's thread adds elements one after the other, so
// that the rounding errors of the parts are no more than those of the elements; 8 where a tree follows the thread's few elements
// (K4, K6, K7, K8 leave about seven roundings in a row of 80). R-MAT scale 20, fp32, TLBs of 32, distance from the 64-bit result:
// the template 4.9e-8 to 5.9e-8; all rows direct 13e-8; limit 128: 4.9e-8, 32: 3.4e-8, 8: 2.4e-8 (scale 21, ten SpMVs: 485, 490, 505 and
// 530 us).
u64 most_direct(const TiledSource &s)
{
    u64 tlb = 0;
    if (s.templ == ASP_DIRECT_ATOM_TEMPLATE_WARP_BLOCK_COMPRESS || is_csr5(s)) tlb = s.a->tlb_size;
    else if (s.templ == ASP_DIRECT_ATOM_TEMPLATE_WARP_COMPRESS || s.templ == ASP_SHARED_MEMORY_TEMPLATE_WARP_COMPRESS)
        for (u64 b = 0; b < s.a->n_units; b++) tlb = std::max<u64>(tlb, s.m[MS_TLB_SIZE].get(b));
    return std::max<u64>(8, tlb);
}
// a part's share of what its row may have (sub-matrices of one row may allow different numbers)
const u32 kDirectShares = 256;
u32 share_of_part(const TiledSource &s) { return (u32)std::max<u64>(1, (kDirectShares + most_direct(s) - 1) / most_direct(s)); }

const u32 kMaxPiece = 32;    // elements of a row's piece: bounds the serial chain of a lane and the padding of a slice
const u32 kWindow = 1024;    // pieces that are sorted by length together: lanes of a slice stay near in y
// Units or slices. A slice's `red` of a warp goes to the rows of 32 pieces of one length, anywhere among 1024 pieces; a unit's goes to
// neighbouring rows, but a unit takes more instructions an element. fp32, random columns, 80 a row, slices / units: 25 tiles 38.2 / 31.2 us
// (200,000 rows), 20 tiles 13.3 / 9.7 (40,000 rows), 13 tiles 9.1 / 6.6 (20,000), 8 tiles 21.3 / 21.0 (150,000), 3 tiles 18.7 / 20.4. Long
// runs: 9,001 rows of 2000 in 25 tiles 25.0 / 28.8, R-MAT scale 21 (8.5 a run) 476 / 643. Rows far apart (strips sorted by length) 19.7 /
// 24.3. fp64 stays with slices: 19 tiles 33.5 / 31.2 us, but 0.95e-16 / 1.27e-16 from the exact sums (the scan's roundings; fp32 4.2e-8 /
// 2.5e-8).
const u64 kRunForUnits = 7;  // at most so many elements a run, on average
const u64 kNearRows = 4;     // and three quarters of the runs at most so many rows behind the run before
const double kRowCost = 1.0; // of a row of a unit, in elements: its entry and its `red`
// fp64: 16 warps, with twice the steps on their way each, or 32. A warp's wait for the steps after these is what most of its time goes to, unless
// most of its slices are a few steps long; those are a chain of their own, of which 32 warps have more under way. 32 / 16, us: FEM of 196,611
// rows 32.9 / 31.4, 30,000 nodes of 17 blocks 13.5 / 11.7; 190,000 rows of 80 in 40 tiles 52.8 / 60.8, in 10 tiles 35.6 / 38. Where rows have several sums
// 16 are no faster (104,543 rows of 80 in 4 tiles 20.4 / 20.7). (fp32 is slower with 16: R-MAT scale 21 46 / 58, 9,001 rows of 2000 24.1 / 24.3.)
// Long streams fill the memory's rate either way: FEM, 27 blocks, 21.9 M elements 42.4 / 40.8, 31.9 M 58.7 / 58.8, 63.7 M 111.2 / 113.5.
const u64 kFewWarpsMost = 26u << 20;
const u64 kDeep = 14; // elements of a long piece; half of all elements are in such: 16
const double kSliceCost = 4.0; // in steps; with 2 the CTAs of sparse tiles ran twice as long as the others
// elements of a block of whole rows, the unit of the parallel build: enough blocks for all cores, and whole windows in each
u64 block_size(u64 n) { return std::min<u64>(1u << 16, std::max<u64>(1u << 13, n / 128)); }

// Shares out what lies in order, tile by tile (begin[t], ..., begin[C]), among the CTAs and their warps: with cost(i) before place i
// and tile_cost for every tile that a CTA loads, so that the largest cost of a CTA is the least that will do (filling the CTAs up to the average,
// one of them had up to twice the others' work: 20,000 rows of 40..120 among 490 K columns 9.8 -> 9.1 us, 9,001 rows of 1000..3000
// 26.3 -> 25.0). at(cost, lo, hi): the place in [lo, hi] that a cost is reached at. A CTA's visits of tiles are `warps` entries of four words
// each, its first one at its own number: put(entry, from, to, tile), link(entry, next visit).
template <class Cost, class At, class Put, class Link>
void share_out(int n_sm, u32 warps, const std::vector<u64> &begin, double tile_cost, const Cost &cost, const At &at, std::vector<u32> &work, const Put &put, const Link &link)
{
    const u64 C = begin.size() - 1, n = begin[C];
    struct Visit
    {
        u64 cta, s, e, tile;
    };
    std::vector<Visit> visits;
    std::vector<double> tile_at(C + 1);
    for (u64 t = 0; t <= C; t++) tile_at[t] = cost(begin[t]);
    // every CTA takes what it can do at a cost of `most`: true, if that is everything
    auto fill = [&](double most) {
        visits.clear();
        u64 s = 0, t = 0;
        double from = 0; // cost(s), but for what one place costs
        for (int cta = 0; cta < n_sm && s < n; cta++)
        {
            double left = most;
            for (bool first = true; s < n && (first || left > tile_cost + warps); first = false)
            {
                while (begin[t + 1] <= s) t++;
                left -= tile_cost;
                const u64 last = begin[t + 1], e = tile_at[t + 1] - from <= left ? last : std::min(last, std::max(s + 1, at(from + left, s, last)));
                visits.push_back({(u64)cta, s, e, t});
                const double to = e < last ? std::max(from, from + left) : tile_at[t + 1];
                left -= to - from;
                from = to;
                s = e;
                if (e < last) break;
            }
        }
        return s == n;
    };
    // to half a percent: eight times 150 searches (a tenth of a millisecond)
    double lo = tile_at[C] / n_sm, hi = (tile_at[C] + tile_cost * (double)(C + (u64)n_sm)) / n_sm;
    while (!fill(hi)) lo = hi, hi *= 1.25;
    while (hi - lo > 0.005 * hi)
    {
        const double mid = (lo + hi) / 2;
        (fill(mid) ? hi : lo) = mid;
    }
    fill(hi);
    work.assign((size_t)n_sm * warps * 4, 0);
    std::vector<u64> place(visits.size());
    for (size_t i = 0; i < visits.size(); i++)
    {
        place[i] = visits[i].cta;
        if (i == 0 || visits[i].cta != visits[i - 1].cta) continue;
        place[i] = work.size() / (warps * 4);
        work.resize(work.size() + warps * 4, 0);
        for (u32 w = 0; w < warps; w++) link(&work[(place[i - 1] * warps + w) * 4], place[i]);
    }
    // (thousands of warps: half of the time of the build when it was done by one thread)
    for_each(visits.size(), true, [&](u64 i) {
        const Visit &v = visits[i];
        const double from = cost(v.s), all = cost(v.e) - from;
        u64 here = v.s;
        for (u32 w = 0; w < warps; w++)
        {
            const u64 to = w + 1 == warps ? v.e : at(from + all * (w + 1) / warps, here, v.e);
            put(&work[(place[i] * warps + w) * 4], here, to, v.tile);
            here = to;
        }
    });
}

struct Chunk
{
    int sub;
    u64 u0, u1;
};

template <class VT>
struct Builder
{
    const std::vector<TiledSource> &src;
    const u64 n_rows, n_cols;
    static constexpr u32 TW = tiled_tile_cols(sizeof(VT) == 8);
    const u64 C; // tiles of x
    const unsigned width = host::crew_width();
    unsigned warps = kTiledWarps; // of a CTA
    // of a warp's share, about: longer pieces are cut, and every cut is one more part of their rows. Of 32 warps: that there are 16 follows from what is counted
    // with it, and those cut less.
    const u64 warp_steps;
    std::vector<Chunk> chunks;
    std::vector<u64> at; // [chunk * C + tile]: first its count, then where its elements go
    std::vector<u64> tile_begin, tile_pieces;
    u64 N = 0, runs = 0, near_runs = 0, deep = 0; // elements; rows' runs in the tiles, and those that lie near the one before; elements of long pieces
    std::vector<u32> row_code; // of every row of y: the shares of its parts, then what stands for it among the slices' rows
    // elements in tile order
    HostBuf<u32> e_row;
    HostBuf<uint16_t> e_col;
    HostBuf<VT> e_val;

    Builder(const std::vector<TiledSource> &s, u64 rows, u64 cols, u64 nnz, int n_sm)
        : src(s), n_rows(rows), n_cols(cols), C((cols + TW - 1) / TW), warp_steps(std::max<u64>(1, nnz / ((u64)n_sm * kTiledWarps * kTiledSlice)))
    {
    }

    // whether a run of row r is a near one behind one of row `before`
    static u64 near(u64 before, u64 r) { return r - before <= kNearRows ? 1 : 0; }
    void count()
    {
        u64 stored = 0;
        for (const TiledSource &s : src) stored += s.stored;
        const u64 want = (u64)width * 4;
        for (size_t i = 0; i < src.size(); i++)
        {
            const u64 units = unit_count(src[i]), parts = std::max<u64>(1, std::min<u64>(units, want * src[i].stored / std::max<u64>(stored, 1)));
            for (u64 p = 0; p < parts; p++) chunks.push_back({(int)i, units * p / parts, units * (p + 1) / parts});
        }
        at.assign(chunks.size() * C, 0);
        tile_pieces.assign(C, 0);
        row_code.assign(n_rows, 0);
        std::vector<u32> share;
        for (const TiledSource &s : src) share.push_back(share_of_part(s));
        ThreadCounters pieces_of_thread(C, width), n_of_thread(C, width); // (neighbours in `at` share cache lines)
        const size_t edges = (2 * C + 31) / 16 * 16;
        std::vector<u32> edge(chunks.size() * edges); // rows of a chunk's first and last element in a tile, on cache lines of its own
        std::atomic<u64> sum_runs(0), sum_near(0), sum_deep(0);
        share_steps(chunks.size(), 1, width, [&](u64 c, u64, unsigned who) {
            u64 *const pieces = pieces_of_thread.of(who), *const n = n_of_thread.of(who);
            u64 all_runs = 0, all_near = 0, all_deep = 0;
            std::fill(n, n + C, 0);
            u32 *const first = edge.data() + (size_t)c * edges, *const last = first + C;
            u64 row = ~0ull, tile = ~0ull, run = 0;
            u32 of_row = 0, elements = 0; // pieces and elements since the row changed
            // rows that are one thread's in the template's kernel have no more parts than it adds elements
            const TiledSource &from = src[chunks[c].sub];
            const bool alone = !from.a->atomic && (from.templ == ASP_DIRECT_ATOM_TEMPLATE_WARP_BLOCK_COMPRESS || from.templ == ASP_DIRECT_ATOM_TEMPLATE_WARP_COMPRESS);
            auto row_ends = [&]() {
                // (several threads may have elements of a row)
                if (of_row && alone) __atomic_store_n(&row_code[row], 1, __ATOMIC_RELAXED);
                else if (of_row) __atomic_fetch_add(&row_code[row], (u32)std::min<u64>(of_row + elements / warp_steps, 1u << 16) * share[chunks[c].sub], __ATOMIC_RELAXED);
                of_row = elements = 0;
            };
            walk_any<VT>(src[chunks[c].sub], chunks[c].u0, chunks[c].u1, [&](u64 r, u64 col, VT) ASP_INLINE {
                const u64 t = (u32)col / TW;
                const bool begins = n[t]++ == 0;
                if (r != row || t != tile || run == kMaxPiece)
                {
                    all_deep += run >= kDeep ? run : 0;
                    pieces[t]++;
                    if (begins) first[t] = (u32)r;
                    else if (r != last[t])
                    {
                        all_runs++;
                        all_near += near(last[t], r);
                    }
                    last[t] = (u32)r;
                    if (r != row) row_ends();
                    of_row++;
                    row = r;
                    tile = t;
                    run = 0;
                }
                run++;
                elements++;
            });
            row_ends();
            std::copy(n, n + C, at.begin() + (size_t)c * C);
            sum_runs.fetch_add(all_runs, std::memory_order_relaxed);
            sum_near.fetch_add(all_near, std::memory_order_relaxed);
            sum_deep.fetch_add(all_deep + (run >= kDeep ? run : 0), std::memory_order_relaxed);
        });
        for (unsigned who = 0; who < width; who++)
            for (u64 t = 0; t < C; t++) tile_pieces[t] += pieces_of_thread.of(who)[t];
        runs = sum_runs.load(std::memory_order_relaxed);
        near_runs = sum_near.load(std::memory_order_relaxed);
        deep = sum_deep.load(std::memory_order_relaxed);
        tile_begin.assign(C + 1, 0);
        u64 sum = 0;
        for (u64 t = 0; t < C; t++)
        {
            tile_begin[t] = sum;
            u64 before = ~0ull; // row of the chunks before
            for (size_t c = 0; c < chunks.size(); c++)
            {
                const u64 n = at[c * C + t];
                if (n > 0)
                {
                    // (whatever the threads made of it: the choice of the layout is the matrix's)
                    const u32 *const first = edge.data() + c * edges, *const last = first + C;
                    runs += before != first[t] ? 1 : 0;
                    near_runs += before != ~0ull && before != first[t] ? near(before, first[t]) : 0;
                    before = last[t];
                }
                at[c * C + t] = sum;
                sum += n;
            }
        }
        tile_begin[C] = N = sum;
    }

    // which rows y takes itself and which have 64-bit sums
    void choose_sums(TiledHost &out)
    {
        // (a long row's pieces lie side by side in a tile and are summed in the warp before they are added: two parts a tile, as a rule,
        // twice as many where warps cut them)
        const u64 most = (warp_steps < kMaxPiece ? 4 : 2) * C * (kDirectShares / 8);
        std::atomic<u64> all_missing(0), all_direct(0), all_shares(0);
        share_ranges(n_rows, true, [&](u64 r, u64 e) {
            u64 missing = 0, direct = 0, shares = 0;
            for (; r < e; r++)
            {
                if (row_code[r] == 0) missing++;
                else if (row_code[r] <= kDirectShares) direct++;
                else shares += std::min<u64>(row_code[r], most);
            }
            all_missing.fetch_add(missing, std::memory_order_relaxed);
            all_direct.fetch_add(direct, std::memory_order_relaxed);
            all_shares.fetch_add(shares, std::memory_order_relaxed);
        });
        const u64 missing = all_missing.load(std::memory_order_relaxed), direct = all_direct.load(std::memory_order_relaxed), shares = all_shares.load(std::memory_order_relaxed);
        const u64 rows = n_rows - missing - direct;
        out.covers_all_rows = missing == 0;
        // fp64: at most half of what may be added up directly goes to one sum of a row, on average
        // (four at least where warps cut the pieces: the longest of a few long rows count for more than the average)
        if (sizeof(VT) == 8 && rows > 0 && warp_steps < kMaxPiece) out.copies = 4;
        if (sizeof(VT) == 8)
            while (out.copies < 16 && shares > kDirectShares / 2 * (u64)out.copies * rows) out.copies *= 2;
        if (sizeof(VT) == 8 && 2 * deep >= N && out.copies == 1 && N <= kFewWarpsMost) warps = kTiledFewWarps;
        // where some rows have sums, the others do better with sums, too, than with one more launch that clears y, unless they are
        // many: 400,000 rows, fp32: 25 -> 21 us; R-MAT scale 21: 50 -> 56 us (a `red` of 64 bits costs more than one of 32)
        const double sums_us = (double)(n_rows - rows) * ((16.0 * out.copies + sizeof(VT)) / 6.0e6 + 4e-6), clear_us = 4.0 + (double)n_rows * sizeof(VT) / 6.0e6;
        out.n_parts = rows == 0 || sums_us > clear_us ? rows : n_rows;
        out.direct = out.n_parts < n_rows;
        if (out.direct) out.parts.resize(rows);
    }
    void number_rows(TiledHost &out)
    {
        if (out.parts.empty()) return; // all rows are alike
        u32 k = 0;
        for (u64 r = 0; r < n_rows; r++)
        {
            const bool in_parts = row_code[r] > kDirectShares;
            if (in_parts) out.parts[k] = (u32)r;
            row_code[r] = in_parts ? kTiledInParts | k++ : (u32)r;
        }
    }

    void scatter()
    {
        e_row.make(N);
        e_col.make(N);
        e_val.make(N);
        ThreadCounters to_of_thread(C, width);
        share_steps(chunks.size(), 1, width, [&](u64 c, u64, unsigned who) {
            u64 *const to = to_of_thread.of(who);
            std::copy(at.begin() + (size_t)c * C, at.begin() + (size_t)(c + 1) * C, to);
            walk_any<VT>(src[chunks[c].sub], chunks[c].u0, chunks[c].u1, [&](u64 r, u64 col, VT v) ASP_INLINE {
                const u64 t = (u32)col / TW, q = to[t]++;
                e_row.p[q] = (u32)r;
                e_col.p[q] = (uint16_t)(col - t * TW);
                e_val.p[q] = v;
            });
        });
    }

    struct Piece
    {
        u32 start, len; // start: relative to the block
    };
    struct Block
    {
        u64 e0, e1;
        u64 step = 0, slice = 0; // first step and slice of the block
    };

    struct Pieces // of one block, in a thread's own memory
    {
        Piece *p, *sorted;
        size_t n = 0;
        size_t size() const { return n; }
        const Piece &operator[](size_t i) const { return sorted[i]; }
    };
    // in windows, every window by descending length (rows in order where lengths agree)
    void pieces_of(const Block &b, Pieces &out) const
    {
        Piece *const p = out.p;
        size_t n = 0;
        for (u64 k = b.e0; k < b.e1;)
        {
            u64 q = k + 1;
            while (q < b.e1 && q - k < kMaxPiece && e_row.p[q] == e_row.p[k]) q++;
            p[n++] = {(u32)(k - b.e0), (u32)(q - k)};
            k = q;
        }
        out.n = n;
        for (size_t i = 0; i < n; i += kWindow)
        {
            const size_t e = std::min<size_t>(n, i + kWindow);
            u32 cnt[kMaxPiece + 2] = {0};
            for (size_t j = i; j < e; j++) cnt[kMaxPiece - p[j].len + 1]++;
            for (u32 l = 1; l <= kMaxPiece; l++) cnt[l] += cnt[l - 1];
            for (size_t j = i; j < e; j++) out.sorted[i + cnt[kMaxPiece - p[j].len]++] = p[j];
        }
    }

    void slices(int n_sm, TiledHost &out)
    {
        std::vector<Block> blocks;
        const u64 kBlock = block_size(N);
        std::vector<size_t> tile_block(C + 1, 0);
        for (u64 t = 0; t < C; t++)
        {
            tile_block[t] = blocks.size();
            for (u64 b = tile_begin[t]; b < tile_begin[t + 1];)
            {
                u64 e = std::min(b + kBlock, tile_begin[t + 1]);
                // whole rows, as long as that does not make the block much longer
                while (e < tile_begin[t + 1] && e - b < 2 * kBlock && e_row.p[e] == e_row.p[e - 1]) e++;
                blocks.push_back({b, e});
                b = e;
            }
        }
        tile_block[C] = blocks.size();
        const u64 B = blocks.size();
        std::vector<u64> n_step(B), n_slice(B);
        u64 longest = 0;
        for (const Block &b : blocks) longest = std::max(longest, b.e1 - b.e0);
        std::unique_ptr<Piece[]> scratch(new Piece[2 * longest * (u64)width]);
        auto scratch_of = [&](unsigned who) {
            Piece *const mine = scratch.get() + 2 * longest * (u64)who;
            return Pieces{mine, mine + longest};
        };
        share_steps(B, 1, width, [&](u64 b, u64, unsigned who) {
            Pieces p = scratch_of(who);
            pieces_of(blocks[b], p);
            u64 s = 0;
            for (size_t i = 0; i < p.size(); i += kTiledSlice) s += p[i].len;
            n_step[b] = s;
            n_slice[b] = (p.size() + kTiledSlice - 1) / kTiledSlice;
        });
        u64 steps = 0, nsl = 0;
        for (u64 b = 0; b < B; b++)
        {
            blocks[b].step = steps;
            blocks[b].slice = nsl;
            steps += n_step[b];
            nsl += n_slice[b];
        }
        const u64 st = steps + kTiledSlackSteps, sl = nsl + kTiledSlackSlices;
        out.val.make(st * kTiledSlice * sizeof(VT));
        out.col.make(st * kTiledSlice);
        out.row.make(sl * kTiledSlice);
        out.end.make(sl);
        VT *val = (VT *)out.val.p;
        // what stands for a row among the slices' rows
        const bool some = !out.parts.empty();
        const u32 all = out.n_parts > 0 && !out.direct ? kTiledInParts : 0;
        share_steps(B, 1, width, [&](u64 b, u64, unsigned who) {
            Pieces p = scratch_of(who);
            pieces_of(blocks[b], p);
            u64 step = blocks[b].step, slice = blocks[b].slice;
            for (size_t i = 0; i < p.size(); i += kTiledSlice, slice++)
            {
                const u32 depth = p[i].len;
                VT *v = val + step * kTiledSlice;
                uint16_t *c = out.col.p + step * kTiledSlice;
                u32 *rows = out.row.p + slice * kTiledSlice;
                memset(v, 0, (size_t)depth * kTiledSlice * sizeof(VT));
                std::fill(c, c + (size_t)depth * kTiledSlice, (uint16_t)TW);
                for (u32 j = 0; j < kTiledSlice; j++)
                {
                    // piece j goes to lane j % 32, so that one `red` of a warp covers 32 neighbouring pieces
                    const u32 o = (j % 32) * kTiledLanePieces + j / 32;
                    rows[o] = kTiledNoRow;
                    if (i + j >= p.size()) continue;
                    const u64 e = blocks[b].e0 + p[i + j].start;
                    rows[o] = some ? row_code[e_row.p[e]] : e_row.p[e] | all;
                    for (u32 k = 0; k < p[i + j].len; k++)
                    {
                        v[k * kTiledSlice + o] = e_val.p[e + k];
                        c[k * kTiledSlice + o] = e_col.p[e + k];
                    }
                }
                step += depth;
                out.end.p[slice] = (u32)step;
            }
        });
        memset(val + steps * kTiledSlice, 0, kTiledSlackSteps * kTiledSlice * sizeof(VT));
        memset(out.col.p + steps * kTiledSlice, 0, kTiledSlackSteps * kTiledSlice * sizeof(uint16_t));
        memset(out.row.p + nsl * kTiledSlice, 0xff, kTiledSlackSlices * kTiledSlice * sizeof(u32));
        for (u32 i = 0; i < kTiledSlackSlices; i++) out.end.p[nsl + i] = 0xffffffffu;
        out.warps = warps;
        out.nnz = N;
        out.steps = steps;
        out.slices = nsl;
        // work of the CTAs: the steps in order, cut so that every CTA has the same cost: its steps, kSliceCost steps for every
        // slice (its two `red` and the wait for its rows), and what loading its tiles takes; inside a CTA's share of a tile
        // the warps are cut the same way
        std::vector<u64> tile_step(C + 1, steps);
        for (u64 t = C; t-- > 0;) tile_step[t] = tile_block[t] < blocks.size() ? blocks[tile_block[t]].step : steps;
        const u32 *end = out.end.p;
        auto slice_of = [&](u64 step) { return (u64)(std::upper_bound(end, end + nsl, (u32)step) - end); };
        auto cost_of = [&](u64 step) { return (double)step + kSliceCost * (double)slice_of(step); };
        // the step in [lo, hi] that a cost is reached at: the slice, then the step inside it
        auto step_at = [&](double cost, u64 lo, u64 hi) {
            u64 j = 0, j1 = nsl;
            while (j < j1)
            {
                const u64 mid = (j + j1) / 2;
                if ((double)end[mid] + kSliceCost * (double)(mid + 1) >= cost) j1 = mid;
                else j = mid + 1;
            }
            const double in = std::ceil(cost - kSliceCost * (double)j);
            u64 step = in > 0 ? (u64)in : 0;
            if (j < nsl) step = std::min<u64>(step, end[j]);
            return std::min(std::max(step, lo), hi);
        };
        const double tile_cost = (double)kTiledTileBytes / (kTiledSlice * (sizeof(VT) + 2.0));
        share_out(
            n_sm, warps, tile_step, tile_cost, cost_of, step_at, out.work,
            [&](u32 *o, u64 from, u64 to, u64 tile) {
                o[0] = (u32)from;
                o[1] = (u32)to;
                o[2] = (u32)slice_of(from);
                o[3] |= (u32)tile;
            },
            [](u32 *o, u64 next) { o[3] |= (u32)next << 16; });
    }

    // ---- units (fp32)
    static constexpr u32 S = kTiledLane, U = kTiledUnit;

    // as scatter(), with a unit of its own at the beginning of every tile
    void scatter_units(TiledHost &out)
    {
        std::vector<u64> to_unit(C), end(C); // what a tile's places move by, and where its elements end
        u64 moved = 0;
        for (u64 t = 0; t < C; t++)
        {
            to_unit[t] = moved;
            end[t] = tile_begin[t + 1] + moved;
            moved += (U - end[t] % U) % U;
        }
        for (u64 t = 1; t <= C; t++) tile_begin[t] = t < C ? tile_begin[t] + to_unit[t] : tile_begin[C] + moved;
        const u64 places = tile_begin[C];
        e_row.make(places);
        out.val.make(places * sizeof(float));
        out.col.make(places);
        float *const val = (float *)out.val.p;
        uint16_t *const cl = out.col.p;
        ThreadCounters to_of_thread(C, width);
        share_steps(chunks.size(), 1, width, [&](u64 c, u64, unsigned who) {
            u64 *const to = to_of_thread.of(who);
            for (u64 t = 0; t < C; t++) to[t] = at[(size_t)c * C + t] + to_unit[t];
            walk_any<float>(src[chunks[c].sub], chunks[c].u0, chunks[c].u1, [&](u64 r, u64 col, float v) ASP_INLINE {
                const u64 t = (u32)col / TW, q = to[t]++;
                e_row.p[q] = (u32)r;
                cl[q] = (uint16_t)(col - t * TW);
                val[unit_val_at(q)] = v;
            });
        });
        // what fills a tile's last unit belongs to its last row and adds 0 * 0
        for (u64 t = 0; t < C; t++)
            for (u64 q = end[t]; q < tile_begin[t + 1]; q++)
            {
                e_row.p[q] = e_row.p[end[t] - 1];
                cl[q] = (uint16_t)TW;
                val[unit_val_at(q)] = 0;
            }
    }

    void units(int n_sm, TiledHost &out)
    {
        const u64 n = tile_begin[C] / U;
        out.word.make(n * 32);
        out.seg.make(n + kTiledSlackUnits);
        // what stands for a row among the units' rows
        const bool some = !out.parts.empty();
        const u32 all = out.n_parts > 0 && !out.direct ? kTiledInParts : 0;
        for_each(n, true, [&](u64 u) {
            u32 *const row = e_row.p + u * U;
            u32 found = 0, before = 0;
            for (u32 l = 0; l < 32; l++)
            {
                u32 word = found << 16;
                for (u32 k = 0; k < S; k++)
                {
                    const u32 r = row[l * S + k];
                    if (l + k > 0 && r == before) continue;
                    before = r;
                    word |= 1u << k;
                    row[found++] = some ? row_code[r] : r | all; // (never beyond what has been read)
                }
                out.word.p[u * 32 + l] = word;
            }
            out.seg.p[u] = found;
        });
        u64 sum = 0;
        for (u64 u = 0; u < n; u++)
        {
            const u32 found = out.seg.p[u];
            out.seg.p[u] = (u32)sum;
            sum += found;
        }
        for (u32 i = 0; i < kTiledSlackUnits; i++) out.seg.p[n + i] = (u32)sum;
        out.row.make(std::max<u64>(sum, 1));
        for_each(n, true, [&](u64 u) { memcpy(out.row.p + out.seg.p[u], e_row.p + u * U, (out.seg.p[u + 1] - out.seg.p[u]) * sizeof(u32)); });
        out.nnz = N;
        out.units = n;
        // work of the CTAs: the units in order; a unit costs its elements and its rows
        std::vector<u64> begin(C + 1);
        for (u64 t = 0; t <= C; t++) begin[t] = tile_begin[t] / U;
        const u32 *seg = out.seg.p;
        auto cost_of = [&](u64 u) { return (double)(u * U) + kRowCost * (double)seg[u]; };
        auto unit_at = [&](double cost, u64 lo, u64 hi) {
            while (lo < hi)
            {
                const u64 mid = (lo + hi) / 2;
                if (cost_of(mid) >= cost) hi = mid;
                else lo = mid + 1;
            }
            return lo;
        };
        const double tile_cost = 0.5 * (double)kTiledTileBytes / (sizeof(float) + 2.0);
        share_out(
            n_sm, kTiledUnitWarps, begin, tile_cost, cost_of, unit_at, out.work,
            [](u32 *o, u64 from, u64 to, u64 tile) {
                o[0] = (u32)from;
                o[1] = (u32)to;
                o[2] = (u32)tile;
            },
            [](u32 *o, u64 next) { o[3] = (u32)next; });
    }
};

template <class VT>
bool build(const std::vector<TiledSource> &src, u64 n_rows, u64 n_cols, int n_sm, TiledHost &out)
{
    const double sv = sizeof(VT);
    // The group's own kernels: one request to L2 per cache line that a gather touches (290 G/s on this part, of which they reach
    // 0.85) or the format's bytes, or their longest serial chain, whichever is longest. Below some 10 us the rates are not reached
    // (20,000 rows of 80 random columns: 13.8 us for 7 us of requests); several kernels add a fork and a join.
    // The kernels for whole rows (one sub-matrix) reach 0.75 of that rate, and take 8 to 12 us for 60,000 rows of 27 to 81 elements that lie near
    // one another. Random columns, K4: 560 K non-zeros 4.3 us, 900 K 6.2, 1.6 M 9.0 to 9.5, 3.2 M 16.4 to 17.2; the layout in units (fp32) 5.2, 5.5,
    // 6.6, 9.3, in slices (fp64) -, 10.5, 11.2, 14.5.
    const bool whole = src.size() == 1 && src[0].whole_rows;
    u64 true_nnz = 0;
    double chain = 0, requests = 0, bytes_us = 0;
    for (const TiledSource &s : src)
    {
        if (unit_count(s) == 0) return false;
        const double slow = whole ? 1.0 : slowness(s);
        true_nnz += s.true_nnz;
        chain = std::max(chain, chain_us(s));
        requests += (double)s.stored * slow;
        bytes_us += (double)s.stored * slow * (sv + 4) / 6.0e6;
    }
    auto own = [&](double lines) {
        if (whole && is_csr5(src[0])) return 0.0; // (small ones: 2.6 to 5 us)
        if (whole) return std::max(2.9, 1.7 + std::max({lines / (0.75 * 290e3), bytes_us * 6.0 / 4.6, src[0].trips * 0.14e-3 + 0.45 * bytes_us * 6.0 / 4.6}));
        const double rate = std::max(lines / (0.85 * 290e3), bytes_us);
        return (src.size() > 1 ? 8.0 : 0.0) + std::max(2.0 + chain, 3.0 + rate + std::min(0.4 * rate, 4.5));
    };
    // (the layout would be faster: three strips, 33,000 non-zeros: 22 us; 73,000: 24 against 6 us)
    if (src.size() > 1 && true_nnz < kSameBits) return false;
    // small matrices, whose time is the launch, stay with their kernels (not worth a look at the columns)
    if (own(requests) < (whole ? 5.0 : 7.0)) return false;
    double lines = 0;
    for (const TiledSource &s : src) lines += lines_per_gather(s, sizeof(VT) == 8) * (double)s.stored * (whole ? 1.0 : slowness(s));
    // of an x of one tile L1 holds most
    const bool short_x = whole && sizeof(VT) == 4 && n_cols <= tiled_tile_cols(false) && true_nnz <= 160 * n_rows;
    if (short_x) lines *= 0.75;
    const double own_us = own(lines);
    // This layout: launches and tail, the first tile of x, 2 + sv bytes per element at 4.6 TB/s, a `red` per piece (below), y
    // cleared, the sums of the rows in many parts.
    auto tiled_us = [&](u64 n, u64 pieces, double red) {
        return 4.5 + 2.5 * std::min(1.0, (double)n_cols / (double)tiled_tile_cols(sizeof(VT) == 8)) + (double)n * (sv + 2) / 4.6e6 + (double)pieces * 4 / 4.6e6 + red / 200e3 +
               ((double)n_rows * sv + (double)out.n_parts * 16.0 * out.copies) / 6.0e6 + (out.n_parts > 0 && out.direct ? 4.0 : 0.0);
    };
    // (what tiled_us says is 1 to 3 us too long for a few million non-zeros, as the time of the other kernels is; that of whole rows is not. fp32, one tile,
    // random rows of 80: 0.8 M 6.3 said, 7.0 taken, by whole rows 4.1; 1.6 M 8.0, 7.8, 6.5; 2 M of three unknowns a node 8.9, 7.9, 6.2)
    const double too_long = short_x ? 1.6 * std::min(1.0, (double)true_nnz / 4e6) : 1.6;
    auto slower = [&](double us) { return whole ? 0.92 * (us - too_long) > own_us : us > 0.85 * own_us; };
    // Pieces of a long dense row are 32 columns apart: the lanes that take them meet in one bank of shared memory. Rows of 81 / 500 / 2000 adjacent
    // columns, fp32, 4 M 10.1 / 13.9 / 18.0 us, 8 M 13.9 / 21.4 / 31.7 (by whole rows 19.3 / - / 12.0), fp64 8 M 17.8 / 29.6 / 35.0.
    const double close = whole && !is_csr5(src[0]) && !slower(tiled_us(true_nnz, 0, 0)) ? closeness<VT>(src[0]) : 0.0;
    auto banks_us = [&](u64 n, double run) { return (double)n * 1.95e-6 * close * std::min(1.0, std::max(0.0, run - 96.0) / 1024.0); };
    auto units_us = [](u64 n) { return 4.4 + 1.45e-6 * (double)n; };
    if (slower(tiled_us(true_nnz, 0, 0) + banks_us(true_nnz, (double)true_nnz / (double)n_rows)) && !(sizeof(VT) == 4 && whole && units_us(true_nnz) <= own_us)) return false;
    if (n_rows >= kTiledInParts || requests >= 1e11) return false;
    Builder<VT> b(src, n_rows, n_cols, true_nnz, n_sm);
    if (b.C + (u64)n_sm >= 65536) return false;
    b.count();
    b.choose_sums(out);
    // (a warp's 32 `red` fall into about an eighth as many lines where the rows of a tile are dense, into 32 where they are sparse)
    double red = 0;
    u64 pieces = 0;
    for (u64 t = 0; t < b.C; t++)
    {
        const double p = (double)b.tile_pieces[t];
        pieces += b.tile_pieces[t];
        if (p > 0) red += p * std::min(1.0, std::max(0.25, 4.0 * (double)n_rows / p / 32.0));
    }
    const bool units = sizeof(VT) == 4 && b.N <= kRunForUnits * b.runs && 4 * b.near_runs >= 3 * b.runs && tiled_units_fit(b.runs, b.N, b.C);
    if (whole && units ? units_us(b.N) > own_us : slower(tiled_us(b.N, pieces, red) + banks_us(b.N, (double)b.N / (double)std::max<u64>(1, b.runs)))) return false;
    b.number_rows(out);
    if constexpr (sizeof(VT) == 4)
    {
        if (units)
        {
            b.scatter_units(out);
            b.units(n_sm, out);
            return true;
        }
    }
    b.scatter();
    b.slices(n_sm, out);
    return true;
}
} // namespace

bool tiled_build(const std::vector<TiledSource> &src, bool f64, uint64_t n_rows, uint64_t n_cols, int n_sm, TiledHost &out)
{
    if (src.empty() || n_sm <= 0) return false;
    return f64 ? build<double>(src, n_rows, n_cols, n_sm, out) : build<float>(src, n_rows, n_cols, n_sm, out);
}
} // namespace asp

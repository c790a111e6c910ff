// Which plans have a list of their rows, and the lists: one pass over the arrays of a plan that say where rows begin and which they are.
#include "../row_lists.h"

#include <algorithm>
#include <atomic>
#include <memory>
#include <new>

#include "crew.hpp"

namespace asp
{
namespace
{
// f(entry of a place): of an array by its type, looked at once
template <class F>
void with_entries(const HostMeta &h, F &&f)
{
    if (h.kind != ASP_COMPRESS_NONE) f([&h](uint64_t i) { return h.get(i); });
    else if (h.dtype == ASP_U8) f([p = (const uint8_t *)h.p](uint64_t i) { return (uint64_t)p[i]; });
    else if (h.dtype == ASP_U16) f([p = (const uint16_t *)h.p](uint64_t i) { return (uint64_t)p[i]; });
    else if (h.dtype == ASP_U32) f([p = (const uint32_t *)h.p](uint64_t i) { return (uint64_t)p[i]; });
    else f([p = (const uint64_t *)h.p](uint64_t i) { return (uint64_t)p[i]; });
}
// Whether rows of y come once each: ascending ones, or a list of what has come (of more than kMostSeen rows: none does)
struct Distinct
{
    const uint64_t n;
    const bool ascending;
    uint64_t next = 0;
    std::vector<bool> seen;
    Distinct(uint64_t rows, bool in_order) : n(in_order || rows <= kMostSeen ? rows : 0), ascending(in_order), seen(in_order ? 0 : n, false) {}
    bool operator()(uint64_t row)
    {
        if (row >= n || (ascending ? row < next : (bool)seen[row])) return false;
        if (ascending) next = row + 1;
        else seen[row] = true;
        return true;
    }
};
uint64_t row_in_y(const asp_plan_desc &d, const HostMeta &perm, int sort_kind, uint64_t r)
{
    return sort_kind == ASP_SORT_GLOBAL ? perm.get(r + d.first_row) : sort_kind == ASP_SORT_LOCAL ? perm.get(r) + d.first_row : r + d.first_row;
}
const uint64_t kMostStrips = 3u << 20, kMostRuns = 1u << 19, kMostTlbs = 2u << 20, kShortTlb = 8; // elements of a plan, of a TLB: row_lists.h
// Row-grouped plans of more elements have no list where rows of some 12 to 64 elements (in fp32, from 1 M on, of 160) lie in columns near one another: their strips
// stream faster than few lanes a row. By strips / by rows, us, rows of 30 in adjacent columns: 0.3 M 3.1 / 2.9, 0.8 M 3.2 / 4.5, 1.6 M 3.9 / 8.0 (fp64 5.8 /
// 8.9), of 80 0.8 M 4.5 / 3.9, 1.2 M 4.1 / 5.1, 1.6 M 5.0 / 6.3 (fp64 8.6 / 7.4); in random ones of 20,000 0.8 M 5.6 / 4.9; rows of 8 in adjacent ones 1.6 M 7.6 / 4.4, of 300
// 12.4 / 4.4.
const uint64_t kMostNear = 5u << 17;
const uint64_t kMostRun = 4096; // elements of a row of the CSR5-like templates that is listed
// Elements of a plan whose rows are listed: as many as both kernels were measured with. By chunks / by rows, us. Chunks of a warp are the slower ones at
// every size: rows of 81, columns in a window of 3000, fp32 1 M 10.1 / 4.7, 16 M 101 / 48.2, 100 M 607 / 287, fp64 10.3 / 6.4, 107 / 70.2, 650 / 425; rows of
// 300, 16 M, 69.5 / 24.7, fp64 68.8 / 36.6. So are chunks of a CTA in fp32, for rows of up to 4096 (rows of 2000 1 M 5.8 / 3.1, 100 M 133 / 121; of
// 600 100 M 239 / 174); for longer ones up to some 16 M (of 8,000 25.3 / 24.9, 32 M 44.7 / 47.1). In fp64 the operations of the sums show: rows of 2000 4 M
// 12.5 / 11.1, 8 M 20.1 / 20.7, 16 M 33.3 / 38.0; of 8,000 1 M 5.5 / 4.1, 2 M 7.3 / 7.4, 4 M 11.7 / 15.6.
const uint64_t kMostByRows = 1u << 27, kMost64 = 1u << 22, kMostLong = 1u << 24, kMostLong64 = 1u << 20;
const uint64_t kSharedRows = 1u << 14; // from so many on, the rows of a list are shared out

// Lists of the rows of a (validated) plan, as the kernels of kernels_rows.cu take them. false: another template, a row in two places, or offsets
// beyond 32 bits.
//
// Chunks of a row one after the other, `longest` row; no more rows than elements (`stored`)
bool list_rows(const asp_plan_desc &d, const std::vector<HostMeta> &hm, const HostMeta &perm, const KArgs &a, uint64_t stored, HostBuf<uint2> &out, uint64_t &longest)
{
    const bool cta = d.template_type == ASP_SHARED_MEMORY_LONG_ROW_TEMPLATE, chunks = cta || d.template_type == ASP_DIRECT_ATOM_TOTAL_WARP_REDUCE_TEMPLATE;
    if ((!chunks && d.template_type != ASP_SHARED_MEMORY_TOTAL_WARP_REDUCE_TEMPLATE) || d.n_rows > 0xffffffffull) return false;
    const HostMeta &offsets = hm[cta ? MS_BLK_NZ : MS_WARP_NZ];
    const uint64_t most = std::min<uint64_t>(d.n_rows, cta ? a.n_units : chunks ? a.effective : std::min<uint64_t>(hm[MS_BLK_ROW].get(a.n_units), a.effective));
    if (most > stored) return false;
    Distinct distinct(d.n_rows, d.sort_kind == ASP_SORT_NONE);
    out.make(most + 1);
    uint64_t end = 0, n = 0;
    longest = 0;
    auto put = [&](uint64_t row, uint64_t from, uint64_t to) {
        if (to < from || to > 0xffffffffull || (n > 0 && from != end) || n == most || !distinct(row)) return false;
        end = to;
        longest = std::max(longest, to - from);
        out.p[n++] = make_uint2((unsigned)from, (unsigned)row);
        return true;
    };
    bool good = true;
    if (chunks)
        with_entries(hm[MS_ROW_OF_UNIT], [&](auto of) {
            with_entries(offsets, [&](auto nz) {
                const uint64_t units = cta ? a.n_units : a.effective, radd = a.row_add ? d.first_row : 0;
                for (uint64_t u = 0; u < units && good;)
                {
                    uint64_t e = u + 1;
                    const uint64_t row = of(u);
                    while (e < units && of(e) == row) e++;
                    good = put(row + radd, nz(u), nz(e));
                    u = e;
                }
            });
        });
    else
    {
        const HostMeta &row = hm[MS_BLK_ROW], &warp = hm[MS_BLK_WARP];
        const uint64_t B = a.n_units, rows = std::min<uint64_t>(row.get(B), a.effective), warps = warp.get(B);
        if (!has_entries(offsets, warps + 1) || !has_entries(hm[MS_ROW_OFF], row.get(B) + 1)) return false;
        with_entries(hm[MS_ROW_OFF], [&](auto off) {
            with_entries(offsets, [&](auto nz) {
                for (uint64_t b = 0; b < B && good; b++)
                {
                    const uint64_t r0 = row.get(b), r1 = std::min(row.get(b + 1), rows), w0 = warp.get(b), g0 = off(r0);
                    for (uint64_t r = r0; r < r1 && good; r++)
                    {
                        const uint64_t lo = w0 + off(r) - g0, hi = w0 + off(r + 1) - g0;
                        good = lo <= warps && hi <= warps && put(row_in_y(d, perm, a.sort_kind, r), nz(lo), nz(hi));
                    }
                }
            });
        });
    }
    if (!good || n == 0) return false;
    out.p[n] = make_uint2((unsigned)end, 0);
    out.n = n + 1;
    return true;
}

// Row-grouped; `tlbs` of all rows, `most` of one
bool list_tlb_rows(const asp_plan_desc &d, const std::vector<HostMeta> &hm, const HostMeta &perm, const KArgs &a, uint64_t stored, HostBuf<uint4> &out, uint64_t &tlbs, uint64_t &most)
{
    if (d.template_type != ASP_SHARED_MEMORY_TEMPLATE_WARP_COMPRESS || d.n_rows > 0xffffffffull) return false;
    const HostMeta &row = hm[MS_BLK_ROW];
    const uint64_t B = a.n_units, rows = std::min<uint64_t>(row.get(B), a.effective);
    if (row.get(0) != 0 || rows == 0 || rows > d.n_rows || rows > stored || !has_entries(hm[MS_ROW_OFF], row.get(B) + 1)) return false;
    Distinct distinct(d.n_rows, a.sort_kind == ASP_SORT_NONE);
    out.make(rows);
    std::atomic<uint64_t> all(0), top(0);
    std::atomic<bool> good(true);
    with_entries(hm[MS_ROW_OFF], [&](auto off) {
        host::share_ranges(B, a.sort_kind == ASP_SORT_NONE && rows >= kSharedRows, [&](uint64_t b, uint64_t e) {
            uint64_t sum = 0, longest = 0;
            bool in = true;
            for (; b < e && in; b++)
            {
                const uint64_t nz = hm[MS_BLK_NZ].get(b), n = hm[MS_BLK_THR].get(b + 1) - hm[MS_BLK_THR].get(b), S = hm[MS_TLB_SIZE].get(b);
                const uint64_t r0 = row.get(b), r1 = std::min(row.get(b + 1), rows), g0 = off(r0);
                in = S > 0 && S <= 0xffff && nz + n * S <= 0xffffffffull;
                for (uint64_t r = r0; r < r1 && in; r++)
                {
                    const uint64_t lo = off(r) - g0, hi = off(r + 1) - g0, y = row_in_y(d, perm, a.sort_kind, r);
                    // (unsorted rows ascend with r, and the BLBs' rows follow one another)
                    in = lo <= hi && hi <= n && hi - lo <= 0xffff && y < d.n_rows && (a.sort_kind == ASP_SORT_NONE || distinct(y));
                    sum += hi - lo;
                    longest = std::max(longest, hi - lo);
                    out.p[r] = make_uint4((unsigned)(nz + lo), (unsigned)y, (unsigned)((hi - lo) | S << 16), (unsigned)n);
                }
                in = in && row.get(b + 1) >= r0;
            }
            all.fetch_add(sum);
            host::raise<uint64_t>(top, longest);
            if (!in) good = false;
        });
    });
    tlbs = all;
    most = top;
    return good;
}

// How near the elements of a (validated) row-grouped plan's TLBs lie, 1: in adjacent columns. Sampled: a TLB each of up to 256 BLBs.
double nearness(const asp_plan_desc &d, const std::vector<HostMeta> &hm, const KArgs &a)
{
    const asp_array_desc *cols = nullptr;
    for (int k = 0; k < d.n_arrays; k++)
        if (d.arrays[k].role == ASP_ARR_COL_INDEX) cols = &d.arrays[k];
    HostMeta col;
    col.p = cols->host_ptr;
    col.dtype = cols->dtype;
    const uint64_t samples = std::min<uint64_t>(a.n_units, 256);
    uint64_t pairs = 0, columns = 0;
    for (uint64_t q = 0; q < samples; q++)
    {
        const uint64_t b = a.n_units * q / samples, nz = hm[MS_BLK_NZ].get(b), n = hm[MS_BLK_THR].get(b + 1) - hm[MS_BLK_THR].get(b), S = hm[MS_TLB_SIZE].get(b);
        for (uint64_t k = 0; n > 0 && k + 1 < S; k++)
        {
            const uint64_t c0 = col.get(nz + k * n), c1 = col.get(nz + (k + 1) * n);
            if (c0 == c1) continue; // (what fills a TLB)
            pairs++;
            columns += c1 > c0 ? c1 - c0 : c0 - c1;
        }
    }
    return columns == 0 ? 0.0 : (double)pairs / (double)columns;
}

// ELL- and SELL-like; `place` stays empty where TLB t is row first + t. `longest` TLB, `rows` that are stored.
bool list_strips(const asp_plan_desc &d, const std::vector<HostMeta> &hm, const KArgs &a, HostBuf<uint4> &out, HostBuf<unsigned> &place, uint64_t &first, uint64_t &longest, uint64_t &rows)
{
    const bool ell = d.template_type == ASP_DIRECT_ATOM_TEMPLATE_WARP_BLOCK_COMPRESS;
    if ((!ell && d.template_type != ASP_DIRECT_ATOM_TEMPLATE_WARP_COMPRESS) || d.n_rows > 0xffffffffull) return false;
    const HostMeta &of = hm[MS_ROW_OF_TLB];
    const uint64_t radd = a.row_add ? d.first_row : 0, B = ell ? 1 : a.n_units;
    const bool numbered = of.kind == ASP_COMPRESS_LINEAR && of.coef == 1;
    longest = rows = 0;
    first = numbered ? of.icpt + radd : 0;
    out.make(std::min<uint64_t>(a.effective, ell ? a.n_tlb : hm[MS_BLK_THR].get(B)) / 32 + B + 1);
    uint64_t k = 0;
    for (uint64_t b = 0; b < B; b++)
    {
        const uint64_t nz = ell ? 0 : hm[MS_BLK_NZ].get(b), t0 = ell ? 0 : hm[MS_BLK_THR].get(b);
        const uint64_t n = ell ? a.n_tlb : hm[MS_BLK_THR].get(b + 1) - t0, S = ell ? a.tlb_size : hm[MS_TLB_SIZE].get(b);
        if (S == 0 || S > 0xffff || nz + n * S > 0xffffffffull || (t0 != rows && t0 < a.effective)) return false;
        longest = std::max(longest, S);
        for (uint64_t t = t0; t < t0 + n && t < a.effective; t += 32)
        {
            const uint64_t m = std::min<uint64_t>({32, t0 + n - t, a.effective - t});
            out.p[k++] = make_uint4((unsigned)(nz + t - t0), (unsigned)t, (unsigned)(S | m << 16), (unsigned)n);
            rows += m;
        }
    }
    out.n = k;
    if (k == 0) return false;
    if (numbered) return first + rows <= d.n_rows;
    if (!has_entries(of, rows)) return false;
    Distinct distinct(d.n_rows, false);
    place.make(rows);
    bool good = true;
    with_entries(of, [&](auto row) {
        for (uint64_t i = 0; i < rows && good; i++)
        {
            good = distinct(row(i) + radd);
            place.p[i] = (unsigned)(row(i) + radd);
        }
    });
    return good;
}

// CSR5-like: {first element, row, elements, 0}
bool list_runs(const asp_plan_desc &d, const std::vector<HostMeta> &hm, const HostMeta &perm, const KArgs &a, HostBuf<uint4> &out)
{
    const uint64_t S = a.tlb_size, rmask = (1ull << a.bits_row) - 1;
    if ((d.template_type != ASP_UNALIGNED_WARP_REDUCE_SAME_TLB_SIZE_TEMPLATE && d.template_type != ASP_UNALIGNED_WARP_REDUCE_SAME_TLB_SIZE_TEMPLATE_WITH_WARP_REDUCE) ||
        d.n_rows > 0xffffffffull || S == 0 || S >= 64)
        return false;
    // (a row that is too long is seen by the warps that begin in it)
    const uint64_t within = kMostRun / (32 * S) + 1;
    for (uint64_t w = 0; w + within < a.n_units; w++)
        if (hm[MS_ROW_OF_UNIT].get(w) == hm[MS_ROW_OF_UNIT].get(w + within)) return false;
    Distinct distinct(d.n_rows, a.sort_kind == ASP_SORT_NONE);
    out.make(std::min<uint64_t>(d.n_rows, a.n_units * 32 * S));
    uint64_t r = ~0ull, n = 0; // of the matrix's rows in order
    bool good = true;
    with_entries(hm[MS_COMBINE], [&](auto words) {
        for (uint64_t w = 0; w < a.n_units && good; w++)
        {
            const uint64_t R0 = hm[MS_ROW_OF_UNIT].get(w);
            good = (words(w * 32) >> (a.bits_word - 1)) & 1ull; // (a warp's first element always starts a row)
            for (uint64_t l = 0; l < 32 && good; l++)
            {
                const uint64_t word = words(w * 32 + l), e0 = (w * 32 + l) * S;
                uint64_t next = R0 + (word & rmask);
                // the flags, first element first, at the top of the word
                for (uint64_t f = word >> (a.bits_word - (int)S) << (64 - S); f != 0 && good; f &= ~(1ull << (63 - __builtin_clzll(f))), next++)
                {
                    if (next == r) continue; // goes on from the warp before
                    r = next;
                    const uint64_t e = e0 + (uint64_t)__builtin_clzll(f), row = row_in_y(d, perm, a.sort_kind, r);
                    good = distinct(row);
                    if (!good) break;
                    if (n > 0) out.p[n - 1].z = (unsigned)(e - out.p[n - 1].x);
                    out.p[n++] = make_uint4((unsigned)e, (unsigned)row, 0, 0);
                }
            }
        }
    });
    if (!good || n == 0) return false;
    out.p[n - 1].z = (unsigned)(a.n_units * 32 * S - out.p[n - 1].x);
    out.n = n;
    return true;
}
} // namespace

void OwnRows::make(const asp_plan_desc &d, const std::vector<HostMeta> &hm, const HostMeta &perm, const KArgs &a, uint64_t stored, int sm_count, bool few)
{
    try
    {
        if (!list(d, hm, perm, a, stored, sm_count, few)) none();
    }
    catch (const std::bad_alloc &) // (not enough host memory: the template's own kernel)
    {
        none();
    }
}

size_t OwnRows::room(const asp_plan_desc &d, const std::vector<HostMeta> &hm, uint64_t stored)
{
    const uint64_t rows = std::min<uint64_t>(d.n_rows, stored);
    switch (d.template_type)
    {
    case ASP_DIRECT_ATOM_TEMPLATE_WARP_BLOCK_COMPRESS:
    case ASP_DIRECT_ATOM_TEMPLATE_WARP_COMPRESS:
    {
        // a group of up to 32 rows an entry, BLBs of 128 rows
        const HostMeta &of = hm[MS_ROW_OF_TLB];
        const bool one = d.template_type == ASP_DIRECT_ATOM_TEMPLATE_WARP_BLOCK_COMPRESS;
        if (stored > kMostStrips || (one && d.tlb_size <= kShortTlb)) return 0;
        return rows / 2 + (one ? 0 : rows / 8) + (of.kind == ASP_COMPRESS_LINEAR && of.coef == 1 ? 0 : 4 * rows) + 512;
    }
    case ASP_UNALIGNED_WARP_REDUCE_SAME_TLB_SIZE_TEMPLATE:
    case ASP_UNALIGNED_WARP_REDUCE_SAME_TLB_SIZE_TEMPLATE_WITH_WARP_REDUCE: return stored > kMostRuns ? 0 : 16 * rows + 256;
    case ASP_SHARED_MEMORY_TEMPLATE_WARP_COMPRESS: return stored > kMostTlbs ? 0 : 16 * rows + 256;
    case ASP_DIRECT_ATOM_TOTAL_WARP_REDUCE_TEMPLATE:
    case ASP_SHARED_MEMORY_LONG_ROW_TEMPLATE:
    case ASP_SHARED_MEMORY_TOTAL_WARP_REDUCE_TEMPLATE: return stored > kMostStrips ? 0 : 8 * rows + 264; // (a block of its own is little beside a larger plan)
    default: return 0;
    }
}

bool OwnRows::list(const asp_plan_desc &d, const std::vector<HostMeta> &hm, const HostMeta &perm, const KArgs &a, uint64_t stored, int sm_count, bool few)
{
    uint64_t longest = 0, all = 0;
    switch (d.template_type)
    {
    case ASP_DIRECT_ATOM_TEMPLATE_WARP_BLOCK_COMPRESS:
    case ASP_DIRECT_ATOM_TEMPLATE_WARP_COMPRESS:
        strips = true;
        if (stored > kMostStrips || !list_strips(d, hm, a, tlbs, place, all, longest, listed)) return false;
        args.first_row = (unsigned)all;
        args.lanes = longest <= 16 ? 4 : longest <= 32 ? 8 : 16;
        args.n = (unsigned)tlbs.n;
        return longest > kShortTlb || few;
    case ASP_UNALIGNED_WARP_REDUCE_SAME_TLB_SIZE_TEMPLATE:
    case ASP_UNALIGNED_WARP_REDUCE_SAME_TLB_SIZE_TEMPLATE_WITH_WARP_REDUCE:
    {
        runs = true;
        if (stored > kMostRuns || !list_runs(d, hm, perm, a, tlbs)) return false;
        listed = tlbs.n;
        args.size = a.tlb_size;
        args.n = (unsigned)listed;
        args.lanes = stored <= 6 * listed ? 4 : stored <= 12 * listed ? 8 : 16;
        for (uint64_t i = 0; i < listed; i++) longest = std::max<uint64_t>(longest, tlbs.p[i].z);
        if (longest > kMostRun) return false;
        // rows that take its lanes more than two trips are a CTA's
        uint4 *const first = std::stable_partition(tlbs.p, tlbs.p + listed, [&](const uint4 &r) { return r.z > 8 * args.lanes; });
        args.hubs = (unsigned)(first - tlbs.p);
        return true;
    }
    case ASP_SHARED_MEMORY_TEMPLATE_WARP_COMPRESS:
        if (stored > kMostTlbs || !list_tlb_rows(d, hm, perm, a, stored, tlbs, all, longest)) return false;
        listed = tlbs.n;
        if (stored > kMostNear && stored >= 12 * listed && (stored <= 64 * listed || (d.val_dtype == ASP_F32 && 2 * stored > 3 * kMostNear && stored <= 160 * listed)) &&
            nearness(d, hm, a) >= 1.0 / 16)
            return false;
        args.n = (unsigned)listed;
        args.lanes = 2;
        while (args.lanes < 32 && args.lanes * listed < all) args.lanes *= 2;
        return longest <= 8 * args.lanes;
    default: break;
    }
    const bool f64 = d.val_dtype == ASP_F64;
    if (stored > kMostByRows || !list_rows(d, hm, perm, a, stored, rows, longest)) return false;
    listed = rows.n - 1;
    const uint64_t elements = rows.p[listed].x - rows.p[0].x, most = longest > 4096 ? (f64 ? kMostLong64 : kMostLong) : f64 ? kMost64 : kMostByRows;
    if (longest > 512 && (longest > 16384 || elements < 256 * listed || (d.template_type == ASP_SHARED_MEMORY_LONG_ROW_TEMPLATE && stored > most))) return false;
    // threads for all of a row in one trip while all rows are on the device at once, else for two
    const uint64_t per = listed <= 2ull * sm_count ? 4 : 8;
    args.cta = longest <= 512 ? 0 : (unsigned)std::min<uint64_t>(1024, std::max<uint64_t>(64, (longest + 32 * per - 1) / (32 * per) * 32));
    args.n = (unsigned)listed;
    for (uint64_t i = 0; i < listed && args.cta == 0; i++) trips += (rows.p[i + 1].x - rows.p[i].x + 127) / 128;
    return true;
}
} // namespace asp

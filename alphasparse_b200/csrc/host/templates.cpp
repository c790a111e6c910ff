// init_<template> + try_all_compress for the ten reduce templates: flatten a tiled sub-matrix into
// the arrays a kernel family reads, apply the row permutation where the reference applies it on
// the host, re-interleave values / column indices, detect closed forms. Array contents, element
// types and closed forms equal the reference's (the ten *_op*.cc files and arr_optimization.cc).
#include <string.h>

#include <algorithm>

#include "format.hpp"


namespace asp
{
namespace host
{

// ---------------------------------------------------------------------------------------------
// closed forms (arr_optimization.cc)
// ---------------------------------------------------------------------------------------------
namespace
{
// f(i) for all i < n; long arrays on all cores once the first entries hold
template <class F>
bool all_of(u64 n, F &&f)
{
    const u64 head = std::min<u64>(n, 1u << 16);
    for (u64 i = 0; i < head; i++)
        if (!f(i)) return false;
    std::atomic<bool> ok(true);
    share_ranges(n - head, n > kParallelRows, [&](u64 i, u64 e) {
        for (i += head, e += head; i < e && f(i);) i++;
        if (i < e) ok.store(false, std::memory_order_relaxed);
    });
    return ok.load(std::memory_order_relaxed);
}
u64 max_entry(U64s a)
{
    std::atomic<u64> all(0);
    share_ranges(a.n, a.n > kParallelRows, [&](u64 i, u64 e) {
        u64 mx = 0;
        for (; i < e; i++) mx = std::max(mx, a[i]);
        raise(all, mx);
    });
    return all.load(std::memory_order_relaxed);
}
} // namespace

bool detect_linear(U64s a, ClosedForm &out)
{
    if (a.size() <= 1) return false;
    if (a[1] < a[0]) return false;
    const u64 coef = a[1] - a[0];
    if (!all_of(a.size() - 1, [&](u64 i) { return a[i + 1] >= a[i] && a[i + 1] - a[i] == coef; })) return false;
    out = ClosedForm();
    out.kind = ASP_COMPRESS_LINEAR;
    out.coef = coef;
    out.icpt = a[0];
    return true;
}

bool detect_constant(U64s a, ClosedForm &out)
{
    if (a.empty()) return false;
    if (!all_of(a.size(), [&](u64 i) { return a[i] == a[0]; })) return false;
    out = ClosedForm();
    out.kind = ASP_COMPRESS_CONSTANT;
    out.icpt = a[0];
    return true;
}

bool detect_branch(U64s a, ClosedForm &out)
{
    // the reference asserts arr_size > 2 here (arr_optimization.cc:117) and aborts on shorter arrays;
    // shorter arrays simply stay uncompressed
    if (a.size() <= 2) return false;
    ClosedForm f;
    f.kind = ASP_COMPRESS_BRANCH;
    f.lo.push_back(0);
    f.val.push_back(a[0]);
    for (size_t i = 0; i < a.size(); i++)
    {
        if (a[i] != f.val.back())
        {
            f.hi.push_back(i - 1);
            f.lo.push_back(i);
            f.val.push_back(a[i]);
            if (f.hi.size() >= ASP_MAX_BRANCH) return false;
        }
    }
    f.hi.push_back(a.size() - 1);
    out = f;
    return true;
}

bool detect_cycle_linear(U64s a, u64 cycle, ClosedForm &out)
{
    if (!(cycle < a.size()) || a.size() % cycle != 0 || cycle <= 1) return false;
    const u64 icpt = a[0], coef = a[1] - a[0];
    for (size_t i = 0; i < a.size(); i++)
    {
        const u64 k = i % cycle;
        if (k == 0) continue;
        // the reference asserts divisibility inside this check (arr_optimization.cc:271); a
        // mismatch is a plain "no" here
        if (a[i] < icpt || (a[i] - icpt) % k != 0 || (a[i] - icpt) / k != coef) return false;
    }
    out = ClosedForm();
    out.kind = ASP_COMPRESS_CYCLE_LINEAR;
    out.cycle = cycle;
    out.coef = coef;
    out.icpt = icpt;
    return true;
}

bool detect_cycle_increase(U64s a, ClosedForm &out)
{
    if (a.size() <= 2) return false;
    u64 cycle = 0;
    for (size_t i = 0; i < a.size(); i++)
        if (a[i] != a[0])
        {
            if (a[i] < a[0]) return false;
            cycle = i;
            break;
        }
    if (cycle == 0) return false; // all equal: the reference asserts here
    if (a.size() % cycle != 0) return false;
    if (!all_of(a.size(), [&](u64 i) { return a[i] == a[0] + i / cycle; })) return false;
    out = ClosedForm();
    out.kind = ASP_COMPRESS_CYCLE_INCREASE;
    out.cycle = cycle;
    out.icpt = a[0];
    return true;
}

namespace
{
template <class T>
Arr<uint8_t> narrow_to(U64s v)
{
    Arr<uint8_t> out;
    T *p = (T *)out.make(v.size() * sizeof(T));
    for_each(v.n, v.n > kParallelRows, [=](u64 i) { p[i] = (T)v[i]; });
    return out;
}
Arr<uint8_t> narrow(U64s v, int dt)
{
    switch (dtype_bytes(dt))
    {
    case 1: return narrow_to<uint8_t>(v);
    case 2: return narrow_to<uint16_t>(v);
    case 4: return narrow_to<uint32_t>(v);
    default: return narrow_to<u64>(v);
    }
}

TemplateArray &add_meta(TemplateData &t, int role, U64s v, int dt)
{
    t.arrays.emplace_back();
    TemplateArray &a = t.arrays.back();
    a.role = role;
    a.dt = dt;
    a.len = v.size();
    a.bytes = narrow(v, dt);
    return a;
}

// dst[k*n + i] = src[i*S + k] for one strip of n TLBs of size S (row-major -> TLB-interleaved)
template <class D, class S_>
void interleave_strip(D *dst, const S_ *src, u64 n, u64 S)
{
    const u64 TB = 256;
    for_each((n + TB - 1) / TB, n * S > kParallelNnz, [=](u64 b) {
        const u64 i0 = b * TB, i1 = std::min(n, i0 + TB);
        for (u64 k = 0; k < S; k++)
            for (u64 i = i0; i < i1; i++) dst[k * n + i] = (D)src[i * S + k];
    });
}

void interleave_cols(uint8_t *dst, int col_dt, const u32 *src, u64 n, u64 S)
{
    switch (col_dt)
    {
    case ASP_U8: interleave_strip((uint8_t *)dst, src, n, S); break;
    case ASP_U16: interleave_strip((uint16_t *)dst, src, n, S); break;
    case ASP_U32: interleave_strip((uint32_t *)dst, src, n, S); break;
    default: interleave_strip((uint64_t *)dst, src, n, S); break;
    }
}
void interleave_vals(uint8_t *dst, int es, const uint8_t *src, u64 n, u64 S)
{
    if (es == 4) interleave_strip((uint32_t *)dst, (const uint32_t *)src, n, S);
    else interleave_strip((uint64_t *)dst, (const uint64_t *)src, n, S);
}

void add_nnz_arrays(TemplateData &t, const CompressedBlock &b, Arr<uint8_t> &col, Arr<uint8_t> &val, u64 n)
{
    t.arrays.emplace_back();
    TemplateArray &v = t.arrays.back();
    v.role = ASP_ARR_VAL;
    v.dt = t.val_dt;
    v.len = n;
    v.bytes.swap(val);
    t.arrays.emplace_back();
    TemplateArray &c = t.arrays.back();
    c.role = ASP_ARR_COL_INDEX;
    c.dt = b.col_dt;
    c.len = n;
    c.bytes.swap(col);
}

// global row (relative to the sub-matrix) of every TLB, in TLB order
Arr<u64> tlb_global_rows(const CompressedBlock &b, bool &adjacent_equal)
{
    const Level &B = b.blb, &W = b.wlb, &T = b.tlb;
    Arr<u64> out;
    u64 *rows = out.make(T.block_num);
    auto of_wlb = [&](u64 i, u64 w, bool share) {
        const u64 base = B.first_row.v[i] + W.first_row.v[w], t0 = W.index.v[w], t1 = W.index.v[w + 1];
        for_each(t1 - t0, share && t1 - t0 > kParallelRows, [&](u64 t) { rows[t0 + t] = base + b.tlb_row[t0 + t]; });
    };
    if (B.block_num < 256) // few BLBs: the TLBs are shared out (and no parallel region is around that), else the BLBs
    {
        for (u64 i = 0; i < B.block_num; i++)
            for (u64 w = B.index.v[i]; w < B.index.v[i + 1]; w++) of_wlb(i, w, true);
    }
    else
        share_steps(B.block_num, 4, T.block_num > kParallelRows ? crew_width() : 1, [&](u64 i, u64 e, unsigned) {
            for (; i < e; i++)
                for (u64 w = B.index.v[i]; w < B.index.v[i + 1]; w++) of_wlb(i, w, false);
        });
    adjacent_equal = T.block_num > 1 && !all_of(T.block_num - 1, [&](u64 t) { return rows[t] != rows[t + 1]; });
    return out;
}

// CSR over TLBs: TLBs of row r are [out[r], out[r + 1])
std::vector<u64> row_offsets(U64s rows, u64 n_rows)
{
    std::vector<u64> out(n_rows + 1, 0);
    if (rows.size() > 1 && all_of(rows.size() - 1, [&](u64 t) { return rows[t] <= rows[t + 1]; }))
    {
        // ascending rows: out[r] is the first TLB whose row is not below r
        for_each(rows.n, rows.n > kParallelRows, [&](u64 t) {
            for (u64 r = t == 0 ? 0 : rows[t - 1] + 1; r <= rows[t]; r++) out[r] = t;
        });
        for (u64 r = rows.back() + 1; r <= n_rows; r++) out[r] = rows.n;
        return out;
    }
    for (u64 t = 0; t < rows.n; t++) out[rows[t] + 1]++;
    for (u64 r = 0; r < n_rows; r++) out[r + 1] += out[r];
    return out;
}

void common_head(const Matrix &m, const CompressedBlock &b, int type, TemplateData &t)
{
    t = TemplateData();
    t.arrays.reserve(16); // references returned by add_meta stay valid while arrays are appended
    t.template_type = type;
    t.val_dt = m.val_dt;
    t.first_row = b.min_row;
    t.first_col = b.min_col;
    t.true_nnz = b.end_coo - b.begin_coo + 1;
    t.sort_kind = m.is_sorted ? ASP_SORT_GLOBAL : ASP_SORT_NONE;
    t.n_blb = b.blb.block_num;
    t.n_wlb = b.wlb.block_num;
    t.n_tlb = b.tlb.block_num;
    // sub-matrices that do not span all columns always accumulate atomically
    t.is_atom_add = !(b.min_col == 0 && b.max_col == m.n_cols - 1);
}

void add_perm(const Matrix &m, TemplateData &t)
{
    if (!m.is_sorted) return;
    t.arrays.emplace_back();
    TemplateArray &a = t.arrays.back();
    a.role = ASP_ARR_ROW_INDEX_BEFORE_SORT;
    a.dt = m.perm_dt;
    a.len = m.n_rows;
    a.shared = m.sorted_row_index;
}

// effective unit count + host-side permutation of a row map (templates whose kernels do not read
// row_index_before_sort): rows >= the dense row count belong to COMPRESSED_ROW_PADDING
// The rows have to be the caller's own buffer.
u64 effective_and_permute(const Matrix &m, const CompressedBlock &b, u64 *rows, u64 n)
{
    const u64 dense_rows = b.max_row - b.min_row + 1;
    std::atomic<u64> first(n);
    if (b.n_rows > dense_rows)
        share_ranges(n, n > kParallelRows, [&](u64 i, u64 e) {
            while (i < e && rows[i] < dense_rows) i++;
            if (i < e) lower(first, i);
        });
    const u64 eff = first.load(std::memory_order_relaxed);
    if (m.is_sorted) for_each(eff, eff > kParallelRows, [&](u64 i) { rows[i] = m.perm[rows[i] + b.min_row]; });
    return eff;
}

void try_linear_then_cycle_increase(TemplateArray &a, U64s v)
{
    if (!detect_linear(v, a.comp)) detect_cycle_increase(v, a.comp);
}

// ---- DIRECT_ATOM_TEMPLATE_WARP_BLOCK_COMPRESS (direct_atom_op_warp_block_compress.cc) --------
bool init_k3(const Matrix &m, const CompressedBlock &b, TemplateData &t, std::string &err)
{
    common_head(m, b, ASP_DIRECT_ATOM_TEMPLATE_WARP_BLOCK_COMPRESS, t);
    const u64 S = b.tlb.coo_size.v[0];
    for (u64 s : b.tlb.coo_size.v)
        if (s != S)
        {
            err = "ELL-like template needs one global TLB size";
            return false;
        }
    bool adj = false;
    Arr<u64> rows = tlb_global_rows(b, adj);
    if (adj) t.is_atom_add = true;
    const u64 n_pad = b.pad_col.size(), P = n_pad / S;
    Arr<uint8_t> col, val;
    interleave_cols(col.make(n_pad * dtype_bytes(b.col_dt)), b.col_dt, b.pad_col.data(), P, S);
    interleave_vals(val.make(n_pad * b.val.es), b.val.es, b.pad_val.b.data(), P, S);
    t.effective_num = effective_and_permute(m, b, rows.mut(), rows.size());
    t.tlb_size = S;
    TemplateArray &rm = add_meta(t, ASP_ARR_GLOBAL_ROW_INDEX_OF_THREAD_LEVEL_BLOCK, rows, suitable_dtype(max_entry(rows)));
    try_linear_then_cycle_increase(rm, rows);
    add_perm(m, t);
    add_nnz_arrays(t, b, col, val, n_pad);
    return true;
}

// per-BLB view shared by the SELL-like and the row-grouped templates: TLB range and TLB size
bool blb_tlb_ranges(const CompressedBlock &b, std::vector<u64> &thr, std::vector<u64> &size, std::string &err)
{
    const Level &B = b.blb, &W = b.wlb, &T = b.tlb;
    thr.resize(B.block_num + 1);
    size.resize(B.block_num);
    for (u64 i = 0; i < B.block_num; i++)
    {
        const u64 w0 = B.index.v[i];
        thr[i] = W.index.v[w0];
        size[i] = T.coo_size.v[w0];
        for (u64 w = w0; w < B.index.v[i + 1]; w++)
            if (T.coo_size.v[w] != size[i])
            {
                err = "TLB size differs inside a BLB";
                return false;
            }
    }
    thr[B.block_num] = W.index.v[W.block_num];
    return true;
}

void interleave_per_blb(const CompressedBlock &b, const std::vector<u64> &thr, const std::vector<u64> &size, Arr<uint8_t> &col, Arr<uint8_t> &val)
{
    const u64 n_pad = b.pad_col.size();
    const int cb = dtype_bytes(b.col_dt), es = b.val.es;
    uint8_t *cp = col.make(n_pad * cb), *vp = val.make(n_pad * es);
    const u64 nb = b.blb.block_num;
    auto of_blb = [&](u64 i) {
        const u64 nz0 = b.blb.coo_begin.v[i], n = thr[i + 1] - thr[i];
        interleave_cols(cp + nz0 * cb, b.col_dt, b.pad_col.data() + nz0, n, size[i]);
        interleave_vals(vp + nz0 * es, es, b.pad_val.b.data() + nz0 * es, n, size[i]);
    };
    share_steps(nb, 4, n_pad > kParallelNnz ? crew_width() : 1, [&](u64 i, u64 e, unsigned) {
        for (; i < e; i++) of_blb(i);
    });
}

// ---- DIRECT_ATOM_TEMPLATE_WARP_COMPRESS (direct_atom_op_warp_compress.cc) --------------------
bool init_k2(const Matrix &m, const CompressedBlock &b, TemplateData &t, std::string &err)
{
    common_head(m, b, ASP_DIRECT_ATOM_TEMPLATE_WARP_COMPRESS, t);
    std::vector<u64> thr, size;
    if (!blb_tlb_ranges(b, thr, size, err)) return false;
    bool adj = false;
    Arr<u64> rows = tlb_global_rows(b, adj);
    if (adj) t.is_atom_add = true;
    Arr<uint8_t> col, val;
    interleave_per_blb(b, thr, size, col, val);
    t.effective_num = effective_and_permute(m, b, rows.mut(), rows.size());
    TemplateArray &rm = add_meta(t, ASP_ARR_GLOBAL_ROW_INDEX_OF_THREAD_LEVEL_BLOCK, rows, suitable_dtype(max_entry(rows)));
    try_linear_then_cycle_increase(rm, rows);
    TemplateArray &bt = add_meta(t, ASP_ARR_BLOCK_BEGIN_THREAD_INDEX_OFFSET, thr, suitable_dtype(thr.back()));
    detect_linear(thr, bt.comp);
    std::vector<u64> bnz(b.blb.coo_begin.v.begin(), b.blb.coo_begin.v.begin() + b.blb.block_num);
    TemplateArray &bn = add_meta(t, ASP_ARR_BLOCK_NZ_BEGIN_OFFSET, bnz, b.blb.coo_begin.dt);
    detect_linear(bnz, bn.comp);
    // The reference narrows this array by its LAST entry (direct_atom_op_warp_compress.cc:239, 544),
    // which is the smallest one after a descending row sort: strips
    // whose widest TLB needs more bits are then truncated (372 stored as 116). The type here is
    // wide enough for the largest entry; it equals the reference's whenever the reference is right.
    TemplateArray &ts = add_meta(t, ASP_ARR_THREAD_BLOCK_SIZE_IN_BLOCK, size, suitable_dtype(*std::max_element(size.begin(), size.end())));
    if (!detect_constant(size, ts.comp)) detect_branch(size, ts.comp);
    add_perm(m, t);
    add_nnz_arrays(t, b, col, val, b.pad_col.size());
    return true;
}

// ---- SHARED_MEMORY_TEMPLATE_WARP_COMPRESS (shared_memory_op_warp_compress.cc) ----------------
bool init_k6(const Matrix &m, const CompressedBlock &b, TemplateData &t, std::string &err)
{
    common_head(m, b, ASP_SHARED_MEMORY_TEMPLATE_WARP_COMPRESS, t);
    const Level &B = b.blb;
    std::vector<u64> thr, size;
    if (!blb_tlb_ranges(b, thr, size, err)) return false;
    // BLBs that overlap in rows (column-divided BLBs) force atomics
    u64 gmax = B.first_row.v[0] + B.row_num.v[0] - 1;
    for (u64 i = 1; i < B.block_num; i++)
    {
        if (B.first_row.v[i] <= gmax)
        {
            t.is_atom_add = true;
            break;
        }
        gmax = std::max(gmax, B.first_row.v[i] + B.row_num.v[i] - 1);
    }
    t.effective_num = b.max_row - b.min_row + 1;
    bool adj = false;
    const Arr<u64> rows = tlb_global_rows(b, adj);
    const std::vector<u64> roff = row_offsets(rows, b.n_rows);
    Arr<uint8_t> col, val;
    interleave_per_blb(b, thr, size, col, val); // every BLB, the last one included (the reference skips it)
    TemplateArray &ro = add_meta(t, ASP_ARR_ROW_OFFSET_IN_THREAD_TMP_RESULT, roff, suitable_dtype(roff.back()));
    std::vector<u64> brow(B.first_row.v);
    brow.push_back(b.n_rows);
    TemplateArray &br = add_meta(t, ASP_ARR_BLOCK_FIRST_ROW_INDEX, brow, suitable_dtype(b.n_rows));
    TemplateArray &bt = add_meta(t, ASP_ARR_BLOCK_BEGIN_THREAD_INDEX_OFFSET, thr, suitable_dtype(thr.back()));
    TemplateArray &ts = add_meta(t, ASP_ARR_THREAD_BLOCK_SIZE_IN_BLOCK, size, b.tlb.coo_size.dt);
    std::vector<u64> bnz(B.coo_begin.v.begin(), B.coo_begin.v.begin() + B.block_num);
    TemplateArray &bn = add_meta(t, ASP_ARR_BLOCK_NZ_BEGIN_OFFSET, bnz, B.coo_begin.dt);
    detect_linear(thr, bt.comp);
    if (!detect_constant(size, ts.comp)) detect_branch(size, ts.comp);
    detect_linear(bnz, bn.comp);
    detect_linear(brow, br.comp);
    detect_linear(roff, ro.comp);
    add_perm(m, t);
    add_nnz_arrays(t, b, col, val, b.pad_col.size());
    return true;
}
// read_index[6] / staggered_padding_val_arr: inside every WLB the TLBs are taken in groups of 32 and
// element k of lane l of group g moves to g*32*S + k*32 + l (op_manager.cc:3569-3589). Identity
// when every TLB holds one non-zero.
void staggered_arrays(const CompressedBlock &b, Arr<uint8_t> &col, Arr<uint8_t> &val)
{
    const u64 n_pad = b.pad_col.size();
    const int cb = dtype_bytes(b.col_dt), es = b.val.es;
    const Level &B = b.blb, &W = b.wlb;
    const U64s sizes(b.tlb.coo_size.v);
    if (all_of(sizes.size(), [&](u64 w) { return sizes[w] == 1; }))
    {
        val = b.pad_val.b;
        if (cb == 4) col = b.pad_col.bytes();
        else interleave_cols(col.make(n_pad * cb), b.col_dt, b.pad_col.data(), n_pad, 1);
        return;
    }
    uint8_t *cp = col.make(n_pad * cb), *vp = val.make(n_pad * es);
    const u64 nb = B.block_num;
    auto of_wlb = [&](u64 i, u64 w) {
        const u64 S = b.tlb.coo_size.v[w];
        const u64 base = B.coo_begin.v[i] + W.coo_begin.v[w];
        const u64 groups = (W.index.v[w + 1] - W.index.v[w]) / 32;
        for (u64 g = 0; g < groups; g++)
        {
            const u64 o = base + g * 32 * S;
            interleave_cols(cp + o * cb, b.col_dt, b.pad_col.data() + o, 32, S);
            interleave_vals(vp + o * es, es, b.pad_val.b.data() + o * es, 32, S);
        }
    };
    if (nb < 256)
        for (u64 i = 0; i < nb; i++)
        {
            const u64 w0 = B.index.v[i], w1 = B.index.v[i + 1];
            for_each(w1 - w0, w1 - w0 > 1024, [&](u64 w) { of_wlb(i, w0 + w); });
        }
    else
        share_steps(nb, 4, n_pad > kParallelNnz ? crew_width() : 1, [&](u64 i, u64 e, unsigned) {
            for (; i < e; i++)
                for (u64 w = B.index.v[i]; w < B.index.v[i + 1]; w++) of_wlb(i, w);
        });
}

std::vector<u64> first_n(const std::vector<u64> &v, u64 n) { return std::vector<u64>(v.begin(), v.begin() + n); }

// ---- DIRECT_ATOM_TOTAL_WARP_REDUCE_TEMPLATE (direct_atom_total_warp_reduce_op.cc) ------------
bool init_k4(const Matrix &m, const CompressedBlock &b, TemplateData &t, std::string &err)
{
    common_head(m, b, ASP_DIRECT_ATOM_TOTAL_WARP_REDUCE_TEMPLATE, t);
    const Level &B = b.blb, &W = b.wlb;
    std::vector<u64> rows(W.block_num), nz(W.block_num + 1);
    for (u64 i = 0; i < B.block_num; i++)
        for (u64 w = B.index.v[i]; w < B.index.v[i + 1]; w++)
        {
            if (W.row_num.v[w] != 1)
            {
                err = "warp-per-row template needs one row per WLB";
                return false;
            }
            rows[w] = B.first_row.v[i] + W.first_row.v[w];
            nz[w] = B.coo_begin.v[i] + W.coo_begin.v[w];
            if (w >= 1 && rows[w] == rows[w - 1]) t.is_atom_add = true;
        }
    nz[W.block_num] = b.pad_col.size();
    t.effective_num = effective_and_permute(m, b, rows.data(), rows.size());
    const u64 mx = max_entry(rows);
    TemplateArray &rm = add_meta(t, ASP_ARR_GLOBAL_ROW_INDEX_OF_WARP_LEVEL_BLOCK, rows, suitable_dtype(mx));
    try_linear_then_cycle_increase(rm, rows);
    TemplateArray &no = add_meta(t, ASP_ARR_GLOBAL_WARP_NZ_BEGIN_OFFSET, nz, suitable_dtype(b.pad_col.size() + 1));
    detect_linear(nz, no.comp);
    add_perm(m, t);
    Arr<uint8_t> col, val;
    staggered_arrays(b, col, val);
    add_nnz_arrays(t, b, col, val, b.pad_col.size());
    return true;
}

// ---- SHARED_MEMORY_LONG_ROW_TEMPLATE (shared_memory_long_row_op.cc) ---------------------------
bool init_k7(const Matrix &m, const CompressedBlock &b, TemplateData &t, std::string &err)
{
    common_head(m, b, ASP_SHARED_MEMORY_LONG_ROW_TEMPLATE, t);
    const Level &B = b.blb;
    for (u64 i = 0; i < B.block_num; i++)
    {
        if (B.row_num.v[i] != 1)
        {
            err = "long-row template needs one row per BLB";
            return false;
        }
        if (i + 1 < B.block_num && B.first_row.v[i] == B.first_row.v[i + 1]) t.is_atom_add = true;
    }
    for (u64 s : b.tlb.coo_size.v)
        if (s != 1)
        {
            err = "long-row template needs TLB size 1";
            return false;
        }
    std::vector<u64> rows(B.first_row.v);
    if (m.is_sorted)
        for (u64 &r : rows) r = m.perm[r + b.min_row];
    u64 mx = 0;
    for (u64 r : rows) mx = std::max(mx, r);
    TemplateArray &rm = add_meta(t, ASP_ARR_ROW_INDEX_OF_BLOCK_LEVEL_BLOCK, rows, suitable_dtype(mx));
    try_linear_then_cycle_increase(rm, rows);
    TemplateArray &bn = add_meta(t, ASP_ARR_BLOCK_NZ_BEGIN_OFFSET, B.coo_begin.v, B.coo_begin.dt);
    detect_linear(B.coo_begin.v, bn.comp);
    add_perm(m, t);
    Arr<uint8_t> col, val;
    staggered_arrays(b, col, val);
    add_nnz_arrays(t, b, col, val, b.pad_col.size());
    return true;
}

bool blbs_overlap_in_rows(const Level &B)
{
    u64 gmax = B.first_row.v[0] + B.row_num.v[0] - 1;
    for (u64 i = 1; i < B.block_num; i++)
    {
        if (B.first_row.v[i] <= gmax) return true;
        gmax = std::max(gmax, B.first_row.v[i] + B.row_num.v[i] - 1);
    }
    return false;
}

// ---- SHARED_MEMORY_TOTAL_WARP_REDUCE_TEMPLATE (shared_memory_total_warp_reduce_op.cc) ---------
bool init_k8(const Matrix &m, const CompressedBlock &b, TemplateData &t, std::string &err)
{
    common_head(m, b, ASP_SHARED_MEMORY_TOTAL_WARP_REDUCE_TEMPLATE, t);
    const Level &B = b.blb, &W = b.wlb;
    if (blbs_overlap_in_rows(B)) t.is_atom_add = true;
    t.effective_num = b.max_row - b.min_row + 1;
    std::vector<u64> roff(b.n_rows + 1, 0), nz(W.block_num + 1);
    for (u64 i = 0; i < B.block_num; i++)
        for (u64 w = B.index.v[i]; w < B.index.v[i + 1]; w++)
        {
            if (W.row_num.v[w] != 1)
            {
                err = "warp-reduce shared-memory template needs one row per WLB";
                return false;
            }
            roff[B.first_row.v[i] + W.first_row.v[w] + 1]++;
            nz[w] = B.coo_begin.v[i] + W.coo_begin.v[w];
        }
    nz[W.block_num] = b.pad_col.size();
    for (u64 r = 0; r < b.n_rows; r++) roff[r + 1] += roff[r];
    TemplateArray &ro = add_meta(t, ASP_ARR_ROW_OFFSET_IN_WARP_TMP_RESULT, roff, suitable_dtype(roff.back()));
    std::vector<u64> brow(B.first_row.v);
    brow.push_back(b.n_rows);
    TemplateArray &br = add_meta(t, ASP_ARR_BLOCK_FIRST_ROW_INDEX, brow, suitable_dtype(b.n_rows));
    TemplateArray &bw = add_meta(t, ASP_ARR_BLOCK_BEGIN_WARP_INDEX_OFFSET, B.index.v, B.index.dt);
    TemplateArray &fn = add_meta(t, ASP_ARR_GLOBAL_WARP_BLOCK_FIRST_NZ, nz, suitable_dtype(nz.back()));
    detect_linear(B.index.v, bw.comp);
    detect_linear(roff, ro.comp);
    detect_linear(brow, br.comp);
    detect_linear(nz, fn.comp);
    add_perm(m, t);
    Arr<uint8_t> col, val;
    staggered_arrays(b, col, val);
    add_nnz_arrays(t, b, col, val, b.pad_col.size());
    return true;
}

// closed form of warp_nz_begin_offset in the 3-level templates: cycle-linear with the cycle taken
// from the linear form of block_begin_warp_index_offset (direct_atom_op.cc:1828-1890)
void try_cycle_linear_warp_nz(TemplateArray &wn, const std::vector<u64> &v, const TemplateArray &bw, const std::vector<u64> &bwv)
{
    u64 cycle = 0;
    if (bw.comp.kind == ASP_COMPRESS_LINEAR) cycle = bw.comp.coef;
    else
    {
        ClosedForm f;
        if (!detect_linear(bwv, f)) return;
        cycle = f.coef;
    }
    detect_cycle_linear(v, cycle, wn.comp);
}

// ---- DIRECT_ATOM_TEMPLATE (direct_atom_op.cc) --------------------------------------------------
bool init_k1(const Matrix &m, const CompressedBlock &b, TemplateData &t, std::string &err)
{
    common_head(m, b, ASP_DIRECT_ATOM_TEMPLATE, t);
    const Level &B = b.blb, &W = b.wlb;
    bool adj = false;
    Arr<u64> rows = tlb_global_rows(b, adj);
    if (adj) t.is_atom_add = true;
    if (m.is_sorted)
        for (u64 i = 0; i < rows.size(); i++) rows.mut()[i] = m.perm[rows[i] + b.min_row]; // every TLB, padded rows included, as the reference does
    u64 mx = 0;
    for (u64 r : rows) mx = std::max(mx, r);
    TemplateArray &rm = add_meta(t, ASP_ARR_GLOBAL_ROW_INDEX_OF_THREAD_LEVEL_BLOCK, rows, suitable_dtype(mx));
    TemplateArray &bw = add_meta(t, ASP_ARR_BLOCK_BEGIN_WARP_INDEX_OFFSET, B.index.v, B.index.dt);
    TemplateArray &wt = add_meta(t, ASP_ARR_WARP_BEGIN_THREAD_INDEX_OFFSET, W.index.v, W.index.dt);
    TemplateArray &ts = add_meta(t, ASP_ARR_THREAD_BLOCK_SIZE_IN_WARP, b.tlb.coo_size.v, b.tlb.coo_size.dt);
    std::vector<u64> bnz = first_n(B.coo_begin.v, B.block_num);
    TemplateArray &bn = add_meta(t, ASP_ARR_BLOCK_NZ_BEGIN_OFFSET, bnz, B.coo_begin.dt);
    TemplateArray &wn = add_meta(t, ASP_ARR_WARP_NZ_BEGIN_OFFSET, W.coo_begin.v, W.coo_begin.dt);
    try_linear_then_cycle_increase(rm, rows);
    detect_linear(B.index.v, bw.comp);
    detect_linear(W.index.v, wt.comp);
    if (!detect_constant(b.tlb.coo_size.v, ts.comp)) detect_branch(b.tlb.coo_size.v, ts.comp);
    detect_linear(bnz, bn.comp);
    try_cycle_linear_warp_nz(wn, W.coo_begin.v, bw, B.index.v);
    add_perm(m, t);
    Arr<uint8_t> col, val;
    staggered_arrays(b, col, val);
    add_nnz_arrays(t, b, col, val, b.pad_col.size());
    (void)err;
    return true;
}

// ---- SHARED_MEMORY_TEMPLATE (shared_memory_op.cc) ----------------------------------------------
bool init_k5(const Matrix &m, const CompressedBlock &b, TemplateData &t, std::string &err)
{
    common_head(m, b, ASP_SHARED_MEMORY_TEMPLATE, t);
    const Level &B = b.blb, &W = b.wlb;
    if (blbs_overlap_in_rows(B)) t.is_atom_add = true;
    bool adj = false;
    const Arr<u64> rows = tlb_global_rows(b, adj);
    const std::vector<u64> roff = row_offsets(rows, b.n_rows);
    // values / columns interleaved per WLB: element k of local TLB i at base + i + k*n_w
    const u64 n_pad = b.pad_col.size();
    const int cb = dtype_bytes(b.col_dt), es = b.val.es;
    Arr<uint8_t> col, val;
    uint8_t *cp = col.make(n_pad * cb), *vp = val.make(n_pad * es);
    for (u64 i = 0; i < B.block_num; i++)
        for (u64 w = B.index.v[i]; w < B.index.v[i + 1]; w++)
        {
            const u64 base = B.coo_begin.v[i] + W.coo_begin.v[w], n = W.index.v[w + 1] - W.index.v[w], S = b.tlb.coo_size.v[w];
            interleave_cols(cp + base * cb, b.col_dt, b.pad_col.data() + base, n, S);
            interleave_vals(vp + base * es, es, b.pad_val.b.data() + base * es, n, S);
        }
    TemplateArray &ro = add_meta(t, ASP_ARR_ROW_OFFSET_IN_THREAD_TMP_RESULT, roff, suitable_dtype(roff.back()));
    std::vector<u64> brow(B.first_row.v);
    brow.push_back(b.n_rows);
    TemplateArray &br = add_meta(t, ASP_ARR_BLOCK_FIRST_ROW_INDEX, brow, suitable_dtype(b.n_rows));
    TemplateArray &bw = add_meta(t, ASP_ARR_BLOCK_BEGIN_WARP_INDEX_OFFSET, B.index.v, B.index.dt);
    TemplateArray &wt = add_meta(t, ASP_ARR_WARP_BEGIN_THREAD_INDEX_OFFSET, W.index.v, W.index.dt);
    TemplateArray &ts = add_meta(t, ASP_ARR_THREAD_BLOCK_SIZE_IN_WARP, b.tlb.coo_size.v, b.tlb.coo_size.dt);
    std::vector<u64> bnz = first_n(B.coo_begin.v, B.block_num);
    TemplateArray &bn = add_meta(t, ASP_ARR_BLOCK_NZ_BEGIN_OFFSET, bnz, B.coo_begin.dt);
    TemplateArray &wn = add_meta(t, ASP_ARR_WARP_NZ_BEGIN_OFFSET, W.coo_begin.v, W.coo_begin.dt);
    detect_linear(B.index.v, bw.comp);
    detect_linear(W.index.v, wt.comp);
    if (!detect_constant(b.tlb.coo_size.v, ts.comp)) detect_branch(b.tlb.coo_size.v, ts.comp);
    detect_linear(bnz, bn.comp);
    try_cycle_linear_warp_nz(wn, W.coo_begin.v, bw, B.index.v);
    detect_linear(brow, br.comp);
    detect_linear(roff, ro.comp);
    add_perm(m, t);
    add_nnz_arrays(t, b, col, val, n_pad);
    (void)err;
    return true;
}

int bit_count(u64 v)
{
    int n = 0;
    while (v)
    {
        v >>= 1;
        n++;
    }
    return n;
}

// ---- UNALIGNED_WARP_REDUCE_SAME_TLB_SIZE_TEMPLATE[_WITH_WARP_REDUCE] ---------------------------
// (unaligned_warp_reduce_same_TLB_size_op.cc:5-297, helpers :434-512 and :1332-1645)
bool init_k9(const Matrix &m, const CompressedBlock &b, bool with_warp_reduce, TemplateData &t, std::string &err)
{
    common_head(m, b, with_warp_reduce ? ASP_UNALIGNED_WARP_REDUCE_SAME_TLB_SIZE_TEMPLATE_WITH_WARP_REDUCE : ASP_UNALIGNED_WARP_REDUCE_SAME_TLB_SIZE_TEMPLATE, t);
    if (!b.tlb_is_nnz_div)
    {
        err = "CSR5-like templates need the TLB level built by the nnz division";
        return false;
    }
    const u64 S = b.tlb.coo_size.v[0];
    if (S > 62)
    {
        err = "CSR5-like: row-start flags + offsets do not fit in 64 bits";
        return false;
    }
    // Elements: the non-zeros in row order; a row without any becomes one zero at column 0 (rows after the last non-zero are
    // dropped); the tail is padded to whole warps by repeating the last (row, column) with value 0. Row r holds elements
    // [first[r], first[r + 1]).
    u64 last_row = 0;
    for (u64 r = b.n_rows; r-- > 0;)
        if (b.rowptr[r + 1] > b.rowptr[r])
        {
            last_row = r;
            break;
        }
    const u64 R = last_row + 1;
    Arr<u64> first_arr;
    u64 *first = first_arr.make(R + 1);
    first[0] = 0;
    for (u64 r = 0; r < R; r++) first[r + 1] = first[r] + std::max<u64>(1, b.rowptr[r + 1] - b.rowptr[r]);
    const u64 n_el = first[R], wn = 32 * S, n = (n_el + wn - 1) / wn * wn, T = n / S, Wn = T / 32;
    const int cb = dtype_bytes(b.col_dt), es = b.val.es;
    // A warp's share is built by one thread: its elements (element k of lane l of warp w goes to w*32*S + k*32 + l), the flags
    // of its TLBs (the first element of a warp always starts a sum) and the first row that starts in each of them, relative to
    // the warp's first row (a TLB without a row start repeats the TLB before it).
    Arr<uint8_t> ocol, oval;
    uint8_t *const cp = ocol.make(n * cb), *const vp = oval.make(n * es);
    Arr<u64> flags_arr;
    u64 *const flags = flags_arr.make(T);
    Arr<u32> frow_arr;
    u32 *const frow = frow_arr.make(T);
    std::vector<u64> wfirst(Wn);
    std::atomic<u64> most_frow(0);
    const auto fill = [&, cp, vp, flags, frow, first, S, R, wn, cb, es, last_row, rowptr = b.rowptr.data(), bcol = b.col.data(), src = b.val.b.data()](u64 w) ASP_INLINE {
        const u64 e0 = w * wn, e1 = e0 + wn;
        u64 top = 0;
        u64 r = std::min<u64>((u64)(std::upper_bound(first, first + R + 1, e0) - first) - 1, last_row);
        wfirst[w] = r;
        for (u64 tl = w * 32; tl < w * 32 + 32; tl++) flags[tl] = 0;
        u64 e = e0, k = 0, lane = 0;
        while (e < e1)
        {
            const u64 end = r < last_row ? std::min(e1, first[r + 1]) : e1; // fillers continue the last row
            const u64 nz0 = rowptr[r], nz = rowptr[r + 1] - nz0;
            if (e == e0 || e == first[r])
            {
                const u64 tl = w * 32 + lane;
                if (flags[tl] == 0) frow[tl] = (u32)(r - wfirst[w]);
                flags[tl] |= 1ull << (S - 1 - k);
            }
            for (; e < end; e++)
            {
                const u64 q = e - first[r], d = e0 + k * 32 + lane;
                if (++k == S) k = 0, lane++;
                const u32 c = nz == 0 ? 0 : bcol[nz0 + std::min(q, nz - 1)];
                switch (cb)
                {
                case 1: cp[d] = (uint8_t)c; break;
                case 2: ((uint16_t *)cp)[d] = (uint16_t)c; break;
                case 4: ((u32 *)cp)[d] = c; break;
                default: ((u64 *)cp)[d] = c; break;
                }
                if (es == 8) ((u64 *)vp)[d] = q < nz ? ((const u64 *)src)[nz0 + q] : 0;
                else ((u32 *)vp)[d] = q < nz ? ((const u32 *)src)[nz0 + q] : 0;
            }
            r++;
        }
        for (u64 tl = w * 32; tl < w * 32 + 32; tl++)
        {
            if (flags[tl] == 0) frow[tl] = frow[tl - 1]; // (the warp's first TLB always has a flag)
            top = std::max<u64>(top, frow[tl]);
        }
        return top;
    };
    share_ranges(Wn, n > kParallelNnz, [&](u64 w, u64 e) {
        const auto mine = fill; // (what it holds by value, in this thread's registers)
        u64 top = 0;
        for (; w < e; w++) top = std::max(top, mine(w));
        raise(most_frow, top);
    });
    const u64 max_frow = most_frow.load(std::memory_order_relaxed);
    // per TLB with a row start: the number of following TLBs without one
    std::vector<u32> roff(T, 0);
    u64 max_roff = 0, last_head = 0;
    for (u64 tl = 1; tl <= T; tl++)
        if (tl == T || flags[tl] != 0)
        {
            roff[last_head] = (u32)(tl - 1 - last_head);
            max_roff = std::max<u64>(max_roff, roff[last_head]);
            last_head = tl;
        }
    int bits_row = bit_count(max_frow), bits_off = bit_count(max_roff);
    if (bits_row == 0) bits_row = 1;
    if (bits_off == 0) bits_off = 1;
    const int total_bits = (int)S + bits_row + bits_off;
    if (total_bits > 64)
    {
        err = "CSR5-like: row-start flags + offsets do not fit in 64 bits";
        return false;
    }
    const int word = total_bits <= 8 ? 8 : total_bits <= 16 ? 16 : total_bits <= 32 ? 32 : 64;
    const int meta_dt = word == 8 ? ASP_U8 : word == 16 ? ASP_U16 : word == 32 ? ASP_U32 : ASP_U64;
    u64 *const meta = flags; // (in place)
    for_each(T, T > kParallelRows, [&](u64 tl) { meta[tl] = (((flags[tl] << (word - (int)S - bits_row)) | roff[tl]) << bits_row) | frow[tl]; });
    t.tlb_size = S;
    t.bits_word = word;
    t.bits_flag = (int)S;
    t.bits_row = bits_row;
    t.bits_off = bits_off;
    t.n_tlb = (b.col.size() + S - 1) / S;
    if (with_warp_reduce) wfirst.push_back(last_row + 1);
    TemplateArray &fr = add_meta(t, ASP_ARR_GLOBAL_FIRST_ROW_INDEX_OF_WARP_LEVEL_BLOCK, wfirst, b.row_dt);
    try_linear_then_cycle_increase(fr, wfirst);
    add_meta(t, ASP_ARR_COMBINE_META_OF_THREAD_LEVEL_BLOCK, flags_arr, meta_dt);
    add_perm(m, t);
    add_nnz_arrays(t, b, ocol, oval, n);
    return true;
}
} // namespace

namespace
{
// block columns (of R x R blocks) of every block row, merged over its rows, from where the non-zeros of its first row begin in
// bcol; returns the most of one block row
template <int R>
u64 block_columns(const CompressedBlock &b, u32 *const bcol, std::vector<u32> &cnt)
{
    std::atomic<u64> W(0);
    const auto merge = [&, rowptr = b.rowptr.data(), col = b.col.data()](u64 br) ASP_INLINE {
        const u64 row0 = br * R, row1 = std::min<u64>(b.n_rows, row0 + R), nz0 = rowptr[row0];
        u32 *const o = bcol + nz0;
        // the columns of a row ascend: its block columns come out in order; further rows usually repeat them
        u64 n = 0;
        for (u64 k = nz0; k < rowptr[row0 + 1]; k++)
        {
            const u32 c0 = col[k] / (u32)R;
            if (n == 0 || o[n - 1] != c0) o[n++] = c0;
        }
        bool merged = false;
        for (u64 row = row0 + 1; row < row1; row++)
        {
            u64 q = 0;
            const u64 sorted = n;
            for (u64 k = rowptr[row]; k < rowptr[row + 1]; k++)
            {
                const u32 c0 = col[k] / (u32)R;
                if (merged)
                {
                    o[n++] = c0; // (at most one entry per non-zero: it stays inside the block row's share)
                    continue;
                }
                while (q < sorted && o[q] < c0) q++;
                if (q < sorted && o[q] == c0) continue;
                o[n++] = c0;
            }
            merged = merged || n > sorted;
        }
        if (merged)
        {
            std::sort(o, o + n);
            n = (u64)(std::unique(o, o + n) - o);
        }
        cnt[br] = (u32)n;
        return n;
    };
    share_ranges(cnt.size(), b.nnz() > kParallelNnz, [&](u64 br, u64 e) {
        const auto mine = merge;
        u64 most = 0;
        for (; br < e; br++) most = std::max(most, mine(br));
        raise(W, most);
    });
    return W.load(std::memory_order_relaxed);
}

// the arrays of block rows [br, e): block columns ip[slot * NB + block row], values vp[((slot * R + i) * R + j) * NB + block row]
template <int R, class V>
void block_values(const CompressedBlock &b, const u32 *const bcol, const u32 *const cnt, u64 W, u64 NB, u32 *const ip, V *const vp, u64 br, u64 e)
{
    const V *const src = (const V *)b.val.b.data();
    const u64 n_rows = b.n_rows;
    const u32 *const col = b.col.data();
    const u64 *const rowptr = b.rowptr.data();
    for (; br < e; br++)
    {
        const u64 n = cnt[br];
        const u32 *bc = bcol + rowptr[br * R];
        for (u64 k = 0; k < W; k++) ip[k * NB + br] = k < n ? bc[k] : (n ? bc[n - 1] : 0); // zero blocks repeat the last block column
        // a block row of full blocks is overwritten whole (no column twice: entries are as many as there are places)
        const u64 q0 = rowptr[br * R], q1 = rowptr[std::min<u64>(n_rows, (br + 1) * R)];
        bool full = q1 - q0 == W * R * R && (br + 1) * R <= n_rows;
        for (u64 row = br * R; full && row < (br + 1) * R; row++)
            for (u64 q = rowptr[row] + 1; q < rowptr[row + 1]; q++) full = full && col[q] != col[q - 1];
        if (!full)
            for (u64 q = 0; q < W * R * R; q++) vp[q * NB + br] = 0;
        for (u64 row = br * R; row < std::min<u64>(n_rows, (br + 1) * R); row++)
        {
            const u64 i = row - br * R;
            u64 k = 0; // the columns of a row ascend, so do its block slots
            for (u64 q = rowptr[row]; q < rowptr[row + 1]; q++)
            {
                const u32 cb = col[q] / (u32)R;
                while (bc[k] != cb) k++;
                const u64 j = col[q] - (u64)cb * R;
                vp[((k * R + i) * R + j) * NB + br] = src[q];
            }
        }
    }
}
} // namespace

// ---- block-value template (this build's; no counterpart in the reference) --------------------------------
// Blocked ELL over dense r x c blocks: block rows of r consecutive rows, block columns of c consecutive columns
// (relative to the sub-matrix's first column); every block that holds a non-zero is stored in full, block rows
// are padded with zero blocks to the width of the widest one, and the block rows to an even count.
bool init_block_ell(const Matrix &m, const CompressedBlock &b, TemplateData &t, std::string &err)
{
    const u64 r = b.block_r, c = b.block_c;
    if (m.is_sorted) return err = "block_value: not for sorted matrices (a block row must be r consecutive rows of y)", false;
    if (!((r == 2 && c == 2) || (r == 3 && c == 3) || (r == 4 && c == 4))) return err = "block_value: blocks of 2 x 2, 3 x 3 or 4 x 4", false;
    const u64 width = b.max_col - b.min_col + 1;
    if (width % c) return err = "block_value: the columns of the sub-matrix are not a multiple of the block width", false;
    const u64 NBR = (b.n_rows + r - 1) / r, NB = (NBR + 1) / 2 * 2;
    Arr<u32> bcol_arr;
    u32 *const bcol = bcol_arr.make(std::max<u64>(1, b.col.size()));
    std::vector<u32> cnt(NBR, 0);
    const u64 W = r == 3 ? block_columns<3>(b, bcol, cnt) : r == 2 ? block_columns<2>(b, bcol, cnt) : block_columns<4>(b, bcol, cnt);
    if (W == 0) return err = "block_value: sub-matrix without non-zeros", false;
    const u64 stored = NB * W * r * c;
    if (b.nnz() == 0 || (double)stored / (double)b.nnz() > 8.0) return err = "block_value: the matrix is not made of dense blocks of this size (more than 8 stored values per non-zero)", false;
    const int es = b.val.es;
    Arr<uint8_t> idx, val;
    u32 *const ip = (u32 *)idx.make_zero(NB * W * 4);
    uint8_t *const vp = val.make(stored * (u64)es);
    for (u64 q = 0; NB > NBR && q < W * r * c; q++) memset(vp + (q * NB + NBR) * es, 0, es); // the block row that pads
    const u32 *const counts = cnt.data();
    share_ranges(NBR, b.nnz() > kParallelNnz, [&](u64 br, u64 e) {
        if (es == 8)
        {
            if (r == 3) block_values<3>(b, bcol, counts, W, NB, ip, (u64 *)vp, br, e);
            else if (r == 2) block_values<2>(b, bcol, counts, W, NB, ip, (u64 *)vp, br, e);
            else block_values<4>(b, bcol, counts, W, NB, ip, (u64 *)vp, br, e);
        }
        else if (r == 3) block_values<3>(b, bcol, counts, W, NB, ip, (u32 *)vp, br, e);
        else if (r == 2) block_values<2>(b, bcol, counts, W, NB, ip, (u32 *)vp, br, e);
        else block_values<4>(b, bcol, counts, W, NB, ip, (u32 *)vp, br, e);
    });
    common_head(m, b, ASP_BLOCK_ELL_TEMPLATE, t);
    t.tlb_size = W;
    t.bits_row = (int)r;
    t.bits_off = (int)c;
    t.effective_num = b.n_rows;
    t.n_blb = NBR;
    t.n_wlb = NBR;
    t.n_tlb = NB;
    t.thread_num_in_block = 128;
    t.tblock_num = (long)std::max<u64>(1, (NB / 2 + 127) / 128);
    t.arrays.emplace_back();
    TemplateArray &v = t.arrays.back();
    v.role = ASP_ARR_VAL;
    v.dt = t.val_dt;
    v.len = stored;
    v.bytes.swap(val);
    t.arrays.emplace_back();
    TemplateArray &ci = t.arrays.back();
    ci.role = ASP_ARR_COL_INDEX;
    ci.dt = ASP_U32;
    ci.len = NB * W;
    ci.bytes.swap(idx);
    return true;
}

// ---- diagonal-value template (this build's; no counterpart in the reference) ------------------------------
// DIA storage: the distinct offsets col - row of the sub-matrix (at most b.diag_max of them), values diagonal-major.
bool init_diag(const Matrix &m, const CompressedBlock &b, TemplateData &t, std::string &err)
{
    if (m.is_sorted) return err = "diag_value: not for sorted matrices (the diagonals are those of the original row order)", false;
    if (!(b.min_col == 0 && b.max_col == m.n_cols - 1)) return err = "diag_value: not for column-sliced sub-matrices", false;
    const int es = b.val.es;
    const u64 V = 16 / (u64)es, NR = (b.n_rows + V - 1) / V * V;
    const int64_t ncols = (int64_t)(b.max_col - b.min_col + 1);
    // distinct offsets, as bits of all there could be; a scattered matrix leaves after a few rows
    std::vector<u64> bits((b.n_rows + (u64)ncols) / 64 + 1, 0);
    u64 found = 0;
    for_each(b.n_rows, b.nnz() > kParallelNnz, [&](u64 r) {
        if (__atomic_load_n(&found, __ATOMIC_RELAXED) > b.diag_max) return;
        for (u64 k = b.rowptr[r]; k < b.rowptr[r + 1]; k++)
        {
            const u64 at = b.col[k] + b.n_rows - r, bit = 1ull << (at % 64);
            if (__atomic_load_n(&bits[at / 64], __ATOMIC_RELAXED) & bit) continue;
            if ((__atomic_fetch_or(&bits[at / 64], bit, __ATOMIC_RELAXED) & bit) == 0) __atomic_fetch_add(&found, 1, __ATOMIC_RELAXED);
        }
    });
    if (found > b.diag_max) return err = "diag_value: more than " + std::to_string(b.diag_max) + " diagonals hold non-zeros", false;
    if (found == 0) return err = "diag_value: sub-matrix without non-zeros", false;
    std::vector<int64_t> off; // ascending
    for (u64 w = 0; w < bits.size(); w++)
        for (u64 left = bits[w]; left; left &= left - 1) off.push_back((int64_t)(w * 64 + (u64)__builtin_ctzll(left)) - (int64_t)b.n_rows);
    const u64 D = off.size();
    Arr<uint8_t> val;
    uint8_t *const vp = val.make_zero(D * NR * (u64)es);
    for_each(b.n_rows, b.nnz() > kParallelNnz, [&](u64 r) {
        for (u64 k = b.rowptr[r]; k < b.rowptr[r + 1]; k++)
        {
            const u64 d = (u64)(std::lower_bound(off.begin(), off.end(), (int64_t)b.col[k] - (int64_t)r) - off.begin());
            memcpy(&vp[(d * NR + r) * es], &b.val.b[k * es], es);
        }
    });
    common_head(m, b, ASP_DIAG_TEMPLATE, t);
    t.tlb_size = D;
    t.effective_num = b.n_rows;
    t.n_blb = 1;
    t.n_wlb = 1;
    t.n_tlb = NR / V;
    t.thread_num_in_block = 256;
    t.tblock_num = (long)std::max<u64>(1, (NR / V + 255) / 256);
    t.arrays.emplace_back();
    TemplateArray &v = t.arrays.back();
    v.role = ASP_ARR_VAL;
    v.dt = t.val_dt;
    v.len = D * NR;
    v.bytes.swap(val);
    std::vector<u64> biased(D);
    for (u64 d = 0; d < D; d++) biased[d] = (u64)(off[d] + ncols);
    add_meta(t, ASP_ARR_COL_INDEX, biased, ASP_U64);
    return true;
}

bool init_template(const Matrix &m, size_t sub, int type, TemplateData &out, std::string &err)
{
    if (sub >= m.blocks.size())
    {
        err = "no such sub-matrix";
        return false;
    }
    const CompressedBlock &b = m.blocks[sub];
    if (type == ASP_DIAG_TEMPLATE)
    {
        if (!b.diag_max) return err = "the template D1 needs the diag_value node", false;
        return init_diag(m, b, out, err);
    }
    if (type == ASP_BLOCK_ELL_TEMPLATE)
    {
        if (!b.block_r) return err = "the template B1 needs the block_value node", false;
        return init_block_ell(m, b, out, err);
    }
    const bool csr5 = type == ASP_UNALIGNED_WARP_REDUCE_SAME_TLB_SIZE_TEMPLATE || type == ASP_UNALIGNED_WARP_REDUCE_SAME_TLB_SIZE_TEMPLATE_WITH_WARP_REDUCE;
    if (!csr5 && b.tlb_is_nnz_div)
    {
        err = "this template needs an ELL-style TLB level";
        return false;
    }
    if (!(b.blb.built && b.wlb.built && b.tlb.built))
    {
        err = "sub-matrix is not tiled at all three levels";
        return false;
    }
    switch (type)
    {
    case ASP_DIRECT_ATOM_TEMPLATE_WARP_BLOCK_COMPRESS: return init_k3(m, b, out, err);
    case ASP_DIRECT_ATOM_TEMPLATE_WARP_COMPRESS: return init_k2(m, b, out, err);
    case ASP_SHARED_MEMORY_TEMPLATE_WARP_COMPRESS: return init_k6(m, b, out, err);
    case ASP_DIRECT_ATOM_TOTAL_WARP_REDUCE_TEMPLATE: return init_k4(m, b, out, err);
    case ASP_SHARED_MEMORY_LONG_ROW_TEMPLATE: return init_k7(m, b, out, err);
    case ASP_SHARED_MEMORY_TOTAL_WARP_REDUCE_TEMPLATE: return init_k8(m, b, out, err);
    case ASP_DIRECT_ATOM_TEMPLATE: return init_k1(m, b, out, err);
    case ASP_SHARED_MEMORY_TEMPLATE: return init_k5(m, b, out, err);
    case ASP_UNALIGNED_WARP_REDUCE_SAME_TLB_SIZE_TEMPLATE: return init_k9(m, b, false, out, err);
    case ASP_UNALIGNED_WARP_REDUCE_SAME_TLB_SIZE_TEMPLATE_WITH_WARP_REDUCE: return init_k9(m, b, true, out, err);
    default: err = "template not implemented by the host lowering"; return false;
    }
}

} // namespace host
} // namespace asp

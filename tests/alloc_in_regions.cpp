// Memory runs out while the host builds formats and layouts. Argument "region": every allocation in a piece of a shared loop fails (an
// exception cannot leave one, so none may be made there); "any": the n-th large allocation fails, for every n until all succeed.
// Ends with status 0 and a line per part, or is ended by the runtime.
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <atomic>
#include <new>
#include <random>
#include <string>
#include <vector>

#include "../include/asp_b200_host.h"
#include "../alphasparse_b200/csrc/tiled.h"

static std::atomic<bool> in_regions{false};
static std::atomic<long> countdown{-1}, refused{0};

void *operator new(size_t n)
{
    bool no = in_regions && asp::host::in_piece();
    if (countdown >= 0 && n >= 4096 && countdown-- == 0) no = true;
    if (no) refused++;
    void *p = no ? nullptr : malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }

static const uint64_t kRows = 60000, kLen = 64, kCols = 1000000;
static std::vector<float> val;
static std::vector<uint32_t> col;
static std::vector<int64_t> ptr;

static bool layout()
{
    asp::KArgs a;
    memset(&a, 0, sizeof a);
    a.n_units = a.effective = kRows;
    a.row_add = 1;
    std::vector<asp::HostMeta> m(asp::MS_COUNT);
    for (int s : {(int)asp::MS_ROW_OF_UNIT, (int)asp::MS_WARP_NZ})
    {
        m[s].kind = ASP_COMPRESS_LINEAR;
        m[s].coef = s == asp::MS_WARP_NZ ? kLen : 1;
        m[s].present = true;
    }
    asp::HostMeta perm;
    asp::TiledSource t;
    t.templ = ASP_DIRECT_ATOM_TOTAL_WARP_REDUCE_TEMPLATE;
    t.m = m.data();
    t.perm = &perm;
    t.a = &a;
    t.val = val.data();
    t.col = col.data();
    t.stored = t.true_nnz = kRows * kLen;
    t.threads = 128;
    asp::TiledHost out;
    return asp::tiled_build({t}, false, kRows, kCols, 148, out);
}

static bool graph(const char *spec) noexcept // (a C interface throws nothing)
{
    asp_matrix *m = nullptr;
    asp_format *f = nullptr;
    if (asp_matrix_view_csr(kRows, kCols, ptr.data(), col.data(), val.data(), ASP_F32, &m) != ASP_OK) return false;
    const asp_status st = asp_graph_execute(m, spec, &f);
    asp_format_destroy(f);
    asp_matrix_destroy(m);
    return st == ASP_OK || (st != ASP_ERR_ALLOC && !refused); // (a graph may not suit the matrix)
}

static bool validate() noexcept
{
    static asp_format *f = nullptr;
    static std::vector<asp_plan_desc> many; // (so that the call's own tables are large allocations)
    if (!f)
    {
        asp_matrix *m = nullptr;
        const long n = countdown.exchange(-1);
        if (asp_matrix_view_csr(kRows, kCols, ptr.data(), col.data(), val.data(), ASP_F32, &m) != ASP_OK) return false;
        if (asp_graph_execute(m, "dense compress\nsub all row_padding 32 1\nsub all tlb_row\nsub all template K3", &f) != ASP_OK) return false;
        asp_matrix_destroy(m);
        many.resize(200);
        for (asp_plan_desc &d : many)
            if (asp_format_plan_descs(f, &d) != ASP_OK) return false;
        countdown = n;
    }
    return asp_plan_descs_validate(many.data(), (int)many.size()) == ASP_OK;
}

int main(int argc, char **argv)
{
    const std::string part = argc > 2 ? argv[2] : "";
    std::mt19937 rng(1);
    val.resize(kRows * kLen);
    col.resize(kRows * kLen);
    for (uint64_t r = 0; r <= kRows; r++) ptr.push_back((int64_t)(r * kLen));
    for (size_t i = 0; i < val.size(); i++)
    {
        val[i] = (float)rng() / 4e9f;
        col[i] = (uint32_t)(i % kLen * (kCols / kLen) + rng() % (kCols / kLen));
    }
    auto run = [&](const char *what, auto &&f) {
        if (part != what) return;
        if (std::string(argv[1]) == "region")
        {
            in_regions = true;
            const bool ok = f();
            in_regions = false;
            printf("%s %s, %ld refused\n", what, ok ? "built" : "failed", refused.load());
            if (!ok || refused) exit(2);
            return;
        }
        long n = 0;
        for (;; n++)
        {
            countdown = n;
            refused = 0;
            bool ok = false;
            try
            {
                ok = f();
            }
            catch (const std::bad_alloc &)
            {
            }
            countdown = -1;
            if (refused == 0)
            {
                if (!ok) exit(3);
                break;
            }
        }
        printf("%s built after %ld failures\n", what, n);
    };
    run("layout", layout);
    run("validate", validate);
    run("K2", [] { return graph("dense compress\nsub all row_padding 32 1\nsub all blb_row_evenly 32\nsub all tlb_row\nsub all template K2"); });
    run("K6", [] { return graph("dense sort 1\ndense compress\nsub all row_padding 32 1\nsub all blb_row_evenly 32\nsub all tlb_col_fixed 4\nsub all template K6"); });
    run("K9", [] { return graph("dense compress\nsub all tlb_nnz 16\nsub all template K9"); });
    run("B1", [] { return graph("dense compress\nsub all block_value 2 2\nsub all template B1"); });
    run("D1", [] { return graph("dense compress\nsub all diag_value 64\nsub all template D1"); });
    return 0;
}

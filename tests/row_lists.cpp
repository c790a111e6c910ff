// Lists of rows as the host makes them, without a GPU. Argument: the part to check. Ends with status 0 where it holds.
#include <stdio.h>
#include <string.h>

#include <string>
#include <vector>

#include "../alphasparse_b200/csrc/row_lists.h"

static asp::HostMeta linear(uint64_t coef)
{
    asp::HostMeta h;
    h.present = true;
    h.kind = ASP_COMPRESS_LINEAR;
    h.coef = coef;
    return h;
}

// `rows` rows of `per` elements one after the other, a chunk (of a warp or, `cta`, of a CTA) each
static asp::OwnRows chunks(uint64_t n_rows, uint64_t rows, uint64_t per, bool f64 = false, bool cta = false)
{
    asp_plan_desc d;
    memset(&d, 0, sizeof d);
    d.template_type = cta ? ASP_SHARED_MEMORY_LONG_ROW_TEMPLATE : ASP_DIRECT_ATOM_TOTAL_WARP_REDUCE_TEMPLATE;
    d.val_dtype = f64 ? ASP_F64 : ASP_F32;
    d.n_rows = n_rows;
    std::vector<asp::HostMeta> m(asp::MS_COUNT);
    m[asp::MS_ROW_OF_UNIT] = linear(1);
    m[cta ? asp::MS_BLK_NZ : asp::MS_WARP_NZ] = linear(per);
    asp::KArgs a;
    memset(&a, 0, sizeof a);
    a.n_units = a.effective = rows;
    asp::OwnRows o;
    o.make(d, m, asp::HostMeta(), a, rows * per, 148);
    return o;
}
static bool listed(const asp::OwnRows &o, uint64_t rows) { return o.bytes() == 8 * (rows + 1) && o.listed == rows; }

// As many elements as both kernels were measured with, and no more.
static int limits()
{
    if (!listed(chunks(1000, 1000, 512), 1000) || !listed(chunks(1000, 1000, 16384), 1000) || chunks(1000, 1000, 16385).bytes() != 0) return 1;
    if (!listed(chunks(1 << 18, 1 << 18, 512), 1 << 18) || chunks((1 << 18) + 1, (1 << 18) + 1, 512).bytes() != 0) return 2;
    if (chunks((1u << 27) + 1, (1u << 27) + 1, 1).bytes() != 0) return 3; // (a warp each: their threads would pass 32 bits)
    if (!listed(chunks(2048, 2048, 2048, true, true), 2048) || chunks(2049, 2049, 2048, true, true).bytes() != 0) return 4;
    if (!listed(chunks(1 << 16, 1 << 16, 2048, false, true), 1 << 16) || chunks((1 << 16) + 1, (1 << 16) + 1, 2048, false, true).bytes() != 0) return 5;
    if (!listed(chunks(128, 128, 8192, true, true), 128) || chunks(129, 129, 8192, true, true).bytes() != 0) return 6;
    if (!listed(chunks(2048, 2048, 8192, false, true), 2048) || chunks(2049, 2049, 8192, false, true).bytes() != 0) return 7;
    return 0;
}

// What a list takes on the host goes with the rows that are in it, not with those of the matrix.
static long peak() // KB of address space
{
    long kb = -1;
    char line[256];
    FILE *f = fopen("/proc/self/status", "r");
    while (f && fgets(line, sizeof line, f)) sscanf(line, "VmPeak: %ld", &kb);
    if (f) fclose(f);
    return kb;
}
static int empty()
{
    const long before = peak();
    if (!listed(chunks(4000000000ull, 5, 3), 5)) return 1;
    if (chunks(100, 50, 0).bytes() != 0) return 2; // more rows than elements
    return peak() - before > 200000 ? 3 : 0;
}

int main(int, char **argv)
{
    const std::string part = argv[1];
    const int r = part == "limits" ? limits() : part == "empty" ? empty() : -1;
    printf("%s: %d\n", part.c_str(), r);
    return r;
}

// The column-tiled layout as the host builds it, without a GPU. Argument: the part to check. Ends with status 0 where it holds.
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <vector>

#include "../include/asp_b200_host.h"
#include "../alphasparse_b200/csrc/tiled.h"

// Row entries of units are found with 32 bits: the most that a matrix may have, and one more.
static int fit()
{
    const uint64_t n = 4000000000ull, tiles = 1500, room = (1ull << 32) - n / asp::kTiledUnit - 2 * tiles - asp::kTiledUnit;
    if (!asp::tiled_units_fit(room - 1, n, tiles) || asp::tiled_units_fit(room, n, tiles)) return 1;
    if (asp::tiled_units_fit(1ull << 32, 1ull << 33, 1) || asp::tiled_units_fit(3ull << 32, 5ull << 34, 65000)) return 2; // (no wrap of its own)
    // 60 million rows of 80 elements, an element a row and tile: below what the layout's other limits refuse
    if (asp::tiled_units_fit(4800000000ull, 4800000000ull, 1500)) return 3;
    // entries that a unit can have: one for each of its elements
    if (!asp::tiled_units_fit(8000000, 16000000, 25)) return 4;
    return 0;
}

// A matrix in the row-per-unit format, its rows in the order `order`.
struct Rows
{
    std::vector<float> val;
    std::vector<uint32_t> col, order;
    std::vector<uint64_t> begin{0};
    uint64_t cols = 0;
    void add(uint32_t row) { order.push_back(row), begin.push_back(col.size()); }
    bool build(asp::TiledHost &out) const
    {
        asp::KArgs a;
        memset(&a, 0, sizeof a);
        a.n_units = a.effective = order.size();
        std::vector<asp::HostMeta> m(asp::MS_COUNT);
        auto array = [](asp::HostMeta &h, const void *p, int dtype, uint64_t n) {
            h.present = true;
            h.kind = ASP_COMPRESS_NONE;
            h.p = p;
            h.dtype = dtype;
            h.len = n;
        };
        array(m[asp::MS_ROW_OF_UNIT], order.data(), ASP_U32, order.size());
        array(m[asp::MS_WARP_NZ], begin.data(), ASP_U64, begin.size());
        asp::HostMeta perm;
        asp::TiledSource t;
        t.templ = ASP_DIRECT_ATOM_TOTAL_WARP_REDUCE_TEMPLATE;
        t.m = m.data();
        t.perm = &perm;
        t.a = &a;
        t.val = val.data();
        t.col = col.data();
        t.stored = t.true_nnz = col.size();
        t.threads = 128;
        return asp::tiled_build({t}, false, order.size(), cols, 148, out);
    }
};

// Units or slices is the matrix's and nobody else's: runs of exactly the length and with exactly the share of near ones that units may
// have, then one element, or one run that is not near, too many. Rows in groups of four that lie side by side, the groups far apart.
static int choice(int seed)
{
    const uint32_t rows = 60000, tiles = 25, run = 7, tile = asp::tiled_tile_cols(false);
    for (int over = 0; over < 3; over++)
    {
        Rows m;
        m.cols = (uint64_t)tiles * tile;
        srand(seed);
        for (uint32_t i = 0; i < rows; i++)
        {
            uint32_t r = i / 4 * 7919 % (rows / 4) * 4 + i % 4;
            if (over == 2 && i / 4 == 5) r = r / 4 * 4 + i * 2 % 4 + i % 4 / 2; // 0, 2, 1, 3: one more step back
            for (uint32_t t = 0; t < tiles; t++)
                for (uint32_t k = 0; k < run + (over == 1 && i == 777 && t == 3 ? 1 : 0); k++) m.col.push_back(t * tile + (uint32_t)rand() % (tile / 8) + k * (tile / 8)), m.val.push_back(1);
            m.add(r);
        }
        asp::TiledHost out;
        if (!m.build(out)) return 10 + over;
        if ((out.units > 0) != (over == 0)) return 20 + over;
    }
    return 0;
}

int main(int argc, char **argv)
{
    const char *part = argc > 1 ? argv[1] : "";
    int r = 99;
    if (!strcmp(part, "fit")) r = fit();
    if (!strcmp(part, "choice")) r = choice(argc > 2 ? atoi(argv[2]) : 1);
    printf("%s %d\n", part, r);
    return r;
}

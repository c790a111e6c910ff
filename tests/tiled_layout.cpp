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
    bool build(asp::TiledHost &out, bool f64 = false) const
    {
        const std::vector<double> val64(val.begin(), f64 ? val.end() : val.begin());
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
        t.val = f64 ? (const void *)val64.data() : val.data();
        t.col = col.data();
        t.stored = t.true_nnz = col.size();
        t.threads = 128;
        return asp::tiled_build({t}, f64, order.size(), cols, 148, out);
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

// Units, followed as the kernel does, against the sums of the matrix: rows added up in y ("y"), all as sums ("sums"), or some each way
// ("both", which takes rows enough for clearing y to be less than their sums). Every element once, in a place of its own tile.
static int units(const char *mode)
{
    const bool y_only = !strcmp(mode, "y"), both = !strcmp(mode, "both");
    const uint32_t rows = both ? 700001 : y_only ? 500000 : 60000, tiles = both || y_only ? 8 : 25, tile = asp::tiled_tile_cols(false);
    Rows m;
    m.cols = (uint64_t)tiles * tile - 77;
    srand(5);
    std::vector<double> x(m.cols), want(rows, 0.0), got(rows, 0.0);
    for (double &v : x) v = rand() % 19 - 9;
    for (uint32_t r = 0; r < rows; r++)
    {
        uint32_t n = both ? 10 + rand() % 8 : y_only ? 8 : 50;
        if (r == 0 || r == rows - 1 || r == rows / 3) n = both ? 9000 : y_only ? 8 : 700; // (over many units and lanes; more parts than y takes)
        if (r % 1000 == 5) n = 0;
        for (uint32_t k = 0; k < n; k++)
        {
            const uint64_t c = (uint64_t)k * m.cols / n + rand() % (m.cols / n);
            m.col.push_back((uint32_t)c);
            m.val.push_back((float)(1 + rand() % 9));
            want[r] += m.val.back() * x[c];
        }
        m.add(r);
    }
    asp::TiledHost out;
    if (!m.build(out)) return 10;
    if (out.units == 0 || out.copies != 1 || out.nnz != m.col.size() || out.covers_all_rows) return 11;
    if (out.direct != (both || y_only) || (out.n_parts > 0) != !y_only || out.parts.empty() == both) return 12;
    if (both && out.n_parts != 3) return 13;
    if (out.seg.n != out.units + asp::kTiledSlackUnits) return 14;
    // the tile of every unit, from the work: every unit is one warp's, and a CTA's warps share a tile
    const uint32_t W = asp::kTiledUnitWarps;
    std::vector<int> tile_of(out.units, -1);
    for (uint32_t cta = 0; cta < 148; cta++)
        for (uint64_t visit = cta, first = 1; first || visit != 0; first = 0)
        {
            const uint32_t *o = &out.work[visit * W * 4], t = o[2], next = o[3];
            for (uint32_t w = 0; w < W; w++, o += 4)
            {
                if (o[0] > o[1] || o[1] > out.units || o[2] != t || o[3] != next) return 15;
                for (uint32_t u = o[0]; u < o[1]; u++)
                {
                    if (tile_of[u] >= 0) return 16;
                    tile_of[u] = (int)t;
                }
            }
            visit = next;
        }
    const float *val = (const float *)out.val.p;
    std::vector<double> sum(out.n_parts, 0.0);
    uint64_t elements = 0;
    for (uint64_t u = 0; u < out.units; u++)
    {
        if (tile_of[u] < 0) return 17;
        uint32_t row = 0, begun = 0;
        for (uint64_t i = 0; i < asp::kTiledUnit; i++)
        {
            const uint64_t q = u * asp::kTiledUnit + i;
            const uint32_t word = out.word.p[u * 32 + i / asp::kTiledLane], k = i % asp::kTiledLane;
            if (k == 0 && word >> 16 != begun) return 18;
            if (word >> k & 1)
            {
                row = out.row.p[out.seg.p[u] + begun];
                begun++;
            }
            else if (i == 0) return 19;
            if (out.col.p[q] == tile) // what fills a tile's last unit
            {
                if (val[asp::unit_val_at(q)] != 0) return 20;
                continue;
            }
            const uint64_t c = (uint64_t)tile_of[u] * tile + out.col.p[q];
            if (out.col.p[q] > tile || c >= m.cols) return 21;
            elements++;
            const bool in_parts = row & asp::kTiledInParts || (out.n_parts > 0 && !out.direct);
            const uint32_t to = row & ~asp::kTiledInParts;
            if (to >= (in_parts ? out.n_parts : rows)) return 22;
            (in_parts ? sum : got)[to] += val[asp::unit_val_at(q)] * x[c];
        }
        if (begun != out.seg.p[u + 1] - out.seg.p[u]) return 23;
    }
    if (elements != m.col.size()) return 24;
    for (uint64_t k = 0; k < out.n_parts; k++) got[out.parts.empty() ? k : out.parts[k]] += sum[k];
    return got == want ? 0 : 25; // (whole numbers: exact)
}

// fp64: 16 warps where half of all elements are in pieces of 14 and more, else 32. Every step is one warp's, in a visit of its CTA.
static int warps()
{
    const uint32_t rows = 200000, tiles = 10, tile = asp::tiled_tile_cols(true);
    for (uint32_t few = 0; few < 4; few++)
    {
        Rows m;
        m.cols = (uint64_t)tiles * tile;
        srand(3);
        // rows of one piece: all of 13, all of 14, and as many of 26 as of 13 times two, then one fewer
        for (uint32_t r = 0; r < rows; r++)
        {
            const bool deep = few == 1 || (few >= 2 && r % 3 == 0 && !(few == 3 && r == 999));
            const uint32_t n = !deep ? 13 : few == 1 ? 14 : 26, t = (uint32_t)rand() % tiles;
            if (few >= 2 && r == rows - 1 && !deep) continue; // (a multiple of three)
            for (uint32_t k = 0; k < n; k++) m.col.push_back(t * tile + k * (tile / n) + (uint32_t)rand() % (tile / n)), m.val.push_back(1);
            m.add(r);
        }
        asp::TiledHost out;
        if (!m.build(out, true)) return 10 + few;
        if (out.units > 0 || out.copies != 1 || out.warps != (few == 1 || few == 2 ? 16u : 32u)) return 20 + few;
        std::vector<char> taken(out.steps, 0);
        for (uint32_t cta = 0; cta < 148; cta++)
            for (uint64_t visit = cta, first = 1; first || visit != 0; first = 0)
            {
                const uint32_t *o = &out.work[visit * out.warps * 4], t = o[3];
                for (uint32_t w = 0; w < out.warps; w++, o += 4)
                {
                    if (o[0] > o[1] || o[1] > out.steps || o[3] != t) return 30 + few;
                    for (uint32_t s = o[0]; s < o[1]; s++)
                        if (taken[s]++) return 40 + few;
                    // the slice that the warp begins in
                    if (o[0] < o[1] && (o[0] >= out.end.p[o[2]] || (o[2] > 0 && o[0] < out.end.p[o[2] - 1]))) return 50 + few;
                }
                visit = t >> 16;
            }
        for (char c : taken)
            if (!c) return 60 + few;
    }
    return 0;
}

int main(int argc, char **argv)
{
    const char *part = argc > 1 ? argv[1] : "";
    int r = 99;
    if (!strcmp(part, "fit")) r = fit();
    if (!strcmp(part, "choice")) r = choice(argc > 2 ? atoi(argv[2]) : 1);
    if (!strcmp(part, "warps")) r = warps();
    if (!strcmp(part, "units")) r = units(argc > 2 ? argv[2] : "");
    printf("%s %d\n", part, r);
    return r;
}

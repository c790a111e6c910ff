// The column-tiled layout as the host builds it, without a GPU. Argument: the part to check. Ends with status 0 where it holds.
#include <stdio.h>
#include <string.h>

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

int main(int argc, char **argv)
{
    const char *part = argc > 1 ? argv[1] : "";
    int r = 99;
    if (!strcmp(part, "fit")) r = fit();
    printf("%s %d\n", part, r);
    return r;
}

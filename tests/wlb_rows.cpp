// Which loop sep_thread_level_col_ell_with_padding shares out among the threads. Ends with status 0 where it is the right one.
#include "../alphasparse_b200/csrc/host/format.hpp"

using namespace asp::host;

int main()
{
    auto by_rows = [](std::vector<u64> rows, u64 per_row) {
        std::vector<u64> nnz;
        for (u64 r : rows) nnz.push_back(r * per_row);
        return shares_rows_of_wlbs(rows, nnz, 4, 16);
    };
    if (!by_rows({500000}, 5)) return 1;                           // one over the whole matrix
    if (by_rows(std::vector<u64>(70, 128), 20)) return 2;          // rows too few to be shared out
    if (by_rows(std::vector<u64>(200, 3000), 20)) return 3;        // all alike
    std::vector<u64> one(60, 170);
    one[37] = 390000;
    if (!by_rows(one, 8)) return 4;                                // one that holds nearly everything: all but one thread would wait
    if (!by_rows({400000, 300000, 350000, 10}, 8)) return 5;       // fewer than the threads
    std::vector<u64> some(100, 7000);
    some[0] = 30000;
    if (by_rows(some, 8)) return 6;                                // a large one, but more in all the others, which nobody would share
    if (by_rows(std::vector<u64>(60, 1), 2000000)) return 8;       // a row each: nothing to share inside
    if (!by_rows({7}, 3) || !by_rows({}, 1)) return 7;             // nothing to share
    return 0;
}

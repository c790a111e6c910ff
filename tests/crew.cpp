// Loops shared among a caller and helpers (csrc/host/crew.hpp). Argument: the part to check. Ends with status 0 where it holds.
#include <omp.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <sys/wait.h>
#include <unistd.h>

#include <thread>
#include <vector>

#include "../alphasparse_b200/csrc/host/crew.cpp"

using namespace asp::host;

// every index once, no two threads with one number at a time
static bool covers(uint64_t n, unsigned width, uint64_t step)
{
    std::vector<std::atomic<int>> hit(n);
    std::vector<std::atomic<int>> busy(width);
    std::atomic<bool> ok(true);
    for (auto &h : hit) h.store(0);
    for (auto &b : busy) b.store(0);
    share_steps(n, step, width, [&](uint64_t i, uint64_t e, unsigned who) {
        if (who >= width || busy[who].fetch_add(1) != 0) ok = false;
        for (; i < e; i++) hit[i]++;
        busy[who].fetch_sub(1);
    });
    for (auto &h : hit) ok = ok && h.load() == 1;
    for (auto &h : hit) h.store(0);
    share_ranges(n, width > 1, [&](uint64_t i, uint64_t e) {
        for (; i < e; i++) hit[i]++;
    });
    for (auto &h : hit) ok = ok && h.load() == 1;
    std::vector<uint64_t> plain(n); // written by whoever, read here: ordered by the loop's end
    for_each(n, width > 1, [&](uint64_t i) { plain[i] = i * 3; });
    for (uint64_t i = 0; i < n; i++) ok = ok && plain[i] == i * 3;
    return ok;
}

static int cover()
{
    for (int t : {1, 2, 3, 8, 40, 300})
    {
        omp_set_num_threads(t);
        for (uint64_t n : {0, 1, 2, 7, 63, 64, 65, 255, 256, 257, 1000, 20011})
            for (uint64_t step : {1, 7, 4096})
                if (!covers(n, crew_width(), step)) return 1;
    }
    return 0;
}

// more callers than there are slots, over and over, with loops inside of pieces
static int callers()
{
    std::atomic<int> bad(0);
    std::vector<std::thread> all;
    for (int k = 0; k < 12; k++)
        all.emplace_back([&, k] {
            omp_set_num_threads(2 + k % 5);
            for (int it = 0; it < 300; it++)
            {
                const Caller caller;
                if (!covers(1 + (uint64_t)(it * 37 + k * 101) % 3000, crew_width(), 1 + it % 50)) bad++;
                std::atomic<uint64_t> sum(0);
                for_each(50, true, [&](uint64_t i) {
                    if (crew_width() != 1 && in_piece()) bad++;
                    for_each(100, true, [&](uint64_t j) { sum += i * j; });
                });
                if (sum != 1225ull * 4950) bad++;
            }
        });
    for (auto &t : all) t.join();
    return bad ? 2 : 0;
}

// A loop ends although every helper is held up in somebody else's: the caller does it by itself.
static int held()
{
    omp_set_num_threads(4);
    std::atomic<bool> go(false), held(false);
    std::atomic<int> in(0);
    std::thread other([&] {
        omp_set_num_threads(4);
        share_pieces(4, 4, [&](unsigned, unsigned) {
            in++;
            for (long i = 0; !go && i < 2000000000; i++) std::this_thread::yield();
            if (!go) held = true; // gave up
        });
    });
    while (in == 0) std::this_thread::yield();
    std::atomic<int> done(0);
    for (int it = 0; it < 50; it++) share_pieces(8, 4, [&](unsigned, unsigned) { done++; });
    const bool before = !go && !held;
    go = true;
    other.join();
    return before && done == 400 ? 0 : 3;
}

static int forked()
{
    omp_set_num_threads(4);
    for (int depth = 0; depth < 3; depth++)
    {
        if (!covers(5000, crew_width(), 16)) return 4;
        const pid_t p = fork();
        if (p < 0) return 5;
        if (p > 0)
        {
            int st = 0;
            for (int i = 0; i < 600; i++)
            {
                if (waitpid(p, &st, WNOHANG) == p) return WIFEXITED(st) ? WEXITSTATUS(st) : 6;
                usleep(50000);
            }
            return 7; // (ended by the test)
        }
    }
    _exit(covers(5000, crew_width(), 16) ? 0 : 8);
}

// inside of a region of the program's own OpenMP, loops are the calling thread's
static int region()
{
    std::atomic<int> bad(0);
#pragma omp parallel num_threads(4)
    {
        if (omp_get_num_threads() > 1 && crew_width() != 1) bad++;
        if (!covers(3000, 1, 5)) bad++;
    }
    omp_set_num_threads(1);
    return bad || crew_width() != 1 ? 9 : 0;
}

int main(int, char **argv)
{
    int r = 99;
    if (!strcmp(argv[1], "cover")) r = cover();
    if (!strcmp(argv[1], "callers")) r = callers();
    if (!strcmp(argv[1], "held")) r = held();
    if (!strcmp(argv[1], "forked")) r = forked();
    if (!strcmp(argv[1], "region")) r = region();
    return r;
}

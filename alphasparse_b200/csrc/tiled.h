// Column-tiled execution layout of a whole plan group (see kernels_tiled.cu for what it is for): built on the host
// from the template arrays at plan creation, read by one kernel that replaces the group's own kernels.
#ifndef ASP_TILED_H
#define ASP_TILED_H

#include <cuda_runtime.h>
#include <stdint.h>

#include <memory>
#include <vector>

#include "host/hostmem.hpp"
#include "host_meta.h"
#include "kernel_args.h"

namespace asp
{
constexpr uint32_t kTiledWarps = 32, kTiledFewWarps = 16; // warps per CTA, one CTA per SM: which of the two say kFewWarpsMost and kDeep (tiled_build.cpp)
const uint32_t kTiledLanePieces = 2;         // pieces of a row per lane
const uint32_t kTiledSlice = 32 * kTiledLanePieces;
// Several plans of fewer non-zeros in all keep their templates' kernels: a row then has the same bits whichever other plans are EMPTY, as before
// there were other kernels. Checks of that kind run on small matrices; for larger ones ASP_LAYOUT_NONE has to be asked for.
const uint64_t kSameBits = 1u << 16;
constexpr uint32_t kTiledTileBytes = 159u << 10; // shared memory of a tile of x
const uint32_t kTiledNoRow = 0xffffffffu;
const uint32_t kTiledInParts = 0x80000000u; // row entry: the rest is a place among the sums of the rows in many parts
// steps and slices the kernel may read past the end (prefetch)
const uint32_t kTiledSlackSteps = 8, kTiledSlackSlices = 2;

constexpr uint32_t kTiledUnitWarps = 16;         // per CTA of the kernel for units
constexpr uint32_t kTiledLane = 8;               // consecutive elements of a lane ...
constexpr uint32_t kTiledUnit = 32 * kTiledLane; // ... and of a warp, which are a unit
constexpr uint32_t kTiledStage = kTiledUnit + 2; // sums of a unit's rows, 8 bytes each, that a warp lays out in the shared memory after the tile
const uint32_t kTiledSlackUnits = 4;             // entries of `seg` that the kernel may read past the end
// Units have an entry per row that they begin, which `seg` finds with 32 bits (a step of slices is 64 elements): whether the offsets, and
// those that the kernel forms behind the last one, stay below 2^32. An entry is a run of a row's elements in a tile, of which there are
// `runs`, or what a unit's or a tile's begin cuts off one.
constexpr bool tiled_units_fit(uint64_t runs, uint64_t elements, uint64_t tiles) { return runs + elements / kTiledUnit + 2 * tiles + kTiledUnit < (1ull << 32); }

// place of element q (unit q / 256, lane q % 256 / 8) among the units' fp32 values: 16 bytes of a lane side by side (its columns are 16 bytes)
constexpr uint64_t unit_val_at(uint64_t q) { return q - q % kTiledUnit + (q % kTiledLane / 4 * 32 + q % kTiledUnit / kTiledLane) * 4 + q % 4; }

// columns of a tile; the shared memory after them holds one zero, which what pads a slice multiplies (never an infinite x)
constexpr uint32_t tiled_tile_cols(bool f64) { return kTiledTileBytes / (f64 ? 8u : 4u) - 32u; }

// one sub-matrix of the group, as its template stores it (host arrays)
struct TiledSource
{
    int templ = 0;
    const HostMeta *m = nullptr; // MS_COUNT slots
    const HostMeta *perm = nullptr;
    const KArgs *a = nullptr;    // scalars of the plan
    const void *val = nullptr, *col = nullptr;
    int col_bytes = 4;
    uint64_t stored = 0; // padded non-zeros
    uint64_t true_nnz = 0;
    unsigned threads = 0; // of a CTA of the template's own kernel
    bool whole_rows = false; // runs the kernels that take whole rows (kernels_rows.cu), in so many trips of a warp:
    uint64_t trips = 0;
};

template <class T>
struct HostBuf
{
    std::shared_ptr<void> s;
    T *p = nullptr;
    uint64_t n = 0;
    void make(uint64_t count) { s = host::big_buffer(count * sizeof(T)), p = (T *)s.get(), n = count; }
    uint64_t bytes() const { return n * sizeof(T); }
};

struct TiledHost
{
    HostBuf<unsigned char> val; // step s, lane l, piece g: value s * 64 + 2 l + g
    HostBuf<uint16_t> col;      // same order, column inside the tile
    HostBuf<uint32_t> row;      // slice s, lane l, piece g: row of y, or kTiledInParts | place (kTiledNoRow: none)
    uint64_t n_parts = 0;        // rows of y that are added up in many parts ...
    std::vector<uint32_t> parts; // ... which these are; empty: all
    HostBuf<uint32_t> end;      // slice s covers steps [end[s - 1], end[s])
    unsigned warps = kTiledWarps;
    std::vector<uint32_t> work; // {first step, end step, slice, tile | next visit << 16} per warp; visit v at v * warps
    uint64_t nnz = 0, steps = 0, slices = 0;
    // units > 0: units instead of slices. Then val and col hold them one after the other, in each the first 16 bytes of every lane, the
    // next 16 bytes of every lane, ...; row[seg[u], seg[u + 1]) are the rows of unit u; work: {first unit, end unit, tile, next visit (0: none)},
    // visit v at v * kTiledUnitWarps
    uint64_t units = 0;
    HostBuf<uint32_t> word; // unit u, lane l: bit k: its k-th element starts a row; from bit 16: rows that start in the lanes before
    HostBuf<uint32_t> seg;
    unsigned copies = 1; // sums of a row, which tiles and warps take in turn: 1, 2, 4, 8 or 16
    bool covers_all_rows = false; // every row of y has at least one element
    bool direct = false;          // some are added up in y itself
};

// false: the group stays with its own kernels
bool tiled_build(const std::vector<TiledSource> &src, bool f64, uint64_t n_rows, uint64_t n_cols, int n_sm, TiledHost &out);

struct TiledArgs
{
    const void *val;
    const uint16_t *col;
    const uint32_t *row, *end;  // slices
    const uint32_t *word, *seg; // units (word: NULL where there are slices)
    const uint4 *work;
    const uint32_t *parts; // n_parts rows (NULL: all rows of y) ...
    double *sum;           // ... and their sums, copies * sum_stride of them, zero between the calls
    unsigned n_parts, copies;
    unsigned long long sum_stride;
    int direct; // y takes other rows' sums: it is cleared first
    unsigned warps; // slices: of a CTA
    const void *x;
    void *y;
    unsigned long long n_rows, n_cols;
};
cudaError_t tiled_setup(int val_is_f64);
// y = A x in up to three launches: y cleared, everything added up, the rows in many parts stored by launch_tiled_rows (n_parts > 0),
// which has to run before the next call's
cudaError_t launch_tiled_sums(int val_is_f64, const TiledArgs &a, unsigned n_sm, cudaStream_t st);
cudaError_t launch_tiled_rows(int val_is_f64, const TiledArgs &a, unsigned n_sm, cudaStream_t st);
} // namespace asp
#endif

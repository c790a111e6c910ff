// Lists of the rows of small plans, as the kernels of kernels_rows.cu take them.
#ifndef ASP_ROW_LISTS_H
#define ASP_ROW_LISTS_H

#include <vector>

#include "host_meta.h"
#include "kernels.h"
#include "tiled.h"

namespace asp
{
const uint64_t kMostSeen = 1u << 26; // rows of a matrix, where which of them have come is kept (8 MB)

// Whole rows for a few lanes, a warp or a CTA, where that is the faster way (kernels_rows.cu). A warp takes up to 512 elements (four trips
// of 1.2 us; chunks in parallel are faster beyond that), a CTA rows of 256 and more on average, up to 16384 (four trips of 1024 threads).
// Rows that are TLBs of more than 8 elements: up to 3 M elements (what L2 holds). CSR5-like: up to 512 K elements (FEM, fp32: 445 K 6 -> 3.1 us, 730 K
// 6.5 -> 5.1, but lists of a million elements cost more to make than that is worth) and rows of 4096 (four trips of a CTA).
// Rows of TLBs: up to 2 M elements, beyond which the CTA's long strips stream better (4.9 M, FEM, fp32: 13.0 us, 17.3 by rows; 1.6 M: 7.2, 5.1).
struct OwnRows
{
    RowArgs args = {};
    HostBuf<uint2> rows; // (one of the two)
    HostBuf<uint4> tlbs;
    HostBuf<unsigned> place;
    uint64_t trips = 0;  // of warps that take a row
    uint64_t listed = 0; // rows of y
    bool strips = false, runs = false; // (in `tlbs`)
    const void *data() const { return tlbs.n == 0 ? (const void *)rows.p : tlbs.p; }
    size_t bytes() const { return rows.bytes() + tlbs.bytes(); }
    void none()
    {
        rows = {};
        tlbs = {};
        place = {};
    }
    // f(row of y) for all of them
    template <class F>
    void each_row(F &&f) const
    {
        for (uint64_t i = 0; i + 1 < rows.n; i++) f(rows.p[i].y);
        for (uint64_t i = 0; i < tlbs.n; i++)
            if (!strips) f(tlbs.p[i].y);
            else if (place.n == 0)
                for (unsigned k = 0; k < tlbs.p[i].z >> 16; k++) f(args.first_row + tlbs.p[i].y + k);
        for (uint64_t i = 0; i < place.n; i++) f(place.p[i]);
    }
    // Device memory that the list of a small plan may take, about: 0 where it can have none. (What does not fit gets a block of its own.) Before anything is known of
    // its arrays' contents: no more rows than elements are listed.
    static size_t room(const asp_plan_desc &d, const std::vector<HostMeta> &hm, uint64_t stored);
    // of a (validated) plan whose values are `stored` ones. few: one of several sub-matrices, which a kernel each takes one after the other
    void make(const asp_plan_desc &d, const std::vector<HostMeta> &hm, const HostMeta &perm, const KArgs &a, uint64_t stored, int sm_count, bool few = false);

  private:
    bool list(const asp_plan_desc &d, const std::vector<HostMeta> &hm, const HostMeta &perm, const KArgs &a, uint64_t stored, int sm_count, bool few);
};
} // namespace asp
#endif

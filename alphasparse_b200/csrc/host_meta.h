// Host-side view of one metadata array of a template, or of the closed form that stands in for it
// (validation, shared-memory sizing, and the walk over a template's elements in tiled_build.cpp).
#ifndef ASP_HOST_META_H
#define ASP_HOST_META_H

#include <stdint.h>

#include "../../include/asp_b200.h"

namespace asp
{
// host copy of a metadata reference, for validation and shared-memory sizing
struct HostMeta
{
    const void *p = nullptr;
    int dtype = ASP_U32;
    uint64_t len = 0;
    int kind = ASP_COMPRESS_NONE;
    uint64_t coef = 0, icpt = 0, cycle = 1;
    int nb = 0;
    uint64_t bhi[5] = {0, 0, 0, 0, 0}, bval[5] = {0, 0, 0, 0, 0};
    bool present = false;
    uint64_t get(uint64_t i) const
    {
        switch (kind)
        {
        case ASP_COMPRESS_NONE:
            switch (dtype)
            {
            case ASP_U8: return ((const uint8_t *)p)[i];
            case ASP_U16: return ((const uint16_t *)p)[i];
            case ASP_U32: return ((const uint32_t *)p)[i];
            default: return ((const uint64_t *)p)[i];
            }
        case ASP_COMPRESS_LINEAR: return i * coef + icpt;
        case ASP_COMPRESS_CONSTANT: return icpt;
        case ASP_COMPRESS_CYCLE_LINEAR: return (i % cycle) * coef + icpt;
        case ASP_COMPRESS_CYCLE_INCREASE: return i / cycle + icpt;
        default:
        {
            uint64_t v = bval[0];
            for (int b = 1; b < nb; b++)
                if (i > bhi[b - 1]) v = bval[b];
            return v;
        }
        }
    }
};
// a closed form, or an array of at least `count` entries
inline bool has_entries(const HostMeta &h, uint64_t count) { return h.kind != ASP_COMPRESS_NONE || h.len >= count; }
} // namespace asp
#endif

// The search loop with a second timer, for its GPU form.
#ifndef ASP_SEARCH_HPP
#define ASP_SEARCH_HPP
#include "../../../include/asp_b200_host.h"

namespace asp
{
namespace host
{
// Times an SpMV over the whole format by what replaces its templates' kernels (a layout, kernels for whole rows); non-zero when nothing does.
typedef int (*time_layout_fn)(void *user, const asp_format *fmt, int warmup, int reps, float *ms_per_spmv);
// asp_search; what replaces the kernels of every dense view's winner, and of every format of a small matrix, is a candidate of its own where `layout_fn` is not NULL
asp_status search(const asp_matrix *m, const asp_search_options *opt, asp_time_fn time_fn, time_layout_fn layout_fn, void *time_user, asp_search_result **out);
} // namespace host
} // namespace asp
#endif

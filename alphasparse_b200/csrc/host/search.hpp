// The search loop with a second timer, for its GPU form.
#ifndef ASP_SEARCH_HPP
#define ASP_SEARCH_HPP
#include "../../../include/asp_b200_host.h"

namespace asp
{
namespace host
{
// Times an SpMV over the whole format in a layout that replaces its templates' kernels; non-zero when there is none for it.
typedef int (*time_layout_fn)(void *user, const asp_format *fmt, int warmup, int reps, float *ms_per_spmv);
// asp_search; the layout of every dense view's winner is a candidate of its own where `layout_fn` is not NULL
asp_status search(const asp_matrix *m, const asp_search_options *opt, asp_time_fn time_fn, time_layout_fn layout_fn, void *time_user, asp_search_result **out);
} // namespace host
} // namespace asp
#endif

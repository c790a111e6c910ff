// asp_search with the GPU as the timer: a trial's format is uploaded once, its launch parameters are
// swept in place, and asp_time measures it (replaces the reference's emit + nvcc + run per trial).
// Trials run the templates' kernels, whole matrices as well as one strip with the others EMPTY. What takes no launch parameters is a candidate of its
// own: the column-tiled layout, which is the same for every template, and kernels for whole rows once per dense view, on the winners' format; whole rows
// of a small matrix in one piece, which are not the same for every template, once per format too.
//
// Launch requests that the kernels fold into the same effective launch (a CTA width above a family's compiled
// bound becomes more CTAs, grids are cut to the CTAs that have work: asp_plan_get_launch) are timed once: a
// sweep over thread_num_in_block often asks for the same kernel launch several times, and the reference, which
// prints the request into a new program each time, cannot know.
#include <stdio.h>

#include <map>
#include <vector>

#include "../../include/asp_b200.h"
#include "../../include/asp_b200_host.h"
#include "host/search.hpp"

namespace
{
struct GpuTimer
{
    asp_ctx *ctx;
    uint64_t cached = 0; // asp_format_id of the uploaded format
    std::vector<asp_plan *> plans;
    std::map<std::vector<int64_t>, float> timed; // effective launch of every plan -> ms, for the uploaded format
    uint64_t reused = 0, measured = 0;

    void drop()
    {
        for (asp_plan *p : plans)
            if (p) asp_plan_destroy(p);
        plans.clear();
        timed.clear();
        cached = 0;
    }
    ~GpuTimer() { drop(); }
};

int time_on_gpu(void *user, const asp_format *fmt, const int64_t *tblock, const int64_t *threads, const int64_t *reduce, int warmup, int reps, float *ms)
{
    GpuTimer *t = static_cast<GpuTimer *>(user);
    const int n = asp_format_num_subs(fmt);
    if (n <= 0) return 1;
    if (t->cached != asp_format_id(fmt))
    {
        t->drop();
        std::vector<asp_plan_desc> descs(n);
        if (asp_format_plan_descs(fmt, descs.data()) != ASP_OK) return 1;
        t->plans.assign(n, nullptr);
        if (asp_plan_group_create_with(t->ctx, descs.data(), n, ASP_LAYOUT_NONE, t->plans.data()) != ASP_OK)
        {
            t->plans.clear();
            return 1;
        }
        t->cached = asp_format_id(fmt);
    }
    std::vector<asp_plan_desc> descs(n);
    if (asp_format_plan_descs(fmt, descs.data()) != ASP_OK) return 1;
    for (int i = 0; i < n; i++)
    {
        if (descs[i].template_type == ASP_EMPTY_TEMPLATE) continue;
        if (asp_plan_set_launch(t->plans[i], tblock[i], threads[i], reduce[i]) != ASP_OK) return 1;
    }
    // the launches the kernels will actually get
    std::vector<int64_t> key;
    key.push_back(warmup);
    key.push_back(reps);
    for (int i = 0; i < n; i++)
    {
        int64_t g = 0, b = 0, r = 0;
        if (descs[i].template_type != ASP_EMPTY_TEMPLATE && asp_plan_get_launch(t->plans[i], &g, &b, &r) != ASP_OK) return 1;
        key.push_back(g);
        key.push_back(b);
        key.push_back(r);
    }
    auto hit = t->timed.find(key);
    if (hit != t->timed.end())
    {
        *ms = hit->second;
        t->reused++;
        return 0;
    }
    float gflops = 0;
    if (asp_time(t->ctx, t->plans.data(), n, warmup, reps, 2, 0.0, ms, &gflops) != ASP_OK) return 1;
    t->timed[key] = *ms;
    t->measured++;
    return 0;
}

int time_layout_on_gpu(void *user, const asp_format *fmt, int warmup, int reps, float *ms)
{
    GpuTimer *t = static_cast<GpuTimer *>(user);
    t->drop(); // (device memory for the layout)
    const int n = asp_format_num_subs(fmt);
    if (n <= 0) return 1;
    std::vector<asp_plan_desc> descs(n);
    if (asp_format_plan_descs(fmt, descs.data()) != ASP_OK) return 1;
    t->plans.assign(n, nullptr);
    bool ok = asp_plan_group_create_with(t->ctx, descs.data(), n, ASP_LAYOUT_AUTO, t->plans.data()) == ASP_OK;
    const bool layout = ok && asp_plan_layout_bytes(t->plans[0]) > 0;
    bool rows = false;
    for (int i = 0; i < n && ok; i++) rows = rows || asp_plan_whole_rows(t->plans[i]);
    float gflops = 0;
    // (the layout with y cleared: the calls in which it runs whatever rows are empty)
    ok = ok && (layout || rows) && asp_time(t->ctx, t->plans.data(), n, warmup, reps, layout ? 1 : 2, 0.0, ms, &gflops) == ASP_OK;
    t->drop();
    return ok ? 0 : 1;
}
} // namespace

extern "C" asp_status asp_search_gpu(asp_ctx *ctx, const void *matrix, const void *options, void **result)
{
    if (!ctx || !matrix || !result) return ASP_ERR_INVALID_ARG;
    GpuTimer timer{ctx};
    asp_search_result *r = nullptr;
    const asp_search_options *opt = static_cast<const asp_search_options *>(options);
    const asp_status st = asp::host::search(static_cast<const asp_matrix *>(matrix), opt, time_on_gpu, time_layout_on_gpu, &timer, &r);
    if (opt && opt->log_fn)
    {
        char line[160];
        snprintf(line, sizeof line, "timer: %llu launches measured, %llu requests folded into a launch already measured", (unsigned long long)timer.measured,
                 (unsigned long long)timer.reused);
        opt->log_fn(opt->log_user, line);
    }
    *result = r;
    return st;
}

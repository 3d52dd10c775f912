// mpm_batch_step on a CUDA runtime that runs nothing and fails where it is told to: what
// the device's counters would hold is followed from the launches, the graphs and the
// memsets, and no later call may start from what a failed one left behind.
#include "mpm_batch.cu"

#include <cstdio>
#include <functional>

namespace {

int bad = 0;
void expect(bool ok, const char* what) {
    if (!ok) { std::printf("%s\n", what); ++bad; }
}

// The device: the step counter, and whether tiles hold the counts of an unfinished sort.
mpm_batch* live = nullptr;
int counter = 0;
bool counted = false;

const void* fail_kernel = nullptr;  // the launch of this kernel fails
int fail_graph = -1;                // the graph launch with this number fails

void stamp() {
    const size_t rows = live->stamps_cap / (size_t)live->nscenes;
    expect((size_t)counter < rows, "a time stamp past the end of its array");
}

}  // namespace

// What fake_cudart.cpp asks and tells.
bool fake_launch_fails(const void* f) { return f == fail_kernel; }
bool fake_graph_fails() { return fail_graph >= 0 && fail_graph-- == 0; }
void fake_kernel_ran(const void* f) {
    if (f == (const void*)k_batch_grid) { stamp(); ++counter; }
    if (f == (const void*)k_batch_end) { stamp(); counter = 0; }
    if (f == (const void*)k_sort_count<2, 4, ManyScenes>) {
        expect(!counted, "a sort on top of the counts of an unfinished one");
        counted = true;
    }
    if (f == (const void*)k_tile_sort<2, 4, ManyScenes>) counted = false;
}
void fake_cleared(void* p) {
    if (live && p == live->arr.step) counter = 0;
    if (live && p == live->ti.tile_count) counted = false;
}

namespace {

mpm_batch* make() {
    mpm_params p{};
    p.dim = 2;
    p.width = p.height = 32;
    p.border_margin = 2;
    p.formulation = MPM_FORMULATION_MLS;
    p.delta_time = 1e-3f;
    p.nu = 0.2f;
    p.youngs = 1e5f;
    p.rho = 400.f;
    const float pos[4] = {10.f, 10.f, 11.f, 11.f}, vol[2] = {1.f, 1.f};
    const mpm_params params[2] = {p, p};
    mpm_particles_init init[2] = {};
    for (auto& i : init) { i.count = 2; i.position = pos; i.volume = vol; }
    counter = 0;
    counted = false;
    live = nullptr;
    mpm_batch* b = nullptr;
    expect(mpm_batch_create(params, init, 2, &b) == MPM_OK, "create");
    live = b;
    return b;
}

void after_failure(const char* what, mpm_batch* b) {
    fail_kernel = nullptr;
    fail_graph = -1;
    expect(mpm_batch_step(b, 40) == MPM_OK, what);
    expect(counter == 0 && !counted, what);
    mpm_batch_destroy(b);
    live = nullptr;
}

}  // namespace

int main() {
    for (int g = 0; g < 3; ++g) {  // 40 steps: graphs of 16, 16 and 8 steps
        mpm_batch* b = make();
        fail_graph = g;
        expect(mpm_batch_step(b, 40) == MPM_ERR_OUT_OF_MEMORY, "a graph that does not launch");
        after_failure("after a graph that did not launch", b);
    }
    const void* sort[] = {(const void*)k_sort_count<2, 4, ManyScenes>, (const void*)k_sort_block_sums, (const void*)k_sort_scan,
                          (const void*)k_sort_bucket, (const void*)k_tile_sort<2, 4, ManyScenes>};
    for (const void* f : sort) {
        mpm_batch* b = make();
        fail_kernel = f;
        expect(mpm_batch_step(b, 3) == MPM_ERR_OUT_OF_MEMORY, "a sort that does not launch");
        expect(b->parity == 0, "the buffers changed places without a sort");
        after_failure("after a sort that did not launch", b);
    }
    {
        mpm_batch* b = make();
        fail_kernel = (const void*)k_batch_end;
        expect(mpm_batch_step(b, 20) == MPM_ERR_OUT_OF_MEMORY, "an end that does not launch");
        after_failure("after a call without its end", b);
    }
    {
        mpm_batch* b = make();
        fail_graph = 1;
        double ms = 0.0;
        expect(mpm_batch_tune(b, 20, nullptr, &ms) == MPM_ERR_OUT_OF_MEMORY, "a trial that fails");
        after_failure("after a trial that failed", b);
    }
    return bad;
}

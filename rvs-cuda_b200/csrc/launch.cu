// Orchestration of one batch of syntheses on a stream.  Every kernel covers
// all slots of the batch in one launch (the slot is a grid dimension), so a
// batch costs the same launches as a single view and the sequence can be
// captured in a CUDA graph.
#include "device_common.cuh"
#include "kernels.hpp"

namespace rvsb {

template <class Tabs>
int launch_mesh(const Tabs& tabs, const BatchShape& sh, int g0, cudaStream_t s, cudaEvent_t* ev);
template <class Tabs>
void launch_resolve(const Tabs& tabs, const BatchShape& sh, int g0, cudaStream_t s);
template <class Tabs>
int launch_inpaint(const Tabs& tabs, const BatchShape& sh, cudaStream_t s);
template <class Tabs>
void launch_aux(const Tabs& tabs, const BatchShape& sh, cudaStream_t s);
template <class Tabs>
int launch_ms(const Tabs& tabs, const BatchShape& sh, cudaStream_t s);

namespace {

// Per slot: the empty status.  Grid (slots).
template <class Tabs>
__global__ void slot_init_kernel(const __grid_constant__ Tabs tabs) {
    dev::grid_dep_wait();
    if (threadIdx.x == 0) {
        DevStatus* st = tabs.at(blockIdx.x).b.status;
        st->n_large = 0;
        st->n_holes = 0;
    }
}

}  // namespace

template <class Tabs>
int launch_batch(const Tabs& tabs, const BatchShape& sh, cudaStream_t s, cudaEvent_t* ev,
                 const std::function<void()>& before_resolve) {
    auto mark = [&](int k) {
        if (ev) cudaEventRecord(ev[k], s);
    };
    mark(8);
    launch_dependent(slot_init_kernel<Tabs>, dim3(sh.slots), dim3(32), 0, s, tabs);
    int launches = 1;
    for (int g0 = 0; g0 < sh.max_views; g0 += sh.vg) {
        launches += launch_mesh(tabs, sh, g0, s, g0 == 0 ? ev : nullptr);
        if (g0 == 0) mark(4);
        if (g0 == 0 && before_resolve) before_resolve();
        launch_resolve(tabs, sh, g0, s);
        ++launches;
    }
    if (sh.ms) launches += launch_ms(tabs, sh, s);
    mark(5);
    mark(6);
    launches += launch_inpaint(tabs, sh, s);
    if (sh.aux) launch_aux(tabs, sh, s);
    if (sh.rescale) launch_resize(tabs, sh, s);
    mark(7);
    mark(9);
    if (cudaPeekAtLastError() != cudaSuccess) return -1;
    return launches + (sh.aux ? 1 : 0) + (sh.rescale ? 1 : 0);
}

template int launch_batch<TableParam>(const TableParam&, const BatchShape&, cudaStream_t, cudaEvent_t*,
                                      const std::function<void()>&);
template int launch_batch<TablePtr>(const TablePtr&, const BatchShape&, cudaStream_t, cudaEvent_t*,
                                    const std::function<void()>&);

}  // namespace rvsb

// testing.cu -- include/dyg_testing.h.
#include "../../include/dyg_testing.h"

#include "dyg_internal.cuh"

using namespace dyg;

extern "C" dyg_status dyg_testing_stall_barrier(dyg_graph *g, uint32_t spin_limit) {
    // far from any grid's size, and below where the count would wrap to one
    const unsigned long long arrivals = 0x40000000ull;
    DYG_CUDA(cudaMemcpy(ptr<unsigned long long>(g->ws.scalars) + S_BAR, &arrivals, sizeof(arrivals),
                        cudaMemcpyHostToDevice));
    g->bar_limit = spin_limit;
    return DYG_OK;
}

extern "C" void dyg_testing_fail_allocations(uint32_t pass, uint32_t fail) { fail_allocations(pass, fail); }

extern "C" dyg_status dyg_testing_stall_scan(dyg_graph *g) {
    g->ws.scan_tickets -= 1;
    return DYG_OK;
}

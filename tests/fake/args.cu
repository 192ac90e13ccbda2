// What cuda_runtime.cpp reads of a launch's DevArgs (kin_device.cuh compiles as CUDA only).
#include "kin_device.cuh"

extern "C" {
size_t fake_args_size() { return sizeof(sgb::DevArgs); }
// lanes, resume, budget, drain, wait_polls, tables
void fake_args_read(const void *args, uint64_t *out6) {
    const sgb::DevArgs &a = *(const sgb::DevArgs *)args;
    out6[0] = a.lanes;
    out6[1] = a.resume;
    out6[2] = a.budget;
    out6[3] = a.drain;
    out6[4] = a.wait_polls;
    out6[5] = (uint64_t)(uintptr_t)a.tables;
}
uint32_t *fake_args_suspend_count(const void *args) { return ((const sgb::DevArgs *)args)->suspend_count; }
}

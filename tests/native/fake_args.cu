// What the stand-in runtime (fake_cudart.cpp) reads of a launch's arguments.
#include "stage_kernel.cuh"

static void raise(sddc::FaultFlags *f)
{
    f->bits |= sddc::kErrNonPositiveDensity;
    if (f->host) *f->host |= sddc::kErrNonPositiveDensity;
}
void raise_stage(const void *stage_args) { raise(static_cast<const sddc::StageArgs *>(stage_args)->err_flags); }
void raise_trace(const void *trace_init) { raise(static_cast<const sddc::TraceInit *>(trace_init)->flags); }
size_t stage_args_bytes() { return sizeof(sddc::StageArgs); }
size_t trace_init_bytes() { return sizeof(sddc::TraceInit); }

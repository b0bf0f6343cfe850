// What the stand-in runtime (fake_cudart.cpp) reads of a launch's arguments.
#include "stage_kernel.cuh"

unsigned *stage_flags(const void *stage_args) { return static_cast<const sddc::StageArgs *>(stage_args)->err_flags; }
unsigned *trace_flags(const void *trace_init) { return static_cast<const sddc::TraceInit *>(trace_init)->flags; }

// The FP64 form of the kernels by lines; one object per N (SDDC_N), SDDC_N = 0 for
// the dispatch.
#define SDDC_R double
#define SDDC_EXACT_FORM false
#define SDDC_LINE launch_line_fp64
#define SDDC_RESID launch_resid_fp64
#define SDDC_TRACE launch_trace_fp64
#define SDDC_VISC launch_visc_fp64
#include "line_launch.inc"

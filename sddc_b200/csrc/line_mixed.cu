// The mixed form of the kernels by lines; one object per N (SDDC_N), SDDC_N = 0 for
// the dispatch.
#define SDDC_R float
#define SDDC_EXACT_FORM false
#define SDDC_LINE launch_line_mixed
#define SDDC_RESID launch_resid_mixed
#define SDDC_TRACE launch_trace_mixed
#define SDDC_VISC launch_visc_mixed
#include "line_launch.inc"

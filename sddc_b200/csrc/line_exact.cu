// The exact FP64 form of the kernels by lines; one object per N (SDDC_N), SDDC_N = 0 for
// the dispatch.
#define SDDC_R double
#define SDDC_EXACT_FORM true
#define SDDC_LINE launch_line_exact
#define SDDC_RESID launch_resid_exact
#define SDDC_TRACE launch_trace_exact
#define SDDC_VISC launch_visc_exact
#include "line_launch.inc"

// The FP64 form of the line kernel; one object per N (SDDC_N), SDDC_N = 0 for
// the dispatch.
#define SDDC_R double
#define SDDC_EXACT_FORM false
#define SDDC_LINE launch_line_fp64
#include "line_launch.inc"

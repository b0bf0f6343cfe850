// The exact FP64 form of the line kernel; one object per N (SDDC_N), SDDC_N = 0 for
// the dispatch.
#define SDDC_R double
#define SDDC_EXACT_FORM true
#define SDDC_LINE launch_line_exact
#include "line_launch.inc"

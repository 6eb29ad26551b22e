// Mixed-radix axis pass, kind MK_NAB (kw_mr_axis.cuh).
#include "kw_mr_axis.cuh"

KW_MR_AXIS_DEFINE(nab, MK_NAB)

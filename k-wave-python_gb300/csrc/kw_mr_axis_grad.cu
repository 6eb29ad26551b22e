// Mixed-radix axis pass, kind MK_GRAD (kw_mr_axis.cuh).
#include "kw_mr_axis.cuh"

KW_MR_AXIS_DEFINE(grad, MK_GRAD)

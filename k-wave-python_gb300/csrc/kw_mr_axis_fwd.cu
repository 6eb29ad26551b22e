// Mixed-radix axis pass, kind MK_FWD (kw_mr_axis.cuh).
#include "kw_mr_axis.cuh"

KW_MR_AXIS_DEFINE(fwd, MK_FWD)

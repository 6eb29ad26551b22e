// Mixed-radix axis pass, kind MK_GEN (kw_mr_axis.cuh).
#include "kw_mr_axis.cuh"

KW_MR_AXIS_DEFINE(gen, MK_GEN)

// Mixed-radix axis pass, kind MK_DIV (kw_mr_axis.cuh).
#include "kw_mr_axis.cuh"

KW_MR_AXIS_DEFINE(div, MK_DIV)

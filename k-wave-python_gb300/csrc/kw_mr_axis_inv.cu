// Mixed-radix axis pass, kind MK_INV (kw_mr_axis.cuh).
#include "kw_mr_axis.cuh"

KW_MR_AXIS_DEFINE(inv, MK_INV)

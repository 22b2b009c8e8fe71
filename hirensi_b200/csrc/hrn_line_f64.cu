// hrn_line_f64.cu -- the line-operator stage kernels in FP64 (hrn_line.cuh).
#include "hrn_line.cuh"

namespace hrn {
int line_stage_f64(hrn_ctx *c, const void *args, int stage, int adj, int sv, int first, bool pdl)
{
    return line_stage_any<double>(c, args, stage, adj, sv, first, pdl);
}
}  // namespace hrn

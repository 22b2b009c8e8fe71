// hrn_line_f32.cu -- the line-operator stage kernels in FP32 (hrn_line.cuh).
#include "hrn_line.cuh"

namespace hrn {
int line_stage_f32(hrn_ctx *c, const void *args, int stage, int adj, int sv, int first, bool pdl)
{
    return line_stage_any<float>(c, args, stage, adj, sv, first, pdl);
}
}  // namespace hrn

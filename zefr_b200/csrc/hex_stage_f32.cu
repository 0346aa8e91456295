// Hexahedral residual kernels, mixed form.
#include "hex_stage.cuh"

namespace zb {
void bind_hex_f32(Ctx &c) { bind_hex<float, float>(c); }
}  // namespace zb

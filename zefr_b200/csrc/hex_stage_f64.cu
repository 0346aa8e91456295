// Hexahedral residual kernels, FP64 form.
#include "hex_stage.cuh"

namespace zb {
void bind_hex_f64(Ctx &c) { bind_hex<double, double>(c); }
}  // namespace zb

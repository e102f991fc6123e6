// fp32 grids outside the quick index arithmetic's range (quick_grid).
#include "render_launch.cuh"

namespace pgb {
int launch_render_general_f32(const RenderArgs<float>& a, int mode, int phase, cudaStream_t s) {
  return launch_render_t<float, float, false, kGeneral>(a, mode, phase, s);
}
}  // namespace pgb

// Integration with one thread per pixel, 65 to 256 frames in two lists
// (integrate_px.cuh).
#include "integrate_px.cuh"

namespace gg {

void launch_integrate_px2(const IntegrateArgs& a, cudaStream_t stream) { launch_px_list<2, 40, 128>(a, stream); }

}  // namespace gg

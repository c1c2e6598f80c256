// Integration with one thread per pixel, up to 64 frames in one list
// (integrate_px.cuh), and the choice of the list.
#include "integrate_px.cuh"

namespace gg {

// One list up to 64 frames, two of half the frames above; list lengths in steps
// of 8, so that a list sorts at most seven rows of padding (two lists: of a
// frame more or less) whatever the count.  Each length and rejection is one more
// unrolled network to compile, hence two files.
void launch_integrate_px(const IntegrateArgs& a, cudaStream_t stream) {
  if (a.frames <= 64) launch_px_list<1, 16, 64>(a, stream);
  else launch_integrate_px2(a, stream);
}

}  // namespace gg

// FP64 plane and z-column launchers: planes 20x20, 21x21, 24x24, 25x25, 27x27, 24x25, 25x24, 25x27, 27x25.
#include "qx_fftplane64_kern.cuh"

namespace qx {
QX_PLANE64_GRID(20, 20)
QX_PLANE64_GRID(21, 21)
QX_PLANE64_GRID(24, 24)
QX_PLANE64_GRID(25, 25)
QX_PLANE64_GRID(27, 27)
QX_PLANE64_GRID(24, 25)
QX_PLANE64_GRID(25, 24)
QX_PLANE64_GRID(25, 27)
QX_PLANE64_GRID(27, 25)
}  // namespace qx

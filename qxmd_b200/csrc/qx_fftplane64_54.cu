// FP64 plane and z-column launchers: planes 54x54, 54x24, 54x25, 54x27.
#include "qx_fftplane64_kern.cuh"

namespace qx {
QX_PLANE64_GRID(54, 54)
QX_PLANE64_GRID(54, 24)
QX_PLANE64_GRID(54, 25)
QX_PLANE64_GRID(54, 27)
QX_ZCOLS64_LENGTH(54)
}  // namespace qx

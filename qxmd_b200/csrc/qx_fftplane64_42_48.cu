// FP64 plane and z-column launchers: planes 42x42, 42x21, 48x48.
#include "qx_fftplane64_kern.cuh"

namespace qx {
QX_PLANE64_GRID(42, 42)
QX_PLANE64_GRID(42, 21)
QX_PLANE64_GRID(48, 48)
QX_ZCOLS64_LENGTH(42)
QX_ZCOLS64_LENGTH(48)
}  // namespace qx

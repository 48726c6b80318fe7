// The face kernels for gamma = 7/5: seventh roots (mlh_faces.cuh).
#include "mlh_faces.cuh"

namespace mlh {
MLH_FACE_INSTANCES(7)
}  // namespace mlh

// The face kernels for gamma = 5/3: fifth roots (mlh_faces.cuh).
#include "mlh_faces.cuh"

namespace mlh {
MLH_FACE_INSTANCES(5)
}  // namespace mlh

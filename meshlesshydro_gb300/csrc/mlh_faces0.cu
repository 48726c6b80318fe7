// The face kernels for any gamma: powers (mlh_faces.cuh).
#include "mlh_faces.cuh"

namespace mlh {
MLH_FACE_INSTANCES(0)
}  // namespace mlh

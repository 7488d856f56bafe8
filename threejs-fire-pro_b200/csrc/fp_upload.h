// Layout of a step's upload: the work rows of FpBatch, the simulations' SimParams, then their scenes
// (each scene's parts 256-byte aligned). The rows and parameters have room for `room` simulations, so
// that their addresses stay the same while simulations come and go; the scenes follow the parameters
// of the `count` simulations that the step has.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include "fp_types.h"

inline size_t fp_align256(size_t v) { return (v + 255) & ~(size_t)255; }
inline size_t fp_upload_params(int room) {
  return fp_align256((size_t)(FP_WORK_HEAD + FP_WORK_KINDS * (room + 1)) * 4);
}
inline size_t fp_upload_scenes(int room, int count) {
  return fp_align256(fp_upload_params(room) + (size_t)count * sizeof(SimParams));
}
// What an upload of any count up to `room` with `scene` bytes of scenes takes at most.
inline size_t fp_upload_bytes(int room, size_t scene) { return fp_upload_scenes(room, room) + scene; }

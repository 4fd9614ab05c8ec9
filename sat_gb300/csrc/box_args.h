// box_args.h -- a validated box-filter descriptor as the kernels take it,
// shared by the kernels that read a SAT (box_filter.cu) and the fused ones
// (box_fused.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/satgb.h"

namespace satgb {

struct BoxArgs {
  int64_t w, h, planes;
  float* sat;
  int64_t sat_pitch, sat_plane;
  int nr;
  int rmax; // the largest radius
  int r[SATGB_MAX_RADII];
  float inv_full[SATGB_MAX_RADII]; // 1 / (2r + 1): the reciprocal window length away from the edges
  float* box[SATGB_MAX_RADII];
  int64_t box_pitch, box_plane;
  int idx32; // every in-plane element offset fits in 32 bits: only then the interior paths run (int offsets)
};

// Checks a descriptor and fills `a`, radii clamped to max(width, height) - 1
// (box_filter.cu).  Empty sizes return SATGB_OK with `a` untouched.
satgb_status box_check_desc(const satgb_box_desc* d, BoxArgs& a);

// Box means of every radius straight from the image (`a.sat` is the image), or
// their gradient with respect to the image straight from the means' gradients
// (`a.sat` is the gradient written), each in one launch.  *done is false, and
// nothing was launched, when the radii are too large for the kernels' shared
// memory or, unless `only_way`, for going in one launch to be the faster way: the
// caller then does that.  launch false: only *done.
satgb_status box_means_fused(const BoxArgs& a, cudaStream_t s, bool only_way, bool launch, bool* done);
satgb_status box_grad_fused(const BoxArgs& a, cudaStream_t s, bool only_way, bool* done);

}  // namespace satgb

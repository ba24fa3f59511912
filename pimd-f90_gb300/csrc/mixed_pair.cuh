// mixed_pair.cuh -- separations of the mixed engine's pairs (mixed.cu, dipole_matrix.cu)
#pragma once
#include "engine.h"

namespace pimd {

PIMD_D float wrapf(float v, float L, float Li) { return v - L * rint_small(__fmul_rn(v, Li)); }

// O_i - O_j, minimum image, from the fixed-point sites: the unsigned difference wraps modulo the
// box, read as signed it is the nearest image; one rounding to FP32 (relative 2^-24) and the scale
PIMD_D void oo_min_image(const KP &kp, uint4 oi, uint4 oj, float R[3]) {
    R[0] = (float)(int)(oi.x - oj.x) * kp.boxq[0];
    R[1] = (float)(int)(oi.y - oj.y) * kp.boxq[1];
    R[2] = (float)(int)(oi.z - oj.z) * kp.boxq[2];
}

}  // namespace pimd

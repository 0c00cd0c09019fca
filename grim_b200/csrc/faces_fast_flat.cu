// faces_fast_flat.cu -- the face-flux kernels of the tangent /
// mixed-precision path (FMA contraction on) in Minkowski.
#define GRIM_KNS fast
#define GRIM_FAST_MATH 1
#define GRIM_ONLY_FACES 1
#define GRIM_FACES_FLAT 1
#include "kernels.cuh"
#include "launch.h"

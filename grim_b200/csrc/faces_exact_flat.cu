// faces_exact_flat.cu -- the face-flux kernels of the FP64 parity path
// (--fmad=false) in Minkowski.
#define GRIM_KNS exact
#define GRIM_ONLY_FACES 1
#define GRIM_FACES_FLAT 1
#include "kernels.cuh"
#include "launch.h"

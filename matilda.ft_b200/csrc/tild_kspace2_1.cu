// The fused k-space z pass of boxes with 1 density field and force group.
#define TILD_KSPACE2_NF 1
#include "tild_kspace2.cuh"

// The fused k-space z pass of boxes with 3 density fields and force groups.
#define TILD_KSPACE2_NF 3
#include "tild_kspace2.cuh"

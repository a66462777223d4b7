// The fused k-space z pass of boxes with 4 density fields and force groups.
#define TILD_KSPACE2_NF 4
#include "tild_kspace2.cuh"

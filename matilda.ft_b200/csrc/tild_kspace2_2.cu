// The fused k-space z pass of boxes with 2 density fields and force groups.
#define TILD_KSPACE2_NF 2
#include "tild_kspace2.cuh"

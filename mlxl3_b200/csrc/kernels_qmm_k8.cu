// Instantiates the tensor-core product for K = 8 bits per weight.
#define B200_QMM_K 8
#include "kernels_qmm.cu"

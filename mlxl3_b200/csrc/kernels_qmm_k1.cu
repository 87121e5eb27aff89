// Instantiates the tensor-core product for K = 1 bits per weight.
#define B200_QMM_K 1
#include "kernels_qmm.cu"

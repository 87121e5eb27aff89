// Instantiates the tensor-core product for K = 2 bits per weight.
#define B200_QMM_K 2
#include "kernels_qmm.cu"

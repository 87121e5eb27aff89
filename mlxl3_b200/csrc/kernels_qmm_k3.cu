// Instantiates the tensor-core product for K = 3 bits per weight.
#define B200_QMM_K 3
#include "kernels_qmm.cu"

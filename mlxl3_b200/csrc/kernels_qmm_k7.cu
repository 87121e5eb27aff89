// Instantiates the tensor-core product for K = 7 bits per weight.
#define B200_QMM_K 7
#include "kernels_qmm.cu"

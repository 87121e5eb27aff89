// Instantiates the tensor-core product for K = 5 bits per weight.
#define B200_QMM_K 5
#include "kernels_qmm.cu"

// Instantiates the tensor-core product for K = 4 bits per weight.
#define B200_QMM_K 4
#include "kernels_qmm.cu"

// Instantiates the tensor-core product for K = 6 bits per weight.
#define B200_QMM_K 6
#include "kernels_qmm.cu"

// The FP64 builds of mc_kernel, compiled beside the FP32 ones.
#define CEMC_MC_F64
#include "cemc_mc.cu"

// eg_arnoldi_batch_f64.cu -- the FP64 batched persistent GMRES kernel
#include "eg_arnoldi_batch.cuh"

const void* eg_gmres_batch_kernel_f64() { return (const void*)k_gmres_batch<double>; }

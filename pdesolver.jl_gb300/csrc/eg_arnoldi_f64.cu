// eg_arnoldi_f64.cu -- the FP64 persistent GMRES kernels (eg_arnoldi.cu has the
// FP32 ones and the description)
#include "eg_arnoldi_launch.cuh"

int eg_gmres_launch_f64(eg_ls* ls) { return launch_T<double>(ls); }

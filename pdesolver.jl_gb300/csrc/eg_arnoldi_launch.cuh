// eg_arnoldi_launch.cuh -- launches of the persistent GMRES solve, included by
// one translation unit per precision (eg_arnoldi.cu: FP32, eg_arnoldi_f64.cu)
#pragma once
#include <algorithm>
#include <mutex>

#include "eg_arnoldi_body.cuh"

namespace {

// the solve of a small system by one thread-block cluster of C blocks;
// EG_ERR_UNSUPPORTED when such a cluster cannot be placed on this device
template <typename T>
int launch_cluster(eg_ls* ls, CoopArgs<T> a, const void* fn, int C) {
  eg_mesh* m = ls->lo->mesh;
  const size_t smem = plan_smem(a, C);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)C);
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = m->stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  // the placement query takes longer than a small solve's launch: asked once
  // per kernel, device and cluster size, for the largest block
  const bool fits = launch_fact(fn, C, [&]() {
    cfg.dynamicSmemBytes = kSmemBudget;
    int clusters = 0;
    const cudaError_t e = cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg);
    cudaGetLastError();
    cfg.dynamicSmemBytes = smem;
    return e == cudaSuccess && clusters >= 1;
  });
  if (!fits) return EG_ERR_UNSUPPORTED;
  void* args[] = {&a};
  EG_CUDA(cudaLaunchKernelExC(&cfg, fn, args));
  m->launches += 1;
  return EG_OK;
}

template <typename T>
int launch_T(eg_ls* ls) {
  eg_mesh* m = ls->lo->mesh;
  const int rc = eg_gmres_tags(ls);
  if (rc != EG_OK) return rc;
  CoopArgs<T> a;
  coop_args<T>(ls, &a);
  const void* fn = gmres_kernel<T>(ls);
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // grid: one cluster for a small system (one block when no cluster can be
  // placed); otherwise one block per SM (at most one per element), one such
  // grid at a time
  const size_t op_bytes = (size_t)m->E * a.n * a.n * sizeof(T);
  if (ls->coop_grid <= 0) {
    // a cluster for a small system, and for one with at most 32 elements
    // per block of a cluster (no device-wide lock needed)
    const int chunks = (m->E + 31) / 32;
    int C = 0;
    if (op_bytes <= kSmallOperatorBytes)
      C = EG_GMRES_CLUSTER_BLOCKS;
    else if (chunks <= EG_GMRES_CLUSTER_BLOCKS)
      C = std::max(2, chunks);
    while (C > 1 && C > m->E) C >>= 1;
    if (C > 1) {
      int st = launch_cluster<T>(ls, a, fn, C);
      if (st == EG_ERR_UNSUPPORTED && C > 8) st = launch_cluster<T>(ls, a, fn, 8);
      if (st != EG_ERR_UNSUPPORTED) return st;
    }
  }
  // a lone multi-block grid (they run one at a time) takes every SM: the
  // full grid was the fastest for every system above the cluster sizes
  int nblk = op_bytes <= kSmallOperatorBytes ? 1 : std::max(2, std::min(sms, m->E));
  if (ls->coop_grid > 0) nblk = std::min(ls->coop_grid, sms);
  if (nblk > m->E) nblk = m->E;
  if (nblk > EG_COOP_MAX_BLOCKS) nblk = EG_COOP_MAX_BLOCKS;
  const size_t smem = plan_smem(a, nblk);
  const bool resident = launch_fact(fn, 0, [&]() {
    int per_sm = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, NT, kSmemBudget) == cudaSuccess && per_sm >= 1;
  });
  if (!resident || nblk <= 0) {
    eg_set_error("persistent GMRES kernel cannot be resident");
    return EG_ERR_UNSUPPORTED;
  }
  void* args[] = {&a};
  if (nblk == 1) {
    EG_CUDA(cudaLaunchCooperativeKernel(fn, dim3(1), dim3(NT), args, smem, m->stream));
    m->launches += 1;
    return EG_OK;
  }
  std::lock_guard<std::mutex> lock(eg_coop_mutex(dev));
  EG_CUDA(cudaLaunchCooperativeKernel(fn, dim3(nblk), dim3(NT), args, smem, m->stream));
  m->launches += 1;
  EG_CUDA(cudaStreamSynchronize(m->stream));  // the grid has finished before the next one starts
  return EG_OK;
}

}  // namespace

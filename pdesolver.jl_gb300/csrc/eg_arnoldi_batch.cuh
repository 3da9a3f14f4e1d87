// eg_arnoldi_batch.cuh -- the batched persistent GMRES kernel, compiled by one
// translation unit per precision (eg_arnoldi_batch.cu: FP32,
// eg_arnoldi_batch_f64.cu)
#pragma once
#include "eg_arnoldi_body.cuh"

namespace {

constexpr int kMaxBatch = 128;               // problems per launch
// one work-list entry: the problem's kernel arguments (device copy), its
// block range, its (dimension, block size) case and its shared-memory plan
struct BatchEntry {
  const void* args;
  int b0, nblk, kind;
  int ec, fs_smem, ws, p0_smem, kv, er, ef0;
};
struct BatchList {
  int n;
  BatchEntry e[kMaxBatch];
};

template <typename T>
__global__ void __launch_bounds__(NT, 1) k_gmres_batch(BatchList list) {
  __shared__ GmresShared<T> sm;
  __shared__ CoopArgs<T> sa;
  __shared__ int s_nblk, s_b0, s_kind;
  if (threadIdx.x == 0) {
    int k = 0;
    while (k + 1 < list.n && (int)blockIdx.x >= list.e[k + 1].b0) ++k;
    const BatchEntry en = list.e[k];
    s_nblk = en.nblk;
    s_b0 = en.b0;
    s_kind = en.kind;
    sa = *reinterpret_cast<const CoopArgs<T>*>(en.args);
    sa.ec = en.ec;
    sa.fs_smem = en.fs_smem;
    sa.ws = en.ws;
    sa.p0_smem = en.p0_smem;
    sa.kv = en.kv;
    sa.er = en.er;
    sa.ef0 = en.ef0;
  }
  __syncthreads();
  const int nblk = s_nblk, b = (int)blockIdx.x - s_b0;
  switch (s_kind) {
    case 0: gmres_body<2, 12, T>(sa, b, nblk, sm); break;
    case 1: gmres_body<2, 24, T>(sa, b, nblk, sm); break;
    case 2: gmres_body<2, 28, T>(sa, b, nblk, sm); break;
    case 3: gmres_body<2, 40, T>(sa, b, nblk, sm); break;
    case 4: gmres_body<2, 48, T>(sa, b, nblk, sm); break;
    case 5: gmres_body<2, 60, T>(sa, b, nblk, sm); break;
    case 6: gmres_body<2, 72, T>(sa, b, nblk, sm); break;
    case 7: gmres_body<2, 0, T>(sa, b, nblk, sm); break;
    case 8: gmres_body<3, 30, T>(sa, b, nblk, sm); break;
    case 9: gmres_body<3, 115, T>(sa, b, nblk, sm); break;
    default: gmres_body<3, 0, T>(sa, b, nblk, sm); break;
  }
}

}  // namespace

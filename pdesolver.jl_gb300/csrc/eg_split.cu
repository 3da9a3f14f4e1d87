// eg_split.cu -- entropy-conservative Hadamard split-form volume integral.
//
// Reference: calcVolumeIntegralsSplitFormCurvilinear
// (src/solver/euler/euler_funcs.jl:295-362) with calcSCurvilinear
// (src/Utils/curvilinear.jl:17-41):
//   S_x[j,k,d] = 1/2 sum_m (dxidx[m,d,j] Q_m(j,k) - dxidx[m,d,k] Q_m(k,j))
//   res_j -= 2 sum_d S_x[j,k,d] F_IR,d(q_j, q_k),  res_k += same   (k < j)
// The IR flux is linear in its direction, so sum_d S_x[j,k,d] F_IR,d equals
// one IR flux in the direction n_jk = S_x[j,k,:]; each pair (j,k) costs one
// Ismail-Roe average and one projection.  The square roots and logarithms of
// the averages are per-node quantities, computed once per node (FP64 is the
// scarce resource on GB300); a pair costs divisions and multiply-adds only.
//
// k_split_element: thread (element, node j) walks the pairs (j, j + s mod Np),
// s = 1 .. Np/2 (for even Np the last distance only from the first half of the
// nodes), so every thread has the same number of pairs.  Its own node's
// quantities and its row of the residual stay in registers; the other node's
// row is added to in shared memory, where the threads of one distance touch
// distinct nodes (one block barrier per distance, no atomics, deterministic).
// The Q entries of a distance are laid out by j, so the threads read them and
// the other node's quantities without bank conflicts.
//
// Bound: the FP64 pipe.  A pair costs 84 FP64 instructions (the averages from
// the per-node quantities with two approximate reciprocals, see
// ir_average_pre); 117 with a division, four threshold tests and separate
// means, and a table of all pair fluxes in shared memory (17 KB per element,
// one CTA per SM).  82,944 tets p=2, residual: 6.72 -> 3.92 ms.
#include "eg_internal.h"
#include "eg_kernels.cuh"
#include "eg_physics.cuh"

using eg::Gas;

namespace {

template <int DIM>
__global__ void k_split_element(DevMesh md, const double* __restrict__ q,
                                const double* __restrict__ fflux, Epilogue ep,
                                unsigned int* __restrict__ status, int epb) {
  constexpr int NV = DIM + 2;
  constexpr int F = DIM + 1;
  constexpr int ND = 7 + DIM * DIM;
  extern __shared__ double smem[];
  const int Np = md.Np, Nf = md.Nf, S = md.S;
  const int H = Np / 2;
  const int rows = epb * Np;
  double* sQa = smem;                         // [H][DIM][Np]: Q_m(j, j + s)
  double* sQb = sQa + H * DIM * Np;           // [H][DIM][Np]: Q_m(j + s, j)
  double* sL = sQb + H * DIM * Np;            // [F][Nf][S]
  int* sPerm = reinterpret_cast<int*>(sL + F * Nf * S);
  double* sN = sL + F * Nf * S + (F * S + 1) / 2;  // [ND][rows]: IR quantities, metrics
  double* sres = sN + (size_t)ND * rows;      // [epb][Np][NV]
  for (int t = threadIdx.x; t < H * DIM * Np; t += blockDim.x) {
    const int s = t / (DIM * Np), r = t - s * DIM * Np;
    const int m = r / Np, j = r - m * Np;
    int k = j + s + 1;
    if (k >= Np) k -= Np;
    sQa[t] = md.Q[((size_t)m * Np + k) * Np + j];  // md.Q[m][k][j] = Q_m(j, k)
    sQb[t] = md.Q[((size_t)m * Np + j) * Np + k];
  }
  for (int k = threadIdx.x; k < F * Nf * S; k += blockDim.x) sL[k] = md.liftS[k];
  for (int k = threadIdx.x; k < F * S; k += blockDim.x) sPerm[k] = md.perm[k];
  const int e0 = blockIdx.x * epb;
  const int nloc = min(epb, md.E - e0);
  const int t = threadIdx.x;
  const int le = t / Np, j = t - le * Np;
  const bool active = le < nloc;
  const Gas g{md.gamma, md.gamma_1};
  eg::IRNode<DIM> nd = {};
  double dx[DIM * DIM];  // [x][xi] of the own node
  double acc[NV];
#pragma unroll
  for (int c = 0; c < NV; ++c) acc[c] = 0.0;
#pragma unroll
  for (int c = 0; c < DIM * DIM; ++c) dx[c] = 0.0;
  if (active) {
    double qj[NV];
    const double* src = q + ((size_t)e0 * Np + t) * NV;
#pragma unroll
    for (int c = 0; c < NV; ++c) qj[c] = src[c];
    const double* dxj = md.dxidx + ((size_t)e0 * Np + t) * DIM * DIM;
#pragma unroll
    for (int c = 0; c < DIM * DIM; ++c) {
      dx[c] = dxj[c];
      sN[(7 + c) * rows + t] = dx[c];
    }
    const double pj = eg::pressure<DIM>(g, qj);
    if (!(qj[0] > 0.0)) atomicOr(status, EG_DEV_NEG_DENSITY);
    if (!(pj > 0.0)) atomicOr(status, EG_DEV_NEG_PRESSURE);
    nd = eg::ir_node<DIM, false>(g, qj);
    sN[0 * rows + t] = nd.z1;
    sN[1 * rows + t] = nd.zp;
    sN[4 * rows + t] = nd.zu;
    sN[5 * rows + t] = nd.zv;
    sN[6 * rows + t] = nd.zw;
#pragma unroll
    for (int c = 0; c < NV; ++c) sres[(size_t)t * NV + c] = 0.0;
  }
  __syncthreads();
  // The logarithms are for pairs whose ratio of z1 or zp exceeds 1.065 (u above
  // 1e-3).  Nodes all within 3 % of the element's first have no such pair
  // (1.03 / 0.97 = 1.062), and the CTA then skips them (two per node were 8 %
  // of the FP64 work at p=2).
  bool far = false;
  if (active) {
    const double z0 = sN[0 * rows + le * Np], p0 = sN[1 * rows + le * Np];
    far = !(fabs(nd.z1 - z0) <= 0.03 * z0) || !(fabs(nd.zp - p0) <= 0.03 * p0);
  }
  if (__syncthreads_or(far)) {
    if (active) {
      sN[2 * rows + t] = nd.lz1 = log(nd.z1);
      sN[3 * rows + t] = nd.lzp = log(nd.zp);
    }
    __syncthreads();
  }
#pragma unroll 1
  for (int s = 0; s < H; ++s) {
    int k = j + s + 1;
    if (k >= Np) k -= Np;
    // even Np: distance Np/2 pairs each node with its opposite once
    if (active && (2 * (s + 1) < Np || j < H)) {
      const int o = le * Np + k;
      const double* qa = sQa + s * DIM * Np + j;
      const double* qb = sQb + s * DIM * Np + j;
      double n[DIM];  // 2 S_x[j,k,:]
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        double v = 0.0;
#pragma unroll
        for (int m = 0; m < DIM; ++m) {
          v = fma(dx[d * DIM + m], qa[m * Np], v);
          v = fma(-sN[(7 + d * DIM + m) * rows + o], qb[m * Np], v);
        }
        n[d] = v;
      }
      const eg::IRNode<DIM> no{sN[0 * rows + o], sN[1 * rows + o], sN[2 * rows + o], sN[3 * rows + o],
                               sN[4 * rows + o], sN[5 * rows + o], sN[6 * rows + o]};
      const auto av = eg::ir_average_pre<DIM>(g, nd, no);
      double G[NV];
      eg::ir_dir<DIM>(av, n, G);
      double* r = sres + (size_t)o * NV;
#pragma unroll
      for (int c = 0; c < NV; ++c) {
        acc[c] -= G[c];
        r[c] += G[c];
      }
    }
    __syncthreads();
  }
  if (active) {
#pragma unroll
    for (int c = 0; c < NV; ++c) sres[(size_t)t * NV + c] += acc[c];
  }
  __syncthreads();
  face_lift_smem<DIM>(md, fflux, sres, sL, sPerm, e0, nloc);
  write_residual<NV>(ep, sres, (size_t)e0 * Np * NV, nloc * Np * NV);
}

}  // namespace

int eg_launch_split_element(eg_mesh* m, const double* q, const Epilogue& ep, int epb) {
  DevMesh md = dev_mesh(m);
  int threads;
  size_t smem;
  const int st = eg_element_shape(m, epb, 0, &threads, &smem);
  if (st != EG_OK) return st;
  const int blocks = (m->E + epb - 1) / epb;
  // once per process (thread-safe static initialisation)
  static const bool attr_set = [] {
    cudaFuncSetAttribute(k_split_element<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(k_split_element<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    return true;
  }();
  (void)attr_set;
  if (m->dim == 2)
    k_split_element<2><<<blocks, threads, smem, m->stream>>>(md, q, m->fflux, ep, m->status, epb);
  else
    k_split_element<3><<<blocks, threads, smem, m->stream>>>(md, q, m->fflux, ep, m->status, epb);
  return EG_OK;
}

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
// The directions n_jk (18 multiply-adds per pair) are formed in the integer
// pipe, which has room: metrics and Q entries as 60-bit fixed-point numbers in
// two 30-bit limbs, a physical direction's metrics relative to the largest of
// that direction in the element, a pair's Q entries relative to its largest;
// n_jk[d] = sum of 2 DIM products, high x high and the two cross terms in
// 64-bit accumulators, converted to FP64 once and scaled by its power of two.
// With R and Qj the largest entries, the roundings of the inputs (2 DIM 2^-60
// each), the low x low terms (at most 2 DIM 2^-60: the low limb is signed) and
// the last shift sum to at most (6 DIM + 1) 2^-60 R Qj, 2^-55.7 in 3-D; FP64
// directions round at 2^-53 of each term.  Scales of their own keep a thin
// direction of a stretched element at that accuracy: with one scale for the
// element an aspect ratio r cost its residual a factor r / 8.
//
// Bound: the FP64 pipe.  A pair costs 69 FP64 instructions (the averages from
// the per-node quantities with two approximate reciprocals, see
// ir_average_pre); 117 with a division, four threshold tests and separate
// means, and a table of all pair fluxes in shared memory (17 KB per element,
// one CTA per SM).  82,944 tets p=2, residual: 6.72 -> 3.81 ms with n_jk in
// FP64, 3.43 ms in fixed point.
#include "eg_internal.h"
#include "eg_kernels.cuh"
#include "eg_physics.cuh"

using eg::Gas;

namespace {

// Fixed point: v = round(x 2^(59 - ex)), |x| < 2^ex, as v = h 2^30 + l with
// |h| <= 2^29 and -2^29 <= l < 2^29.
struct Limbs {
  int h, l;
};
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }
// smallest e with |x| < 2^e for the largest high word of |x| (subnormals count
// as 2^-1022, zero as 1, infinities and NaN as EG_QEXP_NONFINITE)
__device__ __forceinline__ int exponent_above(int hi) {
  const int b = hi >> 20;
  return hi == 0 ? 0 : b == 0x7ff ? EG_QEXP_NONFINITE : (b < 1 ? 1 : b) - 1022;
}
__device__ __forceinline__ Limbs to_limbs(double x, int ex) {
  // two exact scalings: 59 - ex may exceed the exponent range of one
  const int k = 59 - ex, k1 = k / 2;
  const long long v = __double2ll_rn(x * pow2(k1) * pow2(k - k1));
  const int h = (int)((v + (1 << 29)) >> 30);
  return Limbs{h, (int)(v - ((long long)h << 30))};
}
// v 2^k: the exponent field takes k (v = 0 has none), or beyond its range three
// products; NaN where a metric or Q entry is not finite
__device__ __forceinline__ double scaled(long long v, int k) {
  const double x = (double)v;
  if (abs(k) <= 900) return v == 0 ? 0.0 : __hiloint2double(__double2hiint(x) + (k << 20), __double2loint(x));
  if (k > EG_QEXP_NONFINITE / 2) return __longlong_as_double(0x7ff8000000000000LL);
  const int k3 = k / 3;
  return x * pow2(k3) * pow2(k3) * pow2(k - 2 * k3);
}

template <int DIM>
__device__ __forceinline__ void split_element(const DevMesh& md, const double* __restrict__ q,
                                              const double* __restrict__ fflux, const Epilogue& ep,
                                              unsigned int* __restrict__ status, int epb) {
  constexpr int NV = DIM + 2;
  constexpr int F = DIM + 1;
  constexpr int D2 = DIM * DIM;
  extern __shared__ double smem[];
  const int Np = md.Np, Nf = md.Nf, S = md.S;
  const int H = Np / 2;
  const int rows = epb * Np;
  Limbs* sQa = reinterpret_cast<Limbs*>(smem);  // [H][DIM][Np]: Q_m(j, j + s)
  Limbs* sQb = sQa + H * DIM * Np;            // [H][DIM][Np]: Q_m(j + s, j)
  double* sL = reinterpret_cast<double*>(sQb + H * DIM * Np);  // [F][Nf][S]
  int* sPerm = reinterpret_cast<int*>(sL + F * Nf * S);
  double* sN = sL + F * Nf * S + (F * S + 1) / 2;  // [7][rows]: IR quantities
  Limbs* sD = reinterpret_cast<Limbs*>(sN + (size_t)7 * rows);  // [DIM DIM][rows]: metrics
  double* sres = reinterpret_cast<double*>(sD + (size_t)D2 * rows);  // [epb][Np][NV]
  // [epb][DIM] largest high word of |dxidx| of a physical direction, where the
  // logarithms go later
  int* sMax = reinterpret_cast<int*>(sN + (size_t)2 * rows);
  for (int k = threadIdx.x; k < epb * DIM; k += blockDim.x) sMax[k] = 0;
  for (int k = threadIdx.x; k < 2 * H * DIM * Np; k += blockDim.x) {
    const int2 v = md.Qpair[k];
    sQa[k] = Limbs{v.x, v.y};
  }
  for (int k = threadIdx.x; k < F * Nf * S; k += blockDim.x) sL[k] = md.liftS[k];
  for (int k = threadIdx.x; k < F * S; k += blockDim.x) sPerm[k] = md.perm[k];
  __syncthreads();  // sMax
  const int e0 = blockIdx.x * epb;
  const int nloc = min(epb, md.E - e0);
  const int t = threadIdx.x;
  const int le = t / Np, j = t - le * Np;
  const bool active = le < nloc;
  const Gas g{md.gamma, md.gamma_1};
  eg::IRNode<DIM> nd = {};
  double dxd[D2];
  Limbs dx[D2];  // metrics [x][xi] of the own node
  double acc[NV];
#pragma unroll
  for (int c = 0; c < NV; ++c) acc[c] = 0.0;
#pragma unroll
  for (int c = 0; c < D2; ++c) {
    dxd[c] = 0.0;
    dx[c] = Limbs{0, 0};
  }
  if (active) {
    double qj[NV];
    const double* src = q + ((size_t)e0 * Np + t) * NV;
#pragma unroll
    for (int c = 0; c < NV; ++c) qj[c] = src[c];
    const double* dxj = md.dxidx + ((size_t)e0 * Np + t) * D2;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      int hi = 0;
#pragma unroll
      for (int m = 0; m < DIM; ++m) {
        dxd[d * DIM + m] = dxj[d * DIM + m];
        hi = max(hi, __double2hiint(dxd[d * DIM + m]) & 0x7fffffff);
      }
      atomicMax(&sMax[le * DIM + d], hi);
    }
    const double pj = eg::pressure<DIM>(g, qj);
    if (!(qj[0] > 0.0)) atomicOr(status, EG_DEV_NEG_DENSITY);
    if (!(pj > 0.0)) atomicOr(status, EG_DEV_NEG_PRESSURE);
    nd = eg::ir_node<DIM>(g, qj);
    sN[0 * rows + t] = nd.z1;
    sN[1 * rows + t] = nd.zp;
    sN[4 * rows + t] = nd.zu;
    sN[5 * rows + t] = nd.zv;
    sN[6 * rows + t] = nd.zw;
#pragma unroll
    for (int c = 0; c < NV; ++c) sres[(size_t)t * NV + c] = 0.0;
  }
  __syncthreads();
  int ex[DIM];  // n_jk[d] is in units of 2^(ex[d] + pair's exponent)
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    const int e = active ? exponent_above(sMax[le * DIM + d]) : 0;
    if (active) {
#pragma unroll
      for (int m = 0; m < DIM; ++m) sD[(d * DIM + m) * rows + t] = dx[d * DIM + m] = to_limbs(dxd[d * DIM + m], e);
    }
    ex[d] = e - 60;
  }
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
      Limbs qa[DIM], qb[DIM];
#pragma unroll
      for (int m = 0; m < DIM; ++m) {
        qa[m] = sQa[(s * DIM + m) * Np + j];
        qb[m] = sQb[(s * DIM + m) * Np + j];
      }
      const int eq = md.Qexp[s * Np + j];
      double n[DIM];  // 2 S_x[j,k,:]
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        long long hh = 0, x = 0;
#pragma unroll
        for (int m = 0; m < DIM; ++m) {
          const Limbs a = dx[d * DIM + m], b = sD[(d * DIM + m) * rows + o];
          hh += (long long)a.h * qa[m].h - (long long)b.h * qb[m].h;
          x += (long long)a.h * qa[m].l + (long long)a.l * qa[m].h;
          x -= (long long)b.h * qb[m].l + (long long)b.l * qb[m].h;
        }
        n[d] = scaled((hh << 2) + ((x + (1 << 27)) >> 28), ex[d] + eq);
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

template <int DIM>
__global__ void k_split_element(DevMesh md, const double* __restrict__ q, const double* __restrict__ fflux,
                                Epilogue ep, unsigned int* __restrict__ status, int epb) {
  split_element<DIM>(md, q, fflux, ep, status, epb);
}

// The pair loop takes 122 registers (88 on triangles), too many for a block of
// more than 512 (736) threads to launch.  Wider blocks, which only an explicit
// launch configuration or the autotuner asks for, run a build held to the
// registers that MAXT threads leave.
template <int DIM, int MAXT>
__global__ void __launch_bounds__(MAXT) k_split_wide(DevMesh md, const double* __restrict__ q,
                                                     const double* __restrict__ fflux, Epilogue ep,
                                                     unsigned int* __restrict__ status, int epb) {
  split_element<DIM>(md, q, fflux, ep, status, epb);
}

template <int DIM>
int launch_split(eg_mesh* m, const DevMesh& md, const double* q, const Epilogue& ep, int epb, int threads,
                 size_t smem) {
  static EgDeviceOnce once;
  int dev = 0;
  cudaGetDevice(&dev);
  once(dev, [] {
    cudaFuncSetAttribute(k_split_element<DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(k_split_wide<DIM, 768>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(k_split_wide<DIM, 1024>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  });
  // of the code, the same on every device
  static const int narrow = [] {
    cudaFuncAttributes a;
    return cudaFuncGetAttributes(&a, k_split_element<DIM>) == cudaSuccess ? a.maxThreadsPerBlock : 0;
  }();
  const int blocks = (m->E + epb - 1) / epb;
  if (threads <= narrow)
    k_split_element<DIM><<<blocks, threads, smem, m->stream>>>(md, q, m->fflux, ep, m->status, epb);
  else if (threads <= 768)
    k_split_wide<DIM, 768><<<blocks, threads, smem, m->stream>>>(md, q, m->fflux, ep, m->status, epb);
  else
    k_split_wide<DIM, 1024><<<blocks, threads, smem, m->stream>>>(md, q, m->fflux, ep, m->status, epb);
  return EG_OK;
}

}  // namespace

int eg_launch_split_element(eg_mesh* m, const double* q, const Epilogue& ep, int epb) {
  DevMesh md = dev_mesh(m);
  int threads;
  size_t smem;
  const int st = eg_element_shape(m, epb, 0, &threads, &smem);
  if (st != EG_OK) return st;
  return m->dim == 2 ? launch_split<2>(m, md, q, ep, epb, threads, smem)
                     : launch_split<3>(m, md, q, ep, epb, threads, smem);
}

// eg_small.cu -- the weak-form residual of a small mesh in one launch.
//
// Reference: as eg_residual.cu (euler.jl:111-175); the flux, contraction and
// lifting arithmetic is the same, in the same order, so the results are the
// two-kernel path's bit for bit.
//
// On this GPU a warp issues one FP64 instruction per 64 cycles however many
// lanes are active and however independent its instructions are, and an SM
// reaches its rate (19 cycles per instruction) with four warps.  A mesh of a
// few hundred elements therefore costs the chain of its longest thread: face
// interpolation and Roe flux (211 instructions) and then element flux,
// contraction and lifting (about 130), in two launches.  Here a CTA owns the
// `epb` elements that make one CTA per SM and takes the fluxes of all their
// faces itself (an interior face twice on the GPU), so nothing crosses CTAs;
// the work is cut into short tasks for separate warps: interpolation by
// (face node, side, variable), then fluxes beside the Euler fluxes of the
// nodes, then contraction and lifting by (node, variable).  The chain is 6 +
// 163 + 21 instructions, and the RK4 stage is its epilogue.
#include "eg_internal.h"
#include "eg_kernels.cuh"
#include "eg_physics.cuh"

using eg::Gas;

namespace {

constexpr int NT = 256;

template <int DIM>
__global__ void __launch_bounds__(NT) k_small_residual(DevMesh md, const double* __restrict__ q, Epilogue ep,
                                                       unsigned int* __restrict__ status, int epb) {
  constexpr int NV = DIM + 2;
  constexpr int F = DIM + 1;
  extern __shared__ double smem[];
  const int Np = md.Np, Nf = md.Nf, S = md.S;
  double* sQ = smem;                              // [DIM][Np][Np]
  double* sL = sQ + DIM * Np * Np;                // [F][Nf][S]
  double* sI = sL + F * Nf * S;                   // [F][Nf][S] interpolation
  double* sF = sI + F * Nf * S;                   // [epb][DIM][Np][NV]
  double* sS = sF + (size_t)epb * DIM * Np * NV;  // [epb][F][Nf][2][NV] face states
  double* sX = sS + (size_t)epb * F * Nf * 2 * NV;  // [epb][F][Nf][NV] face fluxes
  double* sres = sX + (size_t)epb * F * Nf * NV;  // [epb][Np][NV]
  int* sPerm = reinterpret_cast<int*>(sres + (size_t)epb * Np * NV);  // [F][S]
  EFace* sE = reinterpret_cast<EFace*>(sPerm + ((F * S + 3) & ~3));   // [epb][F]
  const int tid = threadIdx.x;
  const int e0 = blockIdx.x * epb;
  const int nloc = min(epb, md.E - e0);
  for (int k = tid; k < DIM * Np * Np; k += NT) sQ[k] = md.Q[k];
  for (int k = tid; k < F * Nf * S; k += NT) {
    sL[k] = md.liftS[k];
    sI[k] = md.interp[k];
  }
  for (int k = tid; k < F * S; k += NT) sPerm[k] = md.perm[k];
  for (int k = tid; k < nloc * F; k += NT) sE[k] = md.eface[(size_t)e0 * F + k];
  __syncthreads();
  const Gas g{md.gamma, md.gamma_1};
  // ---- face states: (element face, face node, side, variable)
  const int nfn = nloc * F * Nf;  // face nodes
  for (int t = tid; t < nfn * 2 * NV; t += NT) {
    const int c = t % NV, r = t / NV;
    const int side = r & 1, fn = r >> 1;
    const int lf = fn / Nf, i = fn - lf * Nf;
    const EFace ef = sE[lf];
    double v = 0.0;
    if (ef.slot < md.I) {
      const int* itf = md.ifaces + 5 * ef.slot;
      const int e = itf[side], f = itf[2 + side];
      const int row = side ? md.nbrperm[itf[4] * Nf + i] : i;
      const double* x = q + (size_t)e * Np * NV + c;
      if (md.sparse_face) {
        v = x[sPerm[f * S + row] * NV];
      } else {
        const double* w = sI + (f * Nf + row) * S;
        for (int s = 0; s < S; ++s) v = fma(w[s], x[sPerm[f * S + s] * NV], v);
      }
    } else {
      const int b = ef.slot - md.I;
      const int e = md.bfaces[2 * b], f = md.bfaces[2 * b + 1];
      if (side == 0) {
        const double* x = q + (size_t)e * Np * NV + c;
        if (md.sparse_face) {
          v = x[sPerm[f * S + i] * NV];
        } else {
          const double* w = sI + (f * Nf + i) * S;
          for (int s = 0; s < S; ++s) v = fma(w[s], x[sPerm[f * S + s] * NV], v);
        }
      } else if (md.bc_of_b[b] != EG_BC_NOPENETRATION_ES) {
        v = md.qg_bndry[((size_t)b * Nf + i) * NV + c];
      }
    }
    sS[t] = v;
  }
  __syncthreads();
  // ---- face fluxes, and beside them (from the next whole warp on) the Euler
  //      fluxes of the nodes in the parametric directions
  const int nfw = (nfn + 31) & ~31;
  for (int t = tid; t < nfw + nloc * Np; t += NT) {
    if (t < nfw) {
      if (t >= nfn) continue;
      const int lf = t / Nf, i = t - lf * Nf;
      const EFace ef = sE[lf];
      const bool interior = ef.slot < md.I;
      const double* src = interior ? md.nrm_face + ((size_t)ef.slot * Nf + i) * DIM
                                   : md.nrm_bndry + ((size_t)(ef.slot - md.I) * Nf + i) * DIM;
      double nrm[DIM], qL[NV], qR[NV], fl[NV];
#pragma unroll
      for (int k = 0; k < DIM; ++k) nrm[k] = src[k];
#pragma unroll
      for (int c = 0; c < NV; ++c) {
        qL[c] = sS[(size_t)t * 2 * NV + c];
        qR[c] = sS[(size_t)t * 2 * NV + NV + c];
      }
      if (!interior && md.bc_of_b[ef.slot - md.I] == EG_BC_NOPENETRATION_ES) {
        eg::wall_es_flux<DIM>(g, qL, nrm, fl);
      } else if (!interior || md.face_flux == EG_FLUX_ROE) {
        eg::roe_flux<DIM>(g, qL, qR, nrm, fl);
      } else {
        const auto nL = eg::ir_node<DIM>(g, qL);
        const auto nR = eg::ir_node<DIM>(g, qR);
        const auto av = eg::ir_average_pre<DIM, false>(g, nL, nR);
        eg::ir_dir<DIM>(av, nrm, fl);
      }
#pragma unroll
      for (int c = 0; c < NV; ++c) sX[(size_t)t * NV + c] = fl[c];
    } else {
      const int r = t - nfw;  // (element, node)
      const int le = r / Np, j = r - le * Np;
      double qj[NV];
#pragma unroll
      for (int c = 0; c < NV; ++c) qj[c] = q[((size_t)e0 * Np + r) * NV + c];
      const double p = eg::pressure<DIM>(g, qj);
      if (!(qj[0] > 0.0)) atomicOr(status, EG_DEV_NEG_DENSITY);
      if (!(p > 0.0)) atomicOr(status, EG_DEV_NEG_PRESSURE);
      const double* dx = md.dxidx + ((size_t)e0 * Np + r) * DIM * DIM;
#pragma unroll
      for (int k = 0; k < DIM; ++k) {
        double dir[DIM];
#pragma unroll
        for (int pp = 0; pp < DIM; ++pp) dir[pp] = dx[pp * DIM + k];
        eg::euler_flux<DIM>(g, qj, dir, sF + (((size_t)le * DIM + k) * Np + j) * NV);
      }
    }
  }
  __syncthreads();
  // ---- contraction and face lifting by (element, node, variable)
  for (int t = tid; t < nloc * Np * NV; t += NT) {
    const int c = t % NV, r = t / NV;
    const int le = r / Np, j = r - le * Np;
    double acc = 0.0;
    for (int k = 0; k < DIM; ++k) {
      const double* qrow = sQ + ((size_t)k * Np + j) * Np;
      const double* Fk = sF + ((size_t)le * DIM + k) * Np * NV + c;
      for (int i = 0; i < Np; ++i) acc = fma(qrow[i], Fk[i * NV], acc);
    }
    for (int f = 0; f < F; ++f) {
      int s = -1;
      for (int k = 0; k < S; ++k)
        if (sPerm[f * S + k] == j) s = k;
      if (s < 0) continue;
      const EFace ef = sE[le * F + f];
      const double* fl = sX + (size_t)(le * F + f) * Nf * NV + c;
      double a = 0.0;
      if (md.sparse_face) {
        const int i = ef.side ? md.nbrinv[ef.orient * Nf + s] : s;
        a = md.wface[s] * fl[i * NV];
      } else {
        const int* nb = md.nbrperm + ef.orient * Nf;
        for (int i = 0; i < Nf; ++i) a = fma(sL[(f * Nf + (ef.side ? nb[i] : i)) * S + s], fl[i * NV], a);
      }
      if (ef.side == 0) acc -= a;
      else acc += a;
    }
    sres[t] = acc;
  }
  __syncthreads();
  write_residual<NV>(ep, sres, (size_t)e0 * Np * NV, nloc * Np * NV);
}

size_t small_smem(const eg_mesh* m, int epb) {
  const size_t Np = m->Np, Nf = m->Nf, S = m->S, F = m->F, d = m->dim, nv = m->nv;
  return 8 * (d * Np * Np + 2 * F * Nf * S + epb * (d * Np * nv + F * Nf * 3 * nv + Np * nv)) +
         4 * ((F * S + 3) & ~(size_t)3) + sizeof(EFace) * epb * F;
}

// one CTA per SM
int small_epb(const eg_mesh* m) { return (m->E + 151) / 152; }

}  // namespace

// The one-launch path is taken up to kSmallPerSM elements per SM (1,672
// elements): above, the second evaluation of the interior faces costs more
// FP64 time than the short chains and the launch save.  Measured, two kernels
// -> one, us per residual: 128 to 512 triangles 23-39 -> 12.5-20.7 (p=2, 512:
// 24.8 -> 14.5), 1,152 triangles p=4 39 -> 29, 1,568 p=3 28.8 -> 26.8, 1,568
// p=4 41 -> 36, but 2,048 p=3 28.8 -> 28.9 and 2,048 p=4 35 -> 41; 750 tets
// p=1 31 -> 14.5.  An explicit launch configuration and a residual written
// over its own state keep to the two kernels.
bool eg_small_usable(const eg_mesh* m, const double* q, const Epilogue& ep) {
  constexpr int kSmallPerSM = 11;
  return m->params.volume_integral_type == 1 && m->elem_epb == 0 && m->vol_mma == 0 &&
         small_epb(m) <= kSmallPerSM && ep.out != q && small_smem(m, small_epb(m)) <= 200 * 1024;
}

int eg_launch_small(eg_mesh* m, const double* q, const Epilogue& ep) {
  static EgDeviceOnce once;
  int dev = 0;
  cudaGetDevice(&dev);
  once(dev, [] {
    cudaFuncSetAttribute(k_small_residual<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(k_small_residual<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  });
  const DevMesh md = dev_mesh(m);
  const int epb = small_epb(m), blocks = (m->E + epb - 1) / epb;
  const size_t smem = small_smem(m, epb);
  eg_phase_begin(m, EG_PHASE_ELEMENT);
  if (m->dim == 2)
    k_small_residual<2><<<blocks, NT, smem, m->stream>>>(md, q, ep, m->status, epb);
  else
    k_small_residual<3><<<blocks, NT, smem, m->stream>>>(md, q, ep, m->status, epb);
  eg_phase_end(m, EG_PHASE_ELEMENT, 1);
  return EG_OK;
}

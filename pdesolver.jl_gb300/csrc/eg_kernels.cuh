// eg_kernels.cuh -- kernel-side view of an eg_mesh and launch helpers shared
// by the translation units of libeulergpu.
#pragma once
#include "eg_internal.h"

// Plain-pointer view passed to kernels by value.
struct DevMesh {
  int E, Np, Nf, S, I, B;
  int face_flux;
  double gamma, gamma_1;
  const double* Q;        // [dim][Np][Np], Q[k][j][i] = Q_k(i, j)
  const double* interp;   // [F][Nf][S]
  const int* perm;        // [F][S]
  const int* nbrperm;     // [norient][Nf]
  const int2* Qpair;      // [2][Np/2][dim][Np]: Q_m(j, j + s), Q_m(j + s, j) (indices mod Np) in fixed point
  const int* Qexp;        // [Np/2][Np]: 2^Qexp > the pair's largest |Q|
  const double* dxidx;    // [E][Np][dim][dim]
  const int* ifaces;      // [I][5]
  const double* nrm_face; // [I][Nf][dim]
  const int* bfaces;      // [B][2]
  const double* nrm_bndry;// [B][Nf][dim]
  const double* qg_bndry; // [B][Nf][nv]
  const int* bc_of_b;     // [B] boundary condition (eg_bc) of each boundary face
  const EFace* eface;     // [E][F]
  const double* Minv;     // [E][Np]
  const double* w;        // [Np]
  const double* jac;      // [E][Np]
  const double* liftS;    // [F][Nf][S]: interp[f][i][s] * wface[i]
  const int* nbrinv;      // [norient][Nf]: inverse of nbrperm
  const double* wface;    // [Nf]
  int sparse_face;        // face nodes are volume nodes (interp = identity)
};

// Face terms of the SBP weak form added into a shared-memory residual
// sres[epb][Np][NV] of the CTA's elements e0 .. e0+nloc-1 (reference
// interiorfaceintegrate! / boundaryintegrate! with Subtract: elementL and
// boundary faces subtract, elementR adds).  One pass per local face; in a
// pass thread t handles (element, stencil node) so only stencil nodes do
// work, and no two threads touch the same entry (deterministic, no atomics).
template <int DIM>
__device__ __forceinline__ void face_lift_smem(const DevMesh& md, const double* __restrict__ fflux,
                                               double* sres, const double* sLift, const int* sPerm,
                                               int e0, int nloc) {
  constexpr int NV = DIM + 2;
  constexpr int F = DIM + 1;
  const int Np = md.Np, Nf = md.Nf, S = md.S;
#pragma unroll 1
  for (int f = 0; f < F; ++f) {
    for (int t = threadIdx.x; t < nloc * S; t += blockDim.x) {
      const int le = t / S, s = t - le * S;
      const EFace ef = md.eface[(size_t)(e0 + le) * F + f];
      const double* fl = fflux + (size_t)ef.slot * Nf * NV;
      double acc[NV];
#pragma unroll
      for (int c = 0; c < NV; ++c) acc[c] = 0.0;
      if (md.sparse_face) {
        const int i = ef.side ? md.nbrinv[ef.orient * Nf + s] : s;
        const double a = md.wface[s];
#pragma unroll
        for (int c = 0; c < NV; ++c) acc[c] = a * fl[i * NV + c];
      } else if (ef.side == 0) {
        for (int i = 0; i < Nf; ++i) {
          const double a = sLift[(f * Nf + i) * S + s];
#pragma unroll
          for (int c = 0; c < NV; ++c) acc[c] = fma(a, fl[i * NV + c], acc[c]);
        }
      } else {
        const int* nb = md.nbrperm + ef.orient * Nf;
        for (int i = 0; i < Nf; ++i) {
          const double a = sLift[(f * Nf + nb[i]) * S + s];
#pragma unroll
          for (int c = 0; c < NV; ++c) acc[c] = fma(a, fl[i * NV + c], acc[c]);
        }
      }
      double* r = sres + ((size_t)le * Np + sPerm[f * S + s]) * NV;
      if (ef.side == 0) {
#pragma unroll
        for (int c = 0; c < NV; ++c) r[c] -= acc[c];
      } else {
#pragma unroll
        for (int c = 0; c < NV; ++c) r[c] += acc[c];
      }
    }
    __syncthreads();
  }
}

// What an element kernel does with its residual entries: write them (rk 0),
// or finish a stage of the classical RK4 step in place of separate passes over
// the state (reference rk4.jl:201-330 with pde_post_func: k_s = M^-1 R).  The
// stage's input and output vectors differ, since other elements' face fluxes
// of the stage may still be read from the input.
//   1: acc = k, out = x + c k      2: acc += 2 k, out = x + c k
//   3: out = x + c (acc + k), c = h/6 (out may be x)
struct Epilogue {
  int rk;
  double c;
  const double* Minv;
  const double* x;
  double* acc;
  double* out;
};
// entries [0, n) of the CTA's residual block sres, first entry i0 of the vector
template <int NV>
__device__ __forceinline__ void write_residual(const Epilogue& ep, const double* sres, size_t i0, int n) {
  if (ep.rk == 0) {
    for (int t = threadIdx.x; t < n; t += blockDim.x) ep.out[i0 + t] = sres[t];
    return;
  }
  const double* Mi = ep.Minv + i0 / NV;
  for (int t = threadIdx.x; t < n; t += blockDim.x) {
    const double k = Mi[t / NV] * sres[t];
    const size_t i = i0 + t;
    if (ep.rk == 3) {
      ep.out[i] = ep.x[i] + ep.c * (ep.acc[i] + k);
    } else {
      ep.acc[i] = ep.rk == 1 ? k : ep.acc[i] + 2 * k;
      ep.out[i] = ep.x[i] + ep.c * k;
    }
  }
}

DevMesh dev_mesh(const eg_mesh* m);
int eg_launch_residual(eg_mesh* m, const double* q, double* res);
// face fluxes, then the element kernel with its epilogue
int eg_launch_stage(eg_mesh* m, const double* q, const Epilogue& ep);
// the weak form of a small mesh in one launch (eg_small.cu)
bool eg_small_usable(const eg_mesh* m, const double* q, const Epilogue& ep);
int eg_launch_small(eg_mesh* m, const double* q, const Epilogue& ep);
int eg_launch_split_element(eg_mesh* m, const double* q, const Epilogue& ep, int epb);
// elements per CTA of the element kernel: the mesh's setting, else the built-in choice
int eg_elements_per_cta(const eg_mesh* m);
int eg_launch_norm(eg_mesh* m, const double* r, int strongres, double* out_dev);

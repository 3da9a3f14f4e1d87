// eg_arnoldi.cu -- the restarted GMRES solve of a Newton system (or its
// transpose) as one persistent kernel: all restart cycles, one launch.
//
// The Krylov vectors of the Newton systems are small (1.2 MB in FP32 for the
// 8192-triangle p=3 problem), so an Arnoldi step is bound by the exchanges
// between the blocks and by streaming the operator, not by the vector work:
//   * block b owns a contiguous range of elements (and their rows) for the
//     whole solve, so the Gram-Schmidt updates, the scaling of the new basis
//     vector and the solution update touch only its own rows; work vectors,
//     the older half of its basis and as many element operators as fit are
//     resident in its shared memory;
//   * the face coupling is pushed: the owner of element e forms, for each
//     interface face, the neighbour's coupling block times D_e^-1 v_e and
//     writes it to the neighbour's face side.  With dense faces the two
//     factors are multiplied once per solve (G_e = C D_e^-1, restricted to
//     the unknowns the faces see: 48 x 36 values per SBP-Gamma p=3 triangle
//     instead of 48 x 48 + 3 x 16 x 16), so an apply is one pass without a
//     block barrier; face-diagonal couplings (diagonal-E tetrahedra) are
//     cheaper unmultiplied and keep the two steps;
//   * blocks exchange pushed products and dot-product partials as tagged
//     64-bit words that the reader polls (eg_arnoldi_body.cuh): no grid
//     barrier, and each exchange costs one trip through L2;
//   * every block reduces the dot-product partials in the same order, so the
//     Hessenberg column, the re-orthogonalisation test (DGKS), the Givens
//     rotation and the convergence decision are bit-identical in every block:
//     no broadcast is needed and all blocks take the same branches.  The
//     rotation of column j - 1 runs in one warp while the others push K v_j.
// Every block is resident for the whole solve: a cooperative grid, or, for a
// system whose element blocks take at most 2 MB or whose grid would have at
// most 16 blocks, one thread-block cluster (co-scheduled by the hardware, so
// the small solves of concurrent host threads run side by side).  Waits are
// bounded: a block whose wait runs out raises a flag that the other waits
// sample and leaves without publishing, and the host reports EG_ERR_TIMEOUT.
#include <mutex>

#include "eg_arnoldi_launch.cuh"

// one multi-block persistent solve in flight per device: two grids whose
// blocks wait for one another must never hold parts of the GPU at the same time
std::mutex& eg_coop_mutex(int dev) {
  static std::mutex mu[64];
  return mu[dev & 63];
}

int eg_gmres_tags(eg_ls* ls, bool force) {
  // an iteration uses one push tag and at most two reduction tags, a cycle
  // one of each; a solve has at most itermax + 1 cycles
  const int64_t most = 4 * (int64_t)ls->itermax + 16;
  if (!force && ls->tags + most < (int64_t(1) << 31)) {
    ls->tags += most;
    return EG_OK;
  }
  const eg_mesh* m = ls->lo->mesh;
  const size_t es = ls->lo->prec == EG_F64 ? 8 : 4;
  EG_CUDA(cudaMemsetAsync(ls->cfs, 0, eg_face_tag_bytes(m->I, ls->lo->nb, es), m->stream));
  EG_CUDA(cudaMemsetAsync(ls->tpart, 0, eg_part_tag_bytes(es), m->stream));
  EG_CUDA(cudaMemsetAsync(ls->dflags + F_TAGS, 0, 2 * sizeof(int), m->stream));
  ls->tags = most;
  return EG_OK;
}

int eg_gmres_gave_up(eg_ls* ls) {
  const int rc = eg_gmres_tags(ls, true);
  if (rc != EG_OK) return rc;
  eg_set_error("persistent GMRES: a wait between its blocks ran out");
  return EG_ERR_TIMEOUT;
}

// the whole GMRES solve (all restart cycles) as one launch
int eg_gmres_coop(eg_ls* ls) {
  if (eg_gmres_batching() && eg_gmres_wanted_blocks(ls) > 1) return eg_gmres_coop_batched(ls);
  return ls->lo->prec == EG_F64 ? eg_gmres_launch_f64(ls) : launch_T<float>(ls);
}

bool eg_coop_usable(const eg_ls* ls) {
  const eg_mesh* m = ls->lo->mesh;
  return ls->lo->nb <= NB_MAX && m->F == m->dim + 1 && m->F * m->S <= 64 && m->F * m->Np <= 128 && m->Np <= 128 &&
         m->I > 0 && (m->sparse_face || ls->G) && eg_coop_supported();
}

bool eg_coop_supported() {
  int dev = 0, v = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  if (cudaDeviceGetAttribute(&v, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess) return false;
  return v != 0;
}

// eg_arnoldi_batch.cu -- several problems' persistent GMRES solves in one
// cooperative launch (the batched counterpart of eg_arnoldi.cu).
//
// When batching is on (eg_set_gmres_batching), a thread that reaches the
// Krylov solve of its Newton iteration hands the solve to a per-device
// batcher instead of launching it, if the solve runs on several blocks (a
// one-block solve is launched at once: one-block grids of several threads
// already share the GPU without waiting for each other).  The solves handed in within a short
// window (or as soon as every thread inside eg_newton_solve has handed one in)
// go out as one cooperative grid walking a work list: each problem gets a
// contiguous range of blocks (at most one block per SM in total, more blocks
// for larger operators) and runs the same device function as the
// single-problem kernel, whose blocks exchange data through the problem's own
// tagged words.  Several problems then share the GPU inside one launch instead of
// queueing for it one multi-block grid at a time.
//
// Every block of a cooperative launch is resident, so the waits between a
// problem's blocks always end; each is bounded all the same, and a solve with a
// wait that ran out says so in its flags: its caller returns EG_ERR_TIMEOUT.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <mutex>
#include <vector>

#include "eg_arnoldi_batch.cuh"

// k_gmres_batch<double> (eg_arnoldi_batch_f64.cu)
const void* eg_gmres_batch_kernel_f64();

namespace {

// ------------------------------------------------------------------ batcher
struct Submission {
  eg_ls* ls;
  int rc = EG_OK;
  bool done = false;
};

struct Batcher {
  std::mutex mu;
  std::condition_variable cv;
  std::vector<Submission*> pending;
  std::chrono::steady_clock::time_point first;  // oldest pending hand-in
  bool launching = false;
  cudaStream_t stream = nullptr;  // the batched grids' stream
  std::atomic<int> active{0};     // threads inside eg_newton_solve with a
                                  // multi-block Krylov solve
};

Batcher& batcher(int dev) {
  static Batcher b[64];
  return b[dev & 63];
}

std::atomic<int> g_batching{0};
std::atomic<long long> g_window_ns{50000};

int ensure_batcher(Batcher& B) {
  if (B.stream) return EG_OK;
  cudaError_t e = cudaStreamCreateWithFlags(&B.stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) return eg_cuda_fail(e, "GMRES batcher");
  return EG_OK;
}

// blocks of one problem: what the single-problem launcher gives it (one block
// for operators of at most 2 MB, else up to one block per SM with at least 32
// elements each).  A batch never shrinks a problem's share: the block
// partition fixes the order of the dot-product reductions, so a solve gives
// the same bits in any batch and alone.
int wanted_blocks_sms(const eg_ls* ls, int sms) {
  const eg_mesh* m = ls->lo->mesh;
  const size_t es = ls->lo->prec == EG_F64 ? 8 : 4;
  const size_t op = (size_t)m->E * ls->lo->n * ls->lo->n * es;
  // the block count of the same solve alone (eg_arnoldi.cu), so a batched
  // solve keeps its partition and gives the same bits: one (a small system,
  // solved by a cluster and never batched), the cluster's blocks for at most
  // 16 x 32 elements, else one block per SM
  const int chunks = (m->E + 31) / 32;
  int nb = op <= (size_t(2) << 20) ? 1
           : chunks <= EG_GMRES_CLUSTER_BLOCKS ? std::max(2, chunks)
                                               : std::max(2, std::min(sms, m->E));
  nb = std::min(nb, m->E);
  return std::min(nb, EG_COOP_MAX_BLOCKS);
}

template <typename T>
const void* batch_kernel() {
  if constexpr (sizeof(T) == 8)
    return eg_gmres_batch_kernel_f64();
  else
    return (const void*)k_gmres_batch<T>;
}

// a block of the batched kernel is resident with the largest shared memory
// (asked of the runtime once per device; loads the kernel)
template <typename T>
bool batch_kernel_fits() {
  return launch_fact(batch_kernel<T>(), 0, []() {
    int per_sm = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_kernel<T>(), NT, kSmemBudget) ==
               cudaSuccess && per_sm >= 1;
  });
}

template <typename T>
int launch_batch(Batcher& B, const std::vector<Submission*>& batch, int dev) {
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  std::vector<int> nb(batch.size());
  for (size_t i = 0; i < batch.size(); ++i) nb[i] = wanted_blocks_sms(batch[i]->ls, sms);
  BatchList list;
  list.n = (int)batch.size();
  int b0 = 0;
  size_t smem = 0;
  for (size_t i = 0; i < batch.size(); ++i) {
    const eg_ls* ls = batch[i]->ls;
    CoopArgs<T> a = *reinterpret_cast<const CoopArgs<T>*>(ls->hargs);
    smem = std::max(smem, plan_smem(a, nb[i]));
    list.e[i] = BatchEntry{ls->dargs, b0, nb[i], gmres_kind(ls), a.ec, a.fs_smem, a.ws, a.p0_smem, a.kv, a.er, a.ef0};
    b0 += nb[i];
  }
  const void* fn = batch_kernel<T>();
  if (!batch_kernel_fits<T>() || b0 > sms) {
    eg_set_error("batched GMRES kernel cannot be resident");
    return EG_ERR_UNSUPPORTED;
  }
  std::lock_guard<std::mutex> lock(eg_coop_mutex(dev));
  for (Submission* s : batch) EG_CUDA(cudaStreamWaitEvent(B.stream, s->ls->ev_in, 0));
  void* args[] = {&list};
  EG_CUDA(cudaLaunchCooperativeKernel(fn, dim3(b0), dim3(NT), args, smem, B.stream));
  EG_CUDA(cudaStreamSynchronize(B.stream));  // the grid has finished before the next one starts
  batch[0]->ls->lo->mesh->launches += 1;
  return EG_OK;
}

template <typename T>
int stage_args(eg_ls* ls) {
  eg_mesh* m = ls->lo->mesh;
  const int rc = eg_gmres_tags(ls);
  if (rc != EG_OK) return rc;
  if (!ls->dargs) {
    cudaError_t e = cudaMalloc(&ls->dargs, sizeof(CoopArgs<double>));
    if (e == cudaSuccess) e = cudaMallocHost(&ls->hargs, sizeof(CoopArgs<double>));
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ls->ev_in, cudaEventDisableTiming);
    if (e != cudaSuccess) return eg_cuda_fail(e, "batched GMRES set-up");
  }
  // the staging buffer is the solver's own and its previous copy has
  // completed (every Newton iteration synchronises the mesh stream)
  coop_args<T>(ls, reinterpret_cast<CoopArgs<T>*>(ls->hargs));
  EG_CUDA(cudaMemcpyAsync(ls->dargs, ls->hargs, sizeof(CoopArgs<T>), cudaMemcpyHostToDevice, m->stream));
  EG_CUDA(cudaEventRecord(ls->ev_in, m->stream));
  return EG_OK;
}

}  // namespace

bool eg_gmres_batching() { return g_batching.load() != 0; }

int eg_gmres_wanted_blocks(const eg_ls* ls) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return wanted_blocks_sms(ls, sms);
}

void eg_batch_enter(int dev) { batcher(dev).active.fetch_add(1); }
void eg_batch_leave(int dev) { batcher(dev).active.fetch_sub(1); }

int eg_gmres_coop_batched(eg_ls* ls) {
  const bool f64 = ls->lo->prec == EG_F64;
  int st = f64 ? stage_args<double>(ls) : stage_args<float>(ls);
  if (st != EG_OK) return st;
  int dev = 0;
  cudaGetDevice(&dev);
  Batcher& B = batcher(dev);
  Submission sub;
  sub.ls = ls;
  std::unique_lock<std::mutex> lk(B.mu);
  st = ensure_batcher(B);
  if (st != EG_OK) return st;
  if (B.pending.empty()) B.first = std::chrono::steady_clock::now();
  B.pending.push_back(&sub);
  B.cv.notify_all();
  while (!sub.done) {
    const auto now = std::chrono::steady_clock::now();
    const bool full = (int)B.pending.size() >= std::max(1, B.active.load()) ||
                      (int)B.pending.size() >= kMaxBatch;
    const bool late = std::chrono::duration_cast<std::chrono::nanoseconds>(now - B.first).count() >=
                      g_window_ns.load();
    if (!B.launching && !B.pending.empty() && (full || late)) {
      // lead: pack pending solves of the first one's precision, in arrival
      // order, while their blocks fit on the SMs (first fit; the others wait
      // for the next launch)
      B.launching = true;
      int sms = 0;
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      const int prec = B.pending[0]->ls->lo->prec;
      std::vector<Submission*> batch, rest;
      int used = 0;
      for (Submission* s : B.pending) {
        const int w = wanted_blocks_sms(s->ls, sms);
        if (s->ls->lo->prec == prec && (int)batch.size() < kMaxBatch && used + w <= sms) {
          batch.push_back(s);
          used += w;
        } else {
          rest.push_back(s);
        }
      }
      B.pending.swap(rest);
      if (!B.pending.empty()) B.first = now;
      lk.unlock();
      const int rc = prec == EG_F64 ? launch_batch<double>(B, batch, dev) : launch_batch<float>(B, batch, dev);
      lk.lock();
      for (Submission* s : batch) {
        s->rc = rc;
        s->done = true;
      }
      B.launching = false;
      B.cv.notify_all();
    } else {
      B.cv.wait_for(lk, std::chrono::microseconds(20));
    }
  }
  return sub.rc;
}

extern "C" int eg_set_gmres_batching(int32_t enable, double window_us) {
  if ((enable != 0 && enable != 1) || !(window_us >= 0.0)) {
    eg_set_error("eg_set_gmres_batching: enable in {0, 1}, window_us >= 0");
    return EG_ERR_INVALID;
  }
  g_window_ns.store((long long)(window_us * 1000.0));
  if (enable) {
    // the current device's batcher is set up here (stream, both batched
    // kernels loaded), not by the first solve that is handed in
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) {
      Batcher& B = batcher(dev);
      std::lock_guard<std::mutex> lk(B.mu);
      if (ensure_batcher(B) == EG_OK) {
        batch_kernel_fits<float>();
        batch_kernel_fits<double>();
      }
    }
    cudaGetLastError();
  }
  g_batching.store(enable);
  return EG_OK;
}

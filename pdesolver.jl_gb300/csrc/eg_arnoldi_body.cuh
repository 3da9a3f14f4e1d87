// eg_arnoldi_body.cuh -- the persistent GMRES solve as a device function,
// shared by the single-problem launches (eg_arnoldi.cu: a cooperative grid or
// one thread-block cluster) and the batched kernel that runs several
// problems' solves in one launch (eg_arnoldi_batch.cu).  The algorithm and
// its data flow are described in eg_arnoldi.cu.
#pragma once
#include <map>
#include <mutex>
#include <tuple>

#include "eg_internal.h"
#include "eg_kernels.cuh"
#include "eg_krylov.cuh"
#include "eg_linalg.h"

namespace {

constexpr int NT = 1024;  // one block per SM
constexpr int NB_MAX = 64;  // coupling-block rows handled by the face-side pass
// systems whose element blocks take at most this many bytes run on one cluster
constexpr size_t kSmallOperatorBytes = size_t(2) << 20;
constexpr int kLine = 16;  // words of a 128-byte line
// dynamic shared memory of a block (227 KB less the static part)
constexpr size_t kSmemBudget = 208 * 1024, kSmemStream = 176 * 1024;

template <typename T>
struct CoopArgs {
  DevMesh md;
  const T* inv;      // [E][n][n] block inverses (column-major)
  const T* diag;     // [E][n][n] element blocks of J (column-major)
  const T* cpl;      // [I][2][nb][nb] coupling blocks (row-major), or
                     // [I][2][S][NV][NV] when md.sparse_face (face-diagonal)
  const int* spos;   // [F][Np]
  const int* fside;  // [E][F] coupling block of each element face, or -1
  T* G;              // [E][n+1][Rp] pushed operator C D^-1 of each element (dense faces)
  uint64_t* msg;     // [I][2][nbp] tagged coupling products of each face side
  uint64_t* part;    // [2][33][nblk] tagged partial sums
  uint64_t* tot;     // [2][33] tagged sums, one L2 line each (grids above kDirect blocks)
  unsigned int* ep;  // [2] last tags used: pushes, reductions
  const T* bvec;     // [N] right-hand side
  T* x;              // [N] solution (in: initial guess)
  T* V;              // basis v_0 .. v_m and w, block-local: vector k of block b at
                     // (m+2)(e0 nbd (rounded up to 4) + 4 b) + k nrowp
  T* w;              // [N] scratch, natural rows
  T* vint;           // [N] interior rows of v_0
  int* flags;
  double* scal;
  int m, n, E;
  int trans;         // solve J^T x = b
  int l2ef;          // operator + basis exceed L2: operator loads marked evict-first
                     // (dense faces: those of the elements le >= ef0)
  int ef0;
  int nb, nbp, Rp;   // rows of a face side, padded to 4; rows of an element's pushes F nbp
  int nbn;           // nodes on some face stencil (dense faces; all Np with face-diagonal ones)
  int S, F, nv;
  int polls;         // polls of one wait before its block gives up
  // shared-memory plan of the launch (plan_smem)
  int ec;            // elements of a staged chunk (face-diagonal operators)
  int fs_smem, ws, p0_smem;  // face table, work vectors, interior products in shared memory
  int kv;            // basis vectors in shared memory
  int er;            // elements whose pushed operator is resident in shared memory
  int64_t N;
};

// vector type for the streaming passes over a block's rows: 16-byte loads
template <typename T> struct Vec;
template <> struct Vec<float> {
  using V = float4;
  static constexpr int W = 4;
  __device__ static float dot(V a, V b) { return a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w; }
  __device__ static V fma(V a, float h, V c) {
    return make_float4(c.x - a.x * h, c.y - a.y * h, c.z - a.z * h, c.w - a.w * h);
  }
  __device__ static void axpy(V a, float h, V& c) {
    c.x += a.x * h; c.y += a.y * h; c.z += a.z * h; c.w += a.w * h;
  }
  __device__ static V scale(V a, float s) { return make_float4(a.x * s, a.y * s, a.z * s, a.w * s); }
  __device__ static V zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
};
template <> struct Vec<double> {
  using V = double2;
  static constexpr int W = 2;
  __device__ static double dot(V a, V b) { return a.x * b.x + a.y * b.y; }
  __device__ static V fma(V a, double h, V c) { return make_double2(c.x - a.x * h, c.y - a.y * h); }
  __device__ static void axpy(V a, double h, V& c) { c.x += a.x * h; c.y += a.y * h; }
  __device__ static V scale(V a, double s) { return make_double2(a.x * s, a.y * s); }
  __device__ static V zero() { return make_double2(0.0, 0.0); }
};

// ------------------------------------------------------------ tagged words
// Data that crosses blocks travels as 64-bit words {tag, 32 bits of the
// value} (one word for a float, two for a double).  A reader polls the word
// it needs until the tag is that of the phase, so no barrier, fence or
// separate flag stands between producer and consumer: one trip through L2
// instead of three (store, barrier, load).  64-bit accesses are single-copy
// atomic, and every word carries its own tag, so no order between words is
// relied on.  Tags only grow (ep keeps them between solves).
template <typename T>
constexpr int kWords = sizeof(T) / 4;

__device__ __forceinline__ void st2(uint64_t* p, uint64_t a, uint64_t b) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void msg_put(uint64_t* p, float v, unsigned tag) {
  const uint64_t w = ((uint64_t)tag << 32) | (uint64_t)__float_as_uint(v);
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ void msg_put(uint64_t* p, double v, unsigned tag) {
  const uint64_t t = (uint64_t)tag << 32;
  st2(p, t | (uint64_t)(unsigned)__double2loint(v), t | (uint64_t)(unsigned)__double2hiint(v));
}
// the W values of a 16-byte unit
__device__ __forceinline__ void msg_put_v(uint64_t* p, float4 v, unsigned tag) {
  const uint64_t t = (uint64_t)tag << 32;
  st2(p, t | (uint64_t)__float_as_uint(v.x), t | (uint64_t)__float_as_uint(v.y));
  st2(p + 2, t | (uint64_t)__float_as_uint(v.z), t | (uint64_t)__float_as_uint(v.w));
}
__device__ __forceinline__ void msg_put_v(uint64_t* p, double2 v, unsigned tag) {
  msg_put(p, v.x, tag);
  msg_put(p + 2, v.y, tag);
}
__device__ __forceinline__ bool msg_get(const uint64_t* p, unsigned tag, float& v) {
  uint64_t w;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
  v = __uint_as_float((unsigned)w);
  return (unsigned)(w >> 32) == tag;
}
__device__ __forceinline__ bool msg_get(const uint64_t* p, unsigned tag, double& v) {
  uint64_t a, b;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
  v = __hiloint2double((int)(unsigned)b, (int)(unsigned)a);
  return (unsigned)(a >> 32) == tag && (unsigned)(b >> 32) == tag;
}

// NV consecutive values of a coupling row (16-byte loads for 2-D FP32)
template <int NV, typename T>
__device__ __forceinline__ void load_row_piece(const T* __restrict__ p, T* out) {
  if constexpr (NV == 4 && sizeof(T) == 4) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
  } else {
#pragma unroll
    for (int b = 0; b < NV; ++b) out[b] = p[b];
  }
}

// Loads of the operator with an L2 evict-first policy: the operator is
// streamed once per Arnoldi iteration, and its lines should leave L2 before
// the Krylov basis, which every Gram-Schmidt pass reads again.
__device__ __forceinline__ uint64_t l2_evict_first() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ float ld_ef(const float* p, uint64_t pol) {
  float v;
  asm("ld.global.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ double ld_ef(const double* p, uint64_t pol) {
  double v;
  asm("ld.global.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ float4 ld_ef(const float4* p, uint64_t pol) {
  float4 v;
  asm("ld.global.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ double2 ld_ef(const double2* p, uint64_t pol) {
  double2 v;
  asm("ld.global.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;" : "=d"(v.x), "=d"(v.y) : "l"(p), "l"(pol));
  return v;
}
// row r of A xe with U column loads in flight (the streamed inverse blocks of
// the face-diagonal operators): the batches are explicit, so the loads in
// flight do not depend on how the register allocator unrolls the row
template <int NB, bool EF, typename T>
__device__ __forceinline__ T block_row_stream(const T* A, const T* xe, int r, int n, uint64_t pol) {
  constexpr int U = sizeof(T) == 4 ? (NB == 115 ? 23 : 10) : 10;
  T acc0 = T(0), acc1 = T(0);
  const int nc = NB > 0 ? NB : n;
  const T* p = A + r;
  int c = 0;
#pragma unroll 1
  for (; c + U <= nc; c += U) {
    T g[U];
#pragma unroll
    for (int u = 0; u < U; ++u) g[u] = EF ? ld_ef(p + (size_t)u * nc, pol) : p[(size_t)u * nc];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u & 1) acc1 += g[u] * xe[c + u];
      else acc0 += g[u] * xe[c + u];
    }
    p += (size_t)U * nc;
  }
  for (; c < nc; ++c, p += nc) acc0 += *p * xe[c];
  return acc0 + acc1;
}

// row r of A^T xe: column r of the column-major block
template <typename T>
__device__ __forceinline__ T block_col(const T* __restrict__ A, const T* __restrict__ xe, int r, int n) {
  const T* c = A + (size_t)r * n;
  T acc0 = T(0), acc1 = T(0);
  int i = 0;
#pragma unroll 4
  for (; i + 1 < n; i += 2) {
    acc0 += c[i] * xe[i];
    acc1 += c[i + 1] * xe[i + 1];
  }
  if (i < n) acc0 += c[i] * xe[i];
  return acc0 + acc1;
}

__device__ __forceinline__ float wsum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double wsum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// block-level state of the persistent GMRES (static shared memory of the
// kernel that runs it)
template <typename T>
struct GmresShared {
  int sPerm[64], sSpos[128];
  int sOrd[128];  // nodes, face-stencil nodes first
  T sh1[33], sh2[33];
  T sal[33];      // interior part of v_k = sal[k] * vint
  T scs[32], ssn[32], sg[33], syT[33];
  T sR[32 * 33];  // rotated Hessenberg columns: sR[j * (m+1) + k]
  // the same in FP64: columns for the back substitution; transposed FP32 solves
  // rotate in FP64 throughout
  double sRd[sizeof(T) == 4 ? 32 * 33 : 1];
  double dcs[sizeof(T) == 4 ? 32 : 1], dsn[sizeof(T) == 4 ? 32 : 1], dg[sizeof(T) == 4 ? 33 : 1];
  int s_done, s_its, s_jdone, s_conv, s_cycles, s_nreorth, s_err, s_reorth;
  T s_beta, s_g0, s_hn, s_inv, s_a1;
  double s_tol, s_bnorm;
};

// columns of the pushed operator of the compiled block sizes: the unknowns
// of the face-stencil nodes (2-D SBP-Gamma: 7, 12, 18 nodes with 6, 9, 12 on
// the boundary; the other operators: all nodes)
template <int DIM, int NB>
constexpr int kCols = DIM == 2 ? (NB == 28 ? 24 : NB == 48 ? 36 : NB == 72 ? 48 : NB) : NB;

// What a block of the solve knows about itself.
template <typename T>
struct BlockView {
  int b, nblk, e0, nel;
  int nbd;        // Krylov unknowns per element
  int nrow, nrowp;
  T* cur;         // v_j (own rows)
  T* sw;          // w (own rows)
  T* sV;          // basis vectors 0 .. kv-1
  T* gV;          // basis in global memory (block-local)
  T* sG;          // resident pushed operators
  T* sP0;         // interior products
  T* sZ;          // staged chunk (face-diagonal operators)
  const int* fs;  // [nel][F] face table
};

template <typename T>
__device__ __forceinline__ T* basis(const CoopArgs<T>& a, const BlockView<T>& v, int k) {
  return k < a.kv ? v.sV + (size_t)k * v.nrowp : v.gV + (size_t)k * v.nrowp;
}

// ------------------------------------------------------------- reductions
// Up to kDirect blocks, warp k of every block polls and sums the blocks'
// words of partial k in block order.  In a larger grid that is 152 x 152 words
// per partial and the polling delays the writers (20.9 against 18.1 us per
// iteration of the 8192-triangle p=3 system, 11.4 against 8.1 us at p=1), so
// block k (nblk / 33) collects partial k from all blocks and publishes the
// sum: two trips through L2.  Buffers alternate: a block publishes reduction
// t + 2 only after it has the sums of t + 1, to which every block contributed
// after reading those of t.
constexpr int kDirect = 32;

// After a poll that failed: true when the wait is over without its word.  The
// wait that runs out of polls raises flags[F_GAVE_UP], which every wait samples,
// so all blocks leave.  s_err is the block's own flag: its threads wait no more,
// return after the next barrier and publish nothing that depends on the missing
// word, so every word that carries its tag is a good one.  (A flag in shared
// memory, and the rare part out of line: as a vote of the barrier and inlined,
// spills made 8,192 triangles Omega p=2 12 % slower.)
__device__ __noinline__ bool give_up_now(volatile int* gave_up, bool out, volatile int* s_err) {
  if (out) *gave_up = 1;
  if (*gave_up) *s_err = 1;
  return *s_err != 0;
}
template <typename T>
__device__ __forceinline__ bool give_up(const CoopArgs<T>& a, int& polls, int* s_err) {
  ++polls;
  return ((polls & 255) == 0 || polls > a.polls) && give_up_now(a.flags + F_GAVE_UP, polls > a.polls, s_err);
}

// poll one word until it carries the tag
template <typename T>
__device__ __forceinline__ T word_wait(const CoopArgs<T>& a, const uint64_t* p, unsigned tag, int* s_err) {
  T val;
  int polls = 0;
  while (!msg_get(p, tag, val))
    if (give_up(a, polls, s_err)) break;
  return val;
}
// publish this block's partial k of reduction `tag` (lane 0 of a warp)
template <typename T>
__device__ __forceinline__ void part_put(const CoopArgs<T>& a, const BlockView<T>& v, int k, T val, unsigned tag) {
  if ((threadIdx.x & 31) == 0)
    msg_put(a.part + (size_t)(((tag & 1) * 33 + k) * v.nblk + v.b) * kWords<T>, val, tag);
}
// out[k] = sum over the blocks of partial k < cnt, the same bits in every block
template <typename T>
__device__ __forceinline__ void part_sum(const CoopArgs<T>& a, const BlockView<T>& v, int cnt, T* out, unsigned tag,
                                         int* s_err) {
  const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
  if (v.nblk <= kDirect) {
    if (k >= cnt) return;
    const uint64_t* p = a.part + (size_t)((tag & 1) * 33 + k) * v.nblk * kWords<T>;
    T acc = T(0);
    for (int r = lane; r < v.nblk; r += 32) acc += word_wait(a, p + r * kWords<T>, tag, s_err);
    acc = wsum(acc);
    if (lane == 0) out[k] = acc;
    return;
  }
  if (k < cnt && v.b == k * (v.nblk / 33)) {
    const uint64_t* p = a.part + (size_t)((tag & 1) * 33 + k) * v.nblk * kWords<T>;
    T acc = T(0);
    int polls = 0;
    constexpr int U = 5;
    for (int b0 = lane; b0 < v.nblk; b0 += 32 * U) {
      T val[U];
      bool all;
      do {
        all = true;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          val[u] = T(0);
          if (b0 + 32 * u < v.nblk) all &= msg_get(p + (size_t)(b0 + 32 * u) * kWords<T>, tag, val[u]);
        }
        if (!all && give_up(a, polls, s_err)) break;
      } while (!all);
#pragma unroll
      for (int u = 0; u < U; ++u) acc += val[u];
    }
    acc = wsum(acc);
    __syncwarp();
    if (lane == 0 && !*(volatile int*)s_err) msg_put(a.tot + (size_t)((tag & 1) * 33 + k) * kLine, acc, tag);
  }
  if (k == 31 && lane < cnt)
    out[lane] = word_wait(a, a.tot + (size_t)((tag & 1) * 33 + lane) * kLine, tag, s_err);
}

// partial dots of the block's rows against x: warp k < cnt takes V[k] (plus
// add[k] in block 0), warp cnt takes x.x; published as reduction `tag`
template <typename T>
__device__ __forceinline__ void dots_put(const CoopArgs<T>& a, const BlockView<T>& v, const T* x, int cnt, T a1, T g0,
                                         const T* al, unsigned tag) {
  using VT = Vec<T>;
  using VV = typename VT::V;
  const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
  if (k > cnt) return;
  const VV* v4 = reinterpret_cast<const VV*>(k < cnt ? basis(a, v, k) : x);
  const VV* x4 = reinterpret_cast<const VV*>(x);
  const int n4 = v.nrowp / VT::W;
  T acc0 = T(0), acc1 = T(0), acc2 = T(0), acc3 = T(0);
  int i = lane;
  for (; i + 96 < n4; i += 128) {
    const VV a0 = v4[i], a1v = v4[i + 32], a2 = v4[i + 64], a3 = v4[i + 96];
    const VV b0 = x4[i], b1 = x4[i + 32], b2 = x4[i + 64], b3 = x4[i + 96];
    acc0 += VT::dot(a0, b0);
    acc1 += VT::dot(a1v, b1);
    acc2 += VT::dot(a2, b2);
    acc3 += VT::dot(a3, b3);
  }
  for (; i < n4; i += 32) acc0 += VT::dot(v4[i], x4[i]);
  T acc = wsum((acc0 + acc1) + (acc2 + acc3));
  // second pass: the interior part -a1 vint of w' (block 0 adds it once)
  if (v.b == 0 && a1 != T(0)) acc += (k < cnt ? -a1 * al[k] : a1 * a1) * g0;
  part_put(a, v, k, acc, tag);
}

// y = (x - sum_{k<cnt} V[k] h[k]) s on the block's rows, to y0 and y1
template <typename T>
__device__ __forceinline__ void sub_scale(const CoopArgs<T>& a, const BlockView<T>& v, const T* h, int cnt, const T* x,
                                          T s, T* y0, T* y1) {
  using VT = Vec<T>;
  using VV = typename VT::V;
  const int n4 = v.nrowp / VT::W;
  for (int i = threadIdx.x; i < n4; i += NT) {
    VV acc = reinterpret_cast<const VV*>(x)[i];
    auto part = [&](const T* base, int k0, int k1) {
      const VV* p = reinterpret_cast<const VV*>(base) + i;
      const int ld = v.nrowp / VT::W;
      int k = k0;
      for (; k + 4 <= k1; k += 4) {
        const VV v0 = p[(size_t)k * ld], v1 = p[(size_t)(k + 1) * ld];
        const VV v2 = p[(size_t)(k + 2) * ld], v3 = p[(size_t)(k + 3) * ld];
        acc = VT::fma(v0, h[k], acc);
        acc = VT::fma(v1, h[k + 1], acc);
        acc = VT::fma(v2, h[k + 2], acc);
        acc = VT::fma(v3, h[k + 3], acc);
      }
      for (; k < k1; ++k) acc = VT::fma(p[(size_t)k * ld], h[k], acc);
    };
    part(v.sV, 0, min(cnt, a.kv));
    part(v.gV, min(cnt, a.kv), cnt);
    acc = VT::scale(acc, s);
    reinterpret_cast<VV*>(y0)[i] = acc;
    if (y1 != y0) reinterpret_cast<VV*>(y1)[i] = acc;
  }
}

// ---------------------------------------------------------------- pushes
// Coupling C x (transposed: C^T x) of the own elements' values x (natural
// rows, x[le n + r]) to the neighbours' face sides.  t = (element, face, row).
template <int DIM, typename T>
__device__ __forceinline__ void couple_push(const CoopArgs<T>& a, const BlockView<T>& v, const T* x, int c0, int nl,
                                            const int* sPerm, unsigned tag, uint64_t pol) {
  constexpr int NV = DIM + 2;
  const int nb = a.nb, F = a.F, S = a.S, n = a.n;
  const int per = a.Rp;
  for (int t = threadIdx.x; t < nl * per; t += NT) {
    const int le = t / per, q = t - le * per;
    const int f = q / a.nbp, i = q - f * a.nbp;
    const int fs = v.fs[(c0 + le) * F + f];
    if (fs < 0 || i >= nb) continue;
    const int tgt = fs ^ 1;
    const T* xs = x + (size_t)le * n;
    const int* pf = sPerm + f * S;
    T acc0 = T(0), acc1 = T(0);
    if (a.md.sparse_face) {
      // face-diagonal coupling: row (s, r) of the neighbour's side couples to
      // this element's node facing s only (transposed: the facing row's
      // column r)
      const int s = i / NV, r = i - s * NV;
      const int o = a.md.ifaces[5 * (tgt >> 1) + 4];
      const int se = ((tgt & 1) ? a.md.nbrinv : a.md.nbrperm)[o * a.md.Nf + s];
      const T* z = xs + pf[se] * NV;
      if (a.trans) {
        const T* C = a.cpl + ((size_t)fs * S + se) * NV * NV + r;
#pragma unroll
        for (int c = 0; c < NV; ++c) acc0 += C[c * NV] * z[c];
      } else {
        const T* C = a.cpl + (size_t)tgt * nb * NV + (size_t)i * NV;
        if (a.l2ef) {
#pragma unroll
          for (int c = 0; c < NV; ++c) acc0 += ld_ef(C + c, pol) * z[c];
        } else {
#pragma unroll
          for (int c = 0; c < NV; ++c) acc0 += C[c] * z[c];
        }
      }
    } else if (a.trans) {
      const T* C = a.cpl + (size_t)fs * nb * nb + i;
      for (int sp = 0; sp < S; ++sp) {
        const T* z = xs + pf[sp] * NV;
#pragma unroll
        for (int c = 0; c < NV; ++c) acc0 += C[(size_t)(sp * NV + c) * nb] * z[c];
      }
    } else {
      const T* C = a.cpl + ((size_t)tgt * nb + i) * nb;
      for (int sp = 0; sp < S; ++sp) {
        T c[NV];
        load_row_piece<NV, T>(C + sp * NV, c);
        const T* z = xs + pf[sp] * NV;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
          if (k & 1) acc1 += c[k] * z[k];
          else acc0 += c[k] * z[k];
        }
      }
    }
    msg_put(a.msg + ((size_t)tgt * a.nbp + i) * kWords<T>, acc0 + acc1, tag);
  }
}

// W rows of the pushed operator of one element times its v (NC columns in
// groups, all loads of a group in flight)
template <int NC, bool EF, typename T>
__device__ __forceinline__ typename Vec<T>::V push_rows(const T* G, const T* ve, int ncol, int Rp, uint64_t pol) {
  using VT = Vec<T>;
  using VV = typename VT::V;
  constexpr int U = sizeof(T) == 4 ? 6 : 4;
  VV acc = VT::zero();
  int c = 0;
  const int nc = NC > 0 ? NC : ncol;
#pragma unroll 1
  for (; c + U <= nc; c += U) {
    VV g[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const VV* p = reinterpret_cast<const VV*>(G + (size_t)(c + u) * Rp);
      g[u] = EF ? ld_ef(p, pol) : *p;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) VT::axpy(g[u], ve[c + u], acc);
  }
  for (; c < nc; ++c) VT::axpy(*reinterpret_cast<const VV*>(G + (size_t)c * Rp), ve[c], acc);
  return acc;
}

// K v_j of the own elements, pushed to the neighbours' face sides, by
// threads t0 .. NT-1.  Dense faces: the pushed operator G_e = C D_e^-1 (rows:
// the F face sides, columns: the face-stencil unknowns) times v_e, plus
// al = the coefficient of the interior part times its products.
template <int DIM, int NB, typename T>
__device__ __forceinline__ void apply_push(const CoopArgs<T>& a, const BlockView<T>& v, const T* vj, T al,
                                           const int* sPerm, unsigned tag, int t0, uint64_t pol) {
  if (a.md.sparse_face) {
    const int n = NB > 0 ? NB : a.n;
    for (int c0 = 0; c0 < v.nel; c0 += a.ec) {
      const int nl = min(a.ec, v.nel - c0);
      for (int t = threadIdx.x; t < nl * n; t += NT) {
        const int le = t / n, r = t - le * n;
        const T* A = a.inv + (size_t)(v.e0 + c0 + le) * n * n;
        const T* ve = vj + (size_t)(c0 + le) * n;
        v.sZ[t] = a.trans ? block_col<T>(A, ve, r, n)
                  : a.l2ef ? block_row_stream<NB, true, T>(A, ve, r, n, pol)
                           : block_row_stream<NB, false, T>(A, ve, r, n, pol);
      }
      __syncthreads();
      couple_push<DIM, T>(a, v, v.sZ, c0, nl, sPerm, tag, pol);
      __syncthreads();
    }
    return;
  }
  using VT = Vec<T>;
  using VV = typename VT::V;
  constexpr int NC = kCols<DIM, NB>;
  constexpr int W = VT::W;
  const int nbd = NC > 0 ? NC : v.nbd;
  const int Rp = a.Rp, ng = Rp / W;
  const size_t gs = (size_t)(a.n + 1) * Rp;
  for (int t = threadIdx.x - t0; t < v.nel * ng; t += NT - t0) {
    if (t < 0) break;
    const int le = t / ng, row = (t - le * ng) * W;
    const int f = row / a.nbp, i = row - f * a.nbp;
    const int fs = v.fs[le * a.F + f];
    if (fs < 0 || i >= a.nb) continue;
    const T* ve = vj + (size_t)le * nbd;
    const T* Gg = a.G + (size_t)(v.e0 + le) * gs;
    VV acc = le < a.er ? push_rows<NC, false, T>(v.sG + (size_t)le * nbd * Rp + row, ve, nbd, Rp, pol)
             : le >= a.ef0 ? push_rows<NC, true, T>(Gg + row, ve, nbd, Rp, pol)
                       : push_rows<NC, false, T>(Gg + row, ve, nbd, Rp, pol);
    if (nbd < a.n) {
      const T* p0 = a.p0_smem ? v.sP0 + (size_t)le * Rp + row : Gg + (size_t)a.n * Rp + row;
      VT::axpy(*reinterpret_cast<const VV*>(p0), al, acc);
    }
    uint64_t* dst = a.msg + ((size_t)(fs ^ 1) * a.nbp + i) * kWords<T>;
    msg_put_v(dst, acc, tag);  // nbp is a multiple of W: padded rows are never read
  }
}

// The pushed operators of the own elements (dense faces):
//   G[q][f nbp + i] = sum_(s,c) C(tgt)[i][(s,c)] D^-1[(perm_f(s),c)][col(q)]
// (transposed: C(own)^T and D^-T), columns in the order of sOrd (face-stencil
// nodes first).  One thread forms the NV columns of a node of one row.
template <int DIM, typename T>
__device__ __forceinline__ void build_push_operator(const CoopArgs<T>& a, const BlockView<T>& v, const int* sPerm,
                                                    const int* sOrd) {
  constexpr int NV = DIM + 2;
  const int Np = a.md.Np, n = a.n, S = a.S, nb = a.nb, Rp = a.Rp;
  const size_t gs = (size_t)(n + 1) * Rp;
  const int per = Np * Rp;
  for (int t = threadIdx.x; t < v.nel * per; t += NT) {
    const int le = t / per, q = t - le * per;
    const int jn = q / Rp, row = q - jn * Rp;
    const int f = row / a.nbp, i = row - f * a.nbp;
    const int fs = v.fs[le * a.F + f];
    const int node = sOrd[jn];
    T acc[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[k] = T(0);
    if (fs >= 0 && i < nb) {
      const T* A = a.inv + (size_t)(v.e0 + le) * n * n;
      const int* pf = sPerm + f * S;
      for (int s = 0; s < S; ++s) {
        T c[NV];
        if (a.trans) {
#pragma unroll
          for (int k = 0; k < NV; ++k) c[k] = a.cpl[((size_t)fs * nb + s * NV + k) * nb + i];
        } else {
          load_row_piece<NV, T>(a.cpl + ((size_t)(fs ^ 1) * nb + i) * nb + s * NV, c);
        }
        const int r = pf[s] * NV;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
          T z[NV];
          if (a.trans) {
            // D^-T[(r + l)][node NV + k] = inv column r + l, row node NV + k
#pragma unroll
            for (int l = 0; l < NV; ++l) z[l] = A[(size_t)(r + l) * n + node * NV + k];
          } else {
            load_row_piece<NV, T>(A + (size_t)(node * NV + k) * n + r, z);
          }
#pragma unroll
          for (int l = 0; l < NV; ++l) acc[k] += c[l] * z[l];
        }
      }
    }
    T* dst = a.G + (size_t)(v.e0 + le) * gs + (size_t)jn * NV * Rp + row;
#pragma unroll
    for (int k = 0; k < NV; ++k) dst[(size_t)k * Rp] = acc[k];
    if (le < a.er && jn < a.nbn) {
      T* ds = v.sG + (size_t)le * v.nbd * Rp + (size_t)jn * NV * Rp + row;
#pragma unroll
      for (int k = 0; k < NV; ++k) ds[(size_t)k * Rp] = acc[k];
    }
  }
}

// Sum of the pushed products that land on row (node j, variable av) of own
// element le, in face order: one term per simplex face whose stencil holds the
// node and that couples to a neighbour.  Polls until all of them carry `tag`.
template <int DIM, typename T>
__device__ __forceinline__ T gather(const CoopArgs<T>& a, const BlockView<T>& v, const int* sSpos, int le, int j,
                                    int av, unsigned tag, int* s_err) {
  constexpr int NV = DIM + 2, FF = DIM + 1;
  const uint64_t* p[FF];
#pragma unroll
  for (int f = 0; f < FF; ++f) {
    const int sp = sSpos[f * a.md.Np + j];
    const int fs = sp >= 0 ? v.fs[le * FF + f] : -1;
    p[f] = fs >= 0 ? a.msg + ((size_t)fs * a.nbp + sp * NV + av) * kWords<T> : nullptr;
  }
  T val[FF];
  int polls = 0;
  bool all;
  do {
    all = true;
#pragma unroll
    for (int f = 0; f < FF; ++f) {
      val[f] = T(0);
      if (p[f]) all &= msg_get(p[f], tag, val[f]);
    }
    if (!all && give_up(a, polls, s_err)) break;
  } while (!all);
  T acc = T(0);
#pragma unroll
  for (int f = 0; f < FF; ++f) acc += val[f];
  return acc;
}

// Hessenberg column j and its Givens rotation in R (T, or FP64 for a transposed
// FP32 solve) by one warp (identical in every block), to the rotations rcs, rsn,
// the right-hand side rg and the columns rR; h = h1 (+ h2 after a second pass),
// hn = |w'|.  The j earlier rotations act on the column as the affine recurrence
// t_0 = h_0, t_{k+1} = -sn_k t_k + cs_k h_{k+1} (row k becomes cs_k t_k + sn_k
// h_{k+1}), evaluated by a scan over the lanes instead of j dependent steps (the
// serial form took longer than the apply that it runs beside on small systems).
template <typename R, typename T>
__device__ __forceinline__ void givens(GmresShared<T>& sm, int j, int M1, int itermax, R* rcs, R* rsn, R* rg, R* rR) {
  const int lane = threadIdx.x & 31;
  const bool reorth = sm.s_reorth != 0;
  const R hn = R(sm.s_hn);
  // column j of H_K + I, the Hessenberg matrix of I + K: lane k holds h_k
  R h = lane <= j ? R(sm.sh1[lane]) : R(0);
  if (reorth && lane <= j) h += R(sm.sh2[lane]);
  if (lane == j) h += R(1);
  const R h0 = __shfl_sync(0xffffffffu, h, 0);
  const R hup = __shfl_down_sync(0xffffffffu, h, 1);  // h_{k+1}
  const R cs = lane < j ? rcs[lane] : R(1), sn = lane < j ? rsn[lane] : R(0);
  R A = lane < j ? -sn : R(1), B = lane < j ? cs * hup : R(0);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const R Al = __shfl_up_sync(0xffffffffu, A, o), Bl = __shfl_up_sync(0xffffffffu, B, o);
    if (lane >= o) {
      B = A * Bl + B;
      A = A * Al;
    }
  }
  const R tn = A * h0 + B;  // t_{k+1}
  R t = __shfl_up_sync(0xffffffffu, tn, 1);
  if (lane == 0) t = h0;  // t_k
  if (lane < j) rR[j * M1 + lane] = cs * t + sn * hup;
  t = __shfl_sync(0xffffffffu, t, j);
  if (lane == 0) {
    R den, id;
    if constexpr (sizeof(R) > sizeof(T)) {  // squares of FP32 values stay in range
      const R s2 = t * t + hn * hn;
      id = rsqrt(s2);
      den = s2 > R(0) ? s2 * id : s2;
    } else {
      den = hypot(t, hn);
      id = R(1) / den;
    }
    sm.s_its += 1;
    if (!(den > R(0)) || !isfinite(den)) {
      sm.s_done = 1;  // breakdown: keep the j columns built so far
    } else {
      const R c = t * id, s = hn * id;
      rcs[j] = c;
      rsn[j] = s;
      rR[j * M1 + j] = den;
      const R g = rg[j];
      rg[j + 1] = -s * g;
      rg[j] = c * g;
      sm.s_jdone = j + 1;
      const double resid = fabs(double(s * g));
      if (resid <= sm.s_tol || hn == R(0) || sm.s_its >= itermax) sm.s_done = 1;
    }
  }
}
template <typename T>
__device__ __forceinline__ void givens(const CoopArgs<T>& a, GmresShared<T>& sm, int j, int M1) {
  if constexpr (sizeof(T) == 4) {
    if (a.trans) {
      givens<double>(sm, j, M1, a.flags[F_ITERMAX], sm.dcs, sm.dsn, sm.dg, sm.sRd);
      return;
    }
  }
  givens<T>(sm, j, M1, a.flags[F_ITERMAX], sm.scs, sm.ssn, sm.sg, sm.sR);
}

// After a reduction, by one warp: |h|^2 and the interior coefficient sum h_k
// al_k; lane 0 gets both
template <typename T>
__device__ __forceinline__ void column_sums(const T* h, const T* al, int j, T& hh, T& a1) {
  const int lane = threadIdx.x & 31;
  const T hk = lane <= j ? h[lane] : T(0);
  hh = wsum(hk * hk);
  a1 = wsum(lane <= j ? hk * al[lane] : T(0));
}

// first element of block b of nblk over E elements (balanced ranges)
__host__ __device__ __forceinline__ int block_first(int64_t E, int b, int nblk) { return (int)(E * b / nblk); }

// The whole right-preconditioned GMRES(m) solve of J x = b (or J^T x = b) as
// one persistent kernel (reference: the restarted GMRES behind linearSolve,
// ls_standard.jl:230-244, 321-371, with the element block-Jacobi
// preconditioner of NewtonBDiagPC, preconditioning.jl:7-139).
//   * cycle start: r = b - J x (element blocks D and the face push), beta =
//     |r|, converged when beta <= max(reltol |b|, abstol) (the true residual),
//     v_0 = r / beta;
//   * Arnoldi on K = C D^-1 (the coupling part of J M^-1 = I + K): the Krylov
//     spaces of K and I + K are the same, and K V_j = V_{j+1} H_K gives
//     (I + K) V_j = V_{j+1} (H_K + I), so the vectors are orthogonalised
//     without the v_j term that I adds and the identity is added to the
//     Hessenberg column's diagonal; classical Gram-Schmidt with the norm of
//     the orthogonalised vector from the same reduction (|w'|^2 = w.w -
//     |h|^2) and a second classical pass (its reduction also yields w'.w')
//     when |w'|^2 < |w|^2 / 2 (DGKS with eta = 1/sqrt 2);
//   * cycle end: y = R^-1 g (FP64 back substitution, one warp), x += D^-1 V y
//     on the block's own rows.
// Dense faces: K v has rows on the face-stencil nodes only, so the interior
// rows of every v_k are a multiple of those of v_0: v_k = (stencil rows,
// al_k vint).  The basis holds the stencil rows, al_k is a scalar recurrence,
// and K v_k = G v_k + al_k p0 with the pushed operator G = C D^-1 restricted to
// the stencil columns and p0 = C D^-1 (0, vint), once per cycle.
// Block b owns a contiguous element range (and its rows) for the whole solve.
// Blocks exchange the pushed face products and the dot-product partials as
// tagged words; every block sums the partials in the same order, so the
// scalars are bit-identical in every block and all blocks take the same
// branches.  A wait that runs out raises flags[F_GAVE_UP]; its block and every
// block that waits later leave, and the host reports the solve as failed.
template <int DIM, int NB, typename T>
__device__ void gmres_body(const CoopArgs<T>& a, const int b, const int nblk, GmresShared<T>& sm) {
  constexpr int NV = DIM + 2;
  constexpr int NC = kCols<DIM, NB>;
  using VT = Vec<T>;
  const int tid = threadIdx.x;
  const int n = NB > 0 ? NB : a.n, m = a.m, M1 = a.m + 1;
  const int Np = a.md.Np;
  extern __shared__ __align__(16) unsigned char dsmem[];
  BlockView<T> v;
  v.b = b;
  v.nblk = nblk;
  v.e0 = block_first(a.E, b, nblk);
  v.nel = block_first(a.E, b + 1, nblk) - v.e0;
  v.nbd = a.md.sparse_face ? n : NC > 0 ? NC : a.nbn * NV;
  v.nrow = v.nel * v.nbd;
  v.nrowp = (v.nrow + 3) & ~3;
  v.gV = a.V + (size_t)(m + 2) * ((((size_t)v.e0 * v.nbd + 3) & ~(size_t)3) + 4 * b);
  const int64_t r0 = (int64_t)v.e0 * n;  // first natural row
  const int nat = v.nel * n;             // natural rows
  {
    // the largest block's sizes, as in plan_smem
    const int eb = (a.E + nblk - 1) / nblk;
    const size_t rows = ((size_t)eb * v.nbd + 3) & ~(size_t)3;
    T* p = reinterpret_cast<T*>(dsmem);
    v.cur = a.ws ? p : nullptr;
    v.sw = a.ws ? p + rows : v.gV + (size_t)M1 * v.nrowp;
    p += a.ws ? 2 * rows : 0;
    v.sZ = p;
    p += ((size_t)a.ec * n + 3) & ~(size_t)3;
    v.sP0 = p;
    p += a.p0_smem ? (size_t)eb * a.Rp : 0;
    v.sV = p;
    p += (size_t)a.kv * rows;
    v.sG = p;
    p += (size_t)a.er * v.nbd * a.Rp;
    int* fs = reinterpret_cast<int*>(p);
    v.fs = a.fs_smem ? fs : a.fside + (size_t)v.e0 * a.F;
    if (a.fs_smem)
      for (int k = tid; k < v.nel * a.F; k += NT) fs[k] = a.fside[(size_t)v.e0 * a.F + k];
  }
  const int nbd = v.nbd, nrow = v.nrow;
  const uint64_t pol = l2_evict_first();
  unsigned pt = a.ep[0], rt = a.ep[1];  // tags: pushes, reductions
  for (int k = tid; k < a.F * a.S; k += NT) sm.sPerm[k] = a.md.perm[k];
  for (int k = tid; k < a.F * Np; k += NT) sm.sSpos[k] = a.spos[k];
  if (tid == 0) {
    sm.s_its = sm.s_cycles = sm.s_nreorth = sm.s_err = 0;
    sm.s_conv = 0;
    // nodes on some face stencil first (face-diagonal operators: all nodes)
    int q = 0;
    for (int pass = 0; pass < 2; ++pass)
      for (int j = 0; j < Np; ++j) {
        bool on = a.md.sparse_face != 0;
        for (int f = 0; f < a.F; ++f) on = on || a.spos[f * Np + j] >= 0;
        if (on == (pass == 0)) sm.sOrd[q++] = j;
      }
  }
  __syncthreads();
  if (!a.md.sparse_face) {
    build_push_operator<DIM, T>(a, v, sm.sPerm, sm.sOrd);
    if (tid < v.nrowp - nrow && a.ws) v.cur[nrow + tid] = T(0);
  }
  // |b|^2, and whether x is zero (then r = b and J x is not formed)
  {
    const int lane = tid & 31, wq = tid >> 5;
    T bb = T(0), nz = T(0);
    for (int i = tid; i < nat; i += NT) {
      const T bv = a.bvec[r0 + i];
      bb += bv * bv;
      if (!(a.x[r0 + i] == T(0))) nz = T(1);
    }
    bb = wsum(bb);
    nz = wsum(nz);
    if (lane == 0) {
      sm.sR[wq] = bb;
      sm.sR[32 + wq] = nz;
    }
    __syncthreads();
    ++rt;
    if (wq < 2) {
      const T s = wsum(sm.sR[32 * wq + lane]);
      part_put(a, v, wq, s, rt);
    }
    part_sum(a, v, 2, sm.sh1, rt, &sm.s_err);
    __syncthreads();
    if (sm.s_err) return;
    if (tid == 0) {
      sm.s_bnorm = sqrt(double(sm.sh1[0]));
      sm.s_tol = fmax(a.scal[S_RELTOL] * sm.s_bnorm, a.scal[S_ABSTOL]);
    }
  }
  bool xzero = sm.sh1[1] == T(0);
  __syncthreads();
  for (;;) {
    // ---- r = b - J x (natural rows, in a.w); the pushed products cross blocks
    if (xzero) {
      for (int t = tid; t < nat; t += NT) a.w[r0 + t] = a.bvec[r0 + t];
    } else {
      ++pt;
      couple_push<DIM, T>(a, v, a.x + r0, 0, v.nel, sm.sPerm, pt, pol);
      for (int t = tid; t < nat; t += NT) {
        const int le = t / n, r = t - le * n;
        const int e = v.e0 + le;
        const T* A = a.diag + (size_t)e * n * n;
        const T* xe = a.x + (size_t)e * n;
        const T d = a.trans ? block_col<T>(A, xe, r, n) : block_row<NB, T>(A, xe, r, n);
        const int j = r / NV;
        a.w[r0 + t] = a.bvec[r0 + t] - (d + gather<DIM, T>(a, v, sm.sSpos, le, j, r - j * NV, pt, &sm.s_err));
      }
    }
    xzero = false;
    __syncthreads();
    if (sm.s_err) return;
    // |r|^2 of the stencil rows and of the interior rows
    {
      const int lane = tid & 31, wq = tid >> 5;
      T s0 = T(0), s1 = T(0);
      for (int t = tid; t < nat; t += NT) {
        const int le = t / n, q = t - le * n;
        const int jn = q / NV;
        const T r = a.w[r0 + (size_t)le * n + sm.sOrd[jn] * NV + (q - jn * NV)];
        if (q < nbd) s0 += r * r;
        else s1 += r * r;
      }
      s0 = wsum(s0);
      s1 = wsum(s1);
      if (lane == 0) {
        sm.sR[wq] = s0;
        sm.sR[32 + wq] = s1;
      }
      __syncthreads();
      ++rt;
      if (wq < 2) {
        const T s = wsum(sm.sR[32 * wq + lane]);
        part_put(a, v, wq, s, rt);
      }
      part_sum(a, v, 2, sm.sh1, rt, &sm.s_err);
      __syncthreads();
      if (sm.s_err) return;
    }
    if (tid == 0) {
      const T b2 = sm.sh1[0] + sm.sh1[1];
      const T beta = sqrt(b2);
      sm.s_beta = beta;
      sm.s_g0 = b2 > T(0) ? sm.sh1[1] / b2 : T(0);
      sm.sal[0] = T(1);
      if (sm.s_cycles == 0 && b == 0) a.scal[S_BETA0] = double(beta);
      const bool conv = !(double(beta) > sm.s_tol);
      sm.s_conv = conv ? 1 : 0;
      sm.s_done = (conv || sm.s_its >= a.flags[F_ITERMAX] || !isfinite(double(beta))) ? 1 : 0;
      sm.s_jdone = 0;
      sm.sg[0] = beta;
      for (int k = 1; k <= m; ++k) sm.sg[k] = T(0);
      if (sizeof(T) == 4 && a.trans) sm.dg[0] = double(beta);
    }
    __syncthreads();
    if (sm.s_done) break;
    // v_0 = r / beta: stencil rows to the basis, interior rows to vint
    {
      const T s = T(1) / sm.s_beta;
      T* v0 = basis(a, v, 0);
      for (int t = tid; t < nat; t += NT) {
        const int le = t / n, q = t - le * n;
        const int jn = q / NV;
        const T r = a.w[r0 + (size_t)le * n + sm.sOrd[jn] * NV + (q - jn * NV)] * s;
        if (q < nbd) {
          v0[(size_t)le * nbd + q] = r;
          if (a.ws) v.cur[(size_t)le * nbd + q] = r;
        } else {
          a.vint[r0 + (size_t)le * (n - nbd) + (q - nbd)] = r;
        }
      }
      if (tid < v.nrowp - nrow) v0[nrow + tid] = T(0);
      __syncthreads();
      if (nbd < n) {
        // p0 = C D^-1 (0, vint)
        const size_t gs = (size_t)(n + 1) * a.Rp;
        for (int t = tid; t < v.nel * a.Rp; t += NT) {
          const int le = t / a.Rp, row = t - le * a.Rp;
          T* Gg = a.G + (size_t)(v.e0 + le) * gs + row;
          const T* vi = a.vint + r0 + (size_t)le * (n - nbd);
          T acc = T(0);
          for (int c = nbd; c < n; ++c) acc += Gg[(size_t)c * a.Rp] * vi[c - nbd];
          if (a.p0_smem) v.sP0[t] = acc;
          else Gg[(size_t)n * a.Rp] = acc;
        }
        __syncthreads();
      }
    }
    // ---- Arnoldi
    int j = 0;
    for (;;) {
      // (1) push K v_j; meanwhile one warp finishes column j - 1 (Hessenberg,
      //     rotation, convergence)
      ++pt;
      if (tid < 32 && j > 0) givens(a, sm, j - 1, M1);
      apply_push<DIM, NB, T>(a, v, a.ws ? v.cur : basis(a, v, j), sm.sal[j], sm.sPerm, pt,
                             a.md.sparse_face ? 0 : 32, pol);
      __syncthreads();
      if (sm.s_done) break;
      // (2) w = K v_j: the pushed products of the faces holding the row's node
      for (int t = tid; t < nrow; t += NT) {
        const int le = t / nbd, q = t - le * nbd;
        const int jn = q / NV;
        v.sw[t] = gather<DIM, T>(a, v, sm.sSpos, le, sm.sOrd[jn], q - jn * NV, pt, &sm.s_err);
      }
      if (tid < v.nrowp - nrow) v.sw[nrow + tid] = T(0);
      __syncthreads();
      if (sm.s_err) return;
      // (3) first pass: h1 = V^T w and w.w in one reduction
      ++rt;
      dots_put<T>(a, v, v.sw, j + 1, T(0), T(0), sm.sal, rt);
      part_sum(a, v, j + 2, sm.sh1, rt, &sm.s_err);
      __syncthreads();
      if (sm.s_err) return;
      if (tid < 32) {
        T hh, a1;
        column_sums(sm.sh1, sm.sal, j, hh, a1);
        if (tid == 0) {
          const T ww = sm.sh1[j + 1];
          const T n2 = ww - hh;  // |w'|^2
          const int reorth = n2 < T(0.5) * ww;
          const T hn = sqrt(n2), inv = hn > T(0) ? T(1) / hn : T(0);
          sm.s_reorth = reorth;
          sm.s_nreorth += reorth;
          sm.s_a1 = a1;
          sm.s_hn = hn;
          sm.s_inv = inv;
          if (!reorth) sm.sal[j + 1] = -a1 * inv;
        }
      }
      __syncthreads();
      const T* hl = sm.sh1;
      if (sm.s_reorth) {
        // (4) second pass on w' = w - V h1: h2 = V^T w' and w'.w' in one
        //     reduction; the interior rows of w' are -a1 vint
        sub_scale<T>(a, v, sm.sh1, j + 1, v.sw, T(1), v.sw, v.sw);
        __syncthreads();
        ++rt;
        dots_put<T>(a, v, v.sw, j + 1, sm.s_a1, sm.s_g0, sm.sal, rt);
        part_sum(a, v, j + 2, sm.sh2, rt, &sm.s_err);
        __syncthreads();
        if (sm.s_err) return;
        if (tid < 32) {
          T hh, a2;
          column_sums(sm.sh2, sm.sal, j, hh, a2);
          if (tid == 0) {
            const T r = sm.sh2[j + 1] - hh;
            const T hn = sqrt(r > T(0) ? r : T(0)), inv = hn > T(0) ? T(1) / hn : T(0);
            sm.s_hn = hn;
            sm.s_inv = inv;
            sm.sal[j + 1] = -(sm.s_a1 + a2) * inv;
          }
        }
        __syncthreads();
        hl = sm.sh2;
      }
      // (5) v_{j+1} = (w - V h) / hn
      T* vn = basis(a, v, j + 1);
      sub_scale<T>(a, v, hl, j + 1, v.sw, sm.s_inv, vn, a.ws ? v.cur : vn);
      __syncthreads();
      if (++j == m) {
        if (tid < 32) givens(a, sm, m - 1, M1);
        __syncthreads();
        break;
      }
    }
    // ---- y = R^-1 g (FP64 back substitution by warp 0), x += D^-1 V y
    const int nn = sm.s_jdone;
    if constexpr (sizeof(T) == 4) {
      if (!a.trans) {
        for (int t = tid; t < nn * M1; t += NT) sm.sRd[t] = double(sm.sR[t]);
        if (tid < nn) sm.dg[tid] = double(sm.sg[tid]);
        __syncthreads();
      }
    }
    if (tid < 32) {
      // lane i holds g_i and 1 / R_ii; y_k is broadcast from lane k.  The
      // chain per step is one multiply, the broadcast and one FMA: FP64
      // conversions and shared-memory stores in it cost more than the step
      const int lane = tid;
      const double *R, *rg;
      if constexpr (sizeof(T) == 4) R = sm.sRd, rg = sm.dg;
      else R = sm.sR, rg = sm.sg;
      double g = lane < nn ? rg[lane] : 0.0, y = 0.0;
      const double di = lane < nn ? 1.0 / R[lane * M1 + lane] : 0.0;
#pragma unroll 2
      for (int k = nn - 1; k >= 0; --k) {
        const double rik = lane < k ? R[k * M1 + lane] : 0.0;
        const double yl = g * di;
        if (lane == k) y = yl;
        g = fma(-rik, __shfl_sync(0xffffffffu, yl, k), g);
      }
      if (lane < nn) sm.syT[lane] = T(y);
      if (lane == 0) sm.s_cycles += 1;
    }
    __syncthreads();
    // u = V y in natural rows
    T ya = T(0);
    for (int k = 0; k < nn; ++k) ya += sm.sal[k] * sm.syT[k];
    for (int t = tid; t < nat; t += NT) {
      const int le = t / n, q = t - le * n;
      const int jn = q / NV;
      T u0 = T(0), u1 = T(0);
      if (q < nbd) {
        const size_t row = (size_t)le * nbd + q;
        int k = 0;
        for (; k + 2 <= nn; k += 2) {
          u0 += basis(a, v, k)[row] * sm.syT[k];
          u1 += basis(a, v, k + 1)[row] * sm.syT[k + 1];
        }
        if (k < nn) u0 += basis(a, v, k)[row] * sm.syT[k];
      } else {
        u0 = ya * a.vint[r0 + (size_t)le * (n - nbd) + (q - nbd)];
      }
      a.w[r0 + (size_t)le * n + sm.sOrd[jn] * NV + (q - jn * NV)] = u0 + u1;
    }
    __syncthreads();
    for (int t = tid; t < nat; t += NT) {
      const int le = t / n, r = t - le * n;
      const int e = v.e0 + le;
      const T* A = a.inv + (size_t)e * n * n;
      const T* ue = a.w + (size_t)e * n;
      a.x[(size_t)e * n + r] += a.trans ? block_col<T>(A, ue, r, n) : block_row<NB, T>(A, ue, r, n);
    }
    __syncthreads();
  }
  if (b == 0 && tid == 0) {
    a.ep[0] = pt;
    a.ep[1] = rt;
    a.flags[F_ITS] = sm.s_its;
    a.flags[F_JDONE] = sm.s_jdone;
    a.flags[F_DONE] = 1;
    a.flags[F_CONV] = sm.s_conv;
    a.flags[F_CYCLES] = sm.s_cycles;
    a.flags[F_NREORTH] = sm.s_nreorth;
    a.scal[S_BETA] = double(sm.s_beta);
    a.scal[S_RESID] = double(sm.s_beta);
    a.scal[S_BNORM] = sm.s_bnorm;
    a.scal[S_TOL] = sm.s_tol;
  }
}

// kernel arguments of a solver's GMRES solve (the shared-memory plan is set by
// the launcher, which knows the grid)
template <typename T>
void coop_args(const eg_ls* ls, CoopArgs<T>* out) {
  const eg_mesh* m = ls->lo->mesh;
  CoopArgs<T>& a = *out;
  a.md = dev_mesh(m);
  a.inv = (const T*)ls->pc->inv;
  a.diag = (const T*)ls->lo->diag;
  a.cpl = (const T*)ls->lo->cpl;
  a.spos = ls->lo->spos;
  a.fside = ls->lo->fside;
  a.G = (T*)ls->G;
  a.msg = (uint64_t*)ls->cfs;
  a.part = (uint64_t*)ls->tpart;
  a.tot = a.part + (size_t)2 * 33 * EG_COOP_MAX_BLOCKS * kWords<T>;
  a.ep = (unsigned int*)(ls->dflags + F_TAGS);
  a.bvec = (const T*)ls->bT;
  a.x = (T*)ls->xT;
  a.nb = ls->lo->nb;
  a.nbp = eg_face_rows(a.nb);
  a.S = m->S;
  a.F = m->F;  // DIM + 1 (simplices)
  a.Rp = a.F * a.nbp;
  a.nbn = m->sparse_face ? m->Np : ls->lo->face_nodes;
  a.nv = m->nv;
  a.V = (T*)ls->V;
  a.w = (T*)ls->w;
  a.vint = (T*)ls->z;
  a.flags = ls->dflags;
  a.scal = ls->dscal;
  a.m = ls->m;
  a.n = ls->lo->n;
  a.E = m->E;
  a.N = m->ndof;
  a.trans = ls->trans;
  a.polls = ls->polls > 0 ? ls->polls : 1 << 21;  // seconds
  a.ec = a.fs_smem = a.ws = a.p0_smem = a.kv = a.er = a.ef0 = 0;
  // evict-first operator loads when operator and Krylov basis do not fit the
  // 129 MB L2 together (the operator's lines then give way to the basis)
  const size_t es = sizeof(T);
  const size_t op = m->sparse_face ? (size_t)m->E * a.n * a.n * es + eg_lo_coupling_size(ls->lo) * es
                                   : (size_t)m->E * a.Rp * a.nbn * a.nv * es;
  const size_t basis = (size_t)(a.m + 1) * (size_t)a.E * a.nbn * a.nv * es;
  a.l2ef = op + basis > (size_t(96) << 20) ? 1 : 0;
}

// Shared memory of a block when nblk blocks run the solve, in the order of
// use per byte: face table, work vectors, interior products, the first half of
// the basis (vector k is read twice in each of the m - k later iterations),
// pushed operators (read once per iteration), the rest of the basis.
// Returns the dynamic bytes.
template <typename T>
size_t plan_smem(CoopArgs<T>& a, int nblk, size_t budget) {
  const size_t es = sizeof(T);
  const size_t eb = (a.E + nblk - 1) / nblk;
  const size_t nbd = a.md.sparse_face ? (size_t)a.n : (size_t)a.nbn * a.nv;
  const size_t rows = (eb * nbd + 3) & ~(size_t)3;
  size_t left = budget, used = 0;
  auto take = [&](size_t bytes) {
    bytes = (bytes + 15) & ~(size_t)15;
    if (bytes > left) return false;
    left -= bytes;
    used += bytes;
    return true;
  };
  a.ec = 0;
  if (a.md.sparse_face) {
    // one chunk is always there (at most 128 nodes x 5 variables x 8 B)
    a.ec = (int)((40 * 1024) / (a.n * es));
    if (a.ec < 1) a.ec = 1;
    if ((size_t)a.ec > eb) a.ec = (int)eb;
    used = (es * (((size_t)a.ec * a.n + 3) & ~(size_t)3) + 15) & ~(size_t)15;
    left = left > used ? left - used : 0;
  }
  a.fs_smem = eb * a.F * 4 <= 16 * 1024 && take(eb * a.F * 4);
  a.ws = 2 * rows * es <= 96 * 1024 && take(2 * rows * es);
  a.p0_smem = !a.md.sparse_face && (int)nbd < a.n && eb * a.Rp * es <= 32 * 1024 && take(eb * a.Rp * es);
  a.kv = a.er = 0;
  const size_t half = (size_t)(a.m + 1) / 2;
  while ((size_t)a.kv < half && take(rows * es)) ++a.kv;
  if (!a.md.sparse_face)
    while ((size_t)a.er < eb && take(nbd * a.Rp * es)) ++a.er;
  while (a.kv < a.m + 1 && take(rows * es)) ++a.kv;
  a.ef0 = a.l2ef ? a.er : (int)eb;
  return used;
}

// A block whose operators are all resident takes the whole budget.  One that
// streams operators from L2 or HBM leaves 32 KB more to L1, whose lines hold
// the loads in flight (us per iteration with 176 / 208 KB: 149 / 196 for the
// 10,368-tet p=2 system, 70 / 97 for 18,432 triangles p=4, 17.1 / 18.3 for
// 8,192 triangles p=3; 80 KB and less cost again what residence saves).
template <typename T>
size_t plan_smem(CoopArgs<T>& a, int nblk) {
  const size_t used = plan_smem(a, nblk, kSmemBudget);
  const int eb = (a.E + nblk - 1) / nblk;
  return !a.md.sparse_face && a.er == eb ? used : plan_smem(a, nblk, kSmemStream);
}

// (dimension, element-block size) cases with a compiled body; others, and
// dense-face operators whose stencil unknowns are not kCols, run the generic
// one
inline int gmres_kind(const eg_ls* ls) {
  const eg_mesh* m = ls->lo->mesh;
  const int n = ls->lo->n, cols = ls->lo->face_nodes * m->nv;
  if (m->dim == 2) {
    const int ns[] = {12, 24, 28, 40, 48, 60, 72};
    const int cs[] = {kCols<2, 12>, kCols<2, 24>, kCols<2, 28>, kCols<2, 40>, kCols<2, 48>, kCols<2, 60>, kCols<2, 72>};
    for (int k = 0; k < 7; ++k)
      if (n == ns[k] && (m->sparse_face || cols == cs[k])) return k;
    return 7;
  }
  if (n == 30 && (m->sparse_face || cols == 30)) return 8;
  if (n == 115 && (m->sparse_face || cols == 115)) return 9;
  return 10;
}

template <int DIM, int NB, typename T>
__global__ void __launch_bounds__(NT, 1) k_gmres(CoopArgs<T> a) {
  __shared__ GmresShared<T> sm;
  gmres_body<DIM, NB, T>(a, blockIdx.x, gridDim.x, sm);
}

template <typename T>
const void* gmres_kernel(const eg_ls* ls) {
  switch (gmres_kind(ls)) {
    case 0: return (const void*)k_gmres<2, 12, T>;
    case 1: return (const void*)k_gmres<2, 24, T>;
    case 2: return (const void*)k_gmres<2, 28, T>;
    case 3: return (const void*)k_gmres<2, 40, T>;
    case 4: return (const void*)k_gmres<2, 48, T>;
    case 5: return (const void*)k_gmres<2, 60, T>;
    case 6: return (const void*)k_gmres<2, 72, T>;
    case 7: return (const void*)k_gmres<2, 0, T>;
    case 8: return (const void*)k_gmres<3, 30, T>;
    case 9: return (const void*)k_gmres<3, 115, T>;
    default: return (const void*)k_gmres<3, 0, T>;
  }
}

// A fact about launching kernel fn on the current device (key 0: a block of
// it is resident with the largest dynamic shared memory; C: a cluster of C
// blocks can be placed), asked of the runtime once; also sets the kernel's
// attributes on first use.
template <typename F>
bool launch_fact(const void* fn, int key, F ask) {
  static std::mutex mu;
  static std::map<std::tuple<const void*, int, int>, bool> known;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  const auto id = std::make_tuple(fn, dev, key);
  const auto it = known.find(id);
  if (it != known.end()) return it->second;
  cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget);
  cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  const bool yes = ask();
  known[id] = yes;
  return yes;
}

}  // namespace

// eg_block_inverse.cu -- batched inverses of the element blocks (the
// block-Jacobi preconditioner; reference NewtonBDiagPC factors each block with
// getrf!, NonlinearSolvers/preconditioning.jl:7-139).
//
// In-place Gauss-Jordan elimination with partial pivoting, a block's entries
// in registers for all n steps:
//   * lane (lr, lc), lr < RL row lanes, lc < CL = 32 / RL column lanes, holds
//     rows lr + RL r (r < MR) and columns o + CO c (c < MC), o = warp CL + lc of
//     CO = NW CL column owners.  RL x MR and CO x MC are chosen to cover n with
//     as little padding as the register file allows: 48 unknowns are 16 x 3
//     rows and 2 x 24 columns of one warp, exactly;
//   * pivoting is implicit (no rows move): the pivot of column k is the unused
//     row of largest |a|, found with one redux.sync on the magnitude bits and
//     a ballot (FP64: two of each), a NaN ranking above every number;
//   * the column being eliminated is always register column 0: after CO columns
//     the update writes its results one register column to the left (a
//     rotation that costs nothing), so no register is indexed by a runtime
//     value and the steps are not unrolled over k;
//   * pivot rows stay unscaled (every later step treats a row and its
//     multiplier alike, so a row's scale is free until the end): a step costs
//     MR multiplies and MR MC multiply-adds, and each row is divided by its
//     pivot once at the end;
//   * the next column is updated first, so its pivot search does not wait for
//     the rest of the update.
// k_inverse_warp: a block per warp, no block barrier; four such warps share a
// CTA to fill the SM.  k_inverse_cta: a block per NW warps; the warp that owns
// the next column publishes its pivot and multipliers and the others poll a
// flag word in shared memory, so no barrier holds all warps to the slowest.
//
// Bound: FP64 by the FP64 pipe (n^3 FMA; 48 unknowns 1.9 ms of 1.44), FP32 by
// the dependent chain of a step (search, reciprocal, row broadcast) and the
// warps that registers leave room for.  Measured, us for 8192 blocks (10,368
// for 30 and 115 unknowns), one CTA per block with a barrier per step -> now:
//   unknowns     12      28       30       48        60       72        115
//   FP32      99->13  388->48  565->62  423->137  528->352 1032->448 3975->2002
//   FP64     179->90  886->543 1296->741 5694->1887 7117->4191 15457->6499 57.8->36.5 ms
#include <cmath>

#include "eg_internal.h"
#include "eg_kernels.cuh"
#include "eg_linalg.h"

namespace {

constexpr unsigned kAll = 0xffffffffu;
constexpr int kSpin = 1 << 22;  // polls of one wait between a block's warps

// Largest |v[r]| over the unused rows of the warp (bit r of used set: row r of
// the lane is out): the register row in *rp, the lowest such lane returned.
// Ties: lowest r, then lowest lane (the lowest row).
template <int MR>
__device__ __forceinline__ int pivot_search(const float (&v)[MR], unsigned used, int* rp) {
  unsigned key[MR], best = 0;
#pragma unroll
  for (int r = 0; r < MR; ++r) {
    key[r] = (used >> r) & 1u ? 0u : (__float_as_uint(v[r]) & 0x7fffffffu) + 1u;
    best = max(best, key[r]);
  }
  best = __reduce_max_sync(kAll, best);
  int lane = 0, row = 0;
#pragma unroll
  for (int r = MR - 1; r >= 0; --r) {
    const unsigned m = __ballot_sync(kAll, key[r] == best);
    if (m) {
      lane = __ffs(m) - 1;
      row = r;
    }
  }
  *rp = row;
  return lane;
}
template <int MR>
__device__ __forceinline__ int pivot_search(const double (&v)[MR], unsigned used, int* rp) {
  unsigned hi[MR], lo[MR], best = 0;
#pragma unroll
  for (int r = 0; r < MR; ++r) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v[r]);
    hi[r] = (used >> r) & 1u ? 0u : ((unsigned)(b >> 32) & 0x7fffffffu) + 1u;
    lo[r] = (unsigned)b;
    best = max(best, hi[r]);
  }
  best = __reduce_max_sync(kAll, best);
  unsigned low = 0;
#pragma unroll
  for (int r = 0; r < MR; ++r)
    if (hi[r] == best) low = max(low, lo[r]);
  low = __reduce_max_sync(kAll, low);
  int lane = 0, row = 0;
#pragma unroll
  for (int r = MR - 1; r >= 0; --r) {
    const unsigned m = __ballot_sync(kAll, hi[r] == best && lo[r] == low);
    if (m) {
      lane = __ffs(m) - 1;
      row = r;
    }
  }
  *rp = row;
  return lane;
}

// a register row to and from shared memory in 16-byte units (MC values, the
// piece padded to whole units)
template <int MC>
__device__ __forceinline__ void put_row(float* p, const float (&a)[MC]) {
#pragma unroll
  for (int c = 0; c < MC; c += 4)
    *reinterpret_cast<float4*>(p + c) = make_float4(a[c], c + 1 < MC ? a[c + 1] : 0.f, c + 2 < MC ? a[c + 2] : 0.f,
                                                    c + 3 < MC ? a[c + 3] : 0.f);
}
template <int MC>
__device__ __forceinline__ void put_row(double* p, const double (&a)[MC]) {
#pragma unroll
  for (int c = 0; c < MC; c += 2) *reinterpret_cast<double2*>(p + c) = make_double2(a[c], c + 1 < MC ? a[c + 1] : 0.0);
}
// unit u of a row piece
__device__ __forceinline__ void get_unit(const float* p, float (&x)[4]) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
}
__device__ __forceinline__ void get_unit(const double* p, double (&x)[2]) {
  const double2 v = *reinterpret_cast<const double2*>(p);
  x[0] = v.x; x[1] = v.y;
}

// shared memory of one block: the pivot row as each column owner holds it,
// the multipliers of CO published columns and their flag words (NW > 1), the
// pivot rows of the columns, the result
template <typename T, int RL, int MR, int MC, int NW>
struct Tile {
  static constexpr int CL = 32 / RL, CO = NW * CL;
  static constexpr int MCP = (MC + 3) & ~3;  // a lane's pivot-row piece, 16-byte units
  static constexpr int kRow = CO * MCP;      // values
  static constexpr int kMult = NW > 1 ? CO * RL * MR : 0;
  static __host__ __device__ size_t bytes(int n) {
    const size_t b = sizeof(T) * ((size_t)kRow + kMult + (size_t)n * n) + sizeof(int) * ((size_t)n + CO);
    return (b + 15) & ~(size_t)15;
  }
};

// One lane's part of a block.
template <typename T, int RL, int MR, int MC, int NW>
struct Lane {
  using TL = Tile<T, RL, MR, MC, NW>;
  static constexpr int CL = TL::CL, CO = TL::CO, U = 16 / sizeof(T);
  T a[MR][MC], ds[MR];  // entries; 1 / pivot of the own rows
  int kcol[MR];         // column whose pivot row the own row is
  unsigned used;        // bit r: own row r is a pivot row already, or padding
  bool bad;             // a pivot was zero or NaN
  int n, lr, lc, own;
  T *row, *mult, *S;
  int* perm;
  volatile unsigned* sp;

  __device__ __forceinline__ void load(const T* __restrict__ src, unsigned char* base, int n_, int warp) {
    const int lane = threadIdx.x & 31;
    n = n_;
    lr = lane & (RL - 1);
    lc = lane / RL;
    own = warp * CL + lc;
    T* p = reinterpret_cast<T*>(base);
    row = p + own * TL::MCP;
    mult = p + TL::kRow;          // [CO][RL MR]
    S = mult + TL::kMult;         // [n][n]
    perm = reinterpret_cast<int*>(S + (size_t)n * n);  // [n] pivot row of each column
    sp = reinterpret_cast<volatile unsigned*>(perm + n);  // [CO]: column + 1 << 16 | bad << 15 | register row << 8 | lane row
    used = 0;
    bad = false;
#pragma unroll
    for (int r = 0; r < MR; ++r) {
      const int i = lr + RL * r;
      if (i >= n) used |= 1u << r;
      ds[r] = T(0);
      kcol[r] = 0;
#pragma unroll
      for (int c = 0; c < MC; ++c) {
        const int col = own + CO * c;
        a[r][c] = (i < n && col < n) ? src[(size_t)col * n + i] : T(0);
      }
    }
  }
  // pivot of the column whose values the lanes of column lane l hold in col:
  // the column in v, lane row pr, register row rp; returns 1 / pivot, 0 once a
  // pivot was zero or NaN
  __device__ __forceinline__ T pivot(int l, const T (&col)[MR], T (&v)[MR], int& pr, int& rp) {
#pragma unroll
    for (int r = 0; r < MR; ++r) v[r] = CL > 1 ? __shfl_sync(kAll, col[r], lr + RL * l) : col[r];
    pr = pivot_search<MR>(v, used, &rp) & (RL - 1);
    T pv = v[0];
#pragma unroll
    for (int r = 1; r < MR; ++r)
      if (r == rp) pv = v[r];
    pv = __shfl_sync(kAll, pv, pr);
    bad = bad || !(fabs(pv) > T(0));
    return bad ? T(0) : T(1) / pv;
  }
  // the pivot row to shared memory, from the lanes that hold it (rp is
  // uniform: one copy runs)
  __device__ __forceinline__ void share_row(int k, int pr, int rp, T d) {
    __syncwarp();
    if (lr == pr) {
#pragma unroll
      for (int r = 0; r < MR; ++r)
        if (r == rp) {
          put_row<MC>(row, a[r]);
          used |= 1u << r;
          ds[r] = d;
          kcol[r] = k;
        }
    }
    __syncwarp();
  }
  // register column 0 after the step (mine: this lane holds column k), from
  // unit x of the pivot row
  __device__ __forceinline__ void column0(const T (&f)[MR], const T (&x)[U], int pr, int rp, bool mine, T (&x0)[MR]) {
#pragma unroll
    for (int r = 0; r < MR; ++r) {
      const T t = fma(-f[r], x[0], a[r][0]);
      const T q = (lr == pr && r == rp) ? T(1) : -f[r];
      x0[r] = mine ? q : t;
    }
  }
  // the other register columns, rotated by one when ROT
  template <bool ROT>
  __device__ __forceinline__ void update(const T (&f)[MR], T (&x)[U], const T (&x0)[MR]) {
#pragma unroll
    for (int c = 1; c < MC; ++c) {
      if (c % U == 0) get_unit(row + c, x);
#pragma unroll
      for (int r = 0; r < MR; ++r) a[r][ROT ? c - 1 : c] = fma(-f[r], x[c % U], a[r][c]);
    }
#pragma unroll
    for (int r = 0; r < MR; ++r) a[r][ROT ? MC - 1 : 0] = x0[r];
  }
  __device__ __forceinline__ void rotate() {
#pragma unroll
    for (int r = 0; r < MR; ++r) {
      const T t = a[r][0];
#pragma unroll
      for (int c = 0; c + 1 < MC; ++c) a[r][c] = a[r][c + 1];
      a[r][MC - 1] = t;
    }
  }
  // row i is row kcol of the inverse, divided by its pivot; column q of the
  // in-place result is column perm[q]
  __device__ __forceinline__ void gather() {
#pragma unroll
    for (int c = 0; c < MC; ++c) {
      const int q = own + CO * c;
      if (q < n) {
        T* col = S + (size_t)perm[q] * n;
#pragma unroll
        for (int r = 0; r < MR; ++r)
          if (lr + RL * r < n) col[kcol[r]] = a[r][c] * ds[r];
      }
    }
  }
};

template <typename T, int RL, int MR, int MC, int BPC>
__global__ void __launch_bounds__(32 * BPC) k_inverse_warp(const T* __restrict__ blocks, T* __restrict__ inv, int n,
                                                           int E, unsigned int* __restrict__ status) {
  using L = Lane<T, RL, MR, MC, 1>;
  constexpr int CL = L::CL;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int lane = threadIdx.x & 31, sub = threadIdx.x >> 5;
  const int e = blockIdx.x * BPC + sub;
  if (e >= E) return;  // a whole warp
  L t;
  t.load(blocks + (size_t)e * n * n, smraw + (size_t)sub * L::TL::bytes(n), n, 0);
  T f[MR], d, v[MR], col[MR];
  int pr, rp;
  auto next = [&](int k, int l) {  // pivot and multipliers of column k
    d = t.pivot(l, col, v, pr, rp);
#pragma unroll
    for (int r = 0; r < MR; ++r) f[r] = (t.lr == pr && r == rp) ? T(0) : v[r] * d;
    if (lane == 0) t.perm[k] = pr + RL * rp;
  };
#pragma unroll
  for (int r = 0; r < MR; ++r) col[r] = t.a[r][0];
  next(0, 0);
#pragma unroll 1
  for (int g = 0; g < MC; ++g) {
#pragma unroll
    for (int l = 0; l < CL; ++l) {
      const int k = g * CL + l;
      constexpr int kLast = CL - 1;
      if (k >= n) {  // padding columns: only the rotation of the group is left
        if (l == kLast) t.rotate();
        continue;
      }
      t.share_row(k, pr, rp, d);
      T x[L::U], x0[MR], fk[MR];
      get_unit(t.row, x);
      t.column0(f, x, pr, rp, t.lc == l, x0);
#pragma unroll
      for (int r = 0; r < MR; ++r) {
        fk[r] = f[r];
        col[r] = l == kLast && MC > 1 ? fma(-f[r], x[1], t.a[r][MC > 1 ? 1 : 0]) : x0[r];
      }
      if (k + 1 < n) next(k + 1, l == kLast ? 0 : l + 1);
      if (l == kLast) t.template update<true>(fk, x, x0);
      else t.template update<false>(fk, x, x0);
    }
  }
  __syncwarp();
  t.gather();
  __syncwarp();
  T* dst = inv + (size_t)e * n * n;
  for (int q = lane; q < n * n; q += 32) dst[q] = t.S[q];
  if (t.bad && lane == 0) atomicOr(status, EG_DEV_LU_PIVOT);
}

template <typename T, int RL, int MR, int MC, int NW>
__global__ void __launch_bounds__(32 * NW) k_inverse_cta(const T* __restrict__ blocks, T* __restrict__ inv, int n,
                                                         unsigned int* __restrict__ status) {
  using L = Lane<T, RL, MR, MC, NW>;
  constexpr int CL = L::CL, CO = L::CO;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  L t;
  t.load(blocks + (size_t)blockIdx.x * n * n, smraw, n, warp);
  // the warp that holds column k (owner o) writes its multipliers (the pivot
  // row's slot: the reciprocal) and then the flag word.  Buffer o is free:
  // this warp has consumed the CO - 1 columns since column k - CO, and every
  // other warp published one of them after it had read column k - CO.
  auto publish = [&](int k, int o, const T(&col)[MR]) {
    if (k >= n || warp != o / CL) return;
    T v[MR];
    int pr, rp;
    const T d = t.pivot(o & (CL - 1), col, v, pr, rp);
    T* m = t.mult + o * RL * MR;
    if (t.lc == 0) {
#pragma unroll
      for (int r = 0; r < MR; ++r) m[t.lr + RL * r] = (t.lr == pr && r == rp) ? d : v[r] * d;
    }
    if (lane == 0) t.perm[k] = pr + RL * rp;
    __threadfence_block();
    __syncwarp();
    if (lane == 0) t.sp[o] = ((unsigned)(k + 1) << 16) | (t.bad ? 0x8000u : 0u) | (unsigned)(rp << 8) | (unsigned)pr;
  };
  if (threadIdx.x < CO) t.sp[threadIdx.x] = 0;
  __syncthreads();
  {
    T v[MR];
#pragma unroll
    for (int r = 0; r < MR; ++r) v[r] = t.a[r][0];
    publish(0, 0, v);
  }
#pragma unroll 1
  for (int g = 0; g < MC; ++g) {
#pragma unroll 1
    for (int o = 0; o < CO; ++o) {
      const int k = g * CO + o;
      const bool last = o == CO - 1;
      if (k >= n) {  // padding columns: only the rotation of the group is left
        if (last) t.rotate();
        continue;
      }
      const unsigned tag = (unsigned)(k + 1);
      unsigned s = t.sp[o];
      for (int polls = 0; (s >> 16) != tag && polls < kSpin; ++polls) s = t.sp[o];
      __threadfence_block();
      const int pr = s & 255, rp = (s >> 8) & 127;
      t.bad = (s & 0x8000u) != 0 || (s >> 16) != tag;
      const T* m = t.mult + o * RL * MR;
      T f[MR], d = T(0);
#pragma unroll
      for (int r = 0; r < MR; ++r) {
        f[r] = m[t.lr + RL * r];
        if (t.lr == pr && r == rp) {
          d = f[r];
          f[r] = T(0);
        }
      }
      t.share_row(k, pr, rp, d);
      T x[L::U], x0[MR], v[MR];
      get_unit(t.row, x);
      t.column0(f, x, pr, rp, t.own == o, x0);
#pragma unroll
      for (int r = 0; r < MR; ++r) v[r] = last ? fma(-f[r], x[1], t.a[r][1]) : x0[r];
      publish(k + 1, last ? 0 : o + 1, v);
      if (last) t.template update<true>(f, x, x0);
      else t.template update<false>(f, x, x0);
    }
  }
  __syncthreads();
  t.gather();
  __syncthreads();
  T* dst = inv + (size_t)blockIdx.x * n * n;
  for (int q = threadIdx.x; q < n * n; q += 32 * NW) dst[q] = t.S[q];
  if (t.bad && threadIdx.x == 0) atomicOr(status, EG_DEV_LU_PIVOT);
}

// RL row lanes, MR x MC entries per lane, NW warps per block
template <typename T, int RL, int MR, int MC, int NW>
int launch(eg_mesh* m, const T* A, T* X, int n) {
  static_assert(MR <= 32 && (NW & (NW - 1)) == 0, "used mask, published buffers");
  if constexpr (NW == 1) {
    constexpr int BPC = MR * MC * sizeof(T) <= 512 ? 4 : 2;
    const size_t smem = BPC * Tile<T, RL, MR, MC, 1>::bytes(n);
    cudaFuncSetAttribute(k_inverse_warp<T, RL, MR, MC, BPC>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    k_inverse_warp<T, RL, MR, MC, BPC>
        <<<(m->E + BPC - 1) / BPC, 32 * BPC, smem, m->stream>>>(A, X, n, m->E, m->status);
  } else {
    const size_t smem = Tile<T, RL, MR, MC, NW>::bytes(n);
    cudaFuncSetAttribute(k_inverse_cta<T, RL, MR, MC, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    k_inverse_cta<T, RL, MR, MC, NW><<<m->E, 32 * NW, smem, m->stream>>>(A, X, n, m->status);
  }
  return EG_OK;
}

// Tile by block size: one warp as long as its registers hold the block (72
// unknowns in FP32, 48 in FP64; two warps of half the columns each took 1.4
// times as long for 48 unknowns in FP32), then the fewest warps that do.
int inverse_T(eg_mesh* m, const float* A, float* X, int n) {
  if (n <= 12) return launch<float, 16, 1, 6, 1>(m, A, X, n);
  if (n <= 16) return launch<float, 16, 1, 8, 1>(m, A, X, n);
  if (n <= 24) return launch<float, 32, 1, 24, 1>(m, A, X, n);
  if (n <= 32) return launch<float, 32, 1, 32, 1>(m, A, X, n);
  if (n <= 40) return launch<float, 8, 5, 10, 1>(m, A, X, n);
  if (n <= 48) return launch<float, 16, 3, 24, 1>(m, A, X, n);
  if (n <= 64) return launch<float, 16, 4, 16, 2>(m, A, X, n);
  if (n <= 72) return launch<float, 8, 9, 18, 1>(m, A, X, n);
  if (n <= 96) return launch<float, 32, 3, 24, 4>(m, A, X, n);
  if (n <= 116) return launch<float, 32, 4, 29, 4>(m, A, X, n);
  return launch<float, 32, 4, 32, 4>(m, A, X, n);
}
int inverse_T(eg_mesh* m, const double* A, double* X, int n) {
  if (n <= 12) return launch<double, 16, 1, 6, 1>(m, A, X, n);
  if (n <= 16) return launch<double, 16, 1, 8, 1>(m, A, X, n);
  if (n <= 24) return launch<double, 32, 1, 24, 1>(m, A, X, n);
  if (n <= 32) return launch<double, 32, 1, 32, 1>(m, A, X, n);
  if (n <= 40) return launch<double, 8, 5, 10, 1>(m, A, X, n);
  if (n <= 48) return launch<double, 16, 3, 24, 1>(m, A, X, n);
  if (n <= 64) return launch<double, 16, 4, 16, 2>(m, A, X, n);
  if (n <= 72) return launch<double, 8, 9, 9, 2>(m, A, X, n);
  if (n <= 96) return launch<double, 32, 3, 12, 8>(m, A, X, n);
  if (n <= 120) return launch<double, 32, 4, 15, 8>(m, A, X, n);
  return launch<double, 32, 4, 16, 8>(m, A, X, n);
}

}  // namespace

// X_e = A_e^-1 for the E column-major n x n blocks of a mesh (n <= 128); a zero
// or NaN pivot sets EG_DEV_LU_PIVOT in the status word
int eg_block_inverse(eg_mesh* m, int prec, const void* A, void* X, int n) {
  return prec == EG_F64 ? inverse_T(m, (const double*)A, (double*)X, n) : inverse_T(m, (const float*)A, (float*)X, n);
}

// Batched in-place complex FP64 matrix inverse: blocked Gauss-Jordan elimination with
// partial row pivoting.
//
// Replaces Invert_Matrix (Source/MKL_Routines_Cluster.F90:2-33, ZGETRF + ZGETRI).  Both
// are 8n^3 real flops; Gauss-Jordan is chosen because every panel step after the panel
// factorisation is ONE rank-nb update of the whole matrix (a GEMM), with no triangular
// solves, which keeps the FP64 pipe of all SMs busy across a batch of matrices.
//
// Per panel K = [k0, k0+nb), nb = 8 in FP64 up to n = 1024 and 32 otherwise:
//   1. gj_panel:   one CTA per matrix (in FP64 a cluster of eight for a few matrices)
//                  factorises the n x nb panel in shared memory or registers
//                  (pivot = first max of |re|+|im| over rows >= k, as LAPACK izamax).
//   2. gj_swap:    applies the panel's row interchanges to the other columns, copies
//                  their rows K into R (nb x n) and zeroes them.
//   3. gj_update:  A(:, not K) += P * R(:, not K), P = A(:, K) (the factorised panel).
// The FP32 form (a thread a row, n <= 640) factorises each panel after the first beside the update
// before it (gj_step_kernel).
// After the last panel, gj_colswap undoes the row pivoting as column interchanges.
// INFO follows ZGETRF: the 1-based index of the first exactly-zero pivot (0 if none).
#include "negf_internal.cuh"

namespace negf {

namespace {

constexpr int PANEL_THREADS = 512;
constexpr size_t kPanelSmemMax = 200 * 1024;
constexpr int GJ_MOVES = kGjMoves;   // ints of one matrix's interchange list: count, 64 pairs

// V is the real type of the matrix: the FP32 inverse compares floats, so its pivot search
// stays off the FP64 pipe (comparing the floats orders them as their doubles would)
template <typename V>
__device__ __forceinline__ void argmax_combine(V& v, int& i, V v2, int i2) {
  // larger value wins; on ties the lower row index wins (izamax returns the first max)
  if (v2 > v || (v2 == v && i2 < i)) { v = v2; i = i2; }
}

// Factorisation of one n x kb panel held column-major in shared memory, Ps[c * n + i],
// c in [0, kb), i in [0, n), by the whole CTA (blockDim.x a multiple of 32 and >= kb).
// The pivot of each column is the first maximum of |re|+|im| (exact comparisons with the
// lowest index winning ties), and every row is eliminated by one thread with the same
// operations whatever the thread count, so the result does not depend on blockDim.
// red_v / red_i hold one entry per warp.  Ends after a barrier.
template <typename T>
__device__ __forceinline__ void panel_factor(T* Ps, int n, int k0, int kb, int* ip, int* info_b,
                                             typename CplxTraits<T>::R* red_v, int* red_i, int* s_piv, T* s_d) {
  using R = typename CplxTraits<T>::R;
  const int t = threadIdx.x, nth = blockDim.x;
  const int lane = t & 31, warp = t >> 5, nwarps = nth >> 5;
  for (int c = 0; c < kb; ++c) {
    const int r = k0 + c;
    T* col = Ps + (long long)c * n;
    // ---- pivot search over rows r..n-1
    R bv = -1;
    int bi = n;
    for (int i = r + t; i < n; i += nth) argmax_combine(bv, bi, (R)cabs1(col[i]), i);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      R ov = __shfl_down_sync(0xffffffffu, bv, off);
      int oi = __shfl_down_sync(0xffffffffu, bi, off);
      argmax_combine(bv, bi, ov, oi);
    }
    if (lane == 0) { red_v[warp] = bv; red_i[warp] = bi; }
    __syncthreads();
    // second level by warp 0 with shuffles (the maximum under "larger value, then lower
    // index" does not depend on the order of the comparisons)
    if (warp == 0) {
      R v = lane < nwarps ? red_v[lane] : (R)-1;
      int i = lane < nwarps ? red_i[lane] : n;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        R ov = __shfl_down_sync(0xffffffffu, v, off);
        int oi = __shfl_down_sync(0xffffffffu, i, off);
        argmax_combine(v, i, ov, oi);
      }
      if (lane == 0) {
        if (i >= n) i = r;
        *s_piv = i;
        ip[r] = i;
        T pv = col[i];
        if (pv.x == 0 && pv.y == 0) {
          if (*info_b == 0) *info_b = r + 1;
          *s_d = CplxTraits<T>::make(0, 0);
        } else {
          *s_d = crcp(pv);
        }
      }
    }
    __syncthreads();
    const int p = *s_piv;
    const T d = *s_d;
    const bool singular = (d.x == 0 && d.y == 0);
    // ---- interchange rows r and p inside the panel, scale the pivot row
    if (t < kb) {
      T* cj = Ps + (long long)t * n;
      T vr = cj[r], vp = cj[p];
      if (p != r) { cj[p] = vr; }
      // new pivot-row value is the old row p
      cj[r] = (t == c) ? (singular ? vp : d) : (singular ? vp : cmul(vp, d));
    }
    __syncthreads();
    if (singular) continue;
    // ---- eliminate column c from every other row; row i is owned by one thread, which
    // loads EU columns of its row and of the pivot row before any arithmetic or store (the
    // row's elements are independent, so this only removes the wait on each load)
    constexpr int EU = 8;
    for (int i = t; i < n; i += nth) {
      if (i == r) continue;
      const T f = col[i];
      int j0 = 0;
      for (; j0 + EU <= kb; j0 += EU) {
        T rv[EU], v[EU];
#pragma unroll
        for (int q = 0; q < EU; ++q) {
          const T* cj = Ps + (long long)(j0 + q) * n;
          rv[q] = cj[r];
          v[q] = cj[i];
        }
#pragma unroll
        for (int q = 0; q < EU; ++q) {
          if (j0 + q == c) continue;
          v[q].x = fma((R)-f.x, rv[q].x, v[q].x);
          v[q].x = fma(f.y, rv[q].y, v[q].x);
          v[q].y = fma((R)-f.x, rv[q].y, v[q].y);
          v[q].y = fma((R)-f.y, rv[q].x, v[q].y);
          Ps[(long long)(j0 + q) * n + i] = v[q];
        }
      }
      for (int j = j0; j < kb; ++j) {
        if (j == c) continue;
        T* cj = Ps + (long long)j * n;
        const T rv = cj[r];
        T v = cj[i];
        v.x = fma((R)-f.x, rv.x, v.x);
        v.x = fma(f.y, rv.y, v.x);
        v.y = fma((R)-f.x, rv.y, v.y);
        v.y = fma((R)-f.y, rv.x, v.y);
        cj[i] = v;
      }
      col[i] = cmul(CplxTraits<T>::make(-f.x, -f.y), d);
    }
    __syncthreads();
  }
}

// One CTA per matrix: the panel [k0, k0 + kb) factorised in shared memory.
template <typename T>
__global__ void __launch_bounds__(PANEL_THREADS) gj_panel_kernel(T* A, long long sA, int n, int k0, int kb,
                                                                 int* ipiv, int* info) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char panel_raw[];
  T* Ps = reinterpret_cast<T*>(panel_raw);
  using R = typename CplxTraits<T>::R;
  __shared__ R red_v[PANEL_THREADS / 32];
  __shared__ int red_i[PANEL_THREADS / 32];
  __shared__ int s_piv;
  __shared__ T s_d;
  const int b = blockIdx.x;
  T* Ab = A + (long long)b * sA;
  const int t = threadIdx.x;
  const T* src = Ab + (long long)k0 * n;
  for (int e = t; e < n * kb; e += PANEL_THREADS) Ps[e] = src[e];
  __syncthreads();
  panel_factor<T>(Ps, n, k0, kb, ipiv + (long long)b * n, info + b, red_v, red_i, &s_piv, &s_d);
  T* dst = Ab + (long long)k0 * n;
  for (int e = t; e < n * kb; e += PANEL_THREADS) dst[e] = Ps[e];
}

// The FP64 panel of a few matrices: a cluster of eight CTAs a matrix, each with an eighth of the
// rows in its shared memory.  A panel is 4 n nb^2 multiply-adds on FP64 pipes of about two a clock,
// and one SM's was all that gj_panel_kernel used.  A column step is: every CTA's pivot candidates
// to all (distributed shared memory), a cluster barrier, the pivot row scaled by its owner and sent
// to all, the row it changes places with sent to that owner, a second barrier, and the elimination
// of the own rows.  Pivots, ties and every element's operations are those of panel_factor, so the
// panel is bitwise the same.  Bound: FP64 pipes, then the two barriers and the reciprocal of a step.
// On GB300, one CTA against a cluster, a panel of a few matrices: n = 144, 32 columns 277 / 152 us;
// n = 576, 16 columns 251 / 106 us.
constexpr int CLP_CTAS = 8, CLP_THREADS = 256, CLP_WARPS = CLP_THREADS / 32;
__device__ __forceinline__ void clp_barrier() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t clp_remote(const void* p, int rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void clp_store(const void* p, int rank, double2 v) {
  asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(clp_remote(p, rank)), "d"(v.x), "d"(v.y) : "memory");
}
__global__ void __launch_bounds__(CLP_THREADS) gj_panel_cluster_kernel(double2* A, long long sA, int n, int k0, int kb,
                                                                       int* ipiv, int* info) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char clp_raw[];
  __shared__ __align__(16) double2 prow[33];   // new pivot row; [32]: the reciprocal, zero without a pivot
  __shared__ __align__(16) double2 rrow[32];   // the row that goes to the pivot's place (in its owner)
  __shared__ __align__(16) double2 cand[CLP_CTAS][CLP_WARPS];   // (measure, row) of every warp's best
  const int b = blockIdx.x / CLP_CTAS, rank = blockIdx.x % CLP_CTAS;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int share = (n + CLP_CTAS - 1) / CLP_CTAS;   // rows a CTA
  const int r0 = rank * share, nr = max(0, min(share, n - r0));
  double2* Ps = reinterpret_cast<double2*>(clp_raw);   // [kb][share]
  double2* fcol = Ps + (long long)kb * share;          // the column of the step, before it
  double2* Ab = A + (long long)b * sA + (long long)k0 * n;
  for (int e = t; e < nr * kb; e += CLP_THREADS) Ps[e / nr * share + e % nr] = Ab[(long long)(e / nr) * n + r0 + e % nr];
  clp_barrier();   // all CTAs of the cluster are there
  for (int c = 0; c < kb; ++c) {
    const int r = k0 + c;
    // the measure as an integer, which orders as it does: comparisons stay off the FP64 pipe;
    // 0: no candidate (a row above the step, a NaN)
    unsigned long long bv = 0;
    int bi = n;
    for (int il = t; il < nr; il += CLP_THREADS) {
      const double2 v = Ps[c * share + il];
      fcol[il] = v;
      const unsigned long long m = (unsigned long long)__double_as_longlong(cabs1(v));
      if (r0 + il >= r && m <= 0x7FF0000000000000ULL) argmax_combine(bv, bi, m + 1, r0 + il);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const unsigned long long ov = __shfl_xor_sync(0xffffffffu, bv, off);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
      argmax_combine(bv, bi, ov, oi);
    }
    if (lane < CLP_CTAS)
      clp_store(&cand[rank][warp], lane, make_double2(__longlong_as_double((long long)bv), __longlong_as_double(bi)));
    clp_barrier();
    // every warp of every CTA finds the same pivot among the 64 candidates
    static_assert(CLP_CTAS * CLP_WARPS == 64, "two candidates a lane");
    const double2 c0 = cand[0][lane], c1 = cand[CLP_CTAS / 2][lane];
    bv = (unsigned long long)__double_as_longlong(c0.x);
    bi = (int)__double_as_longlong(c0.y);
    argmax_combine(bv, bi, (unsigned long long)__double_as_longlong(c1.x), (int)__double_as_longlong(c1.y));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const unsigned long long ov = __shfl_xor_sync(0xffffffffu, bv, off);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
      argmax_combine(bv, bi, ov, oi);
    }
    const int p = bi >= n ? r : bi;
    if (warp == 0 && p / share == rank) {
      const double2 pv = fcol[p - r0];
      const bool zero = pv.x == 0 && pv.y == 0;
      double2 d = make_double2(0, 0);
      if (!zero) d = crcp(pv);
      if (lane == 0) {
        ipiv[(long long)b * n + r] = p;
        if (zero) atomicCAS(&info[b], 0, r + 1);   // other columns' owners are other CTAs
      }
      const bool singular = d.x == 0 && d.y == 0;
      double2 v = make_double2(0, 0);
      if (lane < kb) {
        v = Ps[lane * share + p - r0];
        if (!singular) v = lane == c ? d : cmul(v, d);
      }
      for (int q = 0; q < CLP_CTAS; ++q) {
        clp_store(&prow[lane], q, v);
        if (lane == 0) clp_store(&prow[32], q, d);
      }
    }
    if (warp == 1 && r / share == rank && lane < kb) clp_store(&rrow[lane], p / share, Ps[lane * share + r - r0]);
    clp_barrier();
    const double2 d = prow[32];
    const bool singular = d.x == 0 && d.y == 0;
    for (int e = t; e < nr * kb; e += CLP_THREADS) {
      const int j = e / nr, il = e % nr, i = r0 + il;
      double2* at = &Ps[j * share + il];
      if (i == r) { *at = prow[j]; continue; }
      const bool moved = i == p;   // holds row r from here on
      double2 v = moved ? rrow[j] : *at;
      if (!singular) {
        const double2 f = moved ? rrow[c] : fcol[il];
        if (j == c) {
          v = cmul(make_double2(-f.x, -f.y), d);
        } else {
          const double2 rv = prow[j];
          v.x = fma(-f.x, rv.x, v.x);
          v.x = fma(f.y, rv.y, v.x);
          v.y = fma(-f.x, rv.y, v.y);
          v.y = fma(-f.y, rv.x, v.y);
        }
      }
      *at = v;
    }
    __syncthreads();
  }
  for (int e = t; e < nr * kb; e += CLP_THREADS) Ab[(long long)(e / nr) * n + r0 + e % nr] = Ps[e / nr * share + e % nr];
}

// The FP32 panel with its rows in registers: thread t holds row t of the panel (32 float2), so
// a column step reads shared memory only for the pivot row, which every thread of a warp reads
// at one address.  The panel in shared memory (panel_factor) spends its time on the 32 x n
// elements that each column step loads and stores there and on four barriers per step; here a
// step has two.  The arrays are indexed statically: every step works on register column 0 and
// writes the updated columns one place to the left, so after 32 steps the columns are back in
// order (a panel of kb < 32 columns ends with 32 - kb plain rotations).  Interchanges move no
// data: each thread carries the position of its row, and the rows are stored to their
// positions at the end.  The candidate of the next step's pivot is formed from the first column
// updated, so its warp reduction overlaps the other 31 columns' arithmetic.
// Bound: issue slots, 128 FMA per row and step, and the latency of the pivot chain (two
// barriers, one reciprocal).  Pivots, their ties (lowest position) and every element's
// operations are those of panel_factor, so the panel is bitwise the same.
// Measured on GB300 (panel alone, 32 matrices), panel_factor against this: n = 144 51 / 23 us, 400
// 72 / 33 us, 576 96 / 44 us.
constexpr int RP_MAX_N = 640;   // 640 threads of up to 102 registers
constexpr int RP_C = 32;
struct PanelShared {
  float2 raw[RP_C], piv[RP_C];   // pivot row, unscaled and scaled
  unsigned w_key[RP_MAX_N / 32];
  int w_pos[RP_MAX_N / 32];
  int extra;
};
__device__ __forceinline__ void named_barrier(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// Threads 0 .. nthreads-1 (whole warps, nthreads >= n) with the panel's rows; ip, info, mv and
// orig are those of the matrix Ab.
template <bool WHOLE>   // nthreads is the whole CTA
__device__ __forceinline__ void panel_rows(float2 (&row)[RP_C], PanelShared& sh, float2* Ab, int n, int k0, int kb,
                                           int* ip, int* info, int* mv, int* orig, int nthreads) {
  float2 *raw = sh.raw, *piv = sh.piv;
  unsigned* w_key = sh.w_key;
  int* w_pos = sh.w_pos;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nwarps = nthreads >> 5;
  auto sync = [&]() {
    if constexpr (WHOLE) __syncthreads();
    else named_barrier(3, nthreads);
  };
  const bool live = t < n;
  int pos = live ? t : 0x7fffffff;
  const int from = live && k0 > 0 ? orig[t] : t;   // the row of A that is here
  if (t == 0) sh.extra = kb;
  // key of a pivot candidate: larger |re|+|im| first (non-negative floats order as their bits),
  // 0 = no candidate (a row above the step, a NaN)
  auto key_of = [&](float2 v, int r) -> unsigned {
    const float a = cabs1(v);
    return (live && pos >= r && a == a) ? __float_as_uint(a) + 1u : 0u;
  };
  unsigned key = key_of(row[0], k0);
  unsigned wmax = __reduce_max_sync(0xffffffffu, key);
#pragma unroll 1
  for (int c = 0; c < kb; ++c) {
    const int r = k0 + c;
    const int wpos = __reduce_min_sync(0xffffffffu, key == wmax ? pos : 0x7fffffff);
    if (lane == 0) { w_key[warp] = wmax; w_pos[warp] = wpos; }
    sync();
    const unsigned ck = lane < nwarps ? w_key[lane] : 0u;
    const unsigned best = __reduce_max_sync(0xffffffffu, ck);
    int p = __reduce_min_sync(0xffffffffu, (lane < nwarps && ck == best) ? w_pos[lane] : 0x7fffffff);
    if (best == 0u) p = r;
    const bool own = pos == p;
    if (__any_sync(0xffffffffu, own)) {
      // the owner's warp scales the pivot row, one element per lane
      if (own) {
#pragma unroll
        for (int j = 0; j < RP_C; j += 2)
          *reinterpret_cast<float4*>(&raw[j]) = make_float4(row[j].x, row[j].y, row[j + 1].x, row[j + 1].y);
        ip[r] = p;
        if (row[0].x == 0.f && row[0].y == 0.f && *info == 0) *info = r + 1;
      }
      __syncwarp();
      const float2 pv = raw[0];
      const float2 d = (pv.x == 0.f && pv.y == 0.f) ? make_float2(0.f, 0.f) : crcp(pv);
      piv[lane] = lane == 0 ? d : cmul(raw[lane], d);
    }
    sync();
    if (own) pos = r;
    else if (pos == r) pos = p;
    const float4 p01 = *reinterpret_cast<const float4*>(&piv[0]);
    const float2 d = make_float2(p01.x, p01.y);
    if (d.x == 0.f && d.y == 0.f) {   // no pivot: the interchange only
      const float2 first = row[0];
#pragma unroll
      for (int j = 0; j < RP_C - 1; ++j) row[j] = row[j + 1];
      row[RP_C - 1] = first;
      key = key_of(row[0], r + 1);
      wmax = __reduce_max_sync(0xffffffffu, key);
      continue;
    }
    const float2 f = row[0];
    auto step = [&](float2 v, float2 rv) -> float2 {
      v.x = fmaf(-f.x, rv.x, v.x);
      v.x = fmaf(f.y, rv.y, v.x);
      v.y = fmaf(-f.x, rv.y, v.y);
      v.y = fmaf(-f.y, rv.x, v.y);
      return v;
    };
    row[0] = own ? make_float2(p01.z, p01.w) : step(row[1], make_float2(p01.z, p01.w));
    key = key_of(row[0], r + 1);
    wmax = __reduce_max_sync(0xffffffffu, key);
    if (own) {   // the pivot row itself: one warp of the CTA takes both branches
#pragma unroll
      for (int j = 2; j < RP_C; ++j) row[j - 1] = piv[j];
      row[RP_C - 1] = d;
    } else {
#pragma unroll
      for (int j = 2; j < RP_C; j += 2) {
        const float4 q = *reinterpret_cast<const float4*>(&piv[j]);
        row[j - 1] = step(row[j], make_float2(q.x, q.y));
        row[j] = step(row[j + 1], make_float2(q.z, q.w));
      }
      row[RP_C - 1] = cmul(make_float2(-f.x, -f.y), d);
    }
  }
#pragma unroll 1
  for (int c = kb; c < RP_C; ++c) {
    const float2 first = row[0];
#pragma unroll
    for (int j = 0; j < RP_C - 1; ++j) row[j] = row[j + 1];
    row[RP_C - 1] = first;
  }
  // the panel's interchanges as (destination, origin) rows for gj_swap, the rows K first: at
  // most kb of the others moved
  if (live) {
#pragma unroll
    for (int j = 0; j < RP_C; ++j)
      if (j < kb) Ab[(long long)(k0 + j) * n + pos] = row[j];
    orig[pos] = from;
    const int q = (pos >= k0 && pos < k0 + kb) ? pos - k0 : (pos != t ? atomicAdd(&sh.extra, 1) : -1);
    if (q >= 0) {
      mv[1 + 2 * q] = pos;
      mv[2 + 2 * q] = t;
    }
  }
  sync();
  if (t == 0) mv[0] = sh.extra;
}

template <int MAXT>   // threads at most: 512 (128 registers each) or RP_MAX_N (96)
__global__ void __launch_bounds__(MAXT, 1) gj_panel_reg_kernel(float2* A, long long sA, int n, int k0, int kb,
                                                               int* ipiv, int* info, int* moves, int* orig, int* tickets) {
  pdl_wait();
  __shared__ __align__(16) PanelShared sh;
  const int b = blockIdx.x, t = threadIdx.x;
  if (b == 0 && t < kGjTickets) tickets[t] = 0;
  float2* Ab = A + (long long)b * sA;
  float2 row[RP_C];
#pragma unroll
  for (int j = 0; j < RP_C; ++j)
    row[j] = (t < n && j < kb) ? Ab[(long long)(k0 + j) * n + t] : make_float2(0.f, 0.f);
  panel_rows<true>(row, sh, Ab, n, k0, kb, ipiv + (long long)b * n, info + b, moves + (long long)b * GJ_MOVES,
             orig + (long long)b * n, blockDim.x);
}

// The FP64 inverse (n <= 1024; not the mixed form's redone ones, see zinv_f64) with panels of
// eight columns.  A panel is one SM's work, 4 n nb^2
// multiply-adds on a pipe of two per clock: with 32 columns and a few matrices the panels were
// most of the time while the other SMs waited, and with many they were the longest part of a
// wave.  The rank-8 updates are split into enough tiles for every SM.  The panel has its rows in
// registers as the FP32 one above: a thread a row, a step on register column 0, two barriers a
// step, the interchanges as moves.
// Whole INVERT calls with the copies on GB300, 32-column panels against these: n = 144, 1 matrix
// 2.76 / 0.92 ms, 304 matrices 13.1 / 9.3 ms; n = 400, 1 10.9 / 3.7 ms, 200 114 / 103 ms;
// n = 784, 1 21.1 / 12.4 ms; n = 1000, 16 149 / 129 ms.
constexpr int NP_C = 8, NP_MAX_N = 1024;
__global__ void __launch_bounds__(NP_MAX_N, 1) gj_panel_narrow_kernel(double2* A, long long sA, int n, int k0, int kb,
                                                                      int* ipiv, int* info, int* moves) {
  pdl_wait();
  __shared__ double2 raw[NP_C], piv[NP_C];   // pivot row, unscaled and scaled
  __shared__ unsigned long long w_key[NP_MAX_N / 32];
  __shared__ int w_pos[NP_MAX_N / 32];
  __shared__ int s_extra;
  const int b = blockIdx.x;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nwarps = blockDim.x >> 5;
  double2* Ab = A + (long long)b * sA;
  int* ip = ipiv + (long long)b * n;
  const bool live = t < n;
  double2 row[NP_C];
#pragma unroll
  for (int j = 0; j < NP_C; ++j)
    row[j] = (live && j < kb) ? Ab[(long long)(k0 + j) * n + t] : make_double2(0.0, 0.0);
  int pos = live ? t : 0x7fffffff;
  if (t == 0) s_extra = kb;
  auto rotate = [&]() {
    const double2 first = row[0];
#pragma unroll
    for (int j = 0; j < NP_C - 1; ++j) row[j] = row[j + 1];
    row[NP_C - 1] = first;
  };
  // largest key of a warp and the lowest position that has it (keys: bits of |re| + |im| plus
  // one, which order as the values; 0 = no candidate)
  auto best_of = [&](unsigned long long key, int at, unsigned long long& best) -> int {
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32) == hi ? (unsigned)key : 0u);
    best = ((unsigned long long)hi << 32) | lo;
    return __reduce_min_sync(0xffffffffu, key == best ? at : 0x7fffffff);
  };
#pragma unroll 1
  for (int c = 0; c < kb; ++c) {
    const int r = k0 + c;
    const double a = cabs1(row[0]);
    unsigned long long best;
    const int wpos = best_of(
        (live && pos >= r && a == a) ? (unsigned long long)__double_as_longlong(a) + 1ULL : 0ULL, pos, best);
    if (lane == 0) { w_key[warp] = best; w_pos[warp] = wpos; }
    __syncthreads();
    int p = best_of(lane < nwarps ? w_key[lane] : 0ULL, lane < nwarps ? w_pos[lane] : 0x7fffffff, best);
    if (best == 0ULL) p = r;
    const bool own = pos == p;
    if (__any_sync(0xffffffffu, own)) {
      if (own) {
#pragma unroll
        for (int j = 0; j < NP_C; ++j) raw[j] = row[j];
        ip[r] = p;
        if (row[0].x == 0.0 && row[0].y == 0.0 && info[b] == 0) info[b] = r + 1;
      }
      __syncwarp();
      const double2 pv = raw[0];
      if (lane < NP_C) {
        const double2 d = (pv.x == 0.0 && pv.y == 0.0) ? pv : crcp(pv);
        piv[lane] = lane == 0 ? d : cmul(raw[lane], d);
      }
    }
    __syncthreads();
    if (own) pos = r;
    else if (pos == r) pos = p;
    const double2 d = piv[0];
    if (d.x == 0.0 && d.y == 0.0) {   // no pivot: the interchange only
      rotate();
      continue;
    }
    const double2 f = row[0];
    if (own) {
#pragma unroll
      for (int j = 1; j < NP_C; ++j) row[j - 1] = piv[j];
      row[NP_C - 1] = d;
    } else {
#pragma unroll
      for (int j = 1; j < NP_C; ++j) {
        const double2 rv = piv[j];
        double2 v = row[j];
        v.x = fma(-f.x, rv.x, v.x);
        v.x = fma(f.y, rv.y, v.x);
        v.y = fma(-f.x, rv.y, v.y);
        v.y = fma(-f.y, rv.x, v.y);
        row[j - 1] = v;
      }
      row[NP_C - 1] = cmul(make_double2(-f.x, -f.y), d);
    }
  }
#pragma unroll 1
  for (int c = kb; c < NP_C; ++c) rotate();
  int* mv = moves + (long long)b * GJ_MOVES;
  if (live) {
#pragma unroll
    for (int j = 0; j < NP_C; ++j)
      if (j < kb) Ab[(long long)(k0 + j) * n + pos] = row[j];
    const int q = (pos >= k0 && pos < k0 + kb) ? pos - k0 : (pos != t ? atomicAdd(&s_extra, 1) : -1);
    if (q >= 0) {
      mv[1 + 2 * q] = pos;
      mv[2 + 2 * q] = t;
    }
  }
  __syncthreads();
  if (t == 0) mv[0] = s_extra;
}

// A(:, j) += P R(:, j) for the columns outside the panel, kb <= KB: tiles of 32 rows x 16
// columns, two outputs a thread, each formed by gj_update_kernel's operations.  One matrix of
// n = 144 is 45 tiles, where gj_update_kernel's 80 x 80 tiles are four; n = 576, K = 32, the few
// matrices of a redone inverse: 107 -> 53 us.
constexpr int NU_M = 32, NU_N = 16;
template <int KB>
__global__ void __launch_bounds__(256) gj_update_tiles_kernel(double2* A, long long sA, int n, int k0, int kb,
                                                              const double2* R, long long sR) {
  pdl_wait();
  __shared__ double2 Ps[KB][NU_M], Rs[KB][NU_N + 1];
  const int b = blockIdx.z, t = threadIdx.x;
  const int m0 = blockIdx.x * NU_M, n0 = blockIdx.y * NU_N;
  double2* Ab = A + (long long)b * sA;
  const double2* Rb = R + (long long)b * sR;
  for (int e = t; e < kb * NU_M; e += 256) {
    const int k = e / NU_M, i = m0 + e % NU_M;
    Ps[k][e % NU_M] = i < n ? Ab[(long long)(k0 + k) * n + i] : make_double2(0.0, 0.0);
  }
  for (int e = t; e < kb * NU_N; e += 256) {
    const int j = n0 + e / kb;
    Rs[e % kb][e / kb] = j < n ? Rb[(long long)j * kb + e % kb] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  const int i = t % NU_M, row = m0 + i;
  for (int jj = t / NU_M; jj < NU_N; jj += 256 / NU_M) {
    const int col = n0 + jj;
    if (row >= n || col >= n || (col >= k0 && col < k0 + kb)) continue;
    double2 s = make_double2(0.0, 0.0);
    for (int k = 0; k < kb; ++k) cfma(s, Ps[k][i], Rs[k][jj]);
    double2* c = Ab + (long long)col * n + row;
    *c = cadd(s, *c);
  }
}

// Row interchanges of one panel for the columns outside it, and the copy of rows K into R.
// The kb interchanges (r, ip[r]) of the panel touch at most 2 kb rows.  The register panel
// leaves them composed as a gather list over the touched rows (row trow[t] receives the value
// of row torig[t]); after the shared-memory panel thread 0 of each CTA composes it.  Then one warp per column loads its touched values (all loads
// before any store, so the gather is a simultaneous permutation), writes rows K to R
// (kb x n, column-major) with zeros in A, and the other touched rows back in place.
// Panel columns get R = 0.
// ahead > 0 (FP32): the first CTAs of a matrix form the next panel's `ahead` columns as the update
// by this panel leaves them, in `next` (n x RP_C), so that the next panel can be factorised beside
// the update of all other columns (gj_step_kernel).  128 rows x 16 columns a CTA, a thread a row
// and eight columns: it gathers the interchanged rows itself and writes elsewhere, so no CTA waits
// for another.  Bound: latency, one chain of list -> rows -> 32 steps from P in registers.
constexpr int SWAP_WARPS = 8;
constexpr int AHEAD_ROWS = 128, AHEAD_COLS = 16;
// the CTA's part of the next panel's columns: rows i0 .., columns k1 + c0 ..
__device__ __forceinline__ void gj_columns_ahead(const float2* Ab, int n, int k0, int kb, int k1, int ahead, int i0, int c0,
                                                 const int* trow, const int* torig, int nt, float2* next) {
  __shared__ __align__(16) float2 rs[RP_C][AHEAD_COLS];   // R of the columns
  __shared__ int origin[AHEAD_ROWS];                      // row that moves to i0 + r
  const int t = threadIdx.x, r = t % AHEAD_ROWS, i = i0 + r;
  const int u0 = t / AHEAD_ROWS * 8;
  if (t < AHEAD_ROWS) origin[t] = i;
  __syncthreads();
  if (t < nt && trow[t] >= i0 && trow[t] < i0 + AHEAD_ROWS) origin[trow[t] - i0] = torig[t];
  // rows K head the list: R(k, j) is row torig[k] of column j
  for (int e = t; e < RP_C * AHEAD_COLS; e += 256) {
    const int k = e / AHEAD_COLS, u = e % AHEAD_COLS;
    rs[k][u] = k < kb && c0 + u < ahead ? Ab[(long long)(k1 + c0 + u) * n + torig[k]] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  if (i >= n) return;
  const bool pivot_row = i >= k0 && i < k1;   // zero before the update
  const int from = origin[r];
  const float2* pk = Ab + (long long)k0 * n + i;
  float2 acc[8], c[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    acc[u] = make_float2(0.f, 0.f);
    c[u] = !pivot_row && c0 + u0 + u < ahead ? Ab[(long long)(k1 + c0 + u0 + u) * n + from] : make_float2(0.f, 0.f);
  }
  constexpr int PF = 16;
#pragma unroll 1
  for (int k = 0; k < kb; k += PF) {   // kb = RP_C
    float2 f[PF];
#pragma unroll
    for (int q = 0; q < PF; ++q) f[q] = pk[(long long)(k + q) * n];
#pragma unroll
    for (int q = 0; q < PF; ++q)
#pragma unroll
      for (int u = 0; u < 8; u += 2) {
        const float4 v = *reinterpret_cast<const float4*>(&rs[k + q][u0 + u]);
        cfma(acc[u], f[q], make_float2(v.x, v.y));
        cfma(acc[u + 1], f[q], make_float2(v.z, v.w));
      }
  }
#pragma unroll
  for (int u = 0; u < 8; ++u)
    if (c0 + u0 + u < ahead) next[(long long)(c0 + u0 + u) * n + i] = cadd(acc[u], c[u]);
}

template <typename T>
__global__ void __launch_bounds__(SWAP_WARPS * 32, sizeof(T) == 8 ? 3 : 1)
    gj_swap_kernel(T* A, long long sA, int n, int k0, int kb, const int* ipiv, const int* moves, T* R, long long sR,
                   int ahead, T* next) {
  pdl_wait();
  __shared__ int trow[64], torig[64];
  __shared__ int s_nt;
  const int b = blockIdx.y;
  T* Ab = A + (long long)b * sA;
  const int* ip = ipiv + (long long)b * n;
  T* Rb = R + (long long)b * sR;
  if (moves) {   // the panel kernel composed the list
    const int* mv = moves + (long long)b * GJ_MOVES;
    if (threadIdx.x < 64 && (int)threadIdx.x < mv[0]) {
      trow[threadIdx.x] = mv[1 + 2 * threadIdx.x];
      torig[threadIdx.x] = mv[2 + 2 * threadIdx.x];
    }
    if (threadIdx.x == 0) s_nt = mv[0];
  } else if (threadIdx.x == 0) {
    int nt = kb;
    for (int c = 0; c < kb; ++c) { trow[c] = k0 + c; torig[c] = k0 + c; }
    for (int c = 0; c < kb; ++c) {
      const int r = k0 + c, p = ip[r];
      if (p == r) continue;
      int ip_ = -1;
      for (int t = 0; t < nt; ++t)
        if (trow[t] == p) { ip_ = t; break; }
      if (ip_ < 0) { ip_ = nt; trow[nt] = p; torig[nt] = p; ++nt; }
      const int tmp = torig[c];   // row r sits at index c
      torig[c] = torig[ip_];
      torig[ip_] = tmp;
    }
    s_nt = nt;
  }
  __syncthreads();
  const int nt = s_nt;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k1 = k0 + kb;
  int block = blockIdx.x;
  if constexpr (sizeof(T) == 8) {
    const int ng = (ahead + AHEAD_COLS - 1) / AHEAD_COLS, nahead = ng * ((n + AHEAD_ROWS - 1) / AHEAD_ROWS);
    if (block < nahead) {
      gj_columns_ahead(Ab, n, k0, kb, k1, ahead, block / ng * AHEAD_ROWS, block % ng * AHEAD_COLS, trow, torig, nt,
                       next + (long long)b * RP_C * n);
      return;
    }
    block -= nahead;
  }
  const int j = block * SWAP_WARPS + warp;
  if (j >= n || (j >= k1 && j < k1 + ahead)) return;
  if (j >= k0 && j < k1) {
    for (int c = lane; c < kb; c += 32) Rb[(long long)j * kb + c] = CplxTraits<T>::make(0, 0);
    return;
  }
  T* colj = Ab + (long long)j * n;
  T v0 = CplxTraits<T>::make(0, 0), v1 = CplxTraits<T>::make(0, 0);
  if (lane < nt) v0 = colj[torig[lane]];
  if (lane + 32 < nt) v1 = colj[torig[lane + 32]];
  __syncwarp();
  if (lane < nt) {
    const int r = trow[lane];
    if (r >= k0 && r < k1) { Rb[(long long)j * kb + (r - k0)] = v0; colj[r] = CplxTraits<T>::make(0, 0); }
    else colj[r] = v0;
  }
  if (lane + 32 < nt) {
    const int r = trow[lane + 32];
    if (r >= k0 && r < k1) { Rb[(long long)j * kb + (r - k0)] = v1; colj[r] = CplxTraits<T>::make(0, 0); }
    else colj[r] = v1;
  }
}

// The rank-kb update of one panel step: A(:, j) += P R(:, j) for every column j outside the
// panel [k0, k0 + kb), P = A(:, k0:k0+kb) (n x kb), R (kb x n) from gj_swap.  K = kb <= 32,
// so each CTA stages its whole P and R slabs in shared memory with one barrier and then
// runs the kb rank-1 steps from there: 80 x 80 output tiles, 256 threads of 5 x 5 complex
// accumulators (25 FMAs per 10 shared loads).  The R slab's rows are padded to 81 entries:
// its loads walk k fastest, and an 80-entry stride would put every thread of a warp on the
// same bank.  In the FP32 form the 25 values of A a thread updates are loaded before the k
// loop, so their latency overlaps the slab loads and the FMAs instead of serialising 25
// load/store round trips at the end (the FP64 form, with twice the registers per value,
// loads them a column of five at a time).  The k order and the final A + sum equal those of
// the general GEMM kernel, so results are bitwise the same.
constexpr int UPD_T = 80, UPD_R = 5, UPD_RS = UPD_T + 1;
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 8 ? 2 : 1) gj_update_kernel(T* A, long long sA, int n, int k0, int kb, const T* R,
                                                        long long sR) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char upd_raw[];
  T* Ps = reinterpret_cast<T*>(upd_raw);              // [kb][UPD_T]
  T* Rs = Ps + 32 * UPD_T;                              // [kb][UPD_RS]
  constexpr bool kPrefetch = sizeof(T) == 8;            // float2
  const int b = blockIdx.z;
  const int m0 = blockIdx.x * UPD_T, n0 = blockIdx.y * UPD_T;
  if (n0 >= k0 && n0 + UPD_T <= k0 + kb) return;        // tile inside the panel columns
  T* Ab = A + (long long)b * sA;
  const T* Rb = R + (long long)b * sR;
  const int t = threadIdx.x;
  const int tx = t & 15, ty = t >> 4;
  auto updated = [&](int i, int j) -> T* {              // nullptr: outside A or in the panel
    const int row = m0 + tx + 16 * i, col = n0 + ty + 16 * j;
    if (row >= n || col >= n || (col >= k0 && col < k0 + kb)) return nullptr;
    return Ab + (long long)col * n + row;
  };
  T cin[kPrefetch ? UPD_R : 1][kPrefetch ? UPD_R : 1];
  if constexpr (kPrefetch) {
#pragma unroll
    for (int j = 0; j < UPD_R; ++j)
#pragma unroll
      for (int i = 0; i < UPD_R; ++i) {
        const T* cp = updated(i, j);
        cin[i][j] = cp ? *cp : CplxTraits<T>::make(0, 0);
      }
  }
  for (int e = t; e < kb * UPD_T; e += 256) {
    const int k = e / UPD_T, i = e % UPD_T;
    Ps[k * UPD_T + i] = (m0 + i < n) ? Ab[(long long)(k0 + k) * n + m0 + i] : CplxTraits<T>::make(0, 0);
    const int j = e / kb, kk = e % kb;                  // R slab: contiguous kb x UPD_T
    Rs[kk * UPD_RS + j] = (n0 + j < n) ? Rb[(long long)(n0 + j) * kb + kk] : CplxTraits<T>::make(0, 0);
  }
  __syncthreads();
  T acc[UPD_R][UPD_R];
#pragma unroll
  for (int i = 0; i < UPD_R; ++i)
#pragma unroll
    for (int j = 0; j < UPD_R; ++j) acc[i][j] = CplxTraits<T>::make(0, 0);
  for (int k = 0; k < kb; ++k) {
    T av[UPD_R], bv[UPD_R];
#pragma unroll
    for (int i = 0; i < UPD_R; ++i) av[i] = Ps[k * UPD_T + tx + 16 * i];
#pragma unroll
    for (int j = 0; j < UPD_R; ++j) bv[j] = Rs[k * UPD_RS + ty + 16 * j];
#pragma unroll
    for (int i = 0; i < UPD_R; ++i)
#pragma unroll
      for (int j = 0; j < UPD_R; ++j) cfma(acc[i][j], av[i], bv[j]);
  }
#pragma unroll
  for (int j = 0; j < UPD_R; ++j) {
    T c[UPD_R];
    if constexpr (!kPrefetch) {   // the column's five loads before its five stores
#pragma unroll
      for (int i = 0; i < UPD_R; ++i) {
        const T* cp = updated(i, j);
        c[i] = cp ? *cp : CplxTraits<T>::make(0, 0);
      }
    }
#pragma unroll
    for (int i = 0; i < UPD_R; ++i) {
      T* cp = updated(i, j);
      if (!cp) continue;
      if constexpr (kPrefetch) *cp = cadd(acc[i][j], cin[i][j]);
      else *cp = cadd(acc[i][j], c[i]);
    }
  }
}

// The FP32 rank-kb update as a persistent, software-pipelined kernel (two CTAs per SM, each
// walking output tiles of 80 x 80).  While a CTA computes one tile, cp.async copies the P
// and R slabs of its next tile into the other half of a double buffer, and the tile's C
// values load into registers behind the k loop; the one-tile-per-CTA form above ran its
// load, compute and store phases back to back with two CTAs per SM to overlap them.  Each
// output element is formed by exactly the operations of gj_update_kernel (the same k order
// of fused multiply-adds from the same slabs, then A + sum), so results are bitwise equal.
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem, int src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)),
               "l"(gmem), "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

constexpr int UPD_SLABS = 32 * UPD_T + 32 * UPD_RS;   // float2 of one buffer: P slab, then R slab

__global__ void __launch_bounds__(256, 2) gj_update_f32_pipelined(float2* A, long long sA, int n, int k0, int kb,
                                                                  const float2* R, long long sR, int ntm, int ntn,
                                                                  long long ntiles) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char upp_raw[];
  float2* bufs = reinterpret_cast<float2*>(upp_raw);   // [2][UPD_SLABS]
  const int t = threadIdx.x;
  const int tx = t & 15, ty = t >> 4;
  const long long per_item = (long long)ntm * ntn;
  // copies of tile q's slabs into buffer Ps (P slab [kb][UPD_T], R slab [kb][UPD_RS]);
  // entries outside A are zero-filled without a read
  auto issue = [&](long long q, float2* Ps) {
    const int b = (int)(q / per_item);
    const int r = (int)(q % per_item);
    const int m0 = (r / ntn) * UPD_T, n0 = (r % ntn) * UPD_T;
    const float2* Ab = A + (long long)b * sA;
    const float2* Rb = R + (long long)b * sR;
    float2* Rs = Ps + 32 * UPD_T;
    for (int e = t; e < kb * UPD_T; e += 256) {
      const int k = e / UPD_T, i = e % UPD_T;
      const bool okp = m0 + i < n;
      cp_async8(&Ps[k * UPD_T + i], okp ? (const void*)&Ab[(long long)(k0 + k) * n + m0 + i] : (const void*)Ab,
                okp ? 8 : 0);
      const int j = e / kb, kk = e % kb;
      const bool okr = n0 + j < n;
      cp_async8(&Rs[kk * UPD_RS + j], okr ? (const void*)&Rb[(long long)(n0 + j) * kb + kk] : (const void*)Rb,
                okr ? 8 : 0);
    }
    cp_async_commit();
  };
  long long q = blockIdx.x;
  if (q < ntiles) issue(q, bufs);
  for (int it = 0; q < ntiles; q += gridDim.x, ++it) {
    const float2* Ps = bufs + (it & 1) * UPD_SLABS;
    const float2* Rs = Ps + 32 * UPD_T;
    const int b = (int)(q / per_item);
    const int r = (int)(q % per_item);
    const int m0 = (r / ntn) * UPD_T, n0 = (r % ntn) * UPD_T;
    float2* Ab = A + (long long)b * sA;
    auto updated = [&](int i, int j) -> float2* {   // nullptr: outside A or in the panel
      const int row = m0 + tx + 16 * i, col = n0 + ty + 16 * j;
      if (row >= n || col >= n || (col >= k0 && col < k0 + kb)) return nullptr;
      return Ab + (long long)col * n + row;
    };
    float2 cin[UPD_R][UPD_R];
#pragma unroll
    for (int j = 0; j < UPD_R; ++j)
#pragma unroll
      for (int i = 0; i < UPD_R; ++i) {
        const float2* cp = updated(i, j);
        cin[i][j] = cp ? *cp : make_float2(0.0f, 0.0f);
      }
    // the next tile's slabs go into the other buffer, which every thread finished reading
    // before the barrier that ended the previous iteration
    if (q + gridDim.x < ntiles) issue(q + gridDim.x, bufs + ((it + 1) & 1) * UPD_SLABS);
    else cp_async_commit();   // an empty group keeps the count: wait_group 1 below = this tile
    cp_async_wait<1>();
    __syncthreads();
    float2 acc[UPD_R][UPD_R];
#pragma unroll
    for (int i = 0; i < UPD_R; ++i)
#pragma unroll
      for (int j = 0; j < UPD_R; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
    for (int k = 0; k < kb; ++k) {
      float2 av[UPD_R], bv[UPD_R];
#pragma unroll
      for (int i = 0; i < UPD_R; ++i) av[i] = Ps[k * UPD_T + tx + 16 * i];
#pragma unroll
      for (int j = 0; j < UPD_R; ++j) bv[j] = Rs[k * UPD_RS + ty + 16 * j];
#pragma unroll
      for (int i = 0; i < UPD_R; ++i)
#pragma unroll
        for (int j = 0; j < UPD_R; ++j) cfma(acc[i][j], av[i], bv[j]);
    }
#pragma unroll
    for (int j = 0; j < UPD_R; ++j)
#pragma unroll
      for (int i = 0; i < UPD_R; ++i) {
        float2* cp = updated(i, j);
        if (cp) *cp = cadd(acc[i][j], cin[i][j]);
      }
    __syncthreads();   // this buffer is free for the tile after next
  }
  cp_async_wait<0>();
}

// One step of the FP32 inverse: the rank-kb update by panel k0 beside the factorisation of the
// next panel, k1 = k0 + kb, whose columns gj_swap_kernel left updated in `next`.  CTA b < batch factorises
// matrix b's; the other CTAs, and these when they are done, take output tiles of 80 x 48 of the
// remaining columns from a counter, each half of a CTA its own tiles, as gj_update_f32_pipelined.
// The two panels' columns are left out of the tiles' count, and 48 wide tiles leave less of it in a
// last ragged one: at n = 400 7 x 48 of 336 columns, where 80 wide tiles of all are 5 x 80.
// A panel is the work of one SM and bound by latency, so on its own it leaves the other SMs idle
// and the update waits.  Bound now: the panel's chain of 32 steps for few matrices, the FP32 pipe
// for many.  A whole inverse on GB300, panel, interchanges and update one after another against
// this: n = 144, 8 matrices 178 / 153 us; n = 400, 8 650 / 526, 32 1028 / 768, 160 3680 / 3322;
// n = 576, 8 1343 / 999, 32 2632 / 2022.
// Every element is formed by the operations of the separate kernels, so the inverse is theirs bit
// for bit.
constexpr int ST_C = 3, ST_N = 16 * ST_C, ST_RS = ST_N + 1;   // columns a thread, of a tile, its stride
constexpr int ST_SLABS = 32 * UPD_T + 32 * ST_RS;             // float2 of one buffer: P slab, then R slab
template <int MAXT>
__global__ void __launch_bounds__(MAXT, 1)
    gj_step_kernel(float2* A, long long sA, int n, int k0, int kb, const float2* R, long long sR, int kb1, int* ipiv,
                   int* info, int* moves, int* orig, int batch, int ntm, int ntn, long long ntiles, int* ticket, int pthreads, bool leave,
                   const float2* next) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char step_raw[];
  __shared__ __align__(16) PanelShared sh;
  __shared__ int s_next[2];
  const int t = threadIdx.x;
  const int k1 = k0 + kb;
  if (blockIdx.x < batch) {
    const int b = blockIdx.x;
    float2* Ab = A + (long long)b * sA;
    if (t < pthreads) {
      float2 row[RP_C];
#pragma unroll
      for (int j = 0; j < RP_C; ++j)
        row[j] = (t < n && j < kb1) ? next[((long long)b * RP_C + j) * n + t] : make_float2(0.f, 0.f);
      panel_rows<false>(row, sh, Ab, n, k1, kb1, ipiv + (long long)b * n, info + b, moves + (long long)b * GJ_MOVES,
                 orig + (long long)b * n, pthreads);
    }
    if (leave) return;
    __syncthreads();
  }
  if (t >= 512) return;
  const int g = t >> 8, tg = t & 255;
  const int tx = tg & 15, ty = tg >> 4;
  float2* bufs = reinterpret_cast<float2*>(step_raw) + (long long)g * 2 * ST_SLABS;   // [2][ST_SLABS]
  const long long per_item = (long long)ntm * ntn;
  const int skip = kb + kb1, cols = n - skip;   // columns outside the two panels: c, from k0 on c + skip
  auto column = [&](int c) { return c < k0 ? c : c + skip; };
  auto issue = [&](long long q, float2* Ps) {
    const int b = (int)(q / per_item);
    const int r = (int)(q % per_item);
    const int m0 = (r / ntn) * UPD_T, n0 = (r % ntn) * ST_N;
    const float2* Ab = A + (long long)b * sA;
    const float2* Rb = R + (long long)b * sR;
    float2* Rs = Ps + 32 * UPD_T;
    for (int e = tg; e < kb * UPD_T; e += 256) {
      const int k = e / UPD_T, i = e % UPD_T;
      const bool okp = m0 + i < n;
      cp_async8(&Ps[k * UPD_T + i], okp ? (const void*)&Ab[(long long)(k0 + k) * n + m0 + i] : (const void*)Ab,
                okp ? 8 : 0);
    }
    for (int e = tg; e < kb * ST_N; e += 256) {
      const int j = e / kb, kk = e % kb;
      const bool okr = n0 + j < cols;
      cp_async8(&Rs[kk * ST_RS + j], okr ? (const void*)&Rb[(long long)column(n0 + j) * kb + kk] : (const void*)Rb,
                okr ? 8 : 0);
    }
    cp_async_commit();
  };
  if (tg == 0) s_next[g] = atomicAdd(ticket, 1);
  named_barrier(1 + g, 256);
  long long q = s_next[g];
  named_barrier(1 + g, 256);
  if (q < ntiles) issue(q, bufs);
  for (int it = 0; q < ntiles; ++it) {
    const float2* Ps = bufs + (it & 1) * ST_SLABS;
    const float2* Rs = Ps + 32 * UPD_T;
    int taken = 0;
    if (tg == 0) taken = atomicAdd(ticket, 1);
    const int b = (int)(q / per_item);
    const int r = (int)(q % per_item);
    const int m0 = (r / ntn) * UPD_T, n0 = (r % ntn) * ST_N;
    float2* Ab = A + (long long)b * sA;
    auto updated = [&](int i, int j) -> float2* {   // nullptr: outside
      const int row = m0 + tx + 16 * i, c = n0 + ty + 16 * j;
      if (row >= n || c >= cols) return nullptr;
      return Ab + (long long)column(c) * n + row;
    };
    float2 cin[UPD_R][ST_C];
#pragma unroll
    for (int j = 0; j < ST_C; ++j)
#pragma unroll
      for (int i = 0; i < UPD_R; ++i) {
        const float2* cp = updated(i, j);
        cin[i][j] = cp ? *cp : make_float2(0.0f, 0.0f);
      }
    cp_async_wait<0>();
    if (tg == 0) s_next[g] = taken;
    named_barrier(1 + g, 256);
    // the next tile's slabs into the other buffer, which every thread finished reading before the
    // barrier that ended the previous tile
    const long long qn = s_next[g];
    if (qn < ntiles) issue(qn, bufs + ((it + 1) & 1) * ST_SLABS);
    float2 acc[UPD_R][ST_C];
#pragma unroll
    for (int i = 0; i < UPD_R; ++i)
#pragma unroll
      for (int j = 0; j < ST_C; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
#pragma unroll 1
    for (int k = 0; k < kb; ++k) {
      float2 av[UPD_R], bv[ST_C];
#pragma unroll
      for (int i = 0; i < UPD_R; ++i) av[i] = Ps[k * UPD_T + tx + 16 * i];
#pragma unroll
      for (int j = 0; j < ST_C; ++j) bv[j] = Rs[k * ST_RS + ty + 16 * j];
#pragma unroll
      for (int i = 0; i < UPD_R; ++i)
#pragma unroll
        for (int j = 0; j < ST_C; ++j) cfma(acc[i][j], av[i], bv[j]);
    }
#pragma unroll
    for (int j = 0; j < ST_C; ++j)
#pragma unroll
      for (int i = 0; i < UPD_R; ++i) {
        float2* cp = updated(i, j);
        if (cp) *cp = cadd(acc[i][j], cin[i][j]);
      }
    named_barrier(1 + g, 256);   // this buffer is free for the tile after next, s_next for its number
    q = qn;
  }
}

// One thread per row: column interchanges in reverse pivot order.
template <typename T>
__global__ void gj_colswap_kernel(T* A, long long sA, int n, const int* ipiv) {
  pdl_wait();
  const int b = blockIdx.y;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  T* Ab = A + (long long)b * sA;
  const int* ip = ipiv + (long long)b * n;
  for (int k = n - 1; k >= 0; --k) {
    const int p = ip[k];
    if (p != k) {
      T tmp = Ab[(long long)k * n + i];
      Ab[(long long)k * n + i] = Ab[(long long)p * n + i];
      Ab[(long long)p * n + i] = tmp;
    }
  }
}

// The whole FP32 Gauss-Jordan of one matrix in one CTA: for every panel, the panel
// factorisation, its row interchanges and its rank-kb update, in the same order and with
// the same operations per element as gj_panel + gj_swap + gj_update, so the inverse is
// bitwise the same as the three-launch form's (the update's k order, its fused multiply-
// adds and the final A + sum are those of gj_update_kernel).  It replaces 3 launches per
// panel by one per inverse and keeps the panel in shared memory across its update.
//   - the panel (n x 32 float2, up to 100 KB at n = 400) stays in shared memory;
//   - the other columns are processed in chunks of 32: one warp per column applies the
//     panel's interchanges (the same gather list as gj_swap) and moves rows K into the
//     chunk's R slab (32 x 32 in shared memory), then all 256 threads update the chunk,
//     each thread 4 rows x 8 columns of accumulators;
//   - two CTAs share an SM, so one's serial panel steps overlap the other's updates.
// Offered when the batch has at least one matrix per SM (below that the three-launch form
// spreads a matrix over many SMs and always finishes first); the engine times both forms
// on its first inverse of a shape and keeps the faster.  The column interchanges that end
// the inverse stay a separate launch (gj_colswap_kernel).
constexpr int FUSED_THREADS = 256, FUSED_JC = 32, FUSED_RS = FUSED_JC + 1, FUSED_MAX_N = 400;
__global__ void __launch_bounds__(FUSED_THREADS, 2) gj_fused_f32_kernel(float2* A, long long sA, int n, int* ipiv,
                                                                        int* info) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char fused_raw[];
  float2* Ps = reinterpret_cast<float2*>(fused_raw);   // [32][n]: the panel, column-major
  float2* Rs = Ps + 32 * n;                             // [32][FUSED_RS]: rows K of a chunk
  __shared__ float red_v[FUSED_THREADS / 32];
  __shared__ int red_i[FUSED_THREADS / 32];
  __shared__ int s_piv, s_nt;
  __shared__ float2 s_d;
  __shared__ int trow[64], torig[64];
  const int b = blockIdx.x;
  float2* Ab = A + (long long)b * sA;
  int* ip = ipiv + (long long)b * n;
  const int t = threadIdx.x;
  const int warp = t >> 5, lane = t & 31;
  const int rg = t & 63, cg = t >> 6;                   // update: row group, column group
  const float2 zero = make_float2(0.f, 0.f);
  for (int k0 = 0; k0 < n; k0 += FUSED_JC) {
    const int kb = n - k0 < FUSED_JC ? n - k0 : FUSED_JC;
    const float2* src = Ab + (long long)k0 * n;
    for (int e = t; e < n * kb; e += FUSED_THREADS) Ps[e] = src[e];
    __syncthreads();
    panel_factor<float2>(Ps, n, k0, kb, ip, info + b, red_v, red_i, &s_piv, &s_d);
    float2* dst = Ab + (long long)k0 * n;
    for (int e = t; e < n * kb; e += FUSED_THREADS) dst[e] = Ps[e];
    if (t == 0) {   // the panel's interchanges as one gather over the touched rows (gj_swap)
      int nt = kb;
      for (int c = 0; c < kb; ++c) { trow[c] = k0 + c; torig[c] = k0 + c; }
      for (int c = 0; c < kb; ++c) {
        const int r = k0 + c, p = ip[r];
        if (p == r) continue;
        int ip_ = -1;
        for (int q = 0; q < nt; ++q)
          if (trow[q] == p) { ip_ = q; break; }
        if (ip_ < 0) { ip_ = nt; trow[nt] = p; torig[nt] = p; ++nt; }
        const int tmp = torig[c];
        torig[c] = torig[ip_];
        torig[ip_] = tmp;
      }
      s_nt = nt;
    }
    __syncthreads();
    const int nt = s_nt;
    for (int j0 = 0; j0 < n; j0 += FUSED_JC) {
      if (j0 == k0) continue;                           // the panel's own columns
      // interchanges of the chunk's columns; rows K go to R and become zero in A
      for (int jj = warp; jj < FUSED_JC; jj += FUSED_THREADS / 32) {
        const int j = j0 + jj;
        if (j >= n) break;
        float2* colj = Ab + (long long)j * n;
        float2 v0 = zero, v1 = zero;
        if (lane < nt) v0 = colj[torig[lane]];
        if (lane + 32 < nt) v1 = colj[torig[lane + 32]];
        __syncwarp();
        if (lane < nt) {
          const int r = trow[lane];
          if (r >= k0 && r < k0 + kb) { Rs[(r - k0) * FUSED_RS + jj] = v0; colj[r] = zero; }
          else colj[r] = v0;
        }
        if (lane + 32 < nt) {
          const int r = trow[lane + 32];
          if (r >= k0 && r < k0 + kb) { Rs[(r - k0) * FUSED_RS + jj] = v1; colj[r] = zero; }
          else colj[r] = v1;
        }
      }
      __syncthreads();
      // A(:, j) += P R(:, j) for the chunk's columns: rows rg + 64 q (+ 256 per pass),
      // columns j0 + 8 cg + c
      for (int i0 = 0; i0 < n; i0 += 256) {
        float2 acc[4][8];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int c = 0; c < 8; ++c) acc[q][c] = zero;
        for (int k = 0; k < kb; ++k) {
          float2 pv[4], rv[8];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int i = i0 + rg + 64 * q;
            pv[q] = i < n ? Ps[k * n + i] : zero;
          }
#pragma unroll
          for (int c = 0; c < 8; ++c) rv[c] = Rs[k * FUSED_RS + 8 * cg + c];
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int c = 0; c < 8; ++c) cfma(acc[q][c], pv[q], rv[c]);
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const int j = j0 + 8 * cg + c;
          if (j >= n) break;
          float2* colj = Ab + (long long)j * n;
          float2 cin[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int i = i0 + rg + 64 * q;
            cin[q] = i < n ? colj[i] : zero;
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int i = i0 + rg + 64 * q;
            if (i < n) colj[i] = cadd(acc[q][c], cin[q]);
          }
        }
      }
      __syncthreads();   // the chunk's A and R are done before the next chunk's interchanges
    }
  }
}

}  // namespace

size_t gj_fused_smem(int n) { return sizeof(float2) * ((size_t)32 * n + 32 * FUSED_RS); }

int panel_width(int n, int elem_bytes) {
  // the panel (n x nb complex) must fit the 227 KB opt-in shared memory of a CTA.  The
  // panel's work grows with nb (n*nb^2 per panel, n^2*nb per inverse) while its rank-nb
  // updates are cheap, so both forms use nb = 32.
  const long long limit = kPanelSmemMax;
  int nb = 32;
  (void)elem_bytes;
  while (nb > 4 && (long long)n * nb * (long long)elem_bytes > limit) nb >>= 1;
  return nb;
}

long long gj_next_bytes(int n, long long batch) { return n <= RP_MAX_N ? 8LL * RP_C * n * batch : 0; }

int inv_work_alloc(InvWork& w, int n, int batch, cudaMemPool_t pool, cudaStream_t st) {
  if (w.n_cap >= n && w.batch_cap >= batch && w.rbuf) return NEGF_OK;
  inv_work_free(w, st);
  w.nb = panel_width(n);
  w.pooled = pool != nullptr;
  auto get = [&](void** p, size_t bytes) {
    return (pool ? cudaMallocFromPoolAsync(p, bytes, pool, st) : cudaMalloc(p, bytes)) == cudaSuccess;
  };
  // R buffer: nb x n complex per matrix, large enough for both forms (FP64 nb, FP32 2nb)
  if (!get((void**)&w.rbuf, sizeof(double2) * (size_t)batch * w.nb * n)) return NEGF_ENOMEM;
  if (!get((void**)&w.ipiv, sizeof(int) * (size_t)batch * n)) return NEGF_ENOMEM;
  if (!get((void**)&w.info, sizeof(int) * (size_t)batch)) return NEGF_ENOMEM;
  if (!get((void**)&w.orig, sizeof(int) * (size_t)batch * n)) return NEGF_ENOMEM;
  if (!get((void**)&w.tickets, sizeof(int) * kGjTickets)) return NEGF_ENOMEM;
  if (n <= RP_MAX_N && !get((void**)&w.next, gj_next_bytes(n, batch))) return NEGF_ENOMEM;
  if (!get((void**)&w.moves, sizeof(int) * (size_t)batch * kGjMoves)) return NEGF_ENOMEM;
  w.n_cap = n;
  w.batch_cap = batch;
  return NEGF_OK;
}

void inv_work_free(InvWork& w, cudaStream_t st) {
  for (void* p : {(void*)w.rbuf, (void*)w.ipiv, (void*)w.info, (void*)w.orig, (void*)w.moves, (void*)w.tickets, (void*)w.next})
    if (p) {
      if (w.pooled) cudaFreeAsync(p, st);
      else cudaFree(p);
    }
  w = InvWork{};
}

namespace {


int sm_count_cached() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
  }
  return n;
}

// FP32 inverse as one fused launch per batch (plus the column interchanges)
int gj_invert_fused_f32(float2* A, long long sA, int n, int batch, InvWork& w, cudaStream_t st) {
  const size_t smem = gj_fused_smem(n);
  w.columns_pending = false;
  NEGF_CUDA_TRY(cudaFuncSetAttribute(gj_fused_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)gj_fused_smem(FUSED_MAX_N)));
  NEGF_CUDA_TRY(cudaMemsetAsync(w.info, 0, sizeof(int) * batch, st));
  cudaEvent_t ev;
  timed_begin(st, TK_F32, 8.0 * (double)n * n * n * batch, &ev);
  pdl_launch(gj_fused_f32_kernel, batch, FUSED_THREADS, smem, st, A, sA, n, w.ipiv, w.info);
  NEGF_CUDA_TRY(cudaGetLastError());
  timed_end(st, TK_F32, ev);
  dim3 g3((n + 127) / 128, batch);
  pdl_launch(gj_colswap_kernel<float2>, g3, 128, 0, st, A, sA, n, w.ipiv);
  NEGF_CUDA_TRY(cudaGetLastError());
  count_launch(2);
  return NEGF_OK;
}

template <typename T>
int gj_invert(T* A, long long sA, int n, int batch, InvWork& w, cudaStream_t st) {
  if (batch <= 0 || n <= 0) return NEGF_OK;
  if (n > w.n_cap || batch > w.batch_cap) return NEGF_EINVAL;
  const int nb = panel_width(n, (int)sizeof(T));
  const size_t smem = sizeof(T) * (size_t)n * nb;
  if (smem > kPanelSmemMax) return NEGF_EINVAL;
  NEGF_CUDA_TRY(cudaFuncSetAttribute(gj_panel_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPanelSmemMax));
  const size_t upd_smem = sizeof(T) * 32 * (UPD_T + UPD_RS);
  NEGF_CUDA_TRY(cudaFuncSetAttribute(gj_update_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)upd_smem));
  const size_t upp_smem = sizeof(float2) * 2 * (size_t)UPD_SLABS;
  if constexpr (sizeof(T) == 8)
    NEGF_CUDA_TRY(cudaFuncSetAttribute(gj_update_f32_pipelined, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)upp_smem));
  if (nb > 32 || batch > 65535) return NEGF_EINVAL;
  NEGF_CUDA_TRY(cudaMemsetAsync(w.info, 0, sizeof(int) * batch, st));
  T* rbuf = reinterpret_cast<T*>(w.rbuf);
  const long long sR = (long long)nb * n;
  // Each panel after the first beside the update before it (gj_step_kernel).  With more matrices
  // than SMs the panels of small ones share an SM better on their own: apart against together,
  // n = 64, 160 matrices 92 / 101 us, 320 121 / 143; n = 144, 320 535 / 578; but n = 256, 320
  // 2632 / 2217 us.
  const bool steps = sizeof(T) == 8 && n <= RP_MAX_N && nb == RP_C && (batch <= sm_count_cached() || n >= 256);
  // FP64 panels of a few matrices on clusters.  Whole inverses, one CTA against clusters: n = 144, 1
  // matrix 1.81 / 1.12 ms, 24 2.34 / 1.77; n = 576, 1 11.4 / 6.2 ms, 24 53.1 / 49.2.  More clusters
  // than that share SMs, and their barriers wait for one another.
  const bool clustered = sizeof(T) == 16 && 4 * batch * CLP_CTAS <= 5 * sm_count_cached();
  for (int k0 = 0; k0 < n; k0 += nb) {
    const int kb = (n - k0 < nb) ? (n - k0) : nb;
    const bool reg = sizeof(T) == 8 && n <= RP_MAX_N;
    const int threads = (n + 31) / 32 * 32;   // of a panel in registers
    const int* moves = reg ? w.moves : nullptr;
    if (!steps || k0 == 0) {   // the others were factorised beside the last update
      cudaEvent_t ev;
      timed_begin(st, TK_PANEL, 8.0 * n * (double)kb * kb * batch, &ev);
      if (reg) {
        auto panel = threads <= 512 ? gj_panel_reg_kernel<512> : gj_panel_reg_kernel<RP_MAX_N>;
        pdl_launch(panel, batch, threads, 0, st, reinterpret_cast<float2*>(A), sA, n, k0, kb, w.ipiv, w.info, w.moves,
                   w.orig, w.tickets);
      } else if (sizeof(T) == 16 && clustered) {
        // an eighth of a panel and of a column: at most 32 KB of what panel_width allows, no opt-in
        const size_t csmem = sizeof(double2) * (size_t)((n + CLP_CTAS - 1) / CLP_CTAS) * (kb + 1);
        pdl_launch_cluster(dim3(CLP_CTAS), gj_panel_cluster_kernel, batch * CLP_CTAS, CLP_THREADS, csmem, st,
                           reinterpret_cast<double2*>(A), sA, n, k0, kb, w.ipiv, w.info);
      } else {
        pdl_launch(gj_panel_kernel<T>, batch, PANEL_THREADS, smem, st, A, sA, n, k0, kb, w.ipiv, w.info);
      }
      NEGF_CUDA_TRY(cudaGetLastError());
      timed_end(st, TK_PANEL, ev);
      count_launch();
    }
    const int ahead = steps ? std::min(nb, n - k0 - kb) : 0;   // the next panel's columns
    const int nahead = (ahead + AHEAD_COLS - 1) / AHEAD_COLS * ((n + AHEAD_ROWS - 1) / AHEAD_ROWS);
    dim3 g2((n + SWAP_WARPS - 1) / SWAP_WARPS + nahead, batch);
    pdl_launch(gj_swap_kernel<T>, g2, SWAP_WARPS * 32, 0, st, A, sA, n, k0, kb, w.ipiv, moves, rbuf, sR, ahead,
               reinterpret_cast<T*>(w.next));
    NEGF_CUDA_TRY(cudaGetLastError());
    count_launch();
    // A(:, j) += P R(:, j) for the columns outside the panel
    {
      cudaEvent_t eu;
      timed_begin(st, sizeof(T) == 8 ? TK_F32 : TK_GEMM, 8.0 * n * (double)(n - kb) * kb * batch, &eu);
      const int nt = (n + UPD_T - 1) / UPD_T;
      if constexpr (sizeof(T) == 8) {
        const long long ntiles = (long long)nt * nt * batch;
        if (ahead > 0) {
          const int sms = sm_count_cached();
          auto stepk = threads <= 512 ? gj_step_kernel<512> : gj_step_kernel<RP_MAX_N>;
          const size_t smem = 4 * sizeof(float2) * (size_t)ST_SLABS;
          NEGF_CUDA_TRY(cudaFuncSetAttribute(stepk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
          const int ntn = (n - kb - ahead + ST_N - 1) / ST_N;
          const long long tiles = (long long)nt * ntn * batch;
          // a CTA an SM; with more matrices than SMs the CTAs for the tiles come after the panels'
          const int grid = batch > sms ? batch + sms : (int)std::min<long long>(batch + (tiles + 1) / 2, sms);
          pdl_launch(stepk, grid, threads <= 512 ? 512 : RP_MAX_N, smem, st, reinterpret_cast<float2*>(A), sA, n, k0, kb,
                     reinterpret_cast<const float2*>(rbuf), sR, ahead, w.ipiv, w.info, w.moves, w.orig, batch, nt, ntn,
                     tiles, w.tickets + k0 / nb, threads, batch > sms, w.next);
        } else {
          const int grid = (int)std::min<long long>(ntiles, 2LL * sm_count_cached());
          pdl_launch(gj_update_f32_pipelined, grid, 256, upp_smem, st, reinterpret_cast<float2*>(A), sA, n, k0, kb,
                     reinterpret_cast<const float2*>(rbuf), sR, nt, nt, ntiles);
        }
      } else {
        // 80 x 80 tiles where they fill the device twice over, smaller ones for a few matrices
        if ((long long)nt * nt * batch < 2LL * sm_count_cached())
          pdl_launch(gj_update_tiles_kernel<32>, dim3((n + NU_M - 1) / NU_M, (n + NU_N - 1) / NU_N, batch), 256, 0, st, A,
                     sA, n, k0, kb, rbuf, sR);
        else
          pdl_launch(gj_update_kernel<T>, dim3(nt, nt, batch), 256, upd_smem, st, A, sA, n, k0, kb, rbuf, sR);
      }
      NEGF_CUDA_TRY(cudaGetLastError());
      timed_end(st, sizeof(T) == 8 ? TK_F32 : TK_GEMM, eu);
      count_launch();
    }
  }
  w.columns_pending = sizeof(T) == 8 && n <= RP_MAX_N;   // the register panels tracked the rows
  if (w.columns_pending) return NEGF_OK;
  dim3 g3((n + 127) / 128, batch);
  pdl_launch(gj_colswap_kernel<T>, g3, 128, 0, st, A, sA, n, w.ipiv);
  NEGF_CUDA_TRY(cudaGetLastError());
  count_launch();
  return NEGF_OK;
}

}  // namespace

namespace {

// n <= NP_MAX_N: panels of NP_C columns
int gj_invert_narrow(double2* A, long long sA, int n, int batch, InvWork& w, cudaStream_t st) {
  NEGF_CUDA_TRY(cudaMemsetAsync(w.info, 0, sizeof(int) * batch, st));
  const long long sR = (long long)NP_C * n;
  for (int k0 = 0; k0 < n; k0 += NP_C) {
    const int kb = std::min(NP_C, n - k0);
    cudaEvent_t ev;
    timed_begin(st, TK_PANEL, 8.0 * n * (double)kb * kb * batch, &ev);
    pdl_launch(gj_panel_narrow_kernel, batch, (n + 31) / 32 * 32, 0, st, A, sA, n, k0, kb, w.ipiv, w.info, w.moves);
    NEGF_CUDA_TRY(cudaGetLastError());
    timed_end(st, TK_PANEL, ev);
    pdl_launch(gj_swap_kernel<double2>, dim3((n + SWAP_WARPS - 1) / SWAP_WARPS, batch), SWAP_WARPS * 32, 0, st, A, sA,
               n, k0, kb, w.ipiv, w.moves, w.rbuf, sR, 0, (double2*)nullptr);
    NEGF_CUDA_TRY(cudaGetLastError());
    timed_begin(st, TK_GEMM, 8.0 * n * (double)(n - kb) * kb * batch, &ev);
    pdl_launch(gj_update_tiles_kernel<NP_C>, dim3((n + NU_M - 1) / NU_M, (n + NU_N - 1) / NU_N, batch), 256, 0, st, A, sA, n,
               k0, kb, w.rbuf, sR);
    NEGF_CUDA_TRY(cudaGetLastError());
    timed_end(st, TK_GEMM, ev);
    count_launch(3);
  }
  pdl_launch(gj_colswap_kernel<double2>, dim3((n + 127) / 128, batch), 128, 0, st, A, sA, n, w.ipiv);
  NEGF_CUDA_TRY(cudaGetLastError());
  count_launch();
  return NEGF_OK;
}

}  // namespace

int zinv_f64(double2* A, long long sA, int n, int batch, InvWork& w, cudaStream_t st, bool wide) {
  if (!wide && n > 0 && n <= NP_MAX_N && batch > 0 && batch <= 65535 && n <= w.n_cap && batch <= w.batch_cap && NP_C <= w.nb)
    return gj_invert_narrow(A, sA, n, batch, w, st);
  return gj_invert<double2>(A, sA, n, batch, w, st);
}

bool cinv_f32_fused_ok(int n, int batch) { return n <= FUSED_MAX_N && batch >= sm_count_cached(); }

int cinv_f32(float2* A, long long sA, int n, int batch, InvWork& w, cudaStream_t st, int form) {
  if (form == 1) {
    if (!cinv_f32_fused_ok(n, batch)) return NEGF_EINVAL;
    if (batch <= 0) return NEGF_OK;
    if (n > w.n_cap || batch > w.batch_cap) return NEGF_EINVAL;
    return gj_invert_fused_f32(A, sA, n, batch, w, st);
  }
  return gj_invert<float2>(A, sA, n, batch, w, st);
}

}  // namespace negf

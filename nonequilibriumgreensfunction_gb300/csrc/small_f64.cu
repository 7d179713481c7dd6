// FP64 solves of small cross-sections (M <= SMALL_MAX_M), one kernel per phase.
//
// A block of a few orbitals is a few microseconds of arithmetic, so a chain of one launch per
// product or panel, as the larger solves use, is all launches and waits.  Here a problem's
// blocks stay in the shared memory of one CTA, or of each CTA of a cluster, through the whole
// phase: the decimation of a lead (Contact_Self_Energy.F90:110-223) until it converges, and the
// two recursive sweeps with the site blocks and traces (Recursive_Greens.F90:2-107,
// Calculate_Gnp.F90:10-114).  Everything is FP64 multiply-adds in the orders of the larger
// path's kernels; inverses are the same Gauss-Jordan elimination with partial pivoting.
//
// Bound: an SM's FP64 pipe (two multiply-adds per clock: 4 M^3 / 2 cycles a product) and, below
// M of about 10, barriers.  A cluster divides the products by columns, each CTA storing its part
// into all of them; the inverses and the O(M^2) steps are repeated in every CTA.
// Measured on GB300 against the larger path: M = 2, 30 slices, an energy at a time 14 -> 0.8 ms;
// M = 36, 4 slices 11 -> 3.7 ms (34 ms with FP64 launches); M = 36, 10 slices, 200 energies in
// one call 30 -> 23 ms.  Beyond SMALL_MAX_M the decimation's blocks do not fit.
#include <algorithm>

#include "negf_internal.cuh"

namespace negf {

namespace {

constexpr int SMALL_THREADS = 256;
constexpr int SR_BLOCKS = 9;    // t, t~, Told L/R, T L/R, tmp, two work blocks
constexpr int RGF_BLOCKS = 6;   // G, column, product, Y, Gamma, work
constexpr int SR_STEPS = 128;   // decimation steps of one launch at most

template <int CS>
__device__ __forceinline__ unsigned cta_rank() {
  if (CS == 1) return 0;
  unsigned r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// all threads that share the problem; shared-memory writes before it, own and remote, are visible
template <int CS>
__device__ __forceinline__ void sync_all() {
  if (CS == 1) __syncthreads();
  else asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// v into place p of every CTA's shared memory
template <int CS>
__device__ __forceinline__ void store_all(double2* p, double2 v) {
  if (CS == 1) {
    *p = v;
    return;
  }
  const uint32_t own = (uint32_t)__cvta_generic_to_shared(p);
#pragma unroll
  for (int r = 0; r < CS; ++r) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(own), "r"(r));
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
  }
}

// C = A B, or C -= A B, in shared memory; C is neither A nor B.  Begins and ends with a barrier.
template <int CS>
__device__ void multiply(double2* C, const double2* A, const double2* B, int n, bool subtract) {
  const int nn = n * n, part = (nn + CS - 1) / CS;
  const int lo = (int)cta_rank<CS>() * part, hi = min(nn, lo + part);
  sync_all<CS>();
  for (int e = lo + (int)threadIdx.x; e < hi; e += SMALL_THREADS) {
    const double2* a = A + e % n;
    const double2* b = B + (long long)(e / n) * n;
    double2 s = make_double2(0.0, 0.0);
    for (int k = 0; k < n; ++k) cfma(s, a[k * n], b[k]);
    store_all<CS>(C + e, subtract ? csub(C[e], s) : s);
  }
  sync_all<CS>();
}

struct InvScratch {
  double2 piv[SMALL_MAX_M], old[SMALL_MAX_M], f[SMALL_MAX_M], tail[SMALL_MAX_M];
  unsigned long long key[SMALL_MAX_M];
  int none;
  int ip[SMALL_MAX_M];
  int info;
};

// bits of |re| + |im|, plus one (they order as the values); 0, no candidate, for a NaN
__device__ __forceinline__ unsigned long long pivot_key(double2 a) {
  const double v = cabs1(a);
  return v == v ? (unsigned long long)__double_as_longlong(v) + 1ULL : 0ULL;
}

// In-place inverse in this CTA's shared memory (every CTA of a cluster does its own copy):
// Gauss-Jordan elimination with partial pivoting (first maximum of |re| + |im| over the rows
// left), the elements of a step spread over all threads without a branch, then the column
// interchanges.  Every warp finds the pivot for itself, from keys that the last step left; the
// first warps scale the pivot row.  INFO into s.info.
__device__ void invert_block(double2* A, int n, InvScratch& s) {
  const int t = threadIdx.x, lane = t & 31;
  const int nn = n * n, di = SMALL_THREADS % n, dj = SMALL_THREADS / n;
  __syncthreads();
  if (t == 0) s.info = 0;
  if (t < n) s.key[t] = pivot_key(A[t]);
  __syncthreads();
  for (int c = 0; c < n; ++c) {
    const double2* col = A + c * n;
    unsigned long long key = 0;
    int at = 0x7fffffff;
    for (int i = lane; i < n; i += 32) {
      const unsigned long long k = i >= c ? s.key[i] : 0ULL;
      if (k > key) { key = k; at = i; }
    }
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32) == hi ? (unsigned)key : 0u);
    int p = __reduce_min_sync(0xffffffffu, ((unsigned)(key >> 32) == hi && (unsigned)key == lo) ? at : 0x7fffffff);
    if (p >= n) p = c;
    if (t < ((n + 31) & ~31)) {
      const double2 pv = col[p];
      const bool zero = pv.x == 0.0 && pv.y == 0.0;
      const double2 d = zero ? pv : small_rcp(pv);
      const bool none = d.x == 0.0 && d.y == 0.0;   // no pivot: the interchange only
      if (t < n) {
        const double2 v = A[t * n + p], f = col[t == p ? c : t];
        s.old[t] = A[t * n + c];
        s.f[t] = none ? make_double2(0.0, 0.0) : f;
        s.piv[t] = none ? v : (t == c ? d : cmul(v, d));
        s.tail[t] = none ? f : cmul(make_double2(-f.x, -f.y), d);
      }
      if (t == 0) {
        s.none = none ? 1 : 0;
        s.ip[c] = p;
        if (zero && s.info == 0) s.info = c + 1;
      }
    }
    __syncthreads();
    const bool none = s.none != 0;
    int i = t % n, j = t / n;
    for (int e = t; e < nn; e += SMALL_THREADS) {
      const double2 v = *(i == p ? &s.old[j] : &A[e]);
      const double2 f = s.f[i], r = s.piv[j];
      const double2 given = *(i == c ? &s.piv[j] : &s.tail[i]);   // the pivot row and column
      double2 w;
      w.x = fma(f.y, r.y, fma(-f.x, r.x, v.x));
      w.y = fma(-f.y, r.x, fma(-f.x, r.y, v.y));
      if (none) w = v;
      if (i == c || j == c) w = given;
      A[e] = w;
      if (j == c + 1) s.key[i] = pivot_key(w);
      i += di;
      j += dj;
      if (i >= n) { i -= n; ++j; }
    }
    __syncthreads();
  }
  if (t < n)
    for (int k = n - 1; k >= 0; --k) {
      const int p = s.ip[k];
      if (p != k) {
        const double2 v = A[k * n + t];
        A[k * n + t] = A[p * n + t];
        A[p * n + t] = v;
      }
    }
  __syncthreads();
}

// H(s no + a, s no + c) of the site-diagonal hop
__device__ __forceinline__ double2 hop_at(const HopBD& h, int s, int a, int c) {
  return h.hb[((long long)s * h.norb + a) * h.norb + c];
}

// (L X)(i, j) with L = H (herm false) or H^H
__device__ __forceinline__ double2 hop_left(const HopBD& h, bool herm, const double2* X, int n, int i, int j) {
  const int no = h.norb, s = i / no, ai = i % no;
  double2 acc = make_double2(0.0, 0.0);
  for (int p = 0; p < no; ++p)
    cfma(acc, herm ? cconj(hop_at(h, s, p, ai)) : hop_at(h, s, ai, p), X[j * n + s * no + p]);
  return acc;
}
// (X R)(i, j) with R = H or H^H
__device__ __forceinline__ double2 hop_right(const HopBD& h, bool herm, const double2* X, int n, int i, int j) {
  const int no = h.norb, s = j / no, aj = j % no;
  double2 acc = make_double2(0.0, 0.0);
  for (int q = 0; q < no; ++q)
    cfma(acc, X[(s * no + q) * n + i], herm ? cconj(hop_at(h, s, aj, q)) : hop_at(h, s, q, aj));
  return acc;
}
// Sum of one value per thread over the CTA, in a fixed order
__device__ double cta_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  for (int w = 0; w < SMALL_THREADS / 32; ++w) s += red[w];
  return s;
}

// The decimation of problem blockIdx.x / CS (Contact_Self_Energy.F90:110-223): the state is
// taken from and left in a.state between launches of at most SR_STEPS steps; when no lead of
// the problem is active any more, its self-energies are formed (:195-209) and a.done set.
template <int CS>
__global__ void __launch_bounds__(SMALL_THREADS) small_sr_kernel(SmallSr a) {
  extern __shared__ __align__(16) double2 blocks[];
  __shared__ InvScratch inv;
  __shared__ double red[SMALL_THREADS / 32];
  __shared__ unsigned long long cmax;
  const int s = blockIdx.x / CS, n = a.n, nn = n * n, t = threadIdx.x;
  const bool writes = cta_rank<CS>() == 0;
  double2* buf[SR_BLOCKS];
#pragma unroll
  for (int i = 0; i < SR_BLOCKS; ++i) buf[i] = blocks + i * nn;
  double2 *T = buf[0], *TT = buf[1], *told[2] = {buf[2], buf[3]}, *sum[2] = {buf[4], buf[5]}, *tmp = buf[6],
          *w1 = buf[7], *w2 = buf[8];
  double2* state = a.state + (long long)s * 6 * nn;
  const double2* H = a.hend[s];
  const double energy = a.energies[s];
  int act[2] = {a.active[s], a.active[a.count + s]};
  const int want[2] = {a.want[s], a.want[a.count + s]};
  int status = a.status[s], info = 0, steps[2] = {a.iters[s], a.iters[a.count + s]};
  if (a.done[s]) {
    sync_all<CS>();
    return;
  }
  auto alpha = [&](int e, double extra) -> double2 {   // (E + i eta) I - H_end (:71-74 / :83-86)
    double2 v = make_double2(-H[e].x, -H[e].y);
    if (e % n == e / n) { v.x += energy; v.y += a.eta + extra; }
    return v;
  };
  auto note = [&]() { if (info == 0) info = inv.info; };
  if (a.first_step == 0) {
    for (int e = t; e < nn; e += SMALL_THREADS) tmp[e] = alpha(e, a.eta);   // (:141)
    invert_block(tmp, n, inv);
    note();
    for (int e = t; e < nn; e += SMALL_THREADS) {   // t = g0 H, t~ = g0 H^H (:147-151)
      T[e] = hop_right(a.hop, false, tmp, n, e % n, e / n);
      TT[e] = hop_right(a.hop, true, tmp, n, e % n, e / n);
      sum[0][e] = T[e];
      sum[1][e] = TT[e];
      told[0][e] = told[1][e] = make_double2(e % n == e / n ? 1.0 : 0.0, 0.0);
    }
  } else {
    for (int e = t; e < nn; e += SMALL_THREADS) {
      T[e] = state[e];
      TT[e] = state[nn + e];
      told[0][e] = state[2 * nn + e];
      told[1][e] = state[3 * nn + e];
      sum[0][e] = state[4 * nn + e];
      sum[1][e] = state[5 * nn + e];
    }
  }
  int it = a.first_step;
  const int stop = min(a.max_iter, a.first_step + SR_STEPS);
  while ((act[0] || act[1]) && it < stop) {
    ++it;
    for (int l = 0; l < 2; ++l) {   // Told_L <- Told_L t~, Told_R <- Told_R t (:157-158)
      if (!want[l]) continue;
      multiply<CS>(w1, told[l], l == 0 ? TT : T, n, false);
      double2* x = told[l];
      told[l] = w1;
      w1 = x;
    }
    for (int e = t; e < nn; e += SMALL_THREADS) tmp[e] = make_double2(e % n == e / n ? 1.0 : 0.0, 0.0);
    multiply<CS>(tmp, T, TT, n, true);   // inv(I - t t~ - t~ t) (:160-163)
    multiply<CS>(tmp, TT, T, n, true);
    invert_block(tmp, n, inv);
    note();
    multiply<CS>(w1, tmp, T, n, false);   // t <- tmp t t, t~ <- tmp t~ t~ (:170-176)
    multiply<CS>(w2, w1, T, n, false);
    { double2* x = T; T = w2; w2 = x; }
    multiply<CS>(w1, tmp, TT, n, false);
    multiply<CS>(w2, w1, TT, n, false);
    { double2* x = TT; TT = w2; w2 = x; }
    for (int l = 0; l < 2; ++l) {   // change = Told t, T += change (:178-191)
      if (!want[l]) continue;
      multiply<CS>(w1, told[l], l == 0 ? T : TT, n, false);
      if (t == 0) cmax = 0;
      __syncthreads();
      double m = 0.0;
      for (int e = t; e < nn; e += SMALL_THREADS) {
        const double2 v = w1[e];
        m = max_or_nan(m, hypot(v.x, v.y));
        if (act[l]) sum[l][e] = cadd(sum[l][e], v);
      }
      atomicMax(&cmax, (unsigned long long)__double_as_longlong(m));   // (a NaN's bits exceed all others)
      __syncthreads();
      const double c = __longlong_as_double((long long)cmax);
      if (act[l] && isnan(c)) {
        status = NEGF_ENAN;
        act[l] = 0;
        steps[l] = it;
      } else if (act[l] && !(c > a.tol)) {
        act[l] = 0;
        steps[l] = it;
      }
      __syncthreads();
    }
  }
  if (it >= a.max_iter)
    for (int l = 0; l < 2; ++l)
      if (act[l]) {
        steps[l] = it;
        if (status == 0 || status > 0) status = NEGF_ESR_NOCONV;
        act[l] = 0;
      }
  const bool finished = !act[0] && !act[1];
  if (!finished && writes) {
    for (int e = t; e < nn; e += SMALL_THREADS) {
      state[e] = T[e];
      state[nn + e] = TT[e];
      state[2 * nn + e] = told[0][e];
      state[3 * nn + e] = told[1][e];
      state[4 * nn + e] = sum[0][e];
      state[5 * nn + e] = sum[1][e];
    }
  }
  // g = inv(alpha + beta T), Sigma = beta g beta^H (:195-209), Gamma and the contact DOS (:94-101)
  if (finished)
    for (int l = 0; l < 2; ++l) {
      if (!want[l]) continue;
      __syncthreads();
      for (int e = t; e < nn; e += SMALL_THREADS)
        tmp[e] = csub(alpha(e, 0.0), hop_left(a.hop, l == 0, sum[l], n, e % n, e / n));
      invert_block(tmp, n, inv);
      note();
      for (int e = t; e < nn; e += SMALL_THREADS) w2[e] = hop_right(a.hop, l == 1, tmp, n, e % n, e / n);
      __syncthreads();
      for (int e = t; e < nn; e += SMALL_THREADS) w1[e] = hop_left(a.hop, l == 0, w2, n, e % n, e / n);
      __syncthreads();
      double2* sig = (l == 0 ? a.sigL : a.sigR) + (long long)s * nn;
      double2* gam = (l == 0 ? a.gamL : a.gamR) + (long long)s * nn;
      if (writes)
        for (int e = t; e < nn; e += SMALL_THREADS) {
          const double2 v = w1[e], h = w1[(e % n) * n + e / n];
          sig[e] = v;
          gam[e] = make_double2(-(v.y + h.y), v.x - h.x);
        }
      double d = 0.0;
      for (int i = t; i < n; i += SMALL_THREADS) d += w1[i * n + i].y;
      d = cta_sum(d, red);
      if (writes && t == 0) a.dos[l * a.count + s] = -d / 3.14159265358979323846;
    }
  if (writes && t == 0) {
    a.active[s] = act[0];
    a.active[a.count + s] = act[1];
    a.iters[s] = steps[0];
    a.iters[a.count + s] = steps[1];
    a.status[s] = status == 0 ? info : status;   // (an INFO gives way to a later NaN or cap)
    a.done[s] = finished ? 1 : 0;
  }
  sync_all<CS>();   // no CTA leaves while another may still store into its shared memory
}

// Both sweeps of item blockIdx.x / CS, with the site blocks of Gn and the end-block traces
// (Engine::solve_rgf_impl's order of slices and products)
template <int CS>
__global__ void __launch_bounds__(SMALL_THREADS) small_rgf_kernel(SmallRgf a) {
  extern __shared__ __align__(16) double2 blocks[];
  __shared__ InvScratch inv;
  __shared__ double red[SMALL_THREADS / 32];
  const int b = blockIdx.x / CS, n = a.n, nn = n * n, t = threadIdx.x, N = a.npx, no = a.hop.norb;
  const bool writes = cta_rank<CS>() == 0;
  double2 *G = blocks, *col = blocks + nn, *Z = blocks + 2 * nn, *Y = blocks + 3 * nn, *gam = blocks + 4 * nn,
          *Q = blocks + 5 * nn;
  const Item item = a.items[b];
  const double2* H = a.Hall + (long long)item.slot * N * nn;
  const double2 *sigL = a.sigL + (long long)item.sr_l * nn, *sigR = a.sigR + (long long)item.sr_r * nn;
  const double2 *gamL = a.gamL + (long long)item.sr_l * nn, *gamR = a.gamR + (long long)item.sr_r * nn;
  double2* store = a.G + (long long)b * N * nn;
  int status = 0;
  // W of slice x and its inverse into G; G holds the neighbour's (side 0: left, side 1: right)
  auto next = [&](int x, int side, bool coupled) {
    __syncthreads();
    if (coupled) {   // L G R: side 0 H^H G H, side 1 H G H^H
      for (int e = t; e < nn; e += SMALL_THREADS) Z[e] = hop_right(a.hop, side == 1, G, n, e % n, e / n);
      __syncthreads();
    }
    for (int e = t; e < nn; e += SMALL_THREADS) {
      const double2 h = H[(long long)x * nn + e];
      double2 v = make_double2(-h.x, -h.y);
      if (e % n == e / n) { v.x += item.energy; v.y += a.eta; }
      if (x == 0) v = csub(v, sigL[e]);
      if (x == N - 1) v = csub(v, sigR[e]);
      if (coupled) v = csub(v, hop_left(a.hop, side == 0, Z, n, e % n, e / n));
      Q[e] = v;
    }
    invert_block(Q, n, inv);
    if (status == 0 && inv.info != 0) status = inv.info;
    double2* q = G;
    G = Q;
    Q = q;
    if (writes)
      for (int e = t; e < nn; e += SMALL_THREADS) store[(long long)x * nn + e] = G[e];
  };
  // column block <- (the stored block of slice x) (hop) (column block)
  auto advance = [&](int x, bool herm) {
    __syncthreads();
    for (int e = t; e < nn; e += SMALL_THREADS) {
      Z[e] = hop_left(a.hop, herm, col, n, e % n, e / n);
      Q[e] = store[(long long)x * nn + e];
    }
    multiply<CS>(col, Q, Z, n, false);
  };
  // P = Y col^H on the site blocks of slice x, Y = col gam
  auto site = [&](int x, double2* P) {
    multiply<CS>(Y, col, gam, n, false);
    double2* out = P + ((long long)b * N + x) * n * no;
    const int count = n * no, part = (count + CS - 1) / CS;
    const int lo = (int)cta_rank<CS>() * part, hi = min(count, lo + part);
    for (int e = lo + t; e < hi; e += SMALL_THREADS) {
      const int r = e / no, c = (r / no) * no + e % no;
      double2 s = make_double2(0.0, 0.0);
      for (int k = 0; k < n; ++k) cfma(s, Y[k * n + r], cconj(col[k * n + c]));
      out[e] = s;
    }
  };
  // Re Tr[g Y col^H], g in global memory; leaves gam's buffer alone
  auto trace = [&](const double2* g, int which) {
    __syncthreads();
    for (int e = t; e < nn; e += SMALL_THREADS) Z[e] = g[e];
    multiply<CS>(Q, Z, Y, n, false);
    double s = 0.0;
    for (int e = t; e < nn; e += SMALL_THREADS) {
      s = fma(Q[e].x, col[e].x, s);
      s = fma(Q[e].y, col[e].y, s);
    }
    s = cta_sum(s, red);
    if (writes && t == 0) a.traces[(long long)b * 4 + which] = s;
  };
  // right-connected sweep (Recursive_Greens.F90:67-86)
  for (int x = N - 1; x >= 0; --x) next(x, 1, x < N - 1);
  // forward: column 1 and the left-connected blocks (:88-96, :16-34).  G(1,1) = gR_1 is in G;
  // the other CTAs' copies of the store are behind a cluster barrier
  sync_all<CS>();
  for (int e = t; e < nn; e += SMALL_THREADS) {
    gam[e] = gamL[e];
    col[e] = G[e];
  }
  for (int x = 0; x < N; ++x) {
    if (x > 0) advance(x, true);
    site(x, a.P1);
    if (x == 0) trace(gamL, 0);
    if (x == N - 1) trace(gamR, 2);
    next(x, 0, x > 0);
  }
  // backward: column N (:53-63)
  sync_all<CS>();
  for (int e = t; e < nn; e += SMALL_THREADS) {
    gam[e] = gamR[e];
    col[e] = G[e];
  }
  for (int x = N - 1; x >= 0; --x) {
    if (x < N - 1) advance(x, false);
    site(x, a.P2);
    if (x == 0) trace(gamL, 1);
    if (x == N - 1) trace(gamR, 3);
  }
  if (writes && t == 0) a.status[b] = status;
  sync_all<CS>();
}

// nblocks: M x M blocks of a CTA
template <typename K, typename A>
int launch(K kernel, int cs, int count, int nblocks, const A& a, cudaStream_t st) {
  const size_t block = sizeof(double2) * nblocks;
  const size_t smem = block * a.n * a.n;
  NEGF_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(block * SMALL_MAX_M * SMALL_MAX_M)));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(count * cs));
  cfg.blockDim = dim3(SMALL_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cs;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  NEGF_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, a));
  count_launch();
  return NEGF_OK;
}

// CTAs of a problem.  Small blocks are barriers rather than arithmetic, and clusters that share
// SMs lose what they divide.  Whole calls of 10 slices on GB300, one CTA / two / four / eight:
//   M = 16:  1 problem 1.64 / 1.52 / 1.52 / 1.52 ms, 200 problems 2.68 / 3.16 / 4.57 / 7.76 ms
//   M = 36:  1 problem 10.2 / 7.3 / 6.2 / 5.4 ms, 19 problems 13.5 / 9.3 / 7.7 / 11.6 ms,
//            64 problems 13.6 / 9.5 / 15.3 / 28.3 ms, 200 problems 23.3 / 25.1 / 39.6 / 79.0 ms
int cluster_size(int n, int count) {
  if (n < 16) return 1;
  if (count * 8 <= 80) return 8;
  if (count * 4 <= 80) return 4;
  return count * 2 <= 152 ? 2 : 1;
}

template <typename A>
int launch_sized(int cs, int count, int nblocks, const A& a, cudaStream_t st, void (*k1)(A), void (*k2)(A),
                 void (*k4)(A), void (*k8)(A)) {
  return launch(cs == 8 ? k8 : cs == 4 ? k4 : cs == 2 ? k2 : k1, cs, count, nblocks, a, st);
}

}  // namespace

int small_sr_steps() { return SR_STEPS; }

int small_sr(const SmallSr& a, cudaStream_t st) {
  return launch_sized(cluster_size(a.n, a.count), a.count, SR_BLOCKS, a, st,
                      small_sr_kernel<1>, small_sr_kernel<2>, small_sr_kernel<4>, small_sr_kernel<8>);
}

int small_rgf(const SmallRgf& a, int count, cudaStream_t st) {
  return launch_sized(cluster_size(a.n, count), count, RGF_BLOCKS, a, st,
                      small_rgf_kernel<1>, small_rgf_kernel<2>, small_rgf_kernel<4>, small_rgf_kernel<8>);
}

}  // namespace negf

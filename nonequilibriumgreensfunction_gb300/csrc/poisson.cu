// Electrostatics of the self-consistent bias point on the device: the role of SIP_V1
// (Source/SIP_Solver.F90:36-201) in the Poisson <-> NEGF loop of Source/NEGF_Main.F90:7-38.
//
// The system is the 7-point Laplacian on the npx x npy x npz site grid with Dirichlet
// values outside it (contacts at x = -1 and x = npx, a gate on every y and z face):
//     6 U_i - sum_{in-grid neighbours j} U_j = kappa rho_i + (boundary values next to i).
// It is symmetric positive definite, so it is solved by conjugate gradients instead of the
// reference's strongly implicit procedure, whose recurrences run along all three axes and
// leave a GPU idle.  A grid has at most a few 10^4 sites, so one CTA solves one grid with
// its four vectors in global memory (they stay in L2), and the dot products are block
// reductions in a fixed order: the result is deterministic.  Grids of different disorder
// samples are independent CTAs of one launch.  A few grids take a cluster of CTAs each.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "negf_internal.cuh"

namespace negf {

namespace {

constexpr int PCG_THREADS = 1024;

__device__ __forceinline__ double apply_a(const double* v, int i, int nx, int ny, int nz) {
  const int x = i % nx, yz = i / nx, y = yz % ny, z = yz / ny;
  double s = 6.0 * v[i];
  if (x > 0) s -= v[i - 1];
  if (x < nx - 1) s -= v[i + 1];
  if (y > 0) s -= v[i - nx];
  if (y < ny - 1) s -= v[i + nx];
  if (z > 0) s -= v[i - nx * ny];
  if (z < nz - 1) s -= v[i + nx * ny];
  return s;
}

// sum over the CTA in a fixed order; every thread gets the result
__device__ double block_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  if (w == 0) {
    double t = l < (int)(blockDim.x >> 5) ? red[l] : 0.0;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (l == 0) red[32] = t;
  }
  __syncthreads();
  return red[32];
}

// b: right-hand sides, u: initial guesses -> solutions, work: 3 vectors per grid.
// Stops when ||b - A u|| <= tol ||b|| or after max_iter steps (a bounded loop).
__global__ void __launch_bounds__(PCG_THREADS) poisson_cg_kernel(int nx, int ny, int nz, const double* b, double* u,
                                                                 double* work, double tol, int max_iter, int* iters,
                                                                 double* rel) {
  __shared__ double red[33];
  const int n = nx * ny * nz;
  const long long g = blockIdx.x;
  const double* bg = b + g * n;
  double* ug = u + g * n;
  double* r = work + g * 3LL * n;
  double* p = r + n;
  double* q = p + n;
  double rr = 0.0, bb = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double ri = bg[i] - apply_a(ug, i, nx, ny, nz);
    r[i] = ri;
    p[i] = ri;
    rr += ri * ri;
    bb += bg[i] * bg[i];
  }
  rr = block_sum(rr, red);
  bb = block_sum(bb, red);
  const double thr = tol * tol * bb;
  int it = 0;
  for (; it < max_iter && rr > thr; ++it) {
    double pq = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const double qi = apply_a(p, i, nx, ny, nz);
      q[i] = qi;
      pq += p[i] * qi;
    }
    pq = block_sum(pq, red);
    if (!(pq > 0.0)) break;             // breakdown (cannot happen for an SPD operator)
    const double alpha = rr / pq;
    double rn = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      ug[i] += alpha * p[i];
      const double ri = r[i] - alpha * q[i];
      r[i] = ri;
      rn += ri * ri;
    }
    rn = block_sum(rn, red);
    const double beta = rn / rr;
    rr = rn;
    for (int i = threadIdx.x; i < n; i += blockDim.x) p[i] = r[i] + beta * p[i];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    iters[g] = it;
    rel[g] = bb > 0.0 ? sqrt(rr / bb) : sqrt(rr);
  }
}

// The same iteration with a grid on a cluster of PCL_CTAS CTAs.  One CTA is bound by its SM's
// FP64 pipe (two multiply-adds per clock: 12 n of them a step, 26 us at n = 8640) and by the
// latency of its loads from L2; a cluster divides the first and keeps every vector in shared
// memory, reading a neighbour's p from the CTA that holds it.  The dot products are added up
// element by element, thread by thread and warp by warp exactly as poisson_cg_kernel adds them,
// so the iterates and the iteration count are the same bits.  What is left is latency: three
// cluster barriers a step.
// Measured on GB300 with the copies of a whole call (114 steps of 60 x 12 x 12 sites): one grid
// 4.55 -> 1.08 ms, 8 grids 4.67 -> 1.37 ms; 200 x 14 x 14: 21.3 -> 3.2 ms.  Eight CTAs of 256
// threads: 1.26 and 1.40 ms; sixteen of 256: 1.08 and 1.61 ms (clusters share SMs).
constexpr int PCL_CTAS = 16, PCL_T = PCG_THREADS / PCL_CTAS, PCL_THREADS = 128;

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t peer_addr(const void* p, unsigned rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ double peer_load(uint32_t a) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void peer_store(uint32_t a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

__global__ void __launch_bounds__(PCL_THREADS) poisson_cg_cluster_kernel(int nx, int ny, int nz, const double* b,
                                                                         double* u, double tol, int max_iter,
                                                                         int* iters, double* rel) {
  extern __shared__ __align__(16) double pcl[];
  __shared__ double red[2][32];   // the 32 warps' sums, alternating between reductions
  const int n = nx * ny * nz;
  const int rows = (n + PCG_THREADS - 1) / PCG_THREADS;
  const int per = rows * PCL_T;   // elements of a CTA, at most
  double* us = pcl;          // element i = v + 1024 k of summing thread v: place k PCL_T + v % PCL_T
  double* rs = us + per;     // of CTA v / PCL_T
  double* qs = rs + per;
  double* ps = qs + per;
  unsigned char* nb = reinterpret_cast<unsigned char*>(ps + per);   // its neighbours inside the grid
  unsigned rank;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const long long g = blockIdx.x / PCL_CTAS;
  const double* bg = b + g * n;
  double* ug = u + g * n;
  const int t = threadIdx.x, lane = t & 31;
  auto index = [&](int e) -> int { return (int)rank * PCL_T + (e % PCL_T) + (e / PCL_T) * PCG_THREADS; };
  // The first PCL_T threads add their elements up one after the other, as poisson_cg_kernel's
  // threads do; the rest of a step is spread over all threads of the CTA.
  const bool adds = t < PCL_T;
  const int first = (int)rank * PCL_T + t;
  const int mine = adds && first < n ? (n - first + PCG_THREADS - 1) / PCG_THREADS : 0;
  int turn = 0;
  auto total = [&](double v) -> double {
    if (adds) {
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      v = __shfl_sync(0xffffffffu, v, 0);
      if (lane < PCL_CTAS) peer_store(peer_addr(&red[turn][first >> 5], lane), v);
    }
    cluster_sync();
    double s = red[turn][lane];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    turn ^= 1;
    return __shfl_sync(0xffffffffu, s, 0);
  };
  auto at = [&](const double* base, int i) -> double {
    const int v = i & (PCG_THREADS - 1);
    return peer_load(peer_addr(base + (i / PCG_THREADS) * PCL_T + (v & (PCL_T - 1)), (unsigned)(v / PCL_T)));
  };
  auto apply = [&](const double* base, int i, int e) -> double {
    const int has = nb[e];
    // every neighbour's load before the sum; an element without one reads its own place
    const double x0 = at(base, has & 1 ? i - 1 : i), x1 = at(base, has & 2 ? i + 1 : i);
    const double y0 = at(base, has & 4 ? i - nx : i), y1 = at(base, has & 8 ? i + nx : i);
    const double z0 = at(base, has & 16 ? i - nx * ny : i), z1 = at(base, has & 32 ? i + nx * ny : i);
    double s = 6.0 * base[e];
    if (has & 1) s -= x0;
    if (has & 2) s -= x1;
    if (has & 4) s -= y0;
    if (has & 8) s -= y1;
    if (has & 16) s -= z0;
    if (has & 32) s -= z1;
    return s;
  };
  for (int e = t; e < per; e += PCL_THREADS) {
    const int i = index(e);
    if (i >= n) continue;
    const int x = i % nx, yz = i / nx, y = yz % ny, z = yz / ny;
    nb[e] = (unsigned char)((x > 0) | (x < nx - 1) << 1 | (y > 0) << 2 | (y < ny - 1) << 3 | (z > 0) << 4 |
                            (z < nz - 1) << 5);
    us[e] = ug[i];
  }
  cluster_sync();
  for (int e = t; e < per; e += PCL_THREADS) {
    const int i = index(e);
    if (i >= n) continue;
    const double ri = bg[i] - apply(us, i, e);
    rs[e] = ri;
    ps[e] = ri;
  }
  __syncthreads();
  double rr = 0.0, bb = 0.0;
  for (int k = 0; k < mine; ++k) {
    const double ri = rs[t + k * PCL_T], bi = bg[first + k * PCG_THREADS];
    rr += ri * ri;
    bb += bi * bi;
  }
  rr = total(rr);
  bb = total(bb);   // (the barriers also order ps before the first step)
  const double thr = tol * tol * bb;
  int it = 0;
  for (; it < max_iter && rr > thr; ++it) {
    for (int e = t; e < per; e += PCL_THREADS) {
      const int i = index(e);
      if (i < n) qs[e] = apply(ps, i, e);
    }
    __syncthreads();
    double pq = 0.0;
    for (int k = 0; k < mine; ++k) pq += ps[t + k * PCL_T] * qs[t + k * PCL_T];
    pq = total(pq);
    if (!(pq > 0.0)) break;             // breakdown (cannot happen for an SPD operator)
    const double alpha = rr / pq;
    for (int e = t; e < per; e += PCL_THREADS) {
      if (index(e) >= n) continue;
      us[e] += alpha * ps[e];
      rs[e] = rs[e] - alpha * qs[e];
    }
    __syncthreads();
    double rn = 0.0;
    for (int k = 0; k < mine; ++k) rn += rs[t + k * PCL_T] * rs[t + k * PCL_T];
    rn = total(rn);
    const double beta = rn / rr;
    rr = rn;
    for (int e = t; e < per; e += PCL_THREADS)
      if (index(e) < n) ps[e] = rs[e] + beta * ps[e];
    cluster_sync();
  }
  for (int e = t; e < per; e += PCL_THREADS)
    if (index(e) < n) ug[index(e)] = us[e];
  if (rank == 0 && t == 0) {
    iters[g] = it;
    rel[g] = bb > 0.0 ? sqrt(rr / bb) : sqrt(rr);
  }
  cluster_sync();   // no CTA leaves while another may still read its shared memory
}

// b = kappa rho + the Dirichlet values of the neighbours outside the grid
__global__ void poisson_rhs_kernel(int nx, int ny, int nz, int grids, const double* rho, double kappa, double ul,
                                   double ur, double ug, double* b) {
  const long long n = (long long)nx * ny * nz;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n * grids;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % n);
    const int x = i % nx, yz = i / nx, y = yz % ny, z = yz / ny;
    double v = kappa * rho[e];
    if (x == 0) v += ul;
    if (x == nx - 1) v += ur;
    if (y == 0) v += ug;
    if (y == ny - 1) v += ug;
    if (z == 0) v += ug;
    if (z == nz - 1) v += ug;
    b[e] = v;
  }
}

// Up to this many grids take a cluster each.  Beyond, the clusters queue for the SMs while one
// CTA per grid still has an SM to itself: 40 grids of 60 x 12 x 12 take 2.7 against 5.1 ms, 80
// grids 5.5 against 5.4 ms, 64 grids of 16 x 8 x 8 1.17 against 1.09 ms.  Small grids are barriers
// rather than arithmetic and gain less from a cluster, so fewer of them pay for the queue, one CTA
// against a cluster: 81 sites, 20 grids 0.41 / 0.39 ms, 24 0.41 / 0.43, 40 0.41 / 0.46; 256 sites, 20
// 0.49 / 0.47, 24 0.50 / 0.51, 40 0.50 / 0.59; 500 sites, 32 0.66 / 0.62, 40 0.66 / 0.68; 1024 sites,
// 40 1.05 / 0.86.
constexpr int pcl_max_grids(long long n) { return n < 400 ? 20 : n < 640 ? 32 : 40; }
constexpr int PCL_SMEM_MAX = 200 * 1024;

// *done: launched; otherwise the grids do not fit clusters
int launch_clustered(int nx, int ny, int nz, int grids, const double* b, double* u, double tol, int max_iter, int* iters,
                     double* rel, bool* done) {
  const long long n = (long long)nx * ny * nz;
  const long long per = (n + PCG_THREADS - 1) / PCG_THREADS * PCL_T;
  const long long smem = per * (4 * (long long)sizeof(double) + 1);
  if (grids > pcl_max_grids(n) || smem > PCL_SMEM_MAX) return NEGF_OK;
  NEGF_CUDA_TRY(cudaFuncSetAttribute(poisson_cg_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PCL_SMEM_MAX));
  NEGF_CUDA_TRY(cudaFuncSetAttribute(poisson_cg_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(grids * PCL_CTAS));
  cfg.blockDim = dim3(PCL_THREADS);
  cfg.dynamicSmemBytes = (size_t)smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = PCL_CTAS;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int fit = 0;
  if (cudaOccupancyMaxActiveClusters(&fit, poisson_cg_cluster_kernel, &cfg) != cudaSuccess || fit < 1) {
    cudaGetLastError();   // no room for such a cluster on this device: one CTA per grid
    return NEGF_OK;
  }
  NEGF_CUDA_TRY(cudaLaunchKernelEx(&cfg, poisson_cg_cluster_kernel, nx, ny, nz, b, u, tol, max_iter, iters, rel));
  *done = true;
  return NEGF_OK;
}

struct DevMem {
  void* p = nullptr;
  ~DevMem() { if (p) cudaFree(p); }
  int alloc(size_t bytes) { return cudaMalloc(&p, bytes) == cudaSuccess ? NEGF_OK : NEGF_ENOMEM; }
};

}  // namespace

}  // namespace negf

extern "C" int negf_poisson_solve(int32_t npx, int32_t npy, int32_t npz, int32_t n_grids, const double* rho,
                                  const double* bc, double kappa, double* U, double tol, int32_t max_iter,
                                  int32_t* iters) {
  using namespace negf;
  if (npx < 1 || npy < 1 || npz < 1 || n_grids < 1 || !rho || !bc || !U || !(tol >= 0.0) || max_iter < 0)
    return NEGF_EINVAL;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return NEGF_ENODEV;
  const long long n = (long long)npx * npy * npz;
  if (n > (1LL << 28)) return NEGF_EINVAL;
  const size_t vec = sizeof(double) * n * n_grids;
  for (long long i = 0; i < n * n_grids; ++i)
    if (!std::isfinite(rho[i])) return NEGF_ENAN;
  for (int i = 0; i < 3; ++i)
    if (!std::isfinite(bc[i])) return NEGF_EINVAL;
  DevMem dRho, dB, dU, dW, dIt, dRel;
  NEGF_TRY(dRho.alloc(vec));
  NEGF_TRY(dB.alloc(vec));
  NEGF_TRY(dU.alloc(vec));
  NEGF_TRY(dW.alloc(3 * vec));
  NEGF_TRY(dIt.alloc(sizeof(int) * n_grids));
  NEGF_TRY(dRel.alloc(sizeof(double) * n_grids));
  NEGF_CUDA_TRY(cudaMemcpy(dRho.p, rho, vec, cudaMemcpyHostToDevice));
  NEGF_CUDA_TRY(cudaMemcpy(dU.p, U, vec, cudaMemcpyHostToDevice));
  const long long total = n * n_grids;
  const int blocks = (int)std::min<long long>((total + 255) / 256, 1024);
  poisson_rhs_kernel<<<blocks, 256>>>(npx, npy, npz, n_grids, (const double*)dRho.p, kappa, bc[0], bc[1], bc[2],
                                      (double*)dB.p);
  NEGF_CUDA_TRY(cudaGetLastError());
  count_launch();
  bool clustered = false;
  NEGF_TRY(launch_clustered(npx, npy, npz, n_grids, (const double*)dB.p, (double*)dU.p, tol, max_iter, (int*)dIt.p,
                            (double*)dRel.p, &clustered));
  if (!clustered) {
    poisson_cg_kernel<<<n_grids, PCG_THREADS>>>(npx, npy, npz, (const double*)dB.p, (double*)dU.p, (double*)dW.p, tol,
                                                max_iter, (int*)dIt.p, (double*)dRel.p);
    NEGF_CUDA_TRY(cudaGetLastError());
  }
  count_launch();
  NEGF_CUDA_TRY(cudaDeviceSynchronize());
  std::vector<int> it(n_grids);
  std::vector<double> rel(n_grids);
  NEGF_CUDA_TRY(cudaMemcpy(it.data(), dIt.p, sizeof(int) * n_grids, cudaMemcpyDeviceToHost));
  NEGF_CUDA_TRY(cudaMemcpy(rel.data(), dRel.p, sizeof(double) * n_grids, cudaMemcpyDeviceToHost));
  NEGF_CUDA_TRY(cudaMemcpy(U, dU.p, vec, cudaMemcpyDeviceToHost));
  int worst = 0;
  bool ok = true;
  for (int g = 0; g < n_grids; ++g) {
    worst = std::max(worst, it[g]);
    if (!(rel[g] <= tol)) ok = false;
  }
  if (iters) *iters = worst;
  return ok ? NEGF_OK : NEGF_EREFINE;
}

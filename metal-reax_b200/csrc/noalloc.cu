// Charge equilibration for callers that cannot allocate device memory.
//
// Some callers own every byte of device memory themselves: a host code with its own pooled allocator and a fixed
// memory budget (a serving loop that admits work by measured bytes, a framework whose allocator must see every
// allocation), or code that runs where a device allocation and the implicit synchronisation it brings are not
// allowed. rx_qeq_solve_static gives them the charge solve of rx_qeq_solve without any allocation: the caller passes
// the matrix and every input and output as device arrays; the CG work vectors live in one file-scope device array of
// fixed size that the library reserves on every GPU that loads it, for as long as the process runs.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <mutex>

#include "../../include/rxcuda.h"
#include "device.cuh"

namespace cg = cooperative_groups;

namespace rx {
namespace {

constexpr int kStaticMaxAtoms = RX_QEQ_STATIC_MAX_ATOMS;
constexpr int kMaxDevices = 64;
constexpr int kStaticThreads = 1024;
constexpr int kOneBlockThreads = 512;
constexpr int kOneBlockAtoms = 112;   // systems of up to this many atoms are one block's
constexpr int kStaticCluster = 16;   // blocks of the solve's cluster (half as many, and so on, where they cannot be had)

}  // namespace

// CG work vectors r, d, q and, for one block, M^-1 r for the s and t systems (8 doubles per atom; 2 MiB for 32768 atoms).
static __device__ __align__(256) double rx_qeq_static_scratch[static_cast<size_t>(kStaticMaxAtoms) * 8];

namespace {

std::mutex g_mu;
double* g_scratch[kMaxDevices] = {};
int g_cluster[kMaxDevices] = {};

void put_err(char* err, int errlen, const char* msg) {
  if (err && errlen > 0) std::snprintf(err, static_cast<size_t>(errlen), "%s", msg);
}

// One row of (diag(eta) + H) v for both right-hand sides, a warp per row. kFlight entries per lane are loaded before the
// first gather is waited for: a row product is bound by the latency of its dependent index -> vector loads. 3, 4, 5, 6 and 8
// in flight, us a solve: 2592 atoms of water 1083, 1059, 1093, 1080, 1175; 12,000 3576, 3543, 3336, 3744, 3444.
constexpr int kFlight = 5;
__device__ inline double2 csr_row_mv(int i, const int* __restrict__ rs, const int* __restrict__ col, const double* __restrict__ val,
                                     double eta, const double2* v) {
  const int lane = threadIdx.x & 31;
  const int end = rs[i + 1];
  const double2 vi = v[i];
  double ys = 0.0, yt = 0.0;
  for (int e0 = rs[i] + lane; e0 < end; e0 += 32 * kFlight) {
    int c[kFlight];
    double h[kFlight];
#pragma unroll
    for (int k = 0; k < kFlight; ++k) {
      const int e = e0 + 32 * k;
      c[k] = e < end ? col[e] : i;
      h[k] = e < end ? val[e] : 0.0;
    }
    // entries past the row's end: weight 0 on the row's own vector entry, so that no load waits behind a branch
    double2 w[kFlight];
#pragma unroll
    for (int k = 0; k < kFlight; ++k) w[k] = v[c[k]];
#pragma unroll
    for (int k = 0; k < kFlight; ++k) {
      ys += h[k] * w[k].x;
      yt += h[k] * w[k].y;
    }
  }
  double y[2] = {ys, yt};
  const double sum = warp_sums<2>(y);
  return make_double2(eta * vi.x + __shfl_sync(0xffffffffu, sum, 0), eta * vi.y + __shfl_sync(0xffffffffu, sum, 16));
}

// Jacobi-PCG of one system held as a CSR matrix, on one thread-block cluster: solves
// (diag(eta) + H) s = -chi and (diag(eta) + H) t = -1 with the stopping rule of the stock fix (sqrt(r.M^-1 r)/|b| <=
// tol, at most imax - 1 iterations per system), then q = s - (sum s / sum t) t. Every work vector is written before
// it is read, so the previous call's contents of the scratch array never reach the result. A breakdown (a step length
// that is not finite, e.g. a singular or indefinite matrix) stops the loop and is reported as iters = -1 for the
// right-hand side(s) it hit.
//
// The matrix (12 bytes an entry) is read once per iteration, so the solve is bound by how many SMs read it: block r of
// the cluster owns the rows [r n / C, (r + 1) n / C). A cluster's hardware barrier and its blocks' shared memory carry
// the dot products, so the launch is a plain one: no grid-wide barrier whose workspace the driver would have to
// provide. Only the search direction d is read by other blocks; r and q = A d stay with their block.
//
// kOneBlock: the system is one block's, which meets at its own barrier and keeps M^-1 r (a division in FP64 takes longer than the
// rest of a small system's vector update). An iteration of one block, of clusters, us: 24 atoms of water 5.3, 7.9; 64 6.2,
// 8.1; 96 7.5, 8.0; 129 9.8, 9.7; 160 11.6, 9.6.
template <bool kOneBlock>
__global__ void __launch_bounds__(kStaticThreads) k_cg_csr_static(int n, const int* rs, const int* col, const double* val,
                                                                  const double* eta, const double* chi, double* s_io, double* t_io,
                                                                  double* q_out, double tol, int imax, int* iters, double* rel,
                                                                  double* scratch) {
  cg::cluster_group cl = cg::this_cluster();
  double2* r = reinterpret_cast<double2*>(scratch);
  double2* d = r + n;
  double2* qv = d + n;
  double2* p = qv + n;
  __shared__ double sh[32 * 4];
  __shared__ double part[2][4];   // this block's partial sums (two sets in turn: one may still be read by a slower block)
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int nb = static_cast<int>(cl.num_blocks()), rank = static_cast<int>(cl.block_rank());
  const int r0 = static_cast<int>(static_cast<long long>(n) * rank / nb), r1 = static_cast<int>(static_cast<long long>(n) * (rank + 1) / nb);
  auto meet = [&]() {
    if (kOneBlock) __syncthreads();
    else cl.sync();
  };
  int flip = 0;
  // sums over the cluster: warps, then the block's warps in order, then the blocks in order (the same in every block)
  auto reduce = [&](double* v, int nv) {
    for (int k = 0; k < nv; ++k) {
      double x = v[k];
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (lane == 0) sh[wid * 4 + k] = x;
    }
    __syncthreads();
    if (threadIdx.x < nv) {
      double t = 0.0;
      for (int w = 0; w < nw; ++w) t += sh[w * 4 + threadIdx.x];
      part[flip][threadIdx.x] = t;
    }
    meet();
    // lane b of every warp fetches block b's partials; the sums run over the blocks in order
    for (int k = 0; k < nv; ++k) {
      if (kOneBlock) {
        v[k] = part[flip][k];
        continue;
      }
      const double mine = lane < nb ? cl.map_shared_rank(&part[flip][0], static_cast<unsigned>(lane))[k] : 0.0;
      double t = 0.0;
      for (int b = 0; b < nb; ++b) t += __shfl_sync(0xffffffffu, mine, b);
      v[k] = t;
    }
    flip ^= 1;
  };
  // the current iterate lives in d for the first product: copy the caller's guesses there
  for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) d[i] = make_double2(s_io[i], t_io[i]);
  meet();
  double loc[4] = {0.0, 0.0, 0.0, 0.0};
  for (int i = r0 + wid; i < r1; i += nw) {
    const double e = eta[i];
    const double2 y = csr_row_mv(i, rs, col, val, e, d);
    if (lane == 0) {
      const double2 b = make_double2(-chi[i], -1.0);
      const double2 rr = make_double2(b.x - y.x, b.y - y.y);
      r[i] = rr;
      loc[0] += b.x * b.x; loc[1] += b.y * b.y; loc[2] += rr.x * (rr.x / e); loc[3] += rr.y * (rr.y / e);
    }
  }
  reduce(loc, 4);
  // x = guesses (kept in the caller's arrays), d = M^-1 r (no block reads the guesses in d any more)
  for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
    const double2 rr = r[i];
    const double e = eta[i];
    d[i] = make_double2(rr.x / e, rr.y / e);
  }
  meet();
  const double bnorm_s = sqrt(loc[0]), bnorm_t = sqrt(loc[1]);
  double sig_s = loc[2], sig_t = loc[3];
  bool act_s = true, act_t = true, broke_s = false, broke_t = false;
  int it_s = 1, it_t = 1;
  for (int it = 1; it < imax; ++it) {
    act_s = act_s && (sqrt(sig_s) / bnorm_s > tol);
    act_t = act_t && (sqrt(sig_t) / bnorm_t > tol);
    if (!act_s && !act_t) break;
    loc[0] = loc[1] = 0.0;
    for (int i = r0 + wid; i < r1; i += nw) {
      const double2 y = csr_row_mv(i, rs, col, val, eta[i], d);
      if (lane == 0) {
        qv[i] = y;
        const double2 dd = d[i];
        loc[0] += dd.x * y.x; loc[1] += dd.y * y.y;
      }
    }
    reduce(loc, 2);
    const double alpha_s = act_s ? sig_s / loc[0] : 0.0;
    const double alpha_t = act_t ? sig_t / loc[1] : 0.0;
    if (!(isfinite(alpha_s) && isfinite(alpha_t))) {
      broke_s = !isfinite(alpha_s);
      broke_t = !isfinite(alpha_t);
      break;
    }
    loc[0] = loc[1] = 0.0;
    for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
      const double2 dd = d[i], qq = qv[i];
      double2 rr = r[i];
      s_io[i] += alpha_s * dd.x;
      t_io[i] += alpha_t * dd.y;
      rr.x -= alpha_s * qq.x; rr.y -= alpha_t * qq.y;
      r[i] = rr;
      const double e = eta[i];
      const double2 pp = make_double2(rr.x / e, rr.y / e);
      if (kOneBlock) p[i] = pp;
      loc[0] += rr.x * pp.x; loc[1] += rr.y * pp.y;
    }
    reduce(loc, 2);
    const double beta_s = act_s ? loc[0] / sig_s : 0.0;
    const double beta_t = act_t ? loc[1] / sig_t : 0.0;
    if (act_s) { sig_s = loc[0]; it_s = it + 1; }
    if (act_t) { sig_t = loc[1]; it_t = it + 1; }
    for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
      double2 pp, dd = d[i];
      if (kOneBlock) {
        pp = p[i];
      } else {
        const double2 rr = r[i];
        const double e = eta[i];
        pp = make_double2(rr.x / e, rr.y / e);
      }
      if (act_s) dd.x = pp.x + beta_s * dd.x;
      if (act_t) dd.y = pp.y + beta_t * dd.y;
      d[i] = dd;
    }
    meet();
  }
  loc[0] = loc[1] = 0.0;
  for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) { loc[0] += s_io[i]; loc[1] += t_io[i]; }
  reduce(loc, 2);
  const double u = loc[0] / loc[1];
  for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) q_out[i] = s_io[i] - u * t_io[i];
  if (rank == 0 && threadIdx.x == 0) {
    if (iters) { iters[0] = broke_s ? -1 : it_s; iters[1] = broke_t ? -1 : it_t; }
    if (rel) { rel[0] = sqrt(sig_s) / bnorm_s; rel[1] = sqrt(sig_t) / bnorm_t; }
  }
  meet();   // no block leaves while another may still read its partial sums
}

cudaLaunchConfig_t static_launch(int cluster, cudaStream_t stream, cudaLaunchAttribute* at) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(cluster));
  cfg.blockDim = dim3(cluster > 1 ? kStaticThreads : kOneBlockThreads);
  cfg.stream = stream;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = static_cast<unsigned>(cluster);
  at->val.clusterDim.y = 1;
  at->val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = cluster > 1 ? 1 : 0;
  return cfg;
}

}  // namespace
}  // namespace rx

extern "C" int rx_qeq_solve_static(int n, const int* row_start, const int* col, const double* val, const double* eta,
                                   const double* chi, double* s, double* t, double* q, double tol, int imax, int* iters,
                                   double* rel, void* stream, char* err, int errlen) {
  using namespace rx;
  if (n < 0 || n > kStaticMaxAtoms) {
    char m[160];
    std::snprintf(m, sizeof m, "rx_qeq_solve_static: %d atoms; this entry point takes 0 (set-up only) to %d atoms (its fixed work array)", n,
                  kStaticMaxAtoms);
    put_err(err, errlen, m);
    return RX_ERR_INVALID;
  }
  if (n > 0 && (!row_start || !col || !val || !eta || !chi || !s || !t || !q)) {
    put_err(err, errlen, "rx_qeq_solve_static: null device array");
    return RX_ERR_INVALID;
  }
  if (n > 0 && (!(tol > 0.0) || imax < 1)) {
    put_err(err, errlen, "rx_qeq_solve_static: need tol > 0 and imax >= 1");
    return RX_ERR_INVALID;
  }
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    put_err(err, errlen, "rx_qeq_solve_static: no current CUDA device");
    return RX_ERR_CUDA;
  }
  double* scratch = nullptr;
  int cluster = 0;
  {
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_scratch[dev]) {
      // the device address of the work array on this (current) device; the host-side name is not one. Looking it up
      // loads this library's device code on the device (with the array) if lazy module loading has not done so yet;
      // the kernel's attributes are queried too, so that its first launch loads nothing more.
      void* ptr = nullptr;
      cudaError_t e = cudaGetSymbolAddress(&ptr, rx_qeq_static_scratch);
      cudaFuncAttributes fa;
      if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_cg_csr_static<true>);
      if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_cg_csr_static<false>);
      if (e == cudaSuccess) {   // a size that the runtime refuses is one that does not fit; what it leaves behind is cleared
        const bool clean = cudaPeekAtLastError() == cudaSuccess;
        int c = kStaticCluster;
        for (; c > 1; c /= 2) {
          cudaLaunchAttribute at;
          cudaLaunchConfig_t cfg = static_launch(c, nullptr, &at);
          int fits = 0;
          cudaError_t q = c > 8 ? cudaFuncSetAttribute(k_cg_csr_static<false>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) : cudaSuccess;
          if (q == cudaSuccess) q = cudaOccupancyMaxActiveClusters(&fits, k_cg_csr_static<false>, &cfg);
          if (q != cudaSuccess && clean) (void)cudaGetLastError();
          if (q == cudaSuccess && fits > 0) break;
        }
        g_cluster[dev] = c;
      }
      if (e != cudaSuccess) {
        char m[200];
        std::snprintf(m, sizeof m, "rx_qeq_solve_static: set-up on device %d failed: %s", dev, cudaGetErrorString(e));
        put_err(err, errlen, m);
        return RX_ERR_CUDA;
      }
      g_scratch[dev] = static_cast<double*>(ptr);
    }
    scratch = g_scratch[dev];
    cluster = g_cluster[dev];
  }
  if (n == 0) {   // set-up only
    put_err(err, errlen, "");
    return RX_OK;
  }
  cudaLaunchAttribute at;
  // no more blocks than have a row for every warp: a small system's barriers cost more than its rows
  const int rows_per_block = kStaticThreads / 32;
  while (cluster > 1 && (cluster / 2) * rows_per_block >= n) cluster /= 2;
  if (n <= kOneBlockAtoms) cluster = 1;
  const cudaLaunchConfig_t cfg = static_launch(cluster, static_cast<cudaStream_t>(stream), &at);
  (void)cudaLaunchKernelEx(&cfg, cluster > 1 ? k_cg_csr_static<false> : k_cg_csr_static<true>, n, row_start, col, val, eta, chi, s, t, q, tol, imax, iters, rel, scratch);
  // peek, not get: the error state is left as it is for the caller (an error still pending from earlier work on this
  // thread is therefore reported here too)
  const cudaError_t e = cudaPeekAtLastError();
  if (e != cudaSuccess) {
    char m[200];
    std::snprintf(m, sizeof m, "rx_qeq_solve_static: launch failed: %s", cudaGetErrorString(e));
    put_err(err, errlen, m);
    return RX_ERR_CUDA;
  }
  put_err(err, errlen, "");
  return RX_OK;
}

// xm_noalloc.cu -- CONGRAD that allocates nothing (efdc_xm_congrad_noalloc).
//
// Who needs it: callers that cannot let a library allocate device memory --
// a host code that hands all of its GPU memory to its own pool or budget, a
// caller inside a time-critical loop where an allocation could stall or fail,
// or one that only has device arrays it manages itself (CUDA Fortran device
// arrays, a framework's tensors).  They pass device arrays for the system and
// the solution; the solver's own vectors live in one fixed-size array of
// device memory declared at file scope below, which exists on every GPU that
// loads this library, from the library's loading until the process exits.
//
// Everything else in the library (efdc_xm_create and the context API) is
// unchanged; this file adds one entry point beside them.
//
// The algorithm is CONGRAD's Jacobi-preconditioned CG (congrad.f90:54-187) in
// FP64 on the reference's own layout: cells L=2..LA in CELLMAP order with the
// LNC/LSC/LEC/LWC neighbour maps (so periodic links work too).  One cooperative
// launch runs the whole solve: a thread keeps its cells' P, RCG, PCG and APCG
// in registers, the others read z = CCCI*RCG and PCG from the scratch, and the
// two reductions of an iteration are also its barriers.

#include <cstdarg>
#include <algorithm>
#include <cstdio>
#include <mutex>
#include <type_traits>

#include "../../include/efdc_xm.h"
#include "xm_kernels.h"
#include "xm_resident.cuh"

namespace {

constexpr int NA_MAX_CELLS = EFDC_XM_NOALLOC_MAX_CELLS;  // water cells, LA-1
constexpr int NA_LEN = ((NA_MAX_CELLS + 2 + 31) / 32) * 32;  // elements 1..LC, padded
constexpr int NA_GRID = 296;                          // partial sums: blocks of 256 threads
constexpr int NA_HALVES = 2;                          // such blocks per CTA
constexpr int NA_CTL = 16;                            // doubles of the control block
constexpr size_t NA_DOUBLES = size_t(3) * NA_LEN + 4 * NA_GRID + NA_CTL;

// The scratch: z | p | p (by turns) | partial sums (by turns) | control block.  In host code this
// name is only a stand-in for the symbol; its device address comes from
// cudaGetSymbolAddress (see scratch_ptr).
static __device__ __align__(256) double g_na_scratch[NA_DOUBLES];

struct NaCtl {  // lives in the last NA_CTL doubles of the scratch
  double rpcg, alpha, beta, rsq;
  int iter, status;
  unsigned int counter, pad;
};
static_assert(sizeof(NaCtl) <= NA_CTL * sizeof(double), "control block too large");

struct NaArgs {
  int la, lc;
  const int *lnc, *lsc, *lec, *lwc;
  const double *ccc, *ccs, *ccn, *ccw, *cce, *fptmp;
  double *P;
  double *z, *pa, *pb, *part;
  NaCtl *ctl;
  int polls;  // of a wait, before it is given up
};

using xm::NT;
using xm::NWARP;

constexpr int NA_NT = NA_HALVES * NT;

__device__ __forceinline__ double na_tree(const double *w) {  // block_sum's last stage (its
  return ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));  // further lanes add 0)
}

// The barrier of the grid: the CTA adds its arrival with release semantics and waits for
// the others' (bounded).  False (in every thread) when the wait ran out.
__device__ __forceinline__ bool na_meet(const NaArgs &a, unsigned &count) {
  count += gridDim.x;
  int dead = 0;
  if (threadIdx.x == 0) {
    xm::red_release(&a.ctl->counter, 1u);
    for (int k = 0; int(xm::ld_acquire(&a.ctl->counter) - count) < 0; ++k)
      if (k >= a.polls) {
        dead = 1;
        break;
      }
  }
  return !__syncthreads_or(dead);
}

// The sums of NS values of the 512 threads `vb` of the launch (a CTA of k_na_solve): each
// block of 256 threads (half of them) sums its values and stores them.
template <int NS>
__device__ __forceinline__ void na_part(const NaArgs &a, int turn, int vb, const double (&v)[NS]) {
  __shared__ double sh[NS][NA_HALVES][NWARP];
  const int t = threadIdx.x, lane = t & 31, half = t / NT, warp = (t % NT) >> 5;
  double2 *part = reinterpret_cast<double2 *>(a.part) + turn * NA_GRID;
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    const double x = xm::warp_sum(v[s]);
    if (lane == 0) sh[s][half][warp] = x + 0.0;
  }
  __syncthreads();  // also: every thread's stores are before the release in na_meet
  if (t < NA_HALVES)
    part[vb * NA_HALVES + t] =
        make_double2(na_tree(sh[0][t]), NS > 1 ? na_tree(sh[NS - 1][t]) : 0.0);
  if (t < 32) __syncwarp();  // (the arrival is the first warp's)
}

// na_meet, and the sums over all nvb*NA_HALVES blocks' values, in every thread: as one
// block of 256 threads sums them.
template <int NS>
__device__ __forceinline__ bool na_total(const NaArgs &a, unsigned &count, int &turn, int nvb,
                                         double (&out)[NS]) {
  __shared__ double red[NS][NWARP];
  const int t = threadIdx.x, nblk = nvb * NA_HALVES;
  const double2 *part = reinterpret_cast<const double2 *>(a.part) + turn * NA_GRID;
  turn ^= 1;
  if (!na_meet(a, count)) return false;
  if (t < NT) {  // reduce_partials
    double z[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) z[s] = 0.0;
    for (int i = t; i < nblk; i += NT) {
      const double2 x = __ldcg(part + i);
      z[0] += x.x;
      if constexpr (NS > 1) z[1] += x.y;
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const double x = xm::warp_sum(z[s]);
      if ((t & 31) == 0) red[s][t >> 5] = x + 0.0;
    }
  }
  __syncthreads();
#pragma unroll
  for (int s = 0; s < NS; ++s) out[s] = na_tree(red[s]);
  return true;
}

// The sums of a launch whose CTAs are the blocks' pairs.
template <int NS>
__device__ __forceinline__ bool na_sum(const NaArgs &a, unsigned &count, int &turn,
                                       const double (&v)[NS], double (&out)[NS]) {
  na_part(a, turn, blockIdx.x, v);
  return na_total(a, count, turn, gridDim.x, out);
}

// What a solve leaves for the host.  A CTA whose last wait ran out has left its cells
// of P unsolved although the others may have come to the end: its status stays.
__device__ __forceinline__ void na_fail(const NaArgs &a) {
  if (threadIdx.x == 0) atomicExch(&a.ctl->status, EFDC_XM_DEVICE_TIMEOUT);
}
struct NaScalars {
  double rpcg, alpha = 0.0, beta = 0.0, rsq = 0.0;
  int iter = 0, status = EFDC_XM_OK;
  // :88, and :143-169; true when the solve has ended
  __device__ __forceinline__ bool start(double sum) {
    rpcg = sum;
    if (!isfinite(rpcg)) status = EFDC_XM_NONFINITE;
    return rpcg == 0.0 || !isfinite(rpcg);
  }
  __device__ __forceinline__ bool next(const double (&sum)[2], double rsqm, int iterm) {
    beta = sum[0] / rpcg;
    rpcg = sum[0];
    rsq = sum[1];
    ++iter;
    if (!isfinite(rsq) || !isfinite(alpha)) {
      status = EFDC_XM_NONFINITE;
      return true;
    }
    if (rsq <= rsqm) return true;
    if (iter >= iterm) {
      status = EFDC_XM_CG_MAXITER;
      return true;
    }
    return false;
  }
  __device__ __forceinline__ void leave(const NaArgs &a) const {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    a.ctl->rpcg = rpcg;
    a.ctl->alpha = alpha;
    a.ctl->beta = beta;
    a.ctl->rsq = rsq;
    a.ctl->iter = iter;
    atomicCAS(&a.ctl->status, EFDC_XM_OK, status);
  }
};
// congrad.f90:42: PCG(1)=PCG(LC)=0
__device__ __forceinline__ void na_ghosts(const NaArgs &a) {
  if (blockIdx.x == 0 && threadIdx.x == 0)
    for (double *q : {a.z, a.pa, a.pb}) {
      q[0] = 0.0;
      q[a.lc - 1] = 0.0;
    }
}
// RCG of cell L = i + 1 (:72)
__device__ __forceinline__ double na_resid(const NaArgs &a, int i, double c, double x) {
  return a.fptmp[i] - c * x - a.ccn[i] * a.P[a.lnc[i] - 1] - a.ccs[i] * a.P[a.lsc[i] - 1] -
         a.ccw[i] * a.P[a.lwc[i] - 1] - a.cce[i] * a.P[a.lec[i] - 1];
}

// congrad.f90:54-187 with NC cells per thread.  What bounds it is the exchange,
// as for the resident solves (xm_resident.cuh): three kernels per iteration and a
// copy to the host every 8 took 410 us for 16 iterations on 112,000 cells; one
// launch takes 168 us (a call of efdc_xm_congrad_noalloc, its copy of P included).
template <int NC>
__global__ void __launch_bounds__(NA_NT) k_na_solve(NaArgs a, double rsqm, int iterm) {
  const int first = 2 + int(blockIdx.x) * NA_NT + int(threadIdx.x), stride = gridDim.x * NA_NT;
  unsigned count = 0u;
  int turn = 0;
  double x[NC], r[NC], p[NC], ap[NC], ci[NC];
  na_ghosts(a);
  NaScalars q;
  bool done;
  {  // :54-88
    double v[1] = {0.0}, sum[1];
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      const int L = first + k * stride;
      if (L > a.la) continue;
      const int i = L - 1;
      x[k] = a.P[i];
      const double c = a.ccc[i];
      r[k] = na_resid(a, i, c, x[k]);
      ci[k] = 1. / c;
      p[k] = r[k] * ci[k];
      a.z[i] = p[k];
      a.pa[i] = p[k];
      v[0] += r[k] * p[k];
    }
    if (!na_sum(a, count, turn, v, sum)) return na_fail(a);
    done = q.start(sum[0]);
  }
  while (!done) {  // ITERM bounds the loop
    const double *pold = q.iter & 1 ? a.pb : a.pa;
    double *pnew = q.iter & 1 ? a.pa : a.pb;
    {  // :151-162 of the iteration before, :107-125
      double v[1] = {0.0}, sum[1];
#pragma unroll
      for (int k = 0; k < NC; ++k) {
        const int L = first + k * stride;
        if (L > a.la) continue;
        const int i = L - 1;
        auto at = [&](int n) { return __ldcg(a.z + n) + q.beta * __ldcg(pold + n); };
        const double ps = at(__ldg(a.lsc + i) - 1), pn = at(__ldg(a.lnc + i) - 1),
                     pw = at(__ldg(a.lwc + i) - 1), pe = at(__ldg(a.lec + i) - 1);
        p[k] = ci[k] * r[k] + q.beta * p[k];
        pnew[i] = p[k];
        ap[k] = __ldg(a.ccc + i) * p[k] + __ldg(a.ccs + i) * ps + __ldg(a.ccn + i) * pn +
                __ldg(a.ccw + i) * pw + __ldg(a.cce + i) * pe;
        v[0] += ap[k] * p[k];
      }
      if (!na_sum(a, count, turn, v, sum)) return na_fail(a);
      q.alpha = q.rpcg / sum[0];
    }
    {  // :127-149
      double v[2] = {0.0, 0.0}, sum[2];
#pragma unroll
      for (int k = 0; k < NC; ++k) {
        const int L = first + k * stride;
        if (L > a.la) continue;
        x[k] = x[k] + q.alpha * p[k];
        r[k] = r[k] - q.alpha * ap[k];
        const double z = ci[k] * r[k];
        a.z[L - 1] = z;
        v[0] += r[k] * z;
        v[1] += r[k] * r[k];
      }
      if (!na_sum(a, count, turn, v, sum)) return na_fail(a);
      done = q.next(sum, rsqm, iterm);
    }
  }
  if (q.iter > 0)
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      const int L = first + k * stride;
      if (L <= a.la) a.P[L - 1] = x[k];
    }
  q.leave(a);
}

// The same solve where fewer CTAs than that can be resident together (a partition of the
// GPU): each CTA does the work of some of the nvb CTAs of k_na_solve, one after another,
// with RCG, PCG and APCG in the scratch and PCG's update in a pass of its own.  The same
// operations and sums, so the same bits; on the whole GPU 112,000 cells take 168 us in
// the launch above.
__global__ void __launch_bounds__(NA_NT) k_na_passes(NaArgs a, double rsqm, int iterm, int nvb) {
  double *const r = a.z, *const p = a.pa, *const ap = a.pb;
  unsigned count = 0u;
  int turn = 0;
  na_ghosts(a);
  NaScalars q;
  // body(i, v) on the CTA's cells, with the sums of each of its nvb CTAs
  auto sweep = [&](auto ns, auto body) {
    constexpr int NS = decltype(ns)::value;
    for (int vb = blockIdx.x; vb < nvb; vb += gridDim.x) {
      double v[NS] = {};
      for (int L = 2 + vb * NA_NT + int(threadIdx.x); L <= a.la; L += nvb * NA_NT) body(L - 1, v);
      na_part(a, turn, vb, v);
      __syncthreads();  // the warps' sums have been read
    }
  };
  using One = std::integral_constant<int, 1>;
  using Two = std::integral_constant<int, 2>;
  double sum[1], sums[2];
  sweep(One{}, [&](int i, double *v) {  // :54-88
    const double c = a.ccc[i];
    const double ri = na_resid(a, i, c, a.P[i]), pi = ri * (1. / c);
    r[i] = ri;
    p[i] = pi;
    v[0] += ri * pi;
  });
  if (!na_total(a, count, turn, nvb, sum)) return na_fail(a);
  bool done = q.start(sum[0]);
  while (!done) {  // ITERM bounds the loop
    for (int vb = blockIdx.x; vb < nvb; vb += gridDim.x)  // :151-162 of the iteration before
      for (int L = 2 + vb * NA_NT + int(threadIdx.x); L <= a.la; L += nvb * NA_NT)
        p[L - 1] = (1. / a.ccc[L - 1]) * r[L - 1] + q.beta * p[L - 1];
    __syncthreads();  // every thread's p is before the release
    if (!na_meet(a, count)) return na_fail(a);
    sweep(One{}, [&](int i, double *v) {  // :107-125
      auto at = [&](int n) { return __ldcg(p + n - 1); };
      const double pi = p[i], ps = at(a.lsc[i]), pn = at(a.lnc[i]), pw = at(a.lwc[i]),
                   pe = at(a.lec[i]);
      const double api = a.ccc[i] * pi + a.ccs[i] * ps + a.ccn[i] * pn + a.ccw[i] * pw +
                         a.cce[i] * pe;
      ap[i] = api;
      v[0] += api * pi;
    });
    if (!na_total(a, count, turn, nvb, sum)) return na_fail(a);
    q.alpha = q.rpcg / sum[0];
    sweep(Two{}, [&](int i, double *v) {  // :127-149
      a.P[i] = a.P[i] + q.alpha * p[i];
      const double ri = r[i] - q.alpha * ap[i], z = (1. / a.ccc[i]) * ri;
      r[i] = ri;
      v[0] += ri * z;
      v[1] += ri * ri;
    });
    if (!na_total(a, count, turn, nvb, sums)) return na_fail(a);
    done = q.next(sums, rsqm, iterm);
  }
  q.leave(a);
}

thread_local char g_na_msg[512];

// the message goes to efdc_xm_last_error(), shared with the rest of the ABI
void na_error(const char *fmt, ...) __attribute__((format(printf, 1, 2)));
void na_error(const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_na_msg, sizeof(g_na_msg), fmt, ap);
  va_end(ap);
  xm::set_last_error_str(g_na_msg);
}

// Device address of the scratch, looked up once per device (with that
// device current) and kept for the life of the process.
std::mutex g_na_mutex;
double *g_na_ptr[64] = {nullptr};

int scratch_ptr(int dev, double **out) {
  if (dev < 0 || dev >= 64) {
    na_error("efdc_xm_congrad_noalloc: device %d out of range", dev);
    return EFDC_XM_BAD_ARGUMENT;
  }
  std::lock_guard<std::mutex> lock(g_na_mutex);
  if (!g_na_ptr[dev]) {
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_na_scratch);
    if (e != cudaSuccess || !p) {
      na_error("efdc_xm_congrad_noalloc: cudaGetSymbolAddress failed on device %d: %s", dev,
               cudaGetErrorString(e));
      return EFDC_XM_CUDA_ERROR;
    }
    g_na_ptr[dev] = static_cast<double *>(p);
  }
  *out = g_na_ptr[dev];
  return EFDC_XM_OK;
}

}  // namespace

extern "C" {

int32_t efdc_xm_congrad_noalloc(int32_t la, const int32_t *lnc, const int32_t *lsc,
                                const int32_t *lec, const int32_t *lwc, const double *ccc,
                                const double *ccs, const double *ccn, const double *ccw,
                                const double *cce, const double *fptmp, double *p, double rsqm,
                                int32_t iterm, void *stream, int32_t *iters, double *rsq) {
  if (la < 2 || iterm < 1 || !lnc || !lsc || !lec || !lwc || !ccc || !ccs || !ccn || !ccw ||
      !cce || !fptmp || !p) {
    na_error("efdc_xm_congrad_noalloc: need LA >= 2, ITERM >= 1 and non-NULL device arrays");
    return EFDC_XM_BAD_ARGUMENT;
  }
  if (la - 1 > NA_MAX_CELLS) {
    na_error("efdc_xm_congrad_noalloc: LA-1 = %d water cells exceeds the fixed scratch of %d "
             "cells; use efdc_xm_create/efdc_xm_congrad for larger systems", la - 1, NA_MAX_CELLS);
    return EFDC_XM_BAD_ARGUMENT;
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  double *base = nullptr;
  int rc = (e == cudaSuccess) ? scratch_ptr(dev, &base) : EFDC_XM_CUDA_ERROR;
  if (rc) {
    if (e != cudaSuccess)
      na_error("efdc_xm_congrad_noalloc: cudaGetDevice: %s", cudaGetErrorString(e));
    return rc;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  NaArgs a;
  a.la = la;
  a.lc = la + 1;
  a.lnc = lnc;
  a.lsc = lsc;
  a.lec = lec;
  a.lwc = lwc;
  a.ccc = ccc;
  a.ccs = ccs;
  a.ccn = ccn;
  a.ccw = ccw;
  a.cce = cce;
  a.fptmp = fptmp;
  a.P = p;
  a.polls = xm::wait_polls();
  a.z = base;
  a.pa = base + NA_LEN;
  a.pb = base + 2 * size_t(NA_LEN);
  a.part = base + 3 * size_t(NA_LEN);
  a.ctl = reinterpret_cast<NaCtl *>(base + 3 * size_t(NA_LEN) + 4 * NA_GRID);
  // one CTA per SM of a B200 at most: the exchange is the cheaper the fewer there are
  const int grid = std::max(1, std::min(NA_GRID / NA_HALVES, (la - 1 + NA_NT - 1) / NA_NT));
  // the control block keeps the previous call's contents: start from zero
  auto fail = [&](cudaError_t err, const char *what) {
    na_error("efdc_xm_congrad_noalloc: %s: %s", what, cudaGetErrorString(err));
    return EFDC_XM_CUDA_ERROR;
  };
  if ((e = cudaMemsetAsync(a.ctl, 0, sizeof(NaCtl), st)) != cudaSuccess) return fail(e, "memset");
  const int nc = (la - 1 + grid * NA_NT - 1) / (grid * NA_NT);
  static_assert((NA_MAX_CELLS + NA_GRID * NT - 1) / (NA_GRID * NT) <= 8, "cells per thread");
  const void *kernel = nc <= 1   ? reinterpret_cast<const void *>(k_na_solve<1>)
                       : nc <= 2 ? reinterpret_cast<const void *>(k_na_solve<2>)
                       : nc <= 4 ? reinterpret_cast<const void *>(k_na_solve<4>)
                                 : reinterpret_cast<const void *>(k_na_solve<8>);
  void *args[] = {&a, &rsqm, &iterm, const_cast<int *>(&grid)};  // (grid: k_na_passes alone)
  e = cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(NA_NT), args, 0, st);
  // the stream's part of the GPU holds fewer CTAs at once
  for (int g = grid / 2; e == cudaErrorCooperativeLaunchTooLarge && g > 0; g /= 2) {
    cudaGetLastError();
    e = cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(k_na_passes), dim3(g),
                                    dim3(NA_NT), args, 0, st);
  }
  if (e != cudaSuccess) return fail(e, "launch");
  NaCtl h{};
  if ((e = cudaMemcpyAsync(&h, a.ctl, sizeof(NaCtl), cudaMemcpyDeviceToHost, st)) != cudaSuccess)
    return fail(e, "copy of the control block");
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return fail(e, "synchronize");
  if (iters) *iters = h.iter;
  if (rsq) *rsq = h.rsq;
  if (h.status == EFDC_XM_DEVICE_TIMEOUT)
    na_error("efdc_xm_congrad_noalloc: a bounded device-side wait ran out; the result is not "
             "valid");
  if (h.status == EFDC_XM_CG_MAXITER)
    na_error("efdc_xm_congrad_noalloc: maximum iterations exceeded (RSQ=%g)", h.rsq);
  if (h.status == EFDC_XM_NONFINITE)
    na_error("efdc_xm_congrad_noalloc: non-finite CG scalars at iteration %d", h.iter);
  return h.status;
}

}  // extern "C"

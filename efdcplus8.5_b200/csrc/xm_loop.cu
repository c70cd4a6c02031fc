// xm_loop.cu -- loop control of a step that runs as one CUDA graph.
//
// The reference's step has three loops whose exit is data-dependent: the CG
// iterations (congrad.f90:91-169, stop at RSQ <= RSQM or ITERM), the MIXED
// form's refinement passes around its FP32 inner iterations, and the wet/dry
// re-solves (GOTO 1000 at calpuv2c.f90:597-601 and :726-749, at most
// NCORDRY = 500).  In a device-driven step each loop is a conditional WHILE
// node of the step's graph, and the small kernels below decide, on the
// device, whether its body runs again: from the member counters the reduce
// kernels keep (Glob::ndone, Glob::nidone) and a body counter with a fixed
// cap, so that every loop ends even if a counter were wrong.  The per-member
// bookkeeping the host did between sweeps (stats, failed members leaving the
// step, the sweep count and its cap) is done here too, so a step needs no
// host synchronisation until it has finished.

#include <algorithm>

#include "xm_cg.cuh"
#include "xm_kernels.h"

namespace xm {

// Start of a loop: its body counter to 0 and the condition of its first
// body: 1, or (pending) "some member has not finished its solve".
__global__ void k_loop_enter(Glob *g, int which, cudaGraphConditionalHandle h, int pending,
                             int nmember) {
  g->loop[which] = 0;
  cudaGraphSetConditional(h, (!pending || g->ndone < nmember) ? 1u : 0u);
}

// End of a loop body: count it and decide on the next.  inner: the MIXED inner
// loop, which runs while some member's inner solve is unfinished.
__global__ void k_loop_next(Glob *g, int which, cudaGraphConditionalHandle h, int cap, int inner,
                            int nmember) {
  g->tot[which] += 1;
  const int c = ++g->loop[which];
  const bool more = inner ? (g->nidone + g->ndone < nmember) : (g->ndone < nmember);
  cudaGraphSetConditional(h, (more && c < cap) ? 1u : 0u);
}

// A member's control block at the start of a step.  One that takes no part keeps
// what describes its assembled system -- the minimum diagonal and the symmetry --:
// the chunks of an efdc_xm_step_batch are steps of a few members each, and the
// scaled system of every member may be asked for after the last.
__device__ __forceinline__ void member_enter(Ctl &c, bool active) {
  Ctl k{};
  if (!active) {
    k.ccmnm_int = c.ccmnm_int;
    k.ccmnm_bc = c.ccmnm_bc;
    k.asym = c.asym;
  }
  k.stepping = active ? 1 : 0;
  member_sweep_reset(k, active);
  c = k;
}
// The control blocks of a step driven by the host.
__global__ void k_ctl_enter(Ctl *ctl, const int *act, int nmember) {
  for (int m = threadIdx.x; m < nmember; m += blockDim.x) member_enter(ctl[m], act[m] != 0);
}

// Start of a step, and of its first sweep: the members' scalars, activity and
// inner preconditioner from the host's mirrors, their control blocks, the
// step's counters.  One kernel of the graph in place of four small copies
// before it.
__global__ void k_step_enter(StepIn in, StepScalars *sc, int *act, int *mpoly, Ctl *ctl, Glob *g,
                             int nmember) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  const unsigned *src = reinterpret_cast<const unsigned *>(in.sc);
  unsigned *dst = reinterpret_cast<unsigned *>(sc);
  if (in.sc != sc)
    for (int i = t; i < nmember * int(sizeof(StepScalars) / 4); i += nt) dst[i] = src[i];
  for (int m = t; m < nmember; m += nt) {
    const int a = in.act[m];
    act[m] = a;
    mpoly[m] = in.mpoly[m];
    member_enter(ctl[m], a != 0);
  }
  if (blockIdx.x == 0) {
    __shared__ int out;
    if (threadIdx.x == 0) out = 0;
    __syncthreads();
    for (int m = threadIdx.x; m < nmember; m += blockDim.x)
      if (!in.act[m]) atomicAdd(&out, 1);
    __syncthreads();
    if (threadIdx.x == 0) {
      g->ndone = out;
      g->nidone = 0;
      g->arrive = 0u;
    }
    if (threadIdx.x < NLOOP) g->tot[threadIdx.x] = 0;
  }
}

// MIXED, after an inner loop: the inner iterations of the pass (those of the
// first pass choose the next step's inner preconditioner).
__global__ void k_inner_done(Ctl *ctl, const int *act, int nmember) {
  for (int m = threadIdx.x; m < nmember; m += blockDim.x) {
    Ctl &k = ctl[m];
    if (!act[m] || k.inner_iter <= 0) continue;
    k.last_inner = k.inner_iter;
    if (k.outer == 1) k.inner_first = k.inner_iter;
  }
}

__global__ void k_after_solve(Ctl *ctl, int *act, int nmember, int mixed) {
  for (int m = threadIdx.x; m < nmember; m += blockDim.x)
    if (act[m]) member_after_solve(ctl[m], act[m], ctl[m].asym, mixed != 0);
}

// End of a sweep (calpuv2c.f90:597-601, 726-749): a member whose faces
// changed sweeps again unless it has reached its cap (then its status is
// WETDRY_MAXSWEEP); the sweep loop runs again while some member does, and
// the members are reset for it.  After a wait that ran out (Glob::err) the step
// has failed and no solve's arrivals match any more: no further sweep.
__global__ void k_sweep_next(DevStatic S, Ctl *ctl, int *act, Glob *g,
                             cudaGraphConditionalHandle h, int cap, int nmember) {
  __shared__ int any;
  if (threadIdx.x == 0) any = 0;
  __syncthreads();
  for (int m = threadIdx.x; m < nmember; m += blockDim.x) {
    Ctl &k = ctl[m];
    int next = 0;
    if (act[m]) {
      const StepScalars &c = S.sc[m];
      if (c.isdry > 0 && c.isdry != 98 && k.icordry) {
        if (++k.sweep < c.max_sweeps)
          next = 1;
        else
          k.mstatus = EFDC_XM_WETDRY_MAXSWEEP;
      }
      act[m] = next;
      if (next) atomicAdd(&any, 1);
    }
  }
  __syncthreads();
  if (any)
    for (int m = threadIdx.x; m < nmember; m += blockDim.x) member_sweep_reset(ctl[m], act[m] != 0);
  if (threadIdx.x == 0) {
    g->ndone = nmember - any;
    g->nidone = 0;
    g->tot[LOOP_SWEEP] += 1;
    const int c = ++g->loop[LOOP_SWEEP];
    cudaGraphSetConditional(h, (any && c < cap && !g->err) ? 1u : 0u);
  }
}

void launch_loop_enter(cudaStream_t st, Glob *g, int which, cudaGraphConditionalHandle h,
                       int pending, int nmember) {
  k_loop_enter<<<1, 1, 0, st>>>(g, which, h, pending, nmember);
  count_launches(1);
}
void launch_loop_next(cudaStream_t st, Glob *g, int which, cudaGraphConditionalHandle h, int cap,
                      int inner, int nmember) {
  k_loop_next<<<1, 1, 0, st>>>(g, which, h, cap, inner, nmember);
  count_launches(1);
}
void launch_step_enter(cudaStream_t st, const StepIn &in, StepScalars *sc, int *act, int *mpoly,
                       Ctl *ctl, Glob *g, int nmember) {
  const int words = nmember * int(sizeof(StepScalars) / 4);
  k_step_enter<<<std::min(64, (words + 255) / 256), 256, 0, st>>>(in, sc, act, mpoly, ctl, g,
                                                                 nmember);
  count_launches(1);
}
void launch_ctl_enter(cudaStream_t st, Ctl *ctl, const int *act, int nmember) {
  k_ctl_enter<<<1, 256, 0, st>>>(ctl, act, nmember);
  count_launches(1);
}
void launch_inner_done(cudaStream_t st, Ctl *ctl, const int *act, int nmember) {
  k_inner_done<<<1, 256, 0, st>>>(ctl, act, nmember);
  count_launches(1);
}
void launch_after_solve(cudaStream_t st, Ctl *ctl, int *act, int nmember, int mixed) {
  k_after_solve<<<1, 256, 0, st>>>(ctl, act, nmember, mixed);
  count_launches(1);
}
void launch_sweep_next(cudaStream_t st, const DevStatic &S, Ctl *ctl, int *act, Glob *g,
                       cudaGraphConditionalHandle h, int cap, int nmember) {
  k_sweep_next<<<1, 256, 0, st>>>(S, ctl, act, g, h, cap, nmember);
  count_launches(1);
}
}  // namespace xm

// xm_resident.cuh -- solves that stay on the chip: what the one-launch CG
// kernels (xm_resident.cu: k_cg_res, xm_resident32.cu: k_mx_res) share.
//
// A member's solve runs in a group of CTAs that are resident together, each
// with W quads side by side (256*W threads) and Q such rows of quads one after
// another, a thread holding its row vectors of each quad in registers from the
// first residual to the stop test.  What leaves a CTA is the border of its
// tiles (the rows and columns a neighbour tile reads) and one partial sum per
// quad, through L2 (FP64 clusters: through shared memory).  The multi-kernel CG pays
// two kernel boundaries per iteration (launch, ramp, tail and a folded reduction: 7 us
// each on a 60,000-cell basin whose row work is below 1 us); here a boundary is one
// exchange between the CTAs of the member, which is also their barrier:
//  * a group of up to 16 CTAs is a thread-block cluster: each CTA stores its
//    quads' partial sums into the shared memory of every CTA, and the cluster
//    barrier orders them and the borders (measured: 1,250 clocks with 2 CTAs,
//    1,380 with 16);
//  * a larger group shares a counter per member in global memory: each CTA
//    stores its partial sums, adds to the counter with release semantics, and
//    waits until the counter has the group's arrivals (a bounded wait), then
//    reads the partial sums of all the member's quads (measured: 3,200 clocks
//    with 64 CTAs, 4,100 with 256; polling the partial sums themselves, without
//    a counter, took 5,200 and 9,700: the polls hold up the stores).  All its
//    CTAs must be resident at once: a cooperative launch.
// The halo of the next row work is loaded as soon as the barrier is passed,
// under the member sums and the divisions.
//
// Same rows, same per-quad partials, same member sums and same epilogues as
// the multi-kernel CG: the iterates are equal bit for bit.
#pragma once

#include <map>
#include <mutex>
#include <tuple>
#include <utility>

#include "xm_cg.cuh"
#include "xm_kernels.h"

namespace xm {

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release(unsigned *p, unsigned v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// a double into the shared memory of CTA `rank` of the cluster, at this CTA's p
__device__ __forceinline__ void st_cluster(double *p, int rank, double v) {
  unsigned a = unsigned(__cvta_generic_to_shared(p)), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(r), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Loads of what another CTA of the group stored during this launch: from L2.
__device__ __forceinline__ V4<double> ldx4(const double *p) {
  const double2 a = __ldcg(reinterpret_cast<const double2 *>(p));
  const double2 b = __ldcg(reinterpret_cast<const double2 *>(p) + 1);
  return {a.x, a.y, b.x, b.y};
}
__device__ __forceinline__ V4<float> ldx4(const float *p) {
  const float4 v = __ldcg(reinterpret_cast<const float4 *>(p));
  return {v.x, v.y, v.z, v.w};
}

// A row vector of one quad of the CTA: its slots and the slots it reads of
// other tiles (those of its tile come from shared memory or the row's lanes).
struct ResRow {
  int d0;  // first slot of the thread's 4 cells
  int hv;  // the same columns in the N (S) neighbour tile, for a row at its N (S) edge
  int hx;  // the W (E) neighbour's slot, for the first (last) row vector of a row
  bool valid;  // the quad exists and the member has the tile
};
__device__ __forceinline__ int res_q() { return threadIdx.x % TPT; }
__device__ __forceinline__ bool res_north() { return res_q() / ROWT == TY - 1; }
__device__ __forceinline__ bool res_south() { return res_q() / ROWT == 0; }
__device__ __forceinline__ bool res_west() { return (res_q() & (ROWT - 1)) == 0; }
__device__ __forceinline__ bool res_east() { return (res_q() & (ROWT - 1)) == ROWT - 1; }

__device__ __forceinline__ RowGeo res_geo(const DevStatic &S, int qd, bool have, ResRow &r) {
  const int sub = threadIdx.x % NT / TPT;
  const int4 cur = have ? S.quads[qd] : int4{0, 0, 0, 0};
  r.valid = have && sub < cur.z;
  const int ti = r.valid ? cur.y + sub : 0;
  const RowGeo g = row_geo_nb(__ldg(&S.tnbr[ti]), ti, res_q());
  r.d0 = g.d0;
  r.hv = res_north() ? g.dn : g.ds;
  r.hx = res_west() ? g.dwe : g.dee;
  return g;
}

// Stores of a row vector's border: whole where the row is the first or last
// of its tile, else the first or last column of the tile.
template <class T>
__device__ __forceinline__ void st_border(T *a, const ResRow &r, const V4<T> &v) {
  if (!r.valid) return;
  if (res_north() || res_south())
    st4(a + r.d0, v);
  else if (res_west())
    a[r.d0] = v.x;
  else if (res_east())
    a[r.d0 + CPT - 1] = v.w;
}

// A CTA of a group: member, quads [q0, q0 + nq) of the member's [qm0, qm0 + nqm).
// Quad q0 + i*W + w is row i of the threads [256w, 256w + 256).
struct ResCta {
  int m, q0, nq, qm0, nqm;
};

// A thread's row vectors of the CTA's quads in shared memory ([row][quad][tile]
// [row][column]), for the rows above and below: TX elements from them.  Of a row
// of 64-bit columns the first halves of its threads' vectors come first, then the
// second: eight threads read 128 bytes in one go.
template <int W>
__device__ __forceinline__ float *res_stage(float *stage, int i) {
  return stage + i * (W * TILES_PER_CTA * TILE) + int(threadIdx.x) * CPT;
}
template <int W>
__device__ __forceinline__ double *res_stage(double *stage, int i) {
  return stage + i * (W * TILES_PER_CTA * TILE) + int(threadIdx.x) / ROWT * TX +
         int(threadIdx.x) % ROWT * 2;
}
__device__ __forceinline__ V4<float> ld_stage(const float *p) { return ld4(p); }
__device__ __forceinline__ V4<double> ld_stage(const double *p) {
  const double2 a = *reinterpret_cast<const double2 *>(p);
  const double2 b = *reinterpret_cast<const double2 *>(p + TX / 2);
  return {a.x, a.y, b.x, b.y};
}
__device__ __forceinline__ void st_stage(float *p, const V4<float> &v) { st4(p, v); }
__device__ __forceinline__ void st_stage(double *p, const V4<double> &v) {
  *reinterpret_cast<double2 *>(p) = make_double2(v.x, v.y);
  *reinterpret_cast<double2 *>(p + TX / 2) = make_double2(v.z, v.w);
}

// Cluster groups hold what their CTAs read of one another's tiles in shared memory:
// the borders of the CTA's tiles in two vectors (z and p_old), a tile as [S row][N row]
// [W column][E column], and past the last tile one of zeros for the ghost tile (where
// every vector is zero).  In global memory they cost the cluster barrier the stores'
// round trip to L2 and the row work behind it another: FP64 steps of 44x28 cells 0.088
// -> 0.079 ms, 60x60 0.091 -> 0.083, 180x150 0.115 -> 0.105, 260x250 (four quads a CTA,
// bound by its row work) 0.131 -> 0.130.
constexpr int RES_EDGE = 2 * TX + 2 * TY;
template <int W, int Q>
__host__ __device__ constexpr int res_edges() {  // elements of one vector
  return (W * Q * TILES_PER_CTA + 1) * RES_EDGE;
}
__device__ __forceinline__ void ld_peer(unsigned a, double &x, double &y) {
  asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(x), "=d"(y) : "r"(a) : "memory");
}
__device__ __forceinline__ V4<double> ld_peer4(unsigned a) {  // a row: see res_stage
  V4<double> v;
  ld_peer(a, v.x, v.y);
  ld_peer(a + TX / 2 * sizeof(double), v.z, v.w);
  return v;
}
__device__ __forceinline__ double ld_peer1(unsigned a) {
  double x;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(x) : "r"(a) : "memory");
  return x;
}
// The row's hv and hx: no slots, the addresses of those cells in the CTAs' edges.
template <int W, int Q>
__device__ __forceinline__ void res_peers(const double *edge, const ResCta &c, int t0,
                                          ResRow &r) {
  const int q = res_q(), cx = q % ROWT, ty = q / ROWT;
  auto at = [&](int slot, int e) {
    const int lt = slot / TILE - t0;  // before the member's tiles: a ghost tile
    const int j = lt < 0 ? W * Q : lt / TILES_PER_CTA % (W * Q);
    const int rank = lt < 0 ? (c.q0 - c.qm0) / (W * Q) : lt / TILES_PER_CTA / (W * Q);
    const double *p = edge + (j * TILES_PER_CTA + (lt < 0 ? 0 : lt % TILES_PER_CTA)) * RES_EDGE + e;
    unsigned a = unsigned(__cvta_generic_to_shared(p)), peer;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(a), "r"(rank));
    return int(peer);
  };
  r.hv = at(r.hv, (res_north() ? 0 : TX) + 2 * cx);
  r.hx = at(r.hx, 2 * TX + (res_west() ? TY : 0) + ty);
}
// The thread's part of its tile's edge (j: the quad of the CTA).
__device__ __forceinline__ void st_edge(double *edge, int j, const V4<double> &v) {
  const int q = res_q(), cx = q % ROWT, ty = q / ROWT;
  double *e = edge + (j * TILES_PER_CTA + threadIdx.x % NT / TPT) * RES_EDGE;
  if (res_north() || res_south()) {
    double2 *p = reinterpret_cast<double2 *>(e + (res_north() ? TX : 0) + 2 * cx);
    p[0] = make_double2(v.x, v.y);
    p[TX / 4] = make_double2(v.z, v.w);
  }
  if (res_west())
    e[2 * TX + ty] = v.x;
  else if (res_east())
    e[2 * TX + TY + ty] = v.w;
}

constexpr int RES_CLUSTER_QUADS = 128;  // of a member in a cluster, at most
template <int W, int Q, bool CLUSTER>
struct ResShared {
  double wsum[2][W * Q][2][NWARP];  // the warps' sums of each quad, by turns
  // the member's partial sums, by turns (cluster); the trees' parts (grid)
  double inbox[CLUSTER ? 2 : 1][2][CLUSTER ? RES_CLUSTER_QUADS : NWARP];
};

// What an exchange carries over: the barrier's turn, and for a grid group the
// member's arrivals so far.
struct ResBarrier {
  unsigned count;
  int turn;
};

// One exchange of NS sums: v[i][s], the thread's part of sum s on its quad of
// row i.  out[s]: the member's sums, in every thread.  halo() runs as soon as
// the other CTAs' borders may be read.  False (in every thread) when a wait
// ran out.
template <int W, int Q, bool CLUSTER, int NS, class Halo>
__device__ __forceinline__ bool res_exchange(const ResPlan &R, const DevStatic &S, const ResCta &c,
                                             ResShared<W, Q, CLUSTER> &sh, ResBarrier &bar,
                                             const double (&v)[Q][NS], double (&out)[NS],
                                             Halo halo) {
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int turn = bar.turn;
  bar.turn ^= 1;
  auto &ws = sh.wsum[turn];
#pragma unroll
  for (int i = 0; i < Q; ++i)
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const double x = warp_sum(v[i][s]);
      if (lane == 0) ws[i * W + warp / NWARP][s][warp % NWARP] = x;
    }
  __syncthreads();
  auto quad_sum = [&](int j, int s) {  // in warp order
    double b = 0.0;
#pragma unroll
    for (int w = 0; w < NWARP; ++w) b += ws[j][s][w];
    return b;
  };
  int dead = 0;
  if constexpr (CLUSTER) {
    const int ncta = gridDim.x / S.nmember;  // of the cluster
    // thread (j, r): the partial sums of quad j to CTA r
    for (int u = t; u < c.nq * ncta; u += W * NT) {
      const int j = u / ncta, r = u - j * ncta;
#pragma unroll
      for (int s = 0; s < NS; ++s)
        st_cluster(&sh.inbox[turn][s][c.q0 - c.qm0 + j], r, quad_sum(j, s));
    }
    cluster_barrier();
    halo();
    // reduce_partials' sum, by every warp: lane l of its warp w holds partial
    // 32w + l, then the trees over the lanes and over the warps
    constexpr int NB = (16 * W * Q + 31) / 32;  // warps with a partial, at most
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      double l[NWARP];
#pragma unroll
      for (int w = 0; w < NWARP; ++w) {
        l[w] = 0.0;
        if (w < NB) {
          const int i = 32 * w + lane;
          l[w] = warp_sum(0.0 + (i < c.nqm ? sh.inbox[turn][s][i] : 0.0)) + 0.0;
        }
      }
      const double x = ((l[0] + l[4]) + (l[2] + l[6])) + ((l[1] + l[5]) + (l[3] + l[7]));
      out[s] = __shfl_sync(0xffffffffu, x, 0);
    }
  } else {
    double2 *part = R.part + size_t(turn) * S.nquad;
    bar.count += unsigned((c.nqm + W * Q - 1) / (W * Q));
    if (warp == 0) {
      if (t < c.nq)
        part[c.q0 + t] = make_double2(quad_sum(t, 0), NS > 1 ? quad_sum(t, NS - 1) : 0.0);
      __syncwarp();
      if (t == 0) {
        unsigned *n = R.count + size_t(c.m) * RES_COUNT_STRIDE;
        red_release(n, 1u);
        for (int k = 0; int(ld_acquire(n) - bar.count) < 0; ++k)
          if (k >= WAIT_POLLS) {
            dead = 1;
            break;
          }
      }
    }
    if (__syncthreads_or(dead)) return false;
    // reduce_partials: thread i adds partials i, i + 256, ... (the first before the
    // halo's loads, which may queue behind it)
    const bool red = t < NT;
    double2 first = make_double2(0.0, 0.0);
    if (red && t < c.nqm) first = __ldcg(part + c.qm0 + t);
    halo();
    if (red) {
      double z[NS];
      z[0] = 0.0 + first.x;
      if constexpr (NS > 1) z[1] = 0.0 + first.y;
      for (int i = t + NT; i < c.nqm; i += NT) {
        const double2 a = __ldcg(part + c.qm0 + i);
        z[0] += a.x;
        if constexpr (NS > 1) z[1] += a.y;
      }
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const double x = warp_sum(z[s]);
        if (lane == 0) sh.inbox[0][s][warp] = x;
      }
    }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < NS; ++s) {  // block_sum's last stage (its further lanes add zeros)
      static_assert(NWARP == 8, "the tree below");
      double l[NWARP];
#pragma unroll
      for (int w = 0; w < NWARP; ++w) l[w] = sh.inbox[0][s][w] + 0.0;
      out[s] = ((l[0] + l[4]) + (l[2] + l[6])) + ((l[1] + l[5]) + (l[3] + l[7]));
    }
  }
  return true;
}

// The open-boundary cells of a row vector report an unsymmetric operator
// (k_obc_asym's test, for contexts whose kernels assume a symmetric one).
__device__ __forceinline__ void res_check_faces(const DevStatic &S, const SysView &V, Ctl &k,
                                                const ResRow &r, const uchar4 &kd,
                                                const ResEnds &ends) {
  if (!ends.check || !r.valid) return;
  const uint8_t kinds[CPT] = {kd.x, kd.y, kd.z, kd.w};
#pragma unroll
  for (int c = 0; c < CPT; ++c)
    if (kinds[c] == OPENBC && unsymmetric_faces(S, V, r.d0 + c)) atomicOr(&k.asym, 2);
}

// A wait ran out: the call fails with a timeout status.  The CTA has not stored its part
// of the solution, and the others may have come through the same exchange: the status
// of the one that ends the solve (res_status) does not replace this one, the largest.
// (A limit of the waits as a kernel argument, or a compare-and-swap here, cost the
// registers of the MIXED 2x1 form: 512x512 cells 0.163 -> 0.166 ms per step.)
__device__ __forceinline__ void res_fail(Ctl &k, int *err) {
  if (threadIdx.x == 0) {
    atomicMax(&k.status, EFDC_XM_DEVICE_TIMEOUT);
    atomicExch(err, 1);
  }
}
__device__ __forceinline__ void res_status(Ctl &k, int status) {  // OK at the entry
  static_assert(EFDC_XM_DEVICE_TIMEOUT > EFDC_XM_NONFINITE &&
                EFDC_XM_DEVICE_TIMEOUT > EFDC_XM_CG_MAXITER, "the largest of a solve");
  atomicMax(&k.status, status);
}

// Row vectors of NC coefficients of the thread's quads: in registers (REG), or
// in shared memory, each thread its own in conflict-free 16-byte words.
template <class T, int W, int Q, int NC, bool REG>
struct ResCoef {
  V4<T> reg[REG ? Q * NC : 1];
  T *sm;
  static constexpr int WORD = 16 / sizeof(T);  // elements of a word
  static constexpr size_t bytes = REG ? 0 : size_t(Q) * NC * W * NT * CPT * sizeof(T);
  __device__ __forceinline__ T *at(int i, int k) const {
    return sm + size_t(i * NC + k) * W * NT * CPT + threadIdx.x * WORD;
  }
  __device__ __forceinline__ void put(int i, int k, const V4<T> &v) {
    if constexpr (REG) {
      reg[i * NC + k] = v;
    } else if constexpr (sizeof(T) == 4) {
      *reinterpret_cast<float4 *>(at(i, k)) = make_float4(v.x, v.y, v.z, v.w);
    } else {
      double2 *p = reinterpret_cast<double2 *>(at(i, k));
      p[0] = make_double2(v.x, v.y);
      p[W * NT] = make_double2(v.z, v.w);
    }
  }
  __device__ __forceinline__ V4<T> get(int i, int k) const {
    if constexpr (REG) {
      return reg[i * NC + k];
    } else if constexpr (sizeof(T) == 4) {
      const float4 v = *reinterpret_cast<const float4 *>(at(i, k));
      return {v.x, v.y, v.z, v.w};
    } else {
      const double2 *p = reinterpret_cast<const double2 *>(at(i, k));
      const double2 a = p[0], b = p[W * NT];
      return {a.x, a.y, b.x, b.y};
    }
  }
};

// The CTA's group and quads: from the launch's table, or, in a cluster, the
// next W*Q quads of the member of the cluster (possibly none).
template <int W, int Q, bool CLUSTER>
__device__ __forceinline__ ResCta res_cta(const ResPlan &R, const DevStatic &S) {
  ResCta c;
  if constexpr (CLUSTER) {
    const int ncta = gridDim.x / S.nmember;
    c.m = blockIdx.x / ncta;
    c.qm0 = S.qstart[c.m];
    c.nqm = S.qstart[c.m + 1] - c.qm0;
    const int first = min(c.nqm, int(blockIdx.x % ncta) * W * Q);
    c.q0 = c.qm0 + first;
    c.nq = min(W * Q, c.nqm - first);
  } else {
    const int4 e = R.cta[blockIdx.x];
    c.m = e.x;
    c.q0 = e.y;
    c.nq = e.z;
    c.qm0 = S.qstart[c.m];
    c.nqm = S.qstart[c.m + 1] - c.qm0;
  }
  return c;
}

// Sets a kernel's dynamic shared memory (and, in clusters, allows 16 CTAs) on
// the current device and returns how many of its CTAs are resident at once
// there, or for a cluster size whether a cluster is (0: it cannot run).
template <class K>
int res_cap(K kernel, int threads, size_t smem, int nsm, int cluster) {
  bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(smem)) == cudaSuccess;
  int b = 0;
  if (cluster > 0) {
    ok = ok && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
                   cudaSuccess;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = cluster;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(cluster);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    // (a millisecond; the answer is the device's: asked once per kernel and size)
    static std::mutex mu;
    static std::map<std::tuple<int, const void *, int>, int> known;
    int dev = 0;
    ok = ok && cudaGetDevice(&dev) == cudaSuccess;
    std::lock_guard<std::mutex> lock(mu);
    const auto key = std::make_tuple(dev, reinterpret_cast<const void *>(kernel), cluster);
    const auto it = known.find(key);
    if (it != known.end()) return ok ? it->second : 0;
    ok = ok && cudaOccupancyMaxActiveClusters(&b, kernel, &cfg) == cudaSuccess;
    if (ok) known[key] = b;
  } else {
    ok = ok && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, threads, smem) ==
                   cudaSuccess;
    b *= nsm;
  }
  if (!ok) {
    cudaGetLastError();
    return 0;
  }
  return b;
}

// A launch in clusters, or with all CTAs resident at once (they wait for one
// another).
template <class... P, class... A>
void launch_resident(void (*kernel)(P...), int ncta, int threads, size_t smem, int cluster,
                     cudaStream_t st, A &&...args) {
  cudaLaunchAttribute at{};
  if (cluster > 0) {
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = cluster;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
  } else {
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(ncta);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

// Calls go with a form as compile-time constants; false for one that is not
// compiled (F64: for FP64).
template <bool F64, class F>
bool res_form(const ResForm &f, F &&go) {
  auto call = [&](auto w, auto q) {
    if (f.cluster > 0)
      go(w, q, std::true_type{});
    else
      go(w, q, std::false_type{});
    return true;
  };
  using I1 = std::integral_constant<int, 1>;
  using I2 = std::integral_constant<int, 2>;
  if (f.w == 1 && f.q == 1) return call(I1{}, I1{});
  if (f.w == 2 && f.q == 2) return call(I2{}, I2{});
  if constexpr (F64) {
    if (f.w == 1 && f.q == 2) return call(I1{}, I2{});
    if (f.w == 2 && f.q == 4 && f.cluster == 0)
      return go(I2{}, std::integral_constant<int, 4>{}, std::false_type{}), true;
  } else {
    if (f.w == 2 && f.q == 1) return call(I2{}, I1{});
  }
  return false;
}

}  // namespace xm

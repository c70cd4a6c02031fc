// xm_resident.cu -- the FP64 CONGRAD of a member in one launch, its vectors in
// registers (see xm_resident.cuh).  Compiled without FMA contraction, like the
// multi-kernel CG (xm_step.cu): each statement rounds as in congrad.f90.

#include "xm_resident.cuh"

namespace xm {

// What a form keeps where.  One quad side by side: the coefficients in registers.
// Two by two: in shared memory.  Four (the lean form): P and PCG live in shared memory too --
// PCG where the rows above and below read it anyway --, CCCI as well, and the
// other coefficients are read and scaled anew (24 of the 112 B per cell-iteration
// of the multi-kernel CG, from L2).
__host__ __device__ constexpr bool res_lean(int Q) { return Q == 4; }
constexpr int RES_NC = 5;  // CCC, CCS, CCW, CCN and CCCI (symmetric) or CCE (MA)
template <int W, int Q>
using Coef64 = ResCoef<double, W, Q, res_lean(Q) ? 2 : RES_NC, Q == 1 || W == 1>;  // lean: CCCI, P
template <int W, int Q, bool CLUSTER>
constexpr size_t res_smem64() {
  return size_t(W) * Q * TILES_PER_CTA * TILE * sizeof(double) + Coef64<W, Q>::bytes +
         (CLUSTER ? 2 * res_edges<W, Q>() * sizeof(double) : 0);
}

// congrad.f90:54-187 for one member per group of CTAs.  What bounds it is the
// exchange (see xm_resident.cuh) and the latency of the row work around it.
// Measured against the multi-kernel CG with folded reductions (one CTA per
// member before, for members of up to 4,000 slots), ms per step, device-resident:
// 60x60 cells 0.33 -> 0.083, 260x250 0.36 -> 0.13, 500x500 0.45 -> 0.177, 700x700
// 0.57 -> 0.33, 256 lakes of 1,100 cells in one batch 0.50 -> 0.38; lean: 900x860
// 0.65 -> 0.49, 1,000x1,000 0.80 -> 0.55 (an iteration 31 -> 20 us, of which the row
// work is 13, the exchanges' waits for the slowest CTA 3 and the exchanges 4).
// Registers: one quad side by side keeps the coefficients there too (255 a thread with
// two rows), two by two (128 a thread) in shared memory; the lean form reads them.  These
// two spill, 312 to 400 bytes stored and 424 to 560 loaded a thread (the forms with one
// quad side by side at most 64); one quad side by side and four or eight rows, which
// would have 255 registers, were not tried.
template <bool MA, int W, int Q, bool CLUSTER>
__global__ void __launch_bounds__(NT *W, W == 1 && Q == 1 && CLUSTER ? 2 : 1)
    k_cg_res(DevStatic S, SysView V, DevSystem Y, double *P, Ctl *ctl, Glob *glob, ResPlan R,
             ResEnds ends) {
  extern __shared__ __align__(16) double dyn[];
  __shared__ ResShared<W, Q, CLUSTER> sh;
  const ResCta me = res_cta<W, Q, CLUSTER>(R, S);
  const int m = me.m;
  if (ctl[m].done) return;  // the same for the member's CTAs: it is set after their exchanges
  if constexpr (CLUSTER) cluster_barrier();  // every CTA has started: its shared memory is there
  const double rsqm = S.sc[m].rsqm;
  const int iterm = S.sc[m].iterm;
  const bool asym = unsym<MA>(ctl[m]);
  ResBarrier bar{CLUSTER ? 0u : R.count[size_t(m) * RES_COUNT_STRIDE + 1], 0};
  double *stage = dyn;
  Coef64<W, Q> C;
  C.sm = dyn + W * Q * TILES_PER_CTA * TILE;
  const bool north = res_north(), south = res_south(), west = res_west(), east = res_east();
  const int w0 = W > 1 ? int(threadIdx.x) / NT : 0;  // quad q0 + i*W + w0 is the thread's row i
  // cluster: the edges of z and of p_old
  constexpr int NE = res_edges<W, Q>();
  double *edge = C.sm + Coef64<W, Q>::bytes / sizeof(double);
  if constexpr (CLUSTER)
    for (int t = threadIdx.x; t < 2 * RES_EDGE; t += W * NT)  // the zeros of the ghost tile
      edge[(t < RES_EDGE ? 1 : 2) * NE - RES_EDGE + t % RES_EDGE] = 0.0;
  auto none = [] {};

  constexpr bool LEAN = res_lean(Q);
  ResRow row[Q];
  V4<double> xr[LEAN ? 1 : Q] = {}, pr[LEAN ? 1 : Q] = {};  // (the registers of the other forms)
  V4<double> r[Q], ap[Q];
  double kwe[LEAN ? 1 : Q];  // symmetric: CCW of the cell east of the row vector
  auto get_x = [&](int i) {
    if constexpr (LEAN)
      return C.get(i, 1);
    else
      return xr[i];
  };
  auto put_x = [&](int i, const V4<double> &v) {
    if constexpr (LEAN)
      C.put(i, 1, v);
    else
      xr[i] = v;
  };
  auto get_p = [&](int i) {
    if constexpr (LEAN)
      return ld_stage(res_stage<W>(stage, i));
    else
      return pr[i];
  };
  auto put_p = [&](int i, const V4<double> &v) {
    st_stage(res_stage<W>(stage, i), v);
    if constexpr (!LEAN) pr[i] = v;
  };
  Ctl k;  // of it: rpcg, papcg, alpha, beta, rsq, iter, status, parity
  k.alpha = 0.0;
  bool fin;
  double v0[Q][1];
  // the scaling of calpuv2c.f90:371-399, as the system is read (k_scale's products)
  const double sc = V.unscaled ? 1. / fmin(ctl[m].ccmnm_int, ctl[m].ccmnm_bc) : 1.0;
  auto ld = [&](const double *a, int d) {
    const V4<double> v = ld4(a + d);
    return V4<double>{v.x * sc, v.y * sc, v.z * sc, v.w * sc};
  };
  unsigned land = 0;  // lean: a bit per cell of the rows
  {  // :54-88
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const int j = i * W + w0;
      const RowGeo g = res_geo(S, me.q0 + j, j < me.nq, row[i]);
      const V4<double> X0 = ld4(P + g.d0), xn = ld4(P + g.dn), xs = ld4(P + g.ds);
      const V4<double> b = ld(V.fp, g.d0), ks = ld(V.cs, g.d0), kw = ld(V.cw, g.d0);
      const V4<double> kn = asym ? ld(V.cn, g.d0) : ld(V.cs, g.dn);
      V4<double> c = ld(V.cc, g.d0);
      const uchar4 kd = *reinterpret_cast<const uchar4 *>(S.kind + g.d0);
      double xw = from_west(X0), xe = from_east(X0);
      double kwee = from_east(kw);
      if (west) xw = P[g.dwe];
      if (east) {
        xe = P[g.dee];
        kwee = V.cw[g.dee] * sc;
      }
      const V4<double> ke = asym ? ld(V.ce, g.d0) : V4<double>{kw.y, kw.z, kw.w, kwee};
      // land slots are inert: CCC = 1, r = 0
      if (kd.x == LAND) c.x = 1.;
      if (kd.y == LAND) c.y = 1.;
      if (kd.z == LAND) c.z = 1.;
      if (kd.w == LAND) c.w = 1.;
      V4<double> d;
      d.x = b.x - c.x * X0.x - kn.x * xn.x - ks.x * xs.x - kw.x * xw - ke.x * X0.y;
      d.y = b.y - c.y * X0.y - kn.y * xn.y - ks.y * xs.y - kw.y * X0.x - ke.y * X0.z;
      d.z = b.z - c.z * X0.z - kn.z * xn.z - ks.z * xs.z - kw.z * X0.y - ke.z * X0.w;
      d.w = b.w - c.w * X0.w - kn.w * xn.w - ks.w * xs.w - kw.w * X0.z - ke.w * xe;
      if (kd.x == LAND) d.x = 0.;
      if (kd.y == LAND) d.y = 0.;
      if (kd.z == LAND) d.z = 0.;
      if (kd.w == LAND) d.w = 0.;
      res_check_faces(S, V, ctl[m], row[i], kd, ends);
      r[i] = d;
      const V4<double> ci = {rcpT(c.x), rcpT(c.y), rcpT(c.z), rcpT(c.w)};
      const V4<double> z = {d.x * ci.x, d.y * ci.y, d.z * ci.z, d.w * ci.w};
      if constexpr (LEAN) {
        land |= unsigned((kd.x == LAND) | (kd.y == LAND) << 1 | (kd.z == LAND) << 2 |
                         (kd.w == LAND) << 3)
                << 4 * i;
        C.put(i, 0, ci);
      } else {
        kwe[i] = kwee;
        C.put(i, 0, c);
        C.put(i, 1, ks);
        C.put(i, 2, kw);
        C.put(i, 3, kn);
        C.put(i, 4, MA ? ke : ci);
      }
      put_x(i, X0);
      put_p(i, z);
      if constexpr (CLUSTER) {
        res_peers<W, Q>(edge, me, S.quads[me.qm0].y, row[i]);
        st_edge(edge, j, z);
        st_edge(edge + NE, j, z);
      } else {
        st_border(Y.z, row[i], z);
        st_border(Y.pa, row[i], z);
      }
      v0[i][0] = row[i].valid ? d.x * z.x + d.y * z.y + d.z * z.z + d.w * z.w : 0.0;
    }
  }
  auto cci = [&](int i) {  // CCCI
    if constexpr (LEAN) {
      return C.get(i, 0);
    } else if constexpr (MA) {
      const V4<double> c = C.get(i, 0);
      return V4<double>{rcpT(c.x), rcpT(c.y), rcpT(c.z), rcpT(c.w)};
    } else {
      return C.get(i, 4);
    }
  };
  // what the neighbour tiles hold of z and p_old, for the next A*p: of every row,
  // loaded under the exchange, or (lean) of the first, each next row's under the
  // one before
  constexpr int NH = LEAN ? 1 : Q;
  V4<double> hz[NH], ho[NH];
  double ez[NH], eo[NH];
  auto halo_row = [&](const double *pold, int i, int h) {
    if constexpr (CLUSTER) {
      constexpr unsigned P_OLD = NE * sizeof(double);
      if (north || south) {
        hz[h] = ld_peer4(row[i].hv);
        ho[h] = ld_peer4(row[i].hv + P_OLD);
      }
      if (west || east) {
        ez[h] = ld_peer1(row[i].hx);
        eo[h] = ld_peer1(row[i].hx + P_OLD);
      }
    } else {
      if (north || south) {
        hz[h] = ldx4(Y.z + row[i].hv);
        ho[h] = ldx4(pold + row[i].hv);
      }
      if (west || east) {
        ez[h] = __ldcg(Y.z + row[i].hx);
        eo[h] = __ldcg(pold + row[i].hx);
      }
    }
  };
  auto halo = [&](const double *pold) {
#pragma unroll
    for (int i = 0; i < NH; ++i) halo_row(pold, i, i);
  };
  {
    double sum[1];
    if (!res_exchange(R, S, me, sh, bar, v0, sum, [&] { halo(Y.pa); }))
      return res_fail(ctl[m], Y.err);
    fin = cg_init_step(k, sum[0]);
  }
  while (!fin) {  // ITERM bounds the loop
    {  // :93-125, and :133 of the previous iteration
      const double beta = k.beta, alpha = k.alpha;
      const double *pold = k.parity ? Y.pb : Y.pa;
      double *pnew = k.parity ? Y.pa : Y.pb;
      const bool dox = k.iter > 0;
      double v[Q][1], sum[1];
#pragma unroll
      for (int i = 0; i < Q; ++i) {
        const V4<double> ci = cci(i), po = get_p(i);
        if (dox) {
          const V4<double> x0 = get_x(i);
          put_x(i, {x0.x + alpha * po.x, x0.y + alpha * po.y, x0.z + alpha * po.z,
                    x0.w + alpha * po.w});
        }
        const V4<double> q = {ci.x * r[i].x + beta * po.x, ci.y * r[i].y + beta * po.y,
                              ci.z * r[i].z + beta * po.z, ci.w * r[i].w + beta * po.w};
        put_p(i, q);
        if constexpr (!CLUSTER) st_border(pnew, row[i], q);
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < Q; ++i) {
        const int hi = LEAN ? 0 : i;
        V4<double> h{};
        double e = 0.0;
        if (north || south)
          h = {hz[hi].x + beta * ho[hi].x, hz[hi].y + beta * ho[hi].y,
               hz[hi].z + beta * ho[hi].z, hz[hi].w + beta * ho[hi].w};
        if (west || east) e = ez[hi] + beta * eo[hi];
        V4<double> c0, ks, kw, kn, ke;
        if constexpr (LEAN) {
          const int d0 = row[i].d0;
          c0 = ld(V.cc, d0);
          if (land >> 4 * i & 1) c0.x = 1.;
          if (land >> 4 * i & 2) c0.y = 1.;
          if (land >> 4 * i & 4) c0.z = 1.;
          if (land >> 4 * i & 8) c0.w = 1.;
          ks = ld(V.cs, d0);
          kw = ld(V.cw, d0);
          kn = asym ? ld(V.cn, d0) : ld(V.cs, north ? row[i].hv : d0 + TX);  // CCN(L) = CCS(LN)
          double kwee = from_east(kw);
          if (east) kwee = V.cw[row[i].hx] * sc;
          ke = asym ? ld(V.ce, d0) : V4<double>{kw.y, kw.z, kw.w, kwee};
          if (i + 1 < Q) halo_row(pold, i + 1, 0);
        } else {
          c0 = C.get(i, 0);
          ks = C.get(i, 1);
          kw = C.get(i, 2);
          kn = C.get(i, 3);
          if constexpr (MA)
            ke = C.get(i, 4);
          else
            ke = {kw.y, kw.z, kw.w, kwe[i]};
        }
        const double *st = res_stage<W>(stage, i);
        const V4<double> pn = north ? h : ld_stage(st + TX), ps = south ? h : ld_stage(st - TX);
        const V4<double> q = get_p(i);
        double pw = from_west(q), pe = from_east(q);
        if (west) pw = e;
        if (east) pe = e;
        V4<double> a;
        a.x = c0.x * q.x + ks.x * ps.x + kn.x * pn.x + kw.x * pw + ke.x * q.y;
        a.y = c0.y * q.y + ks.y * ps.y + kn.y * pn.y + kw.y * q.x + ke.y * q.z;
        a.z = c0.z * q.z + ks.z * ps.z + kn.z * pn.z + kw.z * q.y + ke.z * q.w;
        a.w = c0.w * q.w + ks.w * ps.w + kn.w * pn.w + kw.w * q.z + ke.w * pe;
        ap[i] = a;
        v[i][0] = row[i].valid ? a.x * q.x + a.y * q.y + a.z * q.z + a.w * q.w : 0.0;
      }
      if (!res_exchange(R, S, me, sh, bar, v, sum, none)) return res_fail(ctl[m], Y.err);
      cg_matvec_epi(k, sum[0]);
    }
    {  // :134-169
      const double alpha = k.alpha;
      double v[Q][2], sum[2];
#pragma unroll
      for (int i = 0; i < Q; ++i) {
        const V4<double> ci = cci(i);
        V4<double> rv = r[i];
        rv.x = rv.x - alpha * ap[i].x;
        rv.y = rv.y - alpha * ap[i].y;
        rv.z = rv.z - alpha * ap[i].z;
        rv.w = rv.w - alpha * ap[i].w;
        r[i] = rv;
        const V4<double> z = {ci.x * rv.x, ci.y * rv.y, ci.z * rv.z, ci.w * rv.w};
        if constexpr (CLUSTER) {  // p_old too: the last row work's readers are past the exchange
          st_edge(edge, i * W + w0, z);
          st_edge(edge + NE, i * W + w0, get_p(i));
        } else {
          st_border(Y.z, row[i], z);
        }
        v[i][0] = row[i].valid ? rv.x * z.x + rv.y * z.y + rv.z * z.z + rv.w * z.w : 0.0;
        v[i][1] = row[i].valid ? rv.x * rv.x + rv.y * rv.y + rv.z * rv.z + rv.w * rv.w : 0.0;
      }
      const double *pold = k.parity ? Y.pa : Y.pb;  // the next A*p's: the p just stored
      if (!res_exchange(R, S, me, sh, bar, v, sum, [&] { halo(pold); }))
        return res_fail(ctl[m], Y.err);
      fin = cg_update_step(k, rsqm, iterm, sum[0], sum[1], 0);
    }
  }
  if constexpr (CLUSTER) cluster_barrier();  // the edges have been read
  if (k.iter > 0) {  // :133 of the last iteration
    const double alpha = k.alpha;
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const V4<double> x0 = get_x(i), po = get_p(i);
      if (row[i].valid)
        st4(P + row[i].d0, V4<double>{x0.x + alpha * po.x, x0.y + alpha * po.y,
                                      x0.z + alpha * po.z, x0.w + alpha * po.w});
    }
  }
  if (me.q0 == me.qm0 && me.nq > 0 && threadIdx.x == 0) {  // every CTA of the member has read its entry values
    Ctl &o = ctl[m];
    o.rpcg = k.rpcg;
    o.beta = k.beta;
    o.rsq = k.rsq;
    if (k.iter > 0) {
      o.papcg = k.papcg;
      o.alpha = k.alpha;
    }
    o.iter = k.iter;
    res_status(o, k.status);
    o.parity = k.parity;
    member_done(o, glob);
    if (ends.act) member_after_solve(o, ends.act[m], atomicOr(&o.asym, 0), false);
    if (!CLUSTER) R.count[size_t(m) * RES_COUNT_STRIDE + 1] = bar.count;
  }
}

int cg_res_capacity(const ResForm &f, bool may_asym, int nsm) {
  int cap = 0;
  res_form<true>(f, [&](auto w, auto q, auto cl) {
    constexpr int W = decltype(w)::value, Q = decltype(q)::value;
    constexpr bool CL = decltype(cl)::value;
    cap = may_asym
              ? res_cap(k_cg_res<true, W, Q, CL>, NT * W, res_smem64<W, Q, CL>(), nsm, f.cluster)
              : res_cap(k_cg_res<false, W, Q, CL>, NT * W, res_smem64<W, Q, CL>(), nsm, f.cluster);
  });
  return cap;
}

void launch_cg_res(const Launch &l, const DevStatic &S, const SysView &V, const DevSystem &Y,
                   double *P, Ctl *ctl, Glob *glob, const ResPlan &R, const ResForm &f, int ncta,
                   const ResEnds &ends) {
  res_form<true>(f, [&](auto w, auto q, auto cl) {
    constexpr int W = decltype(w)::value, Q = decltype(q)::value;
    constexpr bool CL = decltype(cl)::value;
    if (l.may_asym)
      launch_resident(k_cg_res<true, W, Q, CL>, ncta, NT * W, res_smem64<W, Q, CL>(), f.cluster,
                      l.stream, S, V, Y, P, ctl, glob, R, ends);
    else
      launch_resident(k_cg_res<false, W, Q, CL>, ncta, NT * W, res_smem64<W, Q, CL>(), f.cluster,
                      l.stream, S, V, Y, P, ctl, glob, R, ends);
  });
  count_launches(1);
}

}  // namespace xm

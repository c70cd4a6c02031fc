// xm_resident32.cu -- the MIXED solve of a member in one launch (see
// xm_resident.cuh): its FP64 refinement passes and their FP32 inner CG
// iterations, the FP32 vectors in registers.  Compiled with FMA contraction,
// like the multi-kernel inner iteration (xm_mixed.cu), whose rows the inner
// iteration repeats; the FP64 refinement, which the multi-kernel form compiles
// without it (xm_step.cu), is written with explicitly rounded operations.

#include "xm_resident.cuh"

namespace xm {

__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
// b - c*x - kn*xn - ks*xs - kw*xw - ke*xe (congrad.f90:72)
__device__ __forceinline__ double resid(double b, double c, double x, double kn, double xn,
                                        double ks, double xs, double kw, double xw, double ke,
                                        double xe) {
  double r = __dsub_rn(b, mul(c, x));
  r = __dsub_rn(r, mul(kn, xn));
  r = __dsub_rn(r, mul(ks, xs));
  r = __dsub_rn(r, mul(kw, xw));
  return __dsub_rn(r, mul(ke, xe));
}
__device__ __forceinline__ double sum_sq(double a, double b, double c, double d) {
  return add(add(add(mul(a, a), mul(b, b)), mul(c, c)), mul(d, d));
}

constexpr int RES_NC32 = 4;  // AS, AW, AN, AE
template <int W, int Q>
using Coef32 = ResCoef<float, W, Q, RES_NC32, Q == 1>;
template <int W, int Q>
constexpr size_t res_smem32() {
  return size_t(W) * Q * TILES_PER_CTA * TILE * sizeof(float) + Coef32<W, Q>::bytes;
}

// What bounds it: the exchanges (two per inner iteration, three per pass) and
// the latency of the row work around them; see k_cg_res.  Measured against the
// multi-kernel form, ms per MIXED step: 317x203 cells 0.124, 400x390 0.147, 512x512
// 0.38 -> 0.163, 700x700 0.45 -> 0.257.
template <bool MA, int W, int Q, bool CLUSTER>
__global__ void __launch_bounds__(NT *W, W == 1 && CLUSTER ? 2 : 1)
    k_mx_res(DevStatic S, SysView V, DevSystem Y, double *P, Ctl *ctl, Glob *glob, ResPlan R,
             RedArgs ra, int max_outer, ResEnds ends) {
  extern __shared__ __align__(16) float dyn32[];
  __shared__ ResShared<W, Q, CLUSTER> sh;
  const ResCta me = res_cta<W, Q, CLUSTER>(R, S);
  const int m = me.m;
  if (ctl[m].done) return;  // the same for the member's CTAs: it is set after their exchanges
  if constexpr (CLUSTER) cluster_barrier();  // every CTA has started: its shared memory is there
  const double rsqm = S.sc[m].rsqm;
  const int iterm = S.sc[m].iterm;
  const bool asym = unsym<MA>(ctl[m]);
  const bool poly = Y.mpoly[m] && !unsym<true>(ctl[m]);
  ResBarrier bar{CLUSTER ? 0u : R.count[size_t(m) * RES_COUNT_STRIDE + 1], 0};
  float *stage = dyn32;
  Coef32<W, Q> C;
  C.sm = dyn32 + W * Q * TILES_PER_CTA * TILE;
  const bool north = res_north(), south = res_south(), west = res_west(), east = res_east();
  const int w0 = W > 1 ? int(threadIdx.x) / NT : 0;  // quad q0 + i*W + w0 is the thread's row i
  auto none = [] {};

  Ctl k;  // the fields of the member's solve, written back at the end
  k.ccmnm_int = ctl[m].ccmnm_int;
  k.ccmnm_bc = ctl[m].ccmnm_bc;
  k.iter = k.inner_iter = k.outer = k.status = k.idone = 0;
  k.alpha = k.papcg = 0.0;
  int last_inner = ctl[m].last_inner, inner_first = ctl[m].inner_first;
  bool done = false;

  ResRow row[Q];
  V4<float> r[Q], z[Q], p[Q], ap[Q], x[Q];
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const int j = i * W + w0;
    const RowGeo g = res_geo(S, me.q0 + j, j < me.nq, row[i]);
    // the Jacobi-scaled operator, as the system is read (k_scale32's products):
    // a coupling towards or from land is 0
    const V4<double> cc = ld4(V.cc + g.d0), cs = ld4(V.cs + g.d0), cw = ld4(V.cw + g.d0);
    const V4<double> cn = ld4(V.cc + g.dn), cS = ld4(V.cc + g.ds), csn = ld4(V.cs + g.dn);
    const uchar4 kd = *reinterpret_cast<const uchar4 *>(S.kind + g.d0);
    const uchar4 kN = *reinterpret_cast<const uchar4 *>(S.kind + g.dn);
    const uchar4 kS = *reinterpret_cast<const uchar4 *>(S.kind + g.ds);
    auto inv4 = [](const V4<double> &c) {
      return V4<double>{inv_sqrt_diag(c.x), inv_sqrt_diag(c.y), inv_sqrt_diag(c.z),
                        inv_sqrt_diag(c.w)};
    };
    auto off = [](double c, double d, double dn, bool wet, bool wetn) {  // C(L)*D(L)*D(LN)
      return wet && wetn ? float(mul(mul(c, d), dn)) : 0.f;
    };
    const V4<double> D = inv4(cc), DN = inv4(cn), DS = inv4(cS);
    const bool wx = kd.x != LAND, wy = kd.y != LAND, wz = kd.z != LAND, ww = kd.w != LAND;
    double dw = from_west(D), de = from_east(D), cwe = 0.;
    // the wet flags of the cells west of the first and east of the last
    bool wetw = __shfl_up_sync(0xffffffffu, int(ww), 1, ROWT) != 0;
    bool wete = __shfl_down_sync(0xffffffffu, int(wx), 1, ROWT) != 0;
    cwe = from_east(cw);
    if (west) {
      dw = inv_sqrt_diag(V.cc[g.dwe]);
      wetw = S.kind[g.dwe] != LAND;
    }
    if (east) {
      de = inv_sqrt_diag(V.cc[g.dee]);
      wete = S.kind[g.dee] != LAND;
      cwe = V.cw[g.dee];
    }
    const V4<float> as = {off(cs.x, D.x, DS.x, wx, kS.x != LAND), off(cs.y, D.y, DS.y, wy, kS.y != LAND),
                          off(cs.z, D.z, DS.z, wz, kS.z != LAND), off(cs.w, D.w, DS.w, ww, kS.w != LAND)};
    const V4<float> aw = {off(cw.x, D.x, dw, wx, wetw), off(cw.y, D.y, D.x, wy, wx),
                          off(cw.z, D.z, D.y, wz, wy), off(cw.w, D.w, D.z, ww, wz)};
    V4<float> an, ae;
    if (asym) {
      const V4<double> c1 = ld4(V.cn + g.d0), c2 = ld4(V.ce + g.d0);
      an = {off(c1.x, D.x, DN.x, wx, kN.x != LAND), off(c1.y, D.y, DN.y, wy, kN.y != LAND),
            off(c1.z, D.z, DN.z, wz, kN.z != LAND), off(c1.w, D.w, DN.w, ww, kN.w != LAND)};
      ae = {off(c2.x, D.x, D.y, wx, wy), off(c2.y, D.y, D.z, wy, wz),
            off(c2.z, D.z, D.w, wz, ww), off(c2.w, D.w, de, ww, wete)};
    } else {  // AN(L) = AS(LN), AE(L) = AW(LE)
      an = {off(csn.x, DN.x, D.x, kN.x != LAND, wx), off(csn.y, DN.y, D.y, kN.y != LAND, wy),
            off(csn.z, DN.z, D.z, kN.z != LAND, wz), off(csn.w, DN.w, D.w, kN.w != LAND, ww)};
      ae = {aw.y, aw.z, aw.w, off(cwe, de, D.w, wete, ww)};
    }
    C.put(i, 0, as);
    C.put(i, 1, aw);
    C.put(i, 2, an);
    C.put(i, 3, ae);
    res_check_faces(S, V, ctl[m], row[i], kd, ends);
  }
  auto fail = [&] { res_fail(ctl[m], Y.err); };
  // what the neighbour tiles hold of one or two vectors, for the next row work
  V4<float> ha[Q], hb[Q];
  float ea[Q], eb[Q];
  auto halo = [&](const float *a, const float *b) {  // b: null for zeros
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      hb[i] = {0.f, 0.f, 0.f, 0.f};
      eb[i] = 0.f;
      if (north || south) {
        ha[i] = ldx4(a + row[i].hv);
        if (b) hb[i] = ldx4(b + row[i].hv);
      }
      if (west || east) {
        ea[i] = __ldcg(a + row[i].hx);
        if (b) eb[i] = __ldcg(b + row[i].hx);
      }
    }
  };

  for (int o = 0; o < max_outer && !done; ++o) {
    {  // the FP64 residual, RSQ, rhat = D^-1/2 r
      double v[Q][2], sum[2];
#pragma unroll
      for (int i = 0; i < Q; ++i) {
        ResRow rw;
        const int j = i * W + w0;
        const RowGeo g = res_geo(S, me.q0 + j, j < me.nq, rw);
        const V4<double> X0 = ldx4(P + g.d0), xn = ldx4(P + g.dn), xs = ldx4(P + g.ds);
        const V4<double> b = ld4(V.fp + g.d0), c = ld4(V.cc + g.d0), ks = ld4(V.cs + g.d0),
                         kw = ld4(V.cw + g.d0);
        const V4<double> kn = asym ? ld4(V.cn + g.d0) : ld4(V.cs + g.dn);
        const uchar4 kd = *reinterpret_cast<const uchar4 *>(S.kind + g.d0);
        double xw = from_west(X0), xe = from_east(X0), kwe = from_east(kw);
        if (west) xw = __ldcg(P + g.dwe);
        if (east) {
          xe = __ldcg(P + g.dee);
          kwe = V.cw[g.dee];
        }
        const V4<double> ke =
            asym ? ld4(V.ce + g.d0) : V4<double>{kw.y, kw.z, kw.w, kwe};
        V4<double> d;
        d.x = resid(b.x, c.x, X0.x, kn.x, xn.x, ks.x, xs.x, kw.x, xw, ke.x, X0.y);
        d.y = resid(b.y, c.y, X0.y, kn.y, xn.y, ks.y, xs.y, kw.y, X0.x, ke.y, X0.z);
        d.z = resid(b.z, c.z, X0.z, kn.z, xn.z, ks.z, xs.z, kw.z, X0.y, ke.z, X0.w);
        d.w = resid(b.w, c.w, X0.w, kn.w, xn.w, ks.w, xs.w, kw.w, X0.z, ke.w, xe);
        if (kd.x == LAND) d.x = 0.;
        if (kd.y == LAND) d.y = 0.;
        if (kd.z == LAND) d.z = 0.;
        if (kd.w == LAND) d.w = 0.;
        r[i] = {float(mul(d.x, inv_sqrt_diag(c.x))), float(mul(d.y, inv_sqrt_diag(c.y))),
                float(mul(d.z, inv_sqrt_diag(c.z))), float(mul(d.w, inv_sqrt_diag(c.w)))};
        x[i] = {0.f, 0.f, 0.f, 0.f};
        const bool ok = row[i].valid;
        v[i][0] = ok ? sum_sq(d.x, d.y, d.z, d.w) : 0.0;
        v[i][1] = ok ? sum_sq(r[i].x, r[i].y, r[i].z, r[i].w) : 0.0;
        st_border(Y.r32, row[i], r[i]);
        if (poly)
          st4(res_stage<W>(stage, i), r[i]);
        else
          st_border(Y.pa32, row[i], r[i]);
      }
      // Jacobi: z = p_old = r
      if (!res_exchange(R, S, me, sh, bar, v, sum, [&] { halo(Y.r32, poly ? nullptr : Y.pa32); }))
        return fail();
      done = mx_resid_step(k, rsqm, iterm, ra, sum[0], sum[1]);
      if (done) break;
    }
    if (poly) {  // z0 = (2I - Ahat) r, p_old = 0, RPCG = r.z0
      double v[Q][1], sum[1];
#pragma unroll
      for (int i = 0; i < Q; ++i) {
        const V4<float> h = ha[i];
        const float e = ea[i];
        const float *st = res_stage<W>(stage, i);
        const V4<float> rN = north ? h : ld4(st + TX), rS = south ? h : ld4(st - TX);
        const V4<float> r0 = r[i];
        float rw = from_west(r0), re = from_east(r0);
        if (west) rw = e;
        if (east) re = e;
        const V4<float> ks = C.get(i, 0), kw = C.get(i, 1), kn = C.get(i, 2), ke = C.get(i, 3);
        const V4<float> zv = neumann_row(r0, rS, rN, rw, re, ks, kn, kw, ke);
        z[i] = zv;
        p[i] = {0.f, 0.f, 0.f, 0.f};
        st_border(Y.z32, row[i], zv);
        v[i][0] = row[i].valid ? dot4(r0, zv)
                               : 0.0;
      }
      if (!res_exchange(R, S, me, sh, bar, v, sum, [&] { halo(Y.z32, nullptr); }))  // p_old = 0
        return fail();
      k.rpcg = sum[0];
    } else {
#pragma unroll
      for (int i = 0; i < Q; ++i) z[i] = p[i] = r[i];
    }
    int fin = 0;
    while (!fin) {  // the inner caps bound the loop (mx_update_step)
      {  // p = z + beta*p_old, Ahat*p, the previous x += alpha*p
        const float beta = float(k.beta), alpha = float(k.alpha);
        const bool dox = k.inner_iter > 0;
        float *pnew = k.parity ? Y.pa32 : Y.pb32;
        double v[Q][1], sum[1];
#pragma unroll
        for (int i = 0; i < Q; ++i) {
          if (dox) x[i] = x_plus_alpha_p(x[i], alpha, p[i]);
          p[i] = {fmaf(beta, p[i].x, z[i].x), fmaf(beta, p[i].y, z[i].y),
                  fmaf(beta, p[i].z, z[i].z), fmaf(beta, p[i].w, z[i].w)};
          st4(res_stage<W>(stage, i), p[i]);
          st_border(pnew, row[i], p[i]);
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < Q; ++i) {
          V4<float> h{};
          float e = 0.f;
          if (north || south)
            h = {fmaf(beta, hb[i].x, ha[i].x), fmaf(beta, hb[i].y, ha[i].y),
                 fmaf(beta, hb[i].z, ha[i].z), fmaf(beta, hb[i].w, ha[i].w)};
          if (west || east) e = fmaf(beta, eb[i], ea[i]);
          const float *st = res_stage<W>(stage, i);
          const V4<float> pn = north ? h : ld4(st + TX), ps = south ? h : ld4(st - TX);
          float pw = from_west(p[i]), pe = from_east(p[i]);
          if (west) pw = e;
          if (east) pe = e;
          const V4<float> ks = C.get(i, 0), kw = C.get(i, 1), kn = C.get(i, 2), ke = C.get(i, 3);
          const V4<float> q = p[i];
          const V4<float> a = scaled_ap(q, ps, pn, pw, pe, ks, kn, kw, ke);
          ap[i] = a;
          if (poly) st_border(Y.ap32, row[i], a);
          v[i][0] = row[i].valid ? dot4(a, q)
                                 : 0.0;
        }
        const float *rold = k.parity ? Y.r32b : Y.r32;
        if (!res_exchange(R, S, me, sh, bar, v, sum, [&] {
              if (poly) halo(rold, Y.ap32);
            }))
          return fail();
        cg_matvec_epi(k, sum[0]);
      }
      {  // r -= alpha*Ap, z, r.z and r.r
        const float alpha = float(k.alpha);
        float *rnew = k.parity ? Y.r32 : Y.r32b;
        double v[Q][2], sum[2];
        if (poly) {
#pragma unroll
          for (int i = 0; i < Q; ++i) {
            r[i] = {fmaf(-alpha, ap[i].x, r[i].x), fmaf(-alpha, ap[i].y, r[i].y),
                    fmaf(-alpha, ap[i].z, r[i].z), fmaf(-alpha, ap[i].w, r[i].w)};
            st4(res_stage<W>(stage, i), r[i]);
            st_border(rnew, row[i], r[i]);
          }
          __syncthreads();
#pragma unroll
          for (int i = 0; i < Q; ++i) {
            V4<float> h{};
            float e = 0.f;
            if (north || south)
              h = {fmaf(-alpha, hb[i].x, ha[i].x), fmaf(-alpha, hb[i].y, ha[i].y),
                   fmaf(-alpha, hb[i].z, ha[i].z), fmaf(-alpha, hb[i].w, ha[i].w)};
            if (west || east) e = fmaf(-alpha, eb[i], ea[i]);
            const float *st = res_stage<W>(stage, i);
            const V4<float> nN = north ? h : ld4(st + TX), nS = south ? h : ld4(st - TX);
            const V4<float> rn0 = r[i];
            float nw = from_west(rn0), ne = from_east(rn0);
            if (west) nw = e;
            if (east) ne = e;
            const V4<float> ks = C.get(i, 0), kw = C.get(i, 1), kn = C.get(i, 2),
                            ke = C.get(i, 3);
            const V4<float> zv = neumann_row(rn0, nS, nN, nw, ne, ks, kn, kw, ke);
            z[i] = zv;
            st_border(Y.z32, row[i], zv);
            double rz = 0.0, rr = 0.0;
            if (row[i].valid) {
              rz += dot4(rn0, zv);
              rr += dot4(rn0, rn0);
            }
            v[i][0] = rz;
            v[i][1] = rr;
          }
        } else {
#pragma unroll
          for (int i = 0; i < Q; ++i) {
            V4<float> rv = r[i];
            rv.x = fmaf(-alpha, ap[i].x, rv.x);
            rv.y = fmaf(-alpha, ap[i].y, rv.y);
            rv.z = fmaf(-alpha, ap[i].z, rv.z);
            rv.w = fmaf(-alpha, ap[i].w, rv.w);
            r[i] = z[i] = rv;
            st_border(rnew, row[i], rv);
            double rr = 0.0;
            if (row[i].valid)
              rr += dot4(rv, rv);
            v[i][0] = rr;
            v[i][1] = rr;
          }
        }
        // the next A*p's: z, and the p just stored
        const float *zb = poly ? Y.z32 : rnew, *pold = k.parity ? Y.pa32 : Y.pb32;
        if (!res_exchange(R, S, me, sh, bar, v, sum, [&] { halo(zb, pold); })) return fail();
        fin = mx_update_step(k, iterm, sum[0], sum[1], 2.0, 0);
      }
    }
    last_inner = k.inner_iter;
    if (k.outer == 1) inner_first = k.inner_iter;
    if (fin == 2) {
      done = true;
      break;
    }
    k.idone = 1;
    {  // P += D^-1/2 (x + alpha*p), then its borders to the neighbours
      const float alpha = float(k.alpha);
      double v[Q][1], sum[1];
#pragma unroll
      for (int i = 0; i < Q; ++i) {
        v[i][0] = 0.0;
        if (!row[i].valid) continue;
        V4<double> X0 = ldx4(P + row[i].d0);
        const V4<double> c = ld4(V.cc + row[i].d0);
        const V4<float> d = x_plus_alpha_p(x[i], alpha, p[i]);
        X0.x = add(X0.x, mul(double(d.x), inv_sqrt_diag(c.x)));
        X0.y = add(X0.y, mul(double(d.y), inv_sqrt_diag(c.y)));
        X0.z = add(X0.z, mul(double(d.z), inv_sqrt_diag(c.z)));
        X0.w = add(X0.w, mul(double(d.w), inv_sqrt_diag(c.w)));
        st4(P + row[i].d0, X0);
      }
      if (!res_exchange(R, S, me, sh, bar, v, sum, none)) return fail();
    }
  }
  if (me.q0 == me.qm0 && me.nq > 0 && threadIdx.x == 0) {  // every CTA of the member has read its entry values
    Ctl &t = ctl[m];
    t.rpcg = k.rpcg;
    t.beta = k.beta;
    t.rsq = k.rsq;
    t.rsq64 = k.rsq64;
    t.rsq_target = k.rsq_target;
    if (k.iter > 0) {
      t.papcg = k.papcg;
      t.alpha = k.alpha;
    }
    t.iter = k.iter;
    res_status(t, k.status);
    t.parity = k.parity;
    t.inner_iter = k.inner_iter;
    t.outer = k.outer;
    t.idone = k.idone;
    t.last_inner = last_inner;
    t.inner_first = inner_first;
    if (done) member_done(t, glob);
    if (ends.act) member_after_solve(t, ends.act[m], atomicOr(&t.asym, 0), true);
    if (!CLUSTER) R.count[size_t(m) * RES_COUNT_STRIDE + 1] = bar.count;
  }
}

int mx_res_capacity(const ResForm &f, bool may_asym, int nsm) {
  int cap = 0;
  res_form<false>(f, [&](auto w, auto q, auto cl) {
    constexpr int W = decltype(w)::value, Q = decltype(q)::value;
    constexpr bool CL = decltype(cl)::value;
    cap = may_asym
              ? res_cap(k_mx_res<true, W, Q, CL>, NT * W, res_smem32<W, Q>(), nsm, f.cluster)
              : res_cap(k_mx_res<false, W, Q, CL>, NT * W, res_smem32<W, Q>(), nsm, f.cluster);
  });
  return cap;
}

void launch_mx_res(const Launch &l, const DevStatic &S, const SysView &V, const DevSystem &Y,
                   double *P, Ctl *ctl, Glob *glob, const ResPlan &R, const ResForm &f, int ncta,
                   double rsqm_fac, double rel_tol, int max_outer, const ResEnds &ends) {
  RedArgs ra{};
  ra.rsqm_fac = rsqm_fac;
  ra.rel_tol = rel_tol;
  ra.margin = l.inner_margin;
  ra.unscaled = V.unscaled;
  res_form<false>(f, [&](auto w, auto q, auto cl) {
    constexpr int W = decltype(w)::value, Q = decltype(q)::value;
    constexpr bool CL = decltype(cl)::value;
    if (l.may_asym)
      launch_resident(k_mx_res<true, W, Q, CL>, ncta, NT * W, res_smem32<W, Q>(), f.cluster,
                      l.stream, S, V, Y, P, ctl, glob, R, ra, max_outer, ends);
    else
      launch_resident(k_mx_res<false, W, Q, CL>, ncta, NT * W, res_smem32<W, Q>(), f.cluster,
                      l.stream, S, V, Y, P, ctl, glob, R, ra, max_outer, ends);
  });
  count_launches(1);
}

}  // namespace xm

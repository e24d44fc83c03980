// gd_grid.cu -- grid-space column kernels of the GFS spectral dycore step.
//
// One thread per grid column; all vertical recurrences of one column run in
// that thread, reads and writes are coalesced along longitude.  Restates
// src/pressure_data.f90:58-100 (calc_pressdata), src/dyn_run.f90:307-373
// (getomega), :375-451 (getpresgrad), :453-476 (getvadv), :478-603
// (getvadv_tracers, Thuburn limiter), the tendency assembly of
// :190-292, and src/phy_run_hs.f90:42-77 (Held-Suarez forcing).
// Vertical order as in the reference: 3-D fields bottom (b=0) to top,
// interface quantities (ak, bk, pk, dpk, rlnp, alfa, etadot) top (t=0) to
// bottom; b = L-1-t.
#include <cfloat>
#include <vector>

#include "gd_grid.cuh"

namespace gd {

constexpr int LMAX = 128;

// Division, reciprocal and logarithm of the column kernel: the hardware
// approximations for the FP32 state (relative error ~1e-7, below the FP32
// state's own rounding), the FP64 state's crcp in gd_common.cuh (operands here
// are pressures, layer thicknesses and tracer differences, normal numbers).
__device__ __forceinline__ double cdiv(double a, double b) { return a * crcp(b); }
__device__ __forceinline__ float cdiv(float a, float b) { return __fdividef(a, b); }
__device__ __forceinline__ float crcp(float a) { return __fdividef(1.f, a); }
__device__ __forceinline__ float clog(float a) { return __logf(a); }

// ln(p1 / p0) and alfa = 1 - p0 / (p1 - p0) ln(p1 / p0) of a layer (dp = p1 -
// p0) in the FP64 state: 2 atanh(z) = 2 z (1 + s), z = dp / (p1 + p0), s = w
// (1/3 + w/5 + ...), w = z^2, and alfa = z - (1 - z) s.  For thin layers this
// is both cheaper than a quotient and a logarithm and free of alfa's
// cancellation.  w < 2^-10: 5 terms, w < 1/64: 8, w < 0.16: 19 (remainders
// below 3e-18); thicker layers take the logarithm.  The ranges are told apart by
// w's high word (comparisons run on the FP64 pipe).
__device__ __forceinline__ void layer_log(double p0, double p1, double dp, double& rl, double& al) {
  const double z = dp * crcp(p1 + p0), w = z * z;
  const int hw = __double2hiint(w);
  double s;
  if (hw < 0x3f500000) {
    s = 1.0 / 11;
#pragma unroll
    for (int k = 9; k >= 3; k -= 2) s = fma(s, w, 1.0 / k);
  } else if (hw < 0x3f900000) {
    s = 1.0 / 17;
#pragma unroll
    for (int k = 15; k >= 3; k -= 2) s = fma(s, w, 1.0 / k);
  } else if (hw < 0x3fc47ae1) {  // 0.16
    s = 1.0 / 39;
#pragma unroll
    for (int k = 37; k >= 3; k -= 2) s = fma(s, w, 1.0 / k);
  } else {
    rl = log(p1 / p0);
    al = 1.0 - (p0 / dp) * rl;
    return;
  }
  s *= w;
  rl = fma(z + z, s, z + z);
  al = fma(z - 1.0, s, z);
}
__device__ __forceinline__ void layer_log(float p0, float p1, float dp, float& rl, float& al) {
  rl = clog(cdiv(p1, p0));
  al = 1.f - (p0 * crcp(dp)) * rl;
}

// Thuburn (1993) limited half-level value at interior interface k
// (dyn_run.f90:574-590): qa = level above the interface, qb = level below,
// dm = dd[k-1], d0 = dd[k], dp = dd[k+1], upwind by the sign of etadot.
// Both upwind cases in one path: the columns of a warp differ in the sign.
// The limiter (phi + |phi|) / (1 + |phi|) of phi = r / d0 (r = dm or dp) is
// 2 phi / (1 + phi) = 2 r / (d0 + r) when r and d0 have one sign and 0
// otherwise: one division instead of two, and finite where r / d0 would
// overflow (d0 is clamped to the smallest normal, not to zero).
__device__ __forceinline__ float thuburn_half(float qa, float qb, float dm, float d0, float dp, float eta) {
  const float h = 0.5f * (qb + qa);
  const bool up = eta > 0.f;
  const float qu = up ? qa : qb;
  const float r = up ? dm : dp;
  const bool same = (r > 0.f) == (d0 > 0.f) && r != 0.f;
  const float lim = same ? cdiv(2.f * r, d0 + r) : 0.f;
  return qu + lim * (h - qu);
}
// FP64: h - qu is half of +-(qb - qa), so the limited value is qu +- (qb - qa)
// r / (d0 + r); the signs are read from the bit patterns (comparisons run on
// the FP64 pipe).  eta = 0 takes the other upwind value than eta > 0 would in
// the form above: its flux is 0 either way.
__device__ __forceinline__ double thuburn_half(double qa, double qb, double dm, double d0, double dp, double eta) {
  const bool up = __double2hiint(eta) >= 0;
  const double qu = up ? qa : qb, r = up ? dm : dp, d = qb - qa;
  const bool same = (__double2hiint(r) ^ __double2hiint(d0)) >= 0;
  const double lim = same ? r * crcp(d0 + r) : 0.0;
  return fma(lim, up ? d : -d, qu);
}

// dd[k] = q(level below k) - q(level above k) at interior interface k,
// clamped away from zero (dyn_run.f90:519-524)
__device__ __forceinline__ float dd_mid(float qbelow, float qabove) {
  const float d = qbelow - qabove;
  return (fabsf(d) < FLT_MIN) ? copysignf(FLT_MIN, d) : d;
}
__device__ __forceinline__ double dd_mid(double qbelow, double qabove) {
  const double d = qbelow - qabove;
  const int hi = __double2hiint(d);  // |d| < DBL_MIN: the exponent field is zero
  return (hi & 0x7ff00000) == 0 ? __hiloint2double((hi & (int)0x80000000) | 0x00100000, 0) : d;
}
// one-sided boundary differences (dyn_run.f90:507-518): dd[0] from the top
// level qt and the one below it, dd[L] from the bottom level qb and the one
// above it
template <typename R>
__device__ __forceinline__ R dd_top(R qt, R qn) {
  return (qt >= R(0)) ? qt - fmax(R(0), R(2) * qt - qn) : qt - fmin(R(0), R(2) * qt - qn);
}
template <typename R>
__device__ __forceinline__ R dd_bottom(R qb, R qn) {
  return (qb >= R(0)) ? fmax(R(0), R(2) * qb - qn) - qb : fmin(R(0), R(2) * qb - qn) - qb;
}

// Level-parallel column kernel.  A CTA owns 32 adjacent grid columns (one per
// lane, so every load and store is a 128-byte row segment) and splits the L
// levels into blocks of LB, one block per warp.  The vertical recurrences
// are scans: each thread sums its block, the block sums meet in shared
// memory, and every thread adds the sums of the blocks above it (getomega's
// top-down prefix sums, dyn_run.f90:327-337) or below it (getpresgrad's
// bottom-up sums, :416-434).  etadot at the interfaces goes through shared
// memory to the two levels that use it.  Phases:
//   1. block sums of div dp, cg dbk (top-down) and of the pressure-gradient
//      terms (bottom-up); Phillips layer pressure (pressure_data.f90:87-88);
//   2. block offsets, dlnps/dt, etadot at the block's interfaces
//      (dyn_run.f90:340-344);
//   3. omega/p (:347-368), pressure gradient, vertical advection of u, v,
//      Tv (getvadv, :453-476) and the tendencies (:190-292);
//   4. tracers, one at a time: Thuburn-limited vertical advection
//      (getvadv_tracers, :478-603) and horizontal advection.
// Levels are indexed b bottom (0) to top; interface quantities t top (0)
// to bottom; layer t = L-1-b.
// at most NWM warps (LB is chosen so); 1024 resident threads per SM for the
// FP32 state (64 registers), 512 for FP64
template <typename R, int LB, int NWM>
__global__ void __launch_bounds__(32 * NWM, (sizeof(R) == 4 ? 32 : 16) / NWM)
    k_dyn_columns(ColumnArgs<R> a, int inverse_only) {
  extern __shared__ __align__(16) unsigned char smcol[];
  // the warp's level block: the same for all its lanes (blockDim.x is 32);
  // taken through a warp reduction so that the compiler knows it too, and
  // every level index, row offset and branch on a level is warp-uniform
  const int lane = threadIdx.x, w = (int)__reduce_min_sync(0xffffffffu, threadIdx.y), NW = blockDim.y;
  const int L = a.L;
  const long ng = (long)a.nlon * a.nlat;
  const long pq = (long)blockIdx.x * 32 + lane;
  const bool valid = pq < ng;
  const long p = valid ? pq : ng - 1;  // lanes past the end compute a copy and store nothing
  const int j = (int)(p / a.nlon);
  R* part = reinterpret_cast<R*>(smcol);  // [5][NW][32] block sums, then [2][32] column totals
  R* etas = part + (5 * NW + 2) * 32;      // [L+1][32] etadot
  // FP64: ln(p(t+1)/p(t)) and alfa of every layer and bk(t)/p(t) of its top
  // interface, from phase 1 for phase 3 (each thread reads back only what it
  // wrote: no barrier); the FP32 kernel recomputes them (hardware
  // approximations).
  constexpr bool kKeep = sizeof(R) == 8;
  R* rls = etas + (L + 1) * 32;  // [L][32] (FP64 only)
  R* als = rls + L * 32;         // [L][32] (FP64 only)
  R* bps = als + L * 32;         // [L][32] (FP64 only)
  // an inverse pass without omega/p needs only the divergence sums
  const bool brief = inverse_only && !a.dlnpdtg;
  auto PART = [&](int q, int ww) -> R& { return part[(q * NW + ww) * 32 + lane]; };
  auto ETA = [&](int t) -> R& { return etas[t * 32 + lane]; };
  // Rows of the grid arrays at this column.  A 32-bit row pitch in bytes makes
  // each address one multiply-add: 64-bit products took a good part of the FP32
  // kernel's 900 instructions per level (its issue slots bound it: T574L64 5.02
  // -> 4.16 ms of a step, T254L64 2.05 -> 1.72).
  const int pitch = (int)(ng * sizeof(R));
  const char* gS = reinterpret_cast<const char*>(a.gS + p);
  auto S = [&](int row) -> R { return __ldg(reinterpret_cast<const R*>(gS + (long)row * pitch)); };
  const R* ak = a.ak;
  const R* bk = a.bk;
  const R* dbk = a.dbk;
  const R rd = a.rd;
  const R ps = exp(S(a.s.lnps));
  const R dlx = S(a.s.dlnpsdx), dly = S(a.s.dlnpsdy);
  auto PK = [&](int t) -> R { return __ldg(ak + t) + __ldg(bk + t) * ps; };
  const int b0 = w * LB;
  const int nb = max(0, min(LB, L - b0));

  // phase 1
  R xdb[LB], xcb[LB];
  R s2 = R(0), su = R(0), sv = R(0);
  // pressure and bk / p at the bottom interface of the current level, carried
  // upward (the top interface of level i is the bottom one of i + 1)
  R pkb = PK(L - b0), bpb = __ldg(bk + L - b0) * crcp(pkb);
  // the block's inputs, all loads issued before the arithmetic (levels past
  // the block's end load its last level again and are not used)
  R lu[LB], lv[LB], ldv[LB], ltv[LB], ltx[LB], lty[LB];
#pragma unroll
  for (int i = 0; i < LB; ++i) {
    const int b = b0 + min(i, nb - 1);
    lu[i] = S(a.s.u + b);
    lv[i] = S(a.s.v + b);
    ldv[i] = S(a.s.div + b);
    ltv[i] = ltx[i] = lty[i] = R(0);
    if (!inverse_only) {  // the inverse transform leaves no temperature gradients
      ltv[i] = S(a.s.tv + b);
      ltx[i] = S(a.s.dtvdx + b);
      lty[i] = S(a.s.dtvdy + b);
    }
  }
#pragma unroll
  for (int i = 0; i < LB; ++i) {
    xdb[i] = R(0);
    xcb[i] = R(0);
    if (i < nb) {
      const int b = b0 + i, t = L - 1 - b;
      const R pkt = PK(t), pkt1 = pkb, dp = pkt1 - pkt;
      pkb = pkt;
      const R cg = lu[i] * dlx + lv[i] * dly;
      xdb[i] = ldv[i] * dp;
      xcb[i] = cg * __ldg(dbk + t);
      if (!brief) {
        const R bpt = t > 0 ? __ldg(bk + t) * crcp(pkt) : R(0);  // unused at the model top (pk = 0)
        R rl = a.rlnp_top, al = a.log2sp;
        if (t > 0) {  // terms of the sums over the layers below a layer
          layer_log(pkt, pkt1, dp, rl, al);
          s2 += (bpb - bpt) * ltv[i];
          su += rl * ltx[i];
          sv += rl * lty[i];
        }
        if (kKeep) {
          rls[t * 32 + lane] = rl;
          als[t * 32 + lane] = al;
          bps[t * 32 + lane] = bpt;
        }
        bpb = bpt;
      }
      if (a.prs && valid)
        a.prs[(long)b * ng + p] =
            pow((pow(pkt1, a.kappa) * pkt1 - pow(pkt, a.kappa) * pkt) / ((a.kappa + R(1)) * dp), R(1) / a.kappa);
    }
  }
  // exclusive top-down prefix within the block (its top level is i = nb-1)
  R dbs = R(0), cbs = R(0);
#pragma unroll
  for (int i = LB - 1; i >= 0; --i) {
    const R d = xdb[i], c = xcb[i];
    xdb[i] = dbs;
    xcb[i] = cbs;
    dbs += d;
    cbs += c;
  }
  PART(0, w) = dbs;
  PART(1, w) = cbs;
  PART(2, w) = s2;
  PART(3, w) = su;
  PART(4, w) = sv;
  __syncthreads();

  // phase 2: offsets from the blocks above (DB, CB) and below (the rest).
  // Warp q scans quantity q over the blocks in place (exclusive sums; DB
  // and CB also keep their column totals), then every warp reads its own.
  for (int q = w; q < 5; q += NW) {
    R run = R(0);
    for (int k = 0; k < NW; ++k) {
      const int ww = q < 2 ? NW - 1 - k : k;
      const R v = PART(q, ww);
      PART(q, ww) = run;
      run += v;
    }
    if (q < 2) part[(5 * NW + q) * 32 + lane] = run;
  }
  __syncthreads();
  const R dbo = PART(0, w), cbo = PART(1, w);
  const R dbt = part[5 * NW * 32 + lane], cbt = part[(5 * NW + 1) * 32 + lane];
  R S2 = PART(2, w), SU = PART(3, w), SV = PART(4, w);
  const R dlnpsdt = -dbt / ps - cbt;
#pragma unroll
  for (int i = 0; i < LB; ++i) {
    xdb[i] += dbo;  // DB(t-1), CB(t-1) of layer t
    xcb[i] += cbo;
    if (i < nb) {
      const int t = L - 1 - (b0 + i);
      const R e = (t == 0) ? R(0) : -ps * (__ldg(bk + t) * dlnpsdt + xcb[i]) - xdb[i];
      ETA(t) = e;
      if (a.etadot && valid) a.etadot[(long)t * ng + p] = e;
    }
  }
  if (w == 0) {
    ETA(L) = R(0);
    if (valid) {
      if (a.etadot) a.etadot[(long)L * ng + p] = R(0);
      a.psg[p] = ps;
      a.dlnpsdt[p] = dlnpsdt;
      if (!inverse_only) a.gA[(long)a.a.dlnps * ng + p] = dlnpsdt;
    }
  }
  if (brief) return;  // uniform over the CTA
  __syncthreads();

  // phase 3
  char* gA = reinterpret_cast<char*>(a.gA + p);
  auto A = [&](int row, R v) {
    if (valid) *reinterpret_cast<R*>(gA + (long)row * pitch) = v;
  };
  const R fcor = a.omega2 * a.sinlat[j];
  const R dphx = a.dphisdx[p], dphy = a.dphisdy[p];
  R uu[LB], vv[LB], idpa[LB];
  R pkb3 = PK(L - b0), bpb3 = __ldg(bk + L - b0) * crcp(pkb3);
  // the level's values and the differences across its bottom interface (from
  // the level below)
  R um = R(0), vm = R(0), tm = R(0);
  R uc = R(0), vc = R(0), tc = R(0);
  if (nb > 0) {
    uc = S(a.s.u + b0);
    vc = S(a.s.v + b0);
    tc = S(a.s.tv + b0);
    if (b0 > 0) {
      um = S(a.s.u + b0 - 1) - uc;
      vm = S(a.s.v + b0 - 1) - vc;
      tm = S(a.s.tv + b0 - 1) - tc;
    }
  }
#pragma unroll
  for (int i = 0; i < LB; ++i) {
    uu[i] = uc;
    vv[i] = vc;
    idpa[i] = R(0);
    if (i >= nb) continue;
    const int b = b0 + i, t = L - 1 - b;
    R up = R(0), vp = R(0), tp = R(0);
    if (b + 1 < L) {
      up = S(a.s.u + b + 1);
      vp = S(a.s.v + b + 1);
      tp = S(a.s.tv + b + 1);
    }
    const R pkt = PK(t), pkt1 = pkb3, dp = pkt1 - pkt, idp = crcp(dp);
    pkb3 = pkt;
    idpa[i] = idp;
    const R bkt = __ldg(bk + t), bkt1 = __ldg(bk + t + 1);
    const R bp1 = bpb3;  // bk(t+1) / p(t+1)
    R rl, al, bpt;
    if constexpr (kKeep) {
      rl = rls[t * 32 + lane];
      al = als[t * 32 + lane];
      bpt = bps[t * 32 + lane];
    } else {
      bpt = t > 0 ? bkt * crcp(pkt) : R(0);
      rl = a.rlnp_top;
      al = a.log2sp;
      if (t > 0) {
        rl = clog(cdiv(pkt1, pkt));
        al = R(1) - (pkt * idp) * rl;
      }
    }
    bpb3 = bpt;
    const R cg = uc * dlx + vc * dly;
    const R dv = S(a.s.div + b);
    const R dbkt = __ldg(dbk + t);
    const R pcg = ps * cg;
    R wb, wc;
    if (t == 0) {
      wb = al * (dv * dp + pcg * dbkt * dbkt);
      wc = pcg * dbkt;
    } else {
      wb = rl * (xdb[i] + ps * xcb[i]) + al * (dv * dp + pcg * dbkt);
      wc = pcg * (dbkt + __ldg(a.ck + t) * (rl * idp));
    }
    const R dlnpdt = (wc - wb) * idp;  // omega / p
    if (a.dlnpdtg && valid) a.dlnpdtg[(long)b * ng + p] = dlnpdt;
    if (!inverse_only) {
      const R dtx = S(a.s.dtvdx + b), dty = S(a.s.dtvdy + b);
      // the pressure gradient's factor of R_d Tv ps grad ln ps, cofb1 - cofa of
      // dyn_run.f90:405-415: with alfa = 1 - pk/dpk rlnp all but -bk(t+1)/pk(t+1)
      // cancels; the top layer's alfa and rlnp are constants of their own
      const R pc = t == 0 ? idp * (bkt1 * pkt * crcp(pkt1) - bkt + rl * (bkt - pkt * dbkt * idp) - al * dbkt) : -bp1;
      const R com = (rd * ps) * (pc * tc - S2);
      const R prsgx = (com * dlx - dphx) - rd * (SU + al * dtx);
      const R prsgy = (com * dly - dphy) - rd * (SV + al * dty);
      const R e1 = ETA(t + 1), e0 = ETA(t);
      const R h = R(0.5) * idp;
      const R h1 = b > 0 ? h * e1 : R(0), h0 = b + 1 < L ? h * e0 : R(0);
      const R du = uc - up, dw = vc - vp, dt = tc - tp;
      const R vu = h1 * um + h0 * du;
      const R vvv = h1 * vm + h0 * dw;
      const R vt = h1 * tm + h0 * dt;
      um = du;
      vm = dw;
      tm = dt;
      R vq = a.kappa * dlnpdt * tc;
      if (a.nt > 0) vq = cdiv(vq, R(1) + a.cvap_cp * S(a.s.trc + b));
      const R vr = S(a.s.vrt + b);
      A(a.a.ttend + b, -uc * dtx - vc * dty - vt + vq);
      A(a.a.fu + b, uc * (vr + fcor) + (vvv - prsgy));
      A(a.a.fv + b, vc * (vr + fcor) - (vu - prsgx));
      A(a.a.ke + b, R(0.5) * (uc * uc + vc * vc));
      if (t > 0) {
        S2 += (bp1 - bpt) * tc;
        SU += rl * dtx;
        SV += rl * dty;
      }
    }
    uc = up;
    vc = vp;
    tc = tp;
  }
  if (inverse_only) return;

  // phase 4: tracers, one at a time.  Interface t (top of level b = L-1-t)
  // has dd[t] = q[b] - q[b+1]; the limited value at t uses dd[t-1], dd[t],
  // dd[t+1], so each level computes one new difference and carries two.
  for (int iq = 0; iq < a.nt; ++iq) {
    const int r0 = a.s.trc + iq * L;
    auto Q = [&](int b) -> R { return (b >= 0 && b < L) ? S(r0 + b) : R(0); };
    // the horizontal gradients of the block's levels, loaded ahead of their use
    R gqx[LB], gqy[LB];
#pragma unroll
    for (int i = 0; i < LB; ++i) {
      gqx[i] = gqy[i] = R(0);
      if (i < nb) {
        gqx[i] = S(a.s.dqdx + iq * L + b0 + i);
        gqy[i] = S(a.s.dqdy + iq * L + b0 + i);
      }
    }
    const int t0 = L - 1 - b0;
    R q0 = Q(b0), q1 = Q(b0 + 1), q2 = Q(b0 + 2);
    // dA = dd[t], dB = dd[t+1] for the level about to be processed; hb =
    // limited value at its bottom interface t+1 (half[L] = q[0])
    R dA, dB, hb;
    if (b0 == 0) {
      hb = q0;
      dA = dd_mid(q0, q1);  // unused when L = 1
      dB = dd_bottom(q0, q1);
    } else {
      const R qm = Q(b0 - 1), qmm = Q(b0 - 2);
      dA = (t0 == 0) ? dd_top(q0, qm) : dd_mid(q0, q1);
      dB = dd_mid(qm, q0);
      const R dC = (b0 == 1) ? dd_bottom(qm, q0) : dd_mid(qmm, qm);
      hb = thuburn_half(q0, qm, dA, dB, dC, ETA(t0 + 1));
    }
    R e1 = ETA(t0 + 1);
#pragma unroll
    for (int i = 0; i < LB; ++i) {
      if (i >= nb) continue;
      const int b = b0 + i, t = L - 1 - b;
      const R e0 = ETA(t);
      R ht = q0;  // half[0] = q at the top level
      if (t > 0) {
        const R dN = (t == 1) ? dd_top(q1, q0) : dd_mid(q1, q2);  // dd[t-1]
        ht = thuburn_half(q1, q0, dN, dA, dB, e0);
        dB = dA;
        dA = dN;
      }
      const R idp = idpa[i];
      const R vadq = (hb * e1 - ht * e0) + (q0 * (e0 - e1));
      A(a.a.qtend + iq * L + b, -uu[i] * gqx[i] - vv[i] * gqy[i] - idp * vadq);
      hb = ht;
      e1 = e0;
      q0 = q1;
      q1 = q2;
      q2 = Q(b + 3);
    }
  }
}

template <typename R, int LB, int NWM>
static void launch_cols_lb(const ColumnArgs<R>& a, bool inverse_only, cudaStream_t s) {
  const long ng = (long)a.nlon * a.nlat;
  const int nw = ceil_div(a.L, LB);
  const size_t sm = (size_t)(5 * nw + 2 + a.L + 1 + (sizeof(R) == 8 ? 3 * a.L : 0)) * 32 * sizeof(R);
  if (sm > 48 * 1024)
    GD_CUDA(cudaFuncSetAttribute(k_dyn_columns<R, LB, NWM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  k_dyn_columns<R, LB, NWM><<<(unsigned)ceil_div(ng, 32), dim3(32, nw), sm, s>>>(a, inverse_only ? 1 : 0);
}

template <typename R>
void launch_dyn_columns(const ColumnArgs<R>& a, bool inverse_only, cudaStream_t s, int lb) {
  if (a.L < 1 || a.L > LMAX) throw std::runtime_error("nlev out of range for the column kernel");
  // Levels per warp (at most 16 warps per CTA): 8 above 64 levels, else as
  // asked.  By default 4 in the FP32 state (8: T574L64 4.49 -> 5.07 ms of a step,
  // T62L28 0.081 -> 0.093).  The FP64 state with more than 32 levels takes 8, which
  // halves the work at the blocks' edges (4 -> 8: T254L64 19.8 -> 18.1 ms,
  // T126L64 4.91 -> 4.52, T42L64 0.558 -> 0.522), once every SM has a CTA; with
  // fewer levels neither is the better one throughout (T126L28 2.16 -> 2.07,
  // T94L28 1.07 -> 1.14, T42L20 0.201 -> 0.212).
  if (lb == 0) lb = sizeof(R) == 8 && a.L > 32 && (long)a.nlon * a.nlat >= 152 * 32 ? 8 : 4;
  if (a.L <= 64 && lb != 8)
    launch_cols_lb<R, 4, 16>(a, inverse_only, s);
  else
    launch_cols_lb<R, 8, 16>(a, inverse_only, s);
  count_launch();
  GD_LAUNCH_CHECK();
}
template void launch_dyn_columns<double>(const ColumnArgs<double>&, bool, cudaStream_t, int);
template void launch_dyn_columns<float>(const ColumnArgs<float>&, bool, cudaStream_t, int);

// Held-Suarez forcing on the grid (phy_run_hs.f90:42-77); prs and psg are
// recomputed from ln(ps) as in calc_pressdata.
//
// The layer pressure prs = ((p1^(k+1) - p0^(k+1)) / ((k+1)(p1 - p0)))^(1/k) of
// the layer p0..p1 is pm times a function of z = (p1 - p0) / (p1 + p0) alone,
// pm = (p1 + p0) / 2: even in z, so ln(prs/pm) and prs/pm are power series in
// w = z^2 (binomial series, coefficients from the launcher).  One logarithm
// and a few multiply-adds replace two powers, a logarithm and an exponential
// per level, and the difference of powers no longer cancels in thin layers.
// w <= 1/64: 9 terms (the remainder is below 1e-18); w <= 0.16: 20 terms
// (below 1e-17); thicker layers (the top two or three of a set that starts at
// p = 0) take the powers.  prs itself matters only below sigma = sigbot.
//
// Bound by the FP64 pipe in the FP64 state and, on small grids, by the threads
// in flight: a thread takes a.lt levels, so a T42L20 grid is 320 CTAs instead
// of 32.  Physics phase of a step (this kernel, the mass fixer and the
// update), before -> after: T254L64 FP64 state 7.77 -> 3.82 ms, T126L64 FP64
// 1.97 -> 0.97 ms, T42L20 FP64 0.330 -> 0.088 ms, T574L64 FP32 0.563 -> 0.467 ms.
template <typename R>
__global__ void __launch_bounds__(128) k_hs(const __grid_constant__ HsArgs<R> a) {
  const long ng = (long)a.nlon * a.nlat;
  const long p = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= ng) return;
  const int j = (int)(p / a.nlon);
  const int L = a.L;
  const R ps = exp(a.gS[(long)a.s.lnps * ng + p]);
  const R sl = a.sinlat[j], cl = a.coslat[j];
  const R s2 = sl * sl, c2 = cl * cl, c4 = c2 * c2;
  const R rp0 = R(1.e-5), ips = R(1) / ps, psbot = a.sigbot * ps, isig = R(1) / (R(1) - a.sigbot);
  const R t0 = R(315) - R(60) * s2, t1 = R(10) * c2, kb = (a.kradb - a.krada) * c4;
  const R sp = a.sppt ? a.sppt[p] : R(0);
  const int b1 = min(L, ((int)blockIdx.y + 1) * a.lt);
  // levels in groups of four: the group's grid loads are issued before its arithmetic
  constexpr int G = 4;
  for (int b0 = blockIdx.y * a.lt; b0 < b1; b0 += G) {
    R tvv[G], vrv[G], dvv[G];
#pragma unroll
    for (int u = 0; u < G; ++u) {
      const int b = min(b0 + u, L - 1);
      tvv[u] = a.gS[(long)(a.s.tv + b) * ng + p];
      vrv[u] = a.gS[(long)(a.s.vrt + b) * ng + p];
      dvv[u] = a.gS[(long)(a.s.div + b) * ng + p];
    }
#pragma unroll
    for (int u = 0; u < G; ++u) {
      const int b = b0 + u;
      if (b >= b1) break;
      const int t = L - 1 - b;
      const R pkt = a.ak[t] + a.bk[t] * ps, pkt1 = a.ak[t + 1] + a.bk[t + 1] * ps;
      const R dp = pkt1 - pkt, sum = pkt1 + pkt, pm = R(0.5) * sum;
      const R z = dp / sum, w = z * z;
      const bool low = !(pkt1 < psbot);  // prs < pkt1: above this level the drag profile is zero
      R lp, bl = R(0);                // ln(prs / p0), (prs / ps - sigbot) / (1 - sigbot)
      if (w <= R(0.16)) {
        lp = log(pm * rp0) + (w <= R(0.015625) ? series<R, 9>(a.lns, w) : series<R, HsArgs<R>::NS>(a.lns, w));
        if (low)
          bl = pm * ips * (w <= R(0.015625) ? series<R, 9>(a.prss, w) : series<R, HsArgs<R>::NS>(a.prss, w));
      } else {
        const R x = (pow(pkt1, a.kappa) * pkt1 - pow(pkt, a.kappa) * pkt) / ((a.kappa + R(1)) * dp);
        const R lx = log(x) / a.kappa;
        lp = lx + log(rp0);
        if (low) bl = exp(lx) * ips;
      }
      bl = low ? (bl - a.sigbot) * isig : R(0);
      if (bl < R(0)) bl = R(0);
      R teq = exp(a.expo * lp) * (t0 - lp * t1);
      if (teq < R(200)) teq = R(200);
      const R tv = tvv[u], vr = vrv[u], dv = dvv[u];
      const R f = a.sppt ? R(1) + a.vfact[b] * sp : R(1);
      a.gA[(long)b * ng + p] = f * ((a.krada + kb * bl) * (teq - tv));
      a.gA[(long)(L + b) * ng + p] = f * (-(bl * a.kdrag) * vr);
      a.gA[(long)(2 * L + b) * ng + p] = f * (-(bl * a.kdrag) * dv);
    }
  }
}
template <typename R>
void phillips_series(R kappa, int n, R* lns, R* prss) {
  // g(w) = ((1+z)^(k+1) - (1-z)^(k+1)) / (2 (k+1) z) = sum_i C(k+1, 2i+1) / (k+1) w^i,
  // h = ln(g) / k and exp(h), each series from the one before by its derivative
  const double kap = (double)kappa;
  std::vector<double> c(n), h(n), e(n);
  double bin = 1.0;  // C(k+1, 2i+1) / (k+1)
  for (int i = 0; i < n; ++i) {
    if (i > 0) bin *= (kap + 2.0 - 2 * i) * (kap + 1.0 - 2 * i) / ((2.0 * i) * (2.0 * i + 1.0));
    c[i] = bin;
  }
  h[0] = 0.0;
  for (int i = 1; i < n; ++i) {
    double v = i * c[i];
    for (int q = 1; q < i; ++q) v -= q * h[q] * kap * c[i - q];
    h[i] = v / (i * kap);
  }
  e[0] = 1.0;
  for (int i = 1; i < n; ++i) {
    double v = 0.0;
    for (int q = 1; q <= i; ++q) v += q * h[q] * e[i - q];
    e[i] = v / i;
  }
  for (int i = 0; i < n; ++i) lns[i] = (R)h[i], prss[i] = (R)e[i];
}
template void phillips_series<double>(double, int, double*, double*);
template void phillips_series<float>(float, int, float*, float*);

template <typename R>
void launch_hs_forcing(const HsArgs<R>& in, cudaStream_t s) {
  HsArgs<R> a = in;
  const long ng = (long)a.nlon * a.nlat;
  constexpr int NS = HsArgs<R>::NS;
  phillips_series(a.kappa, NS, a.lns, a.prss);
  // eight levels per thread share the column's exp and profiles; four while
  // that leaves fewer than eight CTAs per SM
  const int nx = ceil_div(ng, 128);
  a.lt = (long)nx * ceil_div(a.L, 8) >= 8 * 152 ? 8 : 4;
  k_hs<R><<<dim3(nx, ceil_div(a.L, a.lt)), 128, 0, s>>>(a);
  count_launch();
  GD_LAUNCH_CHECK();
}
template void launch_hs_forcing<double>(const HsArgs<double>&, cudaStream_t);
template void launch_hs_forcing<float>(const HsArgs<float>&, cudaStream_t);

// ------------------------------------------------------------ reductions --
__device__ double block_sum(double v) {
  __shared__ double sh[32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  double r = 0;
  if (threadIdx.x == 0)
    for (int i = 0; i < (int)(blockDim.x + 31) / 32; ++i) r += sh[i];
  return r;  // valid in thread 0
}

template <typename R>
__global__ void k_rowsum_ps(const R* psg, const double* w, int nlon, double* rowsum) {
  const int j = blockIdx.x;
  double s = 0;
  for (int i = threadIdx.x; i < nlon; i += blockDim.x) s += (double)psg[(long)j * nlon + i];
  s = block_sum(s);
  if (threadIdx.x == 0) rowsum[j] = s * (w[j] / (2.0 * nlon));
}
__global__ void k_final_sum(const double* rowsum, int n, double* out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double s = 0;
    for (int i = 0; i < n; ++i) s += rowsum[i];
    *out = s;
  }
}
template <typename R>
void launch_area_mean_ps(const R* psg, const double* w, int nlat, int nlon, double* rowsum, double* out,
                         cudaStream_t s) {
  k_rowsum_ps<R><<<nlat, 256, 0, s>>>(psg, w, nlon, rowsum);
  k_final_sum<<<1, 32, 0, s>>>(rowsum, nlat, out);
  count_launch(2);
  GD_LAUNCH_CHECK();
}
template void launch_area_mean_ps<double>(const double*, const double*, int, int, double*, double*, cudaStream_t);
template void launch_area_mean_ps<float>(const float*, const double*, int, int, double*, double*, cudaStream_t);

__global__ void k_pdry_init(const double* pmean, const double* pmoist, double* pdryini) {
  if (threadIdx.x == 0 && *pdryini == 0.0) *pdryini = *pmean - (pmoist ? *pmoist : 0.0);
}
void launch_pdry_init(const double* pmean, const double* pmoist, double* pdryini, cudaStream_t s) {
  k_pdry_init<<<1, 32, 0, s>>>(pmean, pmoist, pdryini);
  count_launch();
  GD_LAUNCH_CHECK();
}

template <typename R>
__global__ void k_massfix_grid(const R* psg, const double* pdryini, const double* pmean, const double* pwatg,
                               double grav, long ng, R* out) {
  const R pcorr = (R)((*pdryini + grav * (pwatg ? *pwatg : 0.0)) / *pmean);
  for (long p = (long)blockIdx.x * blockDim.x + threadIdx.x; p < ng; p += (long)gridDim.x * blockDim.x)
    out[p] = log(psg[p] * pcorr);
}
template <typename R>
void launch_massfix_grid(const R* psg, const double* pdryini, const double* pmean, const double* pwatg, double grav,
                         int ng, R* out, cudaStream_t s) {
  k_massfix_grid<R><<<ceil_div(ng, 256), 256, 0, s>>>(psg, pdryini, pmean, pwatg, grav, ng, out);
  count_launch();
  GD_LAUNCH_CHECK();
}
template void launch_massfix_grid<double>(const double*, const double*, const double*, const double*, double, int,
                                          double*, cudaStream_t);
template void launch_massfix_grid<float>(const float*, const double*, const double*, const double*, double, int,
                                         float*, cudaStream_t);

// per latitude: max wind speed over levels, min/max ps, area-weighted sum of
// (36 ps dlnps/dt)^2
template <typename R>
__global__ void k_diag_rows(const R* u, const R* v, int L, const R* psg, const R* dl, const double* w, int nlat,
                            int nlon, double* part) {
  const int j = blockIdx.x;
  const long ng = (long)nlat * nlon;
  double smax = 0, pmin = 1e300, pmax = -1e300, pt = 0;
  for (int i = threadIdx.x; i < nlon; i += blockDim.x) {
    const long p = (long)j * nlon + i;
    for (int k = 0; k < L; ++k) {
      double uu = u[k * ng + p], vv = v[k * ng + p];
      smax = fmax(smax, sqrt(uu * uu + vv * vv));
    }
    double ps = psg[p];
    pmin = fmin(pmin, ps / 100.);
    pmax = fmax(pmax, ps / 100.);
    double x = 36. * ps * (double)dl[p];
    pt += x * x;
  }
  __shared__ double a[256], b[256], c[256], d[256];
  a[threadIdx.x] = smax;
  b[threadIdx.x] = pmin;
  c[threadIdx.x] = pmax;
  d[threadIdx.x] = pt;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      a[threadIdx.x] = fmax(a[threadIdx.x], a[threadIdx.x + o]);
      b[threadIdx.x] = fmin(b[threadIdx.x], b[threadIdx.x + o]);
      c[threadIdx.x] = fmax(c[threadIdx.x], c[threadIdx.x + o]);
      d[threadIdx.x] += d[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[4 * j + 0] = a[0];
    part[4 * j + 1] = b[0];
    part[4 * j + 2] = c[0];
    part[4 * j + 3] = d[0] * (w[j] / (2.0 * nlon));
  }
}
__global__ void k_diag_final(const double* part, int nlat, double* out) {
  if (threadIdx.x != 0) return;
  double smax = 0, pmin = 1e300, pmax = -1e300, pt = 0;
  for (int j = 0; j < nlat; ++j) {
    smax = fmax(smax, part[4 * j]);
    pmin = fmin(pmin, part[4 * j + 1]);
    pmax = fmax(pmax, part[4 * j + 2]);
    pt += part[4 * j + 3];
  }
  out[0] = smax;
  out[1] = pmin;
  out[2] = pmax;
  out[3] = sqrt(pt);
}
template <typename R>
void launch_diag(const R* u, const R* v, int L, const R* psg, const R* dlnpsdt, const double* w, int nlat, int nlon,
                 double* scratch, double* out, cudaStream_t s) {
  k_diag_rows<R><<<nlat, 256, 0, s>>>(u, v, L, psg, dlnpsdt, w, nlat, nlon, scratch);
  k_diag_final<<<1, 32, 0, s>>>(scratch, nlat, out);
  count_launch(2);
  GD_LAUNCH_CHECK();
}
template void launch_diag<double>(const double*, const double*, int, const double*, const double*, const double*,
                                  int, int, double*, double*, cudaStream_t);
template void launch_diag<float>(const float*, const float*, int, const float*, const float*, const double*, int,
                                 int, double*, double*, cudaStream_t);

}  // namespace gd

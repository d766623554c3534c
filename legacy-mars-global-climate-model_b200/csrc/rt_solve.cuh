// Thread-per-system solves of the pipeline in the arithmetic of
// rt_fastmath.cuh: the passes of rt_fp64_sys.cuh (solve_vis, solve_ir),
// operation for operation, for systems whose operands stay in range.  A
// system that leaves it anywhere (`odd`) is redone by the general solve.
//
// Range: the stage marks bands with |COSBAR| >= 1 or an unusual scattering
// numerator (usual_layer); pass A checks that the optical depths of the
// layer's two levels (visible: and of level 2) are in [0, 2^99) (unusual_depth)
// and its albedo in [0, 1), pass C every eliminated denominator (and, visible,
// the root and the divisor of GAMA).  What else is divided by or rooted then
// lies in range: 1 - W0 COSB >= 2^-53, and ALPHA within 2^27 of 1.  Every
// depth from the top down to a middle of a layer is a sum of depths that are
// not negative, so the exponents of the layers' middles are in [0, 35], EP in
// [1, exp(35)], and those of the beam in [-35, 0].  The sign of the sum of a
// layer's depths is not enough: with -3000 and 3005 the middle's exponent is
// -3000, exp_r wraps, and finite values come out for infinities.
//
// IR solve of 8,192 x 24 columns: 896 instructions issued per layer and warp
// in the general arithmetic, 581 in this one (a pass over the layers less, too).
#pragma once
#include "rt_fp64_sys.cuh"

namespace mgcm {
namespace fp64 {

// Per-layer values of a system in local memory, a record per layer so that
// a thread indexes them with one register, in 16-byte accesses: the rows 2l-1
// and 2l of DSOLVER (AS, DS) and
//   IR       DTAUKI of the layer's two levels;
//   visible  W0, DTAU; TAU at the top and the middle.
struct alignas(16) IrSlot {
    double2 odd, even, pair;
};
struct alignas(16) VisSlot {
    double2 odd, even, pair, depth;
};
union SolveLocal {
    SysLocal g;   // the general solve's
    IrSlot ir[D_MAXNL + 1];
    VisSlot vis[D_MAXNL + 1];
    __device__ SolveLocal() {}
};

// An optical depth outside [0, 2^99): negative (-0 too), infinite or NaN.
__device__ __forceinline__ bool unusual_depth(double d) { return hi32(d) >= 0x46200000u; }
__device__ __forceinline__ bool unusual_depths(double a, double b) { return max(hi32(a), hi32(b)) >= 0x46200000u; }

// The general solves, out of line: systems out of range only.  They carve the
// column block themselves, so that the callers' ColSmem stays in registers.
static __device__ __noinline__ void general_ir(const SegDev &sg, int c, int j, unsigned char *block, int max_nl,
                                        const RtConst &K, const double *__restrict__ ki, SysLocal &w, double *row,
                                        double *rdn, double *scr) {
    unsigned int dummy = 0;
    ColSmem s = carve_smem(block, max_nl, nullptr, false);
    solve_ir<2>(sg, c, j / D_NG + 1, j % D_NG + 1, NSYS_V + j, s, K, ki, w, dummy, row, rdn, scr, ROW_BLK);
}

template <int MODE, bool F32>
static __device__ __noinline__ unsigned int general_vis(const SegDev &sg, int c, int t, unsigned char *block, int max_nl,
                                                 const RtConst &K, const double *__restrict__ kv,
                                                 const float *__restrict__ kvf, SysLocal &w, double *row,
                                                 double *rdn, double *scr) {
    unsigned int nsolved = 0;
    ColSmem s = carve_smem(block, max_nl, nullptr, false);
    solve_vis<MODE, F32>(sg, c, t / D_NG + 1, t % D_NG + 1, t, s, K, kv, w, nsolved, row, rdn, scr, scr + ROW_BLK,
                         scr + 2 * ROW_BLK, kvf, ROW_BLK);
    return nsolved;
}

// TAUGAS of the two levels K = k, k+1 of a layer (taugas_at, taugas_f).  The
// second level's table values are mostly the first one's (KLevel::same): a
// layer's 16 gathered values become 8, its two interpolations one.  With the
// one-pass IR solve below: 64,800 x 24 FP64 11.45 -> 10.3 ms, 16,200 x 48
// 7.80 -> 7.03 ms, 60 x 24 235 -> 215 us.
template <bool F32, class T>
__device__ __forceinline__ void taugas_layer(const ColSmem &s, int k, const T *__restrict__ tb, T &t1, T &t2) {
    const KLv kl = klev_load(s, k);
    const T *p = tb + kl.kd.x;
    const int dh = kl.kd.y;
    T c[4], d[4];
    c[0] = __ldg(p);
    c[1] = __ldg(p + KT_DP);
    c[2] = __ldg(p + KT_DT + KT_DP);
    c[3] = __ldg(p + KT_DT);
    p += dh;
    d[0] = __ldg(p) - c[0];
    d[1] = __ldg(p + KT_DP) - c[1];
    d[2] = __ldg(p + KT_DT + KT_DP) - c[2];
    d[3] = __ldg(p + KT_DT) - c[3];
    auto value = [&](T wr) {
        const T k1 = c[0] + wr * d[0], k2 = c[1] + wr * d[1], k3 = c[2] + wr * d[2], k4 = c[3] + wr * d[3];
        return (T)kl.lk01.x * k1 + (T)kl.lk01.y * k2 + (T)kl.lk23.x * k3 + (T)kl.lk23.y * k4;
    };
    const double2 *q2 = reinterpret_cast<const double2 *>(s.klev + k + 1);
    const double2 wu = q2[2];
    const int same = reinterpret_cast<const int4 *>(q2 + 3)->z;
    const T v = value((T)kl.wu.x);
    t1 = (F32 ? (T)s.dpr[k] : (T)kl.wu.y) * v;
    const T u2 = F32 ? (T)s.dpr[k + 1] : (T)wu.y;
    if (same == SAME_VALUE) t2 = u2 * v;
    else if (same == SAME_CORNERS) t2 = u2 * value((T)wu.x);
    else if constexpr (F32) t2 = taugas_f(s, k + 1, tb);
    else t2 = taugas_at(s, k + 1, tb);
}

// Fetches the line of a global address into L1: the solves ask for the next
// layer's records a layer ahead (64,800 x 24: 9.86 -> 9.62 ms FP64, 9.72 -> 9.37
// ms MIXED).  Asking for the next layer's table values too was slower (11.2 ms):
// with the per-layer values streaming through it, L1 has no room.
__device__ __forceinline__ void prefetch_l1(const void *p) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// x / u0 capped at MAXEXP, y = 1 / u0 (GFLUXV's beam exponents).
__device__ __forceinline__ double beam(double x, double u0, double y) {
    return exp_r(-dmin(quot(x, u0, y), MAXEXP));
}

// Lay's exponential terms from GAMA and LAMDA*DTAU (gfluxi.f90:113-123, gfluxv.f90:150-163).
__device__ __forceinline__ void exp_terms(Lay &y, double x) {
    const double ep = exp_r(dmin(x, TAUMAX)), em = rcp_n(ep);
    const double a = y.gama * em, b = y.gama * ep;
    y.e1 = ep + a;
    y.e2 = ep - a;
    y.e3 = b + em;
    y.e4 = b - em;
}

// rows_of_pair with the fast reciprocal; odd collects the range tests.
__device__ __forceinline__ void fast_rows(const Lay &lo, const Lay &hi, double &as, double &ds, double &as_odd,
                                          double &ds_odd, bool &odd) {
    const double hp = hi.gama - 1.0, c13 = (lo.e1 + lo.e3) * hp;
    const double dp = hi.cpm1 - lo.cp, dm = lo.cm - hi.cmm1;
    {
        const double af = 2.0 * (1.0 - lo.gama * lo.gama);
        const double den = (lo.e1 - lo.e3) * (1.0 + hi.gama) - c13 * as;
        const double df = lo.e3 * dp + lo.e1 * dm;
        odd |= out_of_range(den);
        const double x = rcp_s(den);
        ds = (df - c13 * ds) * x;
        as = af * x;
        as_odd = as;
        ds_odd = ds;
    }
    {
        const double cf = 2.0 * (1.0 - hi.gama * hi.gama);
        const double den = (lo.e2 + lo.e4) * hp - cf * as;
        const double df = hp * dp + (1.0 - hi.gama) * dm;
        odd |= out_of_range(den);
        const double x = rcp_s(den);
        ds = (df - cf * ds) * x;
        as = c13 * x;
    }
}

// ---------------------------------------------------------------- infrared
// TAUGSURF of an IR system in the reference order (code/optci.f90:143-167).
static __device__ __noinline__ double ir_taugsurf(unsigned char *block, int max_nl, int lev,
                                                  const double *__restrict__ tb) {
    const ColSmem s = carve_smem(block, max_nl, nullptr, false);
    double taug = 0.0;
    for (int k = 2; k <= lev; ++k) taug += taugas_at(s, k, tb);
    return taug;
}

// System i % 85 of column i / 85 of the chunk: the TLIMIT decision
// (code/sfluxi.f90:72-75) and the solve.  Returns 0 solved, 1 skipped (TLIMIT), 2 no work, and writes the
// column's skip entry.
//
// Optical depths, coefficients and elimination run in one bottom-up pass, so
// a layer's table gathers overlap the arithmetic of the ones before it; a
// pass of its own for the gathers (top-down, as the reference's) was bound
// by their latency and sent 24 more bytes per layer through local memory.
// What needs the top-down order is formed in pass D (TAUCUMI, for the middle
// of the layers) or decided apart: the gas optical depths are summed bottom-up
// here, and where that sum, at most 1e-13 off the reference's, does not
// decide the TLIMIT test -- or a depth is negative -- they are summed again.
__device__ __forceinline__ int fast_ir(const SegTable *__restrict__ st, int col_begin, int i, int max_nl,
                                       unsigned char *__restrict__ blocks, size_t stride, const RtConst &K,
                                       const double *__restrict__ ki, SolveLocal &w, double *__restrict__ fl,
                                       double *__restrict__ sc) {
    double tc, as1, ds1;
    unsigned flags;   // bit 0: out of range; bit 31: a negative gas optical depth
    // LAMDA, GAMA, TERM of a layer (code/gfluxi.f90:69-93), UBARI = 0.5.
    // Passes C and D both evaluate them, B1 too: cheaper than a round trip
    // of four more values per layer through local memory.
    auto lay3 = [&](double cosb, double w0, double &lam, double &gama, double &term) {
        const double d = 1.0 - w0 * cosb, y = rcp_n(d);
        const double alpha = sqrt_n(quot(1.0 - w0, d, y));
        const double ap1 = 1.0 + alpha;
        lam = alpha * d * 2.0;
        gama = quot(1.0 - alpha, ap1, rcp_n(ap1));
        term = 0.5 * y;
    };
    // The reference's added 1.D-50 has no effect on a DTAUI above its TINY.
    const double tiny = R4(1.0E-9);
    {
        const int cc = i / NSYS_I, j = i - cc * NSYS_I, g = col_begin + cc;
        const SegDev &sg = st->seg[find_seg(st, g)];
        const ColSmem s = carve_smem(blocks + (size_t)cc * stride, max_nl, nullptr, false);
        const int nb = j / D_NG;   // 0-based band
        const int NL = sg.L + 1, LEV = 2 * NL + 1, ng = j - nb * D_NG;
        const bool gas = ng < D_NG - 1;
        if (gas && K.fzeroi[nb] >= R4(0.99)) return s.skip[NSYS_V + j] = 2;
        const double *tb = ki + (size_t)nb * D_NT * D_NP * D_NH * D_NGK + ng;
        flags = (*s.odd >> (D_NV + nb)) & 1;
        double taug;
        double dt1 = 0.0;
        // pass C of one layer
        auto coef = [&](const IrLayer &r, double dtsum) {
            const bool thick = dtsum > tiny;
            const double dt = thick ? dtsum : tiny, ydt = rcp_n(dt);
            const double w0 = thick ? quot(r.wnum, dt, ydt) : 0.0;
            if (hi32(w0) >= 0x3ff00000u) flags |= 1;   // 0 <= WBARI < 1
            dt1 = dt;
            Lay y;
            double lam, term;
            lay3(r.cosb, w0, lam, y.gama, term);
            const double b1 = quot(r.pdif, dt, ydt), b0 = r.b0;
            const double bt = b1 * term, bb = b0 + b1 * dt;
            y.cp = bb + bt;
            y.cm = bb - bt;
            y.cpm1 = b0 + bt;
            y.cmm1 = b0 - bt;
            exp_terms(y, lam * dt);
            return y;
        };
        const IrLayer *r = &s.ir(NL, nb + 1);
        double2 e = r->ext[0];
        double tg = gas ? taugas_at(s, LEV, tb) : 0.0;
        taug = tg;
        flags |= hi32(tg) & 0x80000000u;
        double da = gas ? tg + e.x + e.y : e.x + e.y;
        if (unusual_depth(da)) flags |= 1;
        w.ir[NL].pair = make_double2(da, 0.0);
        Lay hi = coef(*r, da);
        double as, ds;
        bottom_row_v(hi, s.bsurf_i[nb], sg.albi[cc + col_begin - sg.col0], as, ds);
        w.ir[NL].even = make_double2(as, ds);
#pragma unroll 1
        for (int n = NL - 1; n >= 1; --n) {
            --r;
            const double2 e1 = r->ext[0], e2 = r->ext[1];
            double db;
            if (gas) {
                double t1, t2;
                taugas_layer<false>(s, 2 * n + 1, tb, t1, t2);
                taug += t2;
                taug += t1;
                flags |= (hi32(t1) | hi32(t2)) & 0x80000000u;
                da = t1 + e1.x + e1.y;
                db = t2 + e2.x + e2.y;
            } else {
                da = e1.x + e1.y;
                db = e2.x + e2.y;
            }
            if (unusual_depths(da, db)) flags |= 1;
            w.ir[n].pair = make_double2(da, db);
            if (n > 1) {
                prefetch_l1(r - 1);
                prefetch_l1(s.klev + 2 * n - 1);
            }
            const Lay lo = coef(*r, da + db);
            double ao, dd;
            bool odd = false;
            fast_rows(lo, hi, as, ds, ao, dd, odd);
            if (odd) flags |= 1;
            w.ir[n + 1].odd = make_double2(ao, dd);
            w.ir[n].even = make_double2(as, ds);
            hi = lo;
        }
        --r;
        e = r->ext[1];
        tg = gas ? taugas_at(s, 2, tb) : 0.0;
        taug += tg;
        flags |= hi32(tg) & 0x80000000u;
        tc = 0.0 + (gas ? tg + e.x + e.y : e.x + e.y);
        if (gas) {
            bool skip = taug < TLIMITI;
            if ((flags >> 31) || !(fabs(taug - TLIMITI) > 1e-12 * TLIMITI))
                skip = ir_taugsurf(blocks + (size_t)cc * stride, max_nl, LEV, tb) < TLIMITI;
            if (skip) return s.skip[NSYS_V + j] = 1;
        }
        s.skip[NSYS_V + j] = 0;
        const double *plev = sg.plev + (size_t)(cc + col_begin - sg.col0) * LEV;
        const double tautop = dt1 * plev[2 - 1] / (plev[4 - 1] - plev[2 - 1]);
        const double btop = (1.0 - mgcm_rt_exp(-tautop / UBARI)) * s.pltop_i[nb];
        const double cf = hi.gama - 1.0, den = hi.gama + 1.0 - cf * as;
        if (out_of_range(den)) flags |= 1;
        const double x = rcp_s(den);
        as1 = 0.0 * x;
        ds1 = (btop - hi.cmm1 - cf * ds) * x;
    }
    // pass D; what it needs of the column is found again rather than held in
    // registers through pass C
    asm volatile("" : "+r"(i));
    const int cc = i / NSYS_I, nb = (i - cc * NSYS_I) / D_NG;
    const SegDev &sg = st->seg[find_seg(st, col_begin + cc)];
    const int NL = sg.L + 1;
    unsigned char *block = blocks + (size_t)cc * stride;
    double *fmp = fl + row_base(i, max_nl), *fmm = fmp + (size_t)max_nl * ROW_BLK, *sc0 = sc + sc_base(i);
    if (flags & 1) {
        general_ir(sg, col_begin + cc - sg.col0, i - cc * NSYS_I, block, max_nl, K, ki, w.g, fmp, fmm, sc0);
        return 0;
    }
    const IrLayer *r = &carve_smem(block, max_nl, nullptr, false).ir(0, nb + 1);
    double xprev = 0.0;
    double2 n1 = make_double2(as1, ds1), n2 = w.ir[1].even, np = w.ir[1].pair;
#pragma unroll 1
    for (int n = 1; n <= NL; ++n) {
        const double2 r1 = n1, r2 = n2, p = np;
        if (n < NL) {
            n1 = w.ir[n + 1].odd;
            n2 = w.ir[n + 1].even;
            np = w.ir[n + 1].pair;
        }
        ++r;
        if (n < NL) prefetch_l1(r + 1);
        const double tcA = tc + p.x;
        const double dtsum = n < NL ? p.x + p.y : p.x;
        const bool thick = dtsum > tiny;
        const double dt = thick ? dtsum : tiny, ydt = rcp_n(dt);
        const double w0 = thick ? quot(r->wnum, dt, ydt) : 0.0;
        const double dtk = n < NL ? tcA - tc : dt;
        tc = tcA + p.y;
        double lam, gama, term;
        lay3(r->cosb, w0, lam, gama, term);
        const double b1 = quot(r->pdif, dt, ydt), b0 = r->b0;
        const double xa = n == 1 ? r1.y : r1.y - r1.x * xprev;
        const double xb = r2.y - r2.x * xa;
        xprev = xb;
        double xk1, xk2;
        unmix(xa, xb, xk1, xk2);
        const double ep = exp_r(dmin(lam * dtk, TAUMAX)), em = rcp_n(ep);
        const double bt = b1 * term, bb = b0 + b1 * dtk;
        const double u = xk1 * ep, v = gama * xk2 * em;
        const double p1 = u + v + (bb + bt);
        const double m1 = u * gama + xk2 * em + (bb - bt);
        *fmp = p1 * PI_D;
        *fmm = m1 * PI_D;
        fmp += ROW_BLK;
        fmm += ROW_BLK;
        if (n == 1) {
            const double fup = xk1 + gama * xk2 + (b0 + bt);
            const double fdn = xk1 * gama + xk2 + (b0 - bt);
            *sc0 = (fup - fdn) * PI_D;
        }
    }
    return 0;
}

// ---------------------------------------------------------------- visible
// Pass A of system t: TAUs per layer (kept with KEEP), the surface values,
// and whether an operand left the range.
template <bool KEEP, bool F32>
struct VisPassA {
    double taugsurf = 0.0, tau = 0.0, tclev = 0.0, tce1 = 0.0;
    bool odd = false;
    __device__ __forceinline__ void run(const SegDev &sg, int t, const ColSmem &s, const double *__restrict__ kv,
                                        const float *__restrict__ kvf, SolveLocal &w) {
        const int L = sg.L, NL = L + 1;
        const int nb = t / D_NG, ng = t - nb * D_NG;
        const bool gas = ng < D_NG - 1;
        const size_t to = (size_t)nb * D_NT * D_NP * D_NH * D_NGK + ng;
        const double *tb = kv + to;
        const float *tbf = F32 ? kvf + to : nullptr;
        const VisLayer *lay = &s.vis(0, nb + 1);
        auto level = [&](int k, double ray) -> double {
            if (!gas) return ray;
            const double tg = F32 ? (double)taugas_f(s, k, tbf) : taugas_at(s, k, tb);
            taugsurf += tg;
            return tg + ray;
        };
        odd = (*s.odd >> nb) & 1;
        const double tc2 = 0.0 + level(2, lay->ray[1]);
        odd |= unusual_depth(tc2);
        double tc = tc2, fprev = 0.0;
#pragma unroll 1
        for (int l = 1; l <= NL; ++l) {
            const int k = 2 * l + 1;
            ++lay;
            if (l < NL) {
                prefetch_l1(lay + 1);
                prefetch_l1(s.klev + k + 2);
            }
            double da, dt, tcA, tcB;
            if (l <= L) {
                double db;
                if (gas) {
                    if constexpr (F32) {
                        float t1, t2;
                        taugas_layer<true>(s, k, tbf, t1, t2);
                        da = t1;
                        db = t2;
                    } else {
                        taugas_layer<false>(s, k, tb, da, db);
                    }
                    taugsurf += da;
                    taugsurf += db;
                    da = da + lay->ray[0];
                    db = db + lay->ray[1];
                } else {
                    da = lay->ray[0];
                    db = lay->ray[1];
                }
                odd |= unusual_depths(da, db);
                tcA = tc + da;
                tcB = tcA + db;
                dt = da + db;
            } else {
                dt = da = level(k, lay->ray[0]);
                odd |= unusual_depth(da);
                tcA = tcB = tc + da;
            }
            const double cosb = lay->cosb;
            const double wb = quot(lay->wnum, dt, rcp_n(dt));
            const double f = 1.0 - wb * (cosb * cosb);
            odd |= hi32(dt) < 0x2d300000u || hi32(wb) >= 0x3ff00000u;   // below 2^-300; outside [0, 1)
            const double dtl = dt * f;
            if (KEEP) {
                double m = 0.0;
                if (l == 1) {
                    tce1 = tc2 * f;
                    m = tce1 + (tcA - tc2) * f;
                } else if (l < NL) {
                    m = tau + (tcA - tc) * fprev;
                }
                w.vis[l].pair = make_double2(quot(wb * (1.0 - cosb * cosb), f, rcp_n(f)), dtl);
                w.vis[l].depth = make_double2(tau, m);
            }
            tau = tau + dtl;
            fprev = f;
            tc = tcB;
        }
        tclev = tc;
    }
};

// The TLIMIT decision of system t of a day column after its pass A, with
// DETAU and CUMTAUV (code/sfluxv.f90:60-75); true when it is to be solved.
template <class PassA>
__device__ __forceinline__ bool vis_decision(const PassA &a, const SegDev &sg, int c, int t, const ColSmem &s,
                                             const RtConst &K) {
    const int nb = t / D_NG, ng = t - nb * D_NG;
    const size_t o = (size_t)c * NSYS_V + nb + D_NV * ng;
    sg.cumtauv[o] = a.tclev;
    if (ng < D_NG - 1 && K.fzerov[nb] >= R4(0.99)) {
        s.skip[t] = 2;
        return false;
    }
    sg.detau[o] = a.tau;
    const bool skip = ng < D_NG - 1 && a.taugsurf < TLIMITS;
    s.skip[t] = skip ? 1 : 0;
    return !skip;
}

// Screen of system t of a day column; true when it is to be solved.
template <bool F32>
__device__ __forceinline__ bool fast_vis_screen(const SegDev &sg, int c, int t, unsigned char *block, int max_nl,
                                                const ColSmem &s, const RtConst &K, const double *__restrict__ kv,
                                                const float *__restrict__ kvf, SolveLocal &w,
                                                unsigned int &nsolved) {
    VisPassA<false, F32> a;
    a.run(sg, t, s, kv, kvf, w);
    if (a.odd) {
        nsolved += general_vis<1, F32>(sg, c, t, block, max_nl, K, kv, kvf, w.g, nullptr, nullptr, nullptr);
        return s.skip[t] == 0;
    }
    const bool keep = vis_decision(a, sg, c, t, s, K);
    nsolved += keep ? 1 : 0;
    return keep;
}

// Solve of a visible system the screen kept; with DENSE of any system of a day
// column, the decision taken after pass A.  Returns whether it was solved.
template <bool F32, bool DENSE = false>
__device__ __forceinline__ bool fast_vis(const SegDev &sg, int c, int t, unsigned char *block, int max_nl,
                                         const RtConst &K, const double *__restrict__ kv,
                                         const float *__restrict__ kvf, SolveLocal &w, double *fmp, double *fmm,
                                         double *sc) {
    const ColSmem s = carve_smem(block, max_nl, nullptr, false);
    const int NL = sg.L + 1, nb = t / D_NG;
    const double u0 = sg.acosz[c], rsf = sg.als[c], f0pi = sg.sol[nb];
    VisPassA<true, F32> a;
    a.run(sg, t, s, kv, kvf, w);
    if (DENSE) {
        if (a.odd) {
            if (!general_vis<1, F32>(sg, c, t, block, max_nl, K, kv, kvf, w.g, nullptr, nullptr, nullptr)) return false;
        } else if (!vis_decision(a, sg, c, t, s, K)) {
            return false;
        }
    }
    // u0 in [2^-30, 2^30), the band's sun 0 or in [2^-60, 2^60)
    bool odd = a.odd || hi32(u0) - 0x3e100000u >= 0x03c00000u || (f0pi != 0.0 && hi32(f0pi) - 0x3c300000u >= 0x07800000u);
    if (!odd) {
        const VisLayer *lay = &s.vis(NL, nb + 1);
        const double rcp_u0 = rcp_n(u0), rcp_u02 = 1.0 / (u0 * u0);
        const double s3 = (double)sqrtf(3.0f), s3h = (double)(sqrtf(3.0f) * 0.5f);
        const double bsurf = rsf * u0 * f0pi * beam(a.tau, u0, rcp_u0);
        // LAMDA, GAMA, AM, AP of a layer (code/gfluxv.f90:108-150).  Passes C
        // and D both evaluate them: cheaper than 32 more bytes per layer
        // through local memory.
        auto lay4 = [&](double w0, double cb, double &lam, double &gama, double &am, double &ap) {
            const double g1 = s3h * (2.0 - w0 * (1.0 + cb));
            const double g2 = (s3 * w0 * 0.5) * (1.0 - cb);
            const double g3 = 0.5 * (1.0 - s3 * cb * u0);
            const double l2 = g1 * g1 - g2 * g2;
            odd |= hi32(l2) - 0x2d300000u >= 0x25800000u || out_of_range(g2);
            lam = sqrt_n(l2);
            gama = quot(g1 - lam, g2, rcp_s(g2));
            const double g4 = 1.0 - g3;
            double denom = lam * lam - rcp_u02;
            if (denom == 0.0) denom = R4(1.E-10);
            const double rd = rcp_s(denom);
            am = quot(f0pi * w0 * (g4 * (g1 + rcp_u0) + g2 * g3), denom, rd);
            ap = quot(f0pi * w0 * (g3 * (g1 - rcp_u0) + g2 * g4), denom, rd);
        };
        // pass C
        auto coef = [&](double2 p, double cb, double et_top, double et_bot) {
            Lay y;
            double lam, am, ap;
            lay4(p.x, cb, lam, y.gama, am, ap);
            y.cpm1 = ap * et_top;
            y.cmm1 = am * et_top;
            y.cp = ap * et_bot;
            y.cm = am * et_bot;
            exp_terms(y, lam * p.y);
            return y;
        };
        double et_bot = beam(a.tau, u0, rcp_u0), et_top = beam(w.vis[NL].depth.x, u0, rcp_u0);
        Lay hi = coef(w.vis[NL].pair, lay->cbs, et_top, et_bot);
        double as, ds;
        bottom_row_v(hi, bsurf, rsf, as, ds);
        w.vis[NL].even = make_double2(as, ds);
        double2 nxt = w.vis[NL - 1].pair;
        double nd = w.vis[NL - 1].depth.x;
#pragma unroll 1
        for (int n = NL - 1; n >= 1; --n) {
            const double2 cur = nxt;
            const double d = nd;
            if (n > 1) {
                nxt = w.vis[n - 1].pair;
                nd = w.vis[n - 1].depth.x;
            }
            et_bot = et_top;
            et_top = beam(d, u0, rcp_u0);
            --lay;
            if (n > 1) prefetch_l1(&lay[-1].cbs);
            const Lay lo = coef(cur, lay->cbs, et_top, et_bot);
            double ao, dd;
            fast_rows(lo, hi, as, ds, ao, dd, odd);
            w.vis[n + 1].odd = make_double2(ao, dd);
            w.vis[n].even = make_double2(as, ds);
            hi = lo;
        }
        {
            const double cf = hi.gama - 1.0, den = hi.gama + 1.0 - cf * as;
            odd |= out_of_range(den);
            const double x = rcp_s(den);
            w.vis[1].odd = make_double2(0.0 * x, (0.0 - hi.cmm1 - cf * ds) * x);
        }
        if (!odd) {
            // pass D
            double xprev = 0.0;
            double2 n1 = w.vis[1].odd, n2 = w.vis[1].even, nt = w.vis[1].depth;
            double nw = w.vis[1].pair.x;
#pragma unroll 1
            for (int n = 1; n <= NL; ++n) {
                const double2 r1 = n1, r2 = n2, t2 = nt;
                const double w0 = nw;
                if (n < NL) {
                    n1 = w.vis[n + 1].odd;
                    n2 = w.vis[n + 1].even;
                    nw = w.vis[n + 1].pair.x;
                    nt = w.vis[n + 1].depth;
                    prefetch_l1(&lay[1].cbs);
                }
                double lam, gama, am, ap;
                lay4(w0, lay->cbs, lam, gama, am, ap);
                ++lay;
                const double xa = n == 1 ? r1.y : r1.y - r1.x * xprev;
                const double xb = r2.y - r2.x * xa;
                xprev = xb;
                double xk1, xk2;
                unmix(xa, xb, xk1, xk2);
                if (n == 1) {
                    sc[0] = xk1 + gama * xk2 + ap;
                    sc[ROW_BLK] = xk1 * gama + xk2 + am + u0 * f0pi;
                }
                // the middle of the layer; its bottom in the last one
                const double top = n == 1 && n < NL ? a.tce1 : t2.x;
                const double at = n < NL ? t2.y : a.tau;
                const double ep = exp_r(dmin(TAUMAX, lam * (at - top))), em = rcp_n(ep);
                const double et = beam(n < NL ? at : dmin(at, TAUMAX), u0, rcp_u0);
                fmp[(size_t)(n - 1) * ROW_BLK] = xk1 * ep + gama * xk2 * em + ap * et;
                const double m = xk1 * ep * gama + xk2 * em + am * et;
                if (n == NL) sc[2 * ROW_BLK] = m;
                fmm[(size_t)(n - 1) * ROW_BLK] = m + u0 * f0pi * et;
            }
            return true;
        }
    }
    general_vis<2, F32>(sg, c, t, block, max_nl, K, kv, kvf, w.g, fmp, fmm, sc);
    return true;
}

}  // namespace fp64
}  // namespace mgcm
